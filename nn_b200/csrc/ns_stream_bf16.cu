// bf16 product for the few rows of a decoding step: the weights go from global memory straight into registers as the A operand
// of mma.sync, the activations lie in shared memory, K is summed inside the CTA and the epilogue runs in the same launch.
//
// What bounds the product is the weight stream, N * K * 2 bytes.  The tcgen05 kernel of ns_gemm_tc.cu reaches the stream's rate only
// over long loops; with few rows it is a chain of round trips (TMA of the activations, MMA, accumulator read, store of partial sums)
// whose time does not depend on the rows, its 128-column tiles leave SMs without one, and filling the SMs by splitting K makes the
// row kernel behind it read up to eight slabs.  Here the chain is: load, multiply, add across warps, store, and there is one slab.
//
// Work split.  A tile is 16 output columns (16 weight rows); a CTA takes a contiguous range of tiles.  A unit is a tile's 16 rows by
// 128 elements of K: eight 16-byte loads per lane.  The units of a CTA, numbered tile by tile, are dealt to its warps in equal
// contiguous shares (whatever N and K are, the shares differ by one unit), so a warp walks along rows and meets a tile's end a few times
// at most; each meeting leaves its sums in a shared-memory slot of their own (slot tile + warp: both only grow along the units).
// Every register is refilled as soon as it is used, so a warp keeps two units in flight: 128 KB per SM, the latency of HBM times its
// rate with room to spare.  After one barrier, a thread per output adds the warps' slots in their order (fixed by N and K alone, so a
// row's result does not depend on the other rows) and applies the epilogue.
//
// Fragments.  In m16n8k16 a lane (g = lane / 4, q = lane % 4) holds the k of words 2q, 2q + 1 and 2q + 8, 2q + 9 of weight rows g and
// g + 8 and of activation row g.  Any permutation of k may be applied to both operands: a lane takes 16 consecutive bytes of its
// rows and of its activation row, words 0, 1 for one MMA and 2, 3 for the next.  A row of activations takes 64 bytes more than its
// length (a multiple of 128) in shared memory, so the 16-byte reads of a quarter warp (two rows of 64 bytes) meet every bank once.
#include "ns_gemm.cuh"
#include "ns_mma.cuh"

namespace {

constexpr int SB_WARPS = 16;
constexpr int SB_THREADS = SB_WARPS * 32;
constexpr int SB_TILE = 16;          // output columns per tile
constexpr int SB_UNIT = 128;         // elements of K per unit
constexpr int SB_PITCH = 20;         // floats per activation row of a slot (16 columns): 8 q + g meets every bank once
constexpr size_t SB_SMEM_MAX = 164 * 1024;    // see ns_stream_bf16_fits

__host__ __device__ constexpr int sb_slot_floats(int groups) { return groups * 8 * SB_PITCH; }

__device__ __forceinline__ uint4 sb_load_stream(const uint16_t* ptr)
{
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(ptr));
    return v;
}

// Where a warp's loads are: tile, slice of K, and the addresses of this lane's two rows.
struct SbCursor {
    int tile, slice;
    const uint16_t *lo, *hi;
};

// ROWS8: groups of eight activation rows (M <= 8 ROWS8).
template <int ROWS8>
__global__ void __launch_bounds__(SB_THREADS, 1)
ns_stream_bf16_kernel(const NsGemmParams p, const uint16_t* __restrict__ a, const uint16_t* __restrict__ w)
{
    extern __shared__ __align__(128) uint8_t sb_smem[];
    constexpr int SLOT = sb_slot_floats(ROWS8);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, q = lane & 3;
    const int n_tiles = (p.N + SB_TILE - 1) / SB_TILE;
    const int tile_begin = (int)((int64_t)blockIdx.x * n_tiles / gridDim.x);
    const int tile_end = (int)((int64_t)(blockIdx.x + 1) * n_tiles / gridDim.x);
    const int slices = (p.K + SB_UNIT - 1) / SB_UNIT;
    const int units = (tile_end - tile_begin) * slices;
    const int warps = units < SB_WARPS ? units : SB_WARPS;        // fewer units than warps: one each, the rest idle
    const int u0 = warp < warps ? warp * units / warps : units, u1 = warp < warps ? (warp + 1) * units / warps : units;

    const int a_pitch = slices * SB_UNIT + 32;                     // elements
    uint16_t* sa = reinterpret_cast<uint16_t*>(sb_smem);
    float* slots = reinterpret_cast<float*>(sb_smem + (size_t)ROWS8 * 8 * a_pitch * 2);

    SbCursor ld;
    ld.tile = tile_begin + u0 / slices;
    ld.slice = u0 % slices;
    auto rows_of = [&](SbCursor& c) {
        // rows past N repeat the last row (their columns are never stored)
        c.lo = w + (size_t)min(c.tile * SB_TILE + g, p.N - 1) * p.K + q * 8;
        c.hi = w + (size_t)min(c.tile * SB_TILE + g + 8, p.N - 1) * p.K + q * 8;
    };
    rows_of(ld);
    const uint4 zero = make_uint4(0, 0, 0, 0);
    uint4 b0[8], b1[8];
    // piece c of the unit at the cursor: 32 elements of both rows
    auto load_piece = [&](uint4 (&buf)[8], int c, bool there) {
        const int k = ld.slice * SB_UNIT + c * 32;
        const bool ok = there && k + q * 8 < p.K;
        buf[2 * c] = ok ? sb_load_stream(ld.lo + k) : zero;
        buf[2 * c + 1] = ok ? sb_load_stream(ld.hi + k) : zero;
    };
    auto next_unit = [&]() {
        if (++ld.slice == slices) { ld.slice = 0; ld.tile++; rows_of(ld); }
    };
    auto fill = [&]() {
#pragma unroll
        for (int c = 0; c < 4; c++) load_piece(b0, c, u0 < u1);
        next_unit();
#pragma unroll
        for (int c = 0; c < 4; c++) load_piece(b1, c, u0 + 1 < u1);
        next_unit();
    };
    // A Linear's weights are written by no kernel on the stream: the first two units are requested while the kernel before this one
    // is still running.  A caller's own operands wait.
    if (p.prefetch_b) fill();
    ns_pdl_wait();
    ns_pdl_trigger();
    a = ns_after_wait(a);
    const float* bias = ns_after_wait(p.bias);              // a product's bias may be the previous kernel's, too
    if (!p.prefetch_b) fill();

    // activations to shared memory, zeros behind K
    {
        const int pieces = slices * (SB_UNIT / 8);
        for (int i = threadIdx.x; i < p.M * pieces; i += SB_THREADS) {
            const int m = i / pieces, k = (i - m * pieces) * 8;
            if (k < p.K) ns_cp_async16(ns_smem_u32(sa + (size_t)m * a_pitch + k), a + (size_t)m * p.K + k);
            else *reinterpret_cast<uint4*>(sa + (size_t)m * a_pitch + k) = zero;
        }
        ns_cp_commit();
        ns_cp_wait<0>();
    }
    __syncthreads();

    float acc[ROWS8][4];
#pragma unroll
    for (int r = 0; r < ROWS8; r++)
#pragma unroll
        for (int i = 0; i < 4; i++) acc[r][i] = 0.0f;
    int tile = tile_begin + u0 / slices, slice = u0 % slices;
    // one unit out of `buf`, which is refilled with the unit two further on
    auto unit = [&](uint4 (&buf)[8], int u) {
        const uint16_t* x = sa + (size_t)g * a_pitch + slice * SB_UNIT + q * 8;
#pragma unroll
        for (int c = 0; c < 4; c++) {
            const uint32_t f0[4] = {buf[2 * c].x, buf[2 * c + 1].x, buf[2 * c].y, buf[2 * c + 1].y};
            const uint32_t f1[4] = {buf[2 * c].z, buf[2 * c + 1].z, buf[2 * c].w, buf[2 * c + 1].w};
#pragma unroll
            for (int r = 0; r < ROWS8; r++) {
                const uint4 xv = *reinterpret_cast<const uint4*>(x + (size_t)r * 8 * a_pitch + c * 32);
                ns_mma_bf16(acc[r], f0, xv.x, xv.y);
                ns_mma_bf16(acc[r], f1, xv.z, xv.w);
            }
            load_piece(buf, c, u + 2 < u1);
        }
        next_unit();
        if (++slice == slices || u + 1 == u1) {
            // the tile's or the share's end: sums of this warp, [activation row][column]
            float* mine = slots + (size_t)(tile - tile_begin + warp) * SLOT;
#pragma unroll
            for (int r = 0; r < ROWS8; r++) {
                float* at = mine + (r * 8 + 2 * q) * SB_PITCH + g;
                at[0] = acc[r][0]; at[SB_PITCH] = acc[r][1]; at[8] = acc[r][2]; at[SB_PITCH + 8] = acc[r][3];
#pragma unroll
                for (int i = 0; i < 4; i++) acc[r][i] = 0.0f;
            }
            slice = 0;
            tile++;
        }
    };
    for (int u = u0; u < u1; u += 2) {
        unit(b0, u);
        if (u + 1 < u1) unit(b1, u + 1);
    }
    __syncthreads();

    const int cols = min(tile_end * SB_TILE, p.N) - tile_begin * SB_TILE;
    for (int e = threadIdx.x; e < cols * p.M; e += SB_THREADS) {
        const int m = e / cols, c = e - m * cols;
        const int t = c / SB_TILE;
        // the warps that met this tile: unit x belongs to warp (warps (x + 1) - 1) / units
        const int first = (warps * (t * slices + 1) - 1) / units, last = (warps * ((t + 1) * slices) - 1) / units;
        const float* src = slots + (size_t)(t + first) * SLOT + m * SB_PITCH + (c - t * SB_TILE);
        float v = *src;
        for (int i = first; i < last; i++) {
            src += SLOT;
            v = __fadd_rn(v, *src);
        }
        const int n = tile_begin * SB_TILE + c;
        const size_t at = (size_t)m * p.N + n;
        if (p.epilogue != NS_EPI_NONE) v = __fadd_rn(v, __ldg(&bias[n]));
        if (p.epilogue == NS_EPI_BIAS_GELU) v = ns_gelu_fast(v);
        if (p.epilogue == NS_EPI_BIAS_RESIDUAL) v = __fadd_rn(v, ns_gemm_residual(p, at));
        if (p.out_dtype == NS_F32) reinterpret_cast<float*>(p.out)[at] = v;
        else reinterpret_cast<uint16_t*>(p.out)[at] = ns_f32_to_bf16_bits(v);
    }
}

size_t sb_smem_bytes(int sm_count, int groups, int N, int K)
{
    const int tiles = (N + SB_TILE - 1) / SB_TILE, grid = tiles < sm_count ? tiles : sm_count;
    const int most = (tiles + grid - 1) / grid;                    // tiles of one CTA
    const size_t pitch = (size_t)(K + SB_UNIT - 1) / SB_UNIT * SB_UNIT + 32;
    return (size_t)groups * 8 * pitch * 2 + (size_t)(most + SB_WARPS - 1) * sb_slot_floats(groups) * 4;
}

template <int ROWS8>
int launch_stream_bf16(NsDevice* d, const NsGemmParams& p, const void* a, const void* w)
{
    auto kernel = ns_stream_bf16_kernel<ROWS8>;
    static bool configured[64] = {false};
    if (!configured[d->ordinal]) {
        NS_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SB_SMEM_MAX));
        configured[d->ordinal] = true;
    }
    const int tiles = (p.N + SB_TILE - 1) / SB_TILE, grid = tiles < d->sm_count ? tiles : d->sm_count;
    NS_CUDA(ns_launch_pdl(kernel, dim3((unsigned)grid), dim3(SB_THREADS), sb_smem_bytes(d->sm_count, ROWS8, p.N, p.K), d->stream, p,
                          reinterpret_cast<const uint16_t*>(a), reinterpret_cast<const uint16_t*>(w)));
    return NS_OK;
}

}  // namespace

// Up to eight rows: every size whose activations and slots leave L1 a quarter of an SM's 256 KB, because the weights in flight (128 KB
// a SM at most) pass through it.  us, tcgen05 against this, 1 and 8 rows:
//   2048 x 8192 11.5, 7.5 and 11.6, 8.7;  4096 x 9216 17.9, 14.4 and 18.1, 15.6;  4096 x 11264 20.1, 19.7 and 20.5, 21.2;  4096 x 12288 21.6, 37.1 and 22.1, 38.8
// Not where tiles divide badly and K is long: the bytes of weights that the busiest CTA has beyond an even share are time in which the others
// wait.  In front of a row kernel, which reads split sums almost as fast as whole ones, the tcgen05 kernel is ahead sooner.  (With the row kernel) 8 rows:
//   4096 x 4096 (34 KB) 13.6, 12.4;  768 x 8192 (172 KB) 9.1, 9.4;  1024 x 8192 (145 KB) 9.2, 9.8;  2400 x 4096 (126 KB) 10.7, 11.0;  2400 x 5120 (157 KB) 11.3, 12.0
//   2400 x 8192 (252 KB) 13.6, 16.2, and alone 12.2, 13.3;  3000 x 8192 (186 KB) alone 13.4, 13.0
// (One row would gain up to 220 KB, 768 x 8192 9.1, 8.3, and with many columns, 64000 x 1024 24.9, 23.0; but one line for one to eight rows keeps a row's
// bits the same among them.)
// Not many columns over rows of 512 to 1024, where a CTA's 2 400 outputs and more, which it adds up after its last weights, are not made up for: 8 rows
// 100000 x 512 20.8, 23.6;  128256 x 1024 45.1, 48.9;  64000 x 1024 25.7, 26.6;  32000 x 1024 14.2, 14.0.  Shorter rows are tiles of one or two steps to the
// tcgen05 kernel (200000 x 128 25.1, 18.2;  50000 x 256 11.3, 8.8), longer ones weigh more than the outputs (64000 x 2048 47.6, 46.5;  128256 x 4096 174, 167).
// Nine to sixteen rows: short rows and few columns only.  There the tcgen05 kernel is as fast or faster elsewhere, because a CTA of this one copies
// all the activations (16 x 5632: 180 KB) and adds the sums of all its tiles before anything is stored.  With the row kernel that follows, us:
//   8 rows:  2048 x 2048 7.1, 6.4;  11264 x 2048 16.8, 15.2;  2048 x 5632 9.3, 9.4;  32000 x 5632 65.5, 61.0 (floor 55.8);  1 row: 64.4, 58.1
//   16 rows: 2048 x 2048 7.7, 7.0;  3088 x 1024 8.6, 7.6;  3088 x 2048 10.1, 9.3;  4096 x 2048 10.4, 10.1;  6176 x 2048 11.9, 12.3;  32000 x 2048 28.1, 29.7
//            2048 x 5632 9.3, 14.3;  2400 x 2048 (63 KB) 8.6, 8.8;  2600 x 2048 (57 KB) 9.0, 8.7
// In a chain of products alone (8 rows): 12.4, 9.4;  7.1, 3.8;  9.5, 6.3 us (11264 x 2048, 2048 x 2048, 2048 x 5632); 14336 x 4096 23.5, 20.8; 16 rows
// of 4096 x 2048 8.3, 5.7, of 3088 x 1024 6.8, 4.1.
bool ns_stream_bf16_fits(const NsDevice* d, int M, int N, int K, bool deferred)
{
    if (M < 1 || M > 16 || K % 8 != 0) return false;
    if (M > 8 && (K > 2048 || N > 4096)) return false;
    if (sb_smem_bytes(d->sm_count, M <= 8 ? 1 : 2, N, K) > SB_SMEM_MAX) return false;
    const int64_t tiles = (N + SB_TILE - 1) / SB_TILE, most = (tiles + d->sm_count - 1) / d->sm_count;
    if (M <= 8 && K > 256 && K < 2048 && most * SB_TILE * 8 > 2400) return false;
    const int64_t beyond = (most * d->sm_count - tiles) * K * (SB_TILE * 2) / d->sm_count;     // bytes
    return beyond <= (!deferred ? 230 : M <= 8 ? 120 : 62) * 1024;
}

int ns_stream_bf16_run(NsDevice* d, const NsGemmParams& p, const void* a, const void* w)
{
    return p.M <= 8 ? launch_stream_bf16<1>(d, p, a, w) : launch_stream_bf16<2>(d, p, a, w);
}
