// Causal (or full) attention forward for whole sequences, head_dim 128, bf16 in / bf16 out, on the sm_100a tensor cores.
// Q/K/V tiles arrive by TMA, S = Q.K^T and O += P.V are tcgen05.mma with accumulators in tensor memory, the softmax is
// computed online (running maximum and sum per row), so the [T, T] score tensor never exists.
//
// Reference path: MultiHeadAttention.ForwardCore (src/NeuralSharp/Layers/Attention.cs:46-91): three
// narrow+permute copies, matmul_f32 (Q.K^T) into a [N*H, T, T] tensor, scale_mask_softmax_f32 with an
// additive -1e9 mask (one thread per row, PtxKernels.Decoding.cs:24-58), matmul_f32 (P.V), permute back.
// Skipping the key blocks above the diagonal is exact: exp(-1e9 - max) is 0 in float.  The head
// split/merge copies disappear because the tensor maps take the (batch, head, position) strides of
// the caller's buffers.
//
// A tile is (batch, head, 256 query rows); 384 threads, one persistent CTA per SM:
//   warp 0       loads K and V blocks of 128 keys into rings of two slots, for both groups
//   warps 1, 2   issue the MMAs of group 0 and of group 1: O += P.V of a block, then S = Q.K^T of the next
//   warp 3       draws the tiles, hands them to the other roles and loads each group's Q
//   warps 4..11  softmax, two groups of four warps.  Group g owns the tile's query rows [128 g, 128 g + 128): thread r owns
//                row r (= tensor-memory lane r), reads its 128 scores, masks, updates maximum and sum, writes P as bf16 over the
//                scores in tensor memory, from where P.V takes it (each half of the keys as soon as it is there), and rescales O
//                when the row maximum outgrew the reference maximum (the old one may stay: sum and O share it).
// The groups share nothing but the K/V blocks: while one group's MMAs run the other computes exponentials, and one reads out its
// result and begins its next tile while the other is inside a tile.
// What bounds it.  For 128 rows x 128 keys the exponential unit and the tensor pipe need 1 024 cycles each, and shared memory
// (128 bytes a cycle) what is read and written there: Q.K^T 512, V 256, the loads of a K/V block for 256 rows 256.  The form with 128
// rows a tile, its key blocks dealt to the two groups and P in shared memory needed 1 792 there, and merged two results at each
// tile's end.  Against it (same B200, 8 x 32 heads x 2048: us a launch): 369 -> 300; 2 x 32 x 8192: 1 102 -> 1 013; 64 x 16 x 512:
// 186 -> 125; 13 x 16 x 777: 90 -> 74.  It still takes about 1 950 cycles a block: the softmax of a block is 2 000 cycles of one warp's
// instructions, then its P.V and next Q.K^T 1 000.  Measured on the way: blocks of 64 keys with S and two P buffers
// side by side (the next scores ahead of the exponentials): 318 and 1 089; the same with two warps a row: 355 and 1 212; every fourth
// exponential as a polynomial instead of every eighth: level, none: 308 and 1 056.
// Tensor memory of group g: O at columns [256 g, 256 g + 128), S the next 128.
// Every mbarrier wait is bounded; a wait that runs out reports a status code and the CTA leaves.
#include <math.h>

#include <algorithm>

#include "ns_common.cuh"

namespace {

constexpr int PA_THREADS = 384;
constexpr int PA_KB = 128;                             // keys a block
constexpr int PA_SLOTS = 2;
constexpr int PA_EARLY = 4;                            // blocks in which every growth of the maximum is followed
constexpr int PA_POLY = 8;                             // every eighth pair of exponentials is computed on the multiply-add pipe
constexpr uint32_t PA_Q_BYTES = 128 * 128 * 2;         // a group's queries: two [128 x 64] halves
constexpr uint32_t PA_Q_HALF = PA_Q_BYTES / 2;
constexpr uint32_t PA_KV_BYTES = PA_KB * 128 * 2;      // two [128 x 64] halves
constexpr uint32_t PA_KV_HALF = PA_KV_BYTES / 2;
constexpr uint32_t PA_STAGE_BYTES = 32 * 64 * 2;       // a softmax warp's 32 rows x 64 columns on their way out
constexpr uint32_t PA_K_AT = 2 * PA_Q_BYTES;
constexpr uint32_t PA_V_AT = PA_K_AT + PA_SLOTS * PA_KV_BYTES;
constexpr uint32_t PA_STAGE_AT = PA_V_AT + PA_SLOTS * PA_KV_BYTES;
constexpr uint32_t PA_BAR_AT = PA_STAGE_AT + 8 * PA_STAGE_BYTES;
constexpr uint32_t PA_SMEM_BYTES = 1024 + PA_BAR_AT + 512;
constexpr uint32_t PA_S_COL = 128;                     // O at 0; P_j lies over the first half of S_j
static_assert(PA_SMEM_BYTES <= 232448, "shared memory of an SM");

struct PaParams {
    int batch, heads, seq;
    int causal;
    int heads_run;       // (batch, head) pairs whose tiles are drawn together
    float scale_log2;    // scale * log2(e)
    int* status;
    int* tile_counter;   // tiles drawn beyond each CTA's first; zeroed before the launch where there are any
};

struct PaMaps {
    CUtensorMap q;       // box [64 dims, 128 rows]
    CUtensorMap k, v;    // box [64 dims, 128 rows]
    CUtensorMap o;       // box [64 dims, 32 rows]
};

enum { PB_Q_FULL = 0, PB_Q_EMPTY = 2, PB_K_FULL = 4, PB_K_EMPTY = PB_K_FULL + PA_SLOTS, PB_V_FULL = PB_K_EMPTY + PA_SLOTS, PB_V_EMPTY = PB_V_FULL + PA_SLOTS,
       PB_S_FULL = PB_V_EMPTY + PA_SLOTS, PB_P_FULL = PB_S_FULL + 2, PB_O_DONE = PB_P_FULL + 4, PB_TILE_FULL = PB_O_DONE + 2, PB_TILE_EMPTY = PB_TILE_FULL + 2,
       PB_COUNT = PB_TILE_EMPTY + 2 };
static_assert(PB_COUNT * 8 + 16 <= 512, "barriers");

__device__ __forceinline__ float pa_exp2(float x)
{
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// maxima of which a NaN is one
__device__ __forceinline__ float pa_max3(float a, float b, float c)
{
    float y;
    asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(y) : "f"(a), "f"(b), "f"(c));
    return y;
}
__device__ __forceinline__ float pa_max2(float a, float b)
{
    float y;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(y) : "f"(a), "f"(b));
    return y;
}
__device__ __forceinline__ uint64_t pa_pair(float lo, float hi)
{
    uint64_t y;
    asm("mov.b64 %0, {%1, %2};" : "=l"(y) : "f"(lo), "f"(hi));
    return y;
}
__device__ __forceinline__ void pa_split(uint64_t v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
// two sums, two fused multiply-adds: each rounded as the single ones are
__device__ __forceinline__ uint64_t pa_add2(uint64_t a, uint64_t b)
{
    uint64_t y;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(y) : "l"(a), "l"(b));
    return y;
}
__device__ __forceinline__ uint64_t pa_fma2(uint64_t a, uint64_t b, uint64_t c)
{
    uint64_t y;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(y) : "l"(a), "l"(b), "l"(c));
    return y;
}
// The maximum of a row's scores; NaN where one of them is.
__device__ __forceinline__ float pa_row_max(const float (&s)[PA_KB])
{
    float m[8];
#pragma unroll
    for (int q = 0; q < 8; q++) m[q] = s[q];
#pragma unroll
    for (int c = 8; c + 16 <= PA_KB; c += 16)
#pragma unroll
        for (int q = 0; q < 8; q++) m[q] = pa_max3(m[q], s[c + 2 * q], s[c + 2 * q + 1]);
#pragma unroll
    for (int q = 0; q < 8; q++) m[q] = pa_max2(m[q], s[PA_KB - 8 + q]);
    return pa_max3(pa_max3(m[0], m[1], m[2]), pa_max3(m[3], m[4], m[5]), pa_max2(m[6], m[7]));
}

// 2^x of two values on the multiply-add pipe, x <= 126: x = n + f with f in [-1/2, 1/2], 2^f as the polynomial of degree 5 with the
// least relative error under p(0) = 1 (a linear programme over 4001 points of the interval; 2^-22.5 with float rounding, ex2.approx
// states 2^-22), n added to the exponent.  x at or below -127 (a masked score) gives 0, and so does a NaN: see neg_m.
__device__ __forceinline__ void pa_exp2_pair(uint64_t x, float& y0, float& y1)
{
    float x0, x1;
    pa_split(x, x0, x1);
    x = pa_pair(fmaxf(x0, -127.0f), fmaxf(x1, -127.0f));
    const uint64_t shift = pa_pair(12582912.0f, 12582912.0f);         // 1.5 * 2^23: the sum's low bits are the rounded value
    const uint64_t t = pa_add2(x, shift);
    const uint64_t n = pa_add2(t, pa_pair(-12582912.0f, -12582912.0f));
    const uint64_t f = pa_fma2(n, pa_pair(-1.0f, -1.0f), x);
    uint64_t y = pa_fma2(f, pa_pair(0.0013264653f, 0.0013264653f), pa_pair(0.009671511f, 0.009671511f));
    y = pa_fma2(y, f, pa_pair(0.05550734f, 0.05550734f));
    y = pa_fma2(y, f, pa_pair(0.24022242f, 0.24022242f));
    y = pa_fma2(y, f, pa_pair(0.693147f, 0.693147f));
    y = pa_fma2(y, f, pa_pair(1.0f, 1.0f));
    float t0, t1;
    pa_split(t, t0, t1);
    pa_split(y, y0, y1);
    y0 = __int_as_float(__float_as_int(y0) + (__float_as_int(t0) << 23));
    y1 = __int_as_float(__float_as_int(y1) + (__float_as_int(t1) << 23));
}

// P = 2^(s scale + neg_m) of 64 scores as pairs of bf16; the sums of P before that rounding go onto `sum`.
template <int FIRST>
__device__ __forceinline__ void pa_exponentials(const float (&s)[PA_KB], float scale, float neg_m, uint64_t (&sum)[2], uint32_t (&pk)[32])
{
    const uint64_t scale2 = pa_pair(scale, scale), neg2 = pa_pair(neg_m, neg_m);
#pragma unroll
    for (int c = 0; c < 32; c++) {
        const uint64_t x = pa_fma2(pa_pair(s[FIRST + 2 * c], s[FIRST + 2 * c + 1]), scale2, neg2);
        float p0, p1;
        if (c % PA_POLY == PA_POLY - 1) {
            pa_exp2_pair(x, p0, p1);
        } else {
            // one MUFU each (results below 2^-126 flush to zero, which is what P wants)
            pa_split(x, p0, p1);
            p0 = pa_exp2(p0);
            p1 = pa_exp2(p1);
        }
        sum[c & 1] = pa_add2(sum[c & 1], pa_pair(p0, p1));
        pk[c] = ns_pack_bf16x2(p0, p1);
    }
}

// D[tmem] (+)= A[tmem] * B[smem]
__device__ __forceinline__ void pa_mma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// Tiles are drawn in this order: from `heads_run` (batch, head) pairs at a time, the late query rows (which see more keys) first and those
// of one position together.  CTAs that run together then read the same K/V blocks out of L2, and what is left at the end of a run are
// small tiles (with the tiles of one head adjacent, 64 heads x 4096 left the SMs idle 15 % of the time).
template <bool SOLO>
struct PaTile {
    static constexpr int rows = SOLO ? 128 : 256;
    int b, h, q0;
    int n, n0, n1;       // key blocks: of the tile, of each group's rows
    __device__ __forceinline__ int of(int g) const { return g == 0 ? n0 : n1; }
};
template <bool SOLO>
__device__ __forceinline__ void pa_tile(const PaParams& p, int idx, PaTile<SOLO>& t)
{
    const int n_qt = (p.seq + t.rows - 1) / t.rows;
    const int per = p.heads_run * n_qt, first = idx / per * p.heads_run, in = idx - first * n_qt;
    const int heads_here = min(p.heads_run, p.batch * p.heads - first);
    const int bh = first + in % heads_here;
    t.b = bh / p.heads;
    t.h = bh % p.heads;
    t.q0 = (n_qt - 1 - in / heads_here) * t.rows;
    auto blocks = [&](int g) {
        const int first = t.q0 + 128 * g, end = min(first + 128, p.seq);
        return first < p.seq && 128 * g < t.rows ? ((p.causal ? end : p.seq) + PA_KB - 1) / PA_KB : 0;
    };
    t.n0 = blocks(0);
    t.n1 = blocks(1);
    t.n = max(t.n0, t.n1);
}

// a position in a ring of slots and the phase of its barriers
template <int SLOTS>
struct PaRing {
    int s = 0;
    uint32_t phase = 0;
    __device__ __forceinline__ void next()
    {
        if (++s == SLOTS) { s = 0; phase ^= 1u; }
    }
};

// SOLO: a tile of 128 rows is one group's, and the CTA's only one.  The scores of the next block then go where the other group's would be,
// ahead of this block's P.V, and the blocks take turns with both groups' barriers.
template <bool SOLO>
__global__ void __launch_bounds__(PA_THREADS, 1) ns_attention_prompt_kernel(const __grid_constant__ PaMaps maps, const PaParams p)
{
    extern __shared__ uint8_t smem_raw[];
    __shared__ int abort_flag_storage;
    volatile int* abort_flag = &abort_flag_storage;
    const uint32_t smem_base = (ns_smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t bar_base = smem_base + PA_BAR_AT;
    auto bar = [&](int i) { return bar_base + 8u * i; };
    const uint32_t tile_words = bar(PB_COUNT), tmem_slot = tile_words + 8;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    using Tile = PaTile<SOLO>;
    const int total = p.batch * p.heads * ((p.seq + Tile::rows - 1) / Tile::rows);

    if (threadIdx.x == 0) {
        abort_flag_storage = 0;
        for (int i = 0; i < 2; i++) {
            ns_mbar_init(bar(PB_Q_FULL + i), 1);
            ns_mbar_init(bar(PB_Q_EMPTY + i), 1);
            ns_mbar_init(bar(PB_S_FULL + i), 1);
            ns_mbar_init(bar(PB_O_DONE + i), 1);
            ns_mbar_init(bar(PB_TILE_FULL + i), 1);
            ns_mbar_init(bar(PB_TILE_EMPTY + i), 11);   // every warp but the one that draws
        }
        for (int i = 0; i < PA_SLOTS; i++) {
            ns_mbar_init(bar(PB_K_FULL + i), 1);
            ns_mbar_init(bar(PB_K_EMPTY + i), 2);
            ns_mbar_init(bar(PB_V_FULL + i), 1);
            ns_mbar_init(bar(PB_V_EMPTY + i), 2);
        }
        for (int i = 0; i < 4; i++) ns_mbar_init(bar(PB_P_FULL + i), 4);
        ns_fence_barrier_init();
        ns_fence_proxy_async();
        ns_prefetch_tensormap(&maps.q);
        ns_prefetch_tensormap(&maps.k);
        ns_prefetch_tensormap(&maps.v);
        ns_prefetch_tensormap(&maps.o);
    }
    if (warp == 1) {
        ns_tmem_alloc(tmem_slot, 512);
        ns_tmem_relinquish();
    }
    ns_tc_fence_before();
    __syncthreads();
    ns_tc_fence_after();
    uint32_t tmem_base;
    asm volatile("ld.shared.b32 %0, [%1];" : "=r"(tmem_base) : "r"(tmem_slot));
    tmem_base = __shfl_sync(0xffffffffu, tmem_base, 0);
    const int code = 320;
    auto wait = [&](int i, uint32_t parity, int what) { return ns_mbar_wait_warp(bar(i), parity & 1u, abort_flag, p.status, code + what); };
    // the it-th tile of this CTA, by a whole warp; false after the last one
    auto next_tile = [&](int it, Tile& t) {
        if (!wait(PB_TILE_FULL + (it & 1), it >> 1, 1)) return false;
        int idx;
        asm volatile("ld.shared.b32 %0, [%1];" : "=r"(idx) : "r"(tile_words + 4u * (it & 1)) : "memory");
        idx = __shfl_sync(0xffffffffu, idx, 0);
        if (lane == 0) ns_mbar_arrive(bar(PB_TILE_EMPTY + (it & 1)));
        if (idx < 0) return false;
        pa_tile(p, idx, t);
        return true;
    };

    // 168 registers a thread at launch; the softmax warps take what the other four give back: 72 + 2 x 216 = 3 x 168
    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
        if (warp == 0) {
            // ------------------------------------------------------------ K and V
            const bool leader = ns_elect();
            PaRing<PA_SLOTS> ring;
            Tile t;
            bool ok = true;
            for (int it = 0; ok && next_tile(it, t); it++)
                for (int j = 0; j < t.n; j++, ring.next()) {
                    ok = wait(PB_K_EMPTY + ring.s, ring.phase ^ 1u, 2);
                    if (!ok) break;
                    if (leader) {
                        const uint32_t dst = smem_base + PA_K_AT + ring.s * PA_KV_BYTES;
                        ns_mbar_expect_tx(bar(PB_K_FULL + ring.s), PA_KV_BYTES);
                        ns_tma_load_4d(dst, &maps.k, bar(PB_K_FULL + ring.s), 0, j * PA_KB, t.h, t.b);
                        ns_tma_load_4d(dst + PA_KV_HALF, &maps.k, bar(PB_K_FULL + ring.s), 64, j * PA_KB, t.h, t.b);
                    }
                    ok = wait(PB_V_EMPTY + ring.s, ring.phase ^ 1u, 3);
                    if (!ok) break;
                    if (leader) {
                        const uint32_t dst = smem_base + PA_V_AT + ring.s * PA_KV_BYTES;
                        ns_mbar_expect_tx(bar(PB_V_FULL + ring.s), PA_KV_BYTES);
                        ns_tma_load_4d(dst, &maps.v, bar(PB_V_FULL + ring.s), 0, j * PA_KB, t.h, t.b);
                        ns_tma_load_4d(dst + PA_KV_HALF, &maps.v, bar(PB_V_FULL + ring.s), 64, j * PA_KB, t.h, t.b);
                    }
                }
        } else if (warp < 3) {
            // ------------------------------------------------------------ MMAs of one group
            const int g = warp - 1;
            const bool leader = ns_elect();
            constexpr uint32_t idesc_qk = ns_idesc(1, 1, 0, 0, 128, PA_KB), idesc_pv = ns_idesc(1, 1, 0, 1, 128, 128);
            const uint64_t desc_k = ns_desc_base(16, 1024);
            const uint64_t desc_v = ns_desc_base(PA_KV_HALF, 1024);   // MN-major: the halves of 64 columns, 8 key rows 1 KB apart
            const uint32_t o_tmem = tmem_base + 256 * g, q_smem = smem_base + PA_Q_BYTES * g;
            PaRing<PA_SLOTS> kr, vr;
            int nq = 0, ks = 0, kp = 0;   // tiles in which the group had rows, score blocks and P.V products so far
            bool ok = true;
            Tile t;
            auto scores = [&](bool last) {
                ok = wait(PB_K_FULL + kr.s, kr.phase, 4);
                if (!ok) return;
                ns_tc_fence_after();
                if (leader) {
                    const int side = SOLO ? ks & 1 : g;
                    const uint32_t kb = smem_base + PA_K_AT + kr.s * PA_KV_BYTES, s_tmem = tmem_base + 256 * side + PA_S_COL;
#pragma unroll
                    for (int kk = 0; kk < 8; kk++)
                        ns_mma_f16(s_tmem, ns_desc_at(desc_k, q_smem + (kk >> 2) * PA_Q_HALF + (kk & 3) * 32),
                                   ns_desc_at(desc_k, kb + (kk >> 2) * PA_KV_HALF + (kk & 3) * 32), idesc_qk, kk > 0 ? 1u : 0u);
                    ns_tc_commit(bar(PB_S_FULL + side));
                    ns_tc_commit(bar(PB_K_EMPTY + kr.s));
                    if (last) ns_tc_commit(bar(PB_Q_EMPTY + g));
                }
                kr.next();
                ks++;
            };
            for (int it = 0; ok && next_tile(it, t); it++) {
                const int n = t.of(g);
                if (n > 0) {
                    // the scores of a block follow the P.V of the block before in the tensor pipe, which has then read P and finished O
                    ok = wait(PB_Q_FULL + g, nq++, 6);
                    if (ok) scores(n == 1);
                }
                for (int j = 0; j < n && ok; j++, kp++) {
                    const int side = SOLO ? kp & 1 : g;
                    if (SOLO && j + 1 < n) scores(j + 2 == n);
                    ok = ok && wait(PB_V_FULL + vr.s, vr.phase, 8);
#pragma unroll
                    for (int hf = 0; hf < 2; hf++) {
                        ok = ok && wait(PB_P_FULL + 2 * side + hf, kp >> (SOLO ? 1 : 0), 7);
                        if (!ok) break;
                        ns_tc_fence_after();
                        if (leader) {
                            const uint32_t vb = smem_base + PA_V_AT + vr.s * PA_KV_BYTES + hf * (64 * 128), pa = tmem_base + 256 * side + PA_S_COL + hf * 32;
#pragma unroll
                            for (int kk = 0; kk < 4; kk++)
                                pa_mma_ts(o_tmem, pa + kk * 8, ns_desc_at(desc_v, vb + kk * (16 * 128)), idesc_pv, j > 0 || hf > 0 || kk > 0 ? 1u : 0u);
                        }
                    }
                    if (!ok) break;
                    if (leader) {
                        ns_tc_commit(bar(PB_O_DONE + g));
                        ns_tc_commit(bar(PB_V_EMPTY + vr.s));
                    }
                    vr.next();
                    if (!SOLO && j + 1 < n) scores(j + 2 == n);
                }
                // blocks that only the other group's rows see: given back when they have arrived (an earlier arrival would count for the
                // block before them in the slot)
                for (int j = n; j < t.n && ok; j++) {
                    ok = wait(PB_K_FULL + kr.s, kr.phase, 4);
                    if (ok && leader) ns_mbar_arrive(bar(PB_K_EMPTY + kr.s));
                    kr.next();
                    ok = ok && wait(PB_V_FULL + vr.s, vr.phase, 8);
                    if (ok && leader) ns_mbar_arrive(bar(PB_V_EMPTY + vr.s));
                    vr.next();
                }
            }
        } else if (warp == 3) {
            // ------------------------------------------------------------ tiles and queries
            const bool leader = ns_elect();
            int nq0 = 0, nq1 = 0;     // tiles in which each group had rows (group 0 always has)
            int idx = blockIdx.x;
            auto load_q = [&](int g, const Tile& t) {
                const uint32_t dst = smem_base + PA_Q_BYTES * g;
                ns_mbar_expect_tx(bar(PB_Q_FULL + g), PA_Q_BYTES);
                ns_tma_load_4d(dst, &maps.q, bar(PB_Q_FULL + g), 0, t.q0 + 128 * g, t.h, t.b);
                ns_tma_load_4d(dst + PA_Q_HALF, &maps.q, bar(PB_Q_FULL + g), 64, t.q0 + 128 * g, t.h, t.b);
            };
            for (int it = 0;; it++) {
                // a tile is drawn when the last scores of group 0's tile before have been computed
                if (it > 0) {
                    if (!wait(PB_Q_EMPTY, nq0 - 1, 10)) break;
                    idx = total;
                    if ((int)gridDim.x < total) {          // else every tile was some CTA's first
                        if (lane == 0) idx = gridDim.x + atomicAdd(p.tile_counter, 1);
                        idx = __shfl_sync(0xffffffffu, idx, 0);
                    }
                }
                if (!wait(PB_TILE_EMPTY + (it & 1), (it >> 1) + 1, 9)) break;
                if (leader) {
                    asm volatile("st.shared.b32 [%0], %1;" ::"r"(tile_words + 4u * (it & 1)), "r"(idx < total ? idx : -1) : "memory");
                    ns_mbar_arrive(bar(PB_TILE_FULL + (it & 1)));
                }
                if (idx >= total) break;
                Tile t;
                pa_tile(p, idx, t);
                if (leader) load_q(0, t);
                nq0++;
                if (t.n1 > 0) {
                    if (nq1 > 0 && !wait(PB_Q_EMPTY + 1, nq1 - 1, 10)) break;
                    if (leader) load_q(1, t);
                    nq1++;
                }
            }
        }
    } else {
        // ------------------------------------------------------------ softmax and output
        asm volatile("setmaxnreg.inc.sync.aligned.u32 216;");
        const int g = (warp >> 2) - 1, quad = warp & 3;
        const int r = quad * 32 + lane;
        const uint32_t o_addr = tmem_base + (uint32_t(quad * 32) << 16) + 256 * g;
        const uint32_t stage = smem_base + PA_STAGE_AT + (warp - 4) * PA_STAGE_BYTES;
        int k = 0;                               // blocks of this group so far, over all tiles
        bool ok = true;
        Tile t;
        for (int it = 0; ok && next_tile(it, t); it++) {
            const int n = t.of(g);
            if (n == 0) continue;
            const int row0 = t.q0 + 128 * g;
            const int last_key = p.causal ? min(row0 + r, p.seq - 1) : p.seq - 1;
            float m_ref = -INFINITY;             // reference maximum (raw score units)
            float l_run = 0.0f;                  // sum of the exponentials relative to m_ref
            for (int j = 0; j < n; j++, k++) {
                const int side = SOLO ? k & 1 : g;
                const uint32_t s_addr = o_addr + 256 * (side - g) + PA_S_COL;
                ok = wait(PB_S_FULL + side, k >> (SOLO ? 1 : 0), 11);
                if (!ok) break;
                ns_tc_fence_after();
                float s[PA_KB];
                {
                    uint32_t s0[32], s1[32], s2[32], s3[32];
                    ns_tmem_ld32(s_addr, s0);
                    ns_tmem_ld32(s_addr + 32, s1);
                    ns_tmem_ld32(s_addr + 64, s2);
                    ns_tmem_ld32(s_addr + 96, s3);
                    ns_tc_wait_ld();
#pragma unroll
                    for (int c = 0; c < 32; c++) {
                        s[c] = __uint_as_float(s0[c]); s[32 + c] = __uint_as_float(s1[c]);
                        s[64 + c] = __uint_as_float(s2[c]); s[96 + c] = __uint_as_float(s3[c]);
                    }
                }
                // keys after the query (causal) or past the end of the sequence
                const int kv0 = j * PA_KB;
                if ((p.causal && kv0 + PA_KB - 1 > row0) || kv0 + PA_KB > p.seq) {
                    const int live = last_key - kv0;
#pragma unroll
                    for (int c = 0; c < PA_KB; c++)
                        if (c > live) s[c] = -INFINITY;
                }
                // The reference maximum is raised only when the row maximum outgrew it by more than 8 in units of the exponent -- and in the
                // first 512 keys whenever it grew: the largest weight is then exactly 1, which counts where a row has few keys.
                const float mx = pa_row_max(s);
                float alpha = 1.0f;
                bool rescale = false;
                if (mx != -INFINITY && (m_ref == -INFINITY || !((mx - m_ref) * p.scale_log2 <= (j < PA_EARLY ? 0.0f : 8.0f)))) {
                    alpha = m_ref == -INFINITY ? 0.0f : pa_exp2((m_ref - mx) * p.scale_log2);
                    rescale = m_ref != -INFINITY;
                    m_ref = mx;
                }
                if (j > 0 && __any_sync(0xffffffffu, rescale)) {
                    // O belongs to the last P.V; without SOLO these scores have followed it
                    if (SOLO) {
                        ok = wait(PB_O_DONE + g, k - 1, 13);
                        if (!ok) break;
                        ns_tc_fence_after();
                    }
#pragma unroll 1
                    for (int c = 0; c < 4; c++) {
                        uint32_t ob[32];
                        ns_tmem_ld32(o_addr + c * 32, ob);
                        ns_tc_wait_ld();
#pragma unroll
                        for (int q = 0; q < 32; q++) ob[q] = __float_as_uint(__uint_as_float(ob[q]) * alpha);
                        ns_tmem_st32(o_addr + c * 32, ob);
                    }
                }
                // A score of NaN or +infinity makes a row NaN, whichever key's it is.  Both show in the maximum, which then makes every weight of
                // the row NaN (0 m_ref is NaN, else nothing); keeping them through the polynomial cost 1 to 4 % of a launch.
                const float neg_m = m_ref == -INFINITY ? 0.0f : fmaf(m_ref, 0.0f, -m_ref * p.scale_log2);
                uint64_t sum[2] = {0, 0};
                auto hand_over = [&](int hf, const uint32_t (&pk)[32]) {
                    __syncwarp();
                    ns_tmem_st32(s_addr + hf * 32, pk);
                    ns_tc_wait_st();
                    ns_tc_fence_before();
                    __syncwarp();
                    if (lane == 0) ns_mbar_arrive(bar(PB_P_FULL + 2 * side + hf));
                };
                uint32_t pk[32];
                pa_exponentials<0>(s, p.scale_log2, neg_m, sum, pk);
                hand_over(0, pk);
                pa_exponentials<64>(s, p.scale_log2, neg_m, sum, pk);
                // A wait names a phase by its parity, so O_DONE may be asked neither two phases early nor one late.  With SOLO the last scores come before the
                // P.V of the block in front, which may still wait for another warp's P or for its V: that P.V is waited for here, before this block's own
                // can end, and the read-out then waits for the phase that follows.
                if (SOLO && j > 0 && j + 1 == n) {
                    ok = wait(PB_O_DONE + g, k - 1, 12);
                    if (!ok) break;
                }
                hand_over(1, pk);
                float l0, l1;
                pa_split(pa_add2(sum[0], sum[1]), l0, l1);
                l_run = l_run * alpha + (l0 + l1);
            }
            if (!ok) break;
            ok = wait(PB_O_DONE + g, k - 1, 14);
            if (!ok) break;
            ns_tc_fence_after();
            const float inv = l_run > 0.0f ? 1.0f / l_run : 0.0f;
            // O -> bf16 -> shared memory (16-byte piece q of row r at q ^ (r & 7)) -> a TMA store a warp, 64 columns at a time
#pragma unroll 1
            for (int hf = 0; hf < 2; hf++) {
                uint32_t w[32];
#pragma unroll
                for (int c = 0; c < 2; c++) {
                    uint32_t ob[32];
                    ns_tmem_ld32(o_addr + hf * 64 + c * 32, ob);
                    ns_tc_wait_ld();
#pragma unroll
                    for (int q = 0; q < 16; q++) w[c * 16 + q] = ns_pack_bf16x2(__uint_as_float(ob[2 * q]) * inv, __uint_as_float(ob[2 * q + 1]) * inv);
                }
                if (lane == 0) ns_bulk_wait_read<0>();   // the staging rows are still read by the store before
                __syncwarp();
#pragma unroll
                for (int q = 0; q < 8; q++)
                    ns_st_shared_v4(stage + lane * 128 + ((q ^ (lane & 7)) * 16), w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]);
                ns_fence_proxy_async();
                __syncwarp();
                if (lane == 0 && row0 + quad * 32 < p.seq) {
                    ns_tma_store_4d(&maps.o, stage, hf * 64, row0 + quad * 32, t.h, t.b);
                    ns_bulk_commit();
                }
                __syncwarp();
            }
            // the next tile's first P.V overwrites O; it follows this warp's next P
            ns_tc_fence_before();
        }
        if (lane == 0) ns_bulk_wait_read<0>();
    }

    // ---------------------------------------------------------------- teardown
    __syncwarp();
    ns_tc_fence_before();
    __syncthreads();
    if (*abort_flag != 0 && threadIdx.x == 0) {
        long long t0 = clock64();
        while (clock64() - t0 < 400000) { }
    }
    __syncthreads();
    if (warp == 1) {
        ns_tc_fence_after();
        ns_tmem_dealloc(tmem_base, 512);
    }
}

int make_map(CUtensorMap* m, uint64_t base, int batch, int heads, int seq, const int64_t* strides, uint32_t box_rows)
{
    uint64_t dims[4] = {128, (uint64_t)seq, (uint64_t)heads, (uint64_t)batch};
    uint64_t bytes[3] = {(uint64_t)strides[2] * 2, (uint64_t)strides[1] * 2, (uint64_t)strides[0] * 2};
    uint32_t box[4] = {64, box_rows, 1, 1};
    return ns_make_tensor_map(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, reinterpret_cast<const void*>(base), dims, bytes, box, CU_TENSOR_MAP_SWIZZLE_128B);
}

}  // namespace

extern "C" int ns_attention_prefill(ns_device_t h, uint64_t q, uint64_t k, uint64_t v, uint64_t o, int batch, int heads, int seq, int head_dim,
                                    const int64_t* q_strides, const int64_t* k_strides, const int64_t* v_strides, const int64_t* o_strides,
                                    float scale, int causal)
{
    NsDevice* d = ns_dev(h);
    int rc = ns_device_make_current(d);
    if (rc != NS_OK) return rc;
    NS_REQUIRE(q && k && v && o && q_strides && k_strides && v_strides && o_strides, NS_ERR_ARGUMENT, "ns_attention_prefill: null argument");
    NS_REQUIRE(head_dim == 128, NS_ERR_ARGUMENT, "ns_attention_prefill: head_dim must be 128 (got %d)", head_dim);
    NS_REQUIRE(batch > 0 && heads > 0 && seq > 0, NS_ERR_ARGUMENT, "ns_attention_prefill: bad shape");
    const int64_t tiles128 = (int64_t)batch * heads * ((seq + 127) / 128);
    NS_REQUIRE(tiles128 < (1LL << 31), NS_ERR_ARGUMENT, "ns_attention_prefill: too many tiles");
    PaMaps maps;
    rc = make_map(&maps.q, q, batch, heads, seq, q_strides, 128);
    if (rc == NS_OK) rc = make_map(&maps.k, k, batch, heads, seq, k_strides, PA_KB);
    if (rc == NS_OK) rc = make_map(&maps.v, v, batch, heads, seq, v_strides, PA_KB);
    if (rc == NS_OK) rc = make_map(&maps.o, o, batch, heads, seq, o_strides, 32);
    if (rc != NS_OK) return rc;
    PaParams p;
    p.batch = batch; p.heads = heads; p.seq = seq; p.causal = causal ? 1 : 0;
    p.scale_log2 = scale * 1.4426950408889634f;
    p.status = d->status_dev;
    // tiles are drawn from as many heads at a time as have 48 MB of keys and values: those stay in L2 (126 MB)
    p.heads_run = (int)std::max<int64_t>(1, (48 << 20) / ((int64_t)seq * 512));
    // Where each 128 rows can have an SM of their own they get it: a group alone does not share the exponential unit.  A row's
    // arithmetic is the same either way.  Against 128 rows shared by both groups (us): 8 heads x 64 10.7, 7.0; x 512 13.9, 11.3; x 2048 27.2, 25.4; 2 heads x
    // 8192 78.1, 78.9; one head x 16384 145, 151.  (This build spills three words.)
    const bool solo = tiles128 <= d->sm_count;
    const int total = solo ? (int)tiles128 : batch * heads * ((seq + 255) / 256);
    // the counter of drawn tiles: one word at the start of the device object's scratch block, zeroed in stream order
    void* counter = nullptr;
    rc = ns_scratch_reserve(d, 256, &counter);
    if (rc != NS_OK) return rc;
    p.tile_counter = reinterpret_cast<int*>(counter);
    if (total > d->sm_count) NS_CUDA(cudaMemsetAsync(counter, 0, sizeof(int), d->stream));
    auto kernel = solo ? ns_attention_prompt_kernel<true> : ns_attention_prompt_kernel<false>;
    NS_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PA_SMEM_BYTES));
    kernel<<<total < d->sm_count ? total : d->sm_count, PA_THREADS, PA_SMEM_BYTES, d->stream>>>(maps, p);
    NS_CUDA(cudaGetLastError());
    return NS_OK;
}
