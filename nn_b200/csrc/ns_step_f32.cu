// One cached step of the float32 decoder in five launches a layer.
//
// Operator by operator (ns_ops_f32.cu; the call sequence of Sequential.ForwardCached, src/NeuralSharp/Layers/Sequential.cs:59-80)
// such a step is 26 launches a layer of 1 to 3 us each, of which almost all is the launch, one trip to L2 for the input and
// one for the output: 215 us a token for four layers of width 128, whose weights are read in a tenth of a microsecond.  Here a product
// takes the LayerNorm in front of it and the bias, GELU and residual behind it, one kernel does what lies between two
// products of the attention, and the kernels are launched programmatically: a product has its first weights in shared memory before
// its input is ready.  Every output is the same chain of operations as in the operators, so the bits are the same (of finite caches).
// Measured on that decoder (context 128, one sequence): 128 tokens from a prompt of 32 34.4 -> 15.8 ms, a step on the GPU 215 -> 95 us.
#include "ns_common.cuh"

namespace {

constexpr int LT = 32, LK = 64, L_STAGES = 8, L_LD = LT + 4;     // columns of a tile, k of a slice, slices in the ring, words between a slice's rows
constexpr int L_WARPS = 8;
constexpr int LINEAR_A_BYTES = 128 * 1024;                        // most shared memory for a tile's input rows

struct LinearF32Args {
    const float* x;          // [m, k]
    const float* gamma;      // LayerNorm of x first, or null
    const float* beta;
    float eps;
    const float* w;          // [k, n]
    const float* bias;       // or null
    const float* residual;   // [m, n] or null
    float* y;
    int m, n, k, gelu;
};

__device__ __forceinline__ void copy16_async(float* dst, const float* src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(ns_smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ float warp_sum(float v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float warp_max(float v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// One row in shared memory, normalised in place by one warp, with the sums of ns_f32_layernorm_kernel's 128 threads in their order: lane l stands
// for threads l, l + 32, l + 64 and l + 96.
__device__ __forceinline__ void layernorm_row(float* row, int cols, const float* gamma, const float* beta, float eps, int lane)
{
    float p[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
        float s = 0.0f;
        for (int j = lane + 32 * q; j < cols; j += 128) s += row[j];
        p[q] = warp_sum(s);
    }
    const float mean = (((p[0] + p[1]) + p[2]) + p[3]) / (float)cols;
#pragma unroll
    for (int q = 0; q < 4; q++) {
        float v = 0.0f;
        for (int j = lane + 32 * q; j < cols; j += 128) { float d = row[j] - mean; v += d * d; }
        p[q] = warp_sum(v);
    }
    const float var = ((p[0] + p[1]) + p[2]) + p[3];
    const float inv = 1.0f / sqrtf(var / (float)cols + eps);
    for (int j = lane; j < cols; j += 32) row[j] = __fadd_rn(__fmul_rn(__fmul_rn(row[j] - mean, inv), gamma[j]), beta[j]);
}

// DEPTH steps of R chains (DEPTH a multiple of 4); eight steps' operands are fetched ahead of their multiply-adds
template <int R, int DEPTH>
__device__ __forceinline__ void chains(const float* as, int a_ld, const float* bs, float (&acc)[R])
{
    constexpr int AHEAD = DEPTH < 8 ? DEPTH : 8;
    float4 av[2][R][AHEAD / 4];
    float bv[2][AHEAD];
    auto fetch = [&](int buf, int p0) {
#pragma unroll
        for (int p = 0; p < AHEAD; p++) bv[buf][p] = bs[(p0 + p) * L_LD];
#pragma unroll
        for (int r = 0; r < R; r++)
#pragma unroll
            for (int q = 0; q < AHEAD / 4; q++) av[buf][r][q] = *reinterpret_cast<const float4*>(as + r * a_ld + p0 + 4 * q);
    };
    fetch(0, 0);
#pragma unroll
    for (int p0 = 0; p0 < DEPTH; p0 += AHEAD) {
        const int buf = (p0 / AHEAD) & 1;
        if (p0 + AHEAD < DEPTH) fetch(buf ^ 1, p0 + AHEAD);
#pragma unroll
        for (int q = 0; q < AHEAD / 4; q++) {
#pragma unroll
            for (int r = 0; r < R; r++) acc[r] = __fmaf_rn(av[buf][r][q].x, bv[buf][4 * q], acc[r]);
#pragma unroll
            for (int r = 0; r < R; r++) acc[r] = __fmaf_rn(av[buf][r][q].y, bv[buf][4 * q + 1], acc[r]);
#pragma unroll
            for (int r = 0; r < R; r++) acc[r] = __fmaf_rn(av[buf][r][q].z, bv[buf][4 * q + 2], acc[r]);
#pragma unroll
            for (int r = 0; r < R; r++) acc[r] = __fmaf_rn(av[buf][r][q].w, bv[buf][4 * q + 3], acc[r]);
        }
    }
}

// A tile is 8 R rows of 32 columns: a warp owns R rows (loads them, normalises them, multiplies them), a lane one column.  What bounds it is
// latency: one trip for the input rows, k dependent multiply-adds (4 cycles each), so the weights run ahead through a ring of
// 64-step slices (16-byte asynchronous copies; the first 448 steps are under way before the input is ready).
// TURNED: rows of tiles along x, which takes more of them than y does.
template <int R, bool TURNED>
__global__ void __launch_bounds__(32 * L_WARPS) ns_f32_linear_kernel(const LinearF32Args a)
{
    extern __shared__ float4 linear_smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float* rows_smem = reinterpret_cast<float*>(linear_smem);              // [8 R][k]
    float* ring = rows_smem + (size_t)R * L_WARPS * a.k;                  // [L_STAGES][LK][L_LD]
    const int col0 = (TURNED ? blockIdx.y : blockIdx.x) * LT, row0 = ((TURNED ? blockIdx.x : blockIdx.y) * L_WARPS + warp) * R;
    const int slices = (a.k + LK - 1) / LK;

    auto load_w = [&](int slice) {
        if (slice < slices) {
            float* bs = ring + (slice % L_STAGES) * LK * L_LD;
            const int k0 = slice * LK, pieces = min(LK, a.k - k0) * (LT / 4);
            for (int e = threadIdx.x; e < pieces; e += 32 * L_WARPS) {
                const int p = e >> 3, c = (e & 7) * 4;
                if (col0 + c < a.n) copy16_async(bs + p * L_LD + c, a.w + (size_t)(k0 + p) * a.n + col0 + c);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");                // empty groups keep the count
    };
    for (int s = 0; s < L_STAGES - 1; s++) load_w(s);
    ns_pdl_wait();
    ns_pdl_trigger();

    const float* x = ns_after_wait(a.x);
    float* as = rows_smem + (size_t)warp * R * a.k;
    const bool live = row0 < a.m;
#pragma unroll
    for (int r = 0; r < R; r++) {
        if (row0 + r >= a.m) break;
        const float4* src = reinterpret_cast<const float4*>(x + (size_t)(row0 + r) * a.k);
        for (int q = lane; q < a.k / 4; q += 32) reinterpret_cast<float4*>(as + (size_t)r * a.k)[q] = src[q];
    }
    __syncwarp();
    if (a.gamma != nullptr) {
#pragma unroll
        for (int r = 0; r < R; r++)
            if (row0 + r < a.m) layernorm_row(as + (size_t)r * a.k, a.k, a.gamma, a.beta, a.eps, lane);
        __syncwarp();
    }

    const int col = col0 + lane;
    float res[R], acc[R];
    const float* residual = ns_after_wait(a.residual);
    const float bias = a.bias != nullptr && col < a.n ? a.bias[col] : 0.0f;
#pragma unroll
    for (int r = 0; r < R; r++) {
        acc[r] = 0.0f;
        res[r] = residual != nullptr && col < a.n && row0 + r < a.m ? residual[(size_t)(row0 + r) * a.n + col] : 0.0f;
    }
    for (int s = 0; s < slices; s++) {
        asm volatile("cp.async.wait_group %0;" ::"n"(L_STAGES - 2) : "memory");
        __syncthreads();                               // slice s has arrived for everyone; everyone is done with slice s - 1
        load_w(s + L_STAGES - 1);
        if (!live) continue;
        const float* bs = ring + (s % L_STAGES) * LK * L_LD + lane;
        const int depth = min(LK, a.k - s * LK);
        if (depth == LK) chains<R, LK>(as + s * LK, a.k, bs, acc);
        else
            for (int p = 0; p < depth; p += 4) chains<R, 4>(as + s * LK + p, a.k, bs + p * L_LD, acc);
    }
    if (col >= a.n) return;
#pragma unroll
    for (int r = 0; r < R; r++) {
        if (row0 + r >= a.m) break;
        float v = acc[r];
        if (a.bias != nullptr) v = __fadd_rn(v, bias);
        if (a.gelu) v = ns_gelu_tanh(v);
        if (residual != nullptr) v = __fadd_rn(res[r], v);
        a.y[(size_t)(row0 + r) * a.n + col] = v;
    }
}

// ------------------------------------------------------------------------------------------------
// One new position per sequence: this (sequence, head)'s key and value into the cache, scores over the positions there are, softmax,
// weighted values, heads side by side.  One CTA per (sequence, head).  Positions past the current one have weight exp(-1e9 - max) = 0 in
// the operators and are left out, which comes to the same wherever the cache is finite; the sums are those of
// ns_f32_scale_mask_softmax_kernel's 128 threads in their order.
// ------------------------------------------------------------------------------------------------
struct AttentionStepF32Args {
    const float* qkv;        // [batch, 3 heads dim]
    float* keys;             // [batch, heads, capacity, dim]
    float* values;
    const float* position;
    float* y;                // [batch, heads dim]
    int heads, capacity, dim;
    float scale;
};

__global__ void __launch_bounds__(128) ns_f32_attention_step_kernel(const AttentionStepF32Args a)
{
    extern __shared__ float4 attention_smem[];
    __shared__ float red[2][4];
    const int dim = a.dim, b = blockIdx.x / a.heads, h = blockIdx.x % a.heads, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    float* q = reinterpret_cast<float*>(attention_smem);                   // [dim]
    float* vs = q + dim;                                                  // [positions][dim]
    float* p = vs + (size_t)a.capacity * dim;                              // [positions]
    ns_pdl_wait();
    ns_pdl_trigger();
    const int pos = (int)a.position[0];
    const int count = min(max(pos + 1, 0), a.capacity);
    const size_t width = (size_t)a.heads * dim;
    const float* row = a.qkv + (size_t)b * 3 * width + (size_t)h * dim;
    float* keys = a.keys + (size_t)blockIdx.x * a.capacity * dim;
    float* values = a.values + (size_t)blockIdx.x * a.capacity * dim;
    const int old = min(pos, count);                                       // positions that are in the cache already
    for (int e = tid; e < old * dim / 4; e += 128) copy16_async(vs + 4 * e, values + 4 * e);
    asm volatile("cp.async.commit_group;" ::: "memory");
    for (int d = tid; d < dim; d += 128) {
        q[d] = row[d];
        if (pos >= 0 && pos < a.capacity) {
            keys[(size_t)pos * dim + d] = row[width + d];
            const float v = row[2 * width + d];
            values[(size_t)pos * dim + d] = v;
            vs[(size_t)pos * dim + d] = v;
        }
    }
    __syncthreads();
    float mx = -INFINITY;
    for (int j = tid; j < count; j += 128) {
        const float4* k4 = reinterpret_cast<const float4*>(j < pos ? keys + (size_t)j * dim : row + width);
        float acc = 0.0f;
        for (int d0 = 0; d0 < dim / 4; d0 += 8) {
            float4 t[8];
#pragma unroll
            for (int u = 0; u < 8; u++)
                if (d0 + u < dim / 4) t[u] = k4[d0 + u];
#pragma unroll
            for (int u = 0; u < 8; u++)
                if (d0 + u < dim / 4) {
                    const float4 w = reinterpret_cast<const float4*>(q)[d0 + u];
                    acc = __fmaf_rn(w.x, t[u].x, acc); acc = __fmaf_rn(w.y, t[u].y, acc);
                    acc = __fmaf_rn(w.z, t[u].z, acc); acc = __fmaf_rn(w.w, t[u].w, acc);
                }
        }
        const float v = __fadd_rn(__fmul_rn(acc, a.scale), 0.0f);
        p[j] = v;
        mx = fmaxf(mx, v);
    }
    mx = warp_max(mx);
    if (lane == 0) red[0][warp] = mx;
    __syncthreads();
    mx = fmaxf(fmaxf(fmaxf(red[0][0], red[0][1]), red[0][2]), red[0][3]);
    float sum = 0.0f;
    for (int j = tid; j < count; j += 128) {
        float e = expf(p[j] - mx);
        p[j] = e;
        sum += e;
    }
    sum = warp_sum(sum);
    if (lane == 0) red[1][warp] = sum;
    __syncthreads();
    sum = red[1][0] + red[1][1];
    sum += red[1][2];
    sum += red[1][3];
    const float inv = 1.0f / sum;
    for (int j = tid; j < count; j += 128) p[j] *= inv;
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    for (int d = tid; d < dim; d += 128) {
        float acc = 0.0f;
#pragma unroll 16
        for (int j = 0; j < count; j++) acc = __fmaf_rn(p[j], vs[(size_t)j * dim + d], acc);
        a.y[(size_t)b * width + (size_t)h * dim + d] = acc;
    }
}

// x[b, i, :] = table[token] + positions[position + i]; indices as ns_f32_gather takes them (truncated, clamped to the table)
__global__ void ns_f32_embed_positions_kernel(const float* __restrict__ ids, const float* __restrict__ table, const float* __restrict__ positions,
                                              const float* __restrict__ position, float* __restrict__ x, int rows, int steps, int dim, int vocabulary, int capacity)
{
    ns_pdl_wait();
    ns_pdl_trigger();
    const int64_t n = (int64_t)rows * dim;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
        const int r = (int)(e / dim), d = (int)(e % dim);
        const float f = ids[r], g = (float)(r % steps) + position[0];
        const int t = min(f > 0.0f ? (int)f : 0, vocabulary - 1), at = min(g > 0.0f ? (int)g : 0, capacity - 1);
        x[e] = __fadd_rn(table[(size_t)t * dim + d], positions[(size_t)at * dim + d]);
    }
}

}  // namespace

#define NS_ENTER(h)                          \
    NsDevice* d = ns_dev(h);                 \
    {                                        \
        int _rc = ns_device_make_current(d); \
        if (_rc != NS_OK) return _rc;        \
    }

template <int R, bool TURNED>
static int launch_linear_as(NsDevice* d, const LinearF32Args& a, dim3 grid)
{
    constexpr int ring = L_STAGES * LK * L_LD * (int)sizeof(float);
    static bool configured[64] = {false};
    if (!configured[d->ordinal]) {
        NS_CUDA(cudaFuncSetAttribute(ns_f32_linear_kernel<R, TURNED>, cudaFuncAttributeMaxDynamicSharedMemorySize, LINEAR_A_BYTES + ring));
        configured[d->ordinal] = true;
    }
    NS_CUDA(ns_launch_pdl(ns_f32_linear_kernel<R, TURNED>, grid, dim3(32 * L_WARPS), (size_t)R * L_WARPS * a.k * 4 + ring, d->stream, a));
    return NS_OK;
}
template <int R>
static int launch_linear(NsDevice* d, const LinearF32Args& a)
{
    const unsigned across = (unsigned)(((int64_t)a.n + LT - 1) / LT), down = (unsigned)(((int64_t)a.m + L_WARPS * R - 1) / (L_WARPS * R));
    if (down <= 65535) return launch_linear_as<R, false>(d, a, dim3(across, down));
    NS_REQUIRE(across <= 65535, NS_ERR_ARGUMENT, "ns_f32_linear: %d x %d is too large", a.m, a.n);
    return launch_linear_as<R, true>(d, a, dim3(down, across));
}

extern "C" int ns_f32_linear(ns_device_t h, uint64_t x, uint64_t gamma, uint64_t beta, float eps, uint64_t w, uint64_t bias, uint64_t residual, int gelu,
                             uint64_t y, int m, int n, int k)
{
    NS_ENTER(h);
    NS_REQUIRE(x && w && y && m >= 0 && n > 0 && k > 0, NS_ERR_ARGUMENT, "ns_f32_linear: bad argument");
    NS_REQUIRE((gamma == 0) == (beta == 0), NS_ERR_ARGUMENT, "ns_f32_linear: gamma and beta go together");
    NS_REQUIRE(((n | k) & 3) == 0 && ((x | w) & 15) == 0, NS_ERR_ARGUMENT, "ns_f32_linear: n=%d and k=%d must be multiples of 4, x and w on 16 bytes", n, k);
    NS_REQUIRE(k <= LINEAR_A_BYTES / 4 / L_WARPS, NS_ERR_ARGUMENT, "ns_f32_linear: k=%d is more than %d", k, LINEAR_A_BYTES / 4 / L_WARPS);
    NS_REQUIRE(m <= (1 << 30), NS_ERR_ARGUMENT, "ns_f32_linear: %d rows are too many", m);
    if (m == 0) return NS_OK;
    LinearF32Args a;
    a.x = reinterpret_cast<const float*>(x); a.gamma = reinterpret_cast<const float*>(gamma); a.beta = reinterpret_cast<const float*>(beta);
    a.eps = eps; a.w = reinterpret_cast<const float*>(w); a.bias = reinterpret_cast<const float*>(bias);
    a.residual = reinterpret_cast<const float*>(residual); a.y = reinterpret_cast<float*>(y);
    a.m = m; a.n = n; a.k = k; a.gelu = gelu;
    // one row a warp while that makes few tiles (its chain has nothing to wait for but itself), more rows a warp to read w less often
    if (m <= L_WARPS || k > LINEAR_A_BYTES / 8 / L_WARPS) return launch_linear<1>(d, a);
    if (m <= 2 * L_WARPS || k > LINEAR_A_BYTES / 16 / L_WARPS) return launch_linear<2>(d, a);
    return launch_linear<4>(d, a);
}

extern "C" int ns_f32_attention_step(ns_device_t h, uint64_t qkv, uint64_t keys, uint64_t values, uint64_t position, uint64_t y, int batch, int heads,
                                     int capacity, int dim, float scale)
{
    NS_ENTER(h);
    NS_REQUIRE(qkv && keys && values && position && y && batch >= 0 && heads > 0 && capacity > 0 && dim > 0, NS_ERR_ARGUMENT, "ns_f32_attention_step: bad argument");
    NS_REQUIRE((dim & 3) == 0 && ((qkv | keys | values) & 15) == 0, NS_ERR_ARGUMENT, "ns_f32_attention_step: dim=%d must be a multiple of 4, operands on 16 bytes", dim);
    const int64_t smem = ((int64_t)capacity * dim + capacity + dim) * 4;
    NS_REQUIRE(smem <= 200 * 1024, NS_ERR_ARGUMENT, "ns_f32_attention_step: %d positions of %d do not fit shared memory", capacity, dim);
    NS_REQUIRE((int64_t)batch * heads < ((int64_t)1 << 31), NS_ERR_ARGUMENT, "ns_f32_attention_step: %d sequences of %d heads are too many", batch, heads);
    if (batch == 0) return NS_OK;
    static bool configured[64] = {false};
    if (!configured[d->ordinal]) {
        NS_CUDA(cudaFuncSetAttribute(ns_f32_attention_step_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
        configured[d->ordinal] = true;
    }
    AttentionStepF32Args a;
    a.qkv = reinterpret_cast<const float*>(qkv); a.keys = reinterpret_cast<float*>(keys); a.values = reinterpret_cast<float*>(values);
    a.position = reinterpret_cast<const float*>(position); a.y = reinterpret_cast<float*>(y);
    a.heads = heads; a.capacity = capacity; a.dim = dim; a.scale = scale;
    NS_CUDA(ns_launch_pdl(ns_f32_attention_step_kernel, dim3((unsigned)batch * (unsigned)heads), dim3(128), (size_t)smem, d->stream, a));
    return NS_OK;
}

extern "C" int ns_f32_embed_positions(ns_device_t h, uint64_t ids, uint64_t table, uint64_t positions, uint64_t position, uint64_t x, int batch, int steps,
                                      int dim, int vocabulary, int capacity)
{
    NS_ENTER(h);
    NS_REQUIRE(ids && table && positions && position && x && batch >= 0 && steps >= 0 && dim > 0 && vocabulary > 0 && capacity > 0, NS_ERR_ARGUMENT,
               "ns_f32_embed_positions: bad argument");
    const int64_t n = (int64_t)batch * steps * dim;
    if (n == 0) return NS_OK;
    const int64_t blocks = (n + 255) / 256, cap = (int64_t)d->sm_count * 16;
    // nothing to do before its inputs are there: no programmatic start (it lets the first product start early all the same)
    NS_CUDA(ns_launch_plain(ns_f32_embed_positions_kernel, dim3((unsigned)(blocks < cap ? blocks : cap)), dim3(256), 0, d->stream, reinterpret_cast<const float*>(ids),
                          reinterpret_cast<const float*>(table), reinterpret_cast<const float*>(positions), reinterpret_cast<const float*>(position),
                          reinterpret_cast<float*>(x), batch * steps, steps, dim, vocabulary, capacity));
    return NS_OK;
}
