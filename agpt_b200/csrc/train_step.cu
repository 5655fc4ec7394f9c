// One launch group's forward, loss and backward as one native call: the walker's step (src/cuda/agpt_train.cu:4560-5100)
// without a tape or a host decision between the kernels.
//
// What bounds a step on many rows is memory traffic around the dense projections and the tensor pipe inside them; on few
// rows it is the number of launches and the host time between them.  Both come down by giving the projections the work of
// the row kernels around them (step_gemm.cu):
//   * layer norm: its gain is folded into the weights and its shift into the bias (norm * gain * W = norm * (gain W)), the
//     rows are normalised where the projection reads them from the row's {mean, 1/std}, which the projection before wrote.
//     Neither the normalised rows nor the layer-norm output exist in memory.
//   * its parameter gradients come out of the weight gradient: with G = norm^T dY and db = column sums of dY,
//     dW = gain G + shift db,  dgain = sum_n W G,  dshift = sum_n W db  -- no pass over the rows.
//   * bias gradients are column sums of an operand the weight gradient has in its hands anyway.
//   * RoPE, ReLU and its mask (one bit per element), the residual sums and the layer-norm backward are epilogues.
// Per layer: five launches forward, nine and the attention's three backward; the partial weight gradients of all layers
// are summed by two launches at the end.  On few rows all weight gradients are one launch instead of four a layer.
#include <algorithm>
#include <cmath>
#include <vector>

#include "../../include/agpt_b200.h"
#include "internal.h"
#include "pdl.cuh"
#include "step_gemm.h"

namespace {

#define TRY(x)                       \
    do {                             \
        if (int rc_ = (x)) return rc_; \
    } while (0)

int launched(const char *what) {
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return agpt_set_error(AGPT_E_CUDA, "train_step: %s: %s", what, cudaGetErrorString(e));
    return AGPT_OK;
}

__device__ __forceinline__ float wsum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// {mean, 1/std} of a row held by a warp, float4 per lane and step
template <int NV>
__device__ __forceinline__ float2 row_stats(const float4 (&v)[NV], int lane, int d4, int d) {
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < NV; k++) s += (v[k].x + v[k].y) + (v[k].z + v[k].w);
    const float mu = wsum(s) / (float)d;
    float q = 0.f;
#pragma unroll
    for (int k = 0; k < NV; k++)
        if (lane + 32 * k < d4) {
            const float a = v[k].x - mu, b = v[k].y - mu, c = v[k].z - mu, e = v[k].w - mu;
            q += (a * a + b * b) + (c * c + e * e);
        }
    return make_float2(mu, 1.0f / sqrtf(wsum(q) / (float)d + 1e-5f));
}

constexpr int ROWS_PER_BLOCK = 8;
constexpr int NV_MAX = 8;                 // d_model up to 1024

// x[r] = emb[tokens[r]] (tokens == nullptr: x is read as it is), stats[r]; one warp per row, zero statistics behind the end.  Clears n_clear counters on
// the way (a memset between two kernels would keep the second from being placed early).
template <int NV>
__global__ void __launch_bounds__(256) embed_stats_kernel(const float *__restrict__ emb, const int32_t *__restrict__ tokens, float *__restrict__ x,
                                                           float2 *__restrict__ stats, int64_t n, int64_t n_pad, int d, int vocab, int32_t *__restrict__ clear, int n_clear) {
    pdl_wait();
    pdl_next();
    for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < n_clear; i += (int64_t)gridDim.x * 256) clear[i] = 0;
    const int64_t r = (int64_t)blockIdx.x * ROWS_PER_BLOCK + (threadIdx.x >> 5);
    if (r >= n_pad) return;
    const int lane = threadIdx.x & 31, d4 = d >> 2;
    if (r >= n) { if (lane == 0) stats[r] = make_float2(0.f, 0.f); return; }
    const int id = tokens ? __ldg(tokens + r) : 0;
    const bool none = id < 0 || id >= vocab;              // a zero row
    const float4 *src = reinterpret_cast<const float4 *>(tokens ? emb + (int64_t)(none ? 0 : id) * d : x + r * d);
    float4 v[NV];
#pragma unroll
    for (int k = 0; k < NV; k++) {
        v[k] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (lane + 32 * k < d4 && !none) v[k] = tokens ? __ldg(src + lane + 32 * k) : src[lane + 32 * k];
        if (tokens && lane + 32 * k < d4) reinterpret_cast<float4 *>(x + r * d)[lane + 32 * k] = v[k];
    }
    const float2 st = row_stats<NV>(v, lane, d4, d);
    if (lane == 0) stats[r] = st;
}

// dx = (dn - mean(dn) - norm mean(dn norm)) / std (+ add): the rows that do not fit one accumulator tile (d_model > 128)
template <int NV>
__global__ void __launch_bounds__(256) norm_bwd_kernel(const float *__restrict__ dn, const float *__restrict__ x, const float2 *__restrict__ stats,
                                                        const float *add, float *out, int64_t n, int d) {
    pdl_wait();
    pdl_next();
    const int64_t r = (int64_t)blockIdx.x * ROWS_PER_BLOCK + (threadIdx.x >> 5);
    if (r >= n) return;
    const int lane = threadIdx.x & 31, d4 = d >> 2;
    const float2 st = __ldg(stats + r);
    float4 g[NV], nm[NV];
    float s1 = 0.f, s2 = 0.f;
#pragma unroll
    for (int k = 0; k < NV; k++) {
        g[k] = nm[k] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (lane + 32 * k < d4) {
            g[k] = __ldcs(reinterpret_cast<const float4 *>(dn + r * d) + lane + 32 * k);
            const float4 v = __ldg(reinterpret_cast<const float4 *>(x + r * d) + lane + 32 * k);
            nm[k] = make_float4((v.x - st.x) * st.y, (v.y - st.x) * st.y, (v.z - st.x) * st.y, (v.w - st.x) * st.y);
            s1 += (g[k].x + g[k].y) + (g[k].z + g[k].w);
            s2 += (g[k].x * nm[k].x + g[k].y * nm[k].y) + (g[k].z * nm[k].z + g[k].w * nm[k].w);
        }
    }
    s1 = wsum(s1) / (float)d; s2 = wsum(s2) / (float)d;
#pragma unroll
    for (int k = 0; k < NV; k++)
        if (lane + 32 * k < d4) {
            float4 o = make_float4((g[k].x - s1 - nm[k].x * s2) * st.y, (g[k].y - s1 - nm[k].y * s2) * st.y,
                                   (g[k].z - s1 - nm[k].z * s2) * st.y, (g[k].w - s1 - nm[k].w * s2) * st.y);
            if (add) {
                const float4 a = reinterpret_cast<const float4 *>(add + r * d)[lane + 32 * k];
                o.x += a.x; o.y += a.y; o.z += a.z; o.w += a.w;
            }
            reinterpret_cast<float4 *>(out + r * d)[lane + 32 * k] = o;
        }
}

// per-unit numbers of trained queries with a positive loss, and per block the sum of those losses
__global__ void __launch_bounds__(256) loss_count_kernel(const float *__restrict__ loss, const float *__restrict__ trained,
                                                          const int64_t *__restrict__ unit, int64_t n, int32_t *__restrict__ unit_count,
                                                          double *__restrict__ block_sum, int32_t *__restrict__ block_count) {
    pdl_wait();
    pdl_next();
    __shared__ double s_sum[8];
    __shared__ int s_cnt[8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double sum = 0.0;
    int cnt = 0;
    for (int i = 0; i < 4; i++) {
        const int64_t r = (int64_t)blockIdx.x * 1024 + i * 256 + threadIdx.x;
        const float l = r < n ? loss[r] * (trained ? trained[r] : 1.f) : 0.f;
        const bool pos = l > 0.f;
        const int u = r < n ? (int)unit[r] : -1;
        const unsigned m = __ballot_sync(0xffffffffu, pos);
        const int u0 = __shfl_sync(0xffffffffu, u, 0);
        // integer counts: the order of the atomics does not matter.  Rows of a unit are neighbours, so most warps add once.
        if (__all_sync(0xffffffffu, u == u0 || !pos)) { if (lane == 0 && m) atomicAdd(unit_count + u0, __popc(m)); }
        else if (pos) atomicAdd(unit_count + u, 1);
        if (pos) { sum += l; cnt++; }
    }
    for (int o = 16; o > 0; o >>= 1) { sum += __shfl_xor_sync(0xffffffffu, sum, o); cnt += __shfl_xor_sync(0xffffffffu, cnt, o); }
    if (lane == 0) { s_sum[warp] = sum; s_cnt[warp] = cnt; }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; w++) { sum += s_sum[w]; cnt += s_cnt[w]; }
        block_sum[blockIdx.x] = sum; block_count[blockIdx.x] = cnt;
    }
}

// row_scale[r] = trained / (trained queries of the row's unit), zeros behind the end; block 0 adds up the statistics
__global__ void __launch_bounds__(256) row_scale_kernel(const float *__restrict__ trained, const int64_t *__restrict__ unit,
                                                         const int32_t *__restrict__ unit_count, int64_t n, int64_t n_pad, float *__restrict__ scale,
                                                         const double *__restrict__ block_sum, const int32_t *__restrict__ block_count, int blocks,
                                                         double *__restrict__ loss_out, int64_t *__restrict__ count_out, float *__restrict__ tail) {
    pdl_wait();
    pdl_next();
    if (blockIdx.x == 0) {
        __shared__ double s_sum[256];
        __shared__ int64_t s_cnt[256];
        double s = 0.0;
        int64_t c = 0;
        for (int i = threadIdx.x; i < blocks; i += 256) { s += block_sum[i]; c += block_count[i]; }
        s_sum[threadIdx.x] = s; s_cnt[threadIdx.x] = c;
        __syncthreads();
        for (int o = 128; o > 0; o >>= 1) {
            if (threadIdx.x < o) { s_sum[threadIdx.x] += s_sum[threadIdx.x + o]; s_cnt[threadIdx.x] += s_cnt[threadIdx.x + o]; }
            __syncthreads();
        }
        if (threadIdx.x == 0) {
            *loss_out = s_sum[0]; *count_out = s_cnt[0];
            // the count rides in float32 next to the gradients: split so that sums over groups and ranks stay exact
            tail[0] = (float)s_sum[0]; tail[1] = (float)(s_cnt[0] / 4096); tail[2] = (float)(s_cnt[0] % 4096);
        }
    }
    for (int64_t r = (int64_t)blockIdx.x * 256 + threadIdx.x; r < n_pad; r += (int64_t)gridDim.x * 256) {
        float f = 0.f;
        if (r < n) {
            const int c = unit_count[unit[r]];
            f = c > 0 ? 1.0f / (float)c : 0.f;
            if (trained) f *= trained[r];
        }
        scale[r] = f;
    }
}

// out[n] = b[n] + sum_k shift[k] W[k, n]: the bias of a projection behind a layer norm; pad_value behind the last column
struct FoldJob { const float *w, *shift, *b; float *out; int k, n, n_pad; };
constexpr int FOLD_JOBS = 80;
struct FoldArgs { FoldJob job[FOLD_JOBS]; int first_block[FOLD_JOBS + 1]; int n; };
__global__ void __launch_bounds__(256) fold_bias_kernel(const __grid_constant__ FoldArgs a) {
    pdl_wait();
    pdl_next();
    __shared__ float s[8][32];
    int j = 0;
    while (j + 1 < a.n && (int)blockIdx.x >= a.first_block[j + 1]) j++;
    const FoldJob &f = a.job[j];
    const int c = ((int)blockIdx.x - a.first_block[j]) * 32 + (threadIdx.x & 31), w = threadIdx.x >> 5;
    float t = 0.f;
    if (c < f.n)
#pragma unroll 4
        for (int k = w; k < f.k; k += 8) t = fmaf(__ldg(f.shift + k), __ldg(f.w + (int64_t)k * f.n + c), t);
    s[w][threadIdx.x & 31] = t;
    __syncthreads();
    if (w == 0 && c < f.n_pad) {
        float v = -1e30f;
        if (c < f.n) {
            v = __ldg(f.b + c);
            for (int i = 0; i < 8; i++) v += s[i][threadIdx.x];
        }
        f.out[c] = v;
    }
}

// sums the slices of partial weight gradients in slice order and adds them to the gradients
struct GradJob {
    const float *part, *col_part;      // [slices][rows * ld], [slices][col_ld]
    float *col_sum;                    // [cols] scratch: the summed column sums
    float *dw[3], *db[3];              // segments of seg_cols columns
    const float *w[3];                 // NORM: the weights,
    const float *gain, *shift;         //       the layer norm's parameters (null: plain)
    float *dgain, *dshift;
    int slices, rows, cols, ld, seg_cols, col_ld;
};
constexpr int GRAD_JOBS = 20;
struct GradArgs { GradJob job[GRAD_JOBS]; int first_block[GRAD_JOBS + 1]; int n; };

__global__ void __launch_bounds__(256) grad_cols_kernel(const __grid_constant__ GradArgs a) {
    pdl_wait();
    pdl_next();
    __shared__ float s[8][32];
    int j = 0;
    while (j + 1 < a.n && (int)blockIdx.x >= a.first_block[j + 1]) j++;
    const GradJob &g = a.job[j];
    const int c = ((int)blockIdx.x - a.first_block[j]) * 32 + (threadIdx.x & 31), w = threadIdx.x >> 5;
    float t = 0.f;
    if (c < g.cols)
#pragma unroll 4
        for (int i = w; i < g.slices; i += 8) t += __ldg(g.col_part + (int64_t)i * g.col_ld + c);
    s[w][threadIdx.x & 31] = t;
    __syncthreads();
    if (w == 0 && c < g.cols) {
        t = 0.f;
        for (int i = 0; i < 8; i++) t += s[i][threadIdx.x];
        g.col_sum[c] = t;
        const int seg = c / g.seg_cols;
        g.db[seg][c - seg * g.seg_cols] += t;
    }
}

// one block per row of a gradient matrix
__global__ void __launch_bounds__(128) grad_rows_kernel(const __grid_constant__ GradArgs a) {
    pdl_wait();
    pdl_next();
    __shared__ float s[2][4];
    int j = 0;
    while (j + 1 < a.n && (int)blockIdx.x >= a.first_block[j + 1]) j++;
    const GradJob &g = a.job[j];
    const int r = (int)blockIdx.x - a.first_block[j];
    const float gain = g.gain ? __ldg(g.gain + r) : 1.f, shift = g.gain ? __ldg(g.shift + r) : 0.f;
    const int64_t step = (int64_t)g.rows * g.ld;
    float wg = 0.f, wb = 0.f;
    for (int c = threadIdx.x; c < g.cols; c += 128) {
        const float *p = g.part + (int64_t)r * g.ld + c;
        float t = 0.f;
        int i = 0;
        for (; i + 8 <= g.slices; i += 8) {
            float v[8];
#pragma unroll
            for (int q = 0; q < 8; q++) v[q] = __ldcs(p + (i + q) * step);
#pragma unroll
            for (int q = 0; q < 8; q++) t += v[q];
        }
        for (; i < g.slices; i++) t += __ldcs(p + i * step);
        const int seg = c / g.seg_cols, cc = c - seg * g.seg_cols;
        const int64_t at = (int64_t)r * g.seg_cols + cc;
        if (g.gain) {
            const float b = g.col_sum[c], w = __ldg(g.w[seg] + at);
            wg = fmaf(w, t, wg); wb = fmaf(w, b, wb);
            t = gain * t + shift * b;
        }
        g.dw[seg][at] += t;
    }
    if (!g.gain) return;
    wg = wsum(wg); wb = wsum(wb);
    if ((threadIdx.x & 31) == 0) { s[0][threadIdx.x >> 5] = wg; s[1][threadIdx.x >> 5] = wb; }
    __syncthreads();
    if (threadIdx.x == 0) {
        g.dgain[r] += (s[0][0] + s[0][1]) + (s[0][2] + s[0][3]);
        g.dshift[r] += (s[1][0] + s[1][1]) + (s[1][2] + s[1][3]);
    }
}

// ---- workspace ---------------------------------------------------------------------------------------------------------
struct Layer {
    float *q, *a, *xm, *h, *lse;
    float *dh, *dxm, *dqkv;              // gradients of h, of xm, of q, k and v (three times rows x d_model)
    void *k, *v;
    uint32_t *mask;
    float2 *stats2;
    uint8_t *qkv, *qkv_t, *wo, *wo_t, *ff1, *ff1_t, *ff2, *ff2_t;
    float *qkv_b, *ff1_b;
};
struct Space {
    std::vector<Layer> layer;
    std::vector<float *> x;              // layer inputs, and the last layer's output
    std::vector<float2 *> stats;         // their statistics
    uint8_t *head, *head_t;
    float *head_b;
    std::vector<float *> dx;             // gradients of the layer inputs and of the last layer's output (where rows are kept; else one buffer)
    float *u, *tmp;                      // the union below; d_model > 128: gradient of normalised rows
    float *logits, *dlogits, *loss, *scale;
    double *block_sum;
    int32_t *block_count, *unit_count;
    void *attn;
    int64_t attn_bytes;
    float *emb;
    int64_t emb_bytes;
    std::vector<float *> part;           // partial weight gradients, head first, then four per layer
    std::vector<float *> col_part, col_sum;
    int shared_slices;                   // rows kept: slices of every contraction; else 0
    int64_t bytes;
};
constexpr int P_PER_LAYER = 16;
enum { WQ, BQ, WK, BK, WV, BV, WO, BO, G1, B1, W1, BW1, W2, BW2, G2, B2 };

// Blocks are placed early (pdl.cuh) while launches count.  On many rows that costs more than it hides (the blocks of a projection then land on the SMs in
// the order in which these fall free, not side by side).  Whole steps, early / ordinary, us: d_model 64, 59k rows 1234 / 1281, 117k 1945 / 1980, 231k 3240 / 3226;
// d_model 128, 5k 1307 / 1420, 20k 1957 / 2053, 59k 3690 / 3653, 231k 11980 / 11650; d_model 256, 5k 1835 / 2000, 20k 3981 / 4070, 59k 9480 / 9220;
// d_model 384, 5k 2577 / 2755, 20k 7000 / 6890.
constexpr int64_t EARLY_ELEMENTS = 6 << 20;
bool placed_early(const agpt_train_step_args &A) { return A.n * A.d_model <= EARLY_ELEMENTS; }

// All weight gradients are formed by one launch at the end of the backward while that costs little memory: the gradients of the rows, which they contract, are
// then kept layer by layer (d_ff + 5 d_model numbers a row and layer: a megabyte for 60 rows in four layers of d_model 128, d_ff 512); else all
// layers share buffers.  With ffn_recompute, which asks for less memory, they always do.
//
// Whole steps, one launch / a launch each, us: two layers of d_model 64, 60 rows 230 / 302, 16k 484 / 609, 98k 1511 / 1588, 150k 2045 / 2115; of 128, 60 rows 285 / 366,
// 12k 651 / 797, 49k 1559 / 1671, 80k 2309 / 2420; of 256, 6k 824 / 905, 12k 1325 / 1372, 24k 2226 / 2168, 40k 3436 / 3360; four of 384, 6k 2340 / 2473,
// 16k 5646 / 5620.  Wide rows change sides between 3 and 6 Mi elements, narrow ones still gain 5 % beyond 9: the limit of early placement is taken for
// both.  A GiB holds four layers of d_model 128 up to that limit; past it in bytes alone 3 to 14 % are given up (six layers of 128, 49k rows 4354 / 4658).
constexpr int64_t KEPT_BYTES = 1 << 30;
int64_t kept_row_bytes(const agpt_train_step_args &A) { return 4 * (int64_t)A.n_layers * (A.d_ff + 5 * (int64_t)A.d_model); }
int64_t kept_rows(const agpt_train_step_args &A) { return A.ffn_recompute ? 0 : std::min(EARLY_ELEMENTS / A.d_model, KEPT_BYTES / kept_row_bytes(A)); }

int padded_vocab(int v) { return (v + 3) & ~3; }

// blocks per slice of all weight gradients together
int contract_units(const agpt_train_step_args &A) {
    const int D = A.d_model, F = A.d_ff;
    return agpt_row_contract_units(D, padded_vocab(A.vocab)) +
           A.n_layers * (agpt_row_contract_units(D, 3 * D) + agpt_row_contract_units(D, D) + 2 * agpt_row_contract_units(D, F));
}

void lay_out(const agpt_train_step_args &A, char *base, Space &S) {
    int64_t at = 0;
    auto take = [&](int64_t bytes) { char *p = base + at; at += (bytes + 255) & ~(int64_t)255; return p; };
    const int64_t n = A.n, n_pad = (n + 127) & ~(int64_t)127;
    const int D = A.d_model, F = A.d_ff, L = A.n_layers, Vp = padded_vocab(A.vocab), H = A.n_heads;
    const int64_t row = n * D * 4, kv = n * D * (A.bf16_store ? 2 : 4);
    S.layer.resize(L); S.x.resize(L + 1); S.stats.resize(L + 1);
    for (int l = 0; l <= L; l++) { S.x[l] = (float *)take(row); S.stats[l] = (float2 *)take(n_pad * 8); }
    const bool kept = n <= kept_rows(A);
    float *h_shared = A.ffn_recompute ? (float *)take(n * F * 4) : nullptr;
    for (int l = 0; l < L; l++) {
        Layer &y = S.layer[l];
        y.q = (float *)take(row); y.k = take(kv); y.v = take(kv); y.a = (float *)take(row); y.lse = (float *)take(n * H * 4);
        y.xm = (float *)take(row); y.stats2 = (float2 *)take(n_pad * 8);
        y.h = h_shared ? h_shared : (float *)take(n * F * 4);
        y.mask = (uint32_t *)take(n * (F / 32) * 4);
        y.qkv = (uint8_t *)take(agpt_weight_image_bytes(3 * D, D)); y.qkv_t = (uint8_t *)take(agpt_weight_image_bytes(D, 3 * D));
        y.wo = (uint8_t *)take(agpt_weight_image_bytes(D, D)); y.wo_t = (uint8_t *)take(agpt_weight_image_bytes(D, D));
        y.ff1 = (uint8_t *)take(agpt_weight_image_bytes(F, D)); y.ff1_t = (uint8_t *)take(agpt_weight_image_bytes(D, F));
        y.ff2 = (uint8_t *)take(agpt_weight_image_bytes(D, F)); y.ff2_t = (uint8_t *)take(agpt_weight_image_bytes(F, D));
        y.qkv_b = (float *)take(3 * D * 4); y.ff1_b = (float *)take(F * 4);
    }
    S.head = (uint8_t *)take(agpt_weight_image_bytes(Vp, D)); S.head_t = (uint8_t *)take(agpt_weight_image_bytes(D, A.vocab));
    S.head_b = (float *)take(Vp * 4);
    S.dx.resize(L + 1);
    if (kept) {
        for (int l = 0; l <= L; l++) S.dx[l] = (float *)take(row);
        for (int l = 0; l < L; l++) {
            Layer &y = S.layer[l];
            y.dh = (float *)take(n * F * 4); y.dxm = (float *)take(row); y.dqkv = (float *)take(3 * row);
        }
        S.u = (float *)take(row);        // the gradient of the attention's output
        S.logits = (float *)take(n * 8 * (int64_t)Vp);
    } else {
        float *dx = (float *)take(row);
        // one region in turn: logits and their gradient; the feed-forward gradient; the gradients of the attention's output and
        // of q, k, v
        S.u = (float *)take(n * 4 * (int64_t)std::max(std::max(F, 4 * D), 2 * Vp));
        for (int l = 0; l <= L; l++) S.dx[l] = dx;
        for (int l = 0; l < L; l++) { S.layer[l].dh = S.u; S.layer[l].dxm = dx; S.layer[l].dqkv = S.u + n * D; }
        S.logits = S.u;
    }
    S.dlogits = S.logits + n * Vp;
    S.tmp = D > 128 ? (float *)take(row) : nullptr;
    S.loss = (float *)take(n * 4); S.scale = (float *)take(n_pad * 4);
    const int64_t lb = (n + 1023) / 1024;
    S.block_sum = (double *)take(lb * 8); S.block_count = (int32_t *)take(lb * 4); S.unit_count = (int32_t *)take((int64_t)A.n_units * 4);
    S.attn_bytes = agpt_b200_attn_bwd_workspace_bytes(A.plan, D);
    S.attn = take(S.attn_bytes);
    S.emb_bytes = agpt_b200_embedding_grad_workspace_bytes(n, D, A.vocab);
    S.emb = (float *)take(S.emb_bytes);
    S.part.clear(); S.col_part.clear(); S.col_sum.clear();
    S.shared_slices = kept ? agpt_row_contract_shared_slices(n, contract_units(A)) : 0;
    auto part = [&](int m, int k, int cols) {
        const int64_t s = kept ? S.shared_slices : agpt_row_contract_slices(n, m, k);
        S.part.push_back((float *)take(s * m * k * 4)); S.col_part.push_back((float *)take(s * cols * 4)); S.col_sum.push_back((float *)take(cols * 4));
    };
    part(D, Vp, Vp);
    for (int l = 0; l < L; l++) { part(D, 3 * D, 3 * D); part(D, D, D); part(D, F, F); part(D, F, D); }
    S.bytes = at;
}

int check(const agpt_train_step_args &A) {
    if (!A.plan || !A.params || !A.grads || A.n != A.plan->n) return agpt_set_error(AGPT_E_ARG, "train_step: plan, parameters or row count missing");
    if (A.plan->device < 0) return agpt_set_error(AGPT_E_ARG, "train_step: the plan has no device index");
    if (!agpt_b200_train_step_takes(A.d_model, A.n_heads, A.d_ff, A.vocab))
        return agpt_set_error(AGPT_E_ARG, "train_step: d_model %d, %d heads, d_ff %d, vocabulary %d not provided", A.d_model, A.n_heads, A.d_ff, A.vocab);
    if (A.n_layers < 1 || A.n_units < 1 || A.n_pos < 1 || A.n_pos > A.seq_len) return agpt_set_error(AGPT_E_ARG, "train_step: bad argument");
    return AGPT_OK;
}

template <int NV>
int embed_stats_nv(const float *emb, const int32_t *tok, float *x, float2 *st, int64_t n, int d, int vocab, cudaStream_t s, int32_t *clear = nullptr, int n_clear = 0) {
    const int64_t n_pad = (n + 127) & ~(int64_t)127;
    pdl_launch(embed_stats_kernel<NV>, (unsigned)(n_pad / ROWS_PER_BLOCK), 256, 0, s, emb, tok, x, st, n, n_pad, d, vocab, clear, n_clear);
    return launched("row statistics");
}
int embed_stats(const float *emb, const int32_t *tok, float *x, float2 *st, int64_t n, int d, int vocab, cudaStream_t s, int32_t *clear = nullptr, int n_clear = 0) {
    if (d <= 128) return embed_stats_nv<1>(emb, tok, x, st, n, d, vocab, s, clear, n_clear);
    if (d <= 256) return embed_stats_nv<2>(emb, tok, x, st, n, d, vocab, s, clear, n_clear);
    if (d <= 512) return embed_stats_nv<4>(emb, tok, x, st, n, d, vocab, s, clear, n_clear);
    return embed_stats_nv<NV_MAX>(emb, tok, x, st, n, d, vocab, s, clear, n_clear);
}
int norm_bwd(const float *dn, const float *x, const float2 *st, const float *add, float *out, int64_t n, int d, cudaStream_t s) {
    const unsigned g = (unsigned)((n + ROWS_PER_BLOCK - 1) / ROWS_PER_BLOCK);
    if (d <= 128) pdl_launch(norm_bwd_kernel<1>, g, 256, 0, s, dn, x, st, add, out, n, d);
    else if (d <= 256) pdl_launch(norm_bwd_kernel<2>, g, 256, 0, s, dn, x, st, add, out, n, d);
    else if (d <= 512) pdl_launch(norm_bwd_kernel<4>, g, 256, 0, s, dn, x, st, add, out, n, d);
    else pdl_launch(norm_bwd_kernel<NV_MAX>, g, 256, 0, s, dn, x, st, add, out, n, d);
    return launched("layer-norm backward");
}

int up32(int x) { return (x + 31) & ~31; }
int up64(int x) { return (x + 63) & ~63; }

// weight images and folded biases of the whole model
int prepare_weights(const agpt_train_step_args &A, const Space &S, cudaStream_t st) {
    const int D = A.d_model, F = A.d_ff, V = A.vocab;
    std::vector<WeightSplitJob> jobs;
    std::vector<FoldJob> folds;
    // image of W [rows, cols] (n = column) and of its transpose (n = row); gain: per-row factor
    auto both = [&](const float *w, const float *gain, int rows, int cols, uint8_t *img, uint8_t *img_t) {
        jobs.push_back({w, gain, rows, cols, 1, 0, 0, up32(cols), up64(rows), up64(rows) / 64, img});
        jobs.push_back({w, gain, rows, cols, 0, 0, 0, up32(rows), up64(cols), up64(cols) / 64, img_t});
    };
    for (int l = 0; l < A.n_layers; l++) {
        const float *const *p = A.params + 1 + P_PER_LAYER * l;
        const Layer &y = S.layer[l];
        for (int i = 0; i < 3; i++) {
            const float *w = p[WQ + 2 * i];
            jobs.push_back({w, p[G1], D, D, 1, i * D, 0, D, up64(D), up64(D) / 64, y.qkv});
            jobs.push_back({w, p[G1], D, D, 0, 0, i * D, D, i == 2 ? up64(3 * D) - 2 * D : D, up64(3 * D) / 64, y.qkv_t});
            folds.push_back({w, p[B1], p[BQ + 2 * i], y.qkv_b + i * D, D, D, D});
        }
        both(p[WO], nullptr, D, D, y.wo, y.wo_t);
        both(p[W1], p[G2], D, F, y.ff1, y.ff1_t);
        both(p[W2], nullptr, F, D, y.ff2, y.ff2_t);
        folds.push_back({p[W1], p[B2], p[BW1], y.ff1_b, D, F, F});
    }
    const float *const *p = A.params + 1 + P_PER_LAYER * A.n_layers;      // final gain, shift, out.w, out.b
    both(p[2], p[0], D, V, S.head, S.head_t);
    // The vocabulary is padded to a multiple of 4 (rows on 16-byte boundaries): the extra logits get zero weights and a bias
    // of -1e30, so their probability and gradient are exactly 0.
    folds.push_back({p[2], p[1], p[3], S.head_b, D, V, padded_vocab(V)});
    TRY(agpt_split_weights(jobs.data(), (int)jobs.size(), st));
    for (size_t first = 0; first < folds.size(); first += FOLD_JOBS) {
        FoldArgs a;
        a.n = (int)std::min<size_t>(FOLD_JOBS, folds.size() - first);
        int blocks = 0;
        for (int i = 0; i < a.n; i++) { a.job[i] = folds[first + i]; a.first_block[i] = blocks; blocks += (a.job[i].n_pad + 31) / 32; }
        a.first_block[a.n] = blocks;
        pdl_launch(fold_bias_kernel, blocks, 256, 0, st, a);
        TRY(launched("folded biases"));
    }
    return AGPT_OK;
}

RowGemm gemm(const agpt_train_step_args &A, const float *a, int k, const uint8_t *image, int n) {
    RowGemm g;
    g.rows = A.n; g.K = k; g.N = n; g.a[0] = a; g.seg_cols = k; g.lda = k; g.image = image;
    return g;
}
RowContract contract(const agpt_train_step_args &A, const Space &S, int i, const float *a, int m, const float *b, int n) {
    RowContract c;
    c.rows = A.n; c.m = m; c.n = n; c.a = a; c.lda = m; c.b[0] = b; c.seg_cols = n; c.ldb = n;
    c.part = S.part[i]; c.col_part = S.col_part[i]; c.col_ld = n;
    c.slices = S.shared_slices ? S.shared_slices : agpt_row_contract_slices(A.n, m, n);
    return c;
}
// dx = the gradient of the rows in front of a layer norm (+ add) from the product that is the gradient of the normalised rows
int norm_gradient(const agpt_train_step_args &A, const Space &S, RowGemm g, const float *x, const float2 *stats, const float *add, float *dx, cudaStream_t st) {
    if (A.d_model <= 128) {
        g.epi = EPI_NORM_BWD; g.x = x; g.stats = stats; g.add = add; g.out = dx; g.ldo = A.d_model;
        return agpt_row_gemm(g, st);
    }
    g.out = S.tmp; g.ldo = A.d_model;
    TRY(agpt_row_gemm(g, st));
    return norm_bwd(S.tmp, x, stats, add, dx, A.n, A.d_model, st);
}

int ff1_forward(const agpt_train_step_args &A, const Layer &y, cudaStream_t st) {
    RowGemm g = gemm(A, y.xm, A.d_model, y.ff1, A.d_ff);
    g.pro = PRO_NORM; g.stats = y.stats2; g.epi = EPI_RELU; g.bias = y.ff1_b; g.out = y.h; g.ldo = A.d_ff; g.mask_out = y.mask;
    return agpt_row_gemm(g, st);
}

}  // namespace

extern "C" int agpt_b200_train_step_takes(int d_model, int n_heads, int d_ff, int vocab) {
    if (d_model < 32 || d_model > 32 * 4 * NV_MAX || d_model % 32 || d_ff < 32 || d_ff % 32 || n_heads < 1 || d_model % n_heads) return 0;
    const int hd = d_model / n_heads;
    return (hd == 16 || hd == 32 || hd == 64) && vocab >= 1 && vocab <= 400;
}

extern "C" int64_t agpt_b200_train_step_workspace_bytes(const agpt_train_step_args *args) try {
    if (!args) return agpt_set_error(AGPT_E_ARG, "train_step: null arguments");
    TRY(check(*args));
    // A workspace of the largest group serves the smaller ones: a step of fewer rows may need more, at the last row count whose gradients are kept and at the
    // last one with a slice per row block
    const int64_t kept = kept_rows(*args);
    int64_t bytes = 0;
    for (int64_t n : {args->n, kept, std::min(kept, agpt_row_contract_most_slices_rows(contract_units(*args)))})
        if (n >= 1 && n <= args->n) {
            agpt_train_step_args A = *args;
            A.n = n;
            Space S;
            lay_out(A, nullptr, S);
            bytes = std::max(bytes, S.bytes);
        }
    return bytes;
} AGPT_CATCH("train_step_workspace_bytes")

extern "C" int agpt_b200_train_step(const agpt_train_step_args *args, void *workspace, int64_t workspace_bytes, void *stream) try {
    if (!args || !workspace) return agpt_set_error(AGPT_E_ARG, "train_step: null arguments");
    if ((uintptr_t)workspace & 15) return agpt_set_error(AGPT_E_ARG, "train_step: the workspace does not start on a 16-byte boundary");
    const agpt_train_step_args &A = *args;
    TRY(check(A));
    Space S;
    lay_out(A, (char *)workspace, S);
    if (workspace_bytes < S.bytes)
        return agpt_set_error(AGPT_E_ARG, "train_step: workspace %lld bytes < required %lld", (long long)workspace_bytes, (long long)S.bytes);
    cudaStream_t st = (cudaStream_t)stream;
    const int64_t n = A.n;
    const bool kept = S.shared_slices > 0;
    const PdlScope scope(placed_early(A));
    const int D = A.d_model, F = A.d_ff, L = A.n_layers, H = A.n_heads, hd = D / H, V = A.vocab, Vp = padded_vocab(V);
    const float scale = 1.0f / sqrtf((float)hd);
    const int kv_dtype = A.bf16_store ? AGPT_KV_BF16 : AGPT_KV_F32;
    const bool fused_rope = agpt_row_gemm_rope_fits(A.n_pos, hd);
    const bool whole_row = D <= 128;            // a row fits one accumulator tile: statistics and layer-norm backward as epilogues
    // the tensor maps are encoded through the driver, which needs the device's context current on this thread
    cudaError_t e = cudaSetDevice(A.plan->device);
    if (e != cudaSuccess) return agpt_set_error(AGPT_E_CUDA, "train_step: %s", cudaGetErrorString(e));

    TRY(prepare_weights(A, S, st));
    TRY(embed_stats(A.params[0], A.tokens, S.x[0], S.stats[0], n, D, V, st, S.unit_count, A.n_units));

    // ---- forward ----
    for (int l = 0; l < L; l++) {
        const float *const *p = A.params + 1 + P_PER_LAYER * l;
        const Layer &y = S.layer[l];
        RowGemm g = gemm(A, S.x[l], D, y.qkv, 3 * D);
        g.pro = PRO_NORM; g.stats = S.stats[l]; g.epi = EPI_QKV; g.bias = y.qkv_b; g.head_dim = hd;
        float *k32 = y.dqkv, *v32 = y.dqkv + n * D;    // a table too large for shared memory: rotate (and round) in passes of their own
        const bool late = !fused_rope && A.bf16_store;
        g.qkv[0] = y.q; g.qkv[1] = late ? k32 : y.k; g.qkv[2] = late ? v32 : y.v;
        g.kv_bf16 = A.bf16_store && !late;
        if (fused_rope) { g.pos = A.pos; g.cosv = A.cosv; g.sinv = A.sinv; g.n_pos = A.n_pos; }
        TRY(agpt_row_gemm(g, st));
        if (!fused_rope) TRY(agpt_b200_rope_pair(y.q, late ? k32 : (float *)y.k, A.pos, A.cosv, A.sinv, n, H, hd, 0, st));
        if (late) {
            TRY(agpt_b200_kv_store_write_bf16(k32, y.k, n, D, st));
            TRY(agpt_b200_kv_store_write_bf16(v32, y.v, n, D, st));
        }
        TRY(agpt_b200_attn_fwd(A.plan, y.q, y.k, y.v, kv_dtype, y.a, y.lse, H, hd, scale, st));
        g = gemm(A, y.a, D, y.wo, D);
        g.epi = EPI_ADD; g.bias = p[BO]; g.add = S.x[l]; g.out = y.xm; g.ldo = D; g.stats_out = whole_row ? y.stats2 : nullptr;
        TRY(agpt_row_gemm(g, st));
        if (!whole_row) TRY(embed_stats(nullptr, nullptr, y.xm, y.stats2, n, D, 1, st));
        TRY(ff1_forward(A, y, st));
        g = gemm(A, y.h, F, y.ff2, D);
        g.epi = EPI_ADD; g.bias = p[BW2]; g.add = y.xm; g.out = S.x[l + 1]; g.ldo = D; g.stats_out = whole_row ? S.stats[l + 1] : nullptr;
        TRY(agpt_row_gemm(g, st));
        if (!whole_row) TRY(embed_stats(nullptr, nullptr, S.x[l + 1], S.stats[l + 1], n, D, 1, st));
    }
    const float *const *pf = A.params + 1 + P_PER_LAYER * L;
    float *const *gf = A.grads + 1 + P_PER_LAYER * L;
    {
        RowGemm g = gemm(A, S.x[L], D, S.head, Vp);
        g.pro = PRO_NORM; g.stats = S.stats[L]; g.bias = S.head_b; g.out = S.logits; g.ldo = Vp;
        TRY(agpt_row_gemm(g, st));
    }

    // ---- loss ----
    // the kernel's entropy weight divides by ln of the row width: lambda is rescaled so that the true vocabulary counts
    const float lambda = Vp == V ? A.entropy_lambda : (float)(A.entropy_lambda * (std::log((double)Vp) / std::log((double)V)));
    TRY(agpt_b200_loss_per_query(S.logits, A.query_to_node, A.query_offsets, A.radix_ids, A.tokens, A.counts_offset, A.counts_tok, A.counts_val,
                                 A.mass_weights, S.dlogits, S.loss, n, Vp, lambda, A.intermediate_weight, A.ce_only, st));
    const int64_t n_pad = (n + 127) & ~(int64_t)127;
    const int lb = (int)((n + 1023) / 1024);
    pdl_launch(loss_count_kernel, lb, 256, 0, st, S.loss, A.trained, A.unit_of_row, n, S.unit_count, S.block_sum, S.block_count);
    pdl_launch(row_scale_kernel, (unsigned)std::min<int64_t>((n_pad + 255) / 256, 148 * 8), 256, 0, st, A.trained, A.unit_of_row, S.unit_count, n, n_pad, S.scale,
                                                                                                  S.block_sum, S.block_count, lb, A.loss_sum, A.loss_count, A.tail);
    TRY(launched("loss statistics"));

    // ---- backward ----
    std::vector<GradJob> jobs;
    std::vector<RowContract> later;              // rows kept: contractions for the launch at the end
    auto weight_gradient = [&](const RowContract &c) {
        if (!kept) return agpt_row_contract(c, st);
        later.push_back(c);
        return (int)AGPT_OK;
    };
    auto grad_job = [&](int i, const RowContract &c, bool transposed) {
        GradJob j = {};
        j.part = S.part[i]; j.col_part = S.col_part[i]; j.col_sum = S.col_sum[i]; j.slices = c.slices; j.col_ld = c.col_ld;
        j.rows = transposed ? c.n : c.m; j.cols = j.ld = transposed ? c.m : c.n; j.seg_cols = j.cols;
        return j;
    };
    {
        RowContract c = contract(A, S, 0, S.x[L], D, S.dlogits, Vp);
        c.stats = S.stats[L]; c.row_scale = S.scale;
        TRY(weight_gradient(c));
        GradJob j = grad_job(0, c, false);
        j.cols = j.seg_cols = V;
        j.dw[0] = gf[2]; j.db[0] = gf[3]; j.w[0] = pf[2]; j.gain = pf[0]; j.shift = pf[1]; j.dgain = gf[0]; j.dshift = gf[1];
        jobs.push_back(j);
        RowGemm g = gemm(A, S.dlogits, Vp, S.head_t, D);
        g.pro = PRO_SCALE; g.row_scale = S.scale;
        TRY(norm_gradient(A, S, g, S.x[L], S.stats[L], nullptr, S.dx[L], st));
    }
    float *da = S.u;
    for (int l = L - 1; l >= 0; l--) {
        const float *const *p = A.params + 1 + P_PER_LAYER * l;
        float *const *gp = A.grads + 1 + P_PER_LAYER * l;
        const Layer &y = S.layer[l];
        const int i0 = 1 + 4 * l;
        float *dh = y.dh, *dq = y.dqkv, *dk = dq + n * D, *dv = dk + n * D;
        if (A.ffn_recompute) TRY(ff1_forward(A, y, st));
        // feed-forward: dW2 = h^T dx (stored transposed: its rows are h's features), dh = dx W2^T where h > 0
        RowContract c = contract(A, S, i0 + 3, S.dx[l + 1], D, y.h, F);
        c.transposed = 1; c.col_ld = D;
        TRY(weight_gradient(c));
        GradJob j = grad_job(i0 + 3, c, true);
        j.dw[0] = gp[W2]; j.db[0] = gp[BW2];
        jobs.push_back(j);
        RowGemm g = gemm(A, S.dx[l + 1], D, y.ff2_t, F);
        g.epi = EPI_MASKED; g.mask_in = y.mask; g.out = dh; g.ldo = F;
        TRY(agpt_row_gemm(g, st));
        c = contract(A, S, i0 + 2, y.xm, D, dh, F);
        c.stats = y.stats2;
        TRY(weight_gradient(c));
        j = grad_job(i0 + 2, c, false);
        j.dw[0] = gp[W1]; j.db[0] = gp[BW1]; j.w[0] = p[W1]; j.gain = p[G2]; j.shift = p[B2]; j.dgain = gp[G2]; j.dshift = gp[B2];
        jobs.push_back(j);
        TRY(norm_gradient(A, S, gemm(A, dh, F, y.ff1_t, D), y.xm, y.stats2, S.dx[l + 1], y.dxm, st));
        // attention output projection
        c = contract(A, S, i0 + 1, y.a, D, y.dxm, D);
        TRY(weight_gradient(c));
        j = grad_job(i0 + 1, c, false);
        j.dw[0] = gp[WO]; j.db[0] = gp[BO];
        jobs.push_back(j);
        g = gemm(A, y.dxm, D, y.wo_t, D);
        g.out = da; g.ldo = D;
        TRY(agpt_row_gemm(g, st));
        TRY(agpt_b200_attn_bwd_mode(A.plan, y.q, y.k, y.v, kv_dtype, y.a, y.lse, da, dq, dk, dv, S.attn, S.attn_bytes, H, hd, scale, A.grad_mode,
                                    A.edge_first, st));
        TRY(agpt_b200_rope_pair(dq, dk, A.pos, A.cosv, A.sinv, n, H, hd, 1, st));
        // the three projections that read the same normalised rows
        c = contract(A, S, i0, S.x[l], D, dq, 3 * D);
        c.b[1] = dk; c.b[2] = dv; c.n_seg = 3; c.seg_cols = D; c.ldb = D; c.stats = S.stats[l];
        TRY(weight_gradient(c));
        j = grad_job(i0, c, false);
        j.seg_cols = D;
        for (int i = 0; i < 3; i++) { j.dw[i] = gp[WQ + 2 * i]; j.db[i] = gp[BQ + 2 * i]; j.w[i] = p[WQ + 2 * i]; }
        j.gain = p[G1]; j.shift = p[B1]; j.dgain = gp[G1]; j.dshift = gp[B1];
        jobs.push_back(j);
        g = gemm(A, dq, 3 * D, y.qkv_t, D);
        g.a[1] = dk; g.a[2] = dv; g.n_seg = 3; g.seg_cols = D; g.lda = D;
        TRY(norm_gradient(A, S, g, S.x[l], S.stats[l], y.dxm, S.dx[l], st));
    }
    if (kept) TRY(agpt_row_contract_many(later.data(), (int)later.size(), st));
    TRY(agpt_b200_embedding_grad(S.dx[0], A.tokens, A.grads[0], n, D, V, 1, S.emb, S.emb_bytes, st));
    for (size_t first = 0; first < jobs.size(); first += GRAD_JOBS) {
        GradArgs a;
        a.n = (int)std::min<size_t>(GRAD_JOBS, jobs.size() - first);
        int blocks = 0;
        for (int i = 0; i < a.n; i++) { a.job[i] = jobs[first + i]; a.first_block[i] = blocks; blocks += (a.job[i].cols + 31) / 32; }
        a.first_block[a.n] = blocks;
        pdl_launch(grad_cols_kernel, blocks, 256, 0, st, a);
        blocks = 0;
        for (int i = 0; i < a.n; i++) { a.first_block[i] = blocks; blocks += a.job[i].rows; }
        a.first_block[a.n] = blocks;
        pdl_launch(grad_rows_kernel, blocks, 128, 0, st, a);
        TRY(launched("weight gradients"));
    }
    return AGPT_OK;
} AGPT_CATCH("train_step")
