// The dense projections of the training step on the fifth-generation tensor cores, float32 in and out.
//
// Every float32 operand is split into three bfloat16 matrices (x = b0 + b1 + b2, 24 mantissa bits) and a product is
// rebuilt from six bf16 x bf16 partial products with float32 accumulation, a1 b1 + a0 b2 + a2 b0 + a0 b1 + a1 b0 + a0 b0 in
// this order (the accumulator is still small while the small terms are added); the three products left out are below
// 2^-24.  After every 64 k the accumulator leaves tensor memory and is added in registers, round to nearest.
//
// Both kernels put the A operand into TENSOR MEMORY: a converting thread owns one row of the 128-row MMA tile, so it
// writes its packed bf16 pairs with tcgen05.st and no shared-memory pass, and the MMA then reads only B from shared
// memory (64 bytes per clock at N = 128 instead of the 128 that A and B in shared memory would need, which is all an SM
// has).  What the surrounding layers do row by row (layer norm, RoPE, ReLU and its mask, the residual, layer-norm
// backward) happens in the converting or the accumulator threads, which hold a whole row each.
//
// row_gemm_kernel: rows x weights.  Per block: a TMA warp (raw float32 rows, 128-byte swizzle), two MMA warps, four
//   converting warps, and two groups of four accumulator warps that own one 128-row accumulator each, so that one
//   drains while the other is being filled.  The weight image (split once per step) stays in shared memory for the
//   whole kernel when it fits (K <= 128 at 128 columns), else its 64-k blocks stream, each serving two row tiles.
// contract_kernel: A^T B over the rows (weight gradients).  The transposition of A costs nothing: a converting thread
//   owns a feature and walks down the rows of the staged tile.  B is split into shared memory with n contiguous.
//
// What bounds them.  An MMA stream alone runs at 64 clocks per 128 x 128 x 16 whatever shared-memory, tensor-memory or barrier traffic runs beside it; a step of 24
// of them takes 2000 to 3800 clocks here, as the converting warps are never idle (row_gemm_kernel; B's in contract_kernel): a chain of barrier, loads, splits
// and tensor-memory stores, slowed by instruction fetch (a stall of 0.4 to 0.9 per instruction: the roles' code together exceeds the instruction cache) and by
// the other roles' shared-memory traffic.  Sustained, training sits at the board's power limit (985 W, 1690 of 1965 MHz).  Share of active cycles on 288,000 rows of
// d_model 128 (tensor pipe, issue slots): q/k/v 41 %, 37 %; attention output 33, 31 (DRAM 53); feed-forward 48, 43; weight gradients 51, 58.  Tried and slower:
// eight converting warps (1080 -> 1417 us, six projections of d_model 256), one MMA warp that asks barriers ahead (1168), counters in shared memory in place of the
// barriers (1197; with two MMA warps in turn 1163), non-blocking barrier tests in the converters (an epoch of d_model 128 53.8 -> 55.3 ms), B rows of
// contract_kernel loaded one ahead (no change) or four at once (2208 -> 2742), rows stored straight from
// the accumulator threads, 32 bytes to 32 rows at a time (the store path held up the MMA issue too; wide outputs 2x); MMAs
// issued by one lane of a diverged warp (60 clocks each against 29 from an elected lane of a converged warp); scalar
// instead of paired (f32x2) conversions; a drain of the accumulator every 128 k instead of 64 (10 % faster, but the
// truncating tensor-core additions at full magnitude raise the error from 7e-8 to 4e-7).
// Measured, 560,000 rows, d_model 128, d_ff 512 (in brackets: the CUTLASS fast-float32 mainloop and the row kernels around
// it): q/k/v with layer norm and RoPE 419 us (437 + 97 + 187); attention output with residual and statistics 151 (160);
// feed-forward 427 + 369 (550 + 97 + 500); their input gradients 408 + 473 and 389 for q/k/v with the layer-norm backward;
// weight with bias gradients 423 / 215 / 452 / 446.  Since then two MMA warps (d_model 256, two layers: projections 1219 + 865 + 665 + 655 + 576 ->
// 1075 + 817 + 668 + 635 + 542) and one accumulator for narrow weight gradients.  Error against float64 6e-8 to 1.2e-7 (K = 64 to 1536), as before.
#include "step_gemm.h"

#include <algorithm>

#include "../../include/agpt_b200.h"
#include "internal.h"
#include "pdl.cuh"
#include "tc100.cuh"

namespace {

using namespace tc;

constexpr int TM = 128;                  // rows of an MMA tile
constexpr int A_BOX = TM * 128;          // one stage of raw float32 rows: a box of 32 columns
constexpr int SMEM_LIMIT = 232448;
constexpr int ACC_COLS = 128, TA_COLS = 96;      // tensor memory: two accumulators, two A stages of three planes
constexpr int TMEM_COLS = 512;
constexpr int BAR_BYTES = 768;            // barriers, then the abort flag and the tensor-memory address

int sm_count() {
    static int n[64];
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return 148;
    if (!n[dev]) cudaDeviceGetAttribute(&n[dev], cudaDevAttrMultiProcessorCount, dev);
    return n[dev];
}

typedef CUresult (*EncodeFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                             const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                             CUtensorMapFloatOOBfill);

// rows x cols, boxes of 32 columns x box_rows: float32 (128 bytes, swizzled) or bfloat16 (64 bytes)
int encode_map_any(CUtensorMap *m, const void *p, int64_t rows, int cols, int64_t ld_bytes, int box_rows, bool bf16) {
    static EncodeFn fn = nullptr;
    if (!fn) {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult q;
        cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q);
        if (e != cudaSuccess || q != cudaDriverEntryPointSuccess || !f) return agpt_set_error(AGPT_E_CUDA, "cuTensorMapEncodeTiled not found");
        fn = (EncodeFn)f;
    }
    const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)ld_bytes};
    const cuuint32_t box[2] = {32, (cuuint32_t)box_rows}, es[2] = {1, 1};
    CUresult r = fn(m, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void *>(p), dims, strides, box, es,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, bf16 ? CU_TENSOR_MAP_SWIZZLE_NONE : CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return agpt_set_error(AGPT_E_CUDA, "tensor map of %lld x %d: error %d", (long long)rows, cols, (int)r);
    return AGPT_OK;
}
int encode_map(CUtensorMap *m, const float *p, int64_t rows, int cols, int ld, int box_rows) {
    return encode_map_any(m, p, rows, cols, (int64_t)ld * 4, box_rows, false);
}
int encode_map_bf16(CUtensorMap *m, const void *p, int64_t rows, int cols) { return encode_map_any(m, p, rows, cols, (int64_t)cols * 2, 32, true); }

template <typename Kern>
int allow_smem(Kern k, bool *done) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && done[dev]) return AGPT_OK;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_LIMIT);
    if (e != cudaSuccess) return agpt_set_error(AGPT_E_CUDA, "step gemm: shared memory limit: %s", cudaGetErrorString(e));
    if (dev >= 0 && dev < 64) done[dev] = true;
    return AGPT_OK;
}

// bit 1: a bounded wait of one of the kernels below ran out
__device__ int g_step_status = 0;

// a wait of a whole warp whose lanes go on together (tensor-memory instructions follow)
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, volatile int *abort_flag) {
    return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag));
}

// two barriers asked for at once (the latencies of two polls overlap)
__device__ __forceinline__ bool warp_wait2(uint32_t b0, uint32_t p0, uint32_t b1, uint32_t p1, volatile int *abort_flag) {
    const bool d0 = mbar_try(b0, p0), d1 = mbar_try(b1, p1);
    if (__all_sync(0xffffffffu, d0 && d1)) return true;
    return warp_wait(b0, p0, abort_flag) && warp_wait(b1, p1, abort_flag);
}

// the six partial products, small ones first
__device__ __forceinline__ void six_products(uint32_t d, uint32_t a, uint32_t b, uint32_t b_plane16, uint32_t b_step16, uint32_t idesc) {
    constexpr int PA[6] = {1, 0, 2, 0, 1, 0}, PB[6] = {1, 2, 0, 1, 0, 0};
    const uint32_t pl[3] = {b, b + b_plane16, b + 2 * b_plane16};
#pragma unroll
    for (int i = 0; i < 6; i++)
#pragma unroll
        for (int k = 0; k < 4; k++) mma_ts(d, a + PA[i] * 32 + k * 8, pl[PB[i]] + k * b_step16, desc_hi(1024), idesc, i + k > 0);
}

// ---------------------------------------------------------------------------------------------------------------------
// weight images
// ---------------------------------------------------------------------------------------------------------------------
constexpr int SPLIT_JOBS = 56;
struct SplitArgs {
    WeightSplitJob job[SPLIT_JOBS];
    int first_block[SPLIT_JOBS + 1];
    int n;
};

// one block = 32 n x 64 k of one job; reads along the matrix rows, transposes through shared memory
__global__ void __launch_bounds__(256) split_weights_kernel(const __grid_constant__ SplitArgs a) {
    pdl_wait();
    pdl_next();
    __shared__ float s[64][33];
    int j = 0;
    while (j + 1 < a.n && (int)blockIdx.x >= a.first_block[j + 1]) j++;
    const WeightSplitJob &w = a.job[j];
    const int b = blockIdx.x - a.first_block[j];
    const int nn = w.n_is_col ? w.cols : w.rows, kk = w.n_is_col ? w.rows : w.cols;
    const int kblocks = (w.k_pad + 63) / 64;
    const int n_first = (b / kblocks) * 32, k_first = (b % kblocks) * 64;
    for (int i = threadIdx.x; i < 2048; i += 256) {
        int n, k;
        if (w.n_is_col) { n = i & 31; k = i >> 5; } else { k = i & 63; n = i >> 6; }
        float v = 0.f;
        if (n_first + n < nn && k_first + k < kk) {
            const int r = w.n_is_col ? k_first + k : n_first + n, c = w.n_is_col ? n_first + n : k_first + k;
            v = __ldg(w.w + (int64_t)r * w.cols + c);
            if (w.gain) v *= __ldg(w.gain + r);
        }
        s[k][n] = v;
    }
    __syncthreads();
    const int n = threadIdx.x >> 3, c = threadIdx.x & 7;    // 32 n x 8 chunks of 8 k
    if (n_first + n >= w.n_pad || k_first + c * 8 >= w.k_pad) return;
    const int gn = w.n0 + n_first + n, gk = w.k0 + k_first + c * 8;
    uint32_t p[3][4];
#pragma unroll
    for (int q = 0; q < 4; q++) split3(f2_pack(s[c * 8 + 2 * q][n], s[c * 8 + 2 * q + 1][n]), p[0][q], p[1][q], p[2][q]);
    uint8_t *base = w.image + ((int64_t)((gn >> 7) * w.kb + (gk >> 6)) * 3 << 14) + (gn & 127) * 128 + ((((gk & 63) >> 3) ^ (gn & 7)) << 4);
#pragma unroll
    for (int q = 0; q < 3; q++) *reinterpret_cast<uint4 *>(base + (q << 14)) = make_uint4(p[q][0], p[q][1], p[q][2], p[q][3]);
}

// ---------------------------------------------------------------------------------------------------------------------
// rows x weights
// ---------------------------------------------------------------------------------------------------------------------
struct RowArgs {
    RowGemm g;
    int nt, n_tiles, kb;             // width of a column tile, column tiles, 64-k blocks
    int n_a, n_b, stationary;        // shared-memory stages; the weight blocks are loaded once
    int unit_tiles;                  // row tiles that share one pass over the weight blocks (1 or 2)
    int64_t row_tiles, units;
    int rope_stride;                 // entries per position of the shared table (head_dim / 2 + 1)
    int cluster;                     // the column tiles of a row tile are one cluster (whole-row epilogues on few rows), each block has one unit
    uint32_t off_b, off_out, off_bias, off_rope, off_x, off_bar;
};
struct RowMaps { CUtensorMap a[3], o[3], add, x; };

constexpr int ROW_THREADS = 512;
// registers per warpgroup: the launch gives 128 to each of the four (their sum, 512, is what a split may hand out)
constexpr int REG_ISSUE = 48, REG_CONV = 96, REG_ACC = 184;
static_assert(REG_ISSUE + REG_CONV + 2 * REG_ACC <= 4 * 128, "setmaxnreg draws on the registers of the launch");

// Epilogues that need the whole row.  On many rows a block has all its columns; on few (every block has one unit) 32 of them: one block would walk
// the K loop alone, 2.4 us per 64 k, while most SMs have nothing to do.  The blocks of a row tile form a cluster and exchange what they need through each
// other's shared memory.  Measured on 60 rows, 512 k, 128 columns, within a step's chain of launches: 20.5 -> 17 us.
template <int EPI> __device__ __forceinline__ constexpr bool whole_row_epi() { return EPI == EPI_ADD || EPI == EPI_NORM_BWD; }

template <int PRO, int EPI>
__global__ void __launch_bounds__(ROW_THREADS, 1)
row_gemm_kernel(const __grid_constant__ RowMaps maps, const __grid_constant__ RowArgs P) {
    extern __shared__ __align__(1024) unsigned char dyn[];
    const RowGemm &g = P.g;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    unsigned char *smem = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(dyn) + 1023) & ~(uintptr_t)1023);
    const uint32_t sA = smem_u32(smem), sB = sA + P.off_b, bars = sA + P.off_bar;
    volatile int &s_abort = *reinterpret_cast<volatile int *>(smem + P.off_bar + BAR_BYTES - 16);
    uint32_t &s_tmem = *reinterpret_cast<uint32_t *>(smem + P.off_bar + BAR_BYTES - 8);
    float *s_bias = reinterpret_cast<float *>(smem + P.off_bias);
    float4 *s_rope = reinterpret_cast<float4 *>(smem + P.off_rope);       // per pair of columns {cos, cos, -sin, sin}
    // barriers: A stages full / empty, B stages full / empty, tensor-memory A stages full / empty, accumulators full / empty (a pair for each
    // group of accumulator warps and accumulator)
    const uint32_t aF = bars, aE = aF + 8 * P.n_a, bF = aE + 8 * P.n_a, bE = bF + 8 * P.n_b, tF = bE + 8 * P.n_b, tE = tF + 16, cF = tE + 16, cE = cF + 32, oF = cE + 32, xF = oF + 128;
    const int n_tile = blockIdx.x % P.n_tiles, n0 = n_tile * P.nt;
    const int64_t slot = blockIdx.x / P.n_tiles, n_slots = gridDim.x / P.n_tiles;
    const int nt_mma = (min(P.nt, g.N - n0) + 15) & ~15;
    const uint32_t b_plane = (uint32_t)P.nt * 128, b_stage = 3 * b_plane;

    if (warp == 3 && lane == 0) {
        for (int i = 0; i < P.n_b; i++) { mbar_init(bF + 8 * i, 1); mbar_init(bE + 8 * i, P.unit_tiles); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        for (int i = 0; i < g.n_seg; i++) prefetch_map(&maps.a[i]);
        prefetch_map(&maps.o[0]);
        if (EPI == EPI_QKV) { prefetch_map(&maps.o[1]); prefetch_map(&maps.o[2]); }
        if (EPI == EPI_ADD || EPI == EPI_NORM_BWD) { prefetch_map(&maps.add); prefetch_map(&maps.x); }
    }
    if (tid == 0) {
        s_abort = 0;
        for (int i = 0; i < P.n_a; i++) { mbar_init(aF + 8 * i, 1); mbar_init(aE + 8 * i, 4); }
        for (int i = 0; i < 2; i++) { mbar_init(tF + 8 * i, 4); mbar_init(tE + 8 * i, 1); }
        for (int i = 0; i < 4; i++) { mbar_init(cF + 8 * i, 1); mbar_init(cE + 8 * i, 4); }
        for (int i = 0; i < 16; i++) mbar_init(oF + 8 * i, 1);
        for (int i = 0; i < 4; i++) mbar_init(xF + 8 * i, P.n_tiles);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) tmem_alloc(smem_u32(&s_tmem), TMEM_COLS);
    if (whole_row_epi<EPI>() && P.cluster) cluster_sync();       // barriers that other blocks arrive at
    pdl_wait();
    pdl_next();
    auto load_b = [&](int stage, int kb) {
        const uint8_t *img = g.image + (((int64_t)(n0 >> 7) * P.kb) * 3 << 14) + (n0 & 127) * 128;
        mbar_expect(bF + 8 * stage, b_stage);
        for (int q = 0; q < 3; q++) bulk_load(sB + stage * b_stage + q * b_plane, img + ((int64_t)(kb * 3 + q) << 14), b_plane, bF + 8 * stage);
    };
    // weights that stay are asked for by the thread that set their barriers up: by the loading thread, ahead of the rows, they held these up
    if (warp == 3 && lane == 0 && P.stationary) for (int kb = 0; kb < P.kb; kb++) load_b(kb, kb);
    for (int i = tid; i < P.nt; i += ROW_THREADS) s_bias[i] = (g.bias && n0 + i < g.N) ? __ldg(g.bias + n0 + i) : 0.f;
    if (EPI == EPI_QKV && g.cosv) {
        const int half = g.head_dim >> 1;
        for (int i = tid; i < g.n_pos * half; i += ROW_THREADS) {
            const int p = i / half, j = i - p * half;
            const float c = __ldg(g.cosv + (int64_t)p * g.head_dim + 2 * j), s = __ldg(g.sinv + (int64_t)p * g.head_dim + 2 * j);
            s_rope[p * P.rope_stride + j] = make_float4(c, c, -s, s);
        }
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = s_tmem;

    if (warp < 4) {
        regs_dec<REG_ISSUE>();
        if (warp == 0 && lane == 0) {
            // ---------------- loads ----------------
            int as = 0, bs = 0;
            uint32_t ap = 0, bp = 0;
            bool ok = true;
            for (int64_t u = slot; ok && u < P.units; u += n_slots) {
                const int64_t t0 = u * P.unit_tiles;
                const int T = (int)min((int64_t)P.unit_tiles, P.row_tiles - t0);
                for (int kb = 0; ok && kb < P.kb; kb++) {
                    if (!P.stationary) {
                        if (!(ok = mbar_wait(bE + 8 * bs, bp ^ 1, &s_abort))) break;
                        load_b(bs, kb);
                        if (++bs == P.n_b) { bs = 0; bp ^= 1; }
                    }
                    for (int t = 0; ok && t < T; t++)
                        for (int j = 0; j < 2; j++) {
                            if (!(ok = mbar_wait(aE + 8 * as, ap ^ 1, &s_abort))) break;
                            mbar_expect(aF + 8 * as, A_BOX);
                            // columns behind the last segment are read as zeros (out of the map's range)
                            const int cc = kb * 64 + j * 32;
                            const int seg = min(cc / g.seg_cols, g.n_seg - 1);
                            tma_load_2d(sA + as * A_BOX, &maps.a[seg], cc - seg * g.seg_cols, (int)((t0 + t) * TM), aF + 8 * as);
                            if (++as == P.n_a) { as = 0; ap ^= 1; }
                        }
                }
            }
            if (!ok) {                          // copies in flight land before the block leaves
                for (int i = 0; i < P.n_a; i++) { volatile int none = 0; mbar_wait(aF + 8 * i, ap, &none); }
                for (int i = 0; i < P.n_b; i++) { volatile int none = 0; mbar_wait(bF + 8 * i, bp, &none); }
            }
        } else if (warp == 1 || warp == 2) {
            // ---------------- MMAs ----------------
            // A warp per accumulator: a wait costs an issuing warp 140 to 170 clocks even where the barrier is complete, and the tensor pipe
            // queues no more than two or three MMAs, so that one warp alone left it idle for a quarter of the time (24 MMAs of 128 columns behind
            // two waits: 1951 clocks, two warps in turn 1557, the pipe's own 1536).  A warp stays converged, one elected lane issues (29 clocks
            // per MMA instead of 60).  Two row tiles per unit: a warp per tile.  One: the k blocks alternate, and the group of accumulator warps
            // that owns the tile reads both accumulators in turn.
            const int own = warp - 1;
            const bool pair = P.unit_tiles == 2;
            const uint32_t idesc = idesc_bf16(nt_mma, false), acc = tmem + own * ACC_COLS;
            int bs = 0, last = -1;                          // last: the group that reads what this accumulator held before
            uint32_t bp = 0, seen = 0, step = 0, uses[2] = {0, 0};
            int64_t iter = 0;
            bool ok = true;
            for (int64_t u = slot; ok && u < P.units; u += n_slots, iter++) {
                const int T = (int)min((int64_t)P.unit_tiles, P.row_tiles - u * P.unit_tiles);
                for (int kb = 0; ok && kb < P.kb; kb++, step += T) {
                    const uint32_t s = pair ? step + own : step, ts = s & 1;
                    const int grp = pair ? own : (int)(iter & 1);
                    if (pair ? own < T : (int)ts == own) {
                        if (P.stationary) {
                            bs = kb;
                            if (!((seen >> kb) & 1) && !(ok = warp_wait(bF + 8 * bs, 0, &s_abort))) break;
                            seen |= 1u << kb;
                        } else if (!(ok = warp_wait(bF + 8 * bs, bp, &s_abort))) break;
                        if (last >= 0) ok = warp_wait2(cE + 8 * (2 * last + own), ((last ? uses[1] : uses[0]) - 1) & 1, tF + 8 * ts, (s >> 1) & 1, &s_abort);
                        else ok = warp_wait(tF + 8 * ts, (s >> 1) & 1, &s_abort);
                        if (!ok) break;
                        fence_after();
                        if (elect_one()) {
                            six_products(acc, tmem + 2 * ACC_COLS + ts * TA_COLS, desc_lo(sB + bs * b_stage, 16), b_plane >> 4, 2, idesc);
                            commit(tE + 8 * ts);
                            commit(cF + 8 * (2 * grp + own));
                            if (!P.stationary) commit(bE + 8 * bs);
                        }
                        __syncwarp();
                        last = grp;
                        if (grp) uses[1]++; else uses[0]++;
                    } else if (pair && !P.stationary) {
                        // The last unit has one tile; this is the other warp's share of the stage.  It waits as if it read it: an arrival a phase
                        // early would free the stage under the first warp.
                        if (!(ok = warp_wait(bF + 8 * bs, bp, &s_abort))) break;
                        if (lane == 0) mbar_arrive(bE + 8 * bs);
                        __syncwarp();
                    }
                    if (!P.stationary && ++bs == P.n_b) { bs = 0; bp ^= 1; }
                }
            }
            if (!ok && elect_one()) {                          // MMAs in flight finish before tensor memory is released
                commit(tE + 8 * own);
                volatile int none = 0;
                for (int i = 0; i < 2; i++) mbar_wait(tE + 8 * own, i, &none);
            }
            __syncwarp();
        }
    } else if (warp < 8) {
        regs_dec<REG_CONV>();
        // ---------------- float32 rows -> three bf16 planes in tensor memory ----------------
        const int row = tid - 128;
        const uint32_t lane_base = (uint32_t)(row & 96) << 16;
        uint32_t at[8];                                 // the row's 16-byte pieces in order
#pragma unroll
        for (int i = 0; i < 8; i++) at[i] = (i ^ (row & 7)) << 4;
        int as = 0, ts = 0;
        uint32_t ap = 0, tp = 0;
        bool ok = true;
        for (int64_t u = slot; ok && u < P.units; u += n_slots) {
            const int64_t t0 = u * P.unit_tiles;
            const int T = (int)min((int64_t)P.unit_tiles, P.row_tiles - t0);
            float mean[2] = {0.f, 0.f}, mul[2] = {1.f, 1.f};
            if (PRO != PRO_PLAIN) {
#pragma unroll
                for (int t = 0; t < 2; t++) {
                    const int64_t r = (t0 + t) * TM + row;
                    if (t < T && r < g.rows) {
                        if (PRO == PRO_NORM) { const float2 st = __ldg(g.stats + r); mean[t] = st.x; mul[t] = st.y; }
                        else mul[t] = __ldg(g.row_scale + r);
                    }
                }
            }
            for (int kb = 0; ok && kb < P.kb; kb++) {
                for (int t = 0; t < T; t++) {
                    const f2 mn = f2_same(-(t ? mean[1] : mean[0])), ml = f2_same(t ? mul[1] : mul[0]);
                    const uint32_t dst = tmem + 2 * ACC_COLS + ts * TA_COLS + lane_base;
                    // both boxes and the place in tensor memory are asked for at once: three waits one after the other took 500 clocks of a step
                    const int as1 = as + 1 == P.n_a ? 0 : as + 1;
                    const uint32_t ap1 = as1 ? ap : ap ^ 1;
                    const bool full0 = mbar_try(aF + 8 * as, ap), full1 = mbar_try(aF + 8 * as1, ap1), room = mbar_try(tE + 8 * ts, tp ^ 1);
#pragma unroll
                    for (int j = 0; j < 2; j++) {
                        if (!__all_sync(0xffffffffu, j ? full1 : full0) && !(ok = warp_wait(aF + 8 * as, ap, &s_abort))) break;
                        const uint32_t src = sA + as * A_BOX + row * 128;
                        uint32_t p[3][16];
#pragma unroll
                        for (int c = 0; c < 8; c++) {
                            ulonglong2 v = lds_f4(src ^ at[c]);
                            if (PRO == PRO_NORM) { v.x = f2_mul(f2_add(v.x, mn), ml); v.y = f2_mul(f2_add(v.y, mn), ml); }
                            if (PRO == PRO_SCALE) { v.x = f2_mul(v.x, ml); v.y = f2_mul(v.y, ml); }
                            split3(v.x, p[0][2 * c], p[1][2 * c], p[2][2 * c]);
                            split3(v.y, p[0][2 * c + 1], p[1][2 * c + 1], p[2][2 * c + 1]);
                        }
                        __syncwarp();           // the stage has been read
                        if (lane == 0) mbar_arrive(aE + 8 * as);
                        if (++as == P.n_a) { as = 0; ap ^= 1; }
                        if (j == 0) {
                            if (!__all_sync(0xffffffffu, room) && !(ok = warp_wait(tE + 8 * ts, tp ^ 1, &s_abort))) break;
                            fence_after();
                        }
#pragma unroll
                        for (int q = 0; q < 3; q++) tmem_st16(dst + q * 32 + j * 16, p[q]);
                    }
                    if (!ok) break;
                    tmem_wait_st();
                    fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(tF + 8 * ts);
                    if (++ts == 2) { ts = 0; tp ^= 1; }
                }
            }
        }
    } else {
        regs_inc<REG_ACC>();
        // ---------------- accumulators: tensor memory -> registers -> rows ----------------
        // Rows enter and leave through the warp's two staging buffers (32 rows x 32 columns, swizzled) by TMA: a thread owns
        // a row, and 32-byte accesses to 32 different rows per instruction held the whole block up.
        const int grp = warp >= 12, wrow = (warp & 3) * 32 + lane;
        const uint32_t acc_addr = tmem + ((uint32_t)(warp & 3) << 21);
        unsigned char *stg = smem + P.off_out + (warp - 8) * 8192;
        const uint32_t u_stg = smem_u32(stg), lF = oF + (warp - 8) * 16;
        const int sw = lane & 7;
        uint32_t lp[2] = {0, 0};                          // parities of the two buffers' loads
        auto piece = [&](int buf, int c16) { return u_stg + buf * 4096 + lane * 128 + ((c16 ^ sw) << 4); };
        // before chunk c is written: the store that used its buffer last has read it.  That is the store before the last one, but for the first chunk of a
        // tile of an odd number of chunks, whose buffer the tile before ended with.
        auto buffer_free = [&](int c, int chunks) { if (c == 0 && (chunks & 1)) stores_read<0>(); else stores_read<1>(); };
        auto fetch = [&](int buf, const CUtensorMap *m, int x, int y) {       // one lane; the buffer is free
            mbar_expect(lF + 8 * buf, 4096);
            tma_load_2d(u_stg + buf * 4096, m, x, y, lF + 8 * buf);
        };
        uint32_t cp = 0;                                  // phases of this group's two accumulators
        int64_t iter = 0;
        bool ok = true;
        for (int64_t u = slot; ok && u < P.units; u += n_slots, iter++) {
            const int64_t t0 = u * P.unit_tiles;
            int64_t tile = t0 + grp;
            if (P.unit_tiles == 1) { if ((iter & 1) != grp) continue; tile = t0; }
            if (tile >= P.row_tiles) continue;
            const int64_t r = tile * TM + wrow;
            const int y0 = (int)(tile * TM) + (warp & 3) * 32;
            const int chunks = (min(P.nt, g.N - n0) + 31) >> 5;
            // what the first two chunks need is fetched under the MMAs
            const CUtensorMap *in_map = EPI == EPI_NORM_BWD ? &maps.x : &maps.add;
            constexpr bool has_in = EPI == EPI_NORM_BWD || EPI == EPI_ADD;
            if (has_in && lane == 0) {
                stores_read<0>();
                for (int c = 0; c < 2 && c < chunks; c++) fetch(c, in_map, n0 + c * 32, y0);
            }
            __syncwarp();
            f2 acc[ACC_COLS / 2];                         // two columns each; starts from the bias
#pragma unroll
            for (int i = 0; i < ACC_COLS / 2; i++) acc[i] = *reinterpret_cast<const f2 *>(s_bias + 2 * i);
            for (int kb = 0; kb < P.kb; kb++) {
                const int a = P.unit_tiles == 2 ? grp : (int)((iter * P.kb + kb) & 1);
                if (!(ok = warp_wait(cF + 8 * (2 * grp + a), (cp >> a) & 1, &s_abort))) break;
                cp ^= 1u << a;
                fence_after();
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    if (c * 32 < nt_mma) {
                        uint32_t v[32];
                        tmem_ld32(acc_addr + a * ACC_COLS + c * 32, v);
#pragma unroll
                        for (int i = 0; i < 16; i++) acc[c * 16 + i] = f2_add(acc[c * 16 + i], f2_pack(v[2 * i], v[2 * i + 1]));
                    }
                }
                fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(cE + 8 * (2 * grp + a));
            }
            if (!ok) break;
            // epilogue of the tile
            if (EPI == EPI_BIAS || EPI == EPI_RELU || EPI == EPI_MASKED || EPI == EPI_ADD) {
                const int64_t mask_at = r * (g.N >> 5) + (n0 >> 5);
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    if (c >= chunks) continue;
                    const int buf = c & 1;
                    uint32_t bits = 0;
                    if (EPI == EPI_MASKED) bits = r < g.rows ? __ldg(g.mask_in + mask_at + c) : 0u;
                    if (EPI == EPI_ADD) {
                        if (!(ok = warp_wait(lF + 8 * buf, lp[buf], &s_abort))) break;
                        lp[buf] ^= 1;
                    } else {
                        if (lane == 0) buffer_free(c, chunks);
                        __syncwarp();
                    }
#pragma unroll
                    for (int q = 0; q < 8; q++) {
                        ulonglong2 v = make_ulonglong2(acc[c * 16 + 2 * q], acc[c * 16 + 2 * q + 1]);
                        if (EPI == EPI_ADD) {
                            const ulonglong2 x = lds_f4(piece(buf, q));
                            v.x = f2_add(v.x, x.x); v.y = f2_add(v.y, x.y);
                            acc[c * 16 + 2 * q] = v.x; acc[c * 16 + 2 * q + 1] = v.y;
                        }
                        if (EPI == EPI_RELU || EPI == EPI_MASKED) {
                            const float2 a = f2_get(v.x), b = f2_get(v.y);
                            float w[4] = {a.x, a.y, b.x, b.y};
#pragma unroll
                            for (int i = 0; i < 4; i++) {
                                if (EPI == EPI_RELU) {      // 0 - w is negative exactly where w > 0
                                    w[i] = fmaxf(w[i], 0.f);
                                    bits = __funnelshift_l(__float_as_uint(0.f - w[i]), bits, 1);
                                } else {
                                    w[i] = __uint_as_float(__float_as_uint(w[i]) & (uint32_t)((int32_t)(bits << (q * 4 + i)) >> 31));
                                }
                            }
                            v = make_ulonglong2(f2_pack(w[0], w[1]), f2_pack(w[2], w[3]));
                        }
                        sts_f4(piece(buf, q), v.x, v.y);
                    }
                    if (EPI == EPI_RELU && r < g.rows) g.mask_out[mask_at + c] = bits;
                    fence_async_smem();
                    __syncwarp();
                    if (lane == 0) {
                        if (y0 < g.rows) tma_store_2d(&maps.o[0], u_stg + buf * 4096, n0 + c * 32, y0);
                        if (EPI == EPI_ADD && c + 2 < chunks) { stores_read<0>(); fetch(buf, &maps.add, n0 + (c + 2) * 32, y0); }
                    }
                    __syncwarp();
                }
                if (EPI == EPI_ADD && g.stats_out) {               // N <= 128: the thread holds the whole row; zeros behind the last row
                    if (P.cluster) {                               // the first block collects it from the others' staging buffers
                        __syncwarp();
                        if (lane == 0) peer_arrive(peer_addr(xF + 8 * (warp & 3), 0));
                        if (n_tile != 0) continue;
                        if (!(ok = __all_sync(0xffffffffu, mbar_wait_cluster(xF + 8 * (warp & 3), 0, &s_abort)))) break;
#pragma unroll
                        for (int c = 1; c < 4; c++)
                            if (c < P.n_tiles)
#pragma unroll
                                for (int q = 0; q < 8; q++) {
                                    const ulonglong2 v = peer_lds_f4(peer_addr(piece(0, q), c));
                                    acc[c * 16 + 2 * q] = v.x; acc[c * 16 + 2 * q + 1] = v.y;
                                }
                    }
                    f2 sum = 0, sq = 0;
#pragma unroll
                    for (int c = 0; c < 4; c++)
                        if (c * 32 < g.N)
#pragma unroll
                            for (int i = 0; i < 16; i++) sum = f2_add(sum, acc[c * 16 + i]);
                    const float2 s2 = f2_get(sum);
                    const float mu = (s2.x + s2.y) / (float)g.N;
                    const f2 nmu = f2_same(-mu);
#pragma unroll
                    for (int c = 0; c < 4; c++)
                        if (c * 32 < g.N)
#pragma unroll
                            for (int i = 0; i < 16; i++) { const f2 d = f2_add(acc[c * 16 + i], nmu); sq = f2_fma(d, d, sq); }
                    const float2 q2 = f2_get(sq);
                    g.stats_out[r] = r < g.rows ? make_float2(mu, 1.0f / sqrtf((q2.x + q2.y) / (float)g.N + 1e-5f)) : make_float2(0.f, 0.f);
                }
            } else if (EPI == EPI_QKV) {
                const int D = g.N / 3;
                const uint32_t tab = smem_u32(s_rope + (int64_t)(g.cosv && r < g.rows ? min(__ldg(g.pos + r), g.n_pos - 1) : 0) * P.rope_stride);
                const int hmask = (g.head_dim >> 1) - 1;
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    const int col = n0 + c * 32, buf = c & 1;
                    if (c >= chunks) continue;
                    const int which = col / D, dc = col - which * D;
                    if (lane == 0) buffer_free(c, chunks);
                    __syncwarp();
                    if (which < 2 && g.cosv) {
                        const int j0 = (dc & (g.head_dim - 1)) >> 1;
#pragma unroll
                        for (int j = 0; j < 16; j++) {
                            const ulonglong2 cs = lds_f4(tab + (((j0 + j) & hmask) << 4));
                            const float2 v = f2_get(acc[c * 16 + j]);
                            acc[c * 16 + j] = f2_fma(f2_pack(v.y, v.x), cs.y, f2_mul(acc[c * 16 + j], cs.x));
                        }
                    }
                    if (which > 0 && g.kv_bf16) {            // 64-byte rows, not swizzled
                        uint4 *o = reinterpret_cast<uint4 *>(stg + buf * 4096 + lane * 64);
#pragma unroll
                        for (int q = 0; q < 4; q++) {
                            uint32_t w[4];
#pragma unroll
                            for (int i = 0; i < 4; i++) { const float2 v = f2_get(acc[c * 16 + q * 4 + i]); w[i] = pack_bf16(v.x, v.y); }
                            o[q] = make_uint4(w[0], w[1], w[2], w[3]);
                        }
                    } else {
#pragma unroll
                        for (int q = 0; q < 8; q++) sts_f4(piece(buf, q), acc[c * 16 + 2 * q], acc[c * 16 + 2 * q + 1]);
                    }
                    fence_async_smem();
                    __syncwarp();
                    if (lane == 0 && y0 < g.rows) tma_store_2d(&maps.o[which], u_stg + buf * 4096, dc, y0);
                    __syncwarp();
                }
            } else {
                // layer-norm backward of the whole row: dx = (dn - mean(dn) - norm * mean(dn * norm)) / std + add
                const float2 st = __ldg(g.stats + r);
                const f2 nmu = f2_same(-st.x), rs = f2_same(st.y);
                f2 a1 = 0, a2 = 0;
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    if (c >= chunks) continue;
                    const int buf = c & 1;
                    if (!(ok = warp_wait(lF + 8 * buf, lp[buf], &s_abort))) break;
                    lp[buf] ^= 1;
#pragma unroll
                    for (int q = 0; q < 8; q++) {
                        const ulonglong2 x = lds_f4(piece(buf, q));
                        a1 = f2_add(a1, f2_add(acc[c * 16 + 2 * q], acc[c * 16 + 2 * q + 1]));
                        a2 = f2_fma(acc[c * 16 + 2 * q], f2_mul(f2_add(x.x, nmu), rs), a2);
                        a2 = f2_fma(acc[c * 16 + 2 * q + 1], f2_mul(f2_add(x.y, nmu), rs), a2);
                    }
                    __syncwarp();
                    if (lane == 0 && c + 2 < chunks) fetch(buf, &maps.x, n0 + (c + 2) * 32, y0);
                }
                if (!ok) break;
                if (P.cluster) {                                   // every block has its columns' share of the two sums; added in column order
                    const uint32_t mine = sA + P.off_x + (n_tile * TM + wrow) * 16;
                    for (int t = 0; t < P.n_tiles; t++) peer_sts_f4(peer_addr(mine, t), a1, a2);
                    __syncwarp();
                    if (lane < P.n_tiles) peer_arrive(peer_addr(xF + 8 * (warp & 3), lane));
                    if (!(ok = __all_sync(0xffffffffu, mbar_wait_cluster(xF + 8 * (warp & 3), 0, &s_abort)))) break;
                    a1 = a2 = 0;
                    for (int t = 0; t < P.n_tiles; t++) {
                        const ulonglong2 v = lds_f4(sA + P.off_x + (t * TM + wrow) * 16);
                        a1 = f2_add(a1, v.x); a2 = f2_add(a2, v.y);
                    }
                }
                const float2 s1 = f2_get(a1), s2 = f2_get(a2);
                const f2 m1 = f2_same(-(s1.x + s1.y) / (float)g.N), m2 = f2_same(-(s2.x + s2.y) / (float)g.N);
                __syncwarp();
                if (lane == 0) { fetch(0, &maps.x, n0, y0); if (g.add) fetch(1, &maps.add, n0, y0); }
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    if (c >= chunks) continue;
                    if (!(ok = warp_wait(lF, lp[0], &s_abort) && (!g.add || warp_wait(lF + 8, lp[1], &s_abort)))) break;
                    lp[0] ^= 1; lp[1] ^= g.add ? 1 : 0;
#pragma unroll
                    for (int q = 0; q < 8; q++) {
                        ulonglong2 x = lds_f4(piece(0, q));
                        const ulonglong2 y = g.add ? lds_f4(piece(1, q)) : make_ulonglong2(0, 0);
                        x.x = f2_fma(f2_fma(f2_mul(f2_add(x.x, nmu), rs), m2, f2_add(acc[c * 16 + 2 * q], m1)), rs, y.x);
                        x.y = f2_fma(f2_fma(f2_mul(f2_add(x.y, nmu), rs), m2, f2_add(acc[c * 16 + 2 * q + 1], m1)), rs, y.y);
                        sts_f4(piece(0, q), x.x, x.y);
                    }
                    fence_async_smem();
                    __syncwarp();
                    if (lane == 0) {
                        if (y0 < g.rows) tma_store_2d(&maps.o[0], u_stg, n0 + c * 32, y0);
                        if (c + 1 < chunks) {
                            if (g.add) fetch(1, &maps.add, n0 + (c + 1) * 32, y0);
                            stores_read<0>();
                            fetch(0, &maps.x, n0 + (c + 1) * 32, y0);
                        }
                    }
                    __syncwarp();
                }
            }
            if (!ok) break;
            // end of the tile
        }
        if (lane == 0) {
            stores_read<0>();
            volatile int none = 0;
            if (!ok) for (int i = 0; i < 2; i++) mbar_wait(lF + 8 * i, lp[i], &none);      // fetches in flight
        }
        __syncwarp();
    }
    fence_before();
    __syncthreads();
    fence_after();
    if (whole_row_epi<EPI>() && P.cluster) cluster_sync();           // no block leaves while another reads its shared memory
    if (warp == 1) tmem_dealloc(tmem, TMEM_COLS);
    if (tid == 0 && s_abort) atomicOr(&g_step_status, 2);
}

template <int PRO, int EPI>
int launch_row(const RowArgs &P, const RowMaps &m, int grid, size_t smem, cudaStream_t st) {
    static bool done[64];
    if (int rc = allow_smem(row_gemm_kernel<PRO, EPI>, done)) return rc;
    pdl_launch_clusters(row_gemm_kernel<PRO, EPI>, P.cluster ? P.n_tiles : 1, grid, ROW_THREADS, smem, st, m, P);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return agpt_set_error(AGPT_E_CUDA, "row_gemm: %s", cudaGetErrorString(e));
    return AGPT_OK;
}

constexpr int OUT_BYTES = 8 * 8192;      // two staging buffers per accumulator warp
// Rotation in the q/k/v projection while its table takes at most this much of the shared memory that row stages would have: 64 positions of
// head_dim 32, 32 of 64.  An epoch of four layers takes, rotated here / in a pass of its own, us: d_model 128, 4 x 32, 32 positions 27620 /
// 28264, 64 positions (17 KB) 24231 / 24811; d_model 256, 4 x 64, 32 positions (17 KB) 35491 / 36133.  Above it the two are close and trade places:
// 4 x 32, 100 positions (27 KB) 32557 / 33547, but 4 x 64, 64 positions (34 KB) 37961 / 37835.
constexpr int ROPE_SMEM_MAX = 17 * 1024;

}  // namespace

bool agpt_row_gemm_rope_fits(int n_pos, int head_dim) { return (int64_t)n_pos * (head_dim / 2 + 1) * 16 <= ROPE_SMEM_MAX; }

int agpt_row_gemm(const RowGemm &g, cudaStream_t st) {
    if (g.rows <= 0) return AGPT_OK;
    const int sms = sm_count();
    RowArgs P;
    P.g = g;
    P.row_tiles = (g.rows + TM - 1) / TM;
    P.kb = (g.K + 63) / 64;
    const bool whole_row = g.epi == EPI_NORM_BWD || g.stats_out;
    if (whole_row && g.N > 128) return agpt_set_error(AGPT_E_ARG, "row_gemm: a row of %d columns does not fit one tile", g.N);
    // column tile: 128, or narrower (down to 32) while the launch would leave half of the SMs without work; a tile must not
    // cross the 128-column blocks of the image
    P.nt = g.N <= 128 ? (g.N + 15) & ~15 : 128;
    P.cluster = whole_row && g.N % 32 == 0 && g.N > 32 && P.row_tiles * (g.N / 32) <= sms;
    if (P.cluster) P.nt = 32;
    if (!whole_row && g.N % 32 == 0) {
        int nt = P.nt > 64 ? 64 : 32;
        while (nt >= 32 && nt < P.nt && P.row_tiles * ((g.N + P.nt - 1) / P.nt) * 2 <= sms) { P.nt = nt; nt >>= 1; }
    }
    P.n_tiles = (g.N + P.nt - 1) / P.nt;
    P.rope_stride = g.epi == EPI_QKV && g.cosv ? g.head_dim / 2 + 1 : 0;
    const int rope_bytes = P.rope_stride * g.n_pos * 16, b_stage = 3 * P.nt * 128, x_bytes = P.cluster ? P.n_tiles * TM * 16 : 0;
    const int room = SMEM_LIMIT - 1024 - OUT_BYTES - 512 - rope_bytes - x_bytes - BAR_BYTES;
    P.stationary = P.kb * b_stage + 2 * A_BOX <= room;
    P.n_b = P.stationary ? P.kb : 2;
    if (P.n_b > 16) { P.stationary = 0; P.n_b = 2; }
    P.n_a = std::min(8, (room - P.n_b * b_stage) / A_BOX);
    if (P.n_a < 2) return agpt_set_error(AGPT_E_LIMIT, "row_gemm: no shared memory left for the rows");
    P.off_b = (uint32_t)(P.n_a * A_BOX);
    P.off_out = P.off_b + (uint32_t)(P.n_b * b_stage);
    P.off_bias = P.off_out + OUT_BYTES;
    P.off_rope = P.off_bias + 512;
    P.off_x = P.off_rope + (uint32_t)rope_bytes;
    P.off_bar = P.off_x + (uint32_t)x_bytes;
    // two row tiles per pass over the weights once every SM has at least two such units
    P.unit_tiles = !P.cluster && (P.row_tiles + 1) / 2 * P.n_tiles >= 2 * sms ? 2 : 1;
    P.units = (P.row_tiles + P.unit_tiles - 1) / P.unit_tiles;
    const int64_t slots = std::min<int64_t>(P.units, std::max(1, sms / P.n_tiles));
    RowMaps m;
    for (int i = 0; i < 3; i++) {
        if (i >= g.n_seg) m.a[i] = m.a[0];
        else if (int rc = encode_map(&m.a[i], g.a[i], g.rows, g.seg_cols, g.lda, TM)) return rc;
    }
    if (g.epi == EPI_QKV) {
        for (int i = 0; i < 3; i++)
            if (int rc = i && g.kv_bf16 ? encode_map_bf16(&m.o[i], g.qkv[i], g.rows, g.N / 3) : encode_map(&m.o[i], (const float *)g.qkv[i], g.rows, g.N / 3, g.N / 3, 32)) return rc;
    } else {
        if (int rc = encode_map(&m.o[0], g.out, g.rows, g.N, g.ldo, 32)) return rc;
        m.o[1] = m.o[2] = m.o[0];
    }
    m.add = m.x = m.o[0];
    if (g.epi == EPI_ADD && !g.add) return agpt_set_error(AGPT_E_ARG, "row_gemm: nothing to add");
    if (g.add) if (int rc = encode_map(&m.add, g.add, g.rows, g.N, g.ldo, 32)) return rc;
    if (g.epi == EPI_NORM_BWD) {
        if (!g.x) return agpt_set_error(AGPT_E_ARG, "row_gemm: the layer-norm backward needs x");
        if (int rc = encode_map(&m.x, g.x, g.rows, g.N, g.N, 32)) return rc;
    }
    const int grid = (int)(slots * P.n_tiles);
    const size_t smem = (size_t)P.off_bar + BAR_BYTES + 1024;
    switch (g.epi * 3 + g.pro) {
        case EPI_BIAS * 3 + PRO_PLAIN: return launch_row<PRO_PLAIN, EPI_BIAS>(P, m, grid, smem, st);
        case EPI_BIAS * 3 + PRO_NORM: return launch_row<PRO_NORM, EPI_BIAS>(P, m, grid, smem, st);
        case EPI_BIAS * 3 + PRO_SCALE: return launch_row<PRO_SCALE, EPI_BIAS>(P, m, grid, smem, st);
        case EPI_RELU * 3 + PRO_NORM: return launch_row<PRO_NORM, EPI_RELU>(P, m, grid, smem, st);
        case EPI_MASKED * 3 + PRO_PLAIN: return launch_row<PRO_PLAIN, EPI_MASKED>(P, m, grid, smem, st);
        case EPI_ADD * 3 + PRO_PLAIN: return launch_row<PRO_PLAIN, EPI_ADD>(P, m, grid, smem, st);
        case EPI_QKV * 3 + PRO_NORM: return launch_row<PRO_NORM, EPI_QKV>(P, m, grid, smem, st);
        case EPI_NORM_BWD * 3 + PRO_PLAIN: return launch_row<PRO_PLAIN, EPI_NORM_BWD>(P, m, grid, smem, st);
        case EPI_NORM_BWD * 3 + PRO_SCALE: return launch_row<PRO_SCALE, EPI_NORM_BWD>(P, m, grid, smem, st);
    }
    return agpt_set_error(AGPT_E_ARG, "row_gemm: combination not instantiated");
}

int64_t agpt_weight_image_bytes(int n, int k) { return (int64_t)((n + 127) / 128) * ((k + 63) / 64) * 3 << 14; }

int agpt_split_weights(const WeightSplitJob *jobs, int n_jobs, cudaStream_t st) {
    for (int first = 0; first < n_jobs; first += SPLIT_JOBS) {
        SplitArgs a;
        a.n = std::min(SPLIT_JOBS, n_jobs - first);
        int blocks = 0;
        for (int i = 0; i < a.n; i++) {
            a.job[i] = jobs[first + i];
            a.first_block[i] = blocks;
            blocks += ((a.job[i].n_pad + 31) / 32) * ((a.job[i].k_pad + 63) / 64);
        }
        a.first_block[a.n] = blocks;
        pdl_launch(split_weights_kernel, blocks, 256, 0, st, a);
    }
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return agpt_set_error(AGPT_E_CUDA, "split_weights: %s", cudaGetErrorString(e));
    return AGPT_OK;
}

int agpt_step_gemm_status_word(const int **d_word) {
    cudaError_t e = cudaGetSymbolAddress((void **)d_word, g_step_status);
    if (e != cudaSuccess) return agpt_set_error(AGPT_E_CUDA, "device_status: %s", cudaGetErrorString(e));
    return AGPT_OK;
}
int agpt_step_gemm_status(int *out) {
    cudaError_t e = cudaMemcpyFromSymbol(out, g_step_status, sizeof(int));
    if (e != cudaSuccess) return agpt_set_error(AGPT_E_CUDA, "device_status: %s", cudaGetErrorString(e));
    return AGPT_OK;
}

// ---------------------------------------------------------------------------------------------------------------------
// contraction over the rows
// ---------------------------------------------------------------------------------------------------------------------
namespace {

struct alignas(64) ConJob {
    CUtensorMap a, b[3];
    RowContract g;
    int nt, halves, m_tiles, groups; // width of an accumulator, accumulators of a column group, 128-feature tiles, column groups
    int sectors;                     // the rows of partial sums start on 32-byte boundaries
    int64_t row_blocks;
};
// A launch forms one weight gradient, or (few rows) as many as there are at once.
constexpr int CON_JOBS = 40;
template <int JOBS> struct ConBatch {
    ConJob job[JOBS];
    int first_block[JOBS], n;
};
static_assert(sizeof(ConBatch<CON_JOBS>) <= 32764, "kernel parameters");

constexpr int CON_THREADS = 640, CON_ROWS = 64;
constexpr int CON_A = 4 * 8192, CON_B = 4 * 8192, CON_P = 3 * 16384;      // raw A, raw B (one half), B planes
constexpr uint32_t CON_OFF_B = 2 * CON_A, CON_OFF_P = CON_OFF_B + 2 * CON_B, CON_OFF_STAT = CON_OFF_P + 2 * CON_P, CON_OFF_SCALE = CON_OFF_STAT + 2 * 512,
                   CON_OFF_BAR = CON_OFF_SCALE + 2 * 256;
constexpr int CON_BAR_BYTES = 256;
constexpr size_t CON_SMEM = CON_OFF_BAR + CON_BAR_BYTES + 1024;
static_assert(CON_SMEM <= SMEM_LIMIT, "shared memory");
constexpr int CREG_ISSUE = 40, CREG_A = 64, CREG_B = 64, CREG_ACC = 152;
static_assert(CREG_ISSUE + CREG_A + CREG_B + 2 * CREG_ACC <= 5 * 96, "setmaxnreg draws on the registers of the launch");

template <int JOBS>
__global__ void __launch_bounds__(CON_THREADS, 1) contract_kernel(const __grid_constant__ ConBatch<JOBS> batch) {
    extern __shared__ __align__(1024) unsigned char dyn[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, wq = warp & 3;
    int job = 0;
    if (JOBS > 1) {
        for (int i = lane; i - lane < JOBS; i += 32) job += __popc(__ballot_sync(0xffffffffu, i < batch.n && (int)blockIdx.x >= batch.first_block[min(i, JOBS - 1)]));
        job--;
    }
    const ConJob &P = batch.job[job];
    const RowContract &g = P.g;
    const int block = blockIdx.x - (JOBS > 1 ? batch.first_block[job] : 0);
    unsigned char *smem = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(dyn) + 1023) & ~(uintptr_t)1023);
    const uint32_t sA = smem_u32(smem), sB = sA + CON_OFF_B, sP = sA + CON_OFF_P, bars = sA + CON_OFF_BAR;
    volatile int &s_abort = *reinterpret_cast<volatile int *>(smem + CON_OFF_BAR + CON_BAR_BYTES - 16);
    uint32_t &s_tmem = *reinterpret_cast<uint32_t *>(smem + CON_OFF_BAR + CON_BAR_BYTES - 8);
    const uint32_t aF = bars, aE = aF + 16, bF = aE + 16, bE = bF + 16, pF = bE + 16, pE = pF + 16, tF = pE + 16, tE = tF + 16, cF = tE + 16, cE = cF + 16;
    const int units = P.m_tiles * P.groups;
    const int unit = block % units, slice = block / units;
    const int m_first = (unit % P.m_tiles) * 128, n_first = (unit / P.m_tiles) * P.halves * P.nt;
    const int mb = (min(128, g.m - m_first) + 31) >> 5;                    // boxes of 32 features
    const int halves = P.halves == 2 && g.n - n_first > P.nt ? 2 : 1;
    const int w0 = min(P.nt, g.n - n_first), w1 = halves == 2 ? min(P.nt, g.n - n_first - P.nt) : 0;
    const int64_t rb0 = P.row_blocks * slice / g.slices, rb1 = P.row_blocks * (slice + 1) / g.slices;

    if (tid == 0) {
        s_abort = 0;
        for (int i = 0; i < 2; i++) {
            mbar_init(aF + 8 * i, 1); mbar_init(aE + 8 * i, 4); mbar_init(bF + 8 * i, 1); mbar_init(bE + 8 * i, 4);
            mbar_init(pF + 8 * i, 4); mbar_init(pE + 8 * i, 1); mbar_init(tF + 8 * i, 4); mbar_init(tE + 8 * i, halves);
            mbar_init(cF + 8 * i, 1); mbar_init(cE + 8 * i, 4);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) tmem_alloc(smem_u32(&s_tmem), TMEM_COLS);
    pdl_wait();
    pdl_next();
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = s_tmem;

    if (warp < 4) {
        regs_dec<CREG_ISSUE>();
        if (warp == 0 && lane == 0) {
            // ---------------- loads ----------------
            int as = 0, bs = 0;
            uint32_t ap = 0, bp = 0;
            bool ok = true;
            for (int64_t rb = rb0; ok && rb < rb1; rb++) {
                const int y = (int)(rb * CON_ROWS);
                if (!(ok = mbar_wait(aE + 8 * as, ap ^ 1, &s_abort))) break;
                mbar_expect(aF + 8 * as, (uint32_t)(mb * 8192 + (g.stats ? 512 : 0)));
                if (g.stats) bulk_load(sA + CON_OFF_STAT + as * 512, g.stats + rb * CON_ROWS, 512, aF + 8 * as);
                for (int j = 0; j < mb; j++) tma_load_2d(sA + as * CON_A + j * 8192, &P.a, m_first + j * 32, y, aF + 8 * as);
                if (++as == 2) { as = 0; ap ^= 1; }
                for (int h = 0; h < halves; h++) {
                    if (!(ok = mbar_wait(bE + 8 * bs, bp ^ 1, &s_abort))) break;
                    const int nb = ((h ? w1 : w0) + 31) >> 5;
                    mbar_expect(bF + 8 * bs, (uint32_t)(nb * 8192 + (g.row_scale ? 256 : 0)));
                    if (g.row_scale) bulk_load(sA + CON_OFF_SCALE + bs * 256, g.row_scale + rb * CON_ROWS, 256, bF + 8 * bs);
                    for (int j = 0; j < nb; j++) {
                        const int cc = n_first + h * P.nt + j * 32;
                        const int seg = min(cc / g.seg_cols, g.n_seg - 1);
                        tma_load_2d(sB + bs * CON_B + j * 8192, &P.b[seg], cc - seg * g.seg_cols, y, bF + 8 * bs);
                    }
                    if (++bs == 2) { bs = 0; bp ^= 1; }
                }
            }
            if (!ok) {
                volatile int none = 0;
                for (int i = 0; i < 2; i++) { mbar_wait(aF + 8 * i, ap, &none); mbar_wait(bF + 8 * i, bp, &none); }
            }
        } else if (warp >= 1 && warp <= halves) {
            // ---------------- MMAs: a warp per accumulator (see row_gemm_kernel) ----------------
            const int h = warp - 1;
            const uint32_t idesc = idesc_bf16(((h ? w1 : w0) + 15) & ~15, true);
            uint32_t i = 0;                                // each accumulator is used once per row block
            bool ok = true;
            for (int64_t rb = rb0; ok && rb < rb1; rb++, i++) {
                const uint32_t ts = i & 1, s = halves == 2 ? 2 * i + h : i, ps = s & 1;
                if (!(ok = warp_wait2(tF + 8 * ts, (i >> 1) & 1, cE + 8 * h, (i & 1) ^ 1, &s_abort))) break;
                if (!(ok = warp_wait(pF + 8 * ps, (s >> 1) & 1, &s_abort))) break;
                fence_after();
                if (elect_one()) {
                    six_products(tmem + h * ACC_COLS, tmem + 2 * ACC_COLS + ts * TA_COLS, desc_lo(sP + ps * CON_P, 8192), 1024, 128, idesc);
                    commit(pE + 8 * ps);
                    commit(tE + 8 * ts);
                    commit(cF + 8 * h);
                }
                __syncwarp();
            }
            if (!ok && elect_one()) {
                commit(pE + 8 * h);
                volatile int none = 0;
                for (int j = 0; j < 2; j++) mbar_wait(pE + 8 * h, j, &none);
            }
            __syncwarp();
        }
    } else if (warp < 8) {
        regs_dec<CREG_A>();
        // ---------------- A^T: thread = feature, walking down the rows of the staged tile ----------------
        int as = 0, ts = 0;
        uint32_t ap = 0, tp = 0;
        float csum = 0.f;
        const bool live = wq < mb;
        uint32_t at[8];                                 // this feature's place in the eight rows of a swizzle pattern
#pragma unroll
        for (int i = 0; i < 8; i++) at[i] = i * 128 + (((lane >> 2) ^ i) << 4) + ((lane & 3) << 2);
        for (int64_t rb = rb0; rb < rb1; rb++) {
            if (!warp_wait2(aF + 8 * as, ap, tE + 8 * ts, tp ^ 1, &s_abort)) break;
            fence_after();
            if (live) {
                const uint32_t src = sA + as * CON_A + wq * 8192;
                const uint32_t dst = tmem + 2 * ACC_COLS + ts * TA_COLS + ((uint32_t)wq << 21);
                f2 bsum = 0;
#pragma unroll 1
                for (int k0 = 0; k0 < CON_ROWS; k0 += 16) {
                    uint32_t p[3][8];
#pragma unroll
                    for (int k = 0; k < 16; k += 2) {
                        f2 v = f2_pack(lds_f1(src + at[k & 7] + (k0 + (k & 8)) * 128), lds_f1(src + at[(k + 1) & 7] + (k0 + (k & 8)) * 128));
                        if (g.stats) {
                            const float4 st = *reinterpret_cast<const float4 *>(smem + CON_OFF_STAT + as * 512 + (k0 + k) * 8);
                            v = f2_mul(f2_add(v, f2_pack(-st.x, -st.z)), f2_pack(st.y, st.w));
                        }
                        bsum = f2_add(bsum, v);
                        split3(v, p[0][k >> 1], p[1][k >> 1], p[2][k >> 1]);
                    }
#pragma unroll
                    for (int q = 0; q < 3; q++) tmem_st8(dst + q * 32 + (k0 >> 1), p[q]);
                }
                const float2 b2 = f2_get(bsum);
                csum += b2.x + b2.y;
                tmem_wait_st();
            }
            fence_before();
            __syncwarp();
            if (lane == 0) { mbar_arrive(aE + 8 * as); mbar_arrive(tF + 8 * ts); }
            if (++as == 2) { as = 0; ap ^= 1; }
            if (++ts == 2) { ts = 0; tp ^= 1; }
        }
        const int mm = m_first + tid - 128;
        if (g.transposed && g.col_part && n_first == 0 && mm < g.m) g.col_part[(int64_t)slice * g.col_ld + mm] = csum;
    } else if (warp < 12) {
        regs_dec<CREG_B>();
        // ---------------- B: 16-byte pieces of eight neighbouring columns, n contiguous ----------------
        // lane -> (box of 32 columns, group of 8 in it, row of a pair): eight neighbouring lanes read eight different
        // 16-byte chunks and write eight different ones
        const int sub = lane & 3, x4 = (lane >> 2) & 1, y8 = (lane >> 3) & 1, box = ((lane >> 4) << 1) + x4, odd = x4 ^ y8;
        // a warp takes rows 8 i + k of the block: everything but i is fixed
        const int k = 2 * wq + odd;
        const uint32_t get = sB + (box << 13) + k * 128 + (((2 * sub) ^ k) << 4);
        const uint32_t put = sP + ((box >> 1) << 13) + k * 128 + (((((box & 1) << 2) + sub) ^ k) << 4);
        int bs = 0, ps = 0;
        uint32_t bp = 0, pp = 0;
        f2 cs[2][4];
#pragma unroll
        for (int e = 0; e < 4; e++) cs[0][e] = cs[1][e] = 0;
        bool ok = true;
        for (int64_t rb = rb0; ok && rb < rb1; rb++) {
#pragma unroll
            for (int h = 0; h < 2; h++) {
                if (h >= halves) break;
                if (!(ok = warp_wait2(bF + 8 * bs, bp, pE + 8 * ps, pp ^ 1, &s_abort))) break;
                const int nb = ((h ? w1 : w0) + 31) >> 5;
                if (box < nb) {
                    const uint32_t dst = put + ps * CON_P, src = get + bs * CON_B;
                    f2 part[4] = {0, 0, 0, 0};
#pragma unroll 2
                    for (int i = 0; i < CON_ROWS / 8; i++) {
                        ulonglong2 u = lds_f4(src + i * 1024), v = lds_f4((src ^ 16) + i * 1024);
                        if (g.row_scale) {
                            const f2 f = f2_same(*reinterpret_cast<const float *>(smem + CON_OFF_SCALE + bs * 256 + (k + 8 * i) * 4));
                            u.x = f2_mul(u.x, f); u.y = f2_mul(u.y, f); v.x = f2_mul(v.x, f); v.y = f2_mul(v.y, f);
                        }
                        part[0] = f2_add(part[0], u.x); part[1] = f2_add(part[1], u.y); part[2] = f2_add(part[2], v.x); part[3] = f2_add(part[3], v.y);
                        uint32_t p[3][4];
                        split3(u.x, p[0][0], p[1][0], p[2][0]); split3(u.y, p[0][1], p[1][1], p[2][1]);
                        split3(v.x, p[0][2], p[1][2], p[2][2]); split3(v.y, p[0][3], p[1][3], p[2][3]);
#pragma unroll
                        for (int q = 0; q < 3; q++) sts_u4(dst + (q << 14) + i * 1024, p[q]);
                    }
#pragma unroll
                    for (int e = 0; e < 4; e++) cs[h][e] = f2_add(cs[h][e], part[e]);
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) { mbar_arrive(bE + 8 * bs); mbar_arrive(pF + 8 * ps); }
                if (++bs == 2) { bs = 0; bp ^= 1; }
                if (++ps == 2) { ps = 0; pp ^= 1; }
            }
        }
        if (!g.transposed && g.col_part && m_first == 0) {
            // column sums: [4 warps x 2 rows of a pair][2 halves][128] through the raw B area, added in a fixed order
            float *red = reinterpret_cast<float *>(smem + CON_OFF_B);
            asm volatile("bar.sync 1, 128;" ::: "memory");
#pragma unroll
            for (int h = 0; h < 2; h++)
#pragma unroll
                for (int e = 0; e < 4; e++) *reinterpret_cast<f2 *>(red + ((wq * 2 + y8) * 2 + h) * 128 + box * 32 + sub * 8 + 2 * e) = cs[h][e];
            asm volatile("bar.sync 1, 128;" ::: "memory");
            const int c = tid - 256;
            for (int h = 0; h < halves; h++)
                if (c < (h ? w1 : w0)) {
                    float s = 0.f;
                    for (int i = 0; i < 8; i++) s += red[(i * 2 + h) * 128 + c];
                    g.col_part[(int64_t)slice * g.col_ld + n_first + h * P.nt + c] = s;
                }
        }
    } else {
        regs_inc<CREG_ACC>();
        // ---------------- accumulators ----------------
        const int h = warp >= 16;
        const int wh = h ? w1 : w0, nh = n_first + h * P.nt, wm = (wh + 15) & ~15;
        const uint32_t acc_addr = tmem + h * ACC_COLS + ((uint32_t)wq << 21);
        if (h < halves) {
            f2 acc[ACC_COLS / 2];
#pragma unroll
            for (int i = 0; i < ACC_COLS / 2; i++) acc[i] = 0;
            uint32_t cp = 0;
            for (int64_t rb = rb0; rb < rb1; rb++) {
                if (!warp_wait(cF + 8 * h, cp, &s_abort)) break;
                cp ^= 1;
                fence_after();
#pragma unroll
                for (int c = 0; c < 16; c++) {
                    if (c * 8 < wm) {
                        uint32_t v[8];
                        tmem_ld8(acc_addr + c * 8, v);
#pragma unroll
                        for (int i = 0; i < 4; i++) acc[c * 4 + i] = f2_add(acc[c * 4 + i], f2_pack(v[2 * i], v[2 * i + 1]));
                    }
                }
                fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(cE + 8 * h);
            }
            const int mm = m_first + wq * 32 + lane;
            if (mm < g.m) {
                float *part = g.part + (int64_t)slice * g.m * g.n;
                if (g.transposed) {
#pragma unroll
                    for (int i = 0; i < ACC_COLS / 2; i++)
                        if (2 * i < wh) {
                            const float2 v = f2_get(acc[i]);
                            part[(int64_t)(nh + 2 * i) * g.m + mm] = v.x;
                            part[(int64_t)(nh + 2 * i + 1) * g.m + mm] = v.y;
                        }
                } else {
                    float *po = part + (int64_t)mm * g.n + nh;
                    if (P.sectors) {                               // whole sectors by one store; such a store takes no other address
#pragma unroll
                        for (int i = 0; i < ACC_COLS / 8; i++)
                            if (8 * i < wh)
                                asm volatile("st.global.v4.b64 [%0], {%1, %2, %3, %4};" ::"l"(po + 8 * i), "l"(acc[4 * i]), "l"(acc[4 * i + 1]), "l"(acc[4 * i + 2]),
                                             "l"(acc[4 * i + 3]) : "memory");
                    } else {
#pragma unroll
                        for (int i = 0; i < ACC_COLS / 4; i++)
                            if (4 * i < wh) *reinterpret_cast<ulonglong2 *>(po + 4 * i) = make_ulonglong2(acc[2 * i], acc[2 * i + 1]);
                    }
                }
            }
        }
    }
    fence_before();
    __syncthreads();
    fence_after();
    if (warp == 1) tmem_dealloc(tmem, TMEM_COLS);
    if (tid == 0 && s_abort) atomicOr(&g_step_status, 2);
}

// A group has two accumulators; B of up to 128 columns has one: what bounds the kernel is the splitting of B, a pass per accumulator and row block whatever its
// width.  (Three groups of one accumulator for 384 columns, nine for 1152, lose more on A, split once per group: a layer of d_model 384 2618 -> 2912 us.)
void contract_shape(int m, int n, int &nt, int &halves, int &m_tiles, int &groups) {
    m_tiles = (m + 127) / 128;
    halves = n <= 128 ? 1 : 2;
    groups = (n + 255) / 256;
    nt = ((n + halves * groups - 1) / (halves * groups) + 31) & ~31;      // columns split evenly
    groups = (n + halves * nt - 1) / (halves * nt);
}

}  // namespace

// One block per (feature tile, column group, slice of the rows): as many slices as fill the SMs, none without rows.
int agpt_row_contract_units(int m, int n) {
    int nt, halves, mt, gr;
    contract_shape(m, n, nt, halves, mt, gr);
    return mt * gr;
}
int agpt_row_contract_slices(int64_t rows, int m, int n) {
    const int64_t blocks = (rows + CON_ROWS - 1) / CON_ROWS;
    return (int)std::max<int64_t>(1, std::min<int64_t>(sm_count() / agpt_row_contract_units(m, n), blocks));
}
// The same for contractions that share a launch, `units` blocks per slice in all.  A slice costs a block its start, its last drain and stores, 6 us together, and
// a row of partial sums to add, so few: one round of blocks.  Up to four times as many row blocks (20 of 64 rows at four layers of d_model 128, d_ff 512; 64 at two
// of 64, 256) each is a slice of its own, as in a launch apart: the same sums, bit for bit.
static int one_round_slices(int units) { return std::max(1, sm_count() / units); }
int64_t agpt_row_contract_most_slices_rows(int units) { return 4 * (int64_t)one_round_slices(units) * CON_ROWS; }
int agpt_row_contract_shared_slices(int64_t rows, int units) {
    return (int)(rows <= agpt_row_contract_most_slices_rows(units) ? std::max<int64_t>(1, (rows + CON_ROWS - 1) / CON_ROWS) : one_round_slices(units));
}

static int contract_job(const RowContract &g, ConJob &P) {
    P.g = g;
    contract_shape(g.m, g.n, P.nt, P.halves, P.m_tiles, P.groups);
    P.sectors = (g.n & 7) == 0 && ((uintptr_t)g.part & 31) == 0;      // the caller's workspace may start on any 16-byte boundary
    P.row_blocks = (g.rows + CON_ROWS - 1) / CON_ROWS;
    if (int rc = encode_map(&P.a, g.a, g.rows, g.m, g.lda, CON_ROWS)) return rc;
    for (int i = 0; i < g.n_seg; i++)
        if (int rc = encode_map(&P.b[i], g.b[i], g.rows, g.seg_cols, g.ldb, CON_ROWS)) return rc;
    for (int i = g.n_seg; i < 3; i++) P.b[i] = P.b[0];
    return AGPT_OK;
}

template <int JOBS>
static int launch_contract(const ConBatch<JOBS> &batch, int blocks, cudaStream_t st) {
    static bool done[64];
    if (int rc = allow_smem(contract_kernel<JOBS>, done)) return rc;
    pdl_launch(contract_kernel<JOBS>, blocks, CON_THREADS, CON_SMEM, st, batch);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return agpt_set_error(AGPT_E_CUDA, "row_contract: %s", cudaGetErrorString(e));
    return AGPT_OK;
}

int agpt_row_contract(const RowContract &g, cudaStream_t st) {
    if (g.rows <= 0) return AGPT_OK;
    ConBatch<1> b;
    if (int rc = contract_job(g, b.job[0])) return rc;
    b.n = 1; b.first_block[0] = 0;
    return launch_contract(b, b.job[0].m_tiles * b.job[0].groups * g.slices, st);
}

int agpt_row_contract_many(const RowContract *g, int n, cudaStream_t st) {
    for (int first = 0; first < n; first += CON_JOBS) {
        ConBatch<CON_JOBS> b;
        int blocks = 0;
        b.n = std::min(CON_JOBS, n - first);
        for (int i = 0; i < b.n; i++) {
            if (g[first + i].rows <= 0) return AGPT_OK;          // they share their rows
            if (int rc = contract_job(g[first + i], b.job[i])) return rc;
            b.first_block[i] = blocks;
            blocks += b.job[i].m_tiles * b.job[i].groups * g[first + i].slices;
        }
        if (int rc = launch_contract(b, blocks, st)) return rc;
    }
    return AGPT_OK;
}
