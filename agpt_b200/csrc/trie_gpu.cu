// Suffix order of a token corpus on the GPU, for the radix-trie builder (trie_suffix.cpp).
//
// Start positions 0..n-2 are ordered by their first key_len tokens (a position past the end of the corpus orders
// before every token) with a least-significant-digit radix sort: one stable pass per token of the key, from the last
// token to the first.  Each pass is HBM-bound integer work: a gather of one token per suffix (the digit), then one
// 8- or 16-bit radix pass over (digit, position) pairs (cub::DeviceRadixSort, whose passes are stable).  Afterwards
// one thread per neighbouring pair counts the common leading tokens.  For the depth-32 trie of a 5M-token corpus
// this replaces about 80 s of bucket refinement on one host thread by a few milliseconds of device time; the
// linear-time assembly of the trie from the order stays on the host.
#include <cuda_runtime.h>

#include <cub/device/device_radix_sort.cuh>

#include <cstdint>

#include "../../include/agpt_b200.h"
#include "internal.h"

namespace {

#define CUDA_TRY(x)                                                                              \
    do {                                                                                         \
        cudaError_t e_ = (x);                                                                    \
        if (e_ != cudaSuccess) { rc = agpt_set_error(AGPT_E_CUDA, "%s: %s", #x, cudaGetErrorString(e_)); goto done; } \
    } while (0)

// digit of count tokens, the first in the highest bits
template <typename DT>
__global__ void __launch_bounds__(256) digit_kernel(const int32_t *__restrict__ corpus, const int32_t *__restrict__ sa, int64_t n, int32_t m,
                                                     int d, int count, int bits, DT *__restrict__ digit) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t p = (int64_t)sa[i] + d;
        DT v = 0;
        for (int k = 0; k < count; k++) v = (DT)(v << (k ? bits : 0)) | (p + k < n ? (DT)(corpus[p + k] + 1) : (DT)0);
        digit[i] = v;
    }
}

__global__ void __launch_bounds__(256) iota_kernel(int32_t *__restrict__ sa, int32_t m) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x) sa[i] = (int32_t)i;
}

// lcp[i] = number of equal leading tokens of the keys of sa[i-1] and sa[i] (tokens past the corpus end match nothing)
__global__ void __launch_bounds__(256) lcp_kernel(const int32_t *__restrict__ corpus, const int32_t *__restrict__ sa, int64_t n, int32_t m,
                                                   int key_len, int32_t *__restrict__ lcp) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x) {
        if (i == 0) { lcp[0] = 0; continue; }
        const int64_t a = sa[i - 1], b = sa[i];
        int64_t lim = n - (a > b ? a : b);
        if (lim > key_len) lim = key_len;
        int l = 0;
        while (l < lim && corpus[a + l] == corpus[b + l]) l++;
        lcp[i] = l;
    }
}

int64_t up256(int64_t x) { return (x + 255) & ~(int64_t)255; }

// One piece of device memory holds everything: corpus, two position arrays, common prefixes, two digit arrays, cub's scratch.  The
// caller's if it brings some (cudaMalloc and cudaFree of it take one to five ms between them once a program holds other memory, the sort of
// 60,000 tokens half of one), else allocated here.
template <typename DT>
int64_t suffix_workspace(int64_t n, int end_bit) {
    const int32_t m = (int32_t)(n - 1);
    size_t tmp = 0;
    if (cub::DeviceRadixSort::SortPairs(nullptr, tmp, (DT *)nullptr, (DT *)nullptr, (int32_t *)nullptr, (int32_t *)nullptr, m, 0, end_bit) != cudaSuccess) return -1;
    return up256(n * 4) + 3 * up256((int64_t)m * 4) + 2 * up256((int64_t)m * sizeof(DT)) + (int64_t)tmp + 256;
}
// Digits of 64 bits hold nine tokens of 65 symbols and save passes, for 8 bytes a position instead of 1 or 2 in both digit arrays and in the sort's own.
// They are the faster ones on both sides of this line (device ms at 33 tokens a key, wide / narrow: 20,000 positions 0.46 / 0.94, 60,000 0.48 / 0.99,
// 1M 0.84 / 1.32, 4M 2.1 / 2.9, 10M 4.7 / 5.7); it bounds the memory, at a size where a millisecond no longer shows beside the host's assembly.
constexpr int64_t WIDE_DIGITS_BELOW = 4 << 20;
template <typename DT>
int sort_suffixes(const int32_t *corpus, int64_t n, int32_t m, int key_len, int bits, int per_digit, cudaStream_t st, cudaEvent_t e0, cudaEvent_t e1,
                  uint8_t *ws, int64_t ws_bytes, int32_t *sa_out, int32_t *lcp_out) {
    int rc = AGPT_OK;
    uint8_t *arena = ws;
    size_t tmp_bytes = 0;
    const int64_t am = up256((int64_t)m * 4), ad = up256((int64_t)m * sizeof(DT)), an = up256(n * 4);
    const unsigned grid = (unsigned)(((int64_t)m + 255) / 256 < 148 * 16 ? ((int64_t)m + 255) / 256 : 148 * 16);
    int32_t *d_corpus, *in, *outp, *d_lcp;
    DT *dig0, *dig1;
    void *tmp;
    CUDA_TRY(cub::DeviceRadixSort::SortPairs(nullptr, tmp_bytes, (DT *)nullptr, (DT *)nullptr, (int32_t *)nullptr, (int32_t *)nullptr, m, 0,
                                             bits * per_digit, st));
    if (!ws) CUDA_TRY(cudaMalloc(&arena, (size_t)(an + 3 * am + 2 * ad) + tmp_bytes + 16));
    else if (ws_bytes < an + 3 * am + 2 * ad + (int64_t)tmp_bytes) { rc = agpt_set_error(AGPT_E_ARG, "suffix order: workspace of %lld bytes is too small", (long long)ws_bytes); goto done; }
    d_corpus = (int32_t *)arena; in = (int32_t *)(arena + an); outp = (int32_t *)(arena + an + am); d_lcp = (int32_t *)(arena + an + 2 * am);
    dig0 = (DT *)(arena + an + 3 * am); dig1 = (DT *)(arena + an + 3 * am + ad); tmp = arena + an + 3 * am + 2 * ad;
    CUDA_TRY(cudaMemcpyAsync(d_corpus, corpus, (size_t)n * 4, cudaMemcpyHostToDevice, st));
    if (e0) CUDA_TRY(cudaEventRecord(e0, st));
    iota_kernel<<<grid, 256, 0, st>>>(in, m);
    for (int end = key_len; end > 0; end -= per_digit) {
        const int first = end > per_digit ? end - per_digit : 0, count = end - first;
        digit_kernel<DT><<<grid, 256, 0, st>>>(d_corpus, in, n, m, first, count, bits, dig0);
        CUDA_TRY(cub::DeviceRadixSort::SortPairs(tmp, tmp_bytes, dig0, dig1, in, outp, m, 0, bits * count, st));
        int32_t *t = in; in = outp; outp = t;
    }
    lcp_kernel<<<grid, 256, 0, st>>>(d_corpus, in, n, m, key_len, d_lcp);
    CUDA_TRY(cudaGetLastError());
    if (e1) CUDA_TRY(cudaEventRecord(e1, st));
    CUDA_TRY(cudaMemcpyAsync(sa_out, in, (size_t)m * 4, cudaMemcpyDeviceToHost, st));
    CUDA_TRY(cudaMemcpyAsync(lcp_out, d_lcp, (size_t)m * 4, cudaMemcpyDeviceToHost, st));
    CUDA_TRY(cudaStreamSynchronize(st));
done:
    if (!ws) cudaFree(arena);
    return rc;
}

// ws null: own memory and stream
int suffix_order(const int32_t *corpus, int64_t n, int key_len, int device, uint8_t *ws, int64_t ws_bytes, cudaStream_t user, int32_t *sa_out,
                 int32_t *lcp_out, float *device_ms_out) {
    if (!corpus || !sa_out || !lcp_out || n < 2 || key_len < 1) return agpt_set_error(AGPT_E_ARG, "suffix_order_gpu: bad argument");
    if (n >= (1LL << 31)) return agpt_set_error(AGPT_E_LIMIT, "suffix_order_gpu: corpus beyond 2^31 tokens");
    int vocab = 0;
    for (int64_t i = 0; i < n; i++) {
        if (corpus[i] < 0) return agpt_set_error(AGPT_E_ARG, "suffix_order_gpu: negative token");
        if (corpus[i] >= vocab) vocab = corpus[i] + 1;
    }
    if (vocab > 65534) return agpt_set_error(AGPT_E_LIMIT, "suffix_order_gpu: vocabulary beyond 65534");
    int rc = AGPT_OK;
    const int32_t m = (int32_t)(n - 1);
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    cudaStream_t st = user;
    int bits = 1;
    while ((1 << bits) < vocab + 1) bits++;
    CUDA_TRY(cudaSetDevice(device));
    if (!ws) CUDA_TRY(cudaStreamCreate(&st));
    if (device_ms_out) {
        CUDA_TRY(cudaEventCreate(&e0));
        CUDA_TRY(cudaEventCreate(&e1));
    }
    // Below a few million positions a pass is launch latency, so as many tokens as fit 64 bits go into one digit (33 tokens
    // of 7 bits: 44 launches instead of 165); above, one token per pass moves the fewest bytes.
    if (m < WIDE_DIGITS_BELOW) rc = sort_suffixes<uint64_t>(corpus, n, m, key_len, bits, 64 / bits, st, e0, e1, ws, ws_bytes, sa_out, lcp_out);
    else if (vocab + 1 <= 256) rc = sort_suffixes<uint8_t>(corpus, n, m, key_len, bits, 1, st, e0, e1, ws, ws_bytes, sa_out, lcp_out);
    else rc = sort_suffixes<uint16_t>(corpus, n, m, key_len, bits, 1, st, e0, e1, ws, ws_bytes, sa_out, lcp_out);
    if (rc) goto done;
    if (device_ms_out) CUDA_TRY(cudaEventElapsedTime(device_ms_out, e0, e1));
done:
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    if (!ws && st) cudaStreamDestroy(st);
    return rc;
}

int build(const int32_t *corpus, int64_t n, int max_depth, int subtree_level, int prune_min_mass, int prune_min_depth, int device, uint8_t *ws,
          int64_t ws_bytes, cudaStream_t st, agpt_trie **out) {
    if (!corpus || !out || max_depth < 1) return agpt_set_error(AGPT_E_ARG, "trie_build_gpu: bad argument");
    if (n < (int64_t)max_depth + 2) return agpt_set_error(AGPT_E_ARG, "trie_build_gpu: corpus shorter than max_depth + 2 tokens");
    std::vector<int32_t> sa((size_t)(n - 1)), lcp((size_t)(n - 1));
    if (int rc = suffix_order(corpus, n, max_depth + 1, device, ws, ws_bytes, st, sa.data(), lcp.data(), nullptr)) return rc;
    return agpt_b200_trie_from_suffix_order(corpus, n, max_depth, subtree_level, prune_min_mass, prune_min_depth, sa.data(), lcp.data(), out);
}

}  // namespace

extern "C" int agpt_b200_suffix_order_gpu(const int32_t *corpus, int64_t n, int key_len, int device, int32_t *sa_out, int32_t *lcp_out,
                                          float *device_ms_out) try {
    return suffix_order(corpus, n, key_len, device, nullptr, 0, nullptr, sa_out, lcp_out, device_ms_out);
} AGPT_CATCH("suffix_order_gpu")

extern "C" int64_t agpt_b200_trie_build_workspace_bytes(int64_t n) {
    if (n < 2 || n >= (1LL << 31)) return -1;
    return n - 1 < WIDE_DIGITS_BELOW ? suffix_workspace<uint64_t>(n, 64) : std::max(suffix_workspace<uint8_t>(n, 8), suffix_workspace<uint16_t>(n, 16));
}

extern "C" int agpt_b200_trie_build_gpu(const int32_t *corpus, int64_t n, int max_depth, int subtree_level, int prune_min_mass,
                                        int prune_min_depth, int device, agpt_trie **out) try {
    return build(corpus, n, max_depth, subtree_level, prune_min_mass, prune_min_depth, device, nullptr, 0, nullptr, out);
} AGPT_CATCH("trie_build_gpu")

extern "C" int agpt_b200_trie_build_gpu_ws(const int32_t *corpus, int64_t n, int max_depth, int subtree_level, int prune_min_mass, int prune_min_depth,
                                           int device, void *d_workspace, int64_t workspace_bytes, void *stream, agpt_trie **out) try {
    if (!d_workspace) return agpt_set_error(AGPT_E_ARG, "trie_build_gpu_ws: null workspace");
    return build(corpus, n, max_depth, subtree_level, prune_min_mass, prune_min_depth, device, (uint8_t *)d_workspace, workspace_bytes, (cudaStream_t)stream, out);
} AGPT_CATCH("trie_build_gpu_ws")
