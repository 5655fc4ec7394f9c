// Shared between the host walker code and the CUDA translation unit of libagpt_b200.
#pragma once
#include <atomic>
#include <cstdint>
#include <cstdlib>
#include <exception>
#include <mutex>
#include <new>
#include <vector>

#include <sys/mman.h>

#define AGPT_REDUCE_SEG 16    // tiles summed by one warp of the dK/dV reduction before a second pass (at most 32: one offset per lane)

int agpt_set_error(int code, const char *fmt, ...);
// Behind the body of an extern "C" function that allocates (extern "C" int f() try { .. } AGPT_CATCH("f")): no exception crosses the boundary.
#define AGPT_CATCH(who)                                                                                        \
    catch (const std::bad_alloc &) { return agpt_set_error(AGPT_E_NOMEM, who ": out of host memory"); }        \
    catch (const std::exception &e) { return agpt_set_error(AGPT_E_NOMEM, who ": %s", e.what()); }

// Host memory for arrays of megabytes that one call makes and fills once.  Their first touch in 4 KB pages costs more than the
// fill (0.5 us a page: 2 ms for the 1.7M edge characters of 60,000 tokens at depth 32, and zeroing them first as much again), so
// from 1 MB on they lie in huge pages where the system has them, and elements that are not given a value are left as they come.
constexpr size_t AGPT_HUGE_PAGE = (size_t)2 << 20, AGPT_HUGE_FROM = (size_t)1 << 20;
inline void *agpt_big_alloc(size_t bytes) {
    if (bytes < AGPT_HUGE_FROM) return malloc(bytes ? bytes : 1);
    const size_t whole = (bytes + AGPT_HUGE_PAGE - 1) / AGPT_HUGE_PAGE * AGPT_HUGE_PAGE;
    void *p = aligned_alloc(AGPT_HUGE_PAGE, whole);
    if (p) madvise(p, whole, MADV_HUGEPAGE);     // a hint: without huge pages the memory is as good
    return p;
}
struct agpt_big_free { void operator()(void *p) const { free(p); } };
template <typename T>
struct agpt_big_allocator {
    using value_type = T;
    agpt_big_allocator() = default;
    template <typename U> agpt_big_allocator(const agpt_big_allocator<U> &) {}
    T *allocate(size_t n) {
        void *p = n > SIZE_MAX / sizeof(T) - AGPT_HUGE_PAGE ? nullptr : agpt_big_alloc(n * sizeof(T));
        if (!p) throw std::bad_alloc();
        return (T *)p;
    }
    void deallocate(T *p, size_t) { free(p); }
    template <typename U> void construct(U *p) { ::new ((void *)p) U; }       // resize() leaves new elements unset
    template <typename U, typename V> void construct(U *p, V &&v) { ::new ((void *)p) U((V &&)v); }
    template <typename U> bool operator==(const agpt_big_allocator<U> &) const { return true; }
    template <typename U> bool operator!=(const agpt_big_allocator<U> &) const { return false; }
};
template <typename T> using agpt_big_vector = std::vector<T, agpt_big_allocator<T>>;

// Radix trie with the reference's node numbering (ids in the builder's breadth-first emission order), counts, edge
// mass and char positions.
struct agpt_trie {
    int32_t radix_count = 0, n_depth_files = 0;
    int64_t total_edge_chars = 0, leveled_nodes = 0;
    std::vector<int32_t> parent, first_char_depth, edge_len, edge_mass, endpoint_depth, subtree_key, edge_start;
    std::vector<int64_t> edge_off, cnt_off;
    agpt_big_vector<int32_t> edge_tok, cnt_tok, cnt_val;
    void finish_char_positions() {
        // char positions follow depth-file order (src/cuda/agpt_train.cu:813-846)
        edge_start.assign(radix_count, 0);
        std::vector<int64_t> per_depth(n_depth_files + 1, 0);
        for (int32_t r = 1; r < radix_count; r++) per_depth[endpoint_depth[r] + 1] += edge_len[r];
        for (int d = 0; d < n_depth_files; d++) per_depth[d + 1] += per_depth[d];
        for (int32_t r = 1; r < radix_count; r++) {
            edge_start[r] = (int32_t)per_depth[endpoint_depth[r]];
            per_depth[endpoint_depth[r]] += edge_len[r];
        }
    }
};

// Walker plan: a tree laid out in depth-first pre-order.  Position i's subtree is the
// interval [i, sub_end[i]); a is an ancestor-or-self of i iff a <= i < sub_end[a].  Queries
// are processed in tiles of up to tile_m consecutive positions (tile t: [tile_start[t], tile_start[t + 1])); a tile's keys are
// the ancestor chain of its first position (chain_ids, root side first, chain_off per tile) plus the tile's own rows.
//
// A plan for a GPU with tiles of 64 lets a tile end early, where the next one starts at a shallow position: the chain that the
// next tile loads again, and gives partial dK/dV rows for, is as long as its first position is deep, and a trie's depth-first
// order comes back to shallow rows all the time.  The next start is the row k in [32, 64] after this one that makes
// depth + 0.9 (64 - k) least, the later one of equals: a chain row costs about as much as a row left unfilled.  The factor
// stays below 1, because at 1 a run without branches, one deeper per row, leaves every end on it of one cost, the latest is taken and
// next to nothing is cut: the 1.4M-row trie then takes 952 + 2152 us (forward, backward with reduction), at 0.95 907 + 1772.  From 0.5 to 0.95
// times agree to 1 %, though the starts are not the same everywhere (on the 66k-row trie 1,066 tiles at 0.5, 1,061 from 0.75 on); smaller
// factors leave more tiles for little, on bushy trees most (random tree of 600k nodes, 8 x 64: 1635 + 3350 us at 0.25, 1805 + 3644 at 0, 1591 +
// 3303 at 0.9).  (Tiles below 32 rows leave warps without rows.)  Keys per row on the depth-32 trie
// of 1.4M rows 1.27 -> 1.07, partial rows 0.27 -> 0.07 per row and their reduction 274 -> 81 us; forward 945 -> 901 us.
struct agpt_plan {
    int64_t n = 0;
    int32_t tile_m = 64;
    int64_t n_tiles = 0;
    std::vector<int32_t> tile_start;             // [n_tiles + 1]
    int32_t max_keys = 0;                        // chain + rows of the tile that has most
    // An even plan keeps what a sampled training step on a bfloat16 store rounds: its tiles end after tile_m rows, both directions take the
    // chunked kernels (Q, P and dS to 11 bits on both sides of lse; which value P is rounded at depends on the tile's keys in
    // chunks of 32), and a node's partial dK/dV rows are one reduction item.
    bool even = false;
    int32_t max_depth = 0;
    int64_t sum_depth = 0, sum_group_prefix = 0, n_groups = 0, n_reduce_nodes = 0, n_multi_items = 0;
    std::vector<int32_t> dfs_to_node, node_to_dfs, parent_dfs, depth, sub_end;      // filled on demand if lazy: need_host()
    std::vector<int64_t> chain_off;
    int64_t chain_rows = 0;                      // chain_off[n_tiles]
    std::vector<int32_t> chain_ids, chain_end;   // chain_end[j] = sub_end[chain_ids[j]]
    // dK/dV reduction work list: item = (node, inclusive tile range); slot >= 0 when the node's range
    // is cut into several items whose sums meet in a second pass
    std::vector<int32_t> item_node, item_t0, item_t1, item_slot;
    std::vector<int32_t> multi_node, multi_count;
    std::vector<int64_t> multi_first;          // first segment slot of each multi-segment node (its slots are consecutive)
    // a plan made from runs of rows (groups.cu): row arrays are derived from these when the host asks for them
    std::atomic<bool> lazy{false};
    std::vector<int32_t> run_qoff, run_parent, run_depth, run_end;
    std::mutex host_lock;
    void need_host();
    // device copies (owned, or in a buffer of the caller)
    int device = -1;
    bool external = false;
    int32_t *d_depth = nullptr, *d_sub_end = nullptr, *d_chain_ids = nullptr, *d_chain_end = nullptr, *d_tile_start = nullptr;
    int64_t *d_chain_off = nullptr, *d_multi_first = nullptr;
    int32_t *d_item_node = nullptr, *d_item_t0 = nullptr, *d_item_t1 = nullptr, *d_item_slot = nullptr;
    int32_t *d_multi_node = nullptr, *d_multi_count = nullptr;
    // host-buffer step (agpt_b200_attn_fwd_bwd_host): device arena, three streams (upload, compute, download) and
    // per-chunk events; created at first use, kept for later calls, released with the plan
    void *host_arena = nullptr;
    size_t host_arena_bytes = 0;
    void *host_streams[3] = {nullptr, nullptr, nullptr};
    std::vector<void *> host_events;
    void *host_fix = nullptr;                  // pinned staging for rows re-downloaded at the end of a host-buffer step
    size_t host_fix_bytes = 0;
    ~agpt_plan();
};

int agpt_plan_upload(agpt_plan *p, int device);
// Rows of a tile whose first branch (row from 32 on that is not a child of the row before it) lies L > 64 rows away: a chain without branches, as in
// pruned tries with long repeats.  No end before the branch is shallow, so the chain is cut into as few tiles as hold it, whole ones last, and the last
// ends at the branch.  (By cost alone the first end in reach would be taken: tiles of 33 rows.)  On the pruned trie of 719k rows of depth 128: 17,251 -> 11,855
// tiles, chain rows 571k -> 369k, longest tile 141 -> 128 keys; 6 x 64, bfloat16 store, forward 1438 -> 1113 us, backward with reduction 4742 -> 3843; 318k such
// rows, float32 store, 1639 -> 1285 and 5084 -> 2733 (they fit the whole-tile kernels now).  Tries of depth 32 have no such chain.
inline int64_t agpt_tile_of_chain(int64_t L) { const int64_t k = (L - 1) % 64 + 1; return k < 32 ? 32 : k; }
// cost of a tile that starts k rows after the last one's start, at depth d (in tenths of a row)
inline int64_t agpt_tile_cost(int32_t d, int64_t k) { return 10 * (int64_t)d + 9 * (64 - k); }
// mass weight of each loss node (agpt_b200_mass_weights without the expansion to queries)
int agpt_mass_weights_per_node(const int32_t *edge_mass, const int32_t *edge_len, const int32_t *unit_of_node, const uint8_t *counted,
                               int64_t n_nodes, int64_t n_units, int mode, float *out_per_node);
int agpt_step_gemm_status(int *out);       // status word of step_gemm.cu's kernels
int agpt_step_gemm_status_word(const int **d_word);      // and its place on the current device

// tcgen05 float32 GEMM (gemm_sm100.cu): D[l] = act(alpha * op(A[l]) * op(B[l]) + beta * C + bias row), l < L batches
bool agpt_gemm_sm100_takes(int trans_a, int trans_b, int relu, int has_source);
int agpt_gemm_sm100(int trans_a, int trans_b, int M, int N, int K, int L, float alpha, const float *A, int64_t lda, int64_t batch_a,
                    const float *B, int64_t ldb, int64_t batch_b, const float *bias, int relu, float beta, const float *C, int64_t ldc,
                    float *D, int64_t ldd, int64_t batch_d, void *stream);
