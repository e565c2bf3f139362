// Internal structures shared by the host library and the CUDA kernels.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "../../include/gsofa.h"

namespace gsofa {

// Device-side error word bits (read back by the host after every launch).
enum : int32_t {
    DEV_ERR_COL_RANGE = 1,   // a column id outside [0, n)
    DEV_ERR_ROW_RANGE = 2,   // a row interval outside [0, nnz) or begin > end
    DEV_ERR_QUEUE = 4,       // a traversal queue write past its bound
};

// The status code a device error word stands for: row or column ids out of
// range are the caller's input (GSOFA_ERR_ARG), a queue write past its bound
// is GSOFA_ERR_OVERFLOW; no bit set is GSOFA_OK.
inline int device_status_code(int32_t s) {
    if (s & (DEV_ERR_COL_RANGE | DEV_ERR_ROW_RANGE)) return GSOFA_ERR_ARG;
    if (s & DEV_ERR_QUEUE) return GSOFA_ERR_OVERFLOW;
    return GSOFA_OK;
}

// Counter slots of MatOut::counters.
enum : int {
    CNT_FILLS = 0,
    CNT_EDGES_ALG = 1,
    CNT_VERTS_ALG = 2,
    CNT_EDGES_TRAV = 3,
    CNT_NSUP = 4,
    CNT_NNZ_U = 5,
    CNT_NNZ_L = 6,
    CNT_CHAINED = 7,   // source searches that started from the previous source's closure
    CNT_SLOTS = 8,
};

// One matrix as the traversal sees it: A by rows and A^T by rows, both with
// contiguous rows, plus the per-row outputs.
struct MatDesc {
    int32_t n;
    int32_t flags;              // GSOFA_* bits
    const int32_t* rowptr;      // n+1
    const int32_t* col;
    const int32_t* trowptr;     // n+1 (A^T)
    const int32_t* tcol;
    const int32_t* wdeg;        // ceil(n/32): sum of A's row lengths per 32-vertex word
    const uint32_t* dplanes;    // nplanes * ceil(n/32): degree bit-planes of A's rows
    int32_t nplanes;            // bits of A's largest row length
    int32_t method;             // METHOD_*: which counting traversal takes it
    // 0 when A's pattern equals A^T's (set by the ingest's check): the L
    // column searches in A^T then repeat the U row searches in A, and the
    // direction-0 census writes both halves.  asym[1]: non-zero when a row
    // may hold an id twice
    const int32_t* asym;
    int32_t* nnz_u;             // n: |U row|
    int32_t* nz_row_u;          // n: reference nz_row_U counter
    uint64_t* dig_u;            // n (or null)
    int32_t* nnz_lc;            // n: |L column|
    uint64_t* dig_lc;           // n (or null)
    uint32_t* lmask;            // 4n: L(f+1+j, f) bits
    uint32_t* umask;            // 4n or null: U(f, f+1+j) bits (read by chained starts)
    int8_t* sflags;             // n: supernode flags (batched supernode kernel)
    int32_t* nnz_lr;            // n or null (L row scatter)
    uint64_t* dig_lr;           // n or null
    unsigned long long* counters;  // CNT_SLOTS
    const int64_t* uptr;        // pattern pass: U row pointers (n+1) or null
    int32_t* ucols;
    const int64_t* lptr;        // pattern pass: L column pointers (n+1) or null
    int32_t* lrows;
    // 2n bytes or null: link[2 s + d] is 0 until the direction-d search of
    // source s has finished, then 1 + (s+1 is in its closure): for d = 0 that
    // bit is U(s, s+1), for d = 1 it is L(s+1, s).  The search of source s+1
    // in the other direction reads it (see traverse_kernel: chained starts)
    uint8_t* link;
    long long item_base;        // first work item of this matrix
    // gsofa_chain.cu: the chunks of the largest sources, taken by a launch of
    // larger CTAs, and the first of them there
    long long top_items;
    long long top_base;
    // traverse_kernel: only when this device word is not 0 (null: always).  Set
    // in a batch's launch of what gsofa_hub.cu may leave
    const int32_t* only_if;
    // gsofa_hub.cu: place of the matrix in its arrays (a multiple of 32), the
    // room there (n + 1 rounded up), first work item and items (a power of two)
    long long hub_off;
    long long hub_len;
    long long hub_item;
    long long hub_slots;
    // serving only (zero elsewhere)
    long long n_items;          // work items of this request, for either kernel
    long long walk_items;
    unsigned long long seq;     // request number (claim word tag, done flag value)
    int32_t chunk;              // consecutive sources per work item, for either kernel
    int32_t walk_chunk;
    int32_t slot;               // slot of the serving tables
    int32_t pad1;
};

// The serving kernel's view of the request loop.  Each admitted request
// owns a slot: its descriptor, a claim word (request number << 32 | items
// claimed) and a finished-items counter.  The host publishes a request by
// writing its claim word (request number, 0) with a stream-ordered copy after
// the request's build and descriptor, and lists (slot, request number) in a
// device table it rewrites with small copies.  A CTA picks the listed request
// with the fewest unclaimed items and claims one with compare-and-swap; a
// claim only succeeds while the word still carries the entry's request
// number, so stale or torn list entries are harmless.  The CTA that finishes
// a request's last item writes the request number to done_flags[slot]
// (mapped host memory, the one place the kernel touches host memory).
// Every wait is bounded: a CTA that finds nothing to claim for idle_ns (or
// max_idle_polls polls) exits, which also returns its SM to other work.
enum : int32_t {
    SERVE_CHAIN = 0,  // chain_kernel: requests routed to it
    SERVE_WALK = 1,   // traverse_kernel: the same
    SERVE_ALL = 2,    // traverse_kernel, where it serves alone: any request
};
// A slot's route.  The symmetry word of the request's matrix is copied there
// with its build, so that a symmetric request is the chain's at once; the host
// sends others to traverse_kernel.
enum : int32_t { ROUTE_CHAIN = 0, ROUTE_WALK = -2 };
struct ServeLaunch {
    unsigned long long* claim;            // per slot
    const unsigned long long* list;       // (slot << 32) | request number
    const int32_t* ctrl;                  // [0] exit when idle, [1] take no more items, [2] list entries,
                                          // [3], [4] chain_kernel's, traverse_kernel's launches before this
                                          // number take no more items; [5] chain_kernel's SMs end, [6]
                                          // traverse_kernel's begin and [7] end here
    int32_t kind;                         // SERVE_*: the requests it takes
    const int32_t* route;                 // per slot: ROUTE_*, else nobody claims the request's items
    unsigned int* rr;                     // rotating start of the list scan (tie order)
    const MatDesc* slots;                 // one descriptor per slot
    unsigned long long* items_done;       // per slot: finished items
    const int32_t* slot_status;           // per slot: ingest error word
    unsigned long long* done_flags;       // mapped host memory, per slot
    int32_t nslots;
    long long smem_words;                 // bitmap words that fit in shared memory
    long long max_idle_polls;
    long long idle_ns;
    // per-CTA workspace slots (queue, closure ring, global bitmap): several
    // launches may run at once, so a CTA takes a free slot when it starts
    // (bit set in cta_slots) instead of using its block index, and returns
    // it when it exits; a CTA that finds none exits at once
    unsigned int* cta_slots;
    int32_t n_cta_slots;
    int* alive;                           // CTAs holding a slot
    int32_t launch_no;
    unsigned sm_limit;                    // CTAs on SMs of this number or above leave at once
};

struct TraverseLaunch {
    const MatDesc* mats;        // device array
    int32_t nmats;
    long long total_items;
    unsigned long long* work_counter;  // device, zeroed before launch
    int32_t* queue;             // grid * queue_stride ints
    long long queue_stride;
    uint32_t* gbitmap;          // grid * bitmap_words (global-bitmap variant) or null
    uint32_t* gprev;            // grid * ring * bitmap_words: each CTA's recent closures
    int chunk;                  // consecutive sources per work item
    int merge;                  // 1: reuse the closures of reached cached sources
    int chain;                  // 1: start a source from the previous source's closure when it is known to hold
    long long chain_wait_ns;    // wait this long for the other direction's result when it is one source behind
    int ring;                   // cached closures per CTA (power of 2, <= 64)
    long long sample_stride;    // > 1: process only every stride-th item (autotuner timing)
    long long bitmap_words;     // words per bitmap (covers max n + padding)
    int32_t* status;            // device error word
    int pattern_pass;           // 1: write patterns instead of counting
    int bu_alpha;               // top-down -> bottom-up when frontier*alpha > unseen (0: never)
    int bu_beta;                // bottom-up -> top-down when found*beta < unseen
    int bu_min_src;             // sources below this id stay top-down
    int heavy_len;              // padded rows longer than this are walked by a whole warp
    ServeLaunch serve;          // serving kernel only
};

// The counting traversal (gsofa_chain.cu).  Per CTA: a queue of queue_stride
// ints and gbm_count bitmaps of bitmap_words words in global memory (one that is
// zero between uses; another for the dense base when it does not fit in shared
// memory).
enum : int {
    ITEMS_MAIN = 0,  // the matrices' chunks but the top_items
    ITEMS_TOP = 1,   // those
};
struct ChainLaunch {
    const MatDesc* mats;               // device array
    int32_t nmats;
    long long total_items;             // chunks of all matrices
    unsigned long long* work_counter;  // device, zeroed before launch
    int32_t* queue;
    long long queue_stride;
    uint32_t* gbm;
    int gbm_count;
    long long bitmap_words;            // covers the largest n + padding
    long long smem_words;              // bitmap words that fit in shared memory
    int items;                         // ITEMS_*
    int chunk;                         // consecutive sources per work item
    int list_cap;                      // new ids of a search before the whole CTA takes it
    long long sample_stride;           // > 1: only every stride-th item (autotuner timing)
    int32_t* status;                   // device error word
    ServeLaunch serve;                 // serving kernel only
};
// sizes of a set relative to the current source: ids above it, ids below it,
// the degree sum of those below, the digest of those above
struct Tot {
    int gt, v;
    unsigned long long e, dig;
};

// sources counted and the sum of their digests
struct LRowUse {
    unsigned long long count, dig;
};

// How a matrix's counting traversal runs.
enum : int32_t {
    METHOD_CHAIN = 0,   // gsofa_chain.cu
    METHOD_HUB = 1,     // gsofa_hub.cu
    METHOD_DIRECT = 2,  // gsofa_hub.cu without a hub: every source searched alone
    METHOD_WALK = 3,    // traverse_kernel: repeated entries, whose rows those two do not count
};
// A matrix of at most this many rows is METHOD_DIRECT.
constexpr int kDirectMax = 1024;

// The traversal of gsofa_hub.cu over the launch's matrices of the methods hub
// and direct.  `total` is the sum of their hub_len.
struct HubLaunch {
    const MatDesc* mats;
    int32_t nmats;
    int32_t hub_mats;                  // the matrices with a hub are among the first hub_mats
    int group;                         // consecutive sources per work item
    long long total;
    long long total_items;
    unsigned long long* work_counter;  // [0] extra_kernel, [1] large_kernel
    // zeroed before every launch, in one block: Tot base[2 * hub_bases() * total], stamp,
    // label counts, fallback, judged, large_work, counters, large_count
    void* zeroed;
    LRowUse* l_use;                    // per hub and source (with per-row L statistics): see lrow_kernel
    Tot* base;                         // per base, direction and source: the hub set's totals
    int32_t* stamp;                    // as lam
    int32_t* lcnt;                     // 8 per label job
    int32_t* fallback;                 // per matrix: left to traverse_kernel
    int32_t* given_up;                 // per matrix: bit h when hub h has been given up
    int32_t* judged;                   // per matrix: searches done, searches too large
    unsigned long long* large_work;    // per matrix: large searches done, entries they read
    unsigned long long* counters;      // per matrix, CNT_SLOTS
    int* large_count;
    int32_t* lam;                      // labels: hubs x 2 directions x total
    int32_t* lq;                       // label queues: twice lam
    unsigned long long* hubs;          // per matrix and hub (zeroed too)
    unsigned long long* large;         // (matrix, direction, source) of large searches
    int32_t* queue;                    // large_kernel: per CTA queue_stride ints
    long long queue_stride;
    uint32_t* gbm;                     // large_kernel: per CTA bitmap_words (not with large_smem)
    long long bitmap_words;
    int large_smem;                    // its bitmaps are in shared memory
    int32_t* status;
};
struct HubCfg {
    bool any_hub = false;
    int cluster = 0;          // CTAs per label job, labels in shared memory (0: in global memory)
    int32_t n_max = 0;
    int sm_count = 0;
    size_t zeroed_bytes = 0;
    void* scan_tmp = nullptr;
    size_t scan_bytes = 0;
    int large_grid = 0;
    int extra_grid = 0;       // CTAs of the warps' searches at most
    size_t large_smem = 0;
    bool l_rows = false;      // per-row L statistics are wanted
};
int hub_count();  // hubs per matrix
int hub_bases();  // arrays of totals per direction
size_t label_smem_bytes(int32_t n, int cluster);
size_t hub_scan_bytes(long long tots, long long uses);
int large_occupancy(size_t smem);
int label_max_cluster(size_t smem);
// Loads every kernel of launch_hub, with hub_load_bytes() of device memory for a
// scan of nothing.
size_t hub_load_bytes();
cudaError_t hub_load(void* scratch, cudaStream_t stream);
int extra_ctas_per_sm();
cudaError_t launch_hub(const HubLaunch& L, const HubCfg& c, int digests, cudaStream_t stream);

// Shared memory of a CTA besides its bitmaps; the largest list_cap.
size_t chain_sparse_bytes();
int chain_list_cap();
// Resident CTAs per SM with `smem` dynamic bytes (0 = cannot run).
int chain_occupancy(int block, bool serve, size_t smem);
cudaError_t launch_chain(const ChainLaunch& L, int block, bool serve, int grid, size_t smem,
                         cudaStream_t stream);

// Launch helpers (gsofa_kernels.cu).  All asynchronous on `stream`.
int traverse_block_sizes(int* sizes, int max_sizes);
// Returns the resident CTAs per SM for the given configuration (0 = cannot run).
int traverse_occupancy(int block, bool smem_bitmap, size_t smem_bytes);
cudaError_t launch_traverse(const TraverseLaunch& L, int block, int grid, bool smem_bitmap,
                            size_t smem_bytes, cudaStream_t stream);
// The serving kernel: bitmaps of up to L.serve.smem_words words in shared
// memory (smem_bytes), wider ones in L.gbitmap.
int serve_occupancy(int block, size_t smem_bytes);
cudaError_t launch_serve(const TraverseLaunch& L, int block, int grid, size_t smem_bytes,
                         cudaStream_t stream);

// Builds the padded CSR of A (row pointers rp precomputed on the host, with
// pad counts in their low 2 bits) and of A^T.
cudaError_t launch_canonicalize(int32_t n, long long nnz_in, const int32_t* beg,
                                const int32_t* col_in, const int32_t* rp, int32_t* col_out,
                                int32_t* tcount, int32_t* tpad, int32_t* trp, int32_t* tcol,
                                int32_t* tfill, int32_t* wdeg, uint32_t* dplanes, int nplanes,
                                int32_t* asym, int check_symmetry, int check_dup, void* scan_tmp,
                                size_t scan_tmp_bytes, int32_t* status, cudaStream_t stream);
size_t canonicalize_scan_bytes(int32_t n);
// *sum (zeroed by the caller) += sum over A's entries (v, c) of |v - c|.
cudaError_t launch_index_distance(int32_t n, const int32_t* rp, const int32_t* col,
                                  unsigned long long* sum, cudaStream_t stream);
cudaError_t load_supernodes();
cudaError_t launch_supernodes(int32_t n, int32_t mss, const int32_t* nz_row_u,
                              const uint32_t* lmask, int8_t* flags,
                              unsigned long long* counters, cudaStream_t stream);
cudaError_t launch_batch_reset(const MatDesc* mats, int nmats, cudaStream_t stream);
cudaError_t launch_supernodes_batch(const MatDesc* mats, int nmats, int32_t mss,
                                    const long long* seg_base, long long total_segments,
                                    cudaStream_t stream);
long long supernode_segment_count(int32_t n, int32_t mss);
cudaError_t launch_pattern_ptrs(int32_t n, const int32_t* nnz_u, const int32_t* nnz_lc,
                                int64_t* uptr, int64_t* lptr, void* scan_tmp,
                                size_t scan_tmp_bytes, cudaStream_t stream);
size_t pattern_scan_bytes(int32_t n);

// Device-resident view of a loaded matrix (gsofa_capi.cpp), for entry points
// that live in other translation units.
struct MatrixView {
    int device;
    int32_t n;
    const int32_t* rowptr;
    const int32_t* col;
    const int32_t* trowptr;
    const int32_t* tcol;
    const int32_t* wdeg;
    const uint32_t* dplanes;
    int32_t nplanes;
    const int32_t* asym;
};
bool matrix_view(const void* mat, MatrixView* out);

}  // namespace gsofa
