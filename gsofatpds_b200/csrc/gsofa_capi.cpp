// gsofa_capi.cpp -- host side of libgsofa.so: the C-ABI declared in
// include/gsofa.h.  Owns device memory (a dedicated stream-ordered pool with
// budget accounting), device-resident matrices and results, the launch
// configuration of the traversal kernel, and the reference-shaped entry point.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <map>
#include <cerrno>
#include <climits>
#include <chrono>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <memory>
#include <mutex>
#include <new>
#include <string>
#include <vector>

#include "gsofa_host.h"

using namespace gsofa;
using namespace gsofa::host;

// ---------------------------------------------------------------------------
namespace gsofa {
namespace host {

int set_err(gsofa_ctx* ctx, int status, const char* fmt, ...) {
    if (ctx) {
        char buf[512];
        va_list ap;
        va_start(ap, fmt);
        vsnprintf(buf, sizeof(buf), fmt, ap);
        va_end(ap);
        ctx->err = buf;
    }
    return status;
}

int cuda_fail(gsofa_ctx* ctx, cudaError_t e, const char* where) {
    return set_err(ctx, GSOFA_ERR_CUDA, "%s: %s", where, cudaGetErrorString(e));
}

#define CK(call)                                          \
    do {                                                  \
        cudaError_t e_ = (call);                          \
        if (e_ != cudaSuccess) return cuda_fail(ctx, e_, #call); \
    } while (0)

void dev_free_on(gsofa_ctx* ctx, void* p, size_t bytes, cudaStream_t stream) {
    if (!p) return;
    bytes = (bytes + 255) & ~(size_t)255;
    cudaFreeAsync(p, stream);
    ctx->used -= std::min(ctx->used, bytes);
}

size_t kept_workspace(const gsofa_ctx* ctx) {
    return ctx->hub_ws_bytes + ctx->queue_bytes + ctx->gbitmap_bytes + ctx->gprev_bytes;
}

// Gives back the workspace that factorizations keep between calls.
void drop_workspace(gsofa_ctx* ctx) {
    struct {
        void** p;
        size_t* bytes;
    } const kept[] = {{&ctx->hub_ws, &ctx->hub_ws_bytes},
                      {&ctx->queue, &ctx->queue_bytes},
                      {&ctx->gbitmap, &ctx->gbitmap_bytes},
                      {&ctx->gprev, &ctx->gprev_bytes}};
    for (const auto& k : kept) {
        dev_free_on(ctx, *k.p, *k.bytes, ctx->stream);
        *k.p = nullptr;
        *k.bytes = 0;
    }
}

int dev_alloc_on(gsofa_ctx* ctx, size_t bytes, void** p, cudaStream_t stream) {
    *p = nullptr;
    if (bytes == 0) return GSOFA_OK;
    bytes = (bytes + 255) & ~(size_t)255;
    // a factorization's kept workspace gives way to what a caller asks for
    if (ctx->used + bytes > ctx->budget && !ctx->factoring) drop_workspace(ctx);
    if (ctx->used + bytes > ctx->budget)
        return set_err(ctx, GSOFA_ERR_OOM_BUDGET,
                       "allocation of %zu bytes exceeds the budget (%zu of %zu bytes in use)",
                       bytes, ctx->used, ctx->budget);
    cudaError_t e = cudaMallocFromPoolAsync(p, bytes, ctx->pool, stream);
    if (e != cudaSuccess) {
        *p = nullptr;
        return cuda_fail(ctx, e, "cudaMallocFromPoolAsync");
    }
    ctx->used += bytes;
    return GSOFA_OK;
}

int dev_alloc(gsofa_ctx* ctx, size_t bytes, void** p) {
    return dev_alloc_on(ctx, bytes, p, ctx->stream);
}

void dev_free(gsofa_ctx* ctx, void* p, size_t bytes) { dev_free_on(ctx, p, bytes, ctx->stream); }

// Grow-only workspace buffer.
int ensure(gsofa_ctx* ctx, void** p, size_t* have, size_t need) {
    if (*have >= need) return GSOFA_OK;
    dev_free(ctx, *p, *have);
    *p = nullptr;
    *have = 0;
    int rc = dev_alloc(ctx, need, p);
    if (rc) return rc;
    *have = (need + 255) & ~(size_t)255;
    return GSOFA_OK;
}

// Pinned words for the totals and flags of `count` matrices.
int ensure_pinned(gsofa_ctx* ctx, size_t count) {
    if (ctx->h_counters_cap >= count) return GSOFA_OK;
    if (ctx->h_counters) cudaFreeHost(ctx->h_counters);
    if (ctx->h_fallback) cudaFreeHost(ctx->h_fallback);
    ctx->h_counters = nullptr;
    ctx->h_fallback = nullptr;
    ctx->h_counters_cap = 0;
    cudaError_t e = cudaMallocHost((void**)&ctx->h_counters, 8 * CNT_SLOTS * count);
    if (e == cudaSuccess) e = cudaMallocHost((void**)&ctx->h_fallback, 4 * count);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "pinned totals");
    ctx->h_counters_cap = count;
    return GSOFA_OK;
}

size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

long long bitmap_words(int32_t n) { return (((long long)n + 31) >> 5) + 6; }

// Default chunk (consecutive sources per work item): total / grid, a power
// of 2 between 16 and 512 sources, where total weighs each matrix by
// chunk_weight -- about one item per CTA for unsymmetric patterns.  Each
// chunk's first source starts cold (nothing to reuse), while later ones
// mostly start from their predecessor's closure, so long chunks pay; the
// autotuner tries shorter and longer ones.
long long default_chunk(long long total_sources, int grid) {
    long long c = total_sources / (grid > 0 ? grid : 1);
    long long p = 16;
    while (p * 2 <= c && p < 512) p *= 2;
    return p;
}

// Launch order of a batch's matrices: most entries first (longest processing
// time first), so that the persistent kernel's last items are small ones and
// no large matrix starts when the rest of the batch is almost done.
std::vector<int32_t> batch_order(const gsofa_matrix* const* mats, int32_t count) {
    std::vector<int32_t> order((size_t)count);
    for (int32_t i = 0; i < count; i++) order[(size_t)i] = i;
    std::stable_sort(order.begin(), order.end(),
                     [&](int32_t a, int32_t b) { return mats[a]->nnz > mats[b]->nnz; });
    return order;
}

long long chunk_weight(gsofa_ctx* ctx, const gsofa_matrix* m) {
    if (m->host_sym < 0) {
        int sym = 0, dup = 1;
        if (m->n > 0 &&
            cudaMemcpyAsync(ctx->h_status + 1, m->asym, 8, cudaMemcpyDeviceToHost, ctx->stream) ==
                cudaSuccess &&
            cudaStreamSynchronize(ctx->stream) == cudaSuccess) {
            sym = ctx->h_status[1] == 0;
            dup = ctx->h_status[2] != 0;
        } else {
            cudaGetLastError();
        }
        m->host_sym = sym;
        m->host_dup = dup;
    }
    return m->host_sym ? m->n / 4 : 2ll * m->n;
}

// Default CTA size: about 1024 resident threads per SM (the kernel is held
// to 64 registers), given how many shared-memory bitmaps fit per SM.
// Measured on B200: 256-thread CTAs are fastest whenever 4 fit, else fewer,
// larger CTAs.
int default_block(int32_t nmax, int smem_per_sm) {
    const long long words = (((long long)nmax + 31) >> 5) + 6;
    const long long per_cta = ((words * 4 + 15) & ~15ll) + 8 * 1024;
    long long fit = smem_per_sm / per_cta;
    if (fit >= 4) return 256;
    if (fit >= 2) return 512;
    return 1024;
}

struct LaunchCfg {
    int block = 512;
    int grid = 0;
    bool smem_bitmap = true;
    size_t smem = 0;
    long long words = 0;
};

int plan_launch(gsofa_ctx* ctx, int32_t nmax, const gsofa_opts* o, LaunchCfg* c) {
    c->block = o->threads_per_source > 0 ? o->threads_per_source
                                         : default_block(nmax, ctx->smem_per_sm);
    if (c->block != 128 && c->block != 256 && c->block != 512 && c->block != 1024)
        return set_err(ctx, GSOFA_ERR_ARG, "threads_per_source must be 128, 256, 512 or 1024");
    c->words = bitmap_words(nmax);
    size_t bytes = (size_t)c->words * 4;
    bytes = (bytes + 15) & ~(size_t)15;
    // leave room for the kernel's static shared memory (reduction + scan)
    c->smem_bitmap = bytes + 12 * 1024 <= (size_t)ctx->smem_optin &&
                     !(o->flags & GSOFA_FORCE_GLOBAL_BITMAP);
    c->smem = c->smem_bitmap ? bytes : 0;
    int occ = traverse_occupancy(c->block, c->smem_bitmap, c->smem);
    if (occ <= 0)
        return set_err(ctx, GSOFA_ERR_UNSUPPORTED,
                       "traversal kernel cannot be resident (block %d, %zu B shared)", c->block,
                       c->smem);
    c->grid = occ * ctx->sm_count;
    if (o->sources_in_flight > 0) c->grid = std::min(c->grid, o->sources_in_flight);
    return GSOFA_OK;
}

int check_status(gsofa_ctx* ctx) {
    const int32_t s = *ctx->h_status;
    const int code = device_status_code(s);
    if (code == GSOFA_OK) return GSOFA_OK;
    if (s & DEV_ERR_COL_RANGE) return set_err(ctx, code, "column id outside [0, n)");
    if (s & DEV_ERR_ROW_RANGE) return set_err(ctx, code, "row interval outside [0, nnz)");
    return set_err(ctx, code, "traversal queue bound exceeded");
}

int32_t* work_counter_status(gsofa_ctx* ctx, unsigned long long** wc) {
    *wc = reinterpret_cast<unsigned long long*>(ctx->small);
    return reinterpret_cast<int32_t*>(reinterpret_cast<char*>(ctx->small) + 64);
}

void result_free(gsofa_result* r) {
    if (!r) return;
    if (r->ctx) {
        std::lock_guard<std::recursive_mutex> g(r->ctx->mu);
        dev_free(r->ctx, r->arena, r->bytes);
        dev_free(r->ctx, r->parena, r->pbytes);
        supernodal_free(r);
    }
    delete r;
}

// Layout of a result arena: the per-row arrays of an n-row matrix.
static size_t result_layout(int32_t n, uint32_t flags, size_t off[12]) {
    const size_t N = (size_t)std::max(n, 1);
    const bool dig = flags & GSOFA_DIGESTS;
    const bool lrow = flags & GSOFA_L_ROW_STATS;
    size_t sz[12];
    sz[0] = 4 * N;                       // nnz_u
    sz[1] = 4 * N;                       // nz_row_u
    sz[2] = 4 * N;                       // nnz_lc
    sz[3] = dig ? 8 * N : 0;             // dig_u
    sz[4] = dig ? 8 * N : 0;             // dig_lc
    sz[5] = 16 * N;                      // lmask
    sz[6] = 16 * N;                      // umask (chained starts)
    // zeroed from here on
    sz[7] = lrow ? 4 * N : 0;            // nnz_lr
    sz[8] = lrow ? 8 * N : 0;            // dig_lr
    sz[9] = N;                           // supernode flags
    sz[10] = 8 * CNT_SLOTS;              // counters
    sz[11] = 2 * N;                      // link (chained starts)
    size_t total = 0;
    for (int i = 0; i < 12; i++) {
        off[i] = total;
        total += align256(sz[i]);
    }
    return total;
}

size_t result_bytes(int32_t n, uint32_t flags) {
    size_t off[12];
    return result_layout(n, flags, off);
}

// Carve the per-row result arrays out of one arena.
int result_alloc_on(gsofa_ctx* ctx, int32_t n, uint32_t flags, int32_t mss, cudaStream_t stream,
                    gsofa_result** out) {
    gsofa_result* r = new (std::nothrow) gsofa_result();
    if (!r) return set_err(ctx, GSOFA_ERR_OOM_BUDGET, "host allocation failed");
    r->ctx = ctx;
    r->n = n;
    r->flags = flags;
    r->mss = mss;
    const bool dig = flags & GSOFA_DIGESTS;
    const bool lrow = flags & GSOFA_L_ROW_STATS;
    size_t off[12];
    const size_t total = result_layout(n, flags, off);
    int rc = dev_alloc_on(ctx, total, &r->arena, stream);
    if (rc) {
        delete r;
        return rc;
    }
    r->bytes = total;
    char* b = reinterpret_cast<char*>(r->arena);
    r->nnz_u = reinterpret_cast<int32_t*>(b + off[0]);
    r->nz_row_u = reinterpret_cast<int32_t*>(b + off[1]);
    r->nnz_lc = reinterpret_cast<int32_t*>(b + off[2]);
    r->dig_u = dig ? reinterpret_cast<uint64_t*>(b + off[3]) : nullptr;
    r->dig_lc = dig ? reinterpret_cast<uint64_t*>(b + off[4]) : nullptr;
    r->lmask = reinterpret_cast<uint32_t*>(b + off[5]);
    r->umask = reinterpret_cast<uint32_t*>(b + off[6]);
    r->nnz_lr = lrow ? reinterpret_cast<int32_t*>(b + off[7]) : nullptr;
    r->dig_lr = lrow ? reinterpret_cast<uint64_t*>(b + off[8]) : nullptr;
    r->sflags = reinterpret_cast<int8_t*>(b + off[9]);
    r->counters = reinterpret_cast<unsigned long long*>(b + off[10]);
    r->link = reinterpret_cast<uint8_t*>(b + off[11]);
    // zero the scatter targets, the flags, the counters and the links
    cudaError_t e = cudaMemsetAsync(b + off[7], 0, total - off[7], stream);
    if (e != cudaSuccess) {
        dev_free_on(ctx, r->arena, r->bytes, stream);
        delete r;
        return cuda_fail(ctx, e, "result init");
    }
    *out = r;
    return GSOFA_OK;
}

// The arrays a factorization finds zeroed.
cudaError_t result_clear(gsofa_result* r, cudaStream_t stream) {
    size_t off[12];
    const size_t total = result_layout(r->n, r->flags, off);
    return cudaMemsetAsync(static_cast<char*>(r->arena) + off[7], 0, total - off[7], stream);
}

int result_alloc(gsofa_ctx* ctx, int32_t n, uint32_t flags, int32_t mss, gsofa_result** out) {
    return result_alloc_on(ctx, n, flags, mss, ctx->stream, out);
}

MatDesc make_desc(const gsofa_matrix* m, const gsofa_result* r, long long base) {
    MatDesc d{};
    d.n = m->n;
    d.flags = (int32_t)r->flags;
    d.rowptr = m->rowptr;
    d.col = m->col;
    d.trowptr = m->trowptr;
    d.tcol = m->tcol;
    d.wdeg = m->wdeg;
    d.dplanes = m->dplanes;
    d.nplanes = m->nplanes;
    d.asym = m->asym;
    d.nnz_u = r->nnz_u;
    d.nz_row_u = r->nz_row_u;
    d.dig_u = r->dig_u;
    d.nnz_lc = r->nnz_lc;
    d.dig_lc = r->dig_lc;
    d.lmask = r->lmask;
    d.sflags = r->sflags;
    d.nnz_lr = r->nnz_lr;
    d.dig_lr = r->dig_lr;
    d.counters = r->counters;
    d.uptr = r->uptr;
    d.ucols = r->ucols;
    d.lptr = r->lptr;
    d.lrows = r->lrows;
    d.link = r->link;
    d.umask = r->umask;
    d.item_base = base;
    return d;
}

// Whether the counting traversals (gsofa_chain.cu, gsofa_hub.cu) run these
// options: they always reuse closures and search top-down, so the diagnostic
// switches take traverse_kernel.  Per-row L statistics come from gsofa_hub.cu
// alone: with them, only matrices that all go there.  The hubs' arrays of one
// launch hold fewer than 2^31 entries, the count their scans take.
bool chain_runs(const gsofa_opts& o, const gsofa_matrix* const* mats, int32_t count) {
    if ((o.flags & (GSOFA_NO_MERGE | GSOFA_NO_CHAIN)) || o.bu_alpha > 0) return false;
    long long hub_rows = 0;
    bool any = count == 0;
    for (int32_t i = 0; i < count; i++) {
        const int32_t method = method_of(mats[i]);
        any |= method != METHOD_WALK;
        if (method == METHOD_CHAIN && (o.flags & GSOFA_L_ROW_STATS)) return false;
        if (method == METHOD_HUB) hub_rows += mats[i]->n + 32ll;
    }
    return any && hub_rows * std::max(hub_count(), 2 * hub_bases()) <= INT_MAX;
}

int plan_chain(gsofa_ctx* ctx, int32_t nmax, long long total_sources, const gsofa_opts* o, ChainCfg* c) {
    c->words = bitmap_words(nmax);
    const size_t fixed = (chain_sparse_bytes() + 15) & ~(size_t)15;
    size_t bytes = ((size_t)c->words * 4 + 15) & ~(size_t)15;
    if (fixed + bytes + 20 * 1024 > (size_t)ctx->smem_optin || (o->flags & GSOFA_FORCE_GLOBAL_BITMAP))
        bytes = 0;
    c->smem_words = bytes ? c->words : 0;
    c->gbm_count = bytes ? 1 : 2;
    c->smem = fixed + bytes;
    c->block = o->threads_per_source;
    if (c->block <= 0) {
        const long long fit = ctx->smem_per_sm / (long long)(c->smem + 2048);
        // Many small matrices: more chunks at a time (a batch of 64: 5.0 -> 3.9 ms
        // with 128 threads against 256).  A few: their chunks' first searches
        // are the longest chain, shorter with more threads (170 x 170 mesh:
        // 0.97 against 0.82 ms).
        c->block = fit >= 8 && total_sources >= 8ll * nmax ? 128 : fit >= 4 ? 256 : fit >= 2 ? 512 : 1024;
    }
    if (c->block != 128 && c->block != 256 && c->block != 512 && c->block != 1024)
        return set_err(ctx, GSOFA_ERR_ARG, "threads_per_source must be 128, 256, 512 or 1024");
    const int occ = chain_occupancy(c->block, false, c->smem);
    if (occ <= 0)
        return set_err(ctx, GSOFA_ERR_UNSUPPORTED,
                       "traversal kernel cannot be resident (block %d, %zu B shared)", c->block,
                       c->smem);
    c->grid = occ * ctx->sm_count;
    if (o->sources_in_flight > 0) c->grid = std::min(c->grid, o->sources_in_flight);
    return GSOFA_OK;
}

void fill_chain_launch(ChainLaunch* L, const ChainCfg& c, const gsofa_opts& o, int32_t nmax) {
    L->queue_stride = std::max(nmax, 1);
    if (o.flags & GSOFA_DEBUG_QUEUE_CAP) L->queue_stride = std::min<long long>(L->queue_stride, 64);
    L->list_cap = (int)std::min<long long>(chain_list_cap(), L->queue_stride);
    L->gbm_count = c.gbm_count;
    L->bitmap_words = c.words;
    L->smem_words = c.smem_words;
}

int32_t method_of(const gsofa_matrix* m) {
    // the hubs' launch does not count a row's distinct ids, the chain does
    if (m->host_dup != 0 && (m->n <= kDirectMax || m->host_sym <= 0)) return METHOD_WALK;
    if (m->n <= kDirectMax) return METHOD_DIRECT;
    return m->host_sym > 0 ? METHOD_CHAIN : METHOD_HUB;
}

bool plan_hub(gsofa_ctx* ctx, std::vector<MatDesc>* descs, const gsofa_opts& o, void* ws,
              size_t* bytes, size_t room, HubLaunch* L, HubCfg* c, int most) {
    *L = HubLaunch{};
    *c = HubCfg{};
    long long sources = 0, off = 0, items = 0;
    int32_t n_max = 0;
    int hubs = 0, k = 0;
    for (MatDesc& d : *descs) {
        k++;
        if (d.method != METHOD_HUB && d.method != METHOD_DIRECT) continue;
        sources += 2ll * d.n;
        n_max = std::max(n_max, d.n);
        if (d.method != METHOD_HUB) continue;
        hubs++;
        L->hub_mats = k;
        d.hub_off = off;
        d.hub_len = ((long long)d.n + 1 + 31) & ~31ll;
        off += d.hub_len;
    }
    *bytes = 0;
    if (n_max == 0) return false;
    const int nm = (int)descs->size(), W = hub_count();
    c->any_hub = hubs > 0;
    c->n_max = n_max;
    c->sm_count = ctx->sm_count;
    // labels in the shared memory of a cluster: of as many CTAs as leave every
    // job's cluster room on the GPU at once, and hold the largest matrix's labels.
    // Calls with 1, 2, 4, 8 and 16 CTAs (the rule's choice for one matrix): banded
    // n = 11,948 0.39, 0.37, 0.34, 0.31, 0.28 ms; random n = 20,000 0.72, 0.76, 0.76,
    // 0.76, 0.77; random n = 50,000 1.71, 1.65, 1.40, 1.14, 1.35; circuit-like n =
    // 100,000 4.13, 4.12, 3.46, 2.88, 2.47.  Beside a large matrix small ones use its
    // width: 63 of 2,000 to 8,000 rows 3.3 ms, circuit-like n = 659,033 14.0, all in
    // one call 20.4
    const int widest = std::min(ctx->label_cluster, most);
    c->cluster = 1;
    while (c->cluster < widest && 2 * W * hubs * 2 * c->cluster <= ctx->sm_count) c->cluster *= 2;
    while (c->cluster < widest && label_smem_bytes(n_max, c->cluster) + 2048 > (size_t)ctx->smem_optin)
        c->cluster *= 2;
    // by the whole GPU in global memory: matrices too large for that, GPUs that
    // place no cluster, and with the diagnostic GSOFA_FORCE_GLOBAL_BITMAP
    if (widest == 0 || label_smem_bytes(n_max, c->cluster) + 2048 > (size_t)ctx->smem_optin ||
        (o.flags & GSOFA_FORCE_GLOBAL_BITMAP))
        c->cluster = 0;
    L->nmats = nm;
    L->total = off;
    // sources per warp and turn: few enough that the GPU's warps all have some
    long long g = 1;
    while (g < 16 && sources / (2 * g) >= 2ll * 32 * ctx->sm_count) g *= 2;
    L->group = (int)g;
    for (MatDesc& d : *descs) {
        d.hub_item = items;
        d.hub_slots = 0;
        if ((d.method != METHOD_HUB && d.method != METHOD_DIRECT) || d.n == 0) continue;
        d.hub_slots = 1;
        while (d.hub_slots < 2 * ((d.n + g - 1) / g)) d.hub_slots *= 2;
        items += d.hub_slots;
    }
    L->total_items = items;
    // large_kernel: its bitmap in shared memory where four CTAs' fit an SM
    L->bitmap_words = bitmap_words(n_max);
    const size_t bm = ((size_t)L->bitmap_words * 4 + 15) & ~(size_t)15;
    L->large_smem = 4 * (bm + 2048) <= (size_t)ctx->smem_per_sm && !(o.flags & GSOFA_FORCE_GLOBAL_BITMAP);
    c->large_smem = L->large_smem ? bm : 0;
    int occ = large_occupancy(c->large_smem);
    if (occ <= 0) occ = 1;
    c->large_grid = occ * ctx->sm_count;
    c->extra_grid = extra_ctas_per_sm() * ctx->sm_count;
    if (o.sources_in_flight > 0) {
        c->large_grid = std::min(c->large_grid, o.sources_in_flight);
        c->extra_grid = std::min(c->extra_grid, o.sources_in_flight);
    }
    L->queue_stride = n_max;
    if (o.flags & GSOFA_DEBUG_QUEUE_CAP) L->queue_stride = std::min<long long>(L->queue_stride, 64);
    c->l_rows = (o.flags & GSOFA_L_ROW_STATS) != 0;
    const long long uses = c->l_rows ? (long long)W * off : 0;
    c->scan_bytes = c->any_hub ? hub_scan_bytes(2ll * hub_bases() * off, uses) : 0;
    // workspace: the zeroed block first
    size_t at = 0;
    char* const w = static_cast<char*>(ws);
    auto place = [&](size_t b) {
        char* p = w ? w + at : nullptr;
        at += align256(b);
        return static_cast<void*>(p);
    };
    const size_t T = (size_t)off;
    L->zeroed = w;
    L->base = static_cast<Tot*>(place(sizeof(Tot) * 2 * (size_t)hub_bases() * T));
    L->l_use = static_cast<LRowUse*>(place(sizeof(LRowUse) * (size_t)uses));
    L->stamp = static_cast<int32_t*>(place(4 * 2 * (size_t)W * T));
    L->lcnt = static_cast<int32_t*>(place(32 * 2 * (size_t)W * (size_t)nm));
    L->fallback = static_cast<int32_t*>(place(4 * (size_t)nm));
    L->given_up = static_cast<int32_t*>(place(4 * (size_t)nm));
    L->judged = static_cast<int32_t*>(place(8 * (size_t)nm));
    L->large_work = static_cast<unsigned long long*>(place(16 * (size_t)nm));
    L->counters = static_cast<unsigned long long*>(place(8 * CNT_SLOTS * (size_t)nm));
    L->hubs = static_cast<unsigned long long*>(place(8 * (size_t)W * (size_t)nm));
    L->large_count = static_cast<int*>(place(4));
    L->work_counter = static_cast<unsigned long long*>(place(16));
    c->zeroed_bytes = at;
    L->lam = static_cast<int32_t*>(place(4 * 2 * (size_t)W * T));
    L->lq = static_cast<int32_t*>(place(8 * 2 * (size_t)W * T));
    L->large = static_cast<unsigned long long*>(place(8 * (size_t)sources));
    c->scan_tmp = place(c->scan_bytes);
    // the large searches' CTAs, by far the most of it, take turns: as many as fit
    auto large_bytes = [&]() {
        return align256((size_t)c->large_grid * (size_t)L->queue_stride * 4) +
               align256(L->large_smem ? 0 : (size_t)c->large_grid * (size_t)L->bitmap_words * 4);
    };
    while (c->large_grid > 1 && at + large_bytes() > room) c->large_grid = (c->large_grid + 1) / 2;
    L->queue = static_cast<int32_t*>(place((size_t)c->large_grid * (size_t)L->queue_stride * 4));
    L->gbm = static_cast<uint32_t*>(
        place(L->large_smem ? 0 : (size_t)c->large_grid * (size_t)L->bitmap_words * 4));
    *bytes = at;
    return true;
}

// The last separators of a mesh in nested-dissection order reach almost
// everything: their chunks' first searches, from nothing, take as long as all
// the rest of the launch.  From 65,536 rows on, the chunks of the last 2 % of them
// go to CTAs of 1,024 threads, at most one per SM, beside the rest.  Times of a
// call without and with them: 9-point meshes of 260 x 260 1.43 and 1.15 ms, 300 x
// 300 1.83 and 1.36, 362 x 362 2.50 and 1.88, 500 x 500 4.25 and 3.03; 7-point of
// 46^3 1.32 and 1.34, 50^3 1.63 and 1.57, 64^3 2.97 and 2.80; 16 meshes of 300 x 300
// 10.6 and 10.1.  Below, there is little to gain (170 x 170: 0.78 and 0.74) and a
// batch of 64 matrices of up to 30,000 rows loses more by the SMs those CTAs take
// (5.9 and 7.2).
constexpr int32_t kTopRows = 65536;
long long chain_top_items(const gsofa_opts& o, int32_t n, long long chunk) {
    if (o.sources_in_flight > 0 || n < kTopRows) return 0;
    const long long chunks = (n + chunk - 1) / chunk;
    return std::min(chunks - 1, (n / 50 + chunk - 1) / chunk);
}

constexpr int kTopBlock = 1024;

size_t chain_queue_bytes(const gsofa_ctx* ctx, const ChainCfg& c, int32_t nmax, bool top) {
    return ((size_t)c.grid + (top ? (size_t)ctx->sm_count : 0)) * (size_t)std::max(nmax, 1) * 4;
}

size_t chain_gbm_bytes(const gsofa_ctx* ctx, const ChainCfg& c, bool top) {
    return ((size_t)c.grid + (top ? (size_t)ctx->sm_count : 0)) * (size_t)c.gbm_count * (size_t)c.words * 4;
}

cudaError_t launch_chain_both(gsofa_ctx* ctx, const ChainLaunch& L, const ChainCfg& c, long long top_items) {
    cudaError_t e = cudaSuccess;
    if (top_items > 0) {
        ChainLaunch T = L;
        T.items = ITEMS_TOP;
        T.total_items = top_items;
        T.sample_stride = 1;
        T.work_counter = L.work_counter + 1;
        T.queue = L.queue + (size_t)c.grid * (size_t)L.queue_stride;
        T.gbm = L.gbm + (size_t)c.grid * (size_t)c.gbm_count * (size_t)c.words;
        e = cudaEventRecord(ctx->fork, ctx->stream);
        if (e == cudaSuccess) e = cudaStreamWaitEvent(ctx->side_stream, ctx->fork, 0);
        if (e == cudaSuccess)
            e = launch_chain(T, kTopBlock, false, (int)std::min<long long>(top_items, ctx->sm_count), c.smem,
                             ctx->side_stream);
        if (e == cudaSuccess) e = cudaEventRecord(ctx->join, ctx->side_stream);
    }
    if (e == cudaSuccess && L.total_items > 0) e = launch_chain(L, c.block, false, c.grid, c.smem, ctx->stream);
    if (e == cudaSuccess && top_items > 0) e = cudaStreamWaitEvent(ctx->stream, ctx->join, 0);
    return e;
}

long long chain_chunk(const gsofa_opts& o, long long total_sources, int32_t nmax, int grid) {
    if (o.chunk_sources > 0) return o.chunk_sources;
    // A chunk's first source is searched from nothing: about two items per CTA,
    // at most 128 sources each, since items differ in cost (64^3 mesh: 3.3 ms with
    // 128 sources, 4.0 with 443; 40^3: 0.92 with 54, 1.09 with 108).  At most 64
    // below 131,072 rows (a batch's meshes of up to 30,000 rows 5.9 -> 5.3 ms).
    return std::max(1ll, std::min(nmax < 131072 ? 64ll : 128ll, (total_sources + 2ll * grid - 1) / (2ll * grid)));
}

// Runs the traversal (and optionally supernodes / pattern) for `count`
// matrices in one persistent launch.  results[i] must be freshly allocated.
// counting: by the counting traversals where chain_runs, else by traverse_kernel.
int run_factor_with(gsofa_ctx* ctx, const gsofa_matrix* const* mats, int32_t count,
                    const gsofa_opts* o, gsofa_result** res, long long sample_stride,
                    bool counting) {
    int32_t nmax = 0;
    long long total_sources = 0, weight = 0;
    for (int32_t i = 0; i < count; i++) {
        nmax = std::max(nmax, mats[i]->n);
        weight += chunk_weight(ctx, mats[i]);
        total_sources += mats[i]->n;
    }
    const bool chain = counting && chain_runs(*o, mats, count);
    const bool pattern = (o->flags & GSOFA_PATTERN) != 0;
    const bool traverse = !chain || pattern;
    int rc = GSOFA_OK;
    // matrix descriptors, largest matrices first
    const std::vector<int32_t> order = batch_order(mats, count);
    std::vector<MatDesc> descs((size_t)count);
    auto place = [&](long long chunk, int per_chunk) {
        long long base = 0;
        for (int32_t k = 0; k < count; k++) {
            const int32_t i = order[(size_t)k];
            descs[(size_t)k] = make_desc(mats[i], res[i], base);
            base += per_chunk * ((mats[i]->n + chunk - 1) / chunk);
        }
        return base;
    };
    unsigned long long* wc = nullptr;
    int32_t* dstatus = work_counter_status(ctx, &wc);
    const long long stride = sample_stride > 1 ? sample_stride : 1;

    ChainCfg ccfg;
    ChainLaunch CL{};
    HubLaunch HL{};
    HubCfg hcfg;
    bool hub = false;
    long long top_items = 0;
    if (chain) {
        long long chain_sources = 0;
        for (int32_t i = 0; i < count; i++)
            if (method_of(mats[i]) == METHOD_CHAIN) chain_sources += mats[i]->n;
        rc = plan_chain(ctx, std::max(nmax, 1), chain_sources, o, &ccfg);
        if (rc) return rc;
        CL.chunk = (int)chain_chunk(*o, chain_sources, nmax, ccfg.grid);
        long long items = 0;
        place(CL.chunk, 1);
        for (int32_t k = 0; k < count; k++) {
            const gsofa_matrix* m = mats[order[(size_t)k]];
            MatDesc& d = descs[(size_t)k];
            d.method = method_of(m);
            d.item_base = items;
            d.top_base = top_items;
            if (d.method != METHOD_CHAIN) continue;
            d.top_items = stride > 1 ? 0 : chain_top_items(*o, m->n, CL.chunk);
            top_items += d.top_items;
            items += (m->n + CL.chunk - 1) / CL.chunk - d.top_items;
        }
        ccfg.grid = (int)std::max(1ll, std::min<long long>(ccfg.grid, items));
        size_t hub_bytes = 0;
        // the hubs' workspace may take what the budget leaves beside the chain's
        const size_t chain_bytes = align256(chain_queue_bytes(ctx, ccfg, nmax, top_items > 0)) +
                                   align256(chain_gbm_bytes(ctx, ccfg, top_items > 0)) +
                                   align256(sizeof(MatDesc) * (size_t)count);
        const size_t others = ctx->used - std::min(ctx->used, ctx->hub_ws_bytes + ctx->queue_bytes + ctx->gbitmap_bytes);
        const size_t room = ctx->budget > others + chain_bytes ? ctx->budget - others - chain_bytes : 0;
        if (plan_hub(ctx, &descs, *o, nullptr, &hub_bytes, room, &HL, &hcfg)) {
            rc = ensure(ctx, &ctx->hub_ws, &ctx->hub_ws_bytes, hub_bytes);
            if (rc) return rc;
            hub = plan_hub(ctx, &descs, *o, ctx->hub_ws, &hub_bytes, room, &HL, &hcfg);
            HL.status = dstatus;
        }
        rc = ensure(ctx, &ctx->queue, &ctx->queue_bytes, chain_queue_bytes(ctx, ccfg, nmax, top_items > 0));
        if (!rc)
            rc = ensure(ctx, &ctx->gbitmap, &ctx->gbitmap_bytes, chain_gbm_bytes(ctx, ccfg, top_items > 0));
        if (rc) return rc;
        fill_chain_launch(&CL, ccfg, *o, nmax);
        CL.nmats = count;
        CL.total_items = (items + stride - 1) / stride;
        CL.sample_stride = stride;
        CL.work_counter = wc;
        CL.queue = reinterpret_cast<int32_t*>(ctx->queue);
        CL.gbm = reinterpret_cast<uint32_t*>(ctx->gbitmap);
        CL.status = dstatus;
    }
    LaunchCfg cfg;
    TraverseLaunch L{};
    if (traverse) {
        rc = plan_launch(ctx, std::max(nmax, 1), o, &cfg);
        if (rc) return rc;
        // So few sources that each can have a CTA of its own: chunks of one source
        // run them all at once; with more, chunks share closures between
        // consecutive sources.
        const long long chunk = o->chunk_sources > 0 ? o->chunk_sources
                                : 2 * total_sources <= cfg.grid ? 1
                                                                : default_chunk(weight, cfg.grid);
        const long long items = chain ? 0 : place(chunk, 2);
        rc = ensure(ctx, &ctx->queue, &ctx->queue_bytes, (size_t)cfg.grid * (size_t)std::max(nmax, 1) * 4);
        if (!rc && !cfg.smem_bitmap)
            rc = ensure(ctx, &ctx->gbitmap, &ctx->gbitmap_bytes, (size_t)cfg.grid * (size_t)cfg.words * 4);
        const bool merge = !(o->flags & GSOFA_NO_MERGE);
        int ring = o->cached_closures > 0 ? o->cached_closures : kDefaultRing;
        if (ring > kMaxRing) ring = kMaxRing;
        while (ring & (ring - 1)) ring &= ring - 1;  // power of 2
        if (!rc && merge)
            rc = ensure(ctx, &ctx->gprev, &ctx->gprev_bytes,
                        (size_t)cfg.grid * (size_t)ring * (size_t)cfg.words * 4);
        if (rc) return rc;
        L.nmats = count;
        L.total_items = (items + stride - 1) / stride;
        L.sample_stride = stride;
        L.work_counter = wc;
        L.queue = reinterpret_cast<int32_t*>(ctx->queue);
        L.queue_stride = std::max(nmax, 1);
        if (o->flags & GSOFA_DEBUG_QUEUE_CAP) L.queue_stride = std::min<long long>(L.queue_stride, 64);
        L.gbitmap = reinterpret_cast<uint32_t*>(ctx->gbitmap);
        L.bitmap_words = cfg.words;
        L.status = dstatus;
        L.pattern_pass = 0;
        L.bu_alpha = o->bu_alpha > 0 ? o->bu_alpha : (o->bu_alpha < 0 ? 0 : kDefaultBuAlpha);
        L.bu_beta = o->bu_beta > 0 ? o->bu_beta : kDefaultBuBeta;
        L.bu_min_src = o->bu_min_source > 0 ? o->bu_min_source : kBuMinSource;
        L.gprev = reinterpret_cast<uint32_t*>(ctx->gprev);
        L.merge = merge ? 1 : 0;
        L.chain = merge && !(o->flags & GSOFA_NO_CHAIN) ? 1 : 0;
        L.chain_wait_ns = chain_wait_ns(*o);
        L.ring = ring;
        L.chunk = (int)chunk;
        L.heavy_len = o->heavy_row > 0 ? ((o->heavy_row + 3) & ~3) : kDefaultHeavyRow;
        // both traversals share the queue and bitmap buffers, which may have grown
        CL.queue = L.queue;
        CL.gbm = L.gbitmap;
    }
    rc = ensure(ctx, &ctx->desc, &ctx->desc_bytes, sizeof(MatDesc) * (size_t)count);
    if (!rc) rc = ensure_pinned(ctx, (size_t)count);
    if (rc) return rc;
    void* const ddesc = ctx->desc;
    CK(cudaMemcpyAsync(ddesc, descs.data(), sizeof(MatDesc) * (size_t)count, cudaMemcpyHostToDevice,
                       ctx->stream));
    CK(cudaMemsetAsync(ctx->small, 0, 128, ctx->stream));
    L.mats = CL.mats = HL.mats = reinterpret_cast<const MatDesc*>(ddesc);

    CK(cudaEventRecord(ctx->ev0, ctx->stream));
    if (hub) {
        CK(launch_hub(HL, hcfg, (o->flags & GSOFA_DIGESTS) != 0, ctx->stream));
        CK(cudaMemcpyAsync(ctx->h_fallback, HL.fallback, 4 * (size_t)count, cudaMemcpyDeviceToHost,
                           ctx->stream));
    }
    if (chain) CK(launch_chain_both(ctx, CL, ccfg, top_items));
    if (!chain && L.total_items > 0)
        CK(launch_traverse(L, cfg.block, cfg.grid, cfg.smem_bitmap, cfg.smem, ctx->stream));
    CK(cudaEventRecord(ctx->evt, ctx->stream));
    for (int32_t k = 0; k < count; k++) {
        const int32_t i = order[(size_t)k];
        if ((o->flags & GSOFA_SUPERNODES) && mats[i]->n > 0)
            CK(launch_supernodes(mats[i]->n, o->max_supernode_size, res[i]->nz_row_u, res[i]->lmask,
                                 res[i]->sflags, res[i]->counters, ctx->stream));
    }
    CK(cudaEventRecord(ctx->ev1, ctx->stream));
    for (int32_t i = 0; i < count; i++)
        CK(cudaMemcpyAsync(ctx->h_counters + (size_t)i * CNT_SLOTS, res[i]->counters, 8 * CNT_SLOTS,
                           cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaMemcpyAsync(ctx->h_status, dstatus, 4, cudaMemcpyDeviceToHost, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    rc = check_status(ctx);
    if (rc) return rc;
    float ms_f = 0.f, ms_trav_f = 0.f;
    CK(cudaEventElapsedTime(&ms_f, ctx->ev0, ctx->ev1));
    CK(cudaEventElapsedTime(&ms_trav_f, ctx->ev0, ctx->evt));
    double ms = ms_f, ms_trav = ms_trav_f;
    std::vector<unsigned long long> totals(ctx->h_counters, ctx->h_counters + (size_t)count * CNT_SLOTS);

    // those that neither traversal takes and those that the hubs' launch left
    std::vector<int32_t> left;
    for (int32_t k = 0; k < count && chain; k++)
        if (descs[(size_t)k].method == METHOD_WALK || (hub && ctx->h_fallback[k]))
            left.push_back(order[(size_t)k]);
    const int walked = chain ? (int)left.size() : count;
    if (!left.empty()) {
        std::vector<const gsofa_matrix*> lm;
        std::vector<gsofa_result*> lr;
        for (const int32_t i : left) {
            lm.push_back(mats[i]);
            lr.push_back(res[i]);
            CK(result_clear(res[i], ctx->stream));
        }
        gsofa_opts lo = *o;
        lo.flags &= ~(uint32_t)GSOFA_PATTERN;  // made below, with the others'
        rc = run_factor_with(ctx, lm.data(), (int32_t)lm.size(), &lo, lr.data(), sample_stride, false);
        if (rc) return rc;
        for (size_t j = 0; j < left.size(); j++)
            std::copy_n(ctx->h_counters + j * CNT_SLOTS, (size_t)CNT_SLOTS,
                        totals.data() + (size_t)left[j] * CNT_SLOTS);
        ms += lr[0]->counts.ms_device;
        ms_trav += lr[0]->counts.ms_traverse;
        // the buffers may have grown
        L.queue = reinterpret_cast<int32_t*>(ctx->queue);
        L.gbitmap = reinterpret_cast<uint32_t*>(ctx->gbitmap);
        L.gprev = reinterpret_cast<uint32_t*>(ctx->gprev);
    }

    // pattern pass (second traversal writing sorted ids)
    if (pattern) {
        for (int32_t k = 0; k < count; k++) {
            const int32_t i = order[(size_t)k];
            gsofa_result* r = res[i];
            const unsigned long long* c = totals.data() + (size_t)i * CNT_SLOTS;
            const size_t N = (size_t)r->n + 1;
            const size_t nu = c[CNT_NNZ_U], nl = c[CNT_NNZ_L];
            size_t total = align256(8 * N) * 2 + align256(4 * std::max<size_t>(nu, 1)) +
                           align256(4 * std::max<size_t>(nl, 1));
            rc = dev_alloc(ctx, total, &r->parena);
            if (rc) return rc;
            r->pbytes = total;
            char* b = reinterpret_cast<char*>(r->parena);
            r->uptr = reinterpret_cast<int64_t*>(b);
            r->lptr = reinterpret_cast<int64_t*>(b + align256(8 * N));
            r->ucols = reinterpret_cast<int32_t*>(b + 2 * align256(8 * N));
            r->lrows = reinterpret_cast<int32_t*>(b + 2 * align256(8 * N) +
                                                  align256(4 * std::max<size_t>(nu, 1)));
            rc = ensure(ctx, &ctx->scan_tmp, &ctx->scan_tmp_bytes, pattern_scan_bytes(r->n));
            if (rc) return rc;
            CK(launch_pattern_ptrs(r->n, r->nnz_u, r->nnz_lc, r->uptr, r->lptr, ctx->scan_tmp,
                                   ctx->scan_tmp_bytes, ctx->stream));
        }
        L.total_items = place(L.chunk, 2);
        CK(cudaMemcpyAsync(ddesc, descs.data(), sizeof(MatDesc) * (size_t)count,
                           cudaMemcpyHostToDevice, ctx->stream));
        CK(cudaMemsetAsync(ctx->small, 0, 128, ctx->stream));
        L.pattern_pass = 1;
        L.sample_stride = 1;
        if (L.total_items > 0)
            CK(launch_traverse(L, cfg.block, cfg.grid, cfg.smem_bitmap, cfg.smem, ctx->stream));
        CK(cudaMemcpyAsync(ctx->h_status, dstatus, 4, cudaMemcpyDeviceToHost, ctx->stream));
        CK(cudaStreamSynchronize(ctx->stream));
        rc = check_status(ctx);
        if (rc) return rc;
    }

    ctx->walked = walked;
    for (int32_t i = 0; i < count; i++) {
        gsofa_result* r = res[i];
        const unsigned long long* c = totals.data() + (size_t)i * CNT_SLOTS;
        gsofa_counts& k = r->counts;
        k.n = r->n;
        k.fill_count = c[CNT_FILLS];
        k.nnz_l = c[CNT_NNZ_L];
        k.nnz_u = c[CNT_NNZ_U];
        k.nnz_lu = c[CNT_NNZ_L] + c[CNT_NNZ_U] + (uint64_t)r->n;
        k.n_supernodes = (o->flags & GSOFA_SUPERNODES) ? (int64_t)c[CNT_NSUP] + 1 : -1;
        k.edges_alg = c[CNT_EDGES_ALG];
        k.vertices_alg = c[CNT_VERTS_ALG];
        k.edges_traversed = c[CNT_EDGES_TRAV];
        k.sources_chained = c[CNT_CHAINED];
        k.ms_device = (double)ms;  // for a batch: the whole launch
        k.ms_traverse = (double)ms_trav;
    }
    return GSOFA_OK;
}

// The same, within the budget: when the counting traversals' workspace does not
// fit, nothing of earlier calls is kept and traverse_kernel, whose workspace is
// smaller, counts.
int run_factor(gsofa_ctx* ctx, const gsofa_matrix* const* mats, int32_t count, const gsofa_opts* o,
               gsofa_result** res, long long sample_stride = 1) {
    ctx->factoring = true;
    ctx->walked = 0;
    int rc = run_factor_with(ctx, mats, count, o, res, sample_stride, true);
    if (rc == GSOFA_ERR_OOM_BUDGET) {
        drop_workspace(ctx);
        rc = GSOFA_OK;
        for (int32_t i = 0; i < count && rc == GSOFA_OK; i++) {
            gsofa_result* r = res[i];
            dev_free(ctx, r->parena, r->pbytes);
            r->parena = nullptr;
            r->pbytes = 0;
            r->uptr = r->lptr = nullptr;
            r->ucols = r->lrows = nullptr;
            const cudaError_t e = result_clear(r, ctx->stream);
            if (e != cudaSuccess) rc = cuda_fail(ctx, e, "result arrays");
        }
        if (rc == GSOFA_OK) rc = run_factor_with(ctx, mats, count, o, res, sample_stride, false);
    }
    ctx->factoring = false;
    return rc;
}

int validate_opts(gsofa_ctx* ctx, const gsofa_opts* o) {
    if (o->max_supernode_size <= 0)
        return set_err(ctx, GSOFA_ERR_ARG, "max_supernode_size must be positive");
    if (o->threads_per_source < 0 || o->sources_in_flight < 0 || o->chunk_sources < 0 ||
        o->cached_closures < 0)
        return set_err(ctx, GSOFA_ERR_ARG, "negative launch option");
    return GSOFA_OK;
}

// ---- fast ASCII reader --------------------------------------------------------
int read_file(const char* path, std::string* out) {
    FILE* f = fopen(path, "rb");
    if (!f) return -1;
    if (fseek(f, 0, SEEK_END) != 0) { fclose(f); return -1; }
    long sz = ftell(f);
    if (sz < 0) { fclose(f); return -1; }
    rewind(f);
    out->resize((size_t)sz);
    size_t got = sz ? fread(&(*out)[0], 1, (size_t)sz, f) : 0;
    fclose(f);
    return got == (size_t)sz ? 0 : -1;
}

// Parses up to `count` whitespace-separated integers; returns how many.
int64_t parse_ints(const std::string& s, size_t* pos, int64_t count, int32_t* out, bool* bad) {
    const char* p = s.data() + *pos;
    const char* e = s.data() + s.size();
    int64_t i = 0;
    while (i < count) {
        while (p < e && (*p == ' ' || *p == '\n' || *p == '\r' || *p == '\t')) p++;
        if (p >= e) break;
        bool neg = false;
        if (*p == '-') { neg = true; p++; }
        if (p >= e || *p < '0' || *p > '9') { *bad = true; break; }
        int64_t v = 0;
        while (p < e && *p >= '0' && *p <= '9') { v = v * 10 + (*p - '0'); p++; if (v > 4294967295ll) { *bad = true; break; } }
        out[i++] = (int32_t)(neg ? -v : v);
    }
    *pos = (size_t)(p - s.data());
    return i;
}

// The reference's three ASCII files (csr = "E N" then E column ids, beg /
// end = n ids each) into host arrays.  ctx may be null (no message kept).
int parse_dat_files(gsofa_ctx* ctx, const char* beg_file, const char* end_file,
                    const char* csr_file, int32_t* n_out, int64_t* nnz_out,
                    std::vector<int32_t>* beg, std::vector<int32_t>* end,
                    std::vector<int32_t>* col) {
    std::string sc, sb, se;
    if (read_file(csr_file, &sc)) return set_err(ctx, GSOFA_ERR_IO, "cannot read %s", csr_file);
    size_t pos = 0;
    bool bad = false;
    int32_t hdr[2];
    if (parse_ints(sc, &pos, 2, hdr, &bad) != 2 || bad || hdr[0] < 0 || hdr[1] < 0)
        return set_err(ctx, GSOFA_ERR_IO, "%s: bad header (expected E N)", csr_file);
    const int64_t E = hdr[0];
    const int32_t n = hdr[1];
    col->assign((size_t)std::max<int64_t>(E, 1), 0);
    beg->assign((size_t)n + 1, 0);
    end->assign((size_t)n + 1, 0);
    if (parse_ints(sc, &pos, E, col->data(), &bad) != E || bad)
        return set_err(ctx, GSOFA_ERR_IO, "%s: expected %lld column ids", csr_file, (long long)E);
    if (read_file(beg_file, &sb)) return set_err(ctx, GSOFA_ERR_IO, "cannot read %s", beg_file);
    if (read_file(end_file, &se)) return set_err(ctx, GSOFA_ERR_IO, "cannot read %s", end_file);
    pos = 0;
    if (parse_ints(sb, &pos, n, beg->data(), &bad) != n || bad)
        return set_err(ctx, GSOFA_ERR_IO, "%s: expected %d row starts", beg_file, n);
    pos = 0;
    if (parse_ints(se, &pos, n, end->data(), &bad) != n || bad)
        return set_err(ctx, GSOFA_ERR_IO, "%s: expected %d row ends", end_file, n);
    *n_out = n;
    *nnz_out = E;
    return GSOFA_OK;
}

}  // namespace host
}  // namespace gsofa

bool gsofa::matrix_view(const void* mat, MatrixView* out) {
    const gsofa_matrix* m = static_cast<const gsofa_matrix*>(mat);
    if (!m || !out || !m->ctx) return false;
    out->device = m->ctx->device;
    out->n = m->n;
    out->rowptr = m->rowptr;
    out->col = m->col;
    out->trowptr = m->trowptr;
    out->tcol = m->tcol;
    out->wdeg = m->wdeg;
    out->dplanes = m->dplanes;
    out->nplanes = m->nplanes;
    out->asym = m->asym;
    return true;
}

void gsofa::host::ingest_bytes(int32_t n, int64_t nnz, size_t* kept, size_t* staging) {
    // padded A: each row rounded up to 4 entries (at most 3n pads); A^T: the same bound
    const size_t N1 = (size_t)n + 1;
    const size_t PT = (size_t)std::max<int64_t>(nnz + 3ll * n, 4);
    const size_t NW = (size_t)(((int64_t)n + 31) >> 5) + 1;
    *kept = align256(4 * N1) * 2 + align256(4 * PT) * 2 + align256(4 * NW) * 32 + 256;
    const size_t Nin = (size_t)std::max<int64_t>(nnz, 1);
    *staging = align256(4 * N1) + align256(4 * Nin) + align256(4 * N1) * 3 +
               align256(canonicalize_scan_bytes(n)) + 256;
}

cudaError_t gsofa::host::PinnedStager::init() {
    for (int k = 0; k < kBufs; k++) {
        cudaError_t e = cudaHostAlloc(&buf[k], kPiece, cudaHostAllocDefault);
        if (e == cudaSuccess) e = cudaEventCreateWithFlags(&ev[k], cudaEventDisableTiming);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

void gsofa::host::PinnedStager::release() {
    for (int k = 0; k < kBufs; k++) {
        if (ev[k]) cudaEventSynchronize(ev[k]);
        if (buf[k]) cudaFreeHost(buf[k]);
        if (ev[k]) cudaEventDestroy(ev[k]);
        buf[k] = nullptr;
        ev[k] = nullptr;
    }
}

cudaError_t gsofa::host::PinnedStager::upload(void* dst, const void* src, size_t bytes,
                                              cudaStream_t stream) {
    const char* p = static_cast<const char*>(src);
    char* d = static_cast<char*>(dst);
    while (bytes > 0) {
        const size_t k = std::min(bytes, kPiece);
        // the buffer's previous DMA is complete before it is refilled
        cudaError_t e = cudaEventSynchronize(ev[next]);
        if (e != cudaSuccess) return e;
        std::memcpy(buf[next], p, k);
        e = cudaMemcpyAsync(d, buf[next], k, cudaMemcpyHostToDevice, stream);
        if (e == cudaSuccess) e = cudaEventRecord(ev[next], stream);
        if (e != cudaSuccess) return e;
        next = (next + 1) % kBufs;
        p += k;
        d += k;
        bytes -= k;
    }
    return cudaSuccess;
}

int gsofa::host::ingest_csr(gsofa_ctx* ctx, cudaStream_t stream, int32_t* dstatus, int32_t n,
                            int64_t nnz, const int32_t* row_begin, const int32_t* row_end,
                            const int32_t* col, gsofa_matrix** out, PinnedStager* stager) {
    *out = nullptr;
    if (n < 0 || nnz < 0) return set_err(ctx, GSOFA_ERR_ARG, "negative n or nnz");
    if (n > 0 && (!row_begin || !row_end)) return set_err(ctx, GSOFA_ERR_ARG, "null row arrays");
    if (nnz > 0 && !col) return set_err(ctx, GSOFA_ERR_ARG, "null column array");
    if (nnz > INT32_MAX) return set_err(ctx, GSOFA_ERR_UNSUPPORTED, "nnz above 2^31-1");
    // host: padded row pointers of A.  Row v gets a multiple of 4 slots; the
    // number of padding slots of row v sits in the low 2 bits of rp[v+1].
    std::vector<int32_t> rp((size_t)n + 1);
    int64_t acc = 0, real = 0, maxd = 0;
    rp[0] = 0;
    for (int32_t v = 0; v < n; v++) {
        const int64_t b = row_begin[v], e = row_end[v];
        if (b < 0 || e < b || e > nnz)
            return set_err(ctx, GSOFA_ERR_ARG, "row %d interval [%lld,%lld) outside [0,%lld)", v,
                           (long long)b, (long long)e, (long long)nnz);
        const int64_t d = e - b, pd = (d + 3) & ~(int64_t)3;
        real += d;
        if (d > maxd) maxd = d;
        acc += pd;
        if (acc > INT32_MAX - 4 || real + 3ll * n > INT32_MAX - 4)
            return set_err(ctx, GSOFA_ERR_UNSUPPORTED, "padded nnz above 2^31");
        rp[(size_t)v + 1] = (int32_t)(acc | (pd - d));
    }
    const int64_t padded = acc;
    int nplanes = 0;
    while (nplanes < 32 && (maxd >> nplanes) != 0) nplanes++;
    gsofa_matrix* m = nullptr;
    int rc = matrix_alloc(ctx, stream, n, real, padded, nplanes, &m);
    if (rc) return rc;
    // staging: the raw input (row starts, column ids)
    const size_t N1 = (size_t)n + 1;
    const size_t Nin = (size_t)std::max<int64_t>(nnz, 1);
    const size_t stage = align256(4 * N1) + align256(4 * Nin);
    void* sblk = nullptr;
    rc = dev_alloc_on(ctx, stage, &sblk, stream);
    if (rc) { matrix_free_on(m, stream); return rc; }
    int32_t* dbeg = reinterpret_cast<int32_t*>(sblk);
    int32_t* dcol_in = reinterpret_cast<int32_t*>(reinterpret_cast<char*>(sblk) + align256(4 * N1));
    auto up = [&](void* dst, const void* src, size_t bytes) {
        return stager ? stager->upload(dst, src, bytes, stream)
                      : cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, stream);
    };
    cudaError_t e = up(m->rowptr, rp.data(), 4 * N1);
    if (e == cudaSuccess && n > 0) e = up(dbeg, row_begin, 4 * (size_t)n);
    if (e == cudaSuccess && nnz > 0) e = up(dcol_in, col, 4 * (size_t)nnz);
    if (e != cudaSuccess) {
        dev_free_on(ctx, sblk, stage, stream);
        matrix_free_on(m, stream);
        return cuda_fail(ctx, e, "ingest upload");
    }
    rc = matrix_build(ctx, stream, dstatus, m, nnz, dbeg, dcol_in,
                      maxd <= kSymmetryCheckMaxRow ? 1 : 0, 1);
    dev_free_on(ctx, sblk, stage, stream);  // stream-ordered: after the build
    if (rc) { matrix_free_on(m, stream); return rc; }
    *out = m;
    return GSOFA_OK;
}

int gsofa::host::matrix_alloc(gsofa_ctx* ctx, cudaStream_t stream, int32_t n, int64_t real,
                              int64_t padded, int nplanes, gsofa_matrix** out) {
    *out = nullptr;
    gsofa_matrix* m = new (std::nothrow) gsofa_matrix();
    if (!m) return set_err(ctx, GSOFA_ERR_OOM_BUDGET, "host allocation failed");
    m->ctx = ctx;
    m->n = n;
    m->nnz = real;
    m->nplanes = nplanes;
    const size_t N1 = (size_t)n + 1;
    const size_t PA = (size_t)std::max<int64_t>(padded, 4);
    const size_t PT = (size_t)std::max<int64_t>(real + 3ll * n, 4);  // bound for A^T
    const size_t NW = (size_t)(((int64_t)n + 31) >> 5) + 1;
    size_t total = align256(4 * N1) * 2 + align256(4 * PA) + align256(4 * PT) + align256(4 * NW) +
                   align256(4 * NW * (size_t)std::max(nplanes, 1)) + 256;
    void* blk = nullptr;
    int rc = dev_alloc_on(ctx, total, &blk, stream);
    if (rc) { delete m; return rc; }
    m->bytes = total;
    char* b = reinterpret_cast<char*>(blk);
    m->rowptr = reinterpret_cast<int32_t*>(b);
    m->trowptr = reinterpret_cast<int32_t*>(b + align256(4 * N1));
    m->col = reinterpret_cast<int32_t*>(b + 2 * align256(4 * N1));
    m->tcol = reinterpret_cast<int32_t*>(b + 2 * align256(4 * N1) + align256(4 * PA));
    m->wdeg = reinterpret_cast<int32_t*>(b + 2 * align256(4 * N1) + align256(4 * PA) +
                                         align256(4 * PT));
    m->dplanes = reinterpret_cast<uint32_t*>(b + 2 * align256(4 * N1) + align256(4 * PA) +
                                             align256(4 * PT) + align256(4 * NW));
    m->asym = reinterpret_cast<int32_t*>(b + total - 256);
    *out = m;
    return GSOFA_OK;
}

void gsofa::host::matrix_free_on(gsofa_matrix* m, cudaStream_t stream) {
    if (!m) return;
    dev_free_on(m->ctx, m->rowptr, m->bytes, stream);
    delete m;
}

int gsofa::host::matrix_build(gsofa_ctx* ctx, cudaStream_t stream, int32_t* dstatus,
                              gsofa_matrix* m, int64_t nnz_in, const int32_t* dbeg,
                              const int32_t* dcol_in, int check_symmetry,
                              int check_dup) {
    const int32_t n = m->n;
    const size_t N1 = (size_t)n + 1;
    size_t scan_bytes = canonicalize_scan_bytes(n);
    const size_t stage = align256(4 * N1) * 3 + align256(scan_bytes) + 256;
    void* sblk = nullptr;
    int rc = dev_alloc_on(ctx, stage, &sblk, stream);
    if (rc) return rc;
    char* s = reinterpret_cast<char*>(sblk);
    int32_t* tcount = reinterpret_cast<int32_t*>(s);
    s += align256(4 * N1);
    int32_t* tfill = reinterpret_cast<int32_t*>(s);
    s += align256(4 * N1);
    int32_t* tpad = reinterpret_cast<int32_t*>(s);
    s += align256(4 * N1);
    void* scan_tmp = s;
    cudaError_t e = cudaSuccess;
    if (n == 0) e = cudaMemsetAsync(m->trowptr, 0, 4, stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(tcount, 0, 4 * N1, stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(tfill, 0, 4 * N1, stream);
    if (e == cudaSuccess)
        e = launch_canonicalize(n, nnz_in, dbeg, dcol_in, m->rowptr, m->col, tcount, tpad,
                                m->trowptr, m->tcol, tfill, m->wdeg, m->dplanes, m->nplanes,
                                m->asym, check_symmetry, check_dup, scan_tmp, scan_bytes, dstatus, stream);
    dev_free_on(ctx, sblk, stage, stream);  // stream-ordered: after the build
    return e == cudaSuccess ? GSOFA_OK : cuda_fail(ctx, e, "matrix build");
}

// Small arrays share one wait through pinned staging (three 80 KB arrays: 36 ->
// 16 us); large ones go straight to the caller's pages, which the driver's own
// staging fills faster (46 MB: 2.4 ms, against 3.2 through 16 MB pinned pieces and
// four copying threads).
int gsofa::host::fetch_all(gsofa_ctx* ctx, const Fetch* f, int count) {
    size_t total = 0;
    int missing = 0;  // the arrays before a missing one are still brought
    for (; missing < count && (!f[missing].dst || f[missing].src); missing++)
        if (f[missing].dst) total += f[missing].bytes;
    std::lock_guard<std::recursive_mutex> g(ctx->mu);
    cudaError_t e = cudaSuccess;
    if (total + kFetchStep * (size_t)count <= kStageBytes) {
        const FetchPlan p = plan_fetch(f, missing);
        for (int c = 0; c < p.copies && e == cudaSuccess; c++)
            e = cudaMemcpyAsync(ctx->h_stage + p.copy[c].at, p.copy[c].src, p.copy[c].bytes,
                                cudaMemcpyDeviceToHost, ctx->stream);
        if (e == cudaSuccess && p.copies) e = cudaStreamSynchronize(ctx->stream);
        for (int k = 0; k < missing && e == cudaSuccess; k++)
            if (f[k].dst && f[k].bytes) memcpy(f[k].dst, ctx->h_stage + p.at[k], f[k].bytes);
    } else {
        for (int k = 0; k < missing && e == cudaSuccess; k++)
            if (f[k].dst && f[k].bytes)
                e = cudaMemcpyAsync(f[k].dst, f[k].src, f[k].bytes, cudaMemcpyDeviceToHost, ctx->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    }
    if (e != cudaSuccess) return cuda_fail(ctx, e, "result fetch");
    if (missing < count)
        return set_err(ctx, GSOFA_ERR_ARG, "requested array was not computed (option off)");
    return GSOFA_OK;
}

// ============================================================================
extern "C" {

const char* gsofa_status_string(int s) {
    switch (s) {
        case GSOFA_OK: return "ok";
        case GSOFA_ERR_ARG: return "invalid argument";
        case GSOFA_ERR_IO: return "i/o error";
        case GSOFA_ERR_OOM_BUDGET: return "memory budget exceeded";
        case GSOFA_ERR_TIMEOUT: return "device wait timed out";
        case GSOFA_ERR_OVERFLOW: return "queue bound exceeded";
        case GSOFA_ERR_CUDA: return "cuda error";
        case GSOFA_ERR_UNSUPPORTED: return "unsupported size or option";
        case GSOFA_ERR_BUSY: return "busy";
        default: return "unknown status";
    }
}

int gsofa_opts_default(gsofa_opts* o) {
    if (!o) return GSOFA_ERR_ARG;
    o->max_supernode_size = 128;
    o->threads_per_source = 0;
    o->sources_in_flight = 0;
    o->flags = GSOFA_SUPERNODES | GSOFA_DIGESTS;
    o->bu_alpha = 0;
    o->bu_beta = 0;
    o->heavy_row = 0;
    o->bu_min_source = 0;
    o->chunk_sources = 0;
    o->cached_closures = 0;
    o->chain_wait_us = 0;
    o->reserved = 0;
    return GSOFA_OK;
}

int gsofa_create(int device, size_t budget_bytes, gsofa_ctx** out) {
    if (!out) return GSOFA_ERR_ARG;
    *out = nullptr;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev <= 0) {
        cudaGetLastError();
        return GSOFA_ERR_CUDA;
    }
    if (device < 0 || device >= ndev) return GSOFA_ERR_ARG;
    gsofa_ctx* ctx = new (std::nothrow) gsofa_ctx();
    if (!ctx) return GSOFA_ERR_OOM_BUDGET;
    ctx->device = device;
    auto fail = [&](cudaError_t e) {
        (void)e;
        if (ctx->own_stream) cudaStreamDestroy(ctx->own_stream);
        if (ctx->ev0) cudaEventDestroy(ctx->ev0);
        if (ctx->ev1) cudaEventDestroy(ctx->ev1);
        if (ctx->evt) cudaEventDestroy(ctx->evt);
        if (ctx->side_stream) cudaStreamDestroy(ctx->side_stream);
        if (ctx->fork) cudaEventDestroy(ctx->fork);
        if (ctx->join) cudaEventDestroy(ctx->join);
        if (ctx->h_counters) cudaFreeHost(ctx->h_counters);
        if (ctx->h_fallback) cudaFreeHost(ctx->h_fallback);
        if (ctx->h_stage) cudaFreeHost(ctx->h_stage);
        if (ctx->h_status) cudaFreeHost(ctx->h_status);
        if (ctx->pool) cudaMemPoolDestroy(ctx->pool);
        delete ctx;
        return GSOFA_ERR_CUDA;
    };
    cudaError_t e = cudaSetDevice(device);
    if (e != cudaSuccess) return fail(e);
    cudaDeviceGetAttribute(&ctx->sm_count, cudaDevAttrMultiProcessorCount, device);
    cudaDeviceGetAttribute(&ctx->smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
    cudaDeviceGetAttribute(&ctx->smem_per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, device);
    size_t fr = 0, tot = 0;
    if ((e = cudaMemGetInfo(&fr, &tot)) != cudaSuccess) return fail(e);
    ctx->budget = budget_bytes ? budget_bytes : (size_t)(0.9 * (double)fr);
    if ((e = cudaStreamCreateWithFlags(&ctx->own_stream, cudaStreamNonBlocking)) != cudaSuccess)
        return fail(e);
    ctx->stream = ctx->own_stream;
    if ((e = cudaEventCreate(&ctx->ev0)) != cudaSuccess) return fail(e);
    if ((e = cudaEventCreate(&ctx->ev1)) != cudaSuccess) return fail(e);
    if ((e = cudaEventCreate(&ctx->evt)) != cudaSuccess) return fail(e);
    ctx->label_cluster = label_max_cluster(((size_t)ctx->smem_optin - 2048) & ~(size_t)127);
    if ((e = cudaStreamCreateWithFlags(&ctx->side_stream, cudaStreamNonBlocking)) != cudaSuccess ||
        (e = cudaEventCreateWithFlags(&ctx->fork, cudaEventDisableTiming)) != cudaSuccess ||
        (e = cudaEventCreateWithFlags(&ctx->join, cudaEventDisableTiming)) != cudaSuccess)
        return fail(e);
    if (ensure_pinned(ctx, 1) != GSOFA_OK) return fail(cudaErrorMemoryAllocation);
    if ((e = cudaMallocHost((void**)&ctx->h_stage, kStageBytes)) != cudaSuccess) return fail(e);
    if ((e = cudaMallocHost((void**)&ctx->h_status, 64)) != cudaSuccess) return fail(e);
    cudaMemPoolProps props{};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = device;
    if ((e = cudaMemPoolCreate(&ctx->pool, &props)) != cudaSuccess) return fail(e);
    uint64_t thr = UINT64_MAX;
    cudaMemPoolSetAttribute(ctx->pool, cudaMemPoolAttrReleaseThreshold, &thr);
    if (dev_alloc(ctx, 256, &ctx->small) != GSOFA_OK) return fail(cudaErrorMemoryAllocation);
    *out = ctx;
    return GSOFA_OK;
}

int gsofa_destroy(gsofa_ctx* ctx) {
    if (!ctx) return GSOFA_ERR_ARG;
    {
        std::lock_guard<std::recursive_mutex> g(ctx->mu);
        cudaSetDevice(ctx->device);
        dev_free(ctx, ctx->queue, ctx->queue_bytes);
        dev_free(ctx, ctx->gbitmap, ctx->gbitmap_bytes);
        dev_free(ctx, ctx->gprev, ctx->gprev_bytes);
        dev_free(ctx, ctx->scan_tmp, ctx->scan_tmp_bytes);
        dev_free(ctx, ctx->hub_ws, ctx->hub_ws_bytes);
        dev_free(ctx, ctx->desc, ctx->desc_bytes);
        dev_free(ctx, ctx->small, 256);
        cudaStreamSynchronize(ctx->stream);
        cudaStreamSynchronize(ctx->own_stream);
        cudaStreamDestroy(ctx->own_stream);
        cudaEventDestroy(ctx->ev0);
        cudaEventDestroy(ctx->ev1);
        cudaEventDestroy(ctx->evt);
        cudaStreamDestroy(ctx->side_stream);
        cudaEventDestroy(ctx->fork);
        cudaEventDestroy(ctx->join);
        cudaFreeHost(ctx->h_counters);
        cudaFreeHost(ctx->h_fallback);
        cudaFreeHost(ctx->h_stage);
        cudaFreeHost(ctx->h_status);
        cudaMemPoolDestroy(ctx->pool);
    }
    delete ctx;
    return GSOFA_OK;
}

const char* gsofa_last_error(const gsofa_ctx* ctx) {
    if (!ctx) return "null context";
    return ctx->err.c_str();
}

int gsofa_set_stream(gsofa_ctx* ctx, void* s) {
    if (!ctx) return GSOFA_ERR_ARG;
    std::lock_guard<std::recursive_mutex> g(ctx->mu);
    // drain work queued on the previous stream before switching
    cudaStreamSynchronize(ctx->stream);
    ctx->stream = s ? reinterpret_cast<cudaStream_t>(s) : ctx->own_stream;
    return GSOFA_OK;
}

int gsofa_memory_used(const gsofa_ctx* ctx, size_t* bytes) {
    if (!ctx || !bytes) return GSOFA_ERR_ARG;
    *bytes = ctx->used;
    return GSOFA_OK;
}

int gsofa_load_csr(gsofa_ctx* ctx, int32_t n, int64_t nnz, const int32_t* row_begin,
                   const int32_t* row_end, const int32_t* col, gsofa_matrix** out) {
    if (!ctx || !out) return GSOFA_ERR_ARG;
    *out = nullptr;
    std::lock_guard<std::recursive_mutex> g(ctx->mu);
    if (cudaSetDevice(ctx->device) != cudaSuccess) return set_err(ctx, GSOFA_ERR_CUDA, "cudaSetDevice");
    unsigned long long* wc = nullptr;
    int32_t* dstatus = work_counter_status(ctx, &wc);
    CK(cudaMemsetAsync(ctx->small, 0, 128, ctx->stream));
    gsofa_matrix* m = nullptr;
    int rc = ingest_csr(ctx, ctx->stream, dstatus, n, nnz, row_begin, row_end, col, &m);
    if (rc) return rc;
    cudaError_t e = cudaMemcpyAsync(ctx->h_status, dstatus, 4, cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(ctx->h_status + 1, m->asym, 8, cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    if (e == cudaSuccess) {
        m->host_sym = n > 0 && ctx->h_status[1] == 0;
        m->host_dup = n > 0 && ctx->h_status[2] != 0;
    }
    rc = e != cudaSuccess ? cuda_fail(ctx, e, "load") : check_status(ctx);
    if (rc) {
        dev_free(ctx, m->rowptr, m->bytes);
        delete m;
        return rc;
    }
    *out = m;
    return GSOFA_OK;
}

int gsofa_load_csr_files(gsofa_ctx* ctx, const char* beg_file, const char* end_file,
                         const char* csr_file, gsofa_matrix** out) {
    if (!ctx || !out || !beg_file || !end_file || !csr_file) return GSOFA_ERR_ARG;
    int32_t n = 0;
    int64_t E = 0;
    std::vector<int32_t> beg, end, col;
    int rc = parse_dat_files(ctx, beg_file, end_file, csr_file, &n, &E, &beg, &end, &col);
    if (rc) return rc;
    return gsofa_load_csr(ctx, n, E, beg.data(), end.data(), col.data(), out);
}

int gsofa_matrix_info(const gsofa_matrix* m, int32_t* n, int64_t* nnz) {
    if (!m) return GSOFA_ERR_ARG;
    if (n) *n = m->n;
    if (nnz) *nnz = m->nnz;
    return GSOFA_OK;
}

int gsofa_matrix_destroy(gsofa_matrix* m) {
    if (!m) return GSOFA_ERR_ARG;
    {
        std::lock_guard<std::recursive_mutex> g(m->ctx->mu);
        dev_free(m->ctx, m->rowptr, m->bytes);
    }
    delete m;
    return GSOFA_OK;
}

int gsofa_factor_batch(gsofa_ctx* ctx, const gsofa_matrix* const* mats, int32_t count,
                       const gsofa_opts* opts, gsofa_result** results) {
    if (!ctx || count < 0 || (count > 0 && (!mats || !results))) return GSOFA_ERR_ARG;
    std::lock_guard<std::recursive_mutex> g(ctx->mu);
    gsofa_opts o;
    if (opts) o = *opts; else gsofa_opts_default(&o);
    int rc = validate_opts(ctx, &o);
    if (rc) return rc;
    for (int32_t i = 0; i < count; i++) {
        results[i] = nullptr;
        if (!mats[i] || mats[i]->ctx != ctx)
            return set_err(ctx, GSOFA_ERR_ARG, "matrix %d is null or from another context", i);
    }
    if (cudaSetDevice(ctx->device) != cudaSuccess) return set_err(ctx, GSOFA_ERR_CUDA, "cudaSetDevice");
    std::vector<gsofa_result*> res((size_t)count, nullptr);
    for (int32_t i = 0; i < count; i++) {
        rc = result_alloc(ctx, mats[i]->n, o.flags, o.max_supernode_size, &res[i]);
        if (rc) {
            for (auto* r : res) result_free(r);
            return rc;
        }
    }
    rc = run_factor(ctx, mats, count, &o, res.data());
    if (rc) {
        for (auto* r : res) result_free(r);
        return rc;
    }
    for (int32_t i = 0; i < count; i++) results[i] = res[i];
    return GSOFA_OK;
}

static gsofa_opts base_without_l_rows(gsofa_opts o) {
    o.flags &= ~(uint32_t)GSOFA_L_ROW_STATS;
    return o;
}

// Times candidate launch shapes on an evenly spread sample of the matrix's
// work items (large matrices) or on the whole matrix (small ones) and keeps
// the fastest.  The candidates differ only in speed: every setting gives the
// same results.  Choices are cached per size class in the context.
// Coordinate descent over the launch shape, each candidate timed on the device
// as one call over all `count` matrices: CTA size and chunk where the chain or
// traverse_kernel counts any of them (in a list with both, one choice for both),
// and closure ring and warp-walked row threshold where traverse_kernel does.  The
// hubs' launches have no shape to choose.  Writes the best into *opts.
static int autotune_impl(gsofa_ctx* ctx, const gsofa_matrix* const* mats, int32_t count,
                         gsofa_opts* opts) {
    int rc = GSOFA_OK;
    int32_t nmax = 0;
    long long total_sources = 0;
    if (cudaSetDevice(ctx->device) != cudaSuccess) return set_err(ctx, GSOFA_ERR_CUDA, "cudaSetDevice");
    for (int32_t i = 0; i < count; i++) {
        nmax = std::max(nmax, mats[i]->n);
        total_sources += chunk_weight(ctx, mats[i]);
    }
    gsofa_opts base = *opts;
    base.flags &= ~(uint32_t)(GSOFA_SUPERNODES | GSOFA_PATTERN);
    if (chain_runs(*opts, mats, count) || !chain_runs(base_without_l_rows(*opts), mats, count))
        base.flags &= ~(uint32_t)GSOFA_L_ROW_STATS;  // else they decide which kernel counts
    const bool chain = chain_runs(base, mats, count);
    // reference timing with the defaults picks the sampling rate
    std::vector<gsofa_result*> rr((size_t)count, nullptr);
    auto free_all = [&]() {
        for (gsofa_result* x : rr) result_free(x);
    };
    for (int32_t i = 0; i < count; i++) {
        rc = result_alloc(ctx, mats[i]->n, base.flags, base.max_supernode_size, &rr[(size_t)i]);
        if (rc) { free_all(); return rc; }
    }
    rc = run_factor(ctx, mats, count, &base, rr.data());
    if (rc) { free_all(); return rc; }
    const bool walked = ctx->walked > 0;
    const double full_ms = rr[0]->counts.ms_traverse;  // the launch's time
    // Full runs while they are short; above 2 s time every stride-th work
    // item, keeping at least 16 items per CTA so the tail does not dominate.
    long long stride = 1;
    if (full_ms > 2000.0) {
        LaunchCfg c0;
        if (plan_launch(ctx, nmax, &base, &c0) == GSOFA_OK) {
            const long long items = total_sources / 16 + 2ll * count;
            stride = (long long)(full_ms / 1000.0);
            while (stride > 1 && items / stride < 16ll * c0.grid) stride--;
        }
    }
    auto time_opts = [&](const gsofa_opts& p, double* ms) -> int {
        LaunchCfg c;
        if (plan_launch(ctx, nmax, &p, &c) != GSOFA_OK) {
            ctx->err.clear();
            *ms = 1e300;
            return GSOFA_OK;
        }
        int e = run_factor(ctx, mats, count, &p, rr.data(), stride);
        *ms = e ? 1e300 : rr[0]->counts.ms_traverse;
        if (e) {
            const std::string prev = ctx->err;
            set_err(ctx, e, "%s; timing threads %d, ring %d, chunk %d, heavy row %d", prev.c_str(),
                    c.block, p.cached_closures, p.chunk_sources, p.heavy_row);
        }
        return e;
    };
    // coordinate descent from the defaults: CTA size, closure ring, chunk,
    // warp-walked row threshold
    gsofa_opts best = base;
    double best_ms = 0;
    rc = time_opts(best, &best_ms);
    if (rc) { free_all(); return rc; }
    long long auto_chunk = 64;
    long long chain_sources = 0;
    bool walks = walked;  // some matrix's counting depends on the shape
    {
        LaunchCfg c0;
        if (plan_launch(ctx, nmax, &base, &c0) == GSOFA_OK) {
            best.threads_per_source = c0.block;
            auto_chunk = default_chunk(total_sources, c0.grid);
        }
        for (int32_t i = 0; i < count; i++) {
            if (!chain || method_of(mats[i]) != METHOD_CHAIN) continue;
            walks = true;
            chain_sources += mats[i]->n;
        }
        ChainCfg cc;
        if (chain_sources > 0 &&
            plan_chain(ctx, std::max(nmax, 1), chain_sources, &base, &cc) == GSOFA_OK) {
            best.threads_per_source = cc.block;
            auto_chunk = chain_chunk(base, chain_sources, nmax, cc.grid);
            best.chunk_sources = (int32_t)auto_chunk;
        }
        ctx->err.clear();
    }
    const int tps_c[] = {128, 256, 512, 1024};
    for (int tps : tps_c) {
        if (tps == best.threads_per_source || !walks) continue;
        gsofa_opts p = best;
        p.threads_per_source = tps;
        double ms;
        if ((rc = time_opts(p, &ms))) { free_all(); return rc; }
        if (ms < best_ms) { best_ms = ms; best = p; }
    }
    const int ring_c[] = {1, 8, 32, 64};
    const int ring_now = best.cached_closures > 0 ? best.cached_closures : kDefaultRing;
    best.cached_closures = ring_now;
    for (int ring : ring_c) {
        if (ring == ring_now || !walked) continue;
        gsofa_opts p = best;
        p.cached_closures = ring;
        double ms;
        if ((rc = time_opts(p, &ms))) { free_all(); return rc; }
        if (ms < best_ms) { best_ms = ms; best = p; }
    }
    {
        LaunchCfg c;
        if (chain_sources == 0 && plan_launch(ctx, nmax, &best, &c) == GSOFA_OK)
            auto_chunk = default_chunk(total_sources, c.grid);
        ctx->err.clear();
        if (best.chunk_sources <= 0) best.chunk_sources = (int32_t)auto_chunk;
        const long long cands[] = {auto_chunk / 8, auto_chunk / 4, auto_chunk / 2, auto_chunk * 2};
        for (long long ch : cands) {
            if (ch < 16 || ch > 1024 || ch == best.chunk_sources || !walks) continue;
            gsofa_opts p = best;
            p.chunk_sources = (int32_t)ch;
            double ms;
            if ((rc = time_opts(p, &ms))) { free_all(); return rc; }
            if (ms < best_ms) { best_ms = ms; best = p; }
        }
    }
    // rows longer than this are walked by a whole warp
    const int heavy_now = best.heavy_row > 0 ? best.heavy_row : kDefaultHeavyRow;
    best.heavy_row = heavy_now;
    for (int hr : {32, 64}) {
        if (hr == heavy_now || !walked) continue;
        gsofa_opts p = best;
        p.heavy_row = hr;
        double ms;
        if ((rc = time_opts(p, &ms))) { free_all(); return rc; }
        if (ms < best_ms) { best_ms = ms; best = p; }
    }
    (void)best_ms;
    free_all();
    opts->threads_per_source = best.threads_per_source;
    opts->chunk_sources = best.chunk_sources;
    opts->cached_closures = best.cached_closures;
    opts->heavy_row = best.heavy_row;
    return GSOFA_OK;
}

int gsofa_autotune(gsofa_ctx* ctx, const gsofa_matrix* mat, gsofa_opts* opts) {
    if (!ctx || !mat || !opts || mat->ctx != ctx) return GSOFA_ERR_ARG;
    std::lock_guard<std::recursive_mutex> g(ctx->mu);
    int rc = validate_opts(ctx, opts);
    if (rc) return rc;
    if (mat->n <= 0) return GSOFA_OK;
    int lg = 0;
    while ((1ll << (lg + 1)) <= (long long)mat->n) lg++;
    const int deg = (int)((mat->nnz + mat->n / 2) / mat->n);
    // locality: matrices of one size but different orderings want different
    // shapes (a renumbered grid is not its banded original)
    unsigned long long* dsum = reinterpret_cast<unsigned long long*>(
        reinterpret_cast<char*>(ctx->small) + 96);
    unsigned long long hsum = 0;
    cudaError_t ce = cudaMemsetAsync(dsum, 0, 8, ctx->stream);
    if (ce == cudaSuccess) ce = launch_index_distance(mat->n, mat->rowptr, mat->col, dsum, ctx->stream);
    if (ce == cudaSuccess) ce = cudaMemcpyAsync(&hsum, dsum, 8, cudaMemcpyDeviceToHost, ctx->stream);
    if (ce == cudaSuccess) ce = cudaStreamSynchronize(ctx->stream);
    if (ce != cudaSuccess) return cuda_fail(ctx, ce, "autotune locality");
    const double rel = mat->nnz > 0 ? (double)hsum / (double)mat->nnz / (double)mat->n : 0.0;
    const int loc = rel > 1e-9 ? std::max(-60, (int)std::floor(2.0 * std::log2(rel))) : -61;
    // and so do the kernels that may count them
    chunk_weight(ctx, mat);
    const gsofa_matrix* const mats[1] = {mat};
    const std::tuple<int, int, int, int> key(lg, deg, loc, chain_runs(*opts, mats, 1) ? method_of(mat) : -1);
    auto it = ctx->tuned.find(key);
    if (it != ctx->tuned.end()) {
        opts->threads_per_source = it->second.threads_per_source;
        opts->chunk_sources = it->second.chunk_sources;
        opts->cached_closures = it->second.cached_closures;
        opts->heavy_row = it->second.heavy_row;
        return GSOFA_OK;
    }
    rc = autotune_impl(ctx, mats, 1, opts);
    if (rc == GSOFA_OK) ctx->tuned[key] = *opts;
    return rc;
}

int gsofa_autotune_batch(gsofa_ctx* ctx, const gsofa_matrix* const* mats, int32_t count,
                         gsofa_opts* opts) {
    if (!ctx || !opts || count < 0 || (count > 0 && !mats)) return GSOFA_ERR_ARG;
    for (int32_t i = 0; i < count; i++)
        if (!mats[i] || mats[i]->ctx != ctx) return GSOFA_ERR_ARG;
    std::lock_guard<std::recursive_mutex> g(ctx->mu);
    int rc = validate_opts(ctx, opts);
    if (rc) return rc;
    bool any = false;
    for (int32_t i = 0; i < count; i++) any |= mats[i]->n > 0;
    if (!any) return GSOFA_OK;
    return autotune_impl(ctx, mats, count, opts);
}

int gsofa_factor_symbolic(gsofa_ctx* ctx, const gsofa_matrix* mat, const gsofa_opts* opts,
                          gsofa_result** out) {
    if (!out) return GSOFA_ERR_ARG;
    return gsofa_factor_batch(ctx, &mat, 1, opts, out);
}

static void batch_free(gsofa_batch* b) {
    if (!b) return;
    gsofa_ctx* ctx = b->ctx;
    if (ctx) {
        std::lock_guard<std::recursive_mutex> g(ctx->mu);
        cudaSetDevice(ctx->device);
        if (b->exec) cudaGraphExecDestroy(b->exec);
        if (b->graph) cudaGraphDestroy(b->graph);
        for (gsofa_result* r : b->res) {
            if (!r) continue;
            r->batch_owned = false;
            result_free(r);
        }
        dev_free(ctx, b->ws, b->ws_bytes);
        cudaStreamSynchronize(ctx->stream);
        if (b->h_counters) cudaFreeHost(b->h_counters);
        if (b->h_status) cudaFreeHost(b->h_status);
        if (b->e0) cudaEventDestroy(b->e0);
        if (b->et) cudaEventDestroy(b->et);
        if (b->e1) cudaEventDestroy(b->e1);
    }
    delete b;
}

// counting: by the counting traversals where chain_runs, else by traverse_kernel.
static int batch_create_with(gsofa_ctx* ctx, const gsofa_matrix* const* mats, int32_t count,
                             const gsofa_opts& o, bool counting, gsofa_batch** out) {
    int rc = GSOFA_OK;
    int32_t nmax = 1;
    long long weight = 0;
    for (int32_t i = 0; i < count; i++) {
        nmax = std::max(nmax, mats[i]->n);
        weight += chunk_weight(ctx, mats[i]);
    }
    gsofa_batch* b = new (std::nothrow) gsofa_batch();
    if (!b) return set_err(ctx, GSOFA_ERR_OOM_BUDGET, "host allocation failed");
    b->ctx = ctx;
    b->count = count;
    b->opts = o;
    b->res.assign((size_t)count, nullptr);
    auto fail = [&](int code) {
        batch_free(b);
        return code;
    };
    for (int32_t i = 0; i < count; i++) {
        rc = result_alloc(ctx, mats[i]->n, o.flags, o.max_supernode_size, &b->res[(size_t)i]);
        if (rc) return fail(rc);
        b->res[(size_t)i]->batch_owned = true;
    }
    // (per-row L statistics could not be made again inside the captured launch)
    const bool chain = counting && !(o.flags & GSOFA_L_ROW_STATS) && chain_runs(o, mats, count);
    ChainCfg ccfg;
    LaunchCfg cfg;
    // the chain's shape for the symmetric matrices, and traverse_kernel's for
    // those that the hubs' launch may leave it
    long long chain_sources = 0, left_weight = 0;
    int32_t chain_nmax = 1, left_nmax = 1;
    for (int32_t i = 0; i < count; i++) {
        const bool mine = method_of(mats[i]) == METHOD_CHAIN;
        if (mine) chain_sources += mats[i]->n;
        else left_weight += chunk_weight(ctx, mats[i]);
        (mine ? chain_nmax : left_nmax) = std::max(mine ? chain_nmax : left_nmax, mats[i]->n);
    }
    if (chain) rc = plan_chain(ctx, chain_nmax, chain_sources, &o, &ccfg);
    if (!rc) rc = plan_launch(ctx, chain ? left_nmax : nmax, &o, &cfg);
    if (rc) return fail(rc);
    const long long walk_chunk =
        o.chunk_sources > 0 ? o.chunk_sources : default_chunk(chain ? left_weight : weight, cfg.grid);
    const long long chunk = chain ? chain_chunk(o, chain_sources, chain_nmax, ccfg.grid) : walk_chunk;
    const long long per_chunk = chain ? 1 : 2;  // work items
    const bool merge = !(o.flags & GSOFA_NO_MERGE);
    int ring = o.cached_closures > 0 ? o.cached_closures : kDefaultRing;
    if (ring > kMaxRing) ring = kMaxRing;
    while (ring & (ring - 1)) ring &= ring - 1;
    // descriptors, segment prefix, counters, workspace: one private block
    std::vector<MatDesc> descs((size_t)count);
    std::vector<long long> seg((size_t)count + 1, 0);
    long long base = 0;
    const std::vector<int32_t> order = batch_order(mats, count);  // largest first
    for (int32_t k = 0; k < count; k++) {
        const int32_t i = order[(size_t)k];
        descs[(size_t)k] = make_desc(mats[i], b->res[(size_t)i], base);
        base += per_chunk * ((mats[i]->n + chunk - 1) / chunk);
        seg[(size_t)k + 1] = seg[(size_t)k] + supernode_segment_count(mats[i]->n, o.max_supernode_size);
    }
    b->items = base;
    HubLaunch HL{};
    HubCfg hcfg;
    size_t sz_hub = 0;
    bool hub = false;
    long long top_items = 0, left_items = 0;
    std::vector<MatDesc> left;  // of traverse_kernel's launch beside the chain
    if (chain) {
        long long items = 0;
        for (int32_t k = 0; k < count; k++) {
            MatDesc& d = descs[(size_t)k];
            const gsofa_matrix* m = mats[order[(size_t)k]];
            d.method = method_of(m);
            d.item_base = items;
            d.top_base = top_items;
            if (d.method == METHOD_CHAIN) {
                d.top_items = chain_top_items(o, m->n, chunk);
                top_items += d.top_items;
                items += (m->n + chunk - 1) / chunk - d.top_items;
            } else if (m->n > 0) {
                left_items += 2 * ((m->n + walk_chunk - 1) / walk_chunk);
            }
        }
        b->items = items;
        cfg.grid = (int)std::min<long long>(cfg.grid, left_items);
    }
    const size_t sz_small = 256;
    const size_t sz_desc = align256(sizeof(MatDesc) * (size_t)count) * (left_items ? 2 : 1);
    const size_t sz_seg = align256(sizeof(long long) * ((size_t)count + 1));
    const size_t sz_cnt = align256(8ull * CNT_SLOTS * (size_t)count);
    const size_t walk_q = (size_t)cfg.grid * (size_t)(chain ? left_nmax : nmax) * 4;
    const size_t walk_gbm = cfg.smem_bitmap ? 0 : (size_t)cfg.grid * (size_t)cfg.words * 4;
    const size_t sz_q =
        align256(chain ? std::max(chain_queue_bytes(ctx, ccfg, chain_nmax, top_items > 0), walk_q) : walk_q);
    const size_t sz_ring = merge ? align256((size_t)cfg.grid * (size_t)ring * (size_t)cfg.words * 4) : 0;
    const size_t sz_gbm =
        align256(chain ? std::max(chain_gbm_bytes(ctx, ccfg, top_items > 0), walk_gbm) : walk_gbm);
    b->ws_bytes = sz_small + sz_desc + sz_seg + sz_cnt + sz_q + sz_ring + sz_gbm;
    const size_t taken = ctx->used - std::min(ctx->used, kept_workspace(ctx)) + b->ws_bytes;
    const size_t room = ctx->budget > taken ? ctx->budget - taken : 0;
    if (chain) hub = plan_hub(ctx, &descs, o, nullptr, &sz_hub, room, &HL, &hcfg);
    b->ws_bytes += sz_hub;
    rc = dev_alloc(ctx, b->ws_bytes, &b->ws);
    if (rc) return fail(rc);
    char* p = reinterpret_cast<char*>(b->ws);
    unsigned long long* wc = reinterpret_cast<unsigned long long*>(p);
    int32_t* dstatus = reinterpret_cast<int32_t*>(p + 64);
    p += sz_small;
    MatDesc* ddesc = reinterpret_cast<MatDesc*>(p);
    MatDesc* dleft = reinterpret_cast<MatDesc*>(p + align256(sizeof(MatDesc) * (size_t)count));
    p += sz_desc;
    long long* dseg = reinterpret_cast<long long*>(p);
    p += sz_seg;
    unsigned long long* dcnt = reinterpret_cast<unsigned long long*>(p);
    p += sz_cnt;
    int32_t* dq = reinterpret_cast<int32_t*>(p);
    p += sz_q;
    uint32_t* dring = sz_ring ? reinterpret_cast<uint32_t*>(p) : nullptr;
    p += sz_ring;
    uint32_t* dgbm = sz_gbm ? reinterpret_cast<uint32_t*>(p) : nullptr;
    p += sz_gbm;
    if (hub) {
        plan_hub(ctx, &descs, o, p, &sz_hub, room, &HL, &hcfg);
        HL.mats = ddesc;
        HL.status = dstatus;
    }
    for (int32_t k = 0; k < count; k++)  // matrix i's counters at slot i, whatever its launch order
        descs[(size_t)k].counters = dcnt + (size_t)order[(size_t)k] * CNT_SLOTS;
    long long left_base = 0;
    for (int32_t k = 0; k < count && left_items; k++) {
        MatDesc d = descs[(size_t)k];
        if (d.method == METHOD_CHAIN || d.n <= 0) continue;
        d.item_base = left_base;
        left_base += 2 * ((d.n + walk_chunk - 1) / walk_chunk);
        d.only_if = d.method == METHOD_WALK ? nullptr : HL.fallback + k;
        left.push_back(d);
    }
    cudaError_t e;
    if ((e = cudaMemcpyAsync(ddesc, descs.data(), sizeof(MatDesc) * (size_t)count,
                             cudaMemcpyHostToDevice, ctx->stream)) != cudaSuccess ||
        (!left.empty() && (e = cudaMemcpyAsync(dleft, left.data(), sizeof(MatDesc) * left.size(),
                                               cudaMemcpyHostToDevice, ctx->stream)) != cudaSuccess) ||
        (e = cudaMemcpyAsync(dseg, seg.data(), sizeof(long long) * ((size_t)count + 1),
                             cudaMemcpyHostToDevice, ctx->stream)) != cudaSuccess ||
        (e = cudaStreamSynchronize(ctx->stream)) != cudaSuccess ||
        (e = cudaMallocHost((void**)&b->h_counters, 8ull * CNT_SLOTS * (size_t)count)) != cudaSuccess ||
        (e = cudaMallocHost((void**)&b->h_status, 64)) != cudaSuccess ||
        (e = cudaEventCreate(&b->e0)) != cudaSuccess || (e = cudaEventCreate(&b->et)) != cudaSuccess ||
        (e = cudaEventCreate(&b->e1)) != cudaSuccess)
        return fail(cuda_fail(ctx, e, "batch set-up"));

    TraverseLaunch L{};
    L.mats = chain ? dleft : ddesc;
    L.nmats = chain ? (int32_t)left.size() : count;
    L.total_items = chain ? left_items : b->items;
    L.work_counter = chain ? wc + 2 : wc;
    L.queue = dq;
    L.queue_stride = chain ? left_nmax : nmax;
    L.gbitmap = dgbm;
    L.bitmap_words = cfg.words;
    L.status = dstatus;
    L.pattern_pass = 0;
    L.bu_alpha = o.bu_alpha > 0 ? o.bu_alpha : (o.bu_alpha < 0 ? 0 : kDefaultBuAlpha);
    L.bu_beta = o.bu_beta > 0 ? o.bu_beta : kDefaultBuBeta;
    L.bu_min_src = o.bu_min_source > 0 ? o.bu_min_source : kBuMinSource;
    L.heavy_len = o.heavy_row > 0 ? ((o.heavy_row + 3) & ~3) : kDefaultHeavyRow;
    L.gprev = dring;
    L.chunk = (int)walk_chunk;
    L.merge = merge ? 1 : 0;
    L.chain = merge && !(o.flags & GSOFA_NO_CHAIN) ? 1 : 0;
    L.chain_wait_ns = chain_wait_ns(o);
    L.ring = ring;
    L.sample_stride = 1;
    ChainLaunch CL{};
    CL.mats = ddesc;
    CL.nmats = count;
    CL.total_items = b->items;
    CL.work_counter = wc;
    CL.queue = dq;
    CL.gbm = dgbm;
    CL.chunk = (int)chunk;
    CL.sample_stride = 1;
    CL.status = dstatus;
    if (chain) fill_chain_launch(&CL, ccfg, o, chain_nmax);

    // capture: reset -> traversal -> supernodes -> read-back
    struct Fork {  // the hubs' branch: of use during the capture alone
        cudaStream_t stream = nullptr;
        cudaEvent_t fork = nullptr, join = nullptr;
        ~Fork() {
            if (stream) cudaStreamDestroy(stream);
            if (fork) cudaEventDestroy(fork);
            if (join) cudaEventDestroy(join);
        }
    } hf;
    if (hub && ((e = cudaStreamCreateWithFlags(&hf.stream, cudaStreamNonBlocking)) != cudaSuccess ||
                (e = cudaEventCreateWithFlags(&hf.fork, cudaEventDisableTiming)) != cudaSuccess ||
                (e = cudaEventCreateWithFlags(&hf.join, cudaEventDisableTiming)) != cudaSuccess))
        return fail(cuda_fail(ctx, e, "batch streams"));
    if ((e = cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeRelaxed)) != cudaSuccess)
        return fail(cuda_fail(ctx, e, "cudaStreamBeginCapture"));
    e = cudaMemsetAsync(b->ws, 0, 128, ctx->stream);
    if (e == cudaSuccess) e = launch_batch_reset(ddesc, count, ctx->stream);
    if (e == cudaSuccess && chain) {
        // the two traversals side by side, then what the hubs' launch leaves
        if (hub) {
            e = cudaEventRecord(hf.fork, ctx->stream);
            if (e == cudaSuccess) e = cudaStreamWaitEvent(hf.stream, hf.fork, 0);
            if (e == cudaSuccess) e = launch_hub(HL, hcfg, (o.flags & GSOFA_DIGESTS) != 0, hf.stream);
            if (e == cudaSuccess) e = cudaEventRecord(hf.join, hf.stream);
        }
        if (e == cudaSuccess) e = launch_chain_both(ctx, CL, ccfg, top_items);
        if (e == cudaSuccess && hub) {
            e = cudaStreamWaitEvent(ctx->stream, hf.join, 0);
        }
    }
    if (e == cudaSuccess && L.total_items > 0)
        e = launch_traverse(L, cfg.block, cfg.grid, cfg.smem_bitmap, cfg.smem, ctx->stream);
    if (e == cudaSuccess && (o.flags & GSOFA_SUPERNODES))
        e = launch_supernodes_batch(ddesc, count, o.max_supernode_size, dseg, seg[(size_t)count],
                                    ctx->stream);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(b->h_counters, dcnt, 8ull * CNT_SLOTS * (size_t)count,
                            cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(b->h_status, dstatus, 4, cudaMemcpyDeviceToHost, ctx->stream);
    cudaGraph_t graph = nullptr;
    cudaError_t e2 = cudaStreamEndCapture(ctx->stream, &graph);
    if (e != cudaSuccess || e2 != cudaSuccess) {
        if (graph) cudaGraphDestroy(graph);
        return fail(cuda_fail(ctx, e != cudaSuccess ? e : e2, "batch capture"));
    }
    b->graph = graph;
    if ((e = cudaGraphInstantiate(&b->exec, b->graph, 0)) != cudaSuccess)
        return fail(cuda_fail(ctx, e, "cudaGraphInstantiate"));
    *out = b;
    return GSOFA_OK;
}

int gsofa_batch_create(gsofa_ctx* ctx, const gsofa_matrix* const* mats, int32_t count,
                       const gsofa_opts* opts, gsofa_batch** out) {
    if (!ctx || !out || count <= 0 || !mats) return GSOFA_ERR_ARG;
    *out = nullptr;
    std::lock_guard<std::recursive_mutex> g(ctx->mu);
    gsofa_opts o;
    if (opts) o = *opts; else gsofa_opts_default(&o);
    int rc = validate_opts(ctx, &o);
    if (rc) return rc;
    if (o.flags & GSOFA_PATTERN)
        return set_err(ctx, GSOFA_ERR_UNSUPPORTED, "a captured batch cannot materialise patterns");
    for (int32_t i = 0; i < count; i++)
        if (!mats[i] || mats[i]->ctx != ctx)
            return set_err(ctx, GSOFA_ERR_ARG, "matrix %d is null or from another context", i);
    if (cudaSetDevice(ctx->device) != cudaSuccess) return set_err(ctx, GSOFA_ERR_CUDA, "cudaSetDevice");
    rc = batch_create_with(ctx, mats, count, o, true, out);
    // the counting traversals' workspace does not fit: traverse_kernel's is smaller
    if (rc == GSOFA_ERR_OOM_BUDGET) rc = batch_create_with(ctx, mats, count, o, false, out);
    return rc;
}

int gsofa_batch_run(gsofa_batch* b) {
    if (!b) return GSOFA_ERR_ARG;
    gsofa_ctx* ctx = b->ctx;
    std::lock_guard<std::recursive_mutex> g(ctx->mu);
    if (cudaSetDevice(ctx->device) != cudaSuccess) return set_err(ctx, GSOFA_ERR_CUDA, "cudaSetDevice");
    // events around the graph launch: the whole batch's device time
    CK(cudaEventRecord(b->e0, ctx->stream));
    CK(cudaGraphLaunch(b->exec, ctx->stream));
    CK(cudaEventRecord(b->e1, ctx->stream));
    CK(cudaStreamSynchronize(ctx->stream));
    *ctx->h_status = *b->h_status;
    int rc = check_status(ctx);
    if (rc) return rc;
    float ms = 0.f;
    CK(cudaEventElapsedTime(&ms, b->e0, b->e1));
    for (int32_t i = 0; i < b->count; i++) {
        gsofa_result* r = b->res[(size_t)i];
        const unsigned long long* c = b->h_counters + (size_t)i * CNT_SLOTS;
        gsofa_counts& k = r->counts;
        k.n = r->n;
        k.fill_count = c[CNT_FILLS];
        k.nnz_l = c[CNT_NNZ_L];
        k.nnz_u = c[CNT_NNZ_U];
        k.nnz_lu = c[CNT_NNZ_L] + c[CNT_NNZ_U] + (uint64_t)r->n;
        k.n_supernodes = (b->opts.flags & GSOFA_SUPERNODES) ? (int64_t)c[CNT_NSUP] + 1 : -1;
        k.edges_alg = c[CNT_EDGES_ALG];
        k.vertices_alg = c[CNT_VERTS_ALG];
        k.edges_traversed = c[CNT_EDGES_TRAV];
        k.sources_chained = c[CNT_CHAINED];
        k.ms_device = (double)ms;  // the whole batch (one graph launch)
        k.ms_traverse = (double)ms;
    }
    return GSOFA_OK;
}

int gsofa_batch_result(const gsofa_batch* b, int32_t i, gsofa_result** res) {
    if (!b || !res || i < 0 || i >= b->count) return GSOFA_ERR_ARG;
    *res = b->res[(size_t)i];
    return GSOFA_OK;
}

int gsofa_batch_destroy(gsofa_batch* b) {
    if (!b) return GSOFA_ERR_ARG;
    batch_free(b);
    return GSOFA_OK;
}

int gsofa_result_counts(const gsofa_result* r, gsofa_counts* out) {
    if (!r || !out) return GSOFA_ERR_ARG;
    *out = r->counts;
    return GSOFA_OK;
}

static int fetch(const gsofa_result* r, void* dst, const void* src, size_t bytes) {
    if (dst && !src) return set_err(r->ctx, GSOFA_ERR_ARG, "requested array was not computed (option off)");
    const Fetch f{dst, src, bytes, nullptr};
    return fetch_all(r->ctx, &f, 1);
}

int gsofa_result_row_counts(const gsofa_result* r, int32_t* nnz_u_row, int32_t* nz_row_u,
                            int32_t* nnz_l_col, int32_t* nnz_l_row) {
    if (!r) return GSOFA_ERR_ARG;
    const size_t b = 4 * (size_t)r->n;
    const Fetch f[4] = {{nnz_u_row, r->nnz_u, b, r->arena},
                        {nz_row_u, r->nz_row_u, b, r->arena},
                        {nnz_l_col, r->nnz_lc, b, r->arena},
                        {nnz_l_row, r->nnz_lr, b, r->arena}};
    return fetch_all(r->ctx, f, 4);
}

int gsofa_result_digests(const gsofa_result* r, uint64_t* du, uint64_t* dlc, uint64_t* dlr) {
    if (!r) return GSOFA_ERR_ARG;
    const size_t b = 8 * (size_t)r->n;
    const Fetch f[3] = {{du, r->dig_u, b, r->arena},
                        {dlc, r->dig_lc, b, r->arena},
                        {dlr, r->dig_lr, b, r->arena}};
    return fetch_all(r->ctx, f, 3);
}

int gsofa_result_lmask(const gsofa_result* r, uint32_t* mask4n) {
    if (!r) return GSOFA_ERR_ARG;
    return fetch(r, mask4n, r->lmask, 16 * (size_t)r->n);
}

int gsofa_result_supernodes(const gsofa_result* r, int8_t* flags, int32_t* boundaries, int64_t cap,
                            int64_t* count) {
    if (!r) return GSOFA_ERR_ARG;
    if (!(r->flags & GSOFA_SUPERNODES))
        return set_err(r->ctx, GSOFA_ERR_ARG, "supernode detection was not requested");
    std::vector<int8_t> own(flags ? 0 : (size_t)r->n);
    int8_t* const f = flags ? flags : own.data();
    int rc = fetch(r, f, r->sflags, (size_t)r->n);
    if (rc) return rc;
    int64_t k = 0;
    if (!boundaries) {
        for (int32_t v = 0; v < r->n; v++) k += f[v] != 0;
        if (count) *count = k;
        return GSOFA_OK;
    }
    for (int32_t v = 0; v < r->n; v++) {
        if (f[v]) {
            if (boundaries && k < cap) boundaries[k] = v;
            k++;
        }
    }
    if (count) *count = k;
    return GSOFA_OK;
}

static int fetch_pattern(const gsofa_result* r, const int64_t* dptr, const int32_t* dids,
                         int64_t* ptr, int32_t* ids, int64_t cap) {
    if (!(r->flags & GSOFA_PATTERN) || !dptr)
        return set_err(r->ctx, GSOFA_ERR_ARG, "pattern was not requested (GSOFA_PATTERN)");
    std::vector<int64_t> p((size_t)r->n + 1);
    int rc = fetch(r, p.data(), dptr, 8 * ((size_t)r->n + 1));
    if (rc) return rc;
    if (ptr) memcpy(ptr, p.data(), 8 * ((size_t)r->n + 1));
    if (ids) {
        if (cap < p[(size_t)r->n])
            return set_err(r->ctx, GSOFA_ERR_ARG, "id buffer holds %lld, needs %lld", (long long)cap,
                           (long long)p[(size_t)r->n]);
        if (p[(size_t)r->n] > 0) rc = fetch(r, ids, dids, 4 * (size_t)p[(size_t)r->n]);
    }
    return rc;
}

int gsofa_result_pattern_u(const gsofa_result* r, int64_t* ptr, int32_t* cols, int64_t cap) {
    if (!r) return GSOFA_ERR_ARG;
    return fetch_pattern(r, r->uptr, r->ucols, ptr, cols, cap);
}

int gsofa_result_pattern_l(const gsofa_result* r, int64_t* ptr, int32_t* rows, int64_t cap) {
    if (!r) return GSOFA_ERR_ARG;
    return fetch_pattern(r, r->lptr, r->lrows, ptr, rows, cap);
}

int gsofa_result_destroy(gsofa_result* r) {
    if (!r) return GSOFA_ERR_ARG;
    if (r->batch_owned) return set_err(r->ctx, GSOFA_ERR_ARG, "result belongs to a batch");
    result_free(r);
    return GSOFA_OK;
}

// The reference's two command lines (SOA argc == 11, :2532-2545; SPO argc == 6,
// symbfact.cuh:1557-1571), folded onto one device.
int gsofa_symbfact_min_id(int argc, char** argv, int rank, uint64_t* fill_count, double* time_ms,
                          int32_t* n_supernodes, uint64_t* teps_edges) {
    if (!argv || (argc != 11 && argc != 6)) return GSOFA_ERR_ARG;
    gsofa_opts o;
    gsofa_opts_default(&o);
    size_t budget = 0;
    if (argc == 11) {
        int mss = atoi(argv[5]);
        if (mss <= 0) return GSOFA_ERR_ARG;
        o.max_supernode_size = mss;
    } else {
        double gb = atof(argv[5]);
        if (gb < 0) return GSOFA_ERR_ARG;
        // the reference's pool holds its 6 work arrays; here the budget bounds
        // everything the context allocates (matrix, workspace, results)
        budget = gb > 0 ? (size_t)(gb * 1024.0 * 1024.0 * 1024.0) : 0;
        o.flags &= ~(uint32_t)GSOFA_SUPERNODES;
    }
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev <= 0) return GSOFA_ERR_CUDA;
    gsofa_ctx* ctx = nullptr;
    int rc = gsofa_create(rank % ndev, budget, &ctx);
    if (rc) return rc;
    gsofa_matrix* m = nullptr;
    rc = gsofa_load_csr_files(ctx, argv[1], argv[2], argv[3], &m);
    if (rc) {
        fprintf(stderr, "gsofa: %s\n", gsofa_last_error(ctx));
        gsofa_destroy(ctx);
        return rc;
    }
    gsofa_result* r = nullptr;
    rc = gsofa_factor_symbolic(ctx, m, &o, &r);
    if (rc) {
        fprintf(stderr, "gsofa: %s\n", gsofa_last_error(ctx));
        gsofa_matrix_destroy(m);
        gsofa_destroy(ctx);
        return rc;
    }
    gsofa_counts c;
    gsofa_result_counts(r, &c);
    if (fill_count) *fill_count = c.fill_count;
    if (time_ms) *time_ms = c.ms_device;
    if (n_supernodes) *n_supernodes = (int32_t)c.n_supernodes;
    if (teps_edges) *teps_edges = c.edges_alg;
    gsofa_result_destroy(r);
    gsofa_matrix_destroy(m);
    gsofa_destroy(ctx);
    return GSOFA_OK;
}

}  // extern "C"
