// gsofa_server.cpp -- the serving request loop (continuous batching).
//
// One host thread per server drives:
//   * two persistent traversal kernels, chain_kernel for requests with a
//     symmetric pattern and traverse_kernel for those without one that the hubs'
//     launch leaves (for all of them with the diagnostic options, per-row L
//     statistics, or a budget without room for both workspaces).  Their CTAs
//     claim work items of every published request; a kernel stays on the device
//     while published work is waiting and ends by itself when its CTAs have
//     found nothing to claim for a short while;
//   * a few lanes for the other requests: each the hubs' launch of a plain call
//     (gsofa_hub.cu) on a stream and in a workspace of its own.  The SMs are
//     shared out among the two kernels and the lanes while they have work;
//   * a side stream for everything else: the upload and padded-CSR build of
//     each admitted request, its descriptor, the copy that publishes it (its
//     claim word), and, once the request is reported finished, its
//     supernode detection and the read-back of its totals;
//   * a control stream for the small table the kernels poll (the list of live
//     requests the CTAs pick from, the "exit when idle" and "take no more
//     items" controls): the host keeps the master copy in pinned memory and
//     pushes it whole, synchronously, after each change;
//   * mapped host memory for the kernel's per-slot "request done" flags, its
//     only writes to host memory.  Nothing the kernel polls lives in host
//     memory: hundreds of idle CTAs polling across PCIe would compete with
//     the uploads of the requests they wait for.
//
// Admission is first come, first served: the request at the head of the
// queue is admitted when a slot is free and its footprint (padded CSR of A
// and A^T, staging, result arrays) fits the budget beside the workspace and
// the requests in flight.  A request never waits for the kernel: it joins the
// running launch, and a CTA takes its next item from the live request with
// the fewest unclaimed items, so a small request that arrives behind a large
// one is not queued behind the large one's items.  The kernel leaves four SMs free,
// and the side stream has the higher priority, so uploads and builds run
// beside it.
//
// Nothing here waits on the device without a bound: a CTA's idle polling
// ends after kIdleNs, and the host waits only for streams whose work is
// already queued.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <deque>
#include <memory>
#include <mutex>
#include <new>
#include <string>
#include <thread>
#include <unordered_map>
#include <vector>

#include "gsofa_host.h"

using namespace gsofa;
using namespace gsofa::host;

namespace {

enum ReqRoute { TO_NONE, TO_CHAIN, TO_LANE, TO_WALK };
enum ReqState { R_QUEUED, R_RUNNING, R_FINISHING, R_DONE, R_FAILED };

struct Request {
    uint64_t ticket = 0;
    int32_t n = 0;
    int64_t nnz = 0;
    const int32_t* beg = nullptr;
    const int32_t* end = nullptr;
    const int32_t* col = nullptr;
    int state = R_QUEUED;
    int status = GSOFA_ERR_BUSY;
    int slot = -1;
    long long n_items = 0;
    unsigned long long seq = 0;
    size_t footprint = 0;
    gsofa_matrix* mat = nullptr;
    gsofa_result* res = nullptr;
    bool handed_out = false;
    double t_submit = 0, t_admit = 0, t_publish = 0, t_done = 0;
    bool published = false;  // the claim word copy has executed
    int route = 0;           // TO_*: then, who counts it
};

constexpr int kSlots = 256;
constexpr int kKernelStreams = 8;  // launches of a kernel that may run at once (4: 48 requests 126-182 ms, 8: 114-154)
constexpr int kReserveSms = 4;
constexpr int kLanes = 3;                      // hubs' launches that may run at once
constexpr int kLaneCluster = 4;                // CTAs of a lane's label search at most: its SMs are shared
constexpr size_t kLaneBytes = 64u << 20;       // a lane's workspace for large searches, or that of 296 CTAs
constexpr size_t kAhead = 2ull << 30;          // memory the pool gets before the first request, at most
constexpr double kLaneHoldMs = 1.0;            // the lanes' SMs stay free this long after their last work
constexpr long long kMaxIdlePolls = 1000000;  // a cap far above idle_ns worth of polls
constexpr long long kIdleNs = 300000;         // a CTA with nothing to claim for 0.3 ms exits
constexpr double kTopUpCheckMs = 0.5;         // how often a partial launch is topped up
constexpr double kAdmitSliceMs = 1.0;         // admissions per loop pass stop after this long
constexpr size_t kDefaultBudget = 40ull << 30;
constexpr double kShutdownGraceMs = 120000.0;  // destroy waits this long for queued work

// SMs that serving CTAs use; the rest are the uploads' and builds'.
unsigned serve_sms(const gsofa_ctx* ctx) {
    return ctx->sm_count > kReserveSms ? (unsigned)(ctx->sm_count - kReserveSms) : (unsigned)ctx->sm_count;
}

// A serving kernel's launch shape for requests of up to max_n rows and the
// workspace its CTAs need.
struct ServeShape {
    bool chain = false;
    int block = 0, occ = 0, grid = 0;
    size_t smem = 0;  // dynamic, in all
    long long smem_words = 0;
    int32_t max_n = 0;
    int ring = 0;

    size_t queues() const { return align256((size_t)grid * (size_t)max_n * 4); }
    size_t rings(long long words) const {
        return chain ? 0 : align256((size_t)grid * (size_t)ring * (size_t)words * 4);
    }
    // the chain's two, or one for traverse_kernel where shared memory has no room for it
    size_t bitmaps(long long words) const {
        return chain || words > smem_words ? align256((size_t)grid * (chain ? 2 : 1) * (size_t)words * 4) : 0;
    }
    size_t bytes(long long words) const { return queues() + rings(words) + bitmaps(words); }
};

// One of the two serving kernels: its shape, launches and workspace.
enum : int { E_CHAIN = 0, E_WALK = 1, kEngines = 2 };
struct Engine {
    bool on = false;
    ServeShape shape;
    cudaStream_t ks[kKernelStreams] = {};  // launches (low priority)
    cudaEvent_t kdone[kKernelStreams] = {};
    bool krun[kKernelStreams] = {};
    int32_t kno[kKernelStreams] = {};  // the launch's number
    int32_t launches = 0;
    void* ws = nullptr;
    size_t ws_bytes = 0;
    int32_t* queue = nullptr;
    uint32_t* rings = nullptr;
    uint32_t* gbm = nullptr;
    unsigned int* d_cta_slots = nullptr;
    int* d_alive = nullptr;
    double alive_checked = -1.0;

    int streams() const { return shape.chain ? kKernelStreams : kKernelStreams / 2; }
};

// A hubs' launch for one request, and what it needs.
struct Lane {
    cudaStream_t st = nullptr;
    cudaEvent_t done = nullptr;
    std::shared_ptr<Request> r;  // null: free
    void* ws = nullptr;
    size_t bytes = 0;
    MatDesc* h_desc = nullptr;  // pinned
    int32_t* h_left = nullptr;  // pinned: the launch left the request
};

}  // namespace

struct gsofa_server {
    gsofa_ctx* ctx = nullptr;
    gsofa_opts opts{};
    int32_t max_n = 0;
    size_t budget = 0;
    long long words = 0;
    int ring = 32;
    bool merge = true;
    Engine eng[kEngines];
    Lane lanes[kLanes];
    std::deque<std::shared_ptr<Request>> lane_queue;
    double lanes_until = -1.0;
    cudaStream_t as = nullptr, cs = nullptr, fs = nullptr;
    std::vector<cudaEvent_t> slot_ev;  // per slot: read-back done
    std::vector<cudaEvent_t> pub_ev;   // per slot: claim word written
    // device tables (one block; each kernel has a workspace of its own)
    void* tab = nullptr;
    size_t tab_bytes = 0;
    MatDesc* d_slots = nullptr;
    unsigned long long* d_claim = nullptr;
    unsigned long long* d_items_done = nullptr;
    int32_t* d_slot_status = nullptr;
    unsigned int* d_rr = nullptr;
    int* h_alive = nullptr;  // pinned read-back of an engine's *d_alive
    int32_t* d_route = nullptr;  // per slot
    // pinned, 4 words a slot: the matrix's symmetry and repeated-entry words, the
    // build's status, and ROUTE_WALK to be copied from
    int32_t* h_words = nullptr;
    unsigned long long* d_work = nullptr;
    int32_t* d_status = nullptr;
    // control table: int32 ctrl[8] (ServeLaunch says what they hold), then u64
    // list[kSlots] = (slot << 32) | request number.  Master copy in pinned host
    // memory, pushed whole.
    void* d_ctl = nullptr;
    void* h_ctl = nullptr;
    // mapped host memory
    unsigned long long* h_done = nullptr;
    unsigned long long* d_done = nullptr;
    // pinned staging, per slot
    MatDesc* h_desc = nullptr;
    unsigned long long* h_claim = nullptr;
    unsigned long long* h_cnt = nullptr;
    int32_t* h_sstat = nullptr;
    // uploads of the submitted (pageable) host arrays
    gsofa::host::PinnedStager stager;
    // host state (mu guards everything a caller thread touches)
    std::mutex mu;
    std::condition_variable cv_work, cv_done;
    std::thread th;
    bool shutdown = false;
    uint64_t next_ticket = 1;
    std::deque<std::shared_ptr<Request>> queued;
    std::unordered_map<uint64_t, std::shared_ptr<Request>> tickets;
    std::vector<std::shared_ptr<Request>> slot_req;
    std::vector<int> free_slots;
    // loop-thread state
    unsigned long long seq = 0;
    int nlist = 0;
    bool kernel_running = false;
    bool launch_failed = false;
    bool shed = false;  // the chain's workspace has to make room
    int live = 0;
    // accounting
    size_t fixed = 0, least = 0, in_use = 0, peak = 0;  // least: fixed without the chain's workspace
    gsofa_server_stats st{};
    std::string err;
    std::chrono::steady_clock::time_point t0;
};

namespace {

double now_ms(const gsofa_server* s) {
    return std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - s->t0)
        .count();
}

void server_err(gsofa_server* s, const char* fmt, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof(buf), fmt, ap);
    va_end(ap);
    std::lock_guard<std::mutex> g(s->mu);
    s->err = buf;
}

size_t request_footprint(const gsofa_server* s, int32_t n, int64_t nnz) {
    size_t kept = 0, staging = 0;
    ingest_bytes(n, nnz, &kept, &staging);
    return kept + staging + result_bytes(n, s->opts.flags);
}

// Consecutive sources per work item of traverse_kernel: about four items per CTA for this
// order and grid (requests share the CTAs, so items stay shorter than the
// plain path's), capped so that chunk * n stays near 2^28 -- one item of a
// large request then holds its CTA for a bounded time, not for a large part
// of the request, and a request that arrives meanwhile finds CTAs soon.  The
// cap is no tighter because every item's first source starts cold.
int walk_chunk(const gsofa_server* s, int32_t n) {
    if (s->opts.chunk_sources > 0) return s->opts.chunk_sources;
    long long cap = 512;
    while (cap > 16 && cap * (long long)std::max(n, 1) > (1ll << 28)) cap >>= 1;
    return (int)std::min<long long>(default_chunk(2ll * n, 4 * s->eng[E_WALK].shape.grid), cap);
}

// The chain's: about one item per CTA; an item's first source is searched from
// nothing.
int chain_item(const gsofa_server* s, int32_t n) {
    if (s->opts.chunk_sources > 0) return s->opts.chunk_sources;
    const long long grid = std::max(1, s->eng[E_CHAIN].shape.grid);
    return (int)std::max(8ll, std::min(128ll, ((long long)n + grid - 1) / grid));
}

// Default CTA size of traverse_kernel: the plain path's for the largest order
// served (the widest bitmap then fits in shared memory up to n of about 1.8M).
// The chain's throughput is its CTAs' number, whatever max_n: four of 256 threads
// per SM, or as many as keep one bitmap of max_n in shared memory while that
// takes at most 64 KB (a symmetric pattern's only one: the 64^3 mesh at
// max_n = 300,000 took 11.8 ms with it in global memory); wider ones are in
// global memory.
ServeShape serve_shape(const gsofa_ctx* ctx, const gsofa_server& s, bool chain) {
    const gsofa_opts& o = s.opts;
    ServeShape r;
    r.chain = chain;
    r.max_n = s.max_n;
    r.ring = s.merge ? s.ring : 0;
    r.block = o.threads_per_source > 0 ? o.threads_per_source
              : chain                  ? 256
                                       : std::max(256, default_block(s.max_n, ctx->smem_per_sm));
    // shared-memory bitmap: the widest that keeps the block's full residency
    // (none with the diagnostic GSOFA_FORCE_GLOBAL_BITMAP)
    const int occ_target = 1024 / r.block;
    const size_t fixed = chain ? (chain_sparse_bytes() + 15) & ~(size_t)15 : 0;
    auto occupancy = [&](size_t bytes) {
        return chain ? chain_occupancy(r.block, true, fixed + bytes) : serve_occupancy(r.block, bytes);
    };
    size_t smem = 0;
    if (!(o.flags & GSOFA_FORCE_GLOBAL_BITMAP)) {
        smem = (size_t)std::min(ctx->smem_optin, ctx->smem_per_sm / occ_target - 8 * 1024);
        smem &= ~(size_t)1023;
        while (smem >= 4096 && occupancy(smem) < occ_target) smem -= 1024;
        if (smem < 4096) smem = 0;
        const size_t one = ((size_t)s.words * 4 + 1023) & ~(size_t)1023;
        if (chain && one <= 64 * 1024 && smem < one && occupancy(one) > 0) smem = one;
    }
    if (chain) smem = std::min(smem, ((size_t)s.words * 4 + 1023) & ~(size_t)1023);
    r.occ = occupancy(smem);
    r.smem = fixed + smem;
    r.smem_words = (long long)(smem / 4);
    r.grid = r.occ * std::max(1, ctx->sm_count - kReserveSms);
    if (o.sources_in_flight > 0) r.grid = std::min(r.grid, o.sources_in_flight);
    return r;
}

// Gives a request's device memory back, but for a result that is kept.
void drop_buffers(gsofa_server* s, const std::shared_ptr<Request>& r, bool keep_result = false) {
    gsofa_ctx* ctx = s->ctx;
    std::lock_guard<std::recursive_mutex> g(ctx->mu);
    if (r->mat) {
        dev_free_on(ctx, r->mat->rowptr, r->mat->bytes, s->as);
        delete r->mat;
        r->mat = nullptr;
    }
    if (!keep_result && r->res) {
        dev_free_on(ctx, r->res->arena, r->res->bytes, s->as);
        delete r->res;
        r->res = nullptr;
    }
}

// (with s->mu held)
void release_slot(gsofa_server* s, const std::shared_ptr<Request>& r) {
    if (r->slot >= 0) {
        s->slot_req[(size_t)r->slot].reset();
        s->free_slots.push_back(r->slot);
        r->slot = -1;
        s->live--;
    }
    s->in_use -= std::min(s->in_use, r->footprint);
}

// Marks a request finished (done or failed) and releases its slot and memory.
void finish(gsofa_server* s, const std::shared_ptr<Request>& r, int status) {
    drop_buffers(s, r, status == GSOFA_OK);
    std::lock_guard<std::mutex> g(s->mu);
    release_slot(s, r);
    r->t_done = now_ms(s);
    r->status = status;
    r->state = status == GSOFA_OK ? R_DONE : R_FAILED;
    if (status == GSOFA_OK) s->st.completed++;
    else s->st.failed++;
    s->cv_done.notify_all();
}

constexpr size_t kCtlFlags = 32;
constexpr size_t kCtlBytes = kCtlFlags + 8 * (size_t)kSlots;

int32_t* ctl_flags(gsofa_server* s) { return static_cast<int32_t*>(s->h_ctl); }
unsigned long long* ctl_list(gsofa_server* s) {
    return reinterpret_cast<unsigned long long*>(static_cast<char*>(s->h_ctl) + kCtlFlags);
}

// Copies the control table to the device and waits for the copy (tens of
// microseconds), so the master copy can change again at once.
void push_control(gsofa_server* s) {
    cudaError_t e = cudaMemcpyAsync(s->d_ctl, s->h_ctl, kCtlBytes, cudaMemcpyHostToDevice, s->cs);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s->cs);
    if (e != cudaSuccess) server_err(s, "control table update: %s", cudaGetErrorString(e));
}

// The live-request list.  A CTA that reads a stale, duplicated or half
// copied entry fails the claim word's request-number check.
void list_add(gsofa_server* s, int slot, unsigned long long seq) {
    ctl_list(s)[s->nlist++] = ((unsigned long long)slot << 32) | (seq & 0xffffffffull);
    ctl_flags(s)[2] = s->nlist;
    push_control(s);
}

void list_remove(gsofa_server* s, int slot) {
    unsigned long long* L = ctl_list(s);
    for (int i = 0; i < s->nlist; i++) {
        if ((int)(L[i] >> 32) != slot) continue;
        L[i] = L[s->nlist - 1];
        L[--s->nlist] = ~0ull;
        ctl_flags(s)[2] = s->nlist;
        push_control(s);
        return;
    }
}

void set_control(gsofa_server* s, int which, int32_t value) {
    ctl_flags(s)[which] = value;
    push_control(s);
}

// With nothing in flight and a request waiting for room: the chain's workspace
// goes, and traverse_kernel serves alone from here on.
void shed_chain(gsofa_server* s) {
    Engine& C = s->eng[E_CHAIN];
    set_control(s, 3, C.launches);  // its CTAs find nothing to claim: they leave at once
    set_control(s, 4, s->eng[E_WALK].launches);
    for (Engine& E : s->eng)
        for (int k = 0; k < kKernelStreams; k++) {
            if (E.krun[k]) cudaEventSynchronize(E.kdone[k]);
            E.krun[k] = false;
        }
    {
        std::lock_guard<std::recursive_mutex> g(s->ctx->mu);
        dev_free_on(s->ctx, C.ws, C.ws_bytes, s->as);
    }
    std::lock_guard<std::mutex> g(s->mu);
    s->fixed -= C.ws_bytes;
    s->in_use -= C.ws_bytes;
    C.ws = nullptr;
    C.on = false;
    s->shed = false;
    s->st.grid = s->eng[E_WALK].shape.grid;
    s->st.block = s->eng[E_WALK].shape.block;
}

// Admits the request at the head of the queue if it fits; queues its upload,
// build, table writes and publication on the side stream.
bool admit_one(gsofa_server* s) {
    std::shared_ptr<Request> r;
    int slot = -1;
    bool clear = false;
    {
        std::lock_guard<std::mutex> g(s->mu);
        if (s->queued.empty() || s->free_slots.empty()) return false;
        const bool fits = s->in_use + s->queued.front()->footprint <= s->budget;
        if (!fits || s->shed) {
            if (!s->eng[E_CHAIN].on || s->live > 0) return false;
            clear = true;
        }
    }
    if (clear) shed_chain(s);
    const bool both = s->eng[E_CHAIN].on;
    long long items = 0, walk_items = 0;
    int chunk = 0, walk = 0;
    {
        std::lock_guard<std::mutex> g(s->mu);
        if (s->queued.empty()) return false;
        r = s->queued.front();
        walk = walk_chunk(s, r->n);
        walk_items = 2 * (((long long)r->n + walk - 1) / walk);
        chunk = both ? chain_item(s, r->n) : 1;
        items = both ? ((long long)r->n + chunk - 1) / chunk : walk_items;
        s->queued.pop_front();
        slot = s->free_slots.back();
        s->free_slots.pop_back();
        s->slot_req[(size_t)slot] = r;
        s->live++;
        s->st.max_in_flight = std::max(s->st.max_in_flight, s->live);
        s->in_use += r->footprint;
        s->peak = std::max(s->peak, s->in_use);
        r->slot = slot;
        r->state = R_RUNNING;
        r->t_admit = now_ms(s);
    }
    gsofa_ctx* ctx = s->ctx;
    const uint32_t flags = s->opts.flags & (GSOFA_SUPERNODES | GSOFA_DIGESTS | GSOFA_L_ROW_STATS);
    int rc = GSOFA_OK;
    cudaError_t e = cudaMemsetAsync(s->d_slot_status + slot, 0, 4, s->as);
    if (e == cudaSuccess) e = cudaMemsetAsync(s->d_items_done + slot, 0, 8, s->as);
    if (e != cudaSuccess) rc = GSOFA_ERR_CUDA;
    std::string why;
    {
        std::lock_guard<std::recursive_mutex> g(ctx->mu);
        if (rc == GSOFA_OK)
            rc = ingest_csr(ctx, s->as, s->d_slot_status + slot, r->n, r->nnz, r->beg, r->end,
                            r->col, &r->mat, &s->stager);
        if (rc == GSOFA_OK)
            rc = result_alloc_on(ctx, r->n, flags, s->opts.max_supernode_size, s->as, &r->res);
        if (rc != GSOFA_OK) why = ctx->err;
    }
    if (rc == GSOFA_ERR_OOM_BUDGET && both) {
        // the context has no room: again without the chain's workspace, once the
        // requests in flight are done
        drop_buffers(s, r);
        std::lock_guard<std::mutex> g(s->mu);
        release_slot(s, r);
        r->state = R_QUEUED;
        s->queued.push_front(r);
        s->shed = true;
        return true;
    }
    if (rc != GSOFA_OK) {
        server_err(s, "ticket %llu: %s", (unsigned long long)r->ticket, why.c_str());
        finish(s, r, rc);
        return true;
    }
    r->n_items = items;
    r->seq = ++s->seq;
    r->route = TO_NONE;
    MatDesc d = make_desc(r->mat, r->res, 0);
    d.n_items = items;
    d.walk_items = walk_items;
    d.seq = r->seq;
    d.chunk = chunk;
    d.walk_chunk = walk;
    d.slot = slot;
    s->h_desc[slot] = d;
    s->h_done[slot] = 0ull;
    s->h_claim[slot] = (r->seq & 0xffffffffull) << 32;
    e = cudaMemcpyAsync(s->d_slots + slot, s->h_desc + slot, sizeof(MatDesc),
                        cudaMemcpyHostToDevice, s->as);
    if (both) {
        // who counts the request: read there by a CTA before it claims, here to
        // send it on
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(s->d_route + slot, r->mat->asym, 4, cudaMemcpyDeviceToDevice, s->as);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(s->h_words + 4 * slot, r->mat->asym, 8, cudaMemcpyDeviceToHost, s->as);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(s->h_words + 4 * slot + 2, s->d_slot_status + slot, 4, cudaMemcpyDeviceToHost,
                                s->as);
    }
    // the publication: the claim word (request number, 0 claimed), ordered
    // after the build and the descriptor
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(s->d_claim + slot, s->h_claim + slot, 8, cudaMemcpyHostToDevice,
                            s->as);
    if (e == cudaSuccess) e = cudaEventRecord(s->pub_ev[(size_t)slot], s->as);
    if (e != cudaSuccess) {
        // not published: no CTA will claim these items
        server_err(s, "ticket %llu: %s", (unsigned long long)r->ticket, cudaGetErrorString(e));
        finish(s, r, GSOFA_ERR_CUDA);
        return true;
    }
    if (items > 0) list_add(s, slot, r->seq);
    {
        std::lock_guard<std::mutex> g(s->mu);
        s->st.items_published += (uint64_t)items;
    }
    return true;
}

bool launch_kernel(gsofa_server* s, Engine& E, int k, int grid) {
    const gsofa_opts& o = s->opts;
    ServeLaunch V{};
    V.claim = s->d_claim;
    V.list = reinterpret_cast<const unsigned long long*>(static_cast<char*>(s->d_ctl) + kCtlFlags);
    V.ctrl = static_cast<const int32_t*>(s->d_ctl);
    V.kind = E.shape.chain ? SERVE_CHAIN : s->eng[E_CHAIN].on ? SERVE_WALK : SERVE_ALL;
    V.route = s->d_route;
    V.rr = s->d_rr;
    V.nslots = kSlots;
    V.slots = s->d_slots;
    V.items_done = s->d_items_done;
    V.slot_status = s->d_slot_status;
    V.done_flags = s->d_done;
    V.smem_words = E.shape.smem_words;
    V.max_idle_polls = kMaxIdlePolls;
    V.idle_ns = kIdleNs;
    V.cta_slots = E.d_cta_slots;
    V.n_cta_slots = E.shape.grid;
    V.alive = E.d_alive;
    V.launch_no = E.launches;
    V.sm_limit = serve_sms(s->ctx);
    cudaError_t e;
    if (E.shape.chain) {
        ChainLaunch C{};
        C.work_counter = s->d_work;
        C.queue = E.queue;
        C.queue_stride = std::max(s->max_n, 1);
        C.gbm = E.gbm;
        C.gbm_count = 2;
        C.bitmap_words = s->words;
        C.smem_words = E.shape.smem_words;
        C.chunk = 1;
        C.list_cap = (int)std::min<long long>(chain_list_cap(), C.queue_stride);
        C.sample_stride = 1;
        C.status = s->d_status;
        C.serve = V;
        e = launch_chain(C, E.shape.block, true, grid, E.shape.smem, E.ks[k]);
    } else {
        TraverseLaunch L{};
        L.work_counter = s->d_work;
        L.queue = E.queue;
        L.queue_stride = std::max(s->max_n, 1);
        L.gbitmap = E.gbm;
        L.gprev = E.rings;
        L.chunk = 1;
        L.merge = s->merge ? 1 : 0;
        L.chain = s->merge && !(o.flags & GSOFA_NO_CHAIN) ? 1 : 0;
        L.chain_wait_ns = chain_wait_ns(o);
        L.ring = s->ring;
        L.sample_stride = 1;
        L.bitmap_words = s->words;
        L.status = s->d_status;
        L.pattern_pass = 0;
        L.bu_alpha = o.bu_alpha > 0 ? o.bu_alpha : 0;
        L.bu_beta = o.bu_beta > 0 ? o.bu_beta : kDefaultBuBeta;
        L.bu_min_src = o.bu_min_source > 0 ? o.bu_min_source : kBuMinSource;
        L.heavy_len = o.heavy_row > 0 ? ((o.heavy_row + 3) & ~3) : kDefaultHeavyRow;
        L.serve = V;
        e = launch_serve(L, E.shape.block, grid, E.shape.smem, E.ks[k]);
    }
    if (e == cudaSuccess) e = cudaEventRecord(E.kdone[k], E.ks[k]);
    if (e != cudaSuccess) {
        server_err(s, "serving kernel launch: %s", cudaGetErrorString(e));
        s->launch_failed = true;
        return false;
    }
    E.krun[k] = true;
    E.kno[k] = E.launches++;
    s->kernel_running = true;
    std::lock_guard<std::mutex> g(s->mu);
    s->st.kernel_launches++;
    return true;
}

// CTAs currently holding a workspace slot (a short synchronous read).
int alive_ctas(gsofa_server* s, const Engine& E) {
    cudaError_t e = cudaMemcpyAsync(s->h_alive, E.d_alive, 4, cudaMemcpyDeviceToHost, s->cs);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s->cs);
    return e == cudaSuccess ? *s->h_alive : E.shape.grid;
}

// Shares the SMs out among the chain, traverse_kernel and the lanes: equal parts
// for those that have work.  (Parts of every SM's room would never hold a
// 1,024-thread CTA or a cluster.)  A CTA on another's SM leaves after its item.
void share_sms(gsofa_server* s, bool chain, bool walk, bool lanes) {
    const int parts = (chain ? 1 : 0) + (walk ? 1 : 0) + (lanes ? 1 : 0);
    if (!parts) return;
    const int each = (int)serve_sms(s->ctx) / parts;
    const int end = chain ? each : 0, begin = end;
    const int walk_end = walk ? (lanes ? begin + each : (int)serve_sms(s->ctx)) : begin;
    int32_t* f = ctl_flags(s);
    const int chain_end = chain && parts == 1 ? (int)serve_sms(s->ctx) : end;
    if (f[5] == chain_end && f[6] == begin && f[7] == walk_end) return;
    f[5] = chain_end;
    f[6] = begin;
    f[7] = walk_end;
    push_control(s);
    for (Engine& E : s->eng) E.alive_checked = -1.0;
}

// traverse_kernel takes the request.
void to_walk(gsofa_server* s, const std::shared_ptr<Request>& r) {
    r->route = TO_WALK;
    if (!s->eng[E_CHAIN].on) return;  // it takes any
    s->h_words[4 * r->slot + 3] = ROUTE_WALK;
    const cudaError_t e = cudaMemcpyAsync(s->d_route + r->slot, s->h_words + 4 * r->slot + 3, 4,
                                          cudaMemcpyHostToDevice, s->cs);
    if (e != cudaSuccess) server_err(s, "ticket %llu: %s", (unsigned long long)r->ticket, cudaGetErrorString(e));
}

// A lane's workspace: labels, totals and queues take less than 256 bytes a row.
size_t lane_bytes(int32_t n) { return 256 * (size_t)n + std::max(kLaneBytes, 296 * 5 * (size_t)n); }

// Starts the hubs' launch of a request; false: no room for its workspace.
bool lane_start(gsofa_server* s, Lane& l, const std::shared_ptr<Request>& r) {
    gsofa_ctx* ctx = s->ctx;
    size_t room;
    {
        std::lock_guard<std::mutex> g(s->mu);
        room = s->budget - std::min(s->budget, s->in_use);
    }
    std::vector<MatDesc> d(1, make_desc(r->mat, r->res, 0));
    d[0].method = r->n <= kDirectMax ? METHOD_DIRECT : METHOD_HUB;
    const size_t head = align256(sizeof(MatDesc));
    HubLaunch L;
    HubCfg c;
    size_t bytes = 0;
    std::lock_guard<std::recursive_mutex> g(ctx->mu);
    const size_t fit = std::min(room - std::min(room, head), lane_bytes(r->n));
    plan_hub(ctx, &d, s->opts, nullptr, &bytes, fit, &L, &c, kLaneCluster);
    if (head + bytes > room || dev_alloc_on(ctx, head + bytes, &l.ws, l.st) != GSOFA_OK) {
        l.ws = nullptr;
        return false;
    }
    l.bytes = head + bytes;
    plan_hub(ctx, &d, s->opts, static_cast<char*>(l.ws) + head, &bytes, fit, &L, &c, kLaneCluster);
    *l.h_desc = d[0];
    L.mats = static_cast<const MatDesc*>(l.ws);
    L.status = s->d_status;
    cudaError_t e = cudaMemcpyAsync(l.ws, l.h_desc, sizeof(MatDesc), cudaMemcpyHostToDevice, l.st);
    if (e == cudaSuccess) e = launch_hub(L, c, (s->opts.flags & GSOFA_DIGESTS) != 0, l.st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(l.h_left, L.fallback, 4, cudaMemcpyDeviceToHost, l.st);
    if (e == cudaSuccess) e = cudaEventRecord(l.done, l.st);
    if (e != cudaSuccess) {
        cudaStreamSynchronize(l.st);
        server_err(s, "ticket %llu: %s", (unsigned long long)r->ticket, cudaGetErrorString(e));
        dev_free_on(ctx, l.ws, l.bytes, l.st);
        l.ws = nullptr;
        return false;
    }
    l.r = r;
    std::lock_guard<std::mutex> gs(s->mu);
    s->in_use += l.bytes;
    s->peak = std::max(s->peak, s->in_use);
    s->st.kernel_launches++;
    return true;
}

// Lanes whose launch is over; then the next requests for those that are free.
bool manage_lanes(gsofa_server* s) {
    bool progress = false;
    for (Lane& l : s->lanes) {
        if (l.r) {
            const cudaError_t q = cudaEventQuery(l.done);
            if (q == cudaErrorNotReady) continue;
            progress = true;
            const std::shared_ptr<Request> r = l.r;
            l.r.reset();
            {
                std::lock_guard<std::recursive_mutex> g(s->ctx->mu);
                dev_free_on(s->ctx, l.ws, l.bytes, l.st);
                l.ws = nullptr;
            }
            {
                std::lock_guard<std::mutex> g(s->mu);
                s->in_use -= std::min(s->in_use, l.bytes);
            }
            if (q == cudaSuccess && *l.h_left == 0) s->h_done[r->slot] = r->seq;
            else to_walk(s, r);
        }
        if (!s->lane_queue.empty()) {
            const std::shared_ptr<Request> r = s->lane_queue.front();
            s->lane_queue.pop_front();
            if (!lane_start(s, l, r)) to_walk(s, r);
            progress = true;
        }
    }
    return progress;
}

// Keeps a kernel's CTAs on the device while published work is waiting for it.
// A CTA leaves once it has found nothing to claim for kIdleNs, which hands its
// SM back to the side stream (uploads and builds of later requests) and to the
// other kernel.  When work is waiting and fewer CTAs than its SMs hold are
// alive -- none at all, or the rest left during a large request's last items --
// another launch goes out on a free kernel stream (CTAs that find no free slot,
// or are on the other kernel's SMs, exit at once, so a stale count costs
// nothing; with half of the SMs a launch has twice the CTAs that are missing).
// With every stream taken, the oldest launch is told to take no more items: a few
// CTAs of each launch would otherwise keep all streams for as long as there is
// work, and nothing could replace those that left (48 requests at once, largest
// n = 10^6: 0.42, 1.2 and 3.2 s in three runs of 22, 0.13-0.18 s in the others).
bool manage_kernel(gsofa_server* s, int e, bool claimable) {
    Engine& E = s->eng[e];
    if (!E.on) return false;
    bool progress = false;
    bool any = false;
    int free_k = -1;
    for (int k = 0; k < E.streams(); k++) {
        if (E.krun[k] && cudaEventQuery(E.kdone[k]) == cudaSuccess) {
            E.krun[k] = false;
            progress = true;
        }
        if (E.krun[k]) any = true;
        else if (free_k < 0) free_k = k;
    }
    s->kernel_running |= any;
    if (!claimable) return progress;
    if (!any) return launch_kernel(s, E, free_k, E.shape.grid) || progress;
    const double t = now_ms(s);
    if (t - E.alive_checked < kTopUpCheckMs) return progress;
    E.alive_checked = t;
    const int sms = (int)serve_sms(s->ctx);
    const int mine = e == E_CHAIN ? ctl_flags(s)[5] : ctl_flags(s)[7] - ctl_flags(s)[6];
    const bool part = mine < sms;
    const int full = part ? std::min(E.shape.grid, E.shape.occ * std::max(mine, 1)) : E.shape.grid;
    const int missing = full - alive_ctas(s, E);
    if (missing < std::max(full < 8 ? 1 : 8, full / 16)) return progress;
    if (free_k >= 0)
        return launch_kernel(s, E, free_k, part ? std::min(E.shape.grid, 2 * missing) : missing) || progress;
    int32_t oldest = E.kno[0];
    for (int k = 1; k < E.streams(); k++) oldest = std::min(oldest, E.kno[k]);
    if (ctl_flags(s)[3 + e] <= oldest) set_control(s, 3 + e, oldest + 1);
    return progress;
}

// Requests whose last item is done: supernodes + read-back on the side
// stream; then, when that is complete, hand out the result.
bool reap(gsofa_server* s) {
    bool progress = false;
    std::vector<std::shared_ptr<Request>> act;
    {
        std::lock_guard<std::mutex> g(s->mu);
        for (auto& r : s->slot_req)
            if (r && (r->state == R_RUNNING || r->state == R_FINISHING)) act.push_back(r);
    }
    for (auto& r : act) {
        const int slot = r->slot;
        if (r->state == R_RUNNING) {
            const unsigned long long f =
                reinterpret_cast<volatile unsigned long long*>(s->h_done)[slot];
            if (f != r->seq) continue;
            if (r->n_items > 0) list_remove(s, slot);
            cudaError_t e = cudaSuccess;
            if ((s->opts.flags & GSOFA_SUPERNODES) && r->n > 0)
                e = launch_supernodes(r->n, s->opts.max_supernode_size, r->res->nz_row_u,
                                      r->res->lmask, r->res->sflags, r->res->counters, s->fs);
            if (e == cudaSuccess)
                e = cudaMemcpyAsync(s->h_cnt + (size_t)slot * CNT_SLOTS, r->res->counters,
                                    8 * CNT_SLOTS, cudaMemcpyDeviceToHost, s->fs);
            if (e == cudaSuccess)
                e = cudaMemcpyAsync(s->h_sstat + slot, s->d_slot_status + slot, 4,
                                    cudaMemcpyDeviceToHost, s->fs);
            if (e == cudaSuccess) e = cudaEventRecord(s->slot_ev[(size_t)slot], s->fs);
            if (e != cudaSuccess) {
                server_err(s, "ticket %llu: %s", (unsigned long long)r->ticket,
                           cudaGetErrorString(e));
                finish(s, r, GSOFA_ERR_CUDA);
                progress = true;
                continue;
            }
            std::lock_guard<std::mutex> g(s->mu);
            r->state = R_FINISHING;
            progress = true;
        } else {
            cudaError_t q = cudaEventQuery(s->slot_ev[(size_t)slot]);
            if (q == cudaErrorNotReady) continue;
            progress = true;
            if (q != cudaSuccess) {
                server_err(s, "ticket %llu: %s", (unsigned long long)r->ticket,
                           cudaGetErrorString(q));
                finish(s, r, GSOFA_ERR_CUDA);
                continue;
            }
            if (s->h_sstat[slot] != 0) {
                server_err(s, "ticket %llu: %s", (unsigned long long)r->ticket,
                           (s->h_sstat[slot] & DEV_ERR_COL_RANGE) ? "column id outside [0, n)"
                                                                  : "malformed CSR");
                finish(s, r, GSOFA_ERR_ARG);
                continue;
            }
            const unsigned long long* c = s->h_cnt + (size_t)slot * CNT_SLOTS;
            gsofa_counts& k = r->res->counts;
            k.n = r->n;
            k.fill_count = c[CNT_FILLS];
            k.nnz_l = c[CNT_NNZ_L];
            k.nnz_u = c[CNT_NNZ_U];
            k.nnz_lu = c[CNT_NNZ_L] + c[CNT_NNZ_U] + (uint64_t)r->n;
            k.n_supernodes = (s->opts.flags & GSOFA_SUPERNODES) ? (int64_t)c[CNT_NSUP] + 1 : -1;
            k.edges_alg = c[CNT_EDGES_ALG];
            k.vertices_alg = c[CNT_VERTS_ALG];
            k.edges_traversed = c[CNT_EDGES_TRAV];
            k.sources_chained = c[CNT_CHAINED];
            const double t = now_ms(s);
            k.ms_device = t - r->t_publish;  // host clock: publication to completion
            k.ms_traverse = k.ms_device;
            finish(s, r, GSOFA_OK);
        }
    }
    return progress;
}

// Waits for the lanes' launches and drops their requests.
void lanes_stop(gsofa_server* s) {
    s->lane_queue.clear();
    for (Lane& l : s->lanes) {
        if (!l.r) continue;
        cudaStreamSynchronize(l.st);
        l.r.reset();
        {
            std::lock_guard<std::recursive_mutex> g(s->ctx->mu);
            dev_free_on(s->ctx, l.ws, l.bytes, l.st);
            l.ws = nullptr;
        }
        std::lock_guard<std::mutex> g(s->mu);
        s->in_use -= std::min(s->in_use, l.bytes);
    }
}

// Fails every admitted request (the kernel is not running).
void fail_live(gsofa_server* s, int status) {
    lanes_stop(s);
    std::vector<std::shared_ptr<Request>> act;
    {
        std::lock_guard<std::mutex> g(s->mu);
        for (auto& r : s->slot_req)
            if (r) act.push_back(r);
    }
    for (auto& r : act) {
        if (r->n_items > 0 && r->state == R_RUNNING) list_remove(s, r->slot);
        finish(s, r, status);
    }
}

void loop(gsofa_server* s) {
    cudaSetDevice(s->ctx->device);
    int idle_spins = 0;
    double shutdown_at = -1.0;
    for (;;) {
        bool progress = false;
        // admit in slices, so that publication, the kernel launch and the
        // read-back of finished requests are not held up behind the uploads
        // of a long queue
        const double t_adm = now_ms(s);
        while (admit_one(s)) {
            progress = true;
            if (now_ms(s) - t_adm > kAdmitSliceMs) break;
        }
        // requests whose claim word is on the device and whose items are not
        // all finished
        bool claimable[kEngines] = {};
        std::vector<std::shared_ptr<Request>> walk;  // repeated entries, or a build that failed
        {
            std::lock_guard<std::mutex> g(s->mu);
            for (auto& r : s->slot_req) {
                if (!r || r->state != R_RUNNING) continue;
                if (!r->published &&
                    cudaEventQuery(s->pub_ev[(size_t)r->slot]) == cudaSuccess) {
                    r->published = true;
                    r->t_publish = now_ms(s);
                    if (r->n_items == 0) {  // no rows: to be read back, now that its totals are zeroed
                        s->h_done[r->slot] = r->seq;
                        continue;
                    }
                    const int32_t* w = s->h_words + 4 * r->slot;
                    if (!s->eng[E_CHAIN].on) r->route = TO_WALK;
                    else if (w[0] == 0) r->route = TO_CHAIN;
                    else if (w[1] == 0 && w[2] == 0) r->route = TO_LANE;
                    if (r->route == TO_LANE) s->lane_queue.push_back(r);
                    else if (r->route == TO_NONE) walk.push_back(r);
                }
                if (r->route == TO_CHAIN) claimable[E_CHAIN] = true;
                if (r->route == TO_WALK) claimable[E_WALK] = true;
            }
        }
        for (auto& r : walk) to_walk(s, r);
        progress |= manage_lanes(s);
        bool lanes = !s->lane_queue.empty();
        for (const Lane& l : s->lanes) lanes |= l.r != nullptr;
        if (lanes) s->lanes_until = now_ms(s) + kLaneHoldMs;
        const bool held = (claimable[E_CHAIN] || claimable[E_WALK]) && now_ms(s) < s->lanes_until;
        share_sms(s, claimable[E_CHAIN], claimable[E_WALK], lanes || held);
        s->kernel_running = false;
        for (int e = 0; e < kEngines; e++) progress |= manage_kernel(s, e, claimable[e]);
        if (s->launch_failed) {
            // no kernel can run: nothing admitted can finish
            fail_live(s, GSOFA_ERR_CUDA);
            s->launch_failed = false;
        }
        progress |= reap(s);
        std::unique_lock<std::mutex> lk(s->mu);
        const bool idle = s->queued.empty() && s->live == 0;
        if (s->shutdown && idle && !s->kernel_running) break;
        if (s->shutdown && idle && s->kernel_running && ctl_flags(s)[0] == 0) {
            lk.unlock();
            set_control(s, 0, 1);  // idle CTAs leave at once
            continue;
        }
        if (s->shutdown && shutdown_at < 0) shutdown_at = now_ms(s);
        if (s->shutdown && now_ms(s) - shutdown_at > kShutdownGraceMs) {
            // still busy long after destroy began: stop taking items, let the
            // CTAs finish the ones they hold, and fail whatever is left
            lk.unlock();
            set_control(s, 1, 1);
            for (Engine& E : s->eng)
                for (int k = 0; k < kKernelStreams; k++)
                    if (E.krun[k]) cudaEventSynchronize(E.kdone[k]);
            s->kernel_running = false;
            reap(s);
            fail_live(s, GSOFA_ERR_TIMEOUT);
            std::lock_guard<std::mutex> g(s->mu);
            for (auto& r : s->queued) {
                r->state = R_FAILED;
                r->status = GSOFA_ERR_TIMEOUT;
            }
            s->queued.clear();
            s->cv_done.notify_all();
            break;
        }
        if (progress) {
            idle_spins = 0;
            continue;
        }
        if (idle && !s->kernel_running) {
            s->cv_work.wait_for(lk, std::chrono::milliseconds(5));
        } else {
            lk.unlock();
            // poll the device signals: spin briefly, then back off
            if (++idle_spins < 200) std::this_thread::yield();
            else std::this_thread::sleep_for(std::chrono::microseconds(20));
        }
    }
}

void release(gsofa_server* s) {
    gsofa_ctx* ctx = s->ctx;
    cudaSetDevice(ctx->device);
    for (Engine& E : s->eng)
        for (int k = 0; k < kKernelStreams; k++)
            if (E.ks[k]) cudaStreamSynchronize(E.ks[k]);
    for (Lane& l : s->lanes) {
        if (l.st) cudaStreamSynchronize(l.st);
        if (l.done) cudaEventDestroy(l.done);
        if (l.st) cudaStreamDestroy(l.st);
        if (l.h_desc) cudaFreeHost(l.h_desc);
    }
    {
        std::lock_guard<std::recursive_mutex> g(ctx->mu);
        cudaStream_t st = s->as ? s->as : ctx->stream;
        dev_free_on(ctx, s->tab, s->tab_bytes, st);
        for (Engine& E : s->eng) dev_free_on(ctx, E.ws, E.ws_bytes, st);
    }
    if (s->as) cudaStreamSynchronize(s->as);
    if (s->cs) cudaStreamSynchronize(s->cs);
    if (s->fs) cudaStreamSynchronize(s->fs);
    for (cudaEvent_t e : s->slot_ev)
        if (e) cudaEventDestroy(e);
    for (cudaEvent_t e : s->pub_ev)
        if (e) cudaEventDestroy(e);
    for (Engine& E : s->eng)
        for (int k = 0; k < kKernelStreams; k++) {
            if (E.kdone[k]) cudaEventDestroy(E.kdone[k]);
            if (E.ks[k]) cudaStreamDestroy(E.ks[k]);
        }
    if (s->as) cudaStreamDestroy(s->as);
    if (s->h_words) cudaFreeHost(s->h_words);
    if (s->h_alive) cudaFreeHost(s->h_alive);
    if (s->cs) cudaStreamDestroy(s->cs);
    if (s->fs) cudaStreamDestroy(s->fs);
    if (s->h_ctl) cudaFreeHost(s->h_ctl);
    if (s->h_done) cudaFreeHost(s->h_done);
    if (s->h_desc) cudaFreeHost(s->h_desc);
    if (s->h_claim) cudaFreeHost(s->h_claim);
    if (s->h_cnt) cudaFreeHost(s->h_cnt);
    if (s->h_sstat) cudaFreeHost(s->h_sstat);
    s->stager.release();
}

}  // namespace

extern "C" {

int gsofa_server_create(gsofa_ctx* ctx, const gsofa_opts* opts, int32_t max_n,
                        size_t budget_bytes, gsofa_server** out) {
    if (!ctx || !out || max_n <= 0) return GSOFA_ERR_ARG;
    *out = nullptr;
    gsofa_opts o;
    if (opts) o = *opts;
    else gsofa_opts_default(&o);
    if (o.max_supernode_size <= 0 || o.threads_per_source < 0 || o.sources_in_flight < 0 ||
        o.chunk_sources < 0 || o.cached_closures < 0)
        return set_err(ctx, GSOFA_ERR_ARG, "invalid serving options");
    if (o.flags & GSOFA_PATTERN)
        return set_err(ctx, GSOFA_ERR_UNSUPPORTED, "GSOFA_PATTERN is not served");
    if (o.threads_per_source > 0 && o.threads_per_source != 256 && o.threads_per_source != 512 &&
        o.threads_per_source != 1024)
        return set_err(ctx, GSOFA_ERR_ARG, "serving threads_per_source must be 256, 512 or 1024");
    if (cudaSetDevice(ctx->device) != cudaSuccess) return set_err(ctx, GSOFA_ERR_CUDA, "cudaSetDevice");

    gsofa_server* s = new (std::nothrow) gsofa_server();
    if (!s) return set_err(ctx, GSOFA_ERR_OOM_BUDGET, "host allocation failed");
    s->ctx = ctx;
    s->opts = o;
    s->max_n = max_n;
    s->budget = budget_bytes ? budget_bytes : kDefaultBudget;
    s->merge = !(o.flags & GSOFA_NO_MERGE);
    s->ring = o.cached_closures > 0 ? std::min(o.cached_closures, kMaxRing) : kDefaultRing;
    while (s->ring & (s->ring - 1)) s->ring &= s->ring - 1;
    s->t0 = std::chrono::steady_clock::now();
    auto fail = [&](int rc, const char* what, cudaError_t e) {
        if (e != cudaSuccess) set_err(ctx, rc, "%s: %s", what, cudaGetErrorString(e));
        else set_err(ctx, rc, "%s", what);
        release(s);
        delete s;
        return rc;
    };

    s->words = (((long long)max_n + 31) >> 5) + 6;
    const bool counting = chain_runs(o, nullptr, 0) && !(o.flags & GSOFA_L_ROW_STATS);
    // traverse_kernel always, and the chain for symmetric patterns where it can
    // be resident and the budgets have room for its workspace too; that goes
    // again when a request needs its room (shed_chain)
    s->eng[E_WALK].shape = serve_shape(ctx, *s, false);
    s->eng[E_WALK].on = true;
    if (s->eng[E_WALK].shape.occ <= 0)
        return fail(GSOFA_ERR_UNSUPPORTED, "serving kernel cannot be resident", cudaSuccess);
    if (counting) s->eng[E_CHAIN].shape = serve_shape(ctx, *s, true);
    s->eng[E_CHAIN].on = counting && s->eng[E_CHAIN].shape.occ > 0;

    // the side and control streams outrank the kernel stream: when an SM
    // frees up, their pending blocks are placed first
    cudaError_t e;
    int prio_low = 0, prio_high = 0;
    cudaDeviceGetStreamPriorityRange(&prio_low, &prio_high);
    for (Engine& E : s->eng)
        for (int k = 0; k < E.streams() && E.on; k++)
            if ((e = cudaStreamCreateWithPriority(&E.ks[k], cudaStreamNonBlocking, prio_low)) != cudaSuccess ||
                (e = cudaEventCreateWithFlags(&E.kdone[k], cudaEventDisableTiming)) != cudaSuccess)
                return fail(GSOFA_ERR_CUDA, "stream", e);
    // (the lanes' kernels end by themselves: they go before CTAs of the two that stay)
    for (Lane& l : s->lanes) {
        if (!s->eng[E_CHAIN].on) break;
        if ((e = cudaStreamCreateWithPriority(&l.st, cudaStreamNonBlocking, (prio_low + prio_high) / 2)) !=
                cudaSuccess ||
            (e = cudaEventCreateWithFlags(&l.done, cudaEventDisableTiming)) != cudaSuccess ||
            (e = cudaMallocHost((void**)&l.h_desc, align256(sizeof(MatDesc)) + 64)) != cudaSuccess)
            return fail(GSOFA_ERR_CUDA, "lane", e);
        l.h_left = reinterpret_cast<int32_t*>(reinterpret_cast<char*>(l.h_desc) + align256(sizeof(MatDesc)));
    }
    if ((e = cudaStreamCreateWithPriority(&s->as, cudaStreamNonBlocking, prio_high)) != cudaSuccess)
        return fail(GSOFA_ERR_CUDA, "stream", e);
    if ((e = cudaStreamCreateWithPriority(&s->cs, cudaStreamNonBlocking, prio_high)) != cudaSuccess)
        return fail(GSOFA_ERR_CUDA, "stream", e);
    if ((e = cudaStreamCreateWithPriority(&s->fs, cudaStreamNonBlocking, prio_high)) != cudaSuccess)
        return fail(GSOFA_ERR_CUDA, "stream", e);
    s->slot_ev.assign(kSlots, nullptr);
    s->pub_ev.assign(kSlots, nullptr);
    for (auto& ev : s->slot_ev)
        if ((e = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming)) != cudaSuccess)
            return fail(GSOFA_ERR_CUDA, "event", e);
    for (auto& ev : s->pub_ev)
        if ((e = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming)) != cudaSuccess)
            return fail(GSOFA_ERR_CUDA, "event", e);
    if ((e = cudaHostAlloc((void**)&s->h_done, 8 * kSlots, cudaHostAllocMapped)) != cudaSuccess)
        return fail(GSOFA_ERR_CUDA, "mapped host memory", e);
    memset(s->h_done, 0, 8 * kSlots);
    if ((e = cudaHostGetDevicePointer((void**)&s->d_done, s->h_done, 0)) != cudaSuccess)
        return fail(GSOFA_ERR_CUDA, "mapped host memory", e);
    if ((e = cudaMallocHost(&s->h_ctl, kCtlBytes)) != cudaSuccess ||
        (e = cudaMallocHost((void**)&s->h_words, 16 * kSlots)) != cudaSuccess ||
        (e = cudaMallocHost((void**)&s->h_alive, 64)) != cudaSuccess)
        return fail(GSOFA_ERR_CUDA, "pinned host memory", e);
    memset(s->h_ctl, 0, kCtlFlags);
    memset(static_cast<char*>(s->h_ctl) + kCtlFlags, 0xff, kCtlBytes - kCtlFlags);
    if ((e = cudaMallocHost((void**)&s->h_desc, sizeof(MatDesc) * kSlots)) != cudaSuccess ||
        (e = cudaMallocHost((void**)&s->h_claim, 8 * kSlots)) != cudaSuccess ||
        (e = cudaMallocHost((void**)&s->h_cnt, 8 * CNT_SLOTS * kSlots)) != cudaSuccess ||
        (e = cudaMallocHost((void**)&s->h_sstat, 4 * kSlots)) != cudaSuccess ||
        (e = s->stager.init()) != cudaSuccess)
        return fail(GSOFA_ERR_CUDA, "pinned host memory", e);

    // the device tables, then per kernel: per-CTA queues, closure rings and
    // global bitmaps, the CTA slots' bits and the count of those taken
    s->tab_bytes = align256(sizeof(MatDesc) * kSlots) + align256(8 * kSlots) * 2 +
                   align256(4 * kSlots) * 2 + 256 + align256(kCtlBytes);
    auto slot_bytes = [](const Engine& E) { return align256(4 * (size_t)((E.shape.grid + 31) / 32)); };
    for (Engine& E : s->eng)
        if (E.on) E.ws_bytes = E.shape.bytes(s->words) + slot_bytes(E) + 256;
    s->least = s->tab_bytes + s->eng[E_WALK].ws_bytes;
    if (s->least > s->budget)
        return fail(GSOFA_ERR_OOM_BUDGET, "serving workspace exceeds the budget", cudaSuccess);
    if (s->least + s->eng[E_CHAIN].ws_bytes > s->budget) s->eng[E_CHAIN].on = false;
    {
        std::lock_guard<std::recursive_mutex> g(ctx->mu);
        int rc = dev_alloc_on(ctx, s->tab_bytes, &s->tab, s->as);
        if (rc == GSOFA_OK) rc = dev_alloc_on(ctx, s->eng[E_WALK].ws_bytes, &s->eng[E_WALK].ws, s->as);
        if (rc) {
            release(s);
            delete s;
            return rc;
        }
        Engine& C = s->eng[E_CHAIN];
        if (C.on && dev_alloc_on(ctx, C.ws_bytes, &C.ws, s->as) != GSOFA_OK) C.on = false;
        // The pool grows now, for the lanes' workspaces and a few requests of max_n
        // rows: while serving kernels run, its growth waits until they have no work
        // (a request behind a large one's last item; of 56 bursts of 48 requests 3 took
        // about 1 s, of 60 now none took more than 0.15 s).
        size_t ahead[kLanes + 1];
        std::fill_n(ahead, kLanes, C.on ? std::min(lane_bytes(max_n), kAhead / 8) : 0);
        ahead[kLanes] = std::min(4 * request_footprint(s, max_n, 16ll * max_n), kAhead);
        void* warm[kLanes + 1] = {};
        for (int k = 0; k <= kLanes; k++)
            if (s->least + C.ws_bytes + ahead[k] > s->budget ||
                dev_alloc_on(ctx, ahead[k], &warm[k], s->as) != GSOFA_OK)
                warm[k] = nullptr;
        for (int k = 0; k <= kLanes; k++) dev_free_on(ctx, warm[k], ahead[k], s->as);
        // kernels that a request would load while serving kernels run, which its
        // launch then waits for (the first burst of 48 requests of up to 10^6 rows
        // took 0.33-0.75 s, now 0.13)
        void* few = nullptr;
        if (C.on && dev_alloc_on(ctx, hub_load_bytes(), &few, s->as) == GSOFA_OK) {
            e = hub_load(few, s->as);
            dev_free_on(ctx, few, hub_load_bytes(), s->as);
        }
        if (e == cudaSuccess) e = load_supernodes();
    }
    if (e != cudaSuccess) return fail(GSOFA_ERR_CUDA, "serving kernels", e);
    char* b = static_cast<char*>(s->tab);
    s->d_slots = reinterpret_cast<MatDesc*>(b);
    b += align256(sizeof(MatDesc) * kSlots);
    s->d_claim = reinterpret_cast<unsigned long long*>(b);
    b += align256(8 * kSlots);
    s->d_items_done = reinterpret_cast<unsigned long long*>(b);
    b += align256(8 * kSlots);
    s->d_slot_status = reinterpret_cast<int32_t*>(b);
    b += align256(4 * kSlots);
    s->d_route = reinterpret_cast<int32_t*>(b);
    b += align256(4 * kSlots);
    s->d_work = reinterpret_cast<unsigned long long*>(b);
    s->d_rr = reinterpret_cast<unsigned int*>(s->d_work + 1);
    s->d_status = reinterpret_cast<int32_t*>(s->d_work + 2);
    b += 256;
    s->d_ctl = b;
    int32_t* const flags = ctl_flags(s);
    flags[5] = flags[7] = (int32_t)serve_sms(ctx);
    for (Engine& E : s->eng) {
        if (!E.on) continue;
        char* w = static_cast<char*>(E.ws);
        E.queue = reinterpret_cast<int32_t*>(w);
        w += E.shape.queues();
        E.rings = E.shape.rings(s->words) ? reinterpret_cast<uint32_t*>(w) : nullptr;
        w += E.shape.rings(s->words);
        const size_t gb = E.shape.bitmaps(s->words);
        E.gbm = gb ? reinterpret_cast<uint32_t*>(w) : nullptr;
        w += gb;
        E.d_cta_slots = reinterpret_cast<unsigned int*>(w);
        w += slot_bytes(E);
        E.d_alive = reinterpret_cast<int*>(w);
        if ((gb && (e = cudaMemsetAsync(E.gbm, 0, gb, s->as)) != cudaSuccess) ||
            (e = cudaMemsetAsync(E.d_cta_slots, 0, slot_bytes(E) + 256, s->as)) != cudaSuccess)
            return fail(GSOFA_ERR_CUDA, "workspace init", e);
    }
    // claim words start at request number 0 (never used): nothing claimable
    if ((e = cudaMemsetAsync(s->d_claim, 0, 8 * kSlots, s->as)) != cudaSuccess ||
        (e = cudaMemsetAsync(s->d_route, 0, 4 * kSlots, s->as)) != cudaSuccess ||
        (e = cudaMemsetAsync(s->d_work, 0, 256, s->as)) != cudaSuccess ||
        (e = cudaMemcpyAsync(s->d_ctl, s->h_ctl, kCtlBytes, cudaMemcpyHostToDevice, s->as)) !=
            cudaSuccess)
        return fail(GSOFA_ERR_CUDA, "workspace init", e);
    if ((e = cudaStreamSynchronize(s->as)) != cudaSuccess)
        return fail(GSOFA_ERR_CUDA, "workspace init", e);
    s->fixed = s->least + (s->eng[E_CHAIN].on ? s->eng[E_CHAIN].ws_bytes : 0);
    s->in_use = s->peak = s->fixed;
    s->slot_req.assign(kSlots, nullptr);
    for (int i = kSlots - 1; i >= 0; i--) s->free_slots.push_back(i);
    const ServeShape& lead = s->eng[s->eng[E_CHAIN].on ? E_CHAIN : E_WALK].shape;
    s->st.grid = lead.grid;
    s->st.block = lead.block;
    try {
        s->th = std::thread(loop, s);
    } catch (...) {
        return fail(GSOFA_ERR_UNSUPPORTED, "cannot start the serving thread", cudaSuccess);
    }
    *out = s;
    return GSOFA_OK;
}

int gsofa_server_submit(gsofa_server* s, int32_t n, int64_t nnz, const int32_t* row_begin,
                        const int32_t* row_end, const int32_t* col, uint64_t* ticket) {
    if (!s || !ticket) return GSOFA_ERR_ARG;
    *ticket = 0;
    if (n < 0 || nnz < 0 || (n > 0 && (!row_begin || !row_end)) || (nnz > 0 && !col))
        return GSOFA_ERR_ARG;
    if (n > s->max_n) return GSOFA_ERR_UNSUPPORTED;
    auto r = std::make_shared<Request>();
    r->n = n;
    r->nnz = nnz;
    r->beg = row_begin;
    r->end = row_end;
    r->col = col;
    r->footprint = request_footprint(s, n, nnz);
    if (r->footprint + s->least > s->budget) return GSOFA_ERR_OOM_BUDGET;
    std::lock_guard<std::mutex> g(s->mu);
    if (s->shutdown) return GSOFA_ERR_ARG;
    r->ticket = s->next_ticket++;
    r->t_submit = now_ms(s);
    s->queued.push_back(r);
    s->tickets[r->ticket] = r;
    s->st.submitted++;
    *ticket = r->ticket;
    s->cv_work.notify_one();
    return GSOFA_OK;
}

// Hands out a finished request's result (once).  With res == NULL the result
// is returned in *drop for the caller to destroy outside the server's lock.
static int take_result(Request& r, gsofa_result** res, gsofa_result** drop) {
    if (r.state == R_FAILED) return r.status;
    if (r.state != R_DONE) return GSOFA_ERR_BUSY;
    if (r.handed_out || !r.res) return GSOFA_ERR_ARG;
    r.handed_out = true;
    if (res) *res = r.res;
    else *drop = r.res;
    r.res = nullptr;
    return GSOFA_OK;
}

int gsofa_server_poll(gsofa_server* s, uint64_t ticket, gsofa_result** res) {
    if (!s) return GSOFA_ERR_ARG;
    if (res) *res = nullptr;
    gsofa_result* drop = nullptr;
    int rc;
    {
        std::lock_guard<std::mutex> g(s->mu);
        auto it = s->tickets.find(ticket);
        if (it == s->tickets.end()) return GSOFA_ERR_ARG;
        rc = take_result(*it->second, res, &drop);
    }
    if (drop) result_free(drop);
    return rc;
}

int gsofa_server_wait(gsofa_server* s, uint64_t ticket, double timeout_ms, gsofa_result** res) {
    if (!s) return GSOFA_ERR_ARG;
    if (res) *res = nullptr;
    gsofa_result* drop = nullptr;
    int rc;
    {
        std::unique_lock<std::mutex> lk(s->mu);
        auto it = s->tickets.find(ticket);
        if (it == s->tickets.end()) return GSOFA_ERR_ARG;
        std::shared_ptr<Request> r = it->second;
        auto done = [&] { return r->state == R_DONE || r->state == R_FAILED; };
        if (timeout_ms < 0) {
            s->cv_done.wait(lk, done);
        } else if (!s->cv_done.wait_for(lk, std::chrono::duration<double, std::milli>(timeout_ms),
                                        done)) {
            return GSOFA_ERR_TIMEOUT;
        }
        rc = take_result(*r, res, &drop);
    }
    if (drop) result_free(drop);
    return rc;
}

int gsofa_server_ticket_info(gsofa_server* s, uint64_t ticket, gsofa_ticket_info* info) {
    if (!s || !info) return GSOFA_ERR_ARG;
    std::lock_guard<std::mutex> g(s->mu);
    auto it = s->tickets.find(ticket);
    if (it == s->tickets.end()) return GSOFA_ERR_ARG;
    const Request& r = *it->second;
    info->t_submit_ms = r.t_submit;
    info->t_admit_ms = r.t_admit;
    info->t_publish_ms = r.t_publish;
    info->t_done_ms = r.t_done;
    info->footprint_bytes = r.footprint;
    info->status = (r.state == R_DONE || r.state == R_FAILED) ? r.status : GSOFA_ERR_BUSY;
    info->n = r.n;
    return GSOFA_OK;
}

int gsofa_server_get_stats(gsofa_server* s, gsofa_server_stats* out) {
    if (!s || !out) return GSOFA_ERR_ARG;
    std::lock_guard<std::mutex> g(s->mu);
    *out = s->st;
    out->bytes_in_use = s->in_use;
    out->peak_bytes = s->peak;
    out->fixed_bytes = s->fixed;
    return GSOFA_OK;
}

const char* gsofa_server_last_error(const gsofa_server* s) {
    if (!s) return "null server";
    return s->err.c_str();
}

int gsofa_server_destroy(gsofa_server* s) {
    if (!s) return GSOFA_ERR_ARG;
    {
        std::lock_guard<std::mutex> g(s->mu);
        s->shutdown = true;
        s->cv_work.notify_all();
    }
    if (s->th.joinable()) s->th.join();
    // the loop has finished every request and the kernel has exited
    for (auto& kv : s->tickets) {
        Request& r = *kv.second;
        if (r.res) {
            result_free(r.res);
            r.res = nullptr;
        }
    }
    release(s);
    delete s;
    return GSOFA_OK;
}

}  // extern "C"
