// gsofa_hub.cu -- the counting traversal for matrices with a large strongly
// connected core: every source searched on its own, on top of what a hub
// reaches.
//
// For a vertex b let label(v) be the smallest value, over all paths b -> v, of
// the path's largest id before v (b included).  Then b reaches v through ids
// below s exactly when label(v) < s, for every s at once.  With the labels of
// one well connected b in A and in A^T (`lam` of the two directions), a source
// s that reaches b through ids below s -- one comparison, label of s in the
// other direction below s -- has
//     F(s) = { v : label(v) < s }  u  what s reaches beyond it,
// and the first set's sizes and digest are known for every s in advance: each v
// joins it at s = label(v) + 1 and leaves the part above s at s = v, so the
// totals are prefix sums over s of the changes at these times (its digest too:
// a 32-id word's term changes only there).  What is left per source is the
// search beyond the hub's set: on the circuit-like n = 659,033 matrix 21 ids on
// average, and no source waits for another.  gsofa_chain.cu, where a chunk's
// sources are a chain, took 450 ms on that matrix.
//
// Four hubs serve three windows of s (above n/16, n/16 down to n/256, below), two
// of them the first, each among the ids below its window's, so that early sources
// have one too; the smaller windows' labels expand only ids below their end.
//
//   hub_kernel     per matrix and window: the vertex of largest in-degree times
//                  out-degree below the window's start
//   label_*_kernel label-correcting rounds: by a cluster of up to 16 CTAs per
//                  (matrix, hub, direction) in shared memory, which takes n up to
//                  893,000, else one launch of the whole GPU per round (46 and 93
//                  rounds for the first window of the circuit-like matrix, 3.5 to
//                  5.2 reads per entry)
//   event_kernel   a warp per word of 32 ids: the changes of the totals
//   (a scan)       the totals of the hub's set for every s
//   extra_kernel   a warp per (source, direction): the search beyond, in a
//                  table in shared memory
//   large_kernel   the sources whose search outgrew the table: a CTA each, in
//                  a bitmap
//
// A matrix of at most kDirectMax rows has every source searched alone, without
// a hub.  A matrix in which more than a quarter of the searches outgrow the
// table (no core that the hub lies in: meshes) is left: traverse_kernel counts
// it, whose reuse of closures does not need a core (200,000-row band of 4 without
// one: 13 ms, 248 searched source by source along a chain; 90,000-row mesh with a
// third of its couplings one-sided: 16 ms and 26).
#include <algorithm>
#include <climits>

#include <cub/device/device_scan.cuh>

#include "gsofa_device.cuh"
#include "gsofa_label.h"

namespace gsofa {

namespace {

constexpr int kWindows = 3;
constexpr int kHubs = 4;  // two for the first window, one for each other
constexpr int kBases = 2;  // arrays of totals: a source has at most two hubs to choose from
// Label rounds after which a hub is given up.  First window: 24 at n = 5,000, 39
// to 284 at 20,000 and 96 at 40,000 for matrices with a core (random and banded
// with uniform entries, circuit-like), and seldom both of its hubs above 192; a
// band without a core uses up all of them, which at 192 was 0.6 of 2.6 ms at
// n = 5,000.  Far larger ones need more: a band with one uniform entry per row at
// n = 1,200,000 more than 192 (left: 582 ms).  The other windows' few ids are a
// band with hardly an entry besides, where labels travel along: up to 278 at
// 20,000.  (With 192 for all, and a matrix left with its first such hub, 9 of 40
// random n = 20,000 matrices were left, at 2.2 ms; now none, 0.5 to 0.9.)
__host__ __device__ __forceinline__ int label_rounds(int n, int window) {
    if (window) return 64 + n / 32;
    const int a = 64 + n / 64, b = n / 2048 < 192 ? 192 : n / 2048;
    return a < b ? a : b;
}
// The first window's limit once its set has stopped growing (see settled).
__host__ __device__ __forceinline__ int label_rounds_settled(int n) { return 128 + n / 64; }
// A core is reached within a few tens of rounds, the rest only lower labels; in
// a mesh the hub's set still grows then.  The ids first reached in the rounds up
// to kSpread, in the next 16 and in the 16 after that are counted; a matrix is
// left when the last are more than half of those before them and more than n/64
// (see spreads): a 40^3 mesh with a third of its couplings one-sided 8.2 -> 6.5 ms,
// 6.1 by traverse_kernel alone.
constexpr int kSpread = 32, kSpreadStep = 16;
constexpr int kSpreadEnd = kSpread + 2 * kSpreadStep;
constexpr int kLook = 16;  // rounds between looks whether another search has left the matrix
constexpr int kLabelThreads = 1024;
constexpr int kNoLabel = 0x7f7f7f7f;  // label_round_kernel's arrays are set bytewise
constexpr int kExtraThreads = 256;
constexpr int kLargeThreads = 256;
// A matrix is left when more than half of at least kJudgeEarly searches, or more
// than a quarter of kJudgeAfter, have outgrown the table: looked at with every
// such search, and what is under way then ends with it (at the end of every
// item instead, a batch of 48 bands without a core spent 10 of 28 ms there).  An
// eighth or a half instead of the quarter changes no time by more than 1 %: one-sided
// meshes of 4,900 to 90,000 rows, a 200,000-row band, random n = 80,000 with 0.9 to
// 2.5 entries a row.
constexpr int kJudgeEarly = 64, kJudgeAfter = 512;
// A matrix is also left when its large searches, by the mean of those done so
// far, will read more than kLargePerRow entries for each of its rows: large_kernel
// reads 220 G entries/s, traverse_kernel takes 0.3 to 0.5 us a row.  The circuit-like
// n = 659,033 after the hybrid ordering, whose sources below the top separators
// reach no hub, would read 115,000 a row: 355 ms, 210 by traverse_kernel alone.
// After the level-set ordering it reads 4,200 (44 ms against 326), ordered random
// and banded matrices of 20,000 rows 10,000 to 15,000 (1.7-2.0 ms against 2.7-3.9).
constexpr unsigned long long kLargeSample = 1024;
constexpr double kLargePerRow = 65536.0;

struct WarpTable {
    uint32_t key[kSlots];
    uint32_t msk[kSlots];
    int32_t list[kListRoom];
};

// sources of window l: above window_end(n, l + 1), up to window_end(n, l); its
// labels expand ids below window_end(n, l); its hub lies below window_end(n, l + 1)
__host__ __device__ __forceinline__ int window_end(int n, int l) { return n >> (4 * l); }

__device__ __forceinline__ int window_of(int n, int s) {
    return s > window_end(n, 1) ? 0 : s > window_end(n, 2) ? 1 : 2;
}

// hubs 0 and 1 serve the first window, 2 and 3 the others
__host__ __device__ __forceinline__ int window_of_hub(int h) { return h < 2 ? 0 : h - 1; }

__device__ __forceinline__ long long lam_at(const HubLaunch& P, const MatDesc& M, int h, int d) {
    return (2ll * h + d) * P.total + M.hub_off;
}

// The count that round r adds to: 0 up to kSpread, 1 and 2 for the steps after it.
__device__ __forceinline__ int spread_part(int r) { return r < kSpread ? 0 : r < kSpread + kSpreadStep ? 1 : 2; }

// Less than an eighth of the set came in the last step: a core has been reached,
// and the rounds that are left lower labels.
__device__ __forceinline__ bool settled(int all, int last) { return 8ll * last <= all; }

__device__ __forceinline__ bool spreads(int n, int before, int last) { return 2 * last > before && 64 * (long long)last > n; }

// A label search of hub h did not finish.  The hub's labels in that direction
// become none, so that no search starts from it or finds anything in its set; the
// first window has another hub.  Without that one, or another window's only
// hub, the matrix is left.
__device__ __forceinline__ void give_up(const HubLaunch& P, int mi, int h) {
    const int before = atomicOr(P.given_up + mi, 1 << h);
    if (h > 1 || ((before | 1 << h) & 3) == 3) atomicExch(P.fallback + mi, 1);
}

// Per matrix and hub, several CTAs: the largest key (degree product, then
// smallest id).  The first window's two hubs are the best of the even and of
// the odd ids.
__global__ void hub_kernel(HubLaunch P) {
    const int mi = blockIdx.x / kHubs, h = blockIdx.x % kHubs;
    const MatDesc& M = P.mats[mi];
    if (M.method != METHOD_HUB) return;
    const int lim = max(2, window_end(M.n, window_of_hub(h) + 1));
    const int step = h < 2 ? 2 : 1;
    unsigned long long mine = 0;
    for (int v = (h == 1) + step * (blockIdx.y * blockDim.x + threadIdx.x); v < lim;
         v += step * gridDim.y * blockDim.x) {
        const unsigned long long a = (unsigned)row_degree<false>(M.rowptr, v);
        const unsigned long long b = (unsigned)row_degree<false>(M.trowptr, v);
        const unsigned long long p = min(a * b, 0xfffffffeull) + 1ull;
        mine = max(mine, p << 32 | (0xffffffffu - (unsigned)v));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mine = max(mine, __shfl_xor_sync(FULL_MASK, mine, o));
    if ((threadIdx.x & 31) == 0 && mine) atomicMax(P.hubs + blockIdx.x, mine);
}

__device__ __forceinline__ int hub_of(const HubLaunch& P, int mi, int h) {
    return (int)(0xffffffffu - (unsigned)P.hubs[mi * kHubs + h]);
}

__device__ __forceinline__ unsigned cluster_size() {
    unsigned x;
    asm("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(x));
    return x;
}
__device__ __forceinline__ unsigned cluster_rank() {
    unsigned x;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(x));
    return x;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// A shared-memory address of this CTA, as the same place in CTA `rank`.
__device__ __forceinline__ unsigned at_rank(unsigned addr, unsigned rank) {
    unsigned x;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(x) : "r"(addr), "r"(rank));
    return x;
}
__device__ __forceinline__ int dsm_ld(unsigned a) {
    int x;
    asm volatile("ld.volatile.shared::cluster.s32 %0, [%1];" : "=r"(x) : "r"(a) : "memory");
    return x;
}
__device__ __forceinline__ int dsm_min(unsigned a, int v) {
    int x;
    asm volatile("atom.relaxed.cluster.shared::cluster.min.s32 %0, [%1], %2;" : "=r"(x) : "r"(a), "r"(v) : "memory");
    return x;
}
__device__ __forceinline__ int dsm_or(unsigned a, int v) {
    int x;
    asm volatile("atom.relaxed.cluster.shared::cluster.or.b32 %0, [%1], %2;" : "=r"(x) : "r"(a), "r"(v) : "memory");
    return x;
}
__device__ __forceinline__ int dsm_add(unsigned a, int v) {
    int x;
    asm volatile("atom.relaxed.cluster.shared::cluster.add.s32 %0, [%1], %2;" : "=r"(x) : "r"(a), "r"(v) : "memory");
    return x;
}

// Labels of one (matrix, hub, direction) by one thread block cluster, spread
// over its CTAs' shared memory: a word per id (gsofa_label.h), groups of 32 ids
// dealt out in turn.  A round expands the ids queued in the one before; one
// atomic operation marks an id idle and reads its label, so an improvement is
// either read there or queues the id again.  Queues are in global memory.
__global__ void __launch_bounds__(kLabelThreads) label_cluster_kernel(HubLaunch P) {
    extern __shared__ uint4 dyn_smem[];
    // of rank 0: queued ids per round, in turn; whether the matrix is left, every
    // kLook rounds in turn; ids reached by the ends of the three parts
    __shared__ int cnt[3], quit[2], reached[3];
    const unsigned C = cluster_size(), rank = cluster_rank();
    const unsigned shift = 31 - __clz(C);
    const int job = blockIdx.x / C;
    const int mi = job / (2 * kHubs), h = (job >> 1) % kHubs, d = job & 1;
    const MatDesc& M = P.mats[mi];
    if (M.method != METHOD_HUB) return;
    const int l = window_of_hub(h);
    const int n = M.n, nw = (n + 31) >> 5;
    const int bound = l == 0 ? n : window_end(n, l) + 1;  // sources of the window lie below
    const Graph G = d ? Graph{M.trowptr, M.tcol} : Graph{M.rowptr, M.col};
    const long long at = lam_at(P, M, h, d);
    const int mine = (nw + (int)C - 1) >> shift;  // words of this CTA, at most
    int32_t* const lam = reinterpret_cast<int32_t*>(dyn_smem);
    const unsigned lam_a = (unsigned)__cvta_generic_to_shared(lam);
    const unsigned cnt_a = at_rank((unsigned)__cvta_generic_to_shared(cnt), 0);
    const unsigned quit_a = at_rank((unsigned)__cvta_generic_to_shared(quit), 0);
    const unsigned reached_a = at_rank((unsigned)__cvta_generic_to_shared(reached), 0);
    auto group_sync = [&]() {
        if (C == 1) __syncthreads();
        else cluster_sync();
    };
    auto lam_of = [&](int v) {
        const unsigned w = (unsigned)v >> 5;
        return at_rank(lam_a + 4 * (32 * (w >> shift) + ((unsigned)v & 31)), w & (C - 1));
    };
    int32_t* const q[2] = {P.lq + 2 * at, P.lq + 2 * at + M.hub_len};
    const int lane = threadIdx.x & 31;
    const int gw = (int)(rank * kLabelThreads + threadIdx.x) >> 5;
    const int nwarps = (int)C * (kLabelThreads / 32);
    for (int v = threadIdx.x; v < 32 * mine; v += kLabelThreads) lam[v] = kNoLabelWord;
    if (threadIdx.x == 0) {
        cnt[0] = 1;
        cnt[1] = cnt[2] = 0;
        quit[0] = quit[1] = 0;
        reached[0] = reached[1] = reached[2] = 0;
    }
    group_sync();
    if (rank == 0 && threadIdx.x == 0) {
        const int hub = hub_of(P, mi, h);
        dsm_min(lam_of(hub), label_queued(hub));
        __stcg(q[0], hub);
    }
    group_sync();
    int rounds = label_rounds(n, l), r = 0, count = 0;
    for (; r < rounds; r++) {
        count = dsm_ld(cnt_a + 4 * (r % 3));
        if (count == 0) break;
        if (r && r % kLook == 0 && dsm_ld(quit_a + 4 * (r / kLook % 2))) break;
        const int32_t* cur = q[r & 1];
        int32_t* const next = q[(r + 1) & 1];
        const unsigned nc = cnt_a + 4 * ((r + 1) % 3);
        if (rank == 0 && threadIdx.x == 0) cnt[(r + 2) % 3] = 0;
        // few ids queued: fewer per warp, so that more warps work
        const int per = count >= 32 * nwarps ? 32 : (count + nwarps - 1) / nwarps;
        for (int base = gw * per; base < count; base += nwarps * per) {
            int s0 = 0, its = 0, nl = 0;
            if (lane < per && base + lane < count) {
                const int u = __ldcg(cur + base + lane);
                const int a0 = __ldg(G.rp + u), a1 = __ldg(G.rp + u + 1);
                nl = label_queued(max(label_of_word(dsm_or(lam_of(u), kLabelIdle)), u));
                s0 = a0 & ~3;
                its = ((a1 & ~3) - s0) >> 2;
            }
            const int incl = warp_incl_sum(its, lane);
            const int total = __shfl_sync(FULL_MASK, incl, 31);
            int o;
            int p = flat_int4(lane, total, s0, its, incl, &o);
            int4 e = p >= 0 ? ld_row4<false>(G.cl + p) : make_int4(-1, -1, -1, -1);
            for (int j0 = 0; j0 < total; j0 += 32) {
                const int onl = __shfl_sync(FULL_MASK, nl, o);
                int4 en = make_int4(-1, -1, -1, -1);
                if (j0 + 32 < total) {
                    p = flat_int4(j0 + 32 + lane, total, s0, its, incl, &o);
                    if (p >= 0) en = ld_row4<false>(G.cl + p);
                }
                const int ws[4] = {e.x, e.y, e.z, e.w};
                int lw[4];
#pragma unroll
                for (int c = 0; c < 4; c++) lw[c] = ws[c] >= 0 ? dsm_ld(lam_of(ws[c])) : -1;
#pragma unroll
                for (int c = 0; c < 4; c++)
                    lw[c] = label_of_word(onl) < label_of_word(lw[c]) ? dsm_min(lam_of(ws[c]), onl) : -1;
                unsigned bal[4];
                int k = 0;
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    bal[c] = __ballot_sync(FULL_MASK, label_queues(lw[c], onl) && ws[c] < bound);
                    k += __popc(bal[c]);
                }
                if (k) {
                    int to = 0;
                    if (lane == 0) to = dsm_add(nc, k);
                    to = __shfl_sync(FULL_MASK, to, 0);
#pragma unroll
                    for (int c = 0; c < 4; c++) {
                        // a round lists an id once, so at most n
                        const int x = to + __popc(bal[c] & ((1u << lane) - 1u));
                        if (((bal[c] >> lane) & 1u) && x < M.hub_len) __stcg(next + x, ws[c]);
                        to += __popc(bal[c]);
                    }
                }
                e = en;
            }
        }
        // another search of the matrix may have found it to be left
        if (r % kLook == kLook - 1 && rank == 0 && threadIdx.x == 0)
            quit[(r + 1) / kLook % 2] = ld_vol_i32(P.fallback + mi);
        group_sync();
        if (l == 0 && r < kSpreadEnd && (r + 1) % kSpreadStep == 0 && r + 1 >= kSpread) {
            // ids reached so far (counted as they were reached, in every round: 1 to
            // 2 % more of a call, random n = 40,000 1.11 instead of 1.09 ms)
            int got = 0;
            for (int v = threadIdx.x; v < 32 * mine; v += kLabelThreads) got += lam[v] != kNoLabelWord;
            got = __reduce_add_sync(FULL_MASK, got);
            if (lane == 0 && got) dsm_add(reached_a + 4 * spread_part(r), got);
            group_sync();
            if (r == kSpreadEnd - 1) {
                const int all = dsm_ld(reached_a + 8), mid = dsm_ld(reached_a + 4), first = dsm_ld(reached_a);
                if (spreads(n, mid - first, all - mid)) {
                    if (rank == 0 && threadIdx.x == 0) atomicExch(P.fallback + mi, 1);
                    break;
                }
                if (settled(all, all - mid)) rounds = max(rounds, label_rounds_settled(n));
            }
        }
    }
    // unfinished labels are too large: the hub reaches nothing
    const bool none = r == rounds && dsm_ld(cnt_a + 4 * (r % 3)) != 0;
    if (none && rank == 0 && threadIdx.x == 0) give_up(P, mi, h);
    for (int w = (int)rank + (int)C * (threadIdx.x >> 5); w < nw; w += (int)C * (kLabelThreads / 32)) {
        // whole groups: the ids from n on have no label
        P.lam[at + 32ll * w + lane] = label_of_word(none ? kNoLabelWord : lam[32 * (w >> shift) + lane]);
    }
    group_sync();  // no CTA leaves while another may still read its counts
}

// The same by the whole GPU, one launch per round (labels, queues, counts in
// global memory): `per` CTAs a job, a launch that finds nothing queued ends at
// once; after the last, label_drop_kernel looks for unfinished searches.
__global__ void label_start_kernel(HubLaunch P) {
    const int job = blockIdx.x;
    const int mi = job / (2 * kHubs), h = (job >> 1) % kHubs, d = job & 1;
    const MatDesc& M = P.mats[mi];
    if (M.method != METHOD_HUB || threadIdx.x) return;
    const long long at = lam_at(P, M, h, d);
    const int hub = hub_of(P, mi, h);
    P.lam[at + hub] = hub;
    P.lq[2 * at] = hub;
    P.lcnt[8ll * job] = 1;
}

__global__ void __launch_bounds__(kLabelThreads) label_round_kernel(HubLaunch P, int per_job, int r) {
    const int job = blockIdx.x / per_job, part = blockIdx.x % per_job;
    int32_t* const cnt = P.lcnt + 8ll * job;
    int32_t* const reached = cnt + 4;  // ids first reached (see spreads)
    const int count = cnt[r % 3];
    if (part == 0 && threadIdx.x == 0) cnt[(r + 2) % 3] = 0;
    if (count == 0) return;
    const int mi = job / (2 * kHubs), h = (job >> 1) % kHubs, d = job & 1;
    const int lane = threadIdx.x & 31;
    int left = 0;
    if (lane == 0) left = ld_vol_i32(P.fallback + mi);
    if (__shfl_sync(FULL_MASK, left, 0)) return;
    const int l = window_of_hub(h);
    if (part == 0 && threadIdx.x == 0 && l == 0 && r == kSpreadEnd &&
        spreads(P.mats[mi].n, reached[1], reached[2]))
        atomicExch(P.fallback + mi, 1);
    const int gw = (part * kLabelThreads + threadIdx.x) >> 5;
    const int nwarps = per_job * (kLabelThreads / 32);
    // few ids queued: fewer per warp, so that more warps work
    const int per = count >= 32 * nwarps ? 32 : (count + nwarps - 1) / nwarps;
    if (gw * per >= count) return;
    const MatDesc& M = P.mats[mi];
    const int n = M.n;
    const int bound = l == 0 ? n : window_end(n, l) + 1;
    const Graph G = d ? Graph{M.trowptr, M.tcol} : Graph{M.rowptr, M.col};
    const long long at = lam_at(P, M, h, d);
    int got = 0;
    int32_t* const lam = P.lam + at;
    int32_t* const stamp = P.stamp + at;
    const int32_t* cur = P.lq + 2 * at + (r & 1) * M.hub_len;
    int32_t* const next = P.lq + 2 * at + ((r + 1) & 1) * M.hub_len;
    for (int base = gw * per; base < count; base += nwarps * per) {
        int s0 = 0, its = 0, nl = 0;
        if (lane < per && base + lane < count) {
            const int u = cur[base + lane];
            const int a0 = __ldg(G.rp + u), a1 = __ldg(G.rp + u + 1);
            nl = max(__ldcg(lam + u), u);
            s0 = a0 & ~3;
            its = ((a1 & ~3) - s0) >> 2;
        }
        const int incl = warp_incl_sum(its, lane);
        const int total = __shfl_sync(FULL_MASK, incl, 31);
        int o;
        int p = flat_int4(lane, total, s0, its, incl, &o);
        int4 e = p >= 0 ? ld_row4<false>(G.cl + p) : make_int4(-1, -1, -1, -1);
        for (int j0 = 0; j0 < total; j0 += 32) {
            const int onl = __shfl_sync(FULL_MASK, nl, o);
            int4 en = make_int4(-1, -1, -1, -1);
            if (j0 + 32 < total) {
                p = flat_int4(j0 + 32 + lane, total, s0, its, incl, &o);
                if (p >= 0) en = ld_row4<false>(G.cl + p);
            }
            const int ws[4] = {e.x, e.y, e.z, e.w};
            int lw[4], old[4];
#pragma unroll
            for (int c = 0; c < 4; c++) lw[c] = ws[c] >= 0 ? __ldcg(lam + ws[c]) : -1;
#pragma unroll
            for (int c = 0; c < 4; c++) old[c] = onl < lw[c] ? atomicMin(lam + ws[c], onl) : -1;
#pragma unroll
            for (int c = 0; c < 4; c++) got += old[c] == kNoLabel;
#pragma unroll
            for (int c = 0; c < 4; c++)
                old[c] = old[c] > onl && ws[c] < bound ? atomicExch(stamp + ws[c], r + 1) : r + 1;
            unsigned bal[4];
            int k = 0;
#pragma unroll
            for (int c = 0; c < 4; c++) {
                bal[c] = __ballot_sync(FULL_MASK, old[c] != r + 1);
                k += __popc(bal[c]);
            }
            if (k) {
                int to = 0;
                if (lane == 0) to = atomicAdd(cnt + (r + 1) % 3, k);
                to = __shfl_sync(FULL_MASK, to, 0);
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    // a round lists an id once, so at most n
                    const int x = to + __popc(bal[c] & ((1u << lane) - 1u));
                    if (((bal[c] >> lane) & 1u) && x < M.hub_len) next[x] = ws[c];
                    to += __popc(bal[c]);
                }
            }
            e = en;
        }
    }
    if (l == 0 && r < kSpreadEnd) {
        got = __reduce_add_sync(FULL_MASK, got);
        if (lane == 0 && got) atomicAdd(reached + spread_part(r), got);
    }
}

// Searches with ids still queued after the last round.
__global__ void label_drop_kernel(HubLaunch P, int per_job, int rounds) {
    const int job = blockIdx.x / per_job, part = blockIdx.x % per_job;
    if (P.lcnt[8ll * job + rounds % 3] == 0) return;
    const int mi = job / (2 * kHubs), h = (job >> 1) % kHubs, d = job & 1;
    const MatDesc& M = P.mats[mi];
    if (part == 0 && threadIdx.x == 0) give_up(P, mi, h);
    int32_t* const lam = P.lam + lam_at(P, M, h, d);
    for (long long v = part * blockDim.x + threadIdx.x; v < M.hub_len; v += per_job * blockDim.x) lam[v] = kNoLabel;
}

// The changes over s of the hub set's totals.  A warp per word: lane j is id
// v = 32 w + j, in the set from s = label + 1 on, above s until s = v.
__global__ void event_kernel(HubLaunch P, int per_job, int digests) {
    const int job = blockIdx.x / per_job, part = blockIdx.x % per_job;
    const int mi = job / (2 * kHubs), h = (job >> 1) % kHubs, d = job & 1;
    const MatDesc& M = P.mats[mi];
    if (M.method != METHOD_HUB || P.fallback[mi]) return;
    const int n = M.n;
    const int l = window_of_hub(h);
    const int lo = l == kWindows - 1 ? 0 : window_end(n, l + 1) + 1;  // the window's sources
    const int hi = l == 0 ? n - 1 : window_end(n, l);
    if (lo > hi) return;
    const int32_t* lam = P.lam + lam_at(P, M, h, d);
    Tot* const D = P.base + (2ll * (h == 1) + d) * P.total + M.hub_off;
    const int lane = threadIdx.x & 31;
    const int nw = (n + 31) >> 5;
    for (int w = (part * blockDim.x + threadIdx.x) >> 5; w < nw; w += (per_job * blockDim.x) >> 5) {
        const int v = 32 * w + lane;
        const int lv = v < n ? __ldg(lam + v) : INT_MAX;
        int in = -1, out = -1, ve = -1, deg = 0;
        if (lv < hi) {
            in = max(lv + 1, lo);
            out = min(v, hi + 1);
            if (in >= out) in = out = -1;
            ve = max(max(lv, v) + 1, lo);
            if (ve > hi) ve = -1;
            else if (d == 0) deg = row_degree<false>(M.rowptr, v);
        }
        if (!__any_sync(FULL_MASK, in >= 0 || ve >= 0)) continue;
        uint32_t m_in = 0, m_in1 = 0, m_out = 0, m_out1 = 0;  // the word at and before the lane's times
        int c_in = 0, c_out = 0, c_ve = 0;
        unsigned long long s_ve = 0;
        bool lead_in = in >= 0, lead_out = out >= 0, lead_ve = ve >= 0, in_at_out = false;
        for (int i = 0; i < 32; i++) {
            const int ti = __shfl_sync(FULL_MASK, in, i), to = __shfl_sync(FULL_MASK, out, i);
            const int te = __shfl_sync(FULL_MASK, ve, i), dg = __shfl_sync(FULL_MASK, deg, i);
            const uint32_t bit = 1u << i;
            if (ti >= 0) {
                if (ti <= in && in < to) m_in |= bit;
                if (ti <= in - 1 && in - 1 < to) m_in1 |= bit;
                if (ti <= out && out < to) m_out |= bit;
                if (ti <= out - 1 && out - 1 < to) m_out1 |= bit;
                if (ti == in) {
                    c_in++;
                    if (i < lane) lead_in = false;
                }
                if (to == out) {
                    c_out++;
                    if (i < lane) lead_out = false;
                }
                if (ti == out) in_at_out = true;
            }
            if (te >= 0 && te == ve) {
                c_ve++;
                s_ve += (unsigned)dg;
                if (i < lane) lead_ve = false;
            }
        }
        if (lead_in) {
            atomicAdd(&D[in].gt, c_in);
            if (digests) atomicAdd(&D[in].dig, word_digest(w, m_in) - word_digest(w, m_in1));
        }
        if (lead_out) {
            atomicAdd(&D[out].gt, -c_out);
            if (digests && !in_at_out)
                atomicAdd(&D[out].dig, word_digest(w, m_out) - word_digest(w, m_out1));
        }
        if (lead_ve) {
            atomicAdd(&D[ve].v, c_ve);
            if (d == 0) atomicAdd(&D[ve].e, s_ve);
        }
        // the ids below s leave with the window
        const int all = __reduce_add_sync(FULL_MASK, ve >= 0 ? 1 : 0);
        const unsigned long long sum = warp_sum64((unsigned long long)(unsigned)deg);
        if (lane == 0 && all) {
            atomicAdd(&D[hi + 1].v, -all);
            if (d == 0) atomicAdd(&D[hi + 1].e, 0ull - sum);
        }
    }
}

struct TotSum {
    __host__ __device__ Tot operator()(const Tot& a, const Tot& b) const {
        return Tot{a.gt + b.gt, a.v + b.v, a.e + b.e, a.dig + b.dig};
    }
};

// A search's base: the hub's labels in its direction (null: none), and the
// totals of the hub's set.
struct Base {
    const int32_t* lam;
    Tot t;
    int hub;
};

__device__ __forceinline__ Base base_of(const HubLaunch& P, const MatDesc& M, int s, int d, bool sym) {
    Base b{nullptr, {0, 0, 0ull, 0ull}, 0};
    if (M.method != METHOD_HUB) return b;
    const int l = window_of(M.n, s);
    // the hubs s reaches; of two the one that reaches more
    for (int h = l == 0 ? 0 : l + 1; h <= (l == 0 ? 1 : l + 1); h++) {
        if (__ldg(P.lam + lam_at(P, M, h, sym ? d : 1 - d) + s) >= s) continue;
        const Tot t = P.base[(2ll * (h == 1) + d) * P.total + M.hub_off + s];
        if (b.lam && t.gt + t.v <= b.t.gt + b.t.v) continue;
        b.lam = P.lam + lam_at(P, M, h, d);
        b.t = t;
        b.hub = h;
    }
    return b;
}

// Per-row L statistics of L column s: the ids `bits` (of word w, above s) that
// its search found.
__device__ __forceinline__ void lrow_found(const MatDesc& M, int w, uint32_t bits, int s) {
    const unsigned long long ds = mix64((uint64_t)(uint32_t)s);
    for (; bits; bits &= bits - 1) {
        const int v = 32 * w + __ffs(bits) - 1;
        atomicAdd(&M.nnz_lr[v], 1);
        atomicAdd((unsigned long long*)&M.dig_lr[v], ds);
    }
}

// That column s also holds its hub's set above s: noted for lrow_kernel.
__device__ __forceinline__ void lrow_hub(const HubLaunch& P, const MatDesc& M, const Base& b, int s) {
    if (b.lam) P.l_use[(long long)b.hub * P.total + M.hub_off + s] = LRowUse{1ull, mix64((uint64_t)(uint32_t)s)};
}

// the hub set's ids above s in word w
__device__ __forceinline__ uint32_t base_word(const Base& b, int w, int s, int n) {
    if (!b.lam) return 0u;
    uint32_t m = 0;
    const int4* p = reinterpret_cast<const int4*>(b.lam + 32 * w);
#pragma unroll
    for (int k = 0; k < 8; k++) {
        const int4 x = __ldg(p + k);  // the array is padded to whole words
        m |= (x.x < s ? 1u : 0u) << (4 * k) | (x.y < s ? 2u : 0u) << (4 * k) |
             (x.z < s ? 4u : 0u) << (4 * k) | (x.w < s ? 8u : 0u) << (4 * k);
    }
    return m & above(w, s);
}

// Bits of the hub's set among the 128 ids after s: word `lane` for lanes 0..3.
__device__ __forceinline__ uint32_t base_next128(const Base& b, int s, int n) {
    const int lane = threadIdx.x & 31;
    uint32_t mine = 0;
    if (!b.lam) return 0u;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const int v = s + 1 + 32 * j + lane;
        const uint32_t x = __ballot_sync(FULL_MASK, v < n && __ldg(b.lam + v) < s);
        if (lane == j) mine = x;
    }
    return mine;
}

__global__ void __launch_bounds__(kExtraThreads, 1024 / kExtraThreads) extra_kernel(HubLaunch P) {
    extern __shared__ uint4 dyn_smem[];
    const int lane = threadIdx.x & 31;
    WarpTable& T = reinterpret_cast<WarpTable*>(dyn_smem)[threadIdx.x >> 5];
    bool dirty = true;
    for (;;) {
        unsigned long long item = 0;
        if (lane == 0) item = atomicAdd(P.work_counter, 1ull);
        item = __shfl_sync(FULL_MASK, item, 0);
        if ((long long)item >= P.total_items) return;
        int mi = 0;
        {
            int lo = 0, hi = P.nmats - 1;
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (P.mats[mid].hub_item <= (long long)item) lo = mid;
                else hi = mid - 1;
            }
            mi = lo;
        }
        const MatDesc& M = P.mats[mi];
        // one lane looks: another warp may set the flag between two lanes' loads
        int left = 0;
        if (lane == 0) left = ld_vol_i32(P.fallback + mi);
        if (__shfl_sync(FULL_MASK, left, 0)) continue;
        const int n = M.n;
        const bool sym = M.asym[0] == 0;
        const bool digests = M.dig_u != nullptr;
        const int dirs = sym ? 1 : 2;
        const int groups = (n + P.group - 1) / P.group;
        // the matrix's items in an order that spreads the first ones over all
        // of it (an odd multiplier permutes a power of two)
        const unsigned slots = (unsigned)M.hub_slots;
        const unsigned x = ((unsigned)((long long)item - M.hub_item) * 0x9E3779B1u) & (slots - 1);
        if (x >= (unsigned)(groups * dirs)) continue;
        const int d = sym ? 0 : (int)(x & 1u);
        const int g = sym ? (int)x : (int)(x >> 1);
        const Graph G = d ? Graph{M.trowptr, M.tcol} : Graph{M.rowptr, M.col};
        const int s_first = g * P.group, s_end = min(n, s_first + P.group);
        unsigned long long a_fill = 0, a_e = 0, a_v = 0, a_nnz = 0, a_trav = 0;
        int a_hub = 0, judged = s_first;  // the item's sources below `judged` have been counted
        bool abandoned = false;
        int r0 = __ldg(G.rp + s_first), r1 = __ldg(G.rp + s_first + 1);
        int4 pre = make_int4(-1, -1, -1, -1);
        if (4 * lane < (r1 & ~3) - (r0 & ~3)) pre = ld_row4<false>(G.cl + (r0 & ~3) + 4 * lane);
        for (int s = s_first; s < s_end; s++) {
            const int r2 = s + 2 <= n ? __ldg(G.rp + s + 2) : r1;
            const Base B = base_of(P, M, s, d, sym);
            if (dirty) {
                for (int i = lane; i < kSlots; i += 32) {
                    T.key[i] = kFree;
                    T.msk[i] = 0u;
                }
                dirty = false;
                __syncwarp();
            }
            int found = 0, words = 0, raw = 0, v = 0, trav = 0;
            unsigned e = 0;
            bool large = false;
            auto visit = [&](const int4& q4, bool own_row) -> bool {
                const int ws[4] = {q4.x, q4.y, q4.z, q4.w};
                bool todo[4];
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    todo[c] = ws[c] >= 0 && ws[c] != s;
                    if (own_row) raw += ws[c] > s;
                }
                if (B.lam) {
                    int lw[4];
#pragma unroll
                    for (int c = 0; c < 4; c++) lw[c] = todo[c] ? __ldg(B.lam + ws[c]) : -1;
#pragma unroll
                    for (int c = 0; c < 4; c++) todo[c] = todo[c] && lw[c] >= s;
                }
                if (!__any_sync(FULL_MASK, todo[0] || todo[1] || todo[2] || todo[3])) return true;
                dirty = true;
                int nslots = 0, k = 0;
                bool full = false;
                unsigned bal[4];
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    bool fresh = false;
                    if (todo[c]) {
                        const int i = sparse_slot(T.key, ws[c] >> 5, &nslots);
                        const uint32_t bit = 1u << (ws[c] & 31);
                        if (i < 0) full = true;
                        else fresh = !(atomicOr(T.msk + i, bit) & bit);
                    }
                    bal[c] = __ballot_sync(FULL_MASK, fresh);
                    k += __popc(bal[c]);
                }
                words += __reduce_add_sync(FULL_MASK, nslots);
                int to = found;
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    if ((bal[c] >> lane) & 1u) T.list[to + __popc(bal[c] & ((1u << lane) - 1u))] = ws[c];
                    to += __popc(bal[c]);
                }
                found = to;
                __syncwarp();
                return found <= kListCap && words <= kSlotsMax && !__any_sync(FULL_MASK, full);
            };
            {
                const int b = r0 & ~3, plen = (r1 & ~3) - b;
                int4 q4 = pre;
                for (int k0 = 0; k0 < plen && !large; k0 += 128) {
                    int4 qn = make_int4(-1, -1, -1, -1);
                    if (k0 + 128 + 4 * lane < plen) qn = ld_row4<false>(G.cl + b + k0 + 128 + 4 * lane);
                    large = !visit(q4, true);
                    q4 = qn;
                }
                trav += plen;
            }
            pre = make_int4(-1, -1, -1, -1);
            if (4 * lane < (r2 & ~3) - (r1 & ~3)) pre = ld_row4<false>(G.cl + (r1 & ~3) + 4 * lane);
            for (int h = 0; h < found && !large;) {
                const int end = found;
                const int u = h + lane < end ? T.list[h + lane] : INT_MAX;
                int s0 = 0, its = 0;
                if (u < s) {
                    const int a0 = __ldg(G.rp + u), a1 = __ldg(G.rp + u + 1);
                    s0 = a0 & ~3;
                    its = ((a1 & ~3) - s0) >> 2;
                    v++;
                    e += (unsigned)(4 * its - (a1 & 3));
                }
                const int incl = warp_incl_sum(its, lane);
                const int total = __shfl_sync(FULL_MASK, incl, 31);
                trav += 4 * total;
                int o;
                int at = flat_int4(lane, total, s0, its, incl, &o);
                int4 q4 = at >= 0 ? ld_row4<false>(G.cl + at) : make_int4(-1, -1, -1, -1);
                for (int j0 = 0; j0 < total && !large; j0 += 32) {
                    int4 qn = make_int4(-1, -1, -1, -1);
                    if (j0 + 32 < total) {
                        at = flat_int4(j0 + 32 + lane, total, s0, its, incl, &o);
                        if (at >= 0) qn = ld_row4<false>(G.cl + at);
                    }
                    large = !visit(q4, false);
                    q4 = qn;
                }
                h = min(h + 32, end);
            }
            if (large) {
                int left = 0;
                if (lane == 0) {
                    // room for every (source, direction) of the launch
                    const int p = atomicAdd(P.large_count, 1);
                    P.large[p] = (unsigned long long)mi << 33 | (unsigned long long)d << 32 | (unsigned)s;
                    const int done = atomicAdd(P.judged + 2 * mi, s + 1 - judged) + s + 1 - judged;
                    const int big = atomicAdd(P.judged + 2 * mi + 1, 1) + 1;
                    if (n > kDirectMax && ((done >= kJudgeEarly && 2ll * big > done) ||
                                           (done >= kJudgeAfter && 4ll * big > done)))
                        atomicExch(P.fallback + mi, 1);
                    left = ld_vol_i32(P.fallback + mi);
                }
                judged = s + 1;
                abandoned = __shfl_sync(FULL_MASK, left, 0) != 0;
                if (abandoned) break;
            } else {
                Tot t = B.t;
                raw = __reduce_add_sync(FULL_MASK, raw);
                if (found) {
                    // the found ids word by word: occupied slots listed first
                    int k = 0;
                    __syncwarp();
                    for (int i = lane; i < kSlots; i += 32) {
                        const bool has = T.key[i] != kFree && (T.msk[i] & above((int)T.key[i], s));
                        const unsigned b = __ballot_sync(FULL_MASK, has);
                        if (has) T.list[k + __popc(b & ((1u << lane) - 1u))] = i;
                        k += __popc(b);
                    }
                    __syncwarp();
                    int gt = 0;
                    unsigned long long dig = 0;
                    for (int i = lane; i < k; i += 32) {
                        const int slot = T.list[i];
                        const int w = (int)T.key[slot];
                        const uint32_t hi = T.msk[slot] & above(w, s);
                        gt += __popc(hi);
                        if (M.nnz_lr && (d == 1 || sym)) lrow_found(M, w, hi, s);
                        if (digests) {
                            const uint32_t bw = base_word(B, w, s, n);
                            dig += word_digest(w, bw | hi) - word_digest(w, bw);
                        }
                    }
                    t.gt += __reduce_add_sync(FULL_MASK, gt);
                    t.v += __reduce_add_sync(FULL_MASK, v);
                    t.e += (unsigned)__reduce_add_sync(FULL_MASK, e);
                    if (digests && k) t.dig += warp_sum64(dig);
                }
                if (lane == 0) {
                    write_row(M, s, d, sym, t, raw, raw);
                    if (M.nnz_lr && (d == 1 || sym)) lrow_hub(P, M, B, s);
                }
                if (d == 1 || sym) {
                    uint32_t word = base_next128(B, s, n);
                    if (found) {
                        const uint32_t x5 = lane < 5 ? sparse_word(T.key, T.msk, ((s + 1) >> 5) + lane) : 0u;
                        word |= next128(x5, s);
                    }
                    if (lane < 4) M.lmask[4ll * s + lane] = word;
                }
                a_fill += (unsigned long long)(t.gt - raw) * (sym ? 2 : 1);
                a_nnz += (unsigned)t.gt;
                a_trav += (unsigned)trav;
                a_hub += B.lam != nullptr;
                if (d == 0) {
                    a_e += t.e;
                    a_v += (unsigned)t.v;
                }
            }
            r0 = r1;
            r1 = r2;
        }
        if (lane == 0 && !abandoned) {
            unsigned long long* c = P.counters + (long long)mi * CNT_SLOTS;
            atomicAdd(c + CNT_FILLS, a_fill);
            atomicAdd(c + CNT_EDGES_TRAV, a_trav);
            if (d == 0) {
                atomicAdd(c + CNT_EDGES_ALG, a_e);
                atomicAdd(c + CNT_VERTS_ALG, a_v);
                atomicAdd(c + CNT_NNZ_U, a_nnz);
            }
            if (d == 1 || sym) atomicAdd(c + CNT_NNZ_L, a_nnz);
            if (a_hub) atomicAdd(c + CNT_CHAINED, (unsigned long long)a_hub);
            atomicAdd(P.judged + 2 * mi, s_end - judged);
        }
    }
}

template <int BLOCK>
__global__ void __launch_bounds__(BLOCK, 1024 / BLOCK) large_kernel(HubLaunch P) {
    extern __shared__ uint4 dyn_smem[];
    __shared__ BfsSmem<BLOCK> bfs;
    __shared__ long long item;
    __shared__ unsigned long long red[BLOCK / 32][4];
    __shared__ int row[2];
    const int lane = threadIdx.x & 31;
    uint32_t* const bm = P.large_smem ? reinterpret_cast<uint32_t*>(dyn_smem)
                                      : P.gbm + (long long)blockIdx.x * P.bitmap_words;
    int32_t* const q = P.queue + (long long)blockIdx.x * P.queue_stride;
    const int count = *P.large_count;
    if (count == 0) return;
    for (long long i = threadIdx.x; i < P.bitmap_words; i += BLOCK) bm[i] = 0u;
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) {
            const unsigned long long k = atomicAdd(P.work_counter + 1, 1ull);
            item = k < (unsigned long long)count ? (long long)P.large[k] : -1;
            // (one thread looks: another CTA may set the flag)
            if (item >= 0 && ld_vol_i32(P.fallback + (int)(item >> 33))) item = -2;
        }
        __syncthreads();
        if (item == -1) return;
        if (item < 0) continue;
        const int mi = (int)(item >> 33), d = (int)(item >> 32) & 1, s = (int)(item & 0xffffffff);
        const MatDesc& M = P.mats[mi];
        const int n = M.n, nw = (n + 31) >> 5;
        const bool sym = M.asym[0] == 0;
        const bool digests = M.dig_u != nullptr;
        const Graph G = d ? Graph{M.trowptr, M.tcol} : Graph{M.rowptr, M.col};
        const Base B = base_of(P, M, s, d, sym);
        if (threadIdx.x < 32) {
            const int b = __ldg(G.rp + s) & ~3, e = __ldg(G.rp + s + 1) & ~3;
            int raw = 0;
            for (int j = b + lane; j < e; j += 32) raw += __ldg(G.cl + j) > s;
            raw = __reduce_add_sync(FULL_MASK, raw);
            if (lane == 0) {
                row[0] = raw;
                bfs.rtrav = 0;
                q[0] = s;
            }
        }
        __syncthreads();
        if (B.lam)
            block_bfs<BLOCK, false, true>(bfs, G, bm, q, P.queue_stride, 1, s, s, false, P.status, B.lam);
        else
            block_bfs<BLOCK, false, false>(bfs, G, bm, q, P.queue_stride, 1, s, s, false, P.status);
        unsigned long long vals[4] = {0, 0, 0, 0};  // found above, below, degrees below, digest change
        for (int w = threadIdx.x; w < nw; w += BLOCK) {
            const uint32_t x = bm[w];
            if (!x) continue;
            const uint32_t hi = x & above(w, s), low = x & below(w, s);
            vals[0] += __popc(hi);
            vals[1] += __popc(low);
            if (M.nnz_lr && (d == 1 || sym)) lrow_found(M, w, hi, s);
            if (digests && hi) {
                const uint32_t bw = base_word(B, w, s, n);
                vals[3] += word_digest(w, bw | hi) - word_digest(w, bw);
            }
            if (d != 0 || !low) continue;
            if (__popc(low) <= 2) {
                for (uint32_t t = low; t; t &= t - 1)
                    vals[2] += (unsigned)row_degree<false>(M.rowptr, 32 * w + __ffs(t) - 1);
            } else {
                for (int k = 0; k < M.nplanes; k++)
                    vals[2] += (unsigned long long)__popc(low & __ldg(M.dplanes + (long long)k * nw + w)) << k;
            }
        }
#pragma unroll
        for (int j = 0; j < 4; j++) {
            vals[j] = warp_sum64(vals[j]);
            if (lane == 0) red[threadIdx.x >> 5][j] = vals[j];
        }
        __syncthreads();
        if (threadIdx.x < 32) {
            if (d == 1 || sym) {
                uint32_t word = base_next128(B, s, n);
                word |= next128(lane < 5 ? bm[((s + 1) >> 5) + lane] : 0u, s);
                if (lane < 4) M.lmask[4ll * s + lane] = word;
            }
            if (lane == 0) {
                Tot t = B.t;
                for (int i = 0; i < BLOCK / 32; i++) {
                    t.gt += (int)red[i][0];
                    t.v += (int)red[i][1];
                    t.e += red[i][2];
                    t.dig += red[i][3];
                }
                write_row(M, s, d, sym, t, row[0], row[0]);
                if (M.nnz_lr && (d == 1 || sym)) lrow_hub(P, M, B, s);
                unsigned long long* c = P.counters + (long long)mi * CNT_SLOTS;
                atomicAdd(c + CNT_FILLS, (unsigned long long)(t.gt - row[0]) * (sym ? 2 : 1));
                atomicAdd(c + CNT_EDGES_TRAV, bfs.rtrav);
                if (d == 0) {
                    atomicAdd(c + CNT_EDGES_ALG, t.e);
                    atomicAdd(c + CNT_VERTS_ALG, (unsigned long long)(unsigned)t.v);
                    atomicAdd(c + CNT_NNZ_U, (unsigned long long)(unsigned)t.gt);
                }
                if (d == 1 || sym) atomicAdd(c + CNT_NNZ_L, (unsigned long long)(unsigned)t.gt);
                if (B.lam) atomicAdd(c + CNT_CHAINED, 1ull);
                // how many of the matrix's large searches are done, and the entries they read
                const unsigned long long done = atomicAdd(P.large_work + 2 * mi, 1ull) + 1;
                const unsigned long long read = atomicAdd(P.large_work + 2 * mi + 1, bfs.rtrav) + bfs.rtrav;
                if (n > kDirectMax && done >= kLargeSample &&
                    (double)read / (double)done * P.judged[2 * mi + 1] > kLargePerRow * n)
                    atomicExch(P.fallback + mi, 1);
            }
        }
        __syncthreads();
        block_clear<BLOCK>(bm, nw);
    }
}

struct UseSum {
    __host__ __device__ LRowUse operator()(const LRowUse& a, const LRowUse& b) const {
        return LRowUse{a.count + b.count, a.dig + b.dig};
    }
};

// Per-row L statistics from the hubs' sets: row v is in the set of column s
// when label(v) < s < v, so it gains the columns that took hub h's set between
// those two ids: a difference of prefix sums (l_use, scanned).
__global__ void lrow_kernel(HubLaunch P, int per_mat) {
    const int mi = blockIdx.x / per_mat, part = blockIdx.x % per_mat;
    const MatDesc& M = P.mats[mi];
    if (M.method != METHOD_HUB || P.fallback[mi]) return;
    const int d = M.asym[0] == 0 ? 0 : 1;
    for (int v = part * blockDim.x + threadIdx.x; v < M.n; v += per_mat * blockDim.x) {
        unsigned long long count = 0, dig = 0;
        for (int h = 0; h < kHubs; h++) {
            const int l = __ldg(P.lam + lam_at(P, M, h, d) + v);
            if (l >= v - 1) continue;
            const LRowUse* u = P.l_use + (long long)h * P.total + M.hub_off;
            const LRowUse a = u[l], b = u[v - 1];
            count += b.count - a.count;
            dig += b.dig - a.dig;
        }
        if (!count) continue;
        M.nnz_lr[v] += (int)count;
        M.dig_lr[v] += dig;
    }
}

// The counters of every matrix that was not left.
__global__ void commit_kernel(HubLaunch P) {
    const int mi = blockIdx.x;
    const MatDesc& M = P.mats[mi];
    if ((M.method == METHOD_HUB || M.method == METHOD_DIRECT) && !P.fallback[mi] && threadIdx.x < CNT_SLOTS)
        M.counters[threadIdx.x] += P.counters[(long long)mi * CNT_SLOTS + threadIdx.x];
}

}  // namespace


int hub_count() { return kHubs; }
int hub_bases() { return kBases; }
int extra_ctas_per_sm() { return 1024 / kExtraThreads; }

// The largest cluster's shared memory per CTA for a matrix of order n.
size_t label_smem_bytes(int32_t n, int cluster) {
    const size_t words = (((size_t)n + 31) / 32 + (size_t)cluster - 1) / (size_t)cluster;
    return 32 * 4 * words + 16;
}

size_t hub_scan_bytes(long long tots, long long uses) {
    size_t b = 0, c = 0;
    cub::DeviceScan::InclusiveScan(nullptr, b, (const Tot*)nullptr, (Tot*)nullptr, TotSum(), (int)tots);
    if (uses)
        cub::DeviceScan::InclusiveScan(nullptr, c, (const LRowUse*)nullptr, (LRowUse*)nullptr, UseSum(), (int)uses);
    return std::max(b, c);
}

int large_occupancy(size_t smem) {
    int occ = 0;
    cudaError_t e = allow_shared_memory<large_kernel<kLargeThreads>>();
    if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, large_kernel<kLargeThreads>, kLargeThreads, smem);
    if (e != cudaSuccess) cudaGetLastError();
    return e == cudaSuccess ? occ : 0;
}

static cudaError_t label_config(cudaLaunchConfig_t* cfg, cudaLaunchAttribute* attr, int jobs, int cluster,
                                size_t smem, cudaStream_t st) {
    cudaError_t e = allow_shared_memory<label_cluster_kernel>();
    if (e == cudaSuccess && cluster > 8)
        e = cudaFuncSetAttribute(label_cluster_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    *cfg = cudaLaunchConfig_t{};
    cfg->gridDim = dim3((unsigned)(jobs * cluster));
    cfg->blockDim = dim3(kLabelThreads);
    cfg->dynamicSmemBytes = smem;
    cfg->stream = st;
    attr->id = cudaLaunchAttributeClusterDimension;
    attr->val.clusterDim.x = (unsigned)cluster;
    attr->val.clusterDim.y = attr->val.clusterDim.z = 1;
    cfg->attrs = attr;
    cfg->numAttrs = 1;
    return e;
}

// The widest cluster that this GPU can place with `smem` bytes per CTA; 0: none.
int label_max_cluster(size_t smem) {
    for (int c = 16; c > 0; c /= 2) {
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute attr;
        int n = 0;
        cudaError_t e = label_config(&cfg, &attr, 1, c, smem, nullptr);
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&n, label_cluster_kernel, &cfg);
        if (e == cudaSuccess && n > 0) return c;
        cudaGetLastError();
    }
    return 0;
}

size_t hub_load_bytes() { return hub_scan_bytes(2, 2) + 256 + 2 * sizeof(Tot); }

cudaError_t hub_load(void* scratch, cudaStream_t st) {
    cudaFuncAttributes fa;
    const void* const kernels[] = {(const void*)hub_kernel,        (const void*)label_cluster_kernel,
                                   (const void*)label_start_kernel, (const void*)label_round_kernel,
                                   (const void*)label_drop_kernel,  (const void*)event_kernel,
                                   (const void*)extra_kernel,       (const void*)large_kernel<kLargeThreads>,
                                   (const void*)commit_kernel};
    cudaError_t e = cudaSuccess;
    for (const void* k : kernels)
        if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, k);
    Tot* const two = static_cast<Tot*>(scratch);
    size_t sb = hub_scan_bytes(2, 2);
    if (e == cudaSuccess) e = cudaMemsetAsync(two, 0, 2 * sizeof(Tot), st);
    if (e == cudaSuccess)
        e = cub::DeviceScan::InclusiveScan(static_cast<char*>(scratch) + 256, sb, two, two, TotSum(), 2, st);
    return e;
}

// CTAs for each of `jobs` jobs of at most `most` CTAs' work: together no more than
// some tens of waves.
static int parts(int most, int jobs) { return std::max(1, std::min({most, 1024, (1 << 17) / jobs})); }

cudaError_t launch_hub(const HubLaunch& L, const HubCfg& c, int digests, cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(L.zeroed, 0, c.zeroed_bytes, st);
    if (e != cudaSuccess) return e;
    if (c.any_hub) {
        // (grids are one-dimensional: a batch may have more jobs than the 65,535
        // that a second dimension takes)
        const int jobs = L.hub_mats * 2 * kHubs;
        hub_kernel<<<dim3((unsigned)(L.hub_mats * kHubs), 16), 256, 0, st>>>(L);
        if (c.cluster > 0) {
            cudaLaunchConfig_t cfg;
            cudaLaunchAttribute attr;
            e = label_config(&cfg, &attr, jobs, c.cluster, label_smem_bytes(c.n_max, c.cluster), st);
            if (e == cudaSuccess) e = cudaLaunchKernelEx(&cfg, label_cluster_kernel, L);
            if (e != cudaSuccess) return e;
        } else {
            e = cudaMemsetAsync(L.lam, 0x7f, 4ull * 2 * kHubs * (size_t)L.total, st);
            if (e != cudaSuccess) return e;
            label_start_kernel<<<jobs, 32, 0, st>>>(L);
            // two CTAs per SM over a matrix's eight jobs: a round without work costs
            // its CTAs' launch (n = 1,200,000: 16 CTAs per SM 38 ms, two 33)
            const int per = std::max(8, c.sm_count / (4 * std::min(L.hub_mats, 8)));
            const int rounds = label_rounds(c.n_max, 0);
            for (int r = 0; r < rounds; r++) label_round_kernel<<<per * jobs, kLabelThreads, 0, st>>>(L, per, r);
            label_drop_kernel<<<per * jobs, kLabelThreads, 0, st>>>(L, per, rounds);
        }
        const int words = (int)((c.n_max + 31) / 32);
        const int per = parts((words + 7) / 8, jobs);
        event_kernel<<<per * jobs, 256, 0, st>>>(L, per, digests);
        size_t sb = c.scan_bytes;
        e = cub::DeviceScan::InclusiveScan(c.scan_tmp, sb, L.base, L.base, TotSum(), (int)(2 * kBases * L.total), st);
        if (e != cudaSuccess) return e;
    }
    const size_t smem = sizeof(WarpTable) * (kExtraThreads / 32);
    if ((e = allow_shared_memory<extra_kernel>()) != cudaSuccess) return e;
    const long long want = (L.total_items + kExtraThreads / 32 - 1) / (kExtraThreads / 32);
    extra_kernel<<<(int)std::min<long long>(want, c.extra_grid), kExtraThreads, smem, st>>>(L);
    large_kernel<kLargeThreads><<<c.large_grid, kLargeThreads, c.large_smem, st>>>(L);
    if (c.any_hub && c.l_rows) {
        size_t sb = c.scan_bytes;
        e = cub::DeviceScan::InclusiveScan(c.scan_tmp, sb, L.l_use, L.l_use, UseSum(), (int)(kHubs * L.total), st);
        if (e != cudaSuccess) return e;
        const int per = parts((c.n_max + 255) / 256, L.hub_mats);
        lrow_kernel<<<per * L.hub_mats, 256, 0, st>>>(L, per);
    }
    commit_kernel<<<L.nmats, 32, 0, st>>>(L);
    return cudaGetLastError();
}

}  // namespace gsofa
