// Device helpers shared by the traversal kernels (gsofa_kernels.cu,
// gsofa_chain.cu): loads, digests, work-item lookup and serving claims.
#pragma once
#include <atomic>

#include "gsofa_internal.h"

namespace gsofa {

#define FULL_MASK 0xffffffffu

// Lets a kernel's launches ask for all the dynamic shared memory a CTA may
// have.  The limit belongs to the function, for every thread of the process: one
// set to a launch's own need could be lowered by another thread before that
// launch.
template <auto KERNEL>
cudaError_t allow_shared_memory() {
    static std::atomic<int> limits[64];  // per device, once known
    int dev = 0, most = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    int limit = dev < 64 ? limits[dev].load(std::memory_order_relaxed) : 0;
    if (limit == 0) {
        cudaFuncAttributes fa;
        e = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
        if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, KERNEL);
        if (e != cudaSuccess) return e;
        limit = most - (int)fa.sharedSizeBytes;
        if (dev < 64) limits[dev].store(limit, std::memory_order_relaxed);
    }
    return cudaFuncSetAttribute(KERNEL, cudaFuncAttributeMaxDynamicSharedMemorySize, limit);
}

// Digest mixing: splitmix64 finaliser (Steele, Lea, Flood 2014).  A U-row
// or L-column digest sums mix64((w << 32) | mask) over the set's non-zero
// 32-id words w; an L-row digest (scattered) sums mix64(id) over its ids.
__host__ __device__ __forceinline__ uint64_t mix64(uint64_t x) {
    x += 0x9E3779B97F4A7C15ull;
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
    return x ^ (x >> 31);
}

template <long long MatDesc::*BASE = &MatDesc::item_base>
__device__ __forceinline__ int find_matrix(const MatDesc* mats, int nmats, long long item) {
    int lo = 0, hi = nmats - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (mats[mid].*BASE <= item) lo = mid; else hi = mid - 1;
    }
    return lo;
}

__device__ __forceinline__ uint32_t ld_vol(const uint32_t* p) {
    return *reinterpret_cast<const volatile uint32_t*>(p);
}

// Loads of matrix data.  CG = false: the read-only path (L1-cached), valid
// because nothing writes a matrix while a launch reads it.  CG = true (the
// serving kernel): L2 only.  A serving launch outlives the matrices it reads;
// their memory is freed and reused for later requests while it runs, so a
// line it once cached in L1 could be stale.
template <bool CG>
__device__ __forceinline__ int ld_i32(const int32_t* p) {
    return CG ? __ldcg(p) : __ldg(p);
}

template <bool CG>
__device__ __forceinline__ int4 ld_row4(const int32_t* p) {
    const int4* q = reinterpret_cast<const int4*>(p);
    return CG ? __ldcg(q) : __ldg(q);
}

// Original (unpadded) length of row v of a padded graph.
template <bool CG>
__device__ __forceinline__ int row_degree(const int32_t* rp, int v) {
    const int a = ld_i32<CG>(rp + v), b = ld_i32<CG>(rp + v + 1);
    return (b & ~3) - (a & ~3) - (b & 3);
}

// Bitmap words of a matrix of order n: n bits plus zero padding read by the
// 128-bit L-mask extraction past the last vertex.
__host__ __device__ __forceinline__ long long bitmap_words_for(int32_t n) {
    return (((long long)n + 31) >> 5) + 6;
}

__device__ __forceinline__ unsigned long long ld_vol64(const unsigned long long* p) {
    return *reinterpret_cast<const volatile unsigned long long*>(p);
}

__device__ __forceinline__ int ld_vol_i32(const int32_t* p) {
    return *reinterpret_cast<const volatile int32_t*>(p);
}

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Whether this CTA's SM belongs to the other serving kernel now.
__device__ __forceinline__ bool serve_elsewhere(const ServeLaunch& V) {
    unsigned sm;
    asm volatile("mov.u32 %0, %%smid;" : "=r"(sm));
    return V.kind == SERVE_CHAIN
               ? (int)sm >= ld_vol_i32(V.ctrl + 5)
               : (int)sm < ld_vol_i32(V.ctrl + 6) || (int)sm >= ld_vol_i32(V.ctrl + 7);
}

// Serving, called by all 32 lanes of warp 0: claims a work item of any
// published request of the launch's kind.  Each lane checks one list entry
// (rotating start); the claimable entry with the fewest unclaimed items is taken
// with compare-and-swap on its claim word.  Returns false (in every lane) when
// the host says to take no more items (ctrl[1], or by launch: ctrl[3], ctrl[4]),
// when the SM is the other kernel's now, when nothing is claimable and the host
// asks idle CTAs to exit (ctrl[0]), after idle_ns of finding nothing, or after
// max_idle_polls polls.
__device__ inline bool serve_claim(const ServeLaunch& V, int* slot_out, long long* item_out) {
    const int lane = threadIdx.x & 31;
    unsigned ns = 32;
    const unsigned long long t0 = global_ns();
    for (long long polls = 0; polls < V.max_idle_polls; polls++) {
        int c0 = 0, c1 = 0, n = 0;
        unsigned r = 0;
        if (lane == 0) {
            c1 = ld_vol_i32(V.ctrl + 1) | (V.launch_no < ld_vol_i32(V.ctrl + (V.kind == SERVE_CHAIN ? 3 : 4))) |
                 serve_elsewhere(V);
            c0 = ld_vol_i32(V.ctrl);
            n = min(ld_vol_i32(V.ctrl + 2), V.nslots);
            if (!c1 && n > 0) r = atomicAdd(V.rr, 1u);
        }
        c0 = __shfl_sync(FULL_MASK, c0, 0);
        c1 = __shfl_sync(FULL_MASK, c1, 0);
        n = __shfl_sync(FULL_MASK, n, 0);
        r = __shfl_sync(FULL_MASK, r, 0);
        if (c1) return false;
        for (int base = 0; base < n; base += 32) {
            const int k = base + lane;
            bool ok = false;
            int slot = -1;
            unsigned seq = 0;
            unsigned long long v = 0;
            long long nit = 0;
            if (k < n) {
                const unsigned long long e = ld_vol64(V.list + (r + (unsigned)k) % (unsigned)n);
                slot = (int)(e >> 32);
                seq = (unsigned)e;
                if (slot >= 0 && slot < V.nslots) {
                    v = ld_vol64(V.claim + slot);
                    if ((unsigned)(v >> 32) == seq) {
                        __threadfence();  // the descriptor was written before the claim word
                        nit = __ldcg(V.kind == SERVE_CHAIN ? &V.slots[slot].n_items : &V.slots[slot].walk_items);
                        ok = (long long)(v & 0xffffffffull) < nit &&
                             (V.kind == SERVE_ALL ||
                              __ldcg(V.route + slot) == (V.kind == SERVE_CHAIN ? ROUTE_CHAIN : ROUTE_WALK));
                    }
                }
            }
            // shortest remaining work first (fewest unclaimed items), ties in
            // rotation order: small requests overtake large ones item by item
            unsigned rem = 0xffffffffu;
            if (ok) rem = (unsigned)min(nit - (long long)(v & 0xffffffffull), 0xfffffffell);
            for (int round = 0; round < 32; round++) {
                const unsigned best = __reduce_min_sync(FULL_MASK, rem);
                if (best == 0xffffffffu) break;
                const int l = __ffs(__ballot_sync(FULL_MASK, rem == best)) - 1;
                int got = 0;
                long long it = 0;
                if (lane == l) {
                    for (int tries = 0; tries < 256; tries++) {
                        if ((unsigned)(v >> 32) != seq || (long long)(v & 0xffffffffull) >= nit) break;
                        const unsigned long long old = atomicCAS(V.claim + slot, v, v + 1ull);
                        if (old == v) {
                            got = 1;
                            it = (long long)(v & 0xffffffffull);
                            break;
                        }
                        v = old;
                    }
                    rem = 0xffffffffu;  // taken or gone: this entry is done
                }
                if (__shfl_sync(FULL_MASK, got, l)) {
                    *slot_out = __shfl_sync(FULL_MASK, slot, l);
                    *item_out = __shfl_sync(FULL_MASK, it, l);
                    return true;
                }
            }
        }
        if (c0) return false;
        // lane 0's clock decides for the warp
        const int idle = global_ns() - t0 > (unsigned long long)V.idle_ns;
        if (__shfl_sync(FULL_MASK, idle, 0)) return false;
        __nanosleep(ns);
        if (ns < 2048) ns <<= 1;
    }
    return false;
}

// Serving: takes a free per-CTA workspace slot, or returns -1.  None on the SMs
// left to the uploads' and builds' kernels: four CTAs of 256 threads and 64
// registers fill an SM's registers, and single holes spread over many SMs are
// too small for a sort's CTA, which then waits for a serving CTA to leave.
__device__ inline int take_cta_slot(const ServeLaunch& V) {
    unsigned sm;
    asm volatile("mov.u32 %0, %%smid;" : "=r"(sm));
    if (sm >= V.sm_limit || serve_elsewhere(V)) return -1;
    const int nw = (V.n_cta_slots + 31) >> 5;
    for (int w = 0; w < nw; w++) {
        unsigned v = ld_vol_i32(reinterpret_cast<const int32_t*>(V.cta_slots + w));
        for (int tries = 0; tries < 64 && ~v; tries++) {
            const int b = __ffs(~v) - 1;
            if (w * 32 + b >= V.n_cta_slots) break;
            const unsigned old = atomicOr(V.cta_slots + w, 1u << b);
            if (!(old & (1u << b))) {
                atomicAdd(V.alive, 1);
                __threadfence();
                return w * 32 + b;
            }
            v = old | (1u << b);
        }
    }
    return -1;
}

// Thread 0 copies a matrix descriptor to shared memory (through L2 when it
// may have been rewritten since the launch began).
template <bool CG>
__device__ __forceinline__ void copy_desc(MatDesc* dst, const MatDesc* src) {
    static_assert(sizeof(MatDesc) % 8 == 0, "descriptor copied in 8-byte words");
    const unsigned long long* a = reinterpret_cast<const unsigned long long*>(src);
    unsigned long long* b = reinterpret_cast<unsigned long long*>(dst);
#pragma unroll
    for (int k = 0; k < (int)(sizeof(MatDesc) / 8); k++) b[k] = CG ? __ldcg(a + k) : a[k];
}

constexpr int kSlots = 256;              // words a sparse table can hold
constexpr int kSlotsMax = 192;           // words it is filled to
constexpr int kListCap = 512;            // new ids of a search before the CTA takes it
constexpr int kListRoom = kListCap + 128;  // one step of a warp finds at most 128
constexpr uint32_t kFree = 0xffffffffu;

struct Graph {
    const int32_t* __restrict__ rp;
    const int32_t* __restrict__ cl;
};

// bits above s in word w of a bitmap
__device__ __forceinline__ uint32_t above(int w, int s) {
    const int ws = s >> 5;
    if (w != ws) return w > ws ? ~0u : 0u;
    return (s & 31) == 31 ? 0u : ~0u << ((s & 31) + 1);
}

__device__ __forceinline__ uint32_t below(int w, int s) {
    const int ws = s >> 5;
    if (w != ws) return w < ws ? ~0u : 0u;
    return (1u << (s & 31)) - 1u;
}

__device__ __forceinline__ unsigned long long word_digest(int w, uint32_t m) {
    return m ? mix64(((uint64_t)(uint32_t)w << 32) | m) : 0ull;
}

// how the digest of the ids above s changes when word w goes from a to b
__device__ __forceinline__ unsigned long long digest_step(int w, uint32_t a, uint32_t b, int s) {
    const uint32_t m = above(w, s);
    return word_digest(w, b & m) - word_digest(w, a & m);
}

__device__ __forceinline__ unsigned long long warp_sum64(unsigned long long x) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(FULL_MASK, x, o);
    return x;
}

// ---- sparse tables ----------------------------------------------------------------

__device__ __forceinline__ unsigned slot_of(int w) { return ((unsigned)w * 0x9E3779B1u) >> 24; }
static_assert(kSlots == 256, "slot_of gives 8 bits");

__device__ __forceinline__ uint32_t sparse_word(const uint32_t* key, const uint32_t* msk, int w) {
    unsigned i = slot_of(w);
    for (int p = 0; p < kSlots; p++) {
        const uint32_t k = ld_vol(key + i);
        if (k == (uint32_t)w) return ld_vol(msk + i);
        if (k == kFree) return 0u;
        i = (i + 1) & (kSlots - 1);
    }
    return 0u;
}

// The slot of word w, taken when it is new (*fresh counts those); -1: full.
__device__ __forceinline__ int sparse_slot(uint32_t* key, int w, int* fresh) {
    unsigned i = slot_of(w);
    for (int p = 0; p < kSlots; p++) {
        uint32_t k = ld_vol(key + i);
        if (k == kFree) {
            k = atomicCAS(key + i, kFree, (uint32_t)w);
            if (k == kFree) {
                (*fresh)++;
                return (int)i;
            }
        }
        if (k == (uint32_t)w) return (int)i;
        i = (i + 1) & (kSlots - 1);
    }
    return -1;
}

// ---- rows --------------------------------------------------------------------------

// Distinct ids above s in row s (matrices with repeated entries only), by one
// warp; g is a bitmap that is zero before and after.
template <bool CG>
__device__ inline int row_distinct(const Graph& G, int s, uint32_t* g) {
    const int lane = threadIdx.x & 31;
    const int b = ld_i32<CG>(G.rp + s) & ~3, e = ld_i32<CG>(G.rp + s + 1) & ~3;
    int c = 0;
    for (int j = b + lane; j < e; j += 32) {
        const int w = ld_i32<CG>(G.cl + j);
        if (w > s) c += !(atomicOr(g + (w >> 5), 1u << (w & 31)) & (1u << (w & 31)));
    }
    __syncwarp();
    for (int j = b + lane; j < e; j += 32) {
        const int w = ld_i32<CG>(G.cl + j);
        if (w > s) atomicExch(g + (w >> 5), 0u);
    }
    __syncwarp();
    return __reduce_add_sync(FULL_MASK, c);
}

// The rows of up to 32 vertices laid end to end, one int4 per lane and step:
// lane l holds row start s0 and its int4 count, `incl` their inclusive sums.
// Returns this lane's entry index (row start + offset), or -1 past the end;
// *owner is the lane whose row it is.
__device__ __forceinline__ int flat_int4(int j, int total, int s0, int its, int incl, int* owner) {
    // the owner of position j: the number of lanes whose inclusive sum is <= j
    int o = 0;
#pragma unroll
    for (int b = 16; b > 0; b >>= 1) {
        const int v = __shfl_sync(FULL_MASK, incl, o + b - 1);
        if (v <= j) o += b;
    }
    *owner = o;
    const int first = __shfl_sync(FULL_MASK, incl - its, o);
    const int start = __shfl_sync(FULL_MASK, s0, o);
    return j < total ? start + 4 * (j - first) : -1;
}

__device__ __forceinline__ int warp_incl_sum(int x, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(FULL_MASK, x, o);
        if (lane >= o) x += t;
    }
    return x;
}

template <int BLOCK>
__device__ __forceinline__ void block_clear(uint32_t* bm, long long words) {
    for (long long i = threadIdx.x; i < words; i += BLOCK) bm[i] = 0u;
}

// Word `lane` (0..3) of the 128 ids after s, from words `lane` and `lane + 1`
// of the bitmap from (s + 1) >> 5 on (lanes 0..4 hold them).
__device__ __forceinline__ uint32_t next128(uint32_t word, int s) {
    const uint32_t up = __shfl_down_sync(FULL_MASK, word, 1);
    return __funnelshift_r(word, up, (s + 1) & 31);
}

// Row s of a direction's outputs.
__device__ __forceinline__ void write_row(const MatDesc& M, int s, int dir, bool sym, const Tot& t,
                                          int raw, int orig) {
    if (dir == 0) {
        M.nnz_u[s] = t.gt;
        M.nz_row_u[s] = raw + t.gt - orig;
        if (M.dig_u) M.dig_u[s] = t.dig;
    }
    if (dir == 1 || sym) {
        M.nnz_lc[s] = t.gt;
        if (M.dig_lc) M.dig_lc[s] = t.dig;
    }
}

// rows kept of a narrow level by a CTA of BLOCK threads
__host__ __device__ constexpr int bfs_cap(int block) { return block >= 1024 ? 1024 : 512; }

template <int BLOCK>
struct BfsSmem {
    int cnt[3];                // ids queued per level, in turn
    unsigned long long rtrav;  // entries read
    // the rows of a level's first ids: first entry, int4s
    int2 row[2][bfs_cap(BLOCK)];
};

// Breadth-first search in the bitmap bm from the frontier q[0, tail), whose
// ids are marked (but for s itself, which no step marks): every id below
// `bound`, and s, is expanded; ids found are marked and queued (ids from
// `bound` on only when `all`).  Returns the queue's length.  With LAM, ids
// whose label is below s count as marked.  Block-wide.
//
// What bounds it is the chain of dependent accesses per level (a mesh has
// hundreds of narrow levels): in narrow levels an id's row pointers are loaded
// when it is found and its row is kept in shared memory, so that a level is row
// entries -> bitmap -> row pointers -> barrier; wide ones read the queue two
// groups ahead.
template <int BLOCK, bool CG, bool LAM = false>
__device__ long long block_bfs(BfsSmem<BLOCK>& SM, const Graph& G, uint32_t* bm, int32_t* q,
                               long long qcap, long long tail, int s, int bound, bool all,
                               int32_t* status, const int32_t* lam = nullptr) {
    constexpr int NW = BLOCK / 32, kCap = bfs_cap(BLOCK);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) SM.cnt[0] = 0;
    __syncthreads();
    long long lb = 0, le = min(tail, qcap);
    unsigned long long trav = 0;
    bool kept = false;
    for (int level = 0; lb < le; level++) {
        int* const cnt = &SM.cnt[level % 3];
        int2* const next = SM.row[(level + 1) & 1];
        const int2* const cur = SM.row[level & 1];
        if (threadIdx.x == 0) SM.cnt[(level + 1) % 3] = 0;
        const long long n = le - lb;
        const bool keep = n <= BLOCK;  // this level is narrow: the next one's rows are kept
        // the entries of up to 32 rows, 128 at a time: marks them, queues the new ids
        auto expand = [&](int s0, int its) {
            const int incl = warp_incl_sum(its, lane);
            const int total = __shfl_sync(FULL_MASK, incl, 31);
            if (lane == 0) trav += 4ull * total;
            int o;
            int at = flat_int4(lane, total, s0, its, incl, &o);
            int4 e = at >= 0 ? ld_row4<CG>(G.cl + at) : make_int4(-1, -1, -1, -1);
            for (int j0 = 0; j0 < total; j0 += 32) {
                int4 en = make_int4(-1, -1, -1, -1);
                if (j0 + 32 < total) {
                    at = flat_int4(j0 + 32 + lane, total, s0, its, incl, &o);
                    if (at >= 0) en = ld_row4<CG>(G.cl + at);
                }
                const int ws[4] = {e.x, e.y, e.z, e.w};
                e = en;
                uint32_t old[4];
#pragma unroll
                for (int c = 0; c < 4; c++)
                    old[c] = ws[c] >= 0 && ws[c] != s ? ld_vol(bm + (ws[c] >> 5)) : ~0u;
                if constexpr (LAM) {
                    // what the hub reaches through ids below s is not looked at
#pragma unroll
                    for (int c = 0; c < 4; c++)
                        if (ws[c] >= 0 && __ldg(lam + ws[c]) < s) old[c] = ~0u;
                }
                bool any = false;
#pragma unroll
                for (int c = 0; c < 4; c++) any |= !((old[c] >> (ws[c] & 31)) & 1u);
                if (!__any_sync(FULL_MASK, any)) continue;
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    const uint32_t bit = 1u << (ws[c] & 31);
                    old[c] = old[c] & bit ? ~0u : atomicOr(bm + (ws[c] >> 5), bit);
                }
                unsigned bal[4];
                int k = 0;
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    bal[c] = __ballot_sync(FULL_MASK, !((old[c] >> (ws[c] & 31)) & 1u) &&
                                                          (all || ws[c] < bound));
                    k += __popc(bal[c]);
                }
                if (!k) continue;
                int to = 0;
                if (lane == 0) to = atomicAdd(cnt, k);
                to = __shfl_sync(FULL_MASK, to, 0);
                int x[4];
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    x[c] = ((bal[c] >> lane) & 1u) ? to + __popc(bal[c] & ((1u << lane) - 1u)) : -1;
                    to += __popc(bal[c]);
                    if (x[c] < 0) continue;
                    if (le + x[c] < qcap) q[le + x[c]] = ws[c];
                    else atomicOr(status, DEV_ERR_QUEUE);
                }
                if (!keep) continue;
                int a0[4], a1[4];
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    a0[c] = a1[c] = 0;
                    if (x[c] >= 0 && ws[c] < bound) {
                        a0[c] = ld_i32<CG>(G.rp + ws[c]);
                        a1[c] = ld_i32<CG>(G.rp + ws[c] + 1);
                    }
                }
#pragma unroll
                for (int c = 0; c < 4; c++)
                    if (x[c] >= 0 && x[c] < kCap)
                        next[x[c]] = make_int2(a0[c] & ~3, ((a1[c] & ~3) - (a0[c] & ~3)) >> 2);
            }
        };
        if (kept && n <= kCap) {
            const int per = n >= 32 * NW ? 32 : (int)((n + NW - 1) / NW);
            for (long long base = (long long)warp * per; base < n; base += NW * per) {
                int2 r = make_int2(0, 0);
                if (lane < per && base + lane < n) r = cur[base + lane];
                expand(r.x, r.y);
            }
        } else {
            // two groups of 32 ahead: the queue entries load while the group
            // before is expanded, the row pointers while the one before that is
            auto id_of = [&](long long k) { return k < le ? q[k] : -1; };
            auto row_of = [&](int u, int& a0, int& a1) {
                a0 = a1 = 0;
                if (u >= 0 && (u < bound || u == s)) {
                    a0 = ld_i32<CG>(G.rp + u);
                    a1 = ld_i32<CG>(G.rp + u + 1);
                }
            };
            long long base = lb + 32ll * warp;
            int nu = id_of(base + lane), a0, a1;
            row_of(nu, a0, a1);
            nu = id_of(base + 32 * NW + lane);
            for (; base < le; base += 32 * NW) {
                const int nnu = id_of(base + 64 * NW + lane);
                int na0, na1;
                row_of(nu, na0, na1);
                expand(a0 & ~3, ((a1 & ~3) - (a0 & ~3)) >> 2);
                nu = nnu;
                a0 = na0;
                a1 = na1;
            }
        }
        __syncthreads();
        kept = keep;
        lb = le;
        le = min(le + *cnt, qcap);
    }
    if (lane == 0 && trav) atomicAdd(&SM.rtrav, trav);
    __syncthreads();
    return le;
}

}  // namespace gsofa
