// gsofa_chain.cu -- the counting traversal of symmetric patterns: incremental
// reach sets, one warp per chunk.
//
// U row s is the out-neighbourhood above s of everything s reaches in A
// through ids < s (gsofa_kernels.cu states the rule); with a symmetric pattern
// L column s is the same set.  A work item is a chunk of consecutive sources,
// and warp 0 of a CTA walks it in increasing order.  The other warps wait at a
// barrier until a search is too large for one warp.
//
// What makes a source cheap is a base: a vertex b below the current source s
// together with its exact reach set X = {v : b reaches v through ids < s}, kept
// for every s of the chunk.  Then s reaches b exactly when s is in X, and
//   F(s) = X u {what s adds to it}.
// So whether a search may start from the base's set is known from one bit, it
// expands only vertices that the base does not reach, and the counts and
// digests of the result are the base's plus those of the few new ids.  Going
// from s to s + 1, X becomes F(s) if s is in it and stays as it was otherwise.
//
// Two bases are kept.  X is dense: a bitmap of n bits in shared memory (global
// memory when it does not fit).  T is sparse: a table of up to 192 32-id words in
// shared memory, for the small components that lie between the sources of a
// large one.  A source that meets neither is searched alone into a second sparse
// table, which becomes the new T.
//
// A search that finds more than 512 ids or fills its table is handed to the
// whole CTA: it goes on in X if it had begun there, else its table becomes X.
//
// Every set is exact, so nothing here depends on timing: counts, digests and
// masks are the same whatever the chunks, the CTA size or the grid.
//
// What bounds it: a chunk's sources are a serial chain, about 1.1 to 5 rounds
// of dependent loads per source (row pointers, row entries), so throughput is
// the number of chunks in flight over that latency; the rows of the next source
// are loaded a source ahead.  On a 40^3 mesh one warp of a CTA's eight issues, an
// instruction every five cycles of an SM's quarter; seven wait at the barrier.
// (Unsymmetric patterns would need both directions' sets, and a source is in
// them one at a time: one-sided sets are searched anew for each, which took 248 ms
// on a 200,000-row band where traverse_kernel takes 12.)
#include <climits>

#include "gsofa_device.cuh"

namespace gsofa {

namespace {

// the sparse tables (T and the current source's own) and the ids its search has
// found
struct Sparse {
    uint32_t key[2][kSlots];
    uint32_t msk[2][kSlots];
    int32_t list[kListRoom];
    uint32_t was[kListRoom];  // the id's word before it joined
};

// counters of an item
struct Acc {
    unsigned long long fills, e, v, trav, nnz, chained;
};

// Sources that do not meet T before it is dropped: an old T costs a look-up a
// source.  4, 16 and 64 take the same time within 1 % on meshes of 2,025 to 262,144
// rows and on a symmetric random pattern of 20,000.
constexpr int kIdleT = 16;

template <int BLOCK>
struct ChainSmem {
    long long item;
    int mi, skip, cta, dup;
    Tot base;              // X relative to the current source
    int have;              // X is a base
    int s;
    int large, mode, tsel, found;
    int raw, orig;
    Tot tot;
    Acc acc;
    BfsSmem<BLOCK> bfs;
    unsigned long long red[BLOCK / 32][4];
};

// ---- searches by the whole CTA --------------------------------------------------------

// The sizes of a bitmap's set relative to source s, left in SM.tot.  Block-wide.
template <int BLOCK, bool CG>
__device__ void block_census(ChainSmem<BLOCK>& SM, const MatDesc& M, const uint32_t* bm, int s,
                             bool digests) {
    const int lane = threadIdx.x & 31;
    const int nw = (int)(((long long)M.n + 31) >> 5);
    unsigned long long gt = 0, v = 0, e = 0, dig = 0;
    for (int w = threadIdx.x; w < nw; w += BLOCK) {
        const uint32_t x = bm[w];
        if (!x) continue;
        const uint32_t xl = x & below(w, s), xh = x & above(w, s);
        v += __popc(xl);
        gt += __popc(xh);
        if (digests) dig += word_digest(w, xh);
        if (!xl) continue;
        if (xl == ~0u) {
            e += (unsigned long long)ld_i32<CG>(M.wdeg + w);
        } else if (__popc(xl) <= 2 || M.dplanes == nullptr) {
            for (uint32_t t = xl; t; t &= t - 1)
                e += (unsigned long long)row_degree<CG>(M.rowptr, 32 * w + __ffs(t) - 1);
        } else {
            // degree sum from the bit-planes: coalesced loads, four at a time
            const int32_t* pl = reinterpret_cast<const int32_t*>(M.dplanes) + w;
            for (int k = 0; k < M.nplanes; k += 4) {
                uint32_t p4[4];
#pragma unroll
                for (int j = 0; j < 4; j++)
                    p4[j] = k + j < M.nplanes ? (uint32_t)ld_i32<CG>(pl + (long long)(k + j) * nw) : 0u;
#pragma unroll
                for (int j = 0; j < 4; j++) e += (unsigned long long)__popc(xl & p4[j]) << (k + j);
            }
        }
    }
    unsigned long long vals[4] = {gt, v, e, dig};
#pragma unroll
    for (int j = 0; j < 4; j++) {
        vals[j] = warp_sum64(vals[j]);
        if (lane == 0) SM.red[threadIdx.x >> 5][j] = vals[j];
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long r[4] = {0, 0, 0, 0};
        for (int i = 0; i < BLOCK / 32; i++)
            for (int j = 0; j < 4; j++) r[j] += SM.red[i][j];
        SM.tot.gt = (int)r[0];
        SM.tot.v = (int)r[1];
        SM.tot.e = r[2];
        SM.tot.dig = r[3];
    }
    __syncthreads();
}

// The change of word w's digest when its bit s stops being above the source:
// lane 1 digests the word with the bit, the others without.
__device__ __forceinline__ unsigned long long pass_digest(int w, uint32_t x, int s) {
    const bool with = (threadIdx.x & 31) == 1;
    const unsigned long long h = word_digest(w, x & (with ? ~0u << (s & 31) : above(w, s)));
    return __shfl_sync(FULL_MASK, h, 0) - __shfl_sync(FULL_MASK, h, 1);
}

// ---- one warp's walk through a chunk ----------------------------------------------------

// What a chunk's searches need.
struct Side {
    Graph G;
    uint32_t* X;  // the dense base's set
    uint32_t* g;  // a zero bitmap in global memory
    Sparse* P;
};

// The sources SM.s .. s_end - 1, up to the first whose search is left to the
// CTA; SM.s is that source, or s_end.  T begins empty.
template <int BLOCK, bool CG>
__device__ void warp_walk(ChainSmem<BLOCK>& SM, const MatDesc& M, const Side& D, int s_end, int list_cap) {
    const int lane = threadIdx.x & 31;
    const bool dup = SM.dup != 0;
    const bool digests = M.dig_u != nullptr;
    const bool have = SM.have != 0;
    const Graph G = D.G;
    uint32_t* const X = D.X;
    Sparse& P = *D.P;
    int s = SM.s;
    bool have_t = false;
    int tsel = 0, used = 0;
    Tot bx = SM.base, bt = {0, 0, 0ull, 0ull};
    Acc acc = {0, 0, 0, 0, 0, 0};
    auto in_x = [&](int v) { return (ld_vol(X + (v >> 5)) >> (v & 31)) & 1u; };
    auto in_t = [&](int v) { return (sparse_word(P.key[tsel], P.msk[tsel], v >> 5) >> (v & 31)) & 1u; };
    int r0 = ld_i32<CG>(G.rp + s), r1 = ld_i32<CG>(G.rp + s + 1);
    int4 pre = make_int4(-1, -1, -1, -1);  // the first 128 entries of row s
    if (4 * lane < (r1 & ~3) - (r0 & ~3)) pre = ld_row4<CG>(G.cl + (r0 & ~3) + 4 * lane);
    int deg_prev = s > 0 ? row_degree<CG>(G.rp, s - 1) : 0;
    bool large = false;
    int mode = 0, found = 0;
    int idle = 0;  // sources since one met T
    for (; s < s_end; s++) {
        if (idle >= kIdleT) have_t = false;
        const bool xs = have && in_x(s), ts = have_t && in_t(s);
        idle = ts ? 0 : idle + 1;
        mode = xs ? 0 : ts ? 1 : 2;
        // the next row's pointers, then (below) its first entries
        const int r2 = s + 2 <= M.n ? ld_i32<CG>(G.rp + s + 2) : r1;

        // the bases' sizes relative to s instead of s - 1
        {
            const int w = s >> 5, wp = (s - 1) >> 5;
            if (have) {
                if (xs) {
                    bx.gt--;
                    if (digests) bx.dig += pass_digest(w, ld_vol(X + w), s);
                }
                if (s > 0 && in_x(s - 1)) {
                    bx.v++;
                    bx.e += (unsigned)deg_prev;
                }
            }
            if (have_t) {
                if (ts) {
                    bt.gt--;
                    if (digests) bt.dig += pass_digest(w, sparse_word(P.key[tsel], P.msk[tsel], w), s);
                }
                if (s > 0 && (sparse_word(P.key[tsel], P.msk[tsel], wp) >> ((s - 1) & 31)) & 1u) {
                    bt.v++;
                    bt.e += (unsigned)deg_prev;
                }
            }
        }

        uint32_t* const key = P.key[mode == 1 ? tsel : 1 - tsel];
        uint32_t* const msk = P.msk[mode == 1 ? tsel : 1 - tsel];
        int words = mode == 1 ? used : 0;  // table words in use
        if (mode == 2) {
            for (int i = lane; i < kSlots; i += 32) {
                key[i] = kFree;
                msk[i] = 0u;
            }
            __syncwarp();
        }
        large = false;
        found = 0;
        int v = 0, raw = 0, trav = 0;  // this lane's
        unsigned e = 0;
        // marks the four entries and lists the new ids; false: too many for a warp
        auto visit = [&](const int4& q4) -> bool {
            const int ws[4] = {q4.x, q4.y, q4.z, q4.w};
            uint32_t old[4];
            int nslots = 0;
            bool full = false;
            if (mode == 0) {
                bool any = false;
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    old[c] = ws[c] >= 0 && ws[c] != s ? ld_vol(X + (ws[c] >> 5)) : ~0u;
                    any |= !((old[c] >> (ws[c] & 31)) & 1u);
                }
                if (!__any_sync(FULL_MASK, any)) return true;  // all of them known
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    const uint32_t bit = 1u << (ws[c] & 31);
                    old[c] = old[c] & bit ? ~0u : atomicOr(X + (ws[c] >> 5), bit);
                }
            } else {
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    old[c] = ~0u;
                    if (ws[c] < 0 || ws[c] == s) continue;
                    const int i = sparse_slot(key, ws[c] >> 5, &nslots);
                    if (i < 0) full = true;
                    else old[c] = atomicOr(msk + i, 1u << (ws[c] & 31));
                }
                words += __reduce_add_sync(FULL_MASK, nslots);
            }
            unsigned bal[4];
            int to = found;
#pragma unroll
            for (int c = 0; c < 4; c++)
                bal[c] = __ballot_sync(FULL_MASK, !((old[c] >> (ws[c] & 31)) & 1u));
            if (bal[0] | bal[1] | bal[2] | bal[3]) {
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    if ((bal[c] >> lane) & 1u) {
                        const int k = to + __popc(bal[c] & ((1u << lane) - 1u));
                        P.list[k] = ws[c];
                        P.was[k] = old[c];
                    }
                    to += __popc(bal[c]);
                }
                found = to;
                __syncwarp();
            }
            return found <= list_cap && words <= kSlotsMax && !__any_sync(FULL_MASK, full);
        };
        // row s
        {
            const int b = r0 & ~3, plen = (r1 & ~3) - b;
            int4 q4 = pre;
            for (int k0 = 0; k0 < plen && !large; k0 += 128) {
                int4 qn = make_int4(-1, -1, -1, -1);
                if (k0 + 128 + 4 * lane < plen) qn = ld_row4<CG>(G.cl + b + k0 + 128 + 4 * lane);
                raw += (q4.x > s) + (q4.y > s) + (q4.z > s) + (q4.w > s);
                large = !visit(q4);
                q4 = qn;
            }
            if (lane == 0) trav += plen;
        }
        // the next row's first entries load while this search goes on
        pre = make_int4(-1, -1, -1, -1);
        if (4 * lane < (r2 & ~3) - (r1 & ~3)) pre = ld_row4<CG>(G.cl + (r1 & ~3) + 4 * lane);
        for (int h = 0; h < found && !large; h += 32) {
            const int u = h + lane < found ? P.list[h + lane] : INT_MAX;
            int s0 = 0, its = 0;
            if (u < s) {
                const int a0 = ld_i32<CG>(G.rp + u), a1 = ld_i32<CG>(G.rp + u + 1);
                s0 = a0 & ~3;
                its = ((a1 & ~3) - s0) >> 2;
                v++;
                e += (unsigned)(4 * its - (a1 & 3));
            }
            const int have_now = found;
            const int incl = warp_incl_sum(its, lane);
            const int total = __shfl_sync(FULL_MASK, incl, 31);
            if (lane == 0) trav += 4 * total;
            int o;
            int at = flat_int4(lane, total, s0, its, incl, &o);
            int4 q4 = at >= 0 ? ld_row4<CG>(G.cl + at) : make_int4(-1, -1, -1, -1);
            for (int j0 = 0; j0 < total && !large; j0 += 32) {
                int4 qn = make_int4(-1, -1, -1, -1);
                if (j0 + 32 < total) {
                    at = flat_int4(j0 + 32 + lane, total, s0, its, incl, &o);
                    if (at >= 0) qn = ld_row4<CG>(G.cl + at);
                }
                large = !visit(q4);
                q4 = qn;
            }
            // a partial group of 32: the ids found meanwhile start the next one
            if (have_now - h < 32) h = have_now - 32;
        }
        if (large) break;
        Tot t = mode == 0 ? bx : mode == 1 ? bt : Tot{0, 0, 0ull, 0ull};
        if (found) {
            int gt = 0;
            unsigned long long dig = 0;
            for (int i = lane; i < found; i += 32) {
                const int w = P.list[i];
                if (w < s) continue;
                gt++;
                if (digests) dig += digest_step(w >> 5, P.was[i], P.was[i] | (1u << (w & 31)), s);
            }
            gt = __reduce_add_sync(FULL_MASK, gt);
            t.gt += gt;
            t.v += __reduce_add_sync(FULL_MASK, v);
            t.e += (unsigned)__reduce_add_sync(FULL_MASK, e);  // distinct rows: below 2^31
            if (digests && gt) t.dig += warp_sum64(dig);
        }
        raw = __reduce_add_sync(FULL_MASK, raw);
        const int orig = dup ? row_distinct<CG>(G, s, D.g) : raw;
        if (lane == 0) write_row(M, s, 0, true, t, raw, orig);
        {
            // the 128 ids after s of the L column
            uint32_t word = 0;
            if (lane < 5) {
                const int w = ((s + 1) >> 5) + lane;
                word = mode == 0 ? ld_vol(X + w) : sparse_word(key, msk, w);
            }
            word = next128(word, s);
            if (lane < 4) M.lmask[4ll * s + lane] = word;
        }
        acc.fills += 2ull * (unsigned)(t.gt - orig);
        acc.trav += (unsigned)__shfl_sync(FULL_MASK, trav, 0);
        acc.chained += mode != 2;
        acc.nnz += (unsigned)t.gt;
        acc.v += (unsigned)t.v;
        acc.e += t.e;

        // the bases for s + 1
        if (xs) {
            bx = t;
            if (ts) have_t = false;  // T reaches into the dense base: it is as large as that
        } else if (ts) {
            bt = t;
            used = words;
        } else {
            // s met no base: its own set is the new T
            if (lane == 0) {
                int one = 0;
                const int j = sparse_slot(key, s >> 5, &one);
                if (j >= 0) atomicOr(msk + j, 1u << (s & 31));
                words += one;
            }
            words = __shfl_sync(FULL_MASK, words, 0);
            tsel = 1 - tsel;
            used = words;
            bt = t;
            have_t = true;
            idle = 0;
        }
        __syncwarp();
        deg_prev = (r1 & ~3) - (r0 & ~3) - (r1 & 3);
        r0 = r1;
        r1 = r2;
    }
    if (lane == 0) {
        SM.base = bx;
        SM.s = s;
        SM.large = large;
        SM.mode = mode;
        SM.tsel = tsel;
        SM.found = found;
        Acc& A = SM.acc;
        A.fills += acc.fills;
        A.e += acc.e;
        A.v += acc.v;
        A.trav += acc.trav;
        A.nnz += acc.nnz;
        A.chained += acc.chained;
    }
}

// ---- sources the whole CTA takes ---------------------------------------------------------

template <int BLOCK, bool CG>
struct Large {
    ChainSmem<BLOCK>& SM;
    const MatDesc& M;
    const Side& D;
    int32_t* q;
    long long qcap;
    long long words;
    int32_t* status;

    // Row s's entry counts into SM.raw, SM.orig.
    __device__ void row_stats(int s) {
        if (threadIdx.x < 32) {
            const int lane = threadIdx.x;
            const Graph& G = D.G;
            const int b = ld_i32<CG>(G.rp + s) & ~3, e = ld_i32<CG>(G.rp + s + 1) & ~3;
            int raw = 0;
            for (int j = b + lane; j < e; j += 32) raw += ld_i32<CG>(G.cl + j) > s;
            raw = __reduce_add_sync(FULL_MASK, raw);
            const int orig = SM.dup ? row_distinct<CG>(G, s, D.g) : raw;
            if (lane == 0) {
                SM.raw = raw;
                SM.orig = orig;
                SM.bfs.rtrav = 0;
            }
        }
        __syncthreads();
    }

    // Outputs and counters of source s, whose set is X and whose sizes are SM.tot.
    __device__ void emit(int s, bool chained) {
        if (threadIdx.x < 32) {
            const int lane = threadIdx.x;
            uint32_t word = lane < 5 ? D.X[((s + 1) >> 5) + lane] : 0u;
            word = next128(word, s);
            if (lane < 4) M.lmask[4ll * s + lane] = word;
            if (lane == 0) {
                const Tot t = SM.tot;
                write_row(M, s, 0, true, t, SM.raw, SM.orig);
                Acc& A = SM.acc;
                A.fills += 2ull * (unsigned)(t.gt - SM.orig);
                A.e += t.e;
                A.v += (unsigned)t.v;
                A.nnz += (unsigned)t.gt;
                A.trav += SM.bfs.rtrav;
                A.chained += chained ? 1 : 0;
            }
        }
        __syncthreads();
    }

    // Source SM.s, whose search is large: it goes on in X, which is its base's set
    // with what it has found, or, when its search began in a table, what that
    // holds (every id there is reached by s, with T's base, which s reaches, and all
    // but those of the list are expanded).  X is the base from here on.
    __device__ void take() {
        const int s = SM.s, mode = SM.mode, found = SM.found;
        const bool digests = M.dig_u != nullptr;
        const Sparse& P = *D.P;
        row_stats(s);
        if (mode != 0) {
            const int which = mode == 1 ? SM.tsel : 1 - SM.tsel;
            block_clear<BLOCK>(D.X, words);
            __syncthreads();
            for (int i = threadIdx.x; i < kSlots; i += BLOCK)
                if (P.key[which][i] != kFree) D.X[P.key[which][i]] = P.msk[which][i];
            __syncthreads();
            if (threadIdx.x == 0) D.X[s >> 5] |= 1u << (s & 31);
        }
        for (int i = threadIdx.x; i <= found; i += BLOCK) {
            if (i < qcap) q[i] = i ? P.list[i - 1] : s;
            else atomicOr(status, DEV_ERR_QUEUE);
        }
        __syncthreads();
        block_bfs<BLOCK, CG>(SM.bfs, D.G, D.X, q, qcap, found + 1, s, s, false, status);
        block_census<BLOCK, CG>(SM, M, D.X, s, digests);
        emit(s, mode != 2);
        if (threadIdx.x == 0) {
            SM.base = SM.tot;
            SM.have = 1;
            SM.large = 0;
            SM.s = s + 1;
        }
        __syncthreads();
    }
};

// SERVE: items come from the requests the request loop publishes (matrix data
// read through L2, see ld_i32), else from the launch's matrices.
template <int BLOCK, bool SERVE>
__global__ void __launch_bounds__(BLOCK, 1024 / BLOCK) chain_kernel(ChainLaunch P) {
    extern __shared__ uint4 dyn_smem[];
    __shared__ ChainSmem<BLOCK> SM;
    __shared__ MatDesc SD;  // the current item's matrix
    constexpr bool CG = SERVE;
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    if constexpr (SERVE) {
        if (threadIdx.x == 0) SM.cta = take_cta_slot(P.serve);
        __syncthreads();
        if (SM.cta < 0) return;  // every workspace slot is taken
    }
    const long long cta = SERVE ? SM.cta : blockIdx.x;
    Sparse* const sparse = reinterpret_cast<Sparse*>(dyn_smem);
    uint32_t* const sbm = reinterpret_cast<uint32_t*>(sparse + 1);
    uint32_t* const gb = P.gbm + cta * P.gbm_count * P.bitmap_words;
    int32_t* const q = P.queue + cta * P.queue_stride;
    for (long long i = threadIdx.x; i < P.bitmap_words; i += BLOCK) gb[i] = 0u;
    const long long stride = P.sample_stride > 1 ? P.sample_stride : 1;

    for (;;) {
        __syncthreads();  // every thread is done with the previous item
        if constexpr (SERVE) {
            if (warp == 0) {
                int slot = 0;
                long long it = -1;
                const bool got = serve_claim(P.serve, &slot, &it);
                if (lane == 0) {
                    if (got) {
                        copy_desc<true>(&SD, P.serve.slots + slot);
                        SM.skip = __ldcg(P.serve.slot_status + slot) != 0;  // ingest failed
                        SM.dup = __ldcg(SD.asym + 1) != 0;
                    }
                    SM.item = got ? it : -1;
                }
            }
        } else if (threadIdx.x == 0) {
            const unsigned long long c = atomicAdd(P.work_counter, 1ull);
            const long long it = (long long)c < P.total_items ? (long long)c * stride : -1;
            if (it >= 0) {
                SM.mi = P.items == ITEMS_TOP ? find_matrix<&MatDesc::top_base>(P.mats, P.nmats, it)
                                             : find_matrix(P.mats, P.nmats, it);
                copy_desc<false>(&SD, P.mats + SM.mi);
                SM.skip = 0;
                SM.dup = SD.asym[1] != 0;
            }
            SM.item = it;
        }
        __syncthreads();
        if (SM.item < 0) break;
        const MatDesc& M = SD;
        const int32_t n = M.n;
        const long long clen = SERVE ? (long long)M.chunk : (long long)P.chunk;
        const long long nchunks = ((long long)n + clen - 1) / clen;
        // largest sources first; M.top_items of them are the other launch's
        const long long local = SERVE                  ? SM.item
                                : P.items == ITEMS_TOP ? SM.item - M.top_base
                                                       : SM.item - M.item_base + M.top_items;
        const long long chunk = nchunks - 1 - local;
        const int s_first = (int)(chunk * clen);
        const int s_end = SM.skip ? s_first : (int)min((long long)n, (chunk + 1) * clen);
        const long long words = bitmap_words_for(n);
        if (threadIdx.x == 0) {
            SM.s = s_first;
            SM.have = SM.large = 0;
            SM.base = Tot{0, 0, 0ull, 0ull};
            SM.acc = Acc{0, 0, 0, 0, 0, 0};
        }
        const Side D{{M.rowptr, M.col}, words <= P.smem_words ? sbm : gb + P.bitmap_words, gb, sparse};
        __syncthreads();
        while (SM.s < s_end) {
            __syncthreads();  // everyone has read SM.s
            if (warp == 0) warp_walk<BLOCK, CG>(SM, M, D, s_end, P.list_cap);
            __syncthreads();
            if (SM.large) Large<BLOCK, CG>{SM, M, D, q, P.queue_stride, words, P.status}.take();
        }
        if constexpr (SERVE) __threadfence();
        __syncthreads();
        if (threadIdx.x == 0) {
            unsigned long long* c = M.counters;
            const Acc& a = SM.acc;
            atomicAdd(c + CNT_FILLS, a.fills);
            atomicAdd(c + CNT_EDGES_ALG, a.e);
            atomicAdd(c + CNT_VERTS_ALG, a.v);
            atomicAdd(c + CNT_EDGES_TRAV, a.trav);
            atomicAdd(c + CNT_NNZ_U, a.nnz);
            atomicAdd(c + CNT_NNZ_L, a.nnz);
            atomicAdd(c + CNT_CHAINED, a.chained);
            if constexpr (SERVE) {
                // count the item; the CTA that finishes the request's last one tells the host
                __threadfence();
                const unsigned long long done = atomicAdd(P.serve.items_done + M.slot, 1ull) + 1ull;
                if (done == (unsigned long long)M.n_items) {
                    __threadfence_system();
                    *reinterpret_cast<volatile unsigned long long*>(P.serve.done_flags + M.slot) = M.seq;
                }
            }
        }
    }
    if constexpr (SERVE) {
        __syncthreads();  // the workspace is no longer in use
        if (threadIdx.x == 0) {
            __threadfence();
            atomicSub(P.serve.alive, 1);
            atomicAnd(P.serve.cta_slots + (SM.cta >> 5), ~(1u << (SM.cta & 31)));
        }
    }
}

template <int BLOCK, bool SERVE>
int occupancy_one(size_t smem) {
    auto k = chain_kernel<BLOCK, SERVE>;
    int blocks = 0;
    if (allow_shared_memory<chain_kernel<BLOCK, SERVE>>() != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, k, BLOCK, smem) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return blocks;
}

template <int BLOCK, bool SERVE>
cudaError_t launch_one(const ChainLaunch& L, int grid, size_t smem, cudaStream_t st) {
    auto k = chain_kernel<BLOCK, SERVE>;
    cudaError_t e = allow_shared_memory<chain_kernel<BLOCK, SERVE>>();
    if (e != cudaSuccess) return e;
    k<<<grid, BLOCK, smem, st>>>(L);
    return cudaGetLastError();
}

}  // namespace

size_t chain_sparse_bytes() { return sizeof(Sparse); }
int chain_list_cap() { return kListCap; }

int chain_occupancy(int block, bool serve, size_t smem) {
    switch (block) {
        case 128: return serve ? occupancy_one<128, true>(smem) : occupancy_one<128, false>(smem);
        case 256: return serve ? occupancy_one<256, true>(smem) : occupancy_one<256, false>(smem);
        case 512: return serve ? occupancy_one<512, true>(smem) : occupancy_one<512, false>(smem);
        case 1024: return serve ? occupancy_one<1024, true>(smem) : occupancy_one<1024, false>(smem);
        default: return 0;
    }
}

cudaError_t launch_chain(const ChainLaunch& L, int block, bool serve, int grid, size_t smem,
                         cudaStream_t st) {
    switch (block) {
        case 128: return serve ? launch_one<128, true>(L, grid, smem, st) : launch_one<128, false>(L, grid, smem, st);
        case 256: return serve ? launch_one<256, true>(L, grid, smem, st) : launch_one<256, false>(L, grid, smem, st);
        case 512: return serve ? launch_one<512, true>(L, grid, smem, st) : launch_one<512, false>(L, grid, smem, st);
        case 1024: return serve ? launch_one<1024, true>(L, grid, smem, st) : launch_one<1024, false>(L, grid, smem, st);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace gsofa
