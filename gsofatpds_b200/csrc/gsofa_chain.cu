// gsofa_chain.cu -- the counting traversal: incremental reach sets, one warp
// per direction.
//
// U row s is the out-neighbourhood above s of everything s reaches in A
// through ids < s, L column s the same in A^T (gsofa_kernels.cu states the
// rule).  A work item is a chunk of consecutive sources, and a CTA walks it in
// increasing order, both directions of a source at the same time: warp 0 the
// U rows (direction 0), warp 1 the L columns (direction 1; unused when the
// pattern is symmetric).  The other warps wait at a barrier until a search is
// too large for one warp.
//
// What makes a source cheap is a base: a vertex b below the current source s
// together with its exact reach sets X0 = {v : b reaches v through ids < s}
// and X1 = {v : v reaches b through ids < s}, both kept for every s of the
// chunk.  Then
//   s reaches b  <=>  s in X1,  and F(s) = X0 u {what s adds to it},
//   b reaches s  <=>  s in X0,  and B(s) = X1 u {what s adds to it}.
// So whether a search may start from the base's set is known from one bit, it
// expands only vertices that the base does not reach, and the counts and
// digests of the result are the base's plus those of the few new ids.  Going
// from s to s + 1 the base's sets stay exact by one rule per direction:
// X0 becomes X0 u F(s) if b reaches s, and stays as it was otherwise (what an
// overlaid search set is taken back from a list); X1 likewise with B(s).
//
// Two bases are kept.  X is dense: a bitmap of n bits per direction in shared
// memory (global memory when two do not fit).  T is sparse: a table of up to
// 192 32-id words per direction in shared memory, for the small components
// that lie between the sources of a large one.  A source that meets neither is
// searched alone into a second sparse table, which becomes the new T.
//
// A search that finds more than 512 ids or fills its table is handed to the
// whole CTA.  If it met X (or the other direction did), the search goes on
// there; otherwise X is rebuilt: from s itself when both directions are large,
// else from a hub, the found vertex of largest degree in the opposite
// direction, kept when its opposite reach set is large too (a vertex inside
// the strongly connected core, which the one-sided s is not), else the search
// runs alone in a global bitmap.
//
// Every set is exact, so nothing here depends on timing: counts, digests and
// masks are the same whatever the chunks, the CTA size or the grid.
//
// What bounds it: a chunk's sources are a serial chain, about 1.1 to 5 rounds
// of dependent loads per source and direction (row pointers, row entries), so
// throughput is the number of chunks in flight over that latency; the rows of
// the next source are loaded a source ahead.
#include <climits>

#include "gsofa_device.cuh"

namespace gsofa {

namespace {

// a direction's sparse tables (T and the current source's own) and the ids its
// search has found
struct Sparse {
    uint32_t key[2][kSlots];
    uint32_t msk[2][kSlots];
    int32_t list[kListRoom];
    uint32_t was[kListRoom];  // the id's word before it joined
};

// per-direction counters of an item
struct Acc {
    unsigned long long fills, e, v, trav, nnz, chained;
};

constexpr int kPoor = 3;  // large searches a base may miss before another is looked for
constexpr int kIdleT = 16;  // sources that do not meet T before it is dropped

enum : int { PUB_X = 1, PUB_T = 2, PUB_LARGE = 4, PUB_DROP = 8 };

template <int BLOCK>
struct ChainSmem {
    long long item;
    int mi, skip, cta, sym, dup;
    int pub[2][2];         // [source parity][direction]: does X / T of that direction hold the source
    Tot base[2], tbase[2];  // X and T relative to the current source
    Tot pend[2];           // the last source's result, not yet counted
    int pend_fill[2], pend_trav[2], pend_chained[2];
    int have, have_t, tsel, used[2];
    int s, skip_pass;
    int large[2], mode[2], found[2];
    int hits;              // of the source in hand: 1: in X0, 2: in X1
    int hub, hub_at, hub_fails, hub_wait;
    int poor;              // large searches since the base was built that it did not keep
    int raw, orig, plen;
    Tot tot;
    Acc acc[2];
    BfsSmem<BLOCK> bfs;
    unsigned long long red[BLOCK / 32][4];
};

// ---- searches by the whole CTA --------------------------------------------------------

// The sizes of a bitmap's set relative to source s, left in SM.tot.  E (the
// degree sum) is direction 0's.  Block-wide.
template <int BLOCK, bool CG>
__device__ void block_census(ChainSmem<BLOCK>& SM, const MatDesc& M, const uint32_t* bm, int s,
                             int dir, bool digests) {
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
        if (dir != 0 || !xl) continue;
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

// What a warp needs of its direction.
struct Side {
    Graph G;
    uint32_t* X;   // the dense base's set
    uint32_t* g;   // a zero bitmap in global memory
    Sparse* P;
};

// Direction d's half of the sources SM.s .. s_end - 1.  Returns (both warps
// together) at the end of the chunk, or after a source whose search one of
// them left to the CTA; SM.s is that source, or s_end.
template <int BLOCK, bool CG>
__device__ void warp_walk(ChainSmem<BLOCK>& SM, const MatDesc& M, const Side& D, int d, int s_end,
                          int list_cap) {
    const int lane = threadIdx.x & 31;
    const bool sym = SM.sym != 0;
    const bool dup = SM.dup != 0;
    const bool digests = M.dig_u != nullptr;
    Sparse& P = *D.P;
    int s = SM.s;
    bool skip_pass = SM.skip_pass != 0;
    bool have = SM.have != 0, have_t = SM.have_t != 0;
    int tsel = SM.tsel, used = SM.used[d];
    Tot bx = SM.base[d], bt = SM.tbase[d];
    Acc acc = {0, 0, 0, 0, 0, 0};
    auto pair_sync = [&]() {
        if (sym) __syncwarp();
        else asm volatile("bar.sync 1, 64;" ::: "memory");
    };
    auto in_x = [&](int v) { return (ld_vol(D.X + (v >> 5)) >> (v & 31)) & 1u; };
    auto in_t = [&](int v) {
        return have_t ? (sparse_word(P.key[tsel], P.msk[tsel], v >> 5) >> (v & 31)) & 1u : 0u;
    };
    if (lane == 0) SM.pub[s & 1][d] = (have && in_x(s) ? PUB_X : 0) | (in_t(s) ? PUB_T : 0);
    int r0 = ld_i32<CG>(D.G.rp + s), r1 = ld_i32<CG>(D.G.rp + s + 1);
    int4 pre = make_int4(-1, -1, -1, -1);  // the first 128 entries of row s
    if (4 * lane < (r1 & ~3) - (r0 & ~3)) pre = ld_row4<CG>(D.G.cl + (r0 & ~3) + 4 * lane);
    int deg_prev = s > 0 ? row_degree<CG>(D.G.rp, s - 1) : 0;
    // the last source's counters, kept back until the other warp has finished it
    Tot pend = {0, 0, 0ull, 0ull};
    int pend_fill = 0, pend_trav = 0, pend_chained = 0;
    bool large = false;
    int mode = 0, found = 0, hits = 0;
    int idle = 0;  // sources since one met T
    for (;; s++) {
        pair_sync();
        const int f0 = SM.pub[s & 1][0], f1 = sym ? f0 : SM.pub[s & 1][1];
        if ((f0 | f1) & PUB_LARGE) {
            s--;
            break;
        }
        if ((f0 | f1) & PUB_DROP) have_t = false;
        acc.fills += (unsigned)pend_fill;
        acc.trav += (unsigned)pend_trav;
        acc.chained += (unsigned)pend_chained;
        acc.nnz += (unsigned)pend.gt;
        acc.v += (unsigned)pend.v;
        acc.e += pend.e;
        pend_fill = pend_trav = pend_chained = 0;
        pend.gt = pend.v = 0;
        pend.e = 0ull;
        if (s >= s_end) break;
        if (idle >= kIdleT) have_t = false;
        // xs: the base reaches s (direction 0) / s reaches the base (1); ts: the same for T
        const bool xs0 = have && (f0 & PUB_X), xs1 = have && (f1 & PUB_X);
        const bool ts0 = have_t && (f0 & PUB_T), ts1 = have_t && (f1 & PUB_T);
        idle = ts0 || ts1 ? 0 : idle + 1;
        const bool on_x = d ? xs0 : xs1, keep_x = d ? xs1 : xs0;
        const bool on_t = d ? ts0 : ts1, keep_t = d ? ts1 : ts0;
        hits = (xs0 ? 1 : 0) | (xs1 ? 2 : 0);
        mode = on_x ? 0 : on_t ? 1 : 2;
        // the next row's pointers, then (below) its first entries
        const int r2 = s + 2 <= M.n ? ld_i32<CG>(D.G.rp + s + 2) : r1;

        // the bases' sizes relative to s instead of s - 1
        if (!skip_pass) {
            const int w = s >> 5, wp = (s - 1) >> 5;
            if (have) {
                if (keep_x) {
                    bx.gt--;
                    if (digests) bx.dig += pass_digest(w, ld_vol(D.X + w), s);
                }
                if (s > 0 && in_x(s - 1)) {
                    bx.v++;
                    bx.e += (unsigned)deg_prev;
                }
            }
            if (have_t) {
                if (keep_t) {
                    bt.gt--;
                    if (digests) bt.dig += pass_digest(w, sparse_word(P.key[tsel], P.msk[tsel], w), s);
                }
                if (s > 0 && (sparse_word(P.key[tsel], P.msk[tsel], wp) >> ((s - 1) & 31)) & 1u) {
                    bt.v++;
                    bt.e += (unsigned)deg_prev;
                }
            }
        }
        skip_pass = false;

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
                    old[c] = ws[c] >= 0 && ws[c] != s ? ld_vol(D.X + (ws[c] >> 5)) : ~0u;
                    any |= !((old[c] >> (ws[c] & 31)) & 1u);
                }
                if (!__any_sync(FULL_MASK, any)) return true;  // all of them known
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    const uint32_t bit = 1u << (ws[c] & 31);
                    old[c] = old[c] & bit ? ~0u : atomicOr(D.X + (ws[c] >> 5), bit);
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
                if (k0 + 128 + 4 * lane < plen) qn = ld_row4<CG>(D.G.cl + b + k0 + 128 + 4 * lane);
                raw += (q4.x > s) + (q4.y > s) + (q4.z > s) + (q4.w > s);
                large = !visit(q4);
                q4 = qn;
            }
            if (lane == 0) trav += plen;
        }
        // the next row's first entries load while this search goes on
        pre = make_int4(-1, -1, -1, -1);
        if (4 * lane < (r2 & ~3) - (r1 & ~3)) pre = ld_row4<CG>(D.G.cl + (r1 & ~3) + 4 * lane);
        for (int h = 0; h < found && !large; h += 32) {
            const int u = h + lane < found ? P.list[h + lane] : INT_MAX;
            int s0 = 0, its = 0;
            if (u < s) {
                const int a0 = ld_i32<CG>(D.G.rp + u), a1 = ld_i32<CG>(D.G.rp + u + 1);
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
            int4 q4 = at >= 0 ? ld_row4<CG>(D.G.cl + at) : make_int4(-1, -1, -1, -1);
            for (int j0 = 0; j0 < total && !large; j0 += 32) {
                int4 qn = make_int4(-1, -1, -1, -1);
                if (j0 + 32 < total) {
                    at = flat_int4(j0 + 32 + lane, total, s0, its, incl, &o);
                    if (at >= 0) qn = ld_row4<CG>(D.G.cl + at);
                }
                large = !visit(q4);
                q4 = qn;
            }
            // a partial group of 32: the ids found meanwhile start the next one
            if (have_now - h < 32) h = have_now - 32;
        }
        trav = __shfl_sync(FULL_MASK, trav, 0);
        pend_trav = trav;
        if (!large) {
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
            const int orig = dup ? row_distinct<CG>(D.G, s, D.g) : raw;
            if (lane == 0) write_row(M, s, d, sym, t, raw, orig);
            if (d == 1 || sym) {
                // the 128 ids after s of the L column
                uint32_t word = 0;
                if (lane < 5) {
                    const int w = ((s + 1) >> 5) + lane;
                    word = mode == 0 ? ld_vol(D.X + w) : sparse_word(key, msk, w);
                }
                word = next128(word, s);
                if (lane < 4) M.lmask[4ll * s + lane] = word;
            }
            pend = t;
            pend_fill = (t.gt - orig) * (sym ? 2 : 1);
            pend_chained = mode != 2;

            // the bases for s + 1
            int drop = 0;
            if (keep_x) {
                if (mode == 0) {
                    bx = t;
                } else {
                    // F(s) joins X word by word
                    int ag = 0, av = 0;
                    unsigned ae = 0;
                    unsigned long long ad = 0;
                    for (int i = lane; i < kSlots; i += 32) {
                        const uint32_t k = key[i];
                        if (k == kFree) continue;
                        const int w = (int)k;
                        const uint32_t m = msk[i] & ~(w == (s >> 5) ? 1u << (s & 31) : 0u);
                        if (!m) continue;
                        const uint32_t old = atomicOr(D.X + w, m);
                        const uint32_t nb = m & ~old;
                        if (!nb) continue;
                        ag += __popc(nb & above(w, s));
                        if (digests) ad += digest_step(w, old, old | m, s);
                        for (uint32_t t2 = nb & below(w, s); t2; t2 &= t2 - 1) {
                            av++;
                            if (d == 0) ae += (unsigned)row_degree<CG>(M.rowptr, 32 * w + __ffs(t2) - 1);
                        }
                    }
                    bx.gt += __reduce_add_sync(FULL_MASK, ag);
                    bx.v += __reduce_add_sync(FULL_MASK, av);
                    bx.e += (unsigned)__reduce_add_sync(FULL_MASK, ae);
                    if (digests) bx.dig += warp_sum64(ad);
                }
            } else if (mode == 0) {
                for (int i = lane; i < found; i += 32) {
                    const int w = P.list[i];
                    atomicAnd(D.X + (w >> 5), ~(1u << (w & 31)));
                }
            }
            if ((ts0 && xs1) || (ts1 && xs0)) {
                have_t = false;  // T reaches into the dense base (or back): it is as large as that
            } else if (have_t) {
                if (keep_t && mode == 1) {
                    bt = t;
                    used = words;
                } else if (keep_t) {
                    int ag = 0, av = 0, nslots = 0;
                    unsigned ae = 0;
                    unsigned long long ad = 0;
                    bool full = false;
                    uint32_t* const tk = P.key[tsel];
                    uint32_t* const tm = P.msk[tsel];
                    for (int i = lane; i < kSlots; i += 32) {
                        const uint32_t k = key[i];
                        const uint32_t m = msk[i];
                        if (k == kFree || !m) continue;
                        const int w = (int)k;
                        const int j = sparse_slot(tk, w, &nslots);
                        if (j < 0) {
                            full = true;
                            continue;
                        }
                        const uint32_t old = atomicOr(tm + j, m);
                        const uint32_t nb = m & ~old;
                        ag += __popc(nb & above(w, s));
                        if (digests && nb) ad += digest_step(w, old, old | m, s);
                        for (uint32_t t2 = nb & below(w, s); t2; t2 &= t2 - 1) {
                            av++;
                            if (d == 0) ae += (unsigned)row_degree<CG>(M.rowptr, 32 * w + __ffs(t2) - 1);
                        }
                    }
                    bt.gt += __reduce_add_sync(FULL_MASK, ag);
                    bt.v += __reduce_add_sync(FULL_MASK, av);
                    bt.e += (unsigned)__reduce_add_sync(FULL_MASK, ae);
                    if (digests) bt.dig += warp_sum64(ad);
                    used += __reduce_add_sync(FULL_MASK, nslots);
                    if (__any_sync(FULL_MASK, full) || used > kSlotsMax) drop = PUB_DROP;
                } else if (mode == 1) {
                    for (int i = lane; i < found; i += 32) {
                        const int w = P.list[i];
                        int none = 0;
                        const int j = sparse_slot(key, w >> 5, &none);  // present
                        if (j >= 0) atomicAnd(msk + j, ~(1u << (w & 31)));
                    }
                    used = words;
                }
            }
            if (!xs0 && !xs1 && !ts0 && !ts1) {
                // s met no base: its own sets are the new T
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
            if (lane == 0 && s + 1 < M.n)
                SM.pub[(s + 1) & 1][d] =
                    (have && in_x(s + 1) ? PUB_X : 0) | (in_t(s + 1) ? PUB_T : 0) | drop;
            else if (lane == 0)
                SM.pub[(s + 1) & 1][d] = drop;
        } else if (lane == 0) {
            SM.pub[(s + 1) & 1][d] = PUB_LARGE;
        }
        deg_prev = (r1 & ~3) - (r0 & ~3) - (r1 & 3);
        r0 = r1;
        r1 = r2;
    }
    if (lane == 0) {
        SM.base[d] = bx;
        SM.pend[d] = pend;
        SM.pend_fill[d] = pend_fill;
        SM.pend_trav[d] = pend_trav;
        SM.pend_chained[d] = pend_chained;
        SM.large[d] = large;
        SM.mode[d] = mode;
        SM.found[d] = found;
        Acc& A = SM.acc[d];
        A.fills += acc.fills;
        A.e += acc.e;
        A.v += acc.v;
        A.trav += acc.trav;
        A.nnz += acc.nnz;
        A.chained += acc.chained;
        if (d == 0) {
            SM.s = s;
            SM.hits = hits;
            SM.tsel = tsel;
        }
    }
}

// ---- sources the whole CTA takes ---------------------------------------------------------

template <int BLOCK, bool CG>
struct Large {
    ChainSmem<BLOCK>& SM;
    const MatDesc& M;
    const Side* D;  // [2]
    int32_t* q;
    long long qcap;
    long long words;
    int32_t* status;

    // Row s's entry counts into SM.raw, SM.orig.
    __device__ void row_stats(int d, int s) {
        if (threadIdx.x < 32) {
            const int lane = threadIdx.x;
            const Graph& G = D[d].G;
            const int b = ld_i32<CG>(G.rp + s) & ~3, e = ld_i32<CG>(G.rp + s + 1) & ~3;
            int raw = 0;
            for (int j = b + lane; j < e; j += 32) raw += ld_i32<CG>(G.cl + j) > s;
            raw = __reduce_add_sync(FULL_MASK, raw);
            const int orig = SM.dup ? row_distinct<CG>(G, s, D[d].g) : raw;
            if (lane == 0) {
                SM.raw = raw;
                SM.orig = orig;
                SM.bfs.rtrav = 0;
            }
        }
        __syncthreads();
    }

    // Outputs and counters of source s in direction d, whose set is bm and
    // whose sizes are SM.tot.
    __device__ void emit(int d, int s, const uint32_t* bm, bool chained) {
        const bool sym = SM.sym != 0;
        if (threadIdx.x < 32) {
            const int lane = threadIdx.x;
            if (d == 1 || sym) {
                uint32_t word = lane < 5 ? bm[((s + 1) >> 5) + lane] : 0u;
                word = next128(word, s);
                if (lane < 4) M.lmask[4ll * s + lane] = word;
            }
            if (lane == 0) {
                const Tot t = SM.tot;
                write_row(M, s, d, sym, t, SM.raw, SM.orig);
                Acc& A = SM.acc[d];
                A.fills += (unsigned long long)(t.gt - SM.orig) * (sym ? 2 : 1);
                A.e += t.e;
                A.v += (unsigned)t.v;
                A.nnz += (unsigned)t.gt;
                A.trav += SM.bfs.rtrav;
                A.chained += chained ? 1 : 0;
            }
        }
        __syncthreads();
    }

    __device__ void commit_pending(int d) {
        if (threadIdx.x == 0) {
            Acc& A = SM.acc[d];
            A.fills += (unsigned)SM.pend_fill[d];
            A.e += SM.pend[d].e;
            A.v += (unsigned)SM.pend[d].v;
            A.nnz += (unsigned)SM.pend[d].gt;
            A.trav += (unsigned)SM.pend_trav[d];
            A.chained += (unsigned)SM.pend_chained[d];
        }
    }

    // s alone in the dense sets of direction d: the base's set and the result
    __device__ void rebuild_from(int d, int s, bool digests) {
        row_stats(d, s);
        if (threadIdx.x == 0) {
            q[0] = s;
            D[d].X[s >> 5] |= 1u << (s & 31);
        }
        block_bfs<BLOCK, CG>(SM.bfs, D[d].G, D[d].X, q, qcap, 1, s, s, false, status);
        block_census<BLOCK, CG>(SM, M, D[d].X, s, d, digests);
        emit(d, s, D[d].X, false);
        if (threadIdx.x == 0) SM.base[d] = SM.tot;
        __syncthreads();
    }

    // Symmetric patterns: s's search has outgrown its table.  Every id in the
    // table is reached by s (with T's base, which s reaches), and all but those
    // of the list are expanded: the table becomes X, and the search goes on there.
    __device__ void promote(int s, bool digests) {
        const Sparse& P = *D[0].P;
        const int found = SM.found[0];
        const int which = SM.mode[0] == 1 ? SM.tsel : 1 - SM.tsel;
        row_stats(0, s);
        block_clear<BLOCK>(D[0].X, words);
        __syncthreads();
        for (int i = threadIdx.x; i < kSlots; i += BLOCK)
            if (P.key[which][i] != kFree) D[0].X[P.key[which][i]] = P.msk[which][i];
        for (int i = threadIdx.x; i <= found; i += BLOCK) {
            if (i < qcap) q[i] = i ? P.list[i - 1] : s;
            else atomicOr(status, DEV_ERR_QUEUE);
        }
        __syncthreads();
        if (threadIdx.x == 0) D[0].X[s >> 5] |= 1u << (s & 31);
        __syncthreads();
        block_bfs<BLOCK, CG>(SM.bfs, D[0].G, D[0].X, q, qcap, found + 1, s, s, false, status);
        block_census<BLOCK, CG>(SM, M, D[0].X, s, 0, digests);
        emit(0, s, D[0].X, SM.mode[0] == 1);
        if (threadIdx.x == 0) SM.base[0] = SM.tot;
        __syncthreads();
    }

    // the search of s goes on in X
    __device__ void overlaid(int d, int s, bool keep, bool digests) {
        row_stats(d, s);
        const int found = SM.found[d];
        for (int i = threadIdx.x; i <= found; i += BLOCK) {
            if (i < qcap) q[i] = i ? D[d].P->list[i - 1] : s;
            else atomicOr(status, DEV_ERR_QUEUE);
        }
        const long long end = block_bfs<BLOCK, CG>(SM.bfs, D[d].G, D[d].X, q, qcap, found + 1, s, s, true, status);
        block_census<BLOCK, CG>(SM, M, D[d].X, s, d, digests);
        emit(d, s, D[d].X, true);
        if (keep) {
            if (threadIdx.x == 0) SM.base[d] = SM.tot;
        } else {
            for (long long i = 1 + threadIdx.x; i < end; i += BLOCK)
                atomicAnd(D[d].X + (q[i] >> 5), ~(1u << (q[i] & 31)));
        }
        __syncthreads();
    }

    // the search of s alone in the global bitmap; its set joins X when the base reaches s
    __device__ void alone(int d, int s, bool keep, bool digests) {
        uint32_t* const g = D[d].g;
        row_stats(d, s);
        if (threadIdx.x == 0) q[0] = s;
        block_bfs<BLOCK, CG>(SM.bfs, D[d].G, g, q, qcap, 1, s, s, false, status);
        block_census<BLOCK, CG>(SM, M, g, s, d, digests);
        emit(d, s, g, false);
        if (keep) {
            for (long long i = threadIdx.x; i < words; i += BLOCK) D[d].X[i] |= g[i];
            __syncthreads();
            block_census<BLOCK, CG>(SM, M, D[d].X, s, d, digests);
            if (threadIdx.x == 0) SM.base[d] = SM.tot;
        }
        __syncthreads();
        block_clear<BLOCK>(g, words);
        __syncthreads();
    }

    // A hub for the one-sided search of direction d: its reach set in the
    // other direction first, in the global bitmap; not above `least`: no base.
    __device__ bool try_hub(int d, int s, int least, bool digests) {
        if (threadIdx.x < 32) {
            const int lane = threadIdx.x;
            const int32_t* rp = D[1 - d].G.rp;
            int best = -1, id = -1;
            for (int i = lane; i < SM.found[d]; i += 32) {
                const int v = D[d].P->list[i];
                if (v >= s) continue;
                const int deg = row_degree<CG>(rp, v);
                if (deg > best) {
                    best = deg;
                    id = v;
                }
            }
            const int m = __reduce_max_sync(FULL_MASK, best);
            const unsigned who = __ballot_sync(FULL_MASK, best == m && id >= 0);
            id = who ? __shfl_sync(FULL_MASK, id, __ffs(who) - 1) : -1;
            if (lane == 0) {
                SM.hub = id;
                SM.bfs.rtrav = 0;
            }
        }
        __syncthreads();
        const int hub = SM.hub;
        if (hub < 0) return false;
        const int o = 1 - d;
        uint32_t* const g = D[o].g;
        if (threadIdx.x == 0) {
            q[0] = hub;
            g[hub >> 5] = 1u << (hub & 31);
        }
        long long size = block_bfs<BLOCK, CG>(SM.bfs, D[o].G, g, q, qcap, 1, -1, s, false, status);
        const bool ok = size > least;
        if (ok) {
            for (long long i = threadIdx.x; i < words; i += BLOCK) {
                D[o].X[i] = g[i];
                D[d].X[i] = 0u;
            }
            __syncthreads();
            if (threadIdx.x == 0) {
                q[0] = hub;
                D[d].X[hub >> 5] = 1u << (hub & 31);
            }
            block_bfs<BLOCK, CG>(SM.bfs, D[d].G, D[d].X, q, qcap, 1, -1, s, false, status);
            for (int k = 0; k < 2; k++) {
                block_census<BLOCK, CG>(SM, M, D[k].X, s, k, digests);
                if (threadIdx.x == 0) SM.base[k] = SM.tot;
                __syncthreads();
            }
        }
        __syncthreads();
        block_clear<BLOCK>(g, words);
        if (threadIdx.x == 0) SM.acc[d].trav += SM.bfs.rtrav;
        __syncthreads();
        return ok;
    }

    // Failed attempts are further and further apart; one a source, so that every
    // pass through take() makes progress.
    __device__ void note_hub(bool ok, int s) {
        if (threadIdx.x == 0) {
            SM.hub_at = s;
            SM.hub_fails = ok ? 0 : min(SM.hub_fails + 1, 6);
            SM.hub_wait = ok ? 0 : (1 << SM.hub_fails) - 1;
        }
        __syncthreads();
    }

    // Source SM.s, whose search in at least one direction is large.  Leaves
    // SM.s at the source to go on with.
    __device__ void take() {
        const int s = SM.s, hits = SM.hits;
        const bool sym = SM.sym != 0, digests = M.dig_u != nullptr;
        const bool l0 = SM.large[0] != 0, l1 = !sym && SM.large[1] != 0;
        const bool have = SM.have != 0;
        const int hub_wait = SM.hub_wait;
        const bool tried = SM.hub_at == s;  // once a source: every pass through here makes progress
        __syncthreads();
        bool done = true, rebuilt = false;
        // a base that search after search outgrows lies beside the core: a hub
        // among what this one found takes its place if its other set is larger
        // than the base's smaller one
        const int miss = sym ? -1 : l0 && !(hits & 1) ? 0 : l1 && !(hits & 2) ? 1 : -1;
        if (hits && miss >= 0 && !tried && hub_wait == 0 && SM.poor >= kPoor) {
            const bool ok = try_hub(miss, s, max(kListCap, min(SM.base[0].v, SM.base[1].v)), digests);
            note_hub(ok, s);
            if (ok) {
                rebuilt = true;
                done = false;
            }
        }
        if (!hits) {
            // neither direction met the base
            bool rebuild = sym || (l0 && l1) || !have || tried;
            if (!sym && !(l0 && l1) && !tried) {
                bool ok = false;
                if (hub_wait == 0) {
                    ok = try_hub(l0 ? 0 : 1, s, kListCap, digests);
                    note_hub(ok, s);
                } else if (threadIdx.x == 0) {
                    SM.hub_wait = hub_wait - 1;
                }
                if (ok) {
                    rebuild = false;
                    done = false;  // s meets the hub: walk it again
                    rebuilt = true;
                }
            }
            if (rebuild && sym) {
                promote(s, digests);
                rebuilt = true;
            } else if (rebuild) {
                for (int k = 0; k < 2; k++) block_clear<BLOCK>(D[k].X, words);
                __syncthreads();
                for (int k = 0; k < 2; k++) rebuild_from(k, s, digests);
                rebuilt = true;
            }
        }
        if (!rebuilt) {
            for (int k = 0; k < (sym ? 1 : 2); k++) {
                if (!(k ? l1 : l0)) {
                    commit_pending(k);
                    continue;
                }
                const bool keep = sym ? (hits & 1) != 0 : (hits & (k ? 2 : 1)) != 0;
                if (SM.mode[k] == 0) overlaid(k, s, keep, digests);
                else alone(k, s, keep, digests);
            }
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            if (rebuilt) {
                SM.have = 1;
                SM.poor = 0;
            } else if (miss >= 0) {
                SM.poor++;
                if (SM.hub_wait > 0 && hits) SM.hub_wait--;
            }
            SM.have_t = 0;
            SM.tsel = 0;
            SM.s = done ? s + 1 : s;
            SM.skip_pass = done ? 0 : 1;
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
    uint32_t* const sbm = reinterpret_cast<uint32_t*>(sparse + P.sides);
    uint32_t* const gb = P.gbm + cta * P.gbm_count * P.bitmap_words;
    int32_t* const q = P.queue + cta * P.queue_stride;
    for (long long i = threadIdx.x; i < 2 * P.bitmap_words; i += BLOCK) gb[i] = 0u;
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
                        SM.sym = __ldcg(SD.asym) == 0;
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
                SM.sym = SD.asym[0] == 0;
                SM.dup = SD.asym[1] != 0;
            }
            SM.item = it;
        }
        __syncthreads();
        if (SM.item < 0) break;
        const MatDesc& M = SD;
        const int32_t n = M.n;
        const bool sym = SM.sym != 0;
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
        // (a launch planned for symmetric patterns alone has tables for one direction)
        const bool in_smem = (sym ? 1 : 2) * words <= P.smem_words;
        uint32_t* const x0 = in_smem ? sbm : gb + 2 * P.bitmap_words;
        uint32_t* const x1 = in_smem ? sbm + words : gb + 3 * P.bitmap_words;
        if (threadIdx.x == 0) {
            SM.s = s_first;
            SM.skip_pass = 0;
            SM.have = SM.have_t = SM.tsel = 0;
            SM.hub_fails = SM.hub_wait = 0;
            SM.hub_at = -1;
            SM.poor = 0;
            for (int d = 0; d < 2; d++) {
                SM.used[d] = 0;
                SM.large[d] = 0;
                SM.acc[d] = Acc{0, 0, 0, 0, 0, 0};
            }
        }
        const Side D[2] = {{{M.rowptr, M.col}, x0, gb, sparse},
                           {{M.trowptr, M.tcol}, x1, gb + P.bitmap_words, sparse + 1}};
        __syncthreads();
        while (SM.s < s_end) {
            const int dirs = sym ? 1 : 2;
            __syncthreads();  // everyone has read SM.s
            if (warp < dirs) warp_walk<BLOCK, CG>(SM, M, D[warp], warp, s_end, P.list_cap);
            __syncthreads();
            if (SM.large[0] || (!sym && SM.large[1])) {
                Large<BLOCK, CG> L{SM, M, D, q, P.queue_stride, words, P.status};
                L.take();
                if (threadIdx.x == 0) SM.large[0] = SM.large[1] = 0;
                __syncthreads();
            }
        }
        if constexpr (SERVE) __threadfence();
        __syncthreads();
        if (threadIdx.x == 0) {
            unsigned long long* c = M.counters;
            const Acc &a = SM.acc[0], &b = SM.acc[1];
            atomicAdd(c + CNT_FILLS, a.fills + b.fills);
            atomicAdd(c + CNT_EDGES_ALG, a.e);
            atomicAdd(c + CNT_VERTS_ALG, a.v);
            atomicAdd(c + CNT_EDGES_TRAV, a.trav + b.trav);
            atomicAdd(c + CNT_NNZ_U, a.nnz);
            atomicAdd(c + CNT_NNZ_L, sym ? a.nnz : b.nnz);
            atomicAdd(c + CNT_CHAINED, a.chained + b.chained);
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

size_t chain_sparse_bytes(int sides) { return (size_t)sides * sizeof(Sparse); }
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
