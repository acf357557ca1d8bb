// claim_kernels.cuh -- the filter + verify kernels (the plain method's filter
// passes too): k_claim (a CTA per query) and k_tiny (a warp per query of few window entries).  Same
// semantics as k_fused (fused_kernels.cuh), whose keyed slot table remains for
// the strategies a caller asks for, tuned keyed shapes and probe prefixes above
// kClaimPC tokens.
//
// What bounds it: instruction issue and the latency of shared and L2 accesses
// (DRAM at about 1 % of its rate), so the design cuts instructions per window
// entry.  k_fused spends 8.4 warp instructions on an entry, most of them in
// the compare-and-swap loop of its slot table, with half the lanes idle; a claim
// is a store, a load and, for a quarter of the entries, two native atomics.  The
// id ranges of a step come from the join's block table (JoinArgs.tab), shared by
// every query, instead of a binary search per query, probe token and
// range.  Measured (filter kernels of a call, chunk splits included): 1,000,000
// heavy-tailed records at t = 0.7 177 -> 95 ms, 100,000 titles at t = 0.5
// 12.1 -> 4.2 ms, 2 x 60,000 titles R-S at t = 0.6 6.3 -> 3.4 ms, 500,000
// reads at t = 0.8 2.8 -> 0.99 ms, 100,000 titles at t = 0.7 with the plain method's
// two passes 8.4 -> 1.6 ms.
#pragma once

#include "fused_kernels.cuh"
#include "tiles.cuh"

namespace fgss {

// The kernels run in three modes: MODE_FUSED verifies and emits the results (the
// batched method); MODE_COUNT adds every query's sources that need verification to
// a.vcnt, MODE_FILL writes them as (query, source, matches, query position of the
// last) from a.cand[a.voff[query]] (the plain method's two passes; a.ccnt is the
// fill's cursor, zero at launch).  Candidates and window entries are counted in the
// first two.

// Lanes' sources of one query into the plain method's counts or records
// (warp-collective): bit `take` lanes give (s, cj = matches | query position << 16).
template <int MODE>
__device__ __forceinline__ void plain_take(const JoinArgs& a, uint32_t q, bool take, uint32_t s, uint32_t cj) {
    const uint32_t m = __ballot_sync(kFull, take);
    if (m == 0) return;
    uint32_t base = 0;
    if (lane_id() == 0) base = atomicAdd(MODE == MODE_COUNT ? &a.vcnt[q] : &a.ccnt[q], (uint32_t)__popc(m));
    if (MODE == MODE_COUNT) return;
    const uint32_t i = __shfl_sync(kFull, base, 0) + __popc(m & lanemask_lt());
    if (!take) return;
    if (i < a.vcnt[q]) a.cand[a.voff[q] + i] = make_uint4(q, s, cj & 0xffffu, cj >> 16);
    else atomicOr(a.status, ST_HASH_FULL);
}

__device__ __forceinline__ void bar_named(uint32_t id, uint32_t threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
// The barrier with the disjunction of every thread's p.
__device__ __forceinline__ bool bar_or(uint32_t id, uint32_t threads, bool p) {
    uint32_t r;
    asm volatile("{\n .reg .pred x, y;\n setp.ne.u32 x, %3, 0;\n bar.red.or.pred y, %1, %2, x;\n"
                 " selp.u32 %0, 1, 0, y;\n}"
                 : "=r"(r) : "r"(id), "r"(threads), "r"((uint32_t)p) : "memory");
    return r != 0;
}

// ------------------------------------------------------------------- k_claim

// Shared-memory layout of k_claim: NTC consumer threads, U entries of a step in
// each one's registers, 2^HL claim slots.
template <int NTC_, int U_, int HL_>
struct ClaimShape {
    static constexpr uint32_t NTC = NTC_, NT = NTC_ + 32, NWC = NTC_ / 32, U = U_;
    static constexpr uint32_t HLOG = HL_, H = 1u << HL_;
    static constexpr uint32_t PC = kClaimPC;
    static constexpr uint32_t JE = NTC * U;   // entries of a step
    static constexpr uint32_t JW = JE / 32;   // their groups of 32
    static constexpr uint32_t QC = 256;       // query tokens staged (longer: read from global memory)
    static constexpr uint32_t BW = 1024;      // membership words: one bit per term up to 32768 terms
    static constexpr uint32_t MC = 256;       // merge list
    static constexpr size_t off_agg = 0;                          // uint2[JE]
    static constexpr size_t off_src = off_agg + 8ull * JE;        // u32[JE]
    static constexpr size_t off_slot = off_src + 4ull * JE;       // u16[H]
    static constexpr size_t off_vl = off_slot;                    // u16[JE], once the claims are settled
    static constexpr size_t off_wfe = off_slot + 2ull * H;        // u32[2][PC]
    static constexpr size_t off_wj = off_wfe + 2 * 4ull * PC;     // u16[2][PC]
    static constexpr size_t off_grp = off_wj + 2 * 2ull * PC;     // uint2[2][JW]
    static constexpr size_t off_qtok = off_grp + 2 * 8ull * JW;   // u32[2][QC]
    static constexpr size_t off_bm = off_qtok + 2 * 4ull * QC;    // u32[BW]
    static constexpr size_t off_ml = off_bm + 4ull * BW;          // u32[3][MC]
    static constexpr size_t bytes = off_ml + 3 * 4ull * MC;
    static_assert(off_bm % 16 == 0 && off_grp % 8 == 0 && JE <= 65536 && PC <= JE && PC < 1024 && JE <= H, "k_claim layout");
    static_assert(MC <= 32 * NWC, "a warp's share of the merge list fits its lanes");
};

// Work items of k_claim: a list of (join, first query, end), or without one n
// tiles of the map in order from `first` -- records come in descending size, so the
// costly queries still come first.
struct ClaimItems {
    const uint4* list;
    TileMap m;
    uint32_t first, n;
};
__device__ __forceinline__ uint4 claim_item(const ClaimItems& I, uint32_t it) {
    if (I.list) return I.list[it];
    const TileRange t = tile_range(I.m, I.first + it);
    return make_uint4(t.j, t.r0, t.r1, 0);
}

// What the consumers do next: the entries of a range of the query's id
// window, laid out in rank form in buffer (step & 1).
struct ClaimStep {
    uint32_t join, q, lq, pos, L, flags;
};
enum : uint32_t {
    CS_FIRST = 1,    // first step of its query
    CS_END = 2,      // no step left
    CS_UNSORTED = 4  // the join's records are not sorted by size
};

// Producer warp: walks the work items and lays out the steps, one ahead of
// the consumers.
template <typename S, int MODE>
__device__ void claim_producer(const JoinArgs* __restrict__ joins, const FusedArgs* __restrict__ fargs,
                               const ClaimItems& items, uint32_t* counter, unsigned char* smem, ClaimStep* steps) {
    const uint32_t lane = lane_id(), lt = lanemask_lt();
    uint32_t k = 0;  // steps published
    uint32_t cur = 0xffffffffu;
    unsigned long long n_win = 0, n_tok = 0;  // window entries and query tokens of join cur
    auto flush_counts = [&] {
        if (lane == 0 && n_win && MODE != MODE_FILL) {
            atomicAdd(&joins[cur].stats[SS_WINDOW], n_win);
            if (MODE == MODE_FUSED) atomicAdd(&joins[cur].stats[SS_QTOK], n_tok);
        }
        n_win = n_tok = 0;
    };
    auto publish = [&](const ClaimStep& st) {
        if (lane == 0) steps[k & 1] = st;
        __syncwarp();
        bar_named(1, S::NT);
        k++;
    };
    uint32_t it = 0;
    if (lane == 0) it = atomicAdd(counter, 1u);
    it = __shfl_sync(kFull, it, 0);
    while (it < items.n) {
        const uint4 w = claim_item(items, it);
        uint32_t ahead = 0;
        if (lane == 0) ahead = atomicAdd(counter, 1u);
        const JoinArgs& a = joins[w.x];
        const FusedArgs& fa = fargs[w.x];
        if (w.x != cur) {
            flush_counts();
            cur = w.x;
        }
        const uint32_t bits = *a.status;
        const bool unsorted = (bits & ST_UNSORTED) != 0;
        const uint32_t* __restrict__ tab = a.tab;
        const uint64_t nb = a.nb;
        for (uint32_t q0 = w.y; q0 < w.z && !(bits & ST_SKIP_ALL); q0 += 32) {
            const uint4 m = q0 + lane < w.z ? fa.meta[q0 + lane] : make_uint4(0, 0, QC_NONE << 16, 0);
#pragma unroll 1
            for (uint32_t todo = __ballot_sync(kFull, (m.z >> 16) == QC_CLAIM); todo; todo &= todo - 1) {
                const uint32_t src = __ffs(todo) - 1, q = q0 + src;
                ClaimStep st;
                st.join = w.x;
                st.q = q;
                st.pos = __shfl_sync(kFull, m.x, src);
                st.lq = __shfl_sync(kFull, m.y, src);
                const uint32_t W = __shfl_sync(kFull, m.w, src);
                const uint32_t qp = a.probe[st.lq];
                n_win += W;
                n_tok += st.lq;
                st.flags = CS_FIRST | (unsorted ? CS_UNSORTED : 0u);
                const uint32_t send = unsorted ? a.n : a.send[st.lq];
                const uint32_t* __restrict__ qt = a.tok + st.pos;
                const uint2* __restrict__ win = fa.win + fa.poff[q];
                // First entry of probe window j (of list t) at or after source x of [q + 1, send].
                auto bound = [&](uint32_t j, uint32_t t, uint32_t x) -> uint32_t {
                    if (x <= q + 1) return __ldg(&win[j].x);
                    if (x >= send) return __ldg(&win[j].y);
                    if (nb == 0) {
                        const uint2 wn = __ldg(win + j);
                        return lower_bound_src(a.ent, wn.x, wn.y, x);
                    }
                    const uint32_t* row = tab + (uint64_t)t * nb + x / kBlockIds;
                    const uint32_t lo = __ldg(row);
                    return x % kBlockIds ? lower_bound_src(a.ent, lo, __ldg(row + 1), x) : lo;
                };
                // Rank form of the entries with sources in [ra, rb): the windows that hold some get
                // ranks r in order, wfe[r] = first entry - entries of the earlier windows, wj[r] =
                // probe position; grp[g] = (bit per window start, windows starting before entry
                // 32 g; the window that holds that entry writes it).  Returns their number (above
                // JE: more than a step, the layout is not used).
                auto layout = [&](uint32_t ra, uint32_t rb) -> uint32_t {
                    uint32_t* wfe = reinterpret_cast<uint32_t*>(smem + S::off_wfe) + (k & 1) * S::PC;
                    uint16_t* wj = reinterpret_cast<uint16_t*>(smem + S::off_wj) + (k & 1) * S::PC;
                    uint2* grp = reinterpret_cast<uint2*>(smem + S::off_grp) + (k & 1) * S::JW;
                    for (uint32_t g = lane; g < S::JW; g += 32) grp[g].x = 0u;
                    __syncwarp();
                    uint32_t carry = 0, rc = 0;
#pragma unroll 1
                    for (uint32_t j0 = 0; j0 < qp; j0 += 64) {
                        uint32_t lo2[2], hi2[2];
#pragma unroll
                        for (uint32_t x = 0; x < 2; x++) {
                            const uint32_t j = j0 + 32 * x + lane;
                            lo2[x] = hi2[x] = 0;
                            if (j < qp) {
                                const uint32_t t = __ldg(qt + j);
                                lo2[x] = bound(j, t, ra);
                                hi2[x] = bound(j, t, rb);
                            }
                        }
#pragma unroll
                        for (uint32_t x = 0; x < 2; x++) {
                            const uint32_t cnt = hi2[x] - lo2[x];
                            const uint32_t nz = __ballot_sync(kFull, cnt != 0);
                            if (nz == 0) continue;
                            const uint32_t incl = warp_incl_scan(cnt);
                            const uint32_t p = carry + incl - cnt;  // entries of the earlier windows
                            if (cnt != 0 && p < S::JE) {
                                const uint32_t r = rc + __popc(nz & lt), e = min(p + cnt, S::JE);
                                wfe[r] = lo2[x] - p;
                                wj[r] = (uint16_t)(j0 + 32 * x + lane);
                                atomicOr(&grp[p >> 5].x, 1u << (p & 31));
                                for (uint32_t g = (p + 31) >> 5; g * 32 < e; g++) grp[g].y = g * 32 == p ? r : r + 1;
                            }
                            carry += __shfl_sync(kFull, incl, 31);
                            rc += __popc(nz);
                        }
                    }
                    __syncwarp();
                    return carry;
                };
                // Id ranges: the whole window when its entries fit a step, else as many ids as fill
                // 7/8 of a step at the density so far, ending on a block of the table where that
                // gives up little (a bound inside a block takes a search); too many entries halve
                // the range (one id has at most PC of them).
                constexpr uint32_t kAim = S::JE - S::JE / 8;
                uint64_t ids = W > S::JE ? max((uint64_t)kAim * (send - q - 1) / W, (uint64_t)1) : send;
                uint32_t left = W;
#pragma unroll 1
                for (uint32_t ra = q + 1; ra < send && left;) {
                    uint32_t rb = ids < send - ra && left > S::JE ? ra + (uint32_t)ids : send, L;
#pragma unroll 1
                    for (;;) {
                        if (rb < send && rb % kBlockIds < (rb - ra) / 4) rb -= rb % kBlockIds;
                        L = layout(ra, rb);
                        if (L <= S::JE) break;
                        rb = ra + (rb - ra) / 2;
                    }
                    if (L) {
                        st.L = L;
                        publish(st);
                        st.flags &= ~CS_FIRST;
                        ids = max((uint64_t)kAim * (rb - ra) / L, (uint64_t)1);
                        left -= L;
                    }
                    ra = rb;
                }
            }
        }
        it = __shfl_sync(kFull, ahead, 0);
    }
    flush_counts();
    ClaimStep end = {};
    end.flags = CS_END;
    publish(end);
}

// A query as the consumers keep it in shared memory, two by turns.
struct ClaimQuery {
    uint4 bits[4];  // its bitmap (zero beyond bmw)
    uint32_t join, q, lq, pos, qmode;
};

// One source (the same in every lane) merged by the warp at once, the merge
// list being full; the membership structure may not be complete yet, so the
// query's tokens are searched.
__device__ __noinline__ void merge_now(const JoinArgs& a, const FusedArgs& fa, const ClaimQuery& cq, uint32_t s,
                                       uint32_t y, uint32_t cj, const uint32_t* qsrc, unsigned long long* s_cnt) {
    const uint32_t ls = y >> 16, c = cj & 0xffffu, j = cj >> 16, qrest = cq.lq - j - 1, k0 = (y & 0xffffu) + 1;
    const uint4 sm = __ldg(fa.smin + cq.lq + ls);
    const uint32_t* st = a.tok + fa.meta[s].x;
    uint32_t k = k0, cnt = c;
    while (k < ls && cnt + min(ls - k, qrest - (cnt - c)) >= sm.y) {
        const uint32_t kk = k + lane_id();
        const bool hit = kk < ls && contains_gen(qsrc, j + 1, cq.lq, __ldg(st + kk));
        cnt += __popc(__ballot_sync(kFull, hit));
        k = min(k + 32u, ls);
    }
    if (lane_id() == 0) {
        FusedCounters ctr = {0, 0, 0, 0, 0, 0, 0};
        tally_overlap(a, ctr, cq.q, s, cnt, sm.y, sm.z);
        if (ctr.inter) atomicAdd(&s_cnt[0], 1ull);
        if (ctr.res) atomicAdd(&s_cnt[1], 1ull);
        atomicAdd(&s_cnt[2], (unsigned long long)(k - k0));
    }
}

// Consumer warps.  A step's entries, numbered f in (query position, source)
// order, sit in the threads' registers:
//   P1  entry f writes f into the claim slot of its source (the low bits of
//       the id) and its source into src[f]; some entry's number stays;
//   P2  the entry reads the number w that stayed: where src[w] is its own
//       source, w leads that source, and f != w adds itself to agg[w] (further
//       matches, largest entry number + 1) with two native shared atomics.
//       Entries that find another source write and read again under another
//       hash until none is left (a few per cent, once);
//   P3  the largest entry number of a source is its last match (matches ascend
//       on both sides): that entry decides the source with the positions it
//       holds, and if it needs verification puts (y, matches | position) into
//       its own agg slot (its source's other entries, all smaller, either read
//       another slot or cannot take it for theirs) and f into the warp's list;
//   P4  the warp's listed sources' bitmap bounds, a lane each; the survivors go
//       onto the CTA's merge list, which is worked off, a warp per source, at
//       the query's end or when it is half full.
// No slot is compared-and-swapped, probed, listed or cleared: one that is read
// was written in the same step.
template <typename S, int MODE, bool SIDED>
__device__ void claim_consumer(const JoinArgs* __restrict__ joins, const FusedArgs* __restrict__ fargs,
                               unsigned char* smem, const ClaimStep* steps, ClaimQuery* s_query, uint32_t* s_nm,
                               unsigned long long* s_cnt) {
    uint2* const agg = reinterpret_cast<uint2*>(smem + S::off_agg);
    uint32_t* const srcs = reinterpret_cast<uint32_t*>(smem + S::off_src);
    volatile uint16_t* const slot = reinterpret_cast<volatile uint16_t*>(smem + S::off_slot);
    uint32_t* const ml_s = reinterpret_cast<uint32_t*>(smem + S::off_ml);  // source, entry's y,
    uint32_t* const ml_y = ml_s + S::MC;                                   // matches | query position of
    uint32_t* const ml_c = ml_y + S::MC;                                   // the last << 16
    const uint32_t tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const uint32_t le = lanemask_lt() | (1u << lane);
    uint32_t n_cand = 0, n_ver = 0;  // counters of the current join (32 bits: flushed when large)
    uint32_t par = 0;                // the current query is s_query[par], its tokens in buffer par
    bool any_query = false;
    auto tokens_of = [&](uint32_t p) -> const uint32_t* {
        const ClaimQuery& cq = s_query[p];
        return cq.lq <= S::QC ? reinterpret_cast<uint32_t*>(smem + S::off_qtok) + p * S::QC : joins[cq.join].tok + cq.pos;
    };
    uint32_t* const bm = reinterpret_cast<uint32_t*>(smem + S::off_bm);
    auto flush_merge_counts = [&](uint32_t join) {  // thread 0, no merge running
        unsigned long long* stats = joins[join].stats;
        if (s_cnt[0]) atomicAdd(&stats[SS_INTERSECTIONS], s_cnt[0]);
        if (s_cnt[1]) atomicAdd(&stats[SS_RESULTS], s_cnt[1]);
        if (s_cnt[2]) atomicAdd(&stats[SS_MERGED], s_cnt[2]);
        s_cnt[0] = s_cnt[1] = s_cnt[2] = 0;
    };
    auto flush_counts = [&](uint32_t join) {  // warp-collective
        const unsigned long long c = warp_sum((unsigned long long)n_cand), v = warp_sum((unsigned long long)n_ver);
        if (lane == 0) {
            if (c && MODE != MODE_FILL) atomicAdd(&joins[join].stats[SS_CANDIDATES], c);
            if (v && MODE == MODE_FUSED) atomicAdd(&joins[join].stats[SS_VERIFIED], v);
        }
        n_cand = n_ver = 0;
    };
    // The listed sources' merges with the current query, a warp per source.  The lanes first fetch
    // the bounds and offsets of the warp's sources; four chunks of 32 source tokens are
    // loaded at once.
    auto merge_list = [&](uint32_t nm) {
        const ClaimQuery& cq = s_query[par];
        const JoinArgs& a = joins[cq.join];
        const FusedArgs& fa = fargs[cq.join];
        const uint32_t* qsrc = tokens_of(par);
        const uint32_t lq = cq.lq, qmode = cq.qmode;
        const uint32_t mine = wid + lane * S::NWC;
        uint4 sm0 = make_uint4(0, 0, 0, 0);
        uint32_t at0 = 0;
        if (mine < nm) {
            sm0 = __ldg(fa.smin + lq + (ml_y[mine] >> 16));
            at0 = fa.meta[ml_s[mine]].x;
        }
#pragma unroll 1
        for (uint32_t i = wid, x = 0; i < nm; i += S::NWC, x++) {
            const uint32_t s = ml_s[i], y = ml_y[i], cj = ml_c[i];
            const uint32_t im = __shfl_sync(kFull, sm0.y, x), need = __shfl_sync(kFull, sm0.z, x);
            const uint32_t* st = a.tok + __shfl_sync(kFull, at0, x);
            const uint32_t ls = y >> 16, c = cj & 0xffffu, qrest = lq - (cj >> 16) - 1, k0 = (y & 0xffffu) + 1;
            uint32_t k = k0, cnt = c;
#pragma unroll 1
            while (k < ls && cnt + min(ls - k, qrest - (cnt - c)) >= im) {
                uint32_t t[4];
#pragma unroll
                for (uint32_t u = 0; u < 4; u++) {
                    const uint32_t kk = k + 32 * u + lane;
                    t[u] = kk < ls ? __ldg(st + kk) : 0u;
                }
#pragma unroll 1
                for (uint32_t u = 0; u < 4 && k < ls; u++) {
                    const bool hit = k + lane < ls && bm_test(bm, qmode, t[0], qsrc, 0, lq);
                    cnt += __popc(__ballot_sync(kFull, hit));
                    k = min(k + 32u, ls);
                    t[0] = t[1];
                    t[1] = t[2];
                    t[2] = t[3];
                }
            }
            if (lane == 0) {
                FusedCounters ctr = {0, 0, 0, 0, 0, 0, 0};
                tally_overlap(a, ctr, cq.q, s, cnt, im, need);
                if (ctr.inter) atomicAdd(&s_cnt[0], 1ull);
                if (ctr.res) atomicAdd(&s_cnt[1], 1ull);
                atomicAdd(&s_cnt[2], (unsigned long long)(k - k0));
            }
        }
    };
#pragma unroll 1
    for (uint32_t k = 0;; k++) {
        bar_named(1, S::NT);  // step k is laid out; every consumer is done with step k - 1
        const ClaimStep& st = steps[k & 1];
        const uint32_t flags = st.flags;
        const uint32_t nm = min(*(volatile uint32_t*)s_nm, S::MC);
        const bool flush = (flags & (CS_FIRST | CS_END)) || nm > S::MC / 2;
        if (flush && nm) merge_list(nm);
        if (flags & (CS_FIRST | CS_END)) {
            const bool full = __any_sync(kFull, (n_cand | n_ver) >> 30);
            if (any_query && ((flags & CS_END) || st.join != s_query[par].join || full)) flush_counts(s_query[par].join);
            if (flags & CS_END) {
                bar_named(2, S::NTC);
                if (any_query && tid == 0) flush_merge_counts(s_query[par].join);
                break;
            }
            par ^= 1;  // (s_query[par ^ 1] stays readable until the next query)
            const JoinArgs& a = joins[st.join];
            const FusedArgs& fa = fargs[st.join];
            const uint32_t lq = st.lq, pos = st.pos;
            const uint32_t qmode = a.n_terms <= S::BW * 32 ? QM_EXACT : (lq <= kQHashMax ? QM_HASH : QM_BLOOM);
            ClaimQuery& cq = s_query[par];
            if (MODE == MODE_FUSED && tid < 4) cq.bits[tid] = tid < fa.bmw ? __ldg(fa.bmap + (uint64_t)fa.bmw * st.q + tid) : make_uint4(0, 0, 0, 0);
            if (tid == 0) {
                cq.join = st.join;
                cq.q = st.q;
                cq.lq = lq;
                cq.pos = pos;
                cq.qmode = qmode;
            }
            uint32_t* qtok = reinterpret_cast<uint32_t*>(smem + S::off_qtok) + par * S::QC;
            if (MODE == MODE_FUSED && lq <= S::QC)
                for (uint32_t j = tid; j < lq; j += S::NTC) qtok[j] = __ldg(a.tok + pos + j);
        }
        const uint32_t L = st.L, lq = st.lq, join = st.join;
        uint32_t sv[S::U], yv[S::U], jw[S::U];  // source, the entry's y, query position | leader << 16
        uint32_t mine = 0;                      // bit u: entry u takes part
        {
            const uint32_t* wfe = reinterpret_cast<const uint32_t*>(smem + S::off_wfe) + (k & 1) * S::PC;
            const uint16_t* wj = reinterpret_cast<const uint16_t*>(smem + S::off_wj) + (k & 1) * S::PC;
            const uint2* grp = reinterpret_cast<const uint2*>(smem + S::off_grp) + (k & 1) * S::JW;
            const uint2* __restrict__ ent = joins[join].ent;
#pragma unroll
            for (uint32_t u = 0; u < S::U; u++) {
                const uint32_t f = u * S::NTC + tid;
                if (f < L) {
                    const uint2 g = grp[f >> 5];
                    const uint32_t r = g.y + __popc(g.x & le) - 1u;
                    const uint2 e = __ldg(ent + (wfe[r] + f));
                    sv[u] = e.x;
                    yv[u] = e.y;
                    jw[u] = wj[r];
                    mine |= 1u << u;
                }
            }
        }
        if (SIDED || (flags & CS_UNSORTED)) {  // entries that do not take part
            const JoinArgs& a = joins[join];
            const uint32_t side_q = SIDED ? __ldg(a.side + st.q) : 0u;
#pragma unroll
            for (uint32_t u = 0; u < S::U; u++) {
                if (!(mine >> u & 1u)) continue;
                if (((flags & CS_UNSORTED) && !size_ok(a, lq, yv[u] >> 16)) || (SIDED && __ldg(a.side + sv[u]) == side_q))
                    mine &= ~(1u << u);
            }
        }
#pragma unroll
        for (uint32_t u = 0; u < S::U; u++) {
            const uint32_t f = u * S::NTC + tid;
            if (mine >> u & 1u) {
                slot[sv[u] & (S::H - 1)] = (uint16_t)f;
                srcs[f] = sv[u];
                agg[f] = make_uint2(0, 0);
            }
        }
        bar_named(2, S::NTC);
        // every consumer's merges are done: the list is empty again, the previous query's membership
        // cleared, its join's counters added when the join is done
        if (flush && tid == 0) *s_nm = 0;
        if (flags & CS_FIRST) {
            if (any_query && tid == 0 && s_query[par ^ 1].join != join) flush_merge_counts(s_query[par ^ 1].join);
            any_query = true;
            if (MODE == MODE_FUSED)
                for (uint32_t i = tid; i < S::BW / 4; i += S::NTC)
                    reinterpret_cast<uint4*>(bm)[i] = make_uint4(0, 0, 0, 0);
        }
        uint32_t pend = mine;  // bit u: entry u has no leader yet
        uint32_t mul = 0;      // 0: the low bits of the source
#pragma unroll 1
        for (;;) {
            uint32_t ws[S::U];  // source of the number that stayed
#pragma unroll
            for (uint32_t u = 0; u < S::U; u++) {
                if (u * S::NTC + wid * 32 >= L) break;
                if (pend >> u & 1u) {
                    const uint32_t w = slot[mul ? (sv[u] * mul) >> (32 - S::HLOG) : sv[u] & (S::H - 1)];
                    jw[u] = (jw[u] & 0xffffu) | w << 16;
                }
            }
#pragma unroll
            for (uint32_t u = 0; u < S::U; u++) {
                if (u * S::NTC + wid * 32 >= L) break;
                ws[u] = sv[u];
                if ((pend >> u & 1u) && jw[u] >> 16 != u * S::NTC + tid) ws[u] = srcs[jw[u] >> 16];
            }
#pragma unroll
            for (uint32_t u = 0; u < S::U; u++) {
                if (u * S::NTC + wid * 32 >= L) break;
                const uint32_t f = u * S::NTC + tid, w = jw[u] >> 16;
                if ((pend >> u & 1u) && ws[u] == sv[u]) {
                    pend &= ~(1u << u);
                    if (w != f) {
                        atomicAdd(&agg[w].x, 1u);
                        atomicMax(&agg[w].y, f + 1);
                    }
                }
            }
            if (!bar_or(2, S::NTC, pend != 0)) break;
            mul = (mul * 0x9E3779B1u + 0x7f4a7c15u) | 1u;  // another hash for the rest
#pragma unroll
            for (uint32_t u = 0; u < S::U; u++)
                if (pend >> u & 1u) slot[(sv[u] * mul) >> (32 - S::HLOG)] = (uint16_t)(u * S::NTC + tid);
            bar_named(2, S::NTC);
        }
        const FusedArgs& fa = fargs[join];
        if (MODE == MODE_FUSED && (flags & CS_FIRST)) {  // the query's membership structure, for the merges from the next step on
            const uint32_t qmode = s_query[par].qmode;
            const uint32_t* qsrc = tokens_of(par);
#pragma unroll 1
            for (uint32_t j = tid; j < lq; j += S::NTC) bm_insert(bm, qmode, qsrc[j]);
        }
        const uint4* __restrict__ smin = fa.smin + lq;
        uint16_t* const vl = reinterpret_cast<uint16_t*>(smem + S::off_vl) + wid * 32 * S::U;
#pragma unroll
        for (uint32_t u = 0; u < S::U; u++) {  // jw: query position | matches << 16 of an owner (else 0)
            if (u * S::NTC + wid * 32 >= L) break;
            const uint32_t f = u * S::NTC + tid, w = jw[u] >> 16;
            uint2 g = make_uint2(0, 0);
            if (mine >> u & 1u) g = agg[w];
            const bool own = (mine >> u & 1u) && max(w + 1, g.y) == f + 1;
            jw[u] = (jw[u] & 0xffffu) | (own ? (g.x + 1) << 16 : 0u);
        }
        uint32_t ver = 0;  // bit u: the source needs its bitmap bound checked
#pragma unroll
        for (uint32_t u = 0; u < S::U; u++) {
            if (u * S::NTC + wid * 32 >= L) break;
            const uint32_t c = jw[u] >> 16;
            if (!(mine >> u & 1u) || c == 0) continue;
            const uint2 mn = __ldg(reinterpret_cast<const uint2*>(smin + (yv[u] >> 16)));  // (cand, inter)
            const uint32_t most = c + min(lq - (jw[u] & 0xffffu), (yv[u] >> 16) - (yv[u] & 0xffffu));
            n_cand += most >= mn.x;  // filtering.cu:127-135 at the last match
            ver |= (most > mn.y ? 1u : 0u) << u;
        }
        uint32_t nv = 0;
#pragma unroll
        for (uint32_t u = 0; u < S::U; u++) {
            if (u * S::NTC + wid * 32 >= L) break;
            const uint32_t f = u * S::NTC + tid;
            const uint32_t m = __ballot_sync(kFull, ver >> u & 1u);
            if (ver >> u & 1u) {
                agg[f] = make_uint2(yv[u], jw[u] >> 16 | jw[u] << 16);
                vl[nv + __popc(m & (le >> 1))] = (uint16_t)f;
            }
            nv += __popc(m);
        }
        __syncwarp();
        if (lane == 0) n_ver += nv;
#pragma unroll 1
        for (uint32_t i0 = 0; i0 < nv; i0 += 32) {
            const uint32_t f = vl[min(i0 + lane, nv - 1)];
            const uint32_t s = srcs[f];
            const uint2 g = agg[f];  // (y, matches | query position << 16)
            if constexpr (MODE != MODE_FUSED) {
                plain_take<MODE>(joins[join], st.q, i0 + lane < nv, s, g.y);
            } else {
                const bool check = i0 + lane < nv &&
                    bitmap_keeps(s_query[par].bits, fa.bmap + (uint64_t)fa.bmw * s, fa.bmw, lq + (g.x >> 16),
                                 __ldg(&smin[g.x >> 16].y));
                const uint32_t m = __ballot_sync(kFull, check);
                if (m == 0) continue;
                uint32_t base = 0;
                if (lane == 0) base = atomicAdd(s_nm, (uint32_t)__popc(m));
                const uint32_t mi = __shfl_sync(kFull, base, 0) + __popc(m & (le >> 1));
                if (check && mi < S::MC) {
                    ml_s[mi] = s;
                    ml_y[mi] = g.x;
                    ml_c[mi] = g.y;
                }
#pragma unroll 1
                for (uint32_t over = __ballot_sync(kFull, check && mi >= S::MC); over; over &= over - 1) {
                    const uint32_t l = __ffs(over) - 1;
                    merge_now(joins[join], fa, s_query[par], __shfl_sync(kFull, s, l), __shfl_sync(kFull, g.x, l),
                              __shfl_sync(kFull, g.y, l), tokens_of(par), s_cnt);
                }
            }
        }
    }
}

template <typename S, int CTAS, int MODE, bool SIDED>
__global__ void __launch_bounds__(S::NT, CTAS) k_claim(const JoinArgs* __restrict__ joins,
                                                       const FusedArgs* __restrict__ fargs, ClaimItems items,
                                                       uint32_t* counter) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ ClaimStep s_step[2];
    __shared__ ClaimQuery s_query[2];
    __shared__ uint32_t s_nm;
    __shared__ unsigned long long s_cnt[3];  // intersections, results, merged tokens of the current join
    for (uint32_t i = threadIdx.x; i < S::BW; i += S::NT) reinterpret_cast<uint32_t*>(smem + S::off_bm)[i] = 0u;
    if (threadIdx.x < 3) s_cnt[threadIdx.x] = 0;
    if (threadIdx.x == 0) s_nm = 0;
    __syncthreads();
    if (threadIdx.x >= S::NTC)
        claim_producer<S, MODE>(joins, fargs, items, counter, smem, s_step);
    else
        claim_consumer<S, MODE, SIDED>(joins, fargs, smem, s_step, s_query, &s_nm, s_cnt);
}

// -------------------------------------------------------------------- k_tiny

constexpr uint32_t kTinyWarps = 8;

// Warp per query of at most kTinyMax window entries (a CTA per query of
// k_claim would leave most of its 256 threads without an entry), in rows of 32 in the
// lanes' registers in (probe position, source) order.  The claim of k_claim
// within the warp: entry f writes f into its source's slot, the number w that
// stays leads the source, the largest number is the last match.  CTAs take tiles of
// 8 to 32 consecutive records of a join.  Bound by the latency of a query's chain of
// loads (windows, entries, bounds, bitmaps, merges; 0.8 instructions a cycle):
// 64 registers for 4 CTAs an SM, the queries' bounds and offsets and four chunks
// of a merge's tokens fetched at once (this kernel on 500,000 reads at t = 0.8
// 1.05 -> 0.77 ms, on 48 joins of titles 0.57 -> 0.47; at 3 CTAs 0.94 and 0.55, at 5 0.81 and
// 0.61), though MODE_FUSED then spills 40 bytes and loads 68 a thread.
struct TinyShared {
    uint32_t at[kTinyMax];    // entry of number f
    uint32_t src[kTinyMax];
    uint2 agg[kTinyMax];      // (further matches, largest number + 1); of a verified source (y, matches | position << 16)
    uint16_t j[kTinyMax];     // its probe position
    uint16_t slot[4 * kTinyMax];
    uint16_t vl[kTinyMax];    // entries whose source needs verification
};

template <int MODE, bool SIDED>
__global__ void __launch_bounds__(kTinyWarps * 32, 4) k_tiny(const JoinArgs* __restrict__ joins,
                                                          const FusedArgs* __restrict__ fargs, TileMap m) {
    __shared__ TinyShared s_all[kTinyWarps];
    const uint32_t lane = lane_id(), wid = threadIdx.x >> 5, lt = lanemask_lt();
    TinyShared& sh = s_all[wid];
    constexpr uint32_t R = kTinyMax / 32;
    constexpr int HB = 9;
    static_assert((1 << HB) == 4 * kTinyMax, "slot hash bits");
    FusedCounters ctr = {0, 0, 0, 0, 0, 0, 0};
    uint32_t cur = 0xffffffffu;
    for (uint32_t b = blockIdx.x; b < m.ntiles; b += gridDim.x) {  // tiles of at most 32 records
        const TileRange t = tile_range(m, b);
        const uint32_t r0 = t.r0;
        if (r0 >= t.r1) continue;
        if (t.j != cur) {
            if (cur != 0xffffffffu) flush_fused_counters(joins[cur], ctr);
            cur = t.j;
        }
        const JoinArgs& a = joins[cur];
        const FusedArgs& fa = fargs[cur];
        const uint32_t bits = *a.status;
        if (bits & ST_SKIP_ALL) continue;
        // warp w takes records r0 + w, r0 + w + 8, ...
        const uint32_t rec = r0 + wid + lane * kTinyWarps;
        const uint4 mt = lane < 32 / kTinyWarps && rec < t.r1 ? fa.meta[rec] : make_uint4(0, 0, QC_NONE << 16, 0);
        uint32_t qp0 = 0, po0 = 0;  // of each lane's query: their loads are in flight together
        if ((mt.z >> 16) == QC_TINY) {
            qp0 = a.probe[mt.y];
            po0 = fa.poff[rec];
        }
#pragma unroll 1
        for (uint32_t todo = __ballot_sync(kFull, (mt.z >> 16) == QC_TINY); todo; todo &= todo - 1) {
            const uint32_t ln = __ffs(todo) - 1, q = r0 + wid + ln * kTinyWarps;
            const uint32_t lq = __shfl_sync(kFull, mt.y, ln), W = __shfl_sync(kFull, mt.w, ln);
            const uint32_t* __restrict__ qt = a.tok + __shfl_sync(kFull, mt.x, ln);
            const uint32_t qp = __shfl_sync(kFull, qp0, ln), po = __shfl_sync(kFull, po0, ln);
            for (uint32_t j = lane; j < qp; j += 32) {
                const uint2 w = __ldg(fa.win + po + j);
                uint32_t p = __ldg(fa.wpre + po + j);
                for (uint32_t x = w.x; x < w.y; x++, p++) {
                    sh.at[p] = x;
                    sh.j[p] = (uint16_t)j;
                }
            }
            __syncwarp();
            const uint32_t side_q = SIDED ? __ldg(a.side + q) : 0u;
            uint32_t sv[R], yv[R], jw[R];  // source, the entry's y, query position | leader << 16
            uint32_t pend = 0;
#pragma unroll
            for (uint32_t r = 0; r < R; r++) {
                const uint32_t f = r * 32 + lane;
                if (f >= W) continue;
                const uint2 e = __ldg(a.ent + sh.at[f]);
                sv[r] = e.x;
                yv[r] = e.y;
                jw[r] = sh.j[f];
                pend |= 1u << r;
            }
#pragma unroll
            for (uint32_t r = 0; r < R; r++) {
                if (!(pend >> r & 1u)) continue;
                if (((bits & ST_UNSORTED) && !size_ok(a, lq, yv[r] >> 16)) || (SIDED && __ldg(a.side + sv[r]) == side_q)) {
                    pend &= ~(1u << r);
                    continue;
                }
                const uint32_t f = r * 32 + lane;
                sh.slot[sv[r] & ((1u << HB) - 1)] = (uint16_t)f;
                sh.src[f] = sv[r];
                sh.agg[f] = make_uint2(0, 0);
            }
            const uint32_t mine = pend;
            uint32_t mul = 0;  // 0: the low bits of the source
#pragma unroll 1
            for (;;) {
                __syncwarp();
#pragma unroll
                for (uint32_t r = 0; r < R; r++) {
                    if (!(pend >> r & 1u)) continue;
                    const uint32_t f = r * 32 + lane;
                    const uint32_t w = sh.slot[mul ? (sv[r] * mul) >> (32 - HB) : sv[r] & ((1u << HB) - 1)];
                    if (w != f) {
                        if (sh.src[w] != sv[r]) continue;
                        atomicAdd(&sh.agg[w].x, 1u);
                        atomicMax(&sh.agg[w].y, f + 1);
                    }
                    jw[r] |= w << 16;
                    pend &= ~(1u << r);
                }
                if (!__any_sync(kFull, pend)) break;
                mul = (mul * 0x9E3779B1u + 0x7f4a7c15u) | 1u;
#pragma unroll
                for (uint32_t r = 0; r < R; r++)
                    if (pend >> r & 1u) sh.slot[(sv[r] * mul) >> (32 - HB)] = (uint16_t)(r * 32 + lane);
            }
            __syncwarp();
            const uint4* __restrict__ smin = fa.smin + lq;
            uint32_t nv = 0;
#pragma unroll
            for (uint32_t r = 0; r < R; r++) {
                if (r * 32 >= W) break;
                const uint32_t f = r * 32 + lane;
                bool ver = false;
                if (mine >> r & 1u) {
                    const uint32_t w = jw[r] >> 16;
                    const uint2 g = sh.agg[w];
                    if (max(w + 1, g.y) == f + 1) {
                        const uint2 mn = __ldg(reinterpret_cast<const uint2*>(smin + (yv[r] >> 16)));
                        const uint32_t j = jw[r] & 0xffffu, c = g.x + 1;
                        const uint32_t most = c + min(lq - j, (yv[r] >> 16) - (yv[r] & 0xffffu));
                        ctr.cand += most >= mn.x;  // filtering.cu:127-135 at the last match
                        ver = most > mn.y;
                        if (ver) sh.agg[f] = make_uint2(yv[r], c | (j << 16));
                    }
                }
                const uint32_t mm = __ballot_sync(kFull, ver);
                if (ver) sh.vl[nv + __popc(mm & lt)] = (uint16_t)f;
                nv += __popc(mm);
            }
            __syncwarp();
#pragma unroll 1
            for (uint32_t i0 = 0; i0 < nv; i0 += 32) {
                if constexpr (MODE != MODE_FUSED) {
                    const uint32_t f = sh.vl[min(i0 + lane, nv - 1)];
                    plain_take<MODE>(a, q, i0 + lane < nv, sh.src[f], sh.agg[f].y);
                } else {
                    bool check = false;
                    uint32_t s0 = 0, y0 = 0, cj0 = 0, im0 = 0, at0 = 0;
                    if (i0 + lane < nv) {
                        const uint32_t f = sh.vl[i0 + lane];
                        const uint2 g = sh.agg[f];
                        s0 = sh.src[f];
                        y0 = g.x;
                        cj0 = g.y;
                        im0 = __ldg(&smin[y0 >> 16].y);
                        at0 = fa.meta[s0].x;
                        check = bitmap_keeps(fa.bmap + (uint64_t)fa.bmw * q, fa.bmap + (uint64_t)fa.bmw * s0, fa.bmw,
                                             lq + (y0 >> 16), im0);
                    }
#pragma unroll 1
                    for (uint32_t mm = __ballot_sync(kFull, check); mm; mm &= mm - 1) {
                        // merge, 32 source tokens per step, with the early exit of checking.cu:150-157
                        const uint32_t l = __ffs(mm) - 1;
                        const uint32_t s = __shfl_sync(kFull, s0, l), y = __shfl_sync(kFull, y0, l);
                        const uint32_t cj = __shfl_sync(kFull, cj0, l), im = __shfl_sync(kFull, im0, l);
                        const uint32_t ls = y >> 16, c = cj & 0xffffu, j = cj >> 16, qrest = lq - j - 1, k0 = (y & 0xffffu) + 1;
                        const uint32_t* st = a.tok + __shfl_sync(kFull, at0, l);
                        uint32_t k = k0, cnt = c;
#pragma unroll 1
                        while (k < ls && cnt + min(ls - k, qrest - (cnt - c)) >= im) {
                            uint32_t tk[4];  // four chunks of 32 source tokens in flight
#pragma unroll
                            for (uint32_t u = 0; u < 4; u++) tk[u] = k + 32 * u + lane < ls ? __ldg(st + k + 32 * u + lane) : 0u;
#pragma unroll 1
                            for (uint32_t u = 0; u < 4 && k < ls && cnt + min(ls - k, qrest - (cnt - c)) >= im; u++) {
                                const bool hit = k + lane < ls && contains_gen(qt, j + 1, lq, tk[0]);
                                cnt += __popc(__ballot_sync(kFull, hit));
                                k = min(k + 32u, ls);
                                tk[0] = tk[1];
                                tk[1] = tk[2];
                                tk[2] = tk[3];
                            }
                        }
                        if (lane == 0) {
                            ctr.merged += k - k0;
                            tally_overlap(a, ctr, q, s, cnt, im, __ldg(&smin[ls].z));
                        }
                    }
                }
            }
            if (MODE == MODE_FILL) ctr.cand = 0;
            if (lane == 0 && MODE != MODE_FILL) {
                ctr.window += W;
                if (MODE == MODE_FUSED) {
                    ctr.verified += nv;
                    ctr.qtok += lq;
                }
            }
            __syncwarp();
        }
    }
    if (cur != 0xffffffffu) flush_fused_counters(joins[cur], ctr);
}

}  // namespace fgss
