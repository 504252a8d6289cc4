// Tail of the layer-step kernel: exact top-k from the votes and, where the shape allows, the sparse
// attention itself, inside the persistent selection kernel (included by fused.cu).
//
//   phase 3  classify   every CTA reads the request's vote histogram, finds the bin of the k-th vote and
//                       sorts its own candidates into sure winners (above the bin), members of the bin and
//                       losers; it publishes ONE record per (request, CTA): the number of sure winners and
//                       the bin's members (inline when they are few, in a global list otherwise).  When the
//                       CTA's possible winners are few, their key and value rows are requested now, before
//                       the selection is final, so that they are in shared memory when the ranks are known.
//   phase 4  resolve    after a grid barrier every CTA reads the records of the CTAs that share the request:
//                       the members of the bin are ranked on (low vote bits, inverted index), which settles
//                       the set; the sure-winner counts of the CTAs in front give the list position of the
//                       CTA's first winner.  Positions and pool rows of the winners are written out.
//   phase 5  attend     every CTA attends to ITS OWN winners plus its share of the rows that never depended
//                       on votes (initial and local windows; whole lists of requests that reuse a cached set
//                       or attend to everything): rows of 16 per warp and KV head on mma.sync, the query at
//                       position count-1, the row at its list position.  One partial (max, sum, output) per
//                       (request, CTA).
//   phase 6  merge      after a last grid barrier the partials of a (request, head, quarter of the head
//                       dimension) are merged by one CTA each and the output row is written.
//
// Replaces, from patcher/token_retrieval.py: topk + sort (:371-372), the "+ n_init" shift (:433),
// init || top-k || local (:436-446), the slot gather (:448), the cache write (:415) and the paged decode
// attention call (:815-825, planned at :802-813).
#pragma once

namespace ts {

constexpr int kRecInline = 12;               // members of the threshold bin a record holds itself
constexpr unsigned kRecOverflow = 0x80000000u;
constexpr int kAttnRowsMax = 64;             // rows one attention round stages in shared memory
constexpr int kMaxGrid = 256;
constexpr int kDirectRankMax = 128;          // members ranked by direct comparison up to this many

struct alignas(128) SelRecord {
    unsigned sure;                           // winners above the threshold bin in this CTA's range
    unsigned n_members;                      // members of the bin in the range (| kRecOverflow: in the global list)
    uint2 members[15];                       // (candidate index, vote bits); the first kRecInline are used
};
static_assert(sizeof(SelRecord) == 128, "one record is one 128-byte line");

// Scratch of phases 3-6; overlays FusedShared::idx, which only the scoring phase and the statistics merge use.
struct TailScratch {
    int row_slot[kAttnRowsMax];              // pool row of a staged attention row
    int row_rank[kAttnRowsMax];              // its list position (rotation angle); < 0: not attended
    int row_t[kAttnRowsMax];                 // candidate index of a possible winner staged early
    unsigned row_v[kAttnRowsMax];            // its vote bits
    float inv_freq[64];                      // rotation frequencies of the attention positions
    unsigned long long kv_bar;               // mbarrier of the staged K/V rows
    unsigned long long key_at;               // key of the k1-th member (direct ranking)
    int fast, fast_static, fast_pot, fast_b, fast_share;   // (fast_share: this CTA's place in the request's share)
    unsigned n_inl, n_ovf, sure_before, pad;
};
static_assert(sizeof(TailScratch) <= 2 * kIdxBlock * sizeof(int), "tail scratch must fit the index staging area");

__device__ __forceinline__ TailScratch& tail_scratch(FusedShared& sh) { return *reinterpret_cast<TailScratch*>(&sh.idx[0][0]); }

// Rows per attention round and warps that work on them, per KV heads on this rank.
template <int HKV> struct AttnGeom {
    static constexpr int kRows = HKV >= 4 ? 32 : 64;
    static constexpr int kBlocks = kRows / 16;
    static constexpr int kWarpsBusy = kBlocks * HKV;                 // 16, 8, 8, 4
    static constexpr int kRowB = HKV * 256, kRowS = kRowB + 16;      // row bytes in the pool / padded in shared memory
    static constexpr int kKvBytes = 2 * kRows * kRowS;
    static constexpr int kCsOff = (kKvBytes + 127) / 128 * 128;
    static constexpr int kCsBytes = kRows / 8 * 4096;
    static constexpr int kPartOff = kCsOff + kCsBytes;
    static_assert(kWarpsBusy <= kFusedThreads / 32, "more warps than the CTA has");
};
__host__ __device__ constexpr int attn_part_bytes(int warps_busy, int group) { return warps_busy * group * (128 + 2) * 4; }
// Whether an attention round's partial outputs end inside the kernel's dynamic shared memory.  Not so for seven and eight
// query heads on each of eight KV heads (206720 and 215040 bytes of 198656).
template <int HKV>
constexpr bool attn_fits(int group) {
    return AttnGeom<HKV>::kPartOff + attn_part_bytes(AttnGeom<HKV>::kWarpsBusy, group) <= kFusedDynSmem;
}
static_assert(attn_fits<1>(8) && attn_fits<2>(8) && attn_fits<4>(8) && attn_fits<8>(6), "the other shapes fit");

// First and last CTA that own candidates of request b (nc[b] > 0).
__device__ __forceinline__ void owner_range(const LayerParams& p, const FusedShared& sh, int b, int& c0, int& c1) {
    c0 = tile_owner(sh, (unsigned)sh.tile_off[b]);
    c1 = tile_owner(sh, (unsigned)sh.tile_off[b + 1] - 1u);
}

// Rows of request b's list that do not depend on this step's votes, and how many CTAs share them.
//   RECOMPUTE: the initial and local windows, shared by the CTAs that own the request's candidates;
//   REUSE / DENSE: the whole list, shared by `np` CTAs starting at a request-dependent offset.
struct StaticShare {
    int total;       // rows that do not depend on votes
    int np;          // CTAs (= partials) of the request
    int first;       // first CTA of the share (modulo the grid)
    int chunk;       // rows per CTA
};
__device__ __forceinline__ StaticShare static_share(const LayerParams& p, const FusedShared& sh, int b, int rows_per_round) {
    StaticShare s;
    const int n = sh.plan.n[b], flag = sh.plan.flag[b];
    const int req = p.req_pool_indices[b];
    if (n < 1 || n > p.max_ctx || req < 0 || req >= p.max_reqs) { s.total = 0; s.np = 0; s.first = 0; s.chunk = 1; return s; }
    if (flag == TS_FLAG_RECOMPUTE) {
        int c0, c1;
        owner_range(p, sh, b, c0, c1);
        s.total = p.n_init + p.n_local;
        s.np = c1 - c0 + 1;
        s.first = c0;
    } else {
        s.total = flag == TS_FLAG_DENSE ? n : p.n_sel;
        s.np = min(p.grid, (s.total + rows_per_round - 1) / rows_per_round);
        s.first = (int)(((long long)b * 37) % p.grid);
    }
    s.chunk = max(1, (s.total + s.np - 1) / max(s.np, 1));
    return s;
}
// This CTA's place in the share (-1: not part of it).
__device__ __forceinline__ int share_index(const LayerParams& p, const StaticShare& s) {
    if (s.np <= 0) return -1;
    int i = (int)blockIdx.x - s.first;
    if (i < 0) i += p.grid;
    return i < s.np ? i : -1;
}
// List index, logical position of static row `srow` of request b.
__device__ __forceinline__ void static_row(const LayerParams& p, const FusedShared& sh, int b, int srow, int& list_idx, int& pos) {
    const int n = sh.plan.n[b], flag = sh.plan.flag[b];
    if (flag == TS_FLAG_DENSE) { list_idx = srow; pos = srow; return; }
    if (flag == TS_FLAG_RECOMPUTE) list_idx = srow < p.n_init ? srow : srow + p.top_k;
    else list_idx = srow;
    if (list_idx < p.n_init) pos = list_idx;
    else if (list_idx < p.n_init + p.top_k)
        pos = p.pos_cache[((size_t)sh.plan.req[b] * p.n_layers + p.layer) * p.top_k + (list_idx - p.n_init)];
    else pos = n - p.n_local + (list_idx - p.n_init - p.top_k);
}

// Called by all threads before the first use of the tail's scratch.
__device__ __forceinline__ void tail_init(const LayerParams& p, FusedShared& sh) {
    TailScratch& ts = tail_scratch(sh);
    __syncthreads();                                   // the area's previous users are done
    if (threadIdx.x >= 64 && threadIdx.x < 128 && p.attn_inline) ts.inv_freq[threadIdx.x - 64] = p.attn_inv_freq[threadIdx.x - 64];
    if (threadIdx.x == 0) {
        ts.fast = 0; ts.fast_static = 0; ts.fast_pot = 0; ts.fast_b = -1; ts.pad = 0u;
        ts.n_inl = 0u; ts.sure_before = 0u;
        mbar_init(smem_u32(&ts.kv_bar), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
}

// ------------------------------------------------------------------------------------------
// phase 3
// ------------------------------------------------------------------------------------------
// A warp owns the candidates [lo, hi) of a segment, a multiple of 128 for all but the last; lane i holds the candidates
// 4i .. 4i+3 of a group of 128, read with one 16-byte load.  Order inside the warp: lane, then element.
struct WarpRange { int lo, hi; };
__device__ __forceinline__ WarpRange warp_range(const Seg& sg) {
    const int c = (sg.t1 - sg.t0 + 4 * kFusedThreads - 1) / (4 * kFusedThreads) * 128;
    WarpRange r;
    r.lo = min(sg.t1, sg.t0 + (int)(threadIdx.x >> 5) * c);
    r.hi = min(sg.t1, r.lo + c);
    return r;
}
constexpr int kVoteLoads = 4;            // groups of 128 candidates a warp requests together
// Calls f(t, votes of candidates t .. t+3, group base) for every group of the warp's range, in order (all lanes; the
// candidates of a lane at or beyond r.hi are not the warp's).  From shared memory when the CTA's votes were kept there.
template <typename F>
__device__ __forceinline__ void for_own_votes(const FusedShared& sh, const float* votes_s, const float* votes_g, int s,
                                              const WarpRange& r, F&& f) {
    const int lane4 = 4 * (threadIdx.x & 31);
    const float* vs = votes_s + sh.seg_off[s] - sh.seg[s].t0;
    if (sh.own_in_smem) {
#pragma unroll 1
        for (int tb = r.lo; tb < r.hi; tb += 128) {
            const int t = tb + lane4;
            f(t, t < r.hi ? *reinterpret_cast<const float4*>(vs + t) : make_float4(0.f, 0.f, 0.f, 0.f));
        }
        return;
    }
    // (a caller's tensor-parallel vote buffer may start anywhere)
    const bool wide = (reinterpret_cast<uintptr_t>(votes_g) & 15) == 0;
#pragma unroll 1
    for (int tb = r.lo; tb < r.hi; tb += 128 * kVoteLoads) {
        float4 v[kVoteLoads];
#pragma unroll
        for (int u = 0; u < kVoteLoads; ++u) {
            const int t = tb + 128 * u + lane4;
            v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (t < r.hi) {
                if (wide) v[u] = __ldcg(reinterpret_cast<const float4*>(votes_g + t));
                else v[u] = make_float4(__ldcg(votes_g + t), __ldcg(votes_g + t + 1), __ldcg(votes_g + t + 2), __ldcg(votes_g + t + 3));
            }
        }
#pragma unroll
        for (int u = 0; u < kVoteLoads; ++u)
            if (tb + 128 * u < r.hi) f(tb + 128 * u + lane4, v[u]);
    }
}
// Which of the four candidates of every lane satisfy a predicate, and how many of those the warp has in front of each.
struct Quad {
    unsigned bal[4];
    __device__ __forceinline__ unsigned total() const { return __popc(bal[0]) + __popc(bal[1]) + __popc(bal[2]) + __popc(bal[3]); }
    __device__ __forceinline__ unsigned before_lane() const {
        const unsigned lt = (1u << (threadIdx.x & 31)) - 1u;
        return __popc(bal[0] & lt) + __popc(bal[1] & lt) + __popc(bal[2] & lt) + __popc(bal[3] & lt);
    }
    __device__ __forceinline__ bool has(int i) const { return (bal[i] >> (threadIdx.x & 31)) & 1u; }
};
template <typename P>
__device__ __forceinline__ Quad quad_of(const WarpRange& r, int t, const float4& v, P&& pred) {
    const float x[4] = {v.x, v.y, v.z, v.w};
    Quad q;
#pragma unroll
    for (int i = 0; i < 4; ++i) q.bal[i] = __ballot_sync(0xffffffffu, t + i < r.hi && pred(t + i, x[i]));
    return q;
}

constexpr int kWarpMembers = 64;         // members of the threshold bin a warp keeps before they are written out
static_assert(16 * kWarpMembers * sizeof(uint2) <= kHistBins * sizeof(unsigned), "the warps' members fit the histogram's place");

// This CTA's share of the first segment's window rows, which can be staged together with its possible winners: their
// number, and list index and pool row of the one this thread stages.  Looked up while the CTA waits at the barrier that
// publishes the histogram.
struct StaticRows { int cnt, slot, list, share; };
template <int HKV>
__device__ __forceinline__ StaticRows look_up_static_rows(const LayerParams& p, FusedShared& sh) {
    using AG = AttnGeom<HKV>;
    const int tid = threadIdx.x;
    StaticRows st{0, 0, -1, -1};
    if (sh.nseg > 0) {
        const int b = sh.seg[0].b;
        const StaticShare ss = static_share(p, sh, b, AG::kRows);
        st.share = share_index(p, ss);
        if (st.share >= 0) {
            const int s0 = st.share * ss.chunk, s1 = min(ss.total, s0 + ss.chunk);
            st.cnt = max(0, s1 - s0);
            if (tid < st.cnt && st.cnt <= AG::kRows) {
                int pos;
                static_row(p, sh, b, s0 + tid, st.list, pos);
                st.slot = checked_slot(p, p.rtt + (long long)sh.plan.req[b] * p.rtt_stride, pos);
            }
        }
    }
    return st;
}

template <int HKV, bool ATTN>
__device__ __forceinline__ void classify_phase(const LayerParams& p, FusedShared& sh, unsigned char* dyn, const StaticRows& st) {
    constexpr bool attn = ATTN;
    using AG = AttnGeom<(HKV > 0 ? HKV : 1)>;
    const int tid = threadIdx.x;
    TailScratch& ts = tail_scratch(sh);
    const float* votes_s = own_votes(dyn);
    const int* slot_s = own_slots(dyn);
    const int st_cnt = st.cnt;
    fstamp(p, 4);
#pragma unroll 1
    for (int s = 0; s < sh.nseg; ++s) {
        const Seg sg = sh.seg[s];
        const float* votes_g = p.votes_sel + sh.plan.off[sg.b];
        const WarpRange wr = warp_range(sg);
        const int warp = tid >> 5, lane = tid & 31;
        // the bin of the k-th vote, from the request's histogram
        fstamp(p, 5);
        find_threshold<true>(sh, p.hist + (size_t)sg.b * kHistBins, (unsigned)p.top_k);
        fstamp(p, 6);
        const unsigned b1 = (unsigned)sh.res_bin;
        if (tid == 0) { sh.seg_b1[s] = sh.res_bin; sh.seg_above[s] = sh.res_above; sh.seg_cnt[s] = sh.res_cnt; }
        // pass 1: count the sure winners, keep the members of the bin
        uint2* mine = reinterpret_cast<uint2*>(sh.hist) + warp * kWarpMembers;
        unsigned sure = 0, eq = 0;
        for_own_votes(sh, votes_s, votes_g, s, wr, [&](int t, const float4& v) {
            const float x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const unsigned bin = vote_bin(x[i]);
                const bool in = t + i < wr.hi;
                sure += __popc(__ballot_sync(0xffffffffu, in && bin > b1));
                const unsigned m = __ballot_sync(0xffffffffu, in && bin == b1);
                const unsigned at = eq + __popc(m & ((1u << lane) - 1u));
                if (in && bin == b1 && at < (unsigned)kWarpMembers) mine[at] = make_uint2((unsigned)(t + i), __float_as_uint(x[i]));
                eq += __popc(m);
            }
        });
        unsigned sure_before, sure_tot, eq_before, eq_tot;
        if (lane == 0) sh.warp_sum2[warp] = eq;
        sum_over_warps(sure, sh.warp_sum, sure_before, sure_tot);
        {
            const unsigned x = lane < kWarps ? sh.warp_sum2[lane] : 0u;
            eq_tot = __reduce_add_sync(0xffffffffu, x);
            eq_before = __reduce_add_sync(0xffffffffu, lane < warp ? x : 0u);
        }
        fstamp(p, 7);
        const bool overflow = eq_tot > (unsigned)kRecInline;
        SelRecord* rec = p.records + (size_t)sg.b * p.grid + blockIdx.x;
        if (tid == 0) {
            rec->sure = sure_tot;
            rec->n_members = overflow ? (kRecOverflow | eq_tot) : eq_tot;
        }
        const bool fast = attn && s == 0 && sh.own_in_smem && st_cnt <= AG::kRows &&
                          (unsigned)st_cnt + sure_tot + eq_tot <= (unsigned)AG::kRows;
        uint2* dst = rec->members;
        if (overflow) {                                                          // uniform in the CTA
            if (tid == 0) sh.tmp_u[2] = atomicAdd(p.cand_count + sg.b, eq_tot);
            __syncthreads();
            dst = p.cand + sh.plan.off[sg.b] + sh.tmp_u[2];
        }
        // the members go into the record (or the list), in any order
        if (eq <= (unsigned)kWarpMembers) {
            __syncwarp();
#pragma unroll 1
            for (unsigned i = lane; i < eq; i += 32) dst[eq_before + i] = mine[i];
        } else {
            unsigned at = eq_before;
            for_own_votes(sh, votes_s, votes_g, s, wr, [&](int t, const float4& v) {
                const Quad q = quad_of(wr, t, v, [&](int, float x) { return vote_bin(x) == b1; });
                unsigned k = at + q.before_lane();
                const float x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (q.has(i)) dst[k++] = make_uint2((unsigned)(t + i), __float_as_uint(x[i]));
                at += q.total();
            });
        }
        // possible winners are staged in position order
        if (fast && sure + eq > 0u) {
            unsigned at = (unsigned)st_cnt + sure_before + eq_before;
            for_own_votes(sh, votes_s, votes_g, s, wr, [&](int t, const float4& v) {
                const Quad q = quad_of(wr, t, v, [&](int, float x) { return vote_bin(x) >= b1; });
                unsigned r = at + q.before_lane();
                const float x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if (q.has(i)) {
                        ts.row_t[r] = t + i;
                        ts.row_v[r] = __float_as_uint(x[i]);
                        ts.row_slot[r] = slot_s[sh.seg_off[s] + (t + i - sg.t0)];
                        ts.row_rank[r] = -2;
                        ++r;
                    }
                }
                at += q.total();
            });
        }
        if (fast) {
            if (tid < st_cnt) { ts.row_slot[tid] = st.slot; ts.row_rank[tid] = st.list; }
            if (tid == 0) { ts.fast = 1; ts.fast_static = st_cnt; ts.fast_pot = (int)(sure_tot + eq_tot); ts.fast_b = sg.b; ts.fast_share = st.share; }
        }
        __syncthreads();
        fstamp(p, 8);
    }
    fstamp(p, 9);
}

// Requests the rows classify_phase staged.  Called after the CTA has ARRIVED at the grid barrier that follows
// the classification (the copy engine takes ~35 ns per row copy to issue; the other CTAs need not wait for that)
// and before it waits there: the rows land during the wait.
template <int HKV>
__device__ __forceinline__ void issue_staged_rows(const LayerParams& p, FusedShared& sh, unsigned char* dyn) {
    using AG = AttnGeom<HKV>;
    const int tid = threadIdx.x;
    TailScratch& ts = tail_scratch(sh);
    if (ts.fast) {
        const int rows = ts.fast_static + ts.fast_pot;
        const uint32_t kbase = smem_u32(dyn), vbase = kbase + AG::kRows * AG::kRowS;
        const uint32_t bar = smem_u32(&ts.kv_bar);
        asm volatile("fence.proxy.async;" ::: "memory");
        if (tid == 0) mbar_expect_tx(bar, (uint32_t)rows * 2u * AG::kRowB);
        if (tid < rows) {
            const int slot = ts.row_slot[tid];
            bulk_g2s(kbase + tid * AG::kRowS, reinterpret_cast<const unsigned char*>(p.k_pool) + (size_t)slot * AG::kRowB, AG::kRowB, bar);
            bulk_g2s(vbase + tid * AG::kRowS, reinterpret_cast<const unsigned char*>(p.v_pool) + (size_t)slot * AG::kRowB, AG::kRowB, bar);
        }
    }
}

template <int HKV> __device__ __forceinline__ void attend_prepare(const LayerParams& p, FusedShared& sh, unsigned char* dyn, int b,
                                                                  int rows, int cs_rows, bool query);

// Place of the attention's query when it is rotated during the scoring phase, by threads that would idle: between the
// scoring ring and the own-candidate copies (0: no room, or a batch, whose CTAs may attend to several requests).  It
// stays valid up to the attention of the staged rows, whose partial outputs overwrite it once it has been read.  (Rotated
// by all threads after the classification, it held the CTA up for 2 us beyond the barrier: with the vectorised scoring
// fragments, one request of 8192 tokens 45.0 -> 41.0 us a layer step, of 131072 88.7 -> 85.5 us.)
constexpr int kQStride = 136;            // floats per head of the staged rotated query (8 floats of padding: bank spread)
__device__ __forceinline__ int early_query_offset(const LayerParams& p, int ring_bytes) {
    return p.batch == 1 && ring_bytes + p.hq * kQStride * 4 <= kFusedDynSmem - 2 * kOwnCap * 4 ? ring_bytes : 0;
}
template <int HKV>
__device__ __forceinline__ bool query_is_early(const LayerParams& p, const FusedShared& sh) {
    return early_query_offset(p, kScoreStages * ScoreGeom<HKV>::kStageBytes) != 0 && sh.tile_off[p.batch] != 0;
}

// Where the threshold bin's members are staged when the attention's inputs are prepared early: behind the query
// and the partial outputs, running into the shared-memory copies of the CTA's own votes and pool rows (no longer
// needed once the possible winners are staged).
template <int HKV>
__device__ __forceinline__ int early_cand_offset(const LayerParams& p) {
    using AG = AttnGeom<HKV>;
    const int q_off = early_query_offset(p, kScoreStages * ScoreGeom<HKV>::kStageBytes);
    const int q_end = q_off ? q_off + p.hq * kQStride * 4 : 0;
    return (max(AG::kPartOff + attn_part_bytes(AG::kWarpsBusy, p.group), q_end) + 15) & ~15;
}

// While the CTA waits at the grid barrier after the classification: everything the attention over the staged
// rows needs except the winners' final list positions (rotated query, zeros in unused rows, rotation rows of the
// window rows).  Only when the members of all records are sure to fit their alternative staging place.
template <int HKV>
__device__ __forceinline__ void early_prepare(const LayerParams& p, FusedShared& sh, unsigned char* dyn) {
    TailScratch& ts = tail_scratch(sh);
    if (ts.fast == 0 || sh.nseg != 1) return;     // (a second segment would still read the own-vote copies)
    int c0, c1;
    owner_range(p, sh, ts.fast_b, c0, c1);
    const int room = (kFusedDynSmem - early_cand_offset<HKV>(p)) / 8;
    if ((c1 - c0 + 1) * kRecInline > room) return;
    attend_prepare<HKV>(p, sh, dyn, ts.fast_b, ts.fast_static + ts.fast_pot, ts.fast_static, !query_is_early<HKV>(p, sh));
    if (threadIdx.x == 0) ts.pad = 1u;
}

// ------------------------------------------------------------------------------------------
// phase 4
// ------------------------------------------------------------------------------------------
struct Resolved {
    unsigned long long prefix, mask;     // a member is selected iff (key & mask) >= prefix
    unsigned before;                     // winners of the request in front of this CTA's range
    unsigned b1;
};

// Gathers the records of the CTAs that share request sg.b, settles which members of the threshold bin are
// selected and counts the winners in front of this CTA's candidates.  cand_s: staging for the members.
__device__ __forceinline__ Resolved resolve_segment(const LayerParams& p, FusedShared& sh, int s, uint2* cand_s, unsigned cand_cap) {
    const int tid = threadIdx.x;
    TailScratch& ts = tail_scratch(sh);
    const Seg sg = sh.seg[s];
    int c0, c1;
    owner_range(p, sh, sg.b, c0, c1);
    const int nown = c1 - c0 + 1;
    const SelRecord* recs = p.records + (size_t)sg.b * p.grid + c0;
    fstamp(p, 10);
    // One round trip for whole records (sixteen threads each: header, inline members) and the overflow list's length.  The
    // order of the members is free; a warp reserves the places of its ten records' members together.
    const int lane = tid & 31, k16 = tid & 15;
    unsigned ovf = 0;
    if (tid == kFusedThreads - 1) ovf = __ldcg(p.cand_count + sg.b);
    constexpr int kRecAhead = 5;                           // 160 records a pass: one pass for grids up to 160 CTAs
    unsigned sure_front = 0;
#pragma unroll 1
    for (int base = 0; base < nown * 16; base += kFusedThreads * kRecAhead) {
        uint2 v[kRecAhead];
#pragma unroll
        for (int u = 0; u < kRecAhead; ++u) {
            const int rec = (base + kFusedThreads * u + tid) >> 4;
            v[u] = make_uint2(0u, 0u);
            if (rec < nown && k16 <= kRecInline) v[u] = __ldcg(reinterpret_cast<const uint2*>(recs + rec) + k16);
        }
        unsigned inl[kRecAhead], sum = 0;
#pragma unroll
        for (int u = 0; u < kRecAhead; ++u) {
            const unsigned nm = __shfl_sync(0xffffffffu, v[u].y, lane & 16);
            inl[u] = (nm & kRecOverflow) ? 0u : nm;
            const int rec = (base + kFusedThreads * u + tid) >> 4;
            if (k16 == 0 && c0 + rec < (int)blockIdx.x) sure_front += v[u].x;
            sum += inl[u] + __shfl_xor_sync(0xffffffffu, inl[u], 16);
        }
        unsigned at = 0;
        if (lane == 0 && sum) at = atomicAdd(&ts.n_inl, sum);
        at = __shfl_sync(0xffffffffu, at, 0);
#pragma unroll
        for (int u = 0; u < kRecAhead; ++u) {
            const unsigned other = __shfl_xor_sync(0xffffffffu, inl[u], 16);
            if (k16 >= 1 && (unsigned)(k16 - 1) < inl[u]) cand_s[at + (lane & 16 ? other : 0u) + k16 - 1] = v[u];
            at += inl[u] + other;
        }
    }
    sure_front = __reduce_add_sync(0xffffffffu, sure_front);
    if (lane == 0 && sure_front) atomicAdd(&ts.sure_before, sure_front);
    if (tid == kFusedThreads - 1) ts.n_ovf = ovf;
    __syncthreads();
    fstamp(p, 12);
    const unsigned n_inl = ts.n_inl, n_ovf = ts.n_ovf, n_c = n_inl + n_ovf;
    // the list's members when there is room (the inline ones always fit)
    const uint2* cand_g = p.cand + sh.plan.off[sg.b];
    const bool staged = n_c <= cand_cap;
    if (staged)
#pragma unroll 1
        for (unsigned i = tid; i < n_ovf; i += kFusedThreads) cand_s[n_inl + i] = __ldcg(cand_g + i);
    __syncthreads();
    auto get_cand = [&](unsigned i) -> uint2 { return (i < n_inl || staged) ? cand_s[i] : __ldcg(cand_g + (i - n_inl)); };
    fstamp(p, 13);

    Resolved r;
    r.b1 = (unsigned)sh.seg_b1[s];
    const unsigned k1 = (unsigned)p.top_k - sh.seg_above[s];     // 1 <= k1 <= n_c members still to take
    unsigned long long prefix = 0ull, mask_above = 0ull;
    if (k1 >= n_c) {
        // every member is taken
    } else if (n_c <= (unsigned)kDirectRankMax) {
        // few members: the one with exactly k1-1 larger keys is the last one taken
        const unsigned i = (unsigned)tid >> 2;             // four threads a member
        unsigned long long key = 0ull;
        unsigned larger = 0;
        if (i < n_c) {
            key = cand_key(cand_s[i]);
#pragma unroll 2
            for (unsigned j = tid & 3; j < n_c; j += 4) larger += cand_key(cand_s[j]) > key;
        }
        larger += __shfl_xor_sync(0xffffffffu, larger, 1);
        larger += __shfl_xor_sync(0xffffffffu, larger, 2);
        if (i < n_c && larger == k1 - 1) ts.key_at = key;
        __syncthreads();
        prefix = ts.key_at;
        mask_above = ~0ull;
    } else {
        // radix levels on (low 20 vote bits | inverted index): 10, 10, 11, 11, 10 bits from the top
        unsigned k_rem = k1, active = n_c;
        const int shifts[5] = {42, 32, 21, 10, 0};
        const unsigned widths[5] = {10, 10, 11, 11, 10};
#pragma unroll 1
        for (int lv = 0; lv < 5; ++lv) {
            if (k_rem >= active) break;                    // everything still active is taken
            __syncthreads();
#pragma unroll 1
            for (int i = tid; i < kHistBins; i += kFusedThreads) sh.hist[i] = 0u;
            __syncthreads();
            const unsigned long long dmask = (1ull << widths[lv]) - 1ull;
#pragma unroll 1
            for (unsigned i = tid; i < n_c; i += kFusedThreads) {
                const unsigned long long key = cand_key(get_cand(i));
                if ((key & mask_above) == prefix) atomicAdd(&sh.hist[(unsigned)((key >> shifts[lv]) & dmask)], 1u);
            }
            __syncthreads();
            find_threshold<false>(sh, sh.hist, k_rem);
            prefix |= (unsigned long long)(unsigned)sh.res_bin << shifts[lv];
            mask_above |= dmask << shifts[lv];
            k_rem -= sh.res_above;
            active = sh.res_cnt;
        }
    }
    fstamp(p, 14);
    // selected members in front of this CTA's range
    unsigned before = 0;
#pragma unroll 1
    for (unsigned i = tid; i < n_c; i += kFusedThreads) {
        const uint2 c = get_cand(i);
        if ((int)c.x < sg.t0 && (cand_key(c) & mask_above) >= prefix) ++before;
    }
    unsigned none, tot;                                    // (cand_s may be reused by the caller after this)
    sum_over_warps(__reduce_add_sync(0xffffffffu, before), sh.warp_sum2, none, tot);
    r.prefix = prefix;
    r.mask = mask_above;
    r.before = ts.sure_before + tot;
    fstamp(p, 15);
    return r;
}

__device__ __forceinline__ bool vote_selected(const Resolved& r, int t, unsigned vbits) {
    const unsigned bin = (vbits >> 20) & (kHistBins - 1);
    if (bin > r.b1) return true;
    if (bin < r.b1) return false;
    return (cand_key(make_uint2((unsigned)t, vbits)) & r.mask) >= r.prefix;
}

// Writes the winners of segment s in position order (list index n_init + rank) and leaves, in
// seg_above[s] / seg_cnt[s], the list index of the CTA's first winner and their number.
__device__ __forceinline__ void emit_segment(const LayerParams& p, FusedShared& sh, unsigned char* dyn, int s, const Resolved& r,
                                             bool fast) {
    const int tid = threadIdx.x;
    TailScratch& ts = tail_scratch(sh);
    const Seg sg = sh.seg[s];
    const int k = p.top_k;
    const int req = sh.plan.req[sg.b];
    const int* row = p.rtt + (long long)req * p.rtt_stride;
    int* out_slots = p.sel_slots + (size_t)sg.b * p.n_sel;
    int* out_pos = p.sel_pos + (size_t)sg.b * p.n_sel;
    int* cache_pos = p.pos_cache + ((size_t)req * p.n_layers + p.layer) * k;
    unsigned total_here;
    if (fast) {
        // the possible winners sit in the staged rows, in position order: rank them with one warp
        const int st = ts.fast_static, np = ts.fast_pot;
        if (tid < 32) {
            unsigned carry = 0;
#pragma unroll 1
            for (int base = 0; base < np; base += 32) {
                const int i = base + tid;
                const bool sel = i < np && vote_selected(r, ts.row_t[st + i], ts.row_v[st + i]);
                const unsigned bal = __ballot_sync(0xffffffffu, sel);
                if (i < np) {
                    const unsigned rank = r.before + carry + __popc(bal & ((1u << tid) - 1u));
                    ts.row_rank[st + i] = sel ? (int)(p.n_init + rank) : -1;
                    if (sel) {
                        if (rank < (unsigned)k) {
                            const int pos = p.n_init + ts.row_t[st + i];
                            out_pos[p.n_init + rank] = pos;
                            out_slots[p.n_init + rank] = ts.row_slot[st + i];
                            if (p.query_cache) cache_pos[rank] = pos;          // topk_indices_cache[layer] = ... (:415)
                        } else {
                            set_error(p.err, TS_ERR_INTERNAL, (int)rank);
                        }
                    }
                }
                carry += __popc(bal);
            }
            if (tid == 0) { sh.tmp_u[0] = r.before; sh.tmp_u[1] = carry; }
        }
        __syncthreads();
        total_here = sh.tmp_u[0] + sh.tmp_u[1];
    } else {
        const float* votes_s = own_votes(dyn);
        const float* votes_g = p.votes_sel + sh.plan.off[sg.b];
        const WarpRange wr = warp_range(sg);
        auto selected = [&](int t, float v) { return vote_selected(r, t, __float_as_uint(v)); };
        unsigned mine = 0;
        for_own_votes(sh, votes_s, votes_g, s, wr, [&](int t, const float4& v) { mine += quad_of(wr, t, v, selected).total(); });
        unsigned in_front, tot;
        sum_over_warps(mine, sh.warp_sum, in_front, tot);
        if (tid == 0) { sh.tmp_u[0] = r.before; sh.tmp_u[1] = tot; }
        if (mine > 0u) {
            unsigned at = r.before + in_front;
            for_own_votes(sh, votes_s, votes_g, s, wr, [&](int t, const float4& v) {
                const Quad q = quad_of(wr, t, v, selected);
                unsigned rank = at + q.before_lane();
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if (!q.has(i)) continue;
                    if (rank < (unsigned)k) {
                        const int pos = p.n_init + t + i;
                        out_pos[p.n_init + rank] = pos;
                        out_slots[p.n_init + rank] =
                            sh.own_in_smem ? own_slots(dyn)[sh.seg_off[s] + (t + i - sg.t0)] : checked_slot(p, row, pos);
                        if (p.query_cache) cache_pos[rank] = pos;          // topk_indices_cache[layer] = ... (:415)
                    } else {
                        set_error(p.err, TS_ERR_INTERNAL, (int)rank);
                    }
                    ++rank;
                }
                at += q.total();
            });
        }
        __syncthreads();
        total_here = sh.tmp_u[0] + sh.tmp_u[1];
    }
    // the CTA owning the request's last candidates checks the total
    if (sg.t1 >= pooled_len(sh.plan.nc[sg.b], p.kernel_size) && tid == 0 && total_here != (unsigned)k) set_error(p.err, TS_ERR_INTERNAL, (int)total_here);
    __syncthreads();
    if (tid == 0) {
        sh.seg_above[s] = (unsigned)p.n_init + sh.tmp_u[0];
        sh.seg_cnt[s] = sh.tmp_u[1];
        ts.n_inl = 0u; ts.sure_before = 0u;                // for the next segment
    }
    __syncthreads();
}

// ------------------------------------------------------------------------------------------
// phase 5: attention over staged rows
// ------------------------------------------------------------------------------------------
// sin and cos of a non-negative angle of up to a few thousand radians: two-constant reduction to [-pi, pi]
// (2*pi = 6.2831854820251465 - 1.7484555e-7 in fp32 pieces), then the special-function unit (absolute error
// below 1e-6, far inside the attention tolerance; the library's sincosf would cost hundreds of instruction
// bytes at each place it is used).
__device__ __forceinline__ void sincos_reduced(float a, float& sn, float& cn) {
    const float n = rintf(a * 0.15915494309189535f);
    float r = fmaf(n, -6.2831854820251465f, a);
    r = fmaf(n, 1.7484555e-7f, r);
    sn = __sinf(r);
    cn = __cosf(r);
}

// Rotation rows of the staged rows' list positions, in the order the lanes of the multiplying warps read them:
// positions in tiles of eight; inside a tile the (cos, sin) of frequency i = 16s + 8u + 2t + w of position g
// sits in float2 (((s*2+u)*8 + g)*4 + t)*2 + w.
__device__ __forceinline__ void fill_rotation_rows(const LayerParams& p, const TailScratch& ts, float2* cs, int row0, int row1) {
#pragma unroll 1
    for (int idx = row0 * 64 + (int)threadIdx.x; idx < row1 * 64; idx += kFusedThreads) {
        const int r = idx >> 6, i = idx & 63;
        const int rank = max(ts.row_rank[r], 0);
        float sn, cn;
        sincos_reduced(__fmul_rn((float)rank, ts.inv_freq[i]), sn, cn);
        const int tile = r >> 3, g = r & 7;
        const int s = i >> 4, u = (i >> 3) & 1, t = (i >> 1) & 3, w = i & 1;
        cs[(tile * 256 + ((s * 2 + u) * 8 + g) * 4 + t) * 2 + w] = make_float2(cn, sn);
    }
}

// The request's query rotated at position count-1, fp32, [hq][kQStride] in shared memory.
__device__ __forceinline__ void fill_rotated_query(const LayerParams& p, const float* inv_freq, const __nv_bfloat16* q_b, int count,
                                                   float* q_s, int tid, int nthr) {
#pragma unroll 1
    for (int idx = tid; idx < p.hq * 64; idx += nthr) {
        const int h = idx >> 6, i = idx & 63;
        float sn, cn;
        sincos_reduced(__fmul_rn((float)(count - 1), inv_freq[i]), sn, cn);
        const float x1 = __bfloat162float(q_b[h * 128 + i]), x2 = __bfloat162float(q_b[h * 128 + i + 64]);
        q_s[h * kQStride + i] = x1 * cn - x2 * sn;
        q_s[h * kQStride + i + 64] = x2 * cn + x1 * sn;
    }
}

__device__ __forceinline__ void rotate_query_early(const LayerParams& p, FusedShared& sh, unsigned char* dyn, int off, int tid, int nthr) {
    fill_rotated_query(p, p.attn_inv_freq, reinterpret_cast<const __nv_bfloat16*>(p.q), min(sh.plan.n[0], p.n_sel),
                       reinterpret_cast<float*>(dyn + off), tid, nthr);
}

// What the attention over a round's staged rows needs besides the rows' final list positions: zeros in the
// unused rows of the last, partly filled block (0-weight products must stay finite), "not attended" marks for
// them, the rotated query (`query`), and (from row `cs_rows` down) the rotation rows of positions already known.
template <int HKV>
__device__ __forceinline__ void attend_prepare(const LayerParams& p, FusedShared& sh, unsigned char* dyn, int b, int rows,
                                               int cs_rows, bool query) {
    using AG = AttnGeom<HKV>;
    const int t = (int)threadIdx.x;
    constexpr int nthr = kFusedThreads;
    TailScratch& ts = tail_scratch(sh);
    unsigned char* sm_k = dyn;
    unsigned char* sm_v = dyn + AG::kRows * AG::kRowS;
    const int rows16 = (rows + 15) / 16 * 16;
#pragma unroll 1
    for (int i = rows * (AG::kRowB / 16) + t; i < rows16 * (AG::kRowB / 16); i += nthr) {
        const int r = i / (AG::kRowB / 16), c = i - r * (AG::kRowB / 16);
        *reinterpret_cast<uint4*>(sm_k + r * AG::kRowS + c * 16) = make_uint4(0u, 0u, 0u, 0u);
        *reinterpret_cast<uint4*>(sm_v + r * AG::kRowS + c * 16) = make_uint4(0u, 0u, 0u, 0u);
    }
    if (t >= rows && t < rows16) ts.row_rank[t] = -1;
    if (query)
        fill_rotated_query(p, ts.inv_freq, reinterpret_cast<const __nv_bfloat16*>(p.q) + (size_t)b * p.hq * 128,
                           min(sh.plan.n[b], p.n_sel), reinterpret_cast<float*>(dyn + AG::kPartOff), t, nthr);
    if (cs_rows > 0) fill_rotation_rows(p, ts, reinterpret_cast<float2*>(dyn + AG::kCsOff), 0, cs_rows);
}

// One warp: S^T of 16 staged rows x one KV head's query heads on mma.sync, rows in groups of eight (the N of
// the instruction); a group without rows is skipped.  The rotated query and keys (fp32) go into the tensor
// cores as fp16: 11 significant bits, i.e. a logit error of a few 1e-4 at these shapes -- an order of magnitude
// inside what the bf16 output rounding already costs -- for ONE instruction per k-step (the bf16 high/low
// split of attend.cu needs three; this path is bound by the tensor pipe's rate for mma.sync).  Values beyond
// the fp16 range saturate.  The loops are kept rolled: this code runs once per launch.
template <int HKV>
__device__ __forceinline__ void attend_scores(const LayerParams& p, const unsigned char* sm_k, const float4* sm_cs,
                                              const float* q_s, int wb, int kv, int rows, float (&sc)[2][4]) {
    using AG = AttnGeom<HKV>;
    const int lane = threadIdx.x & 31;
    const int g = lane >> 2, t = lane & 3;
    const int G = p.group;
    const bool on = g < G;
    const float* qh = q_s + (size_t)(kv * G + min(g, G - 1)) * kQStride;
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) sc[j][i] = 0.f;
    const int lrow = lane & 7, lsel = lane >> 3;
    const int ngroups = min(2, (rows - wb * 16 + 7) >> 3);        // groups of eight rows this block really has
#pragma unroll 1
    for (int s = 0; s < 4; ++s) {
        // A fragments of k-steps s and s+4 (rows 8..15 of A are unused: zero)
        uint32_t af[2][2];
#pragma unroll
        for (int k2 = 0; k2 < 2; ++k2)
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const float2 x = *reinterpret_cast<const float2*>(qh + 16 * (s + 4 * k2) + 8 * u + 2 * t);
                af[k2][u] = pack_f16x2_sat(on ? x.x : 0.f, on ? x.y : 0.f);
            }
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            if (j < ngroups) {
                const float4* cst = sm_cs + (size_t)(wb * 2 + j) * 256;
                uint32_t r[4];
                const int doff = 16 * s + (lsel & 1) * 8 + (lsel >> 1) * 64;
                ldmatrix_x4(r, smem_u32(sm_k) + (wb * 16 + 8 * j + lrow) * AG::kRowS + kv * 256 + doff * 2);
                uint32_t bf[2][2];                         // [k-step s | s+4][b0 | b1]
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const float4 cs = cst[((s * 2 + u) * 8 + g) * 4 + t];
                    const float x1a = __uint_as_float(r[u] << 16), x1b = __uint_as_float(r[u] & 0xFFFF0000u);
                    const float x2a = __uint_as_float(r[2 + u] << 16), x2b = __uint_as_float(r[2 + u] & 0xFFFF0000u);
                    bf[0][u] = pack_f16x2_sat(x1a * cs.x - x2a * cs.y, x1b * cs.z - x2b * cs.w);
                    bf[1][u] = pack_f16x2_sat(x2a * cs.x + x1a * cs.y, x2b * cs.z + x1b * cs.w);
                }
#pragma unroll
                for (int k2 = 0; k2 < 2; ++k2) {
                    const uint32_t a4[4] = {af[k2][0], 0u, af[k2][1], 0u};
                    mma_f16_16816(sc[j], a4, bf[k2][0], bf[k2][1]);
                }
            }
        }
    }
}

// Softmax numerators of the block (base 2) and O^T = V^T . P^T into part_o [G][128], (max, sum) into part_ml [G].
template <int HKV>
__device__ __forceinline__ void attend_values(const LayerParams& p, const TailScratch& ts, const unsigned char* sm_v, int wb,
                                              int kv, int rows, const float (&sc)[2][4], float* part_o, float2* part_ml) {
    using AG = AttnGeom<HKV>;
    const int lane = threadIdx.x & 31;
    const int g = lane >> 2, t = lane & 3;
    const int G = p.group;
    const int lrow = lane & 7;
    float x[2][2], mx = -INFINITY;
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            float v = sc[j][u] * p.sm_scale;
            if (p.logit_cap > 0.f) v = p.logit_cap * tanhf(v / p.logit_cap);
            const int rr = wb * 16 + 8 * j + 2 * t + u;
            v = (rr < rows && ts.row_rank[rr] >= 0) ? v * kLog2e : -INFINITY;
            x[j][u] = v;
            mx = fmaxf(mx, v);
        }
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
    float pe[2][2], lsum = 0.f;
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            pe[j][u] = (x[j][u] == -INFINITY) ? 0.f : ex2_ftz(fmaxf(x[j][u] - mx, -126.f));
            lsum += pe[j][u];
        }
    lsum += __shfl_xor_sync(0xffffffffu, lsum, 1);
    lsum += __shfl_xor_sync(0xffffffffu, lsum, 2);
    uint32_t ph[2], pl[2];
    split_bf16x2(pe[0][0], pe[0][1], ph[0], pl[0]);
    split_bf16x2(pe[1][0], pe[1][1], ph[1], pl[1]);
#pragma unroll 1
    for (int db = 0; db < 8; ++db) {
        uint32_t a[4];
        ldmatrix_x4_trans(a, smem_u32(sm_v) + (wb * 16 + ((lane >> 4) & 1) * 8 + lrow) * AG::kRowS + kv * 256 +
                                 (16 * db + ((lane >> 3) & 1) * 8) * 2);
        float o[4] = {0.f, 0.f, 0.f, 0.f};
        mma_bf16_16816(o, a, ph[0], ph[1]);
        mma_bf16_16816(o, a, pl[0], pl[1]);
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int hh = 2 * t + u;
            if (hh < G) {
                part_o[hh * 128 + 16 * db + g] = o[u];
                part_o[hh * 128 + 16 * db + g + 8] = o[2 + u];
            }
        }
    }
    if (t == 0 && g < G) part_ml[g] = make_float2(mx, lsum);
}

// The rows of one (request, CTA): `st_cnt` rows that never depended on votes starting at static row st0,
// then `own_cnt` winners of this CTA starting at list index own0.  `staged`: all rows are already on their
// way (requested by classify_phase) and listed in the scratch.  Writes partial `pslot` of the request.
template <int HKV>
__device__ __forceinline__ void attend_rowset(const LayerParams& p, FusedShared& sh, unsigned char* dyn, int b, int pslot,
                                              int st0, int st_cnt, int own0, int own_cnt, bool staged, bool prepared,
                                              uint32_t& kv_parity, bool& dead) {
    using AG = AttnGeom<HKV>;
    const int tid = threadIdx.x, warp = tid >> 5;
    TailScratch& ts = tail_scratch(sh);
    const int G = p.group, hq = p.hq;
    unsigned char* sm_k = dyn;
    unsigned char* sm_v = dyn + AG::kRows * AG::kRowS;
    float2* cs = reinterpret_cast<float2*>(dyn + AG::kCsOff);
    float* part = reinterpret_cast<float*>(dyn + AG::kPartOff);       // [warps busy][G][130]; first the rotated query
    const uint32_t bar = smem_u32(&ts.kv_bar);
    const int count = min(sh.plan.n[b], p.n_sel);
    float* g_o = p.part_o + (size_t)pslot * hq * 128;
    float2* g_ml = p.part_ml + (size_t)pslot * hq;
    const int total = st_cnt + own_cnt;
    if (total == 0) {
#pragma unroll 1
        for (int h = tid; h < hq; h += kFusedThreads) g_ml[h] = make_float2(-INFINITY, 0.f);
        return;
    }
    const int* rtt_row = p.rtt + (long long)sh.plan.req[b] * p.rtt_stride;
#pragma unroll 1
    for (int r0 = 0; r0 < total; r0 += AG::kRows) {
        const int rows = min(AG::kRows, total - r0);
        const int rows16 = (rows + 15) / 16 * 16;
        if (!staged) {
            // look the round's rows up and request them
            __syncthreads();                               // the previous round's readers are done
            if (tid < rows) {
                const int i = r0 + tid;
                int slot, rank;
                if (i < st_cnt) {
                    int pos;
                    static_row(p, sh, b, st0 + i, rank, pos);
                    slot = checked_slot(p, rtt_row, pos);
                } else {
                    rank = own0 + (i - st_cnt);
                    slot = __ldcg(p.sel_slots + (size_t)b * p.n_sel + rank);
                    if ((unsigned long long)(long long)slot >= (unsigned long long)p.pool_rows) {
                        set_error(p.err, TS_ERR_BAD_SLOT, slot);
                        slot = 0;
                    }
                }
                ts.row_slot[tid] = slot;
                ts.row_rank[tid] = rank;
            }
            asm volatile("fence.proxy.async;" ::: "memory");
            __syncthreads();
            if (tid == 0) mbar_expect_tx(bar, (uint32_t)rows * 2u * AG::kRowB);
            if (tid < rows) {
                const int slot = ts.row_slot[tid];
                bulk_g2s(smem_u32(sm_k) + tid * AG::kRowS, reinterpret_cast<const unsigned char*>(p.k_pool) + (size_t)slot * AG::kRowB,
                         AG::kRowB, bar);
                bulk_g2s(smem_u32(sm_v) + tid * AG::kRowS, reinterpret_cast<const unsigned char*>(p.v_pool) + (size_t)slot * AG::kRowB,
                         AG::kRowB, bar);
            }
        }
        if (prepared && r0 == 0) {
            // the caller zeroed the unused rows, rotated the query and filled the static rows' rotation rows
            // while the final set was being settled; only the winners' rotation rows are left
            fill_rotation_rows(p, ts, cs, ts.fast_static, rows16);
        } else {
            attend_prepare<HKV>(p, sh, dyn, b, rows, 0, true);
            __syncthreads();
            fill_rotation_rows(p, ts, cs, 0, rows16);
        }
        __syncthreads();
        fstamp(p, 18);
        mbar_wait(bar, kv_parity, p.err, dead, 5, p.wait_cycles);
        kv_parity ^= 1u;
        fstamp(p, 19);
        const int nblk = rows16 / 16;
        const int wb = warp / HKV, kv = warp % HKV;
        float sc[2][4];
        const float* q_s = prepared && r0 == 0 && query_is_early<HKV>(p, sh) ? reinterpret_cast<const float*>(dyn + sh.vote_top) : part;
        if (wb < nblk) attend_scores<HKV>(p, sm_k, reinterpret_cast<const float4*>(cs), q_s, wb, kv, rows, sc);
        __syncthreads();                                   // the rotated query has been read: its place takes the partials
        float* my_o = part + (size_t)warp * G * 130;
        if (wb < nblk) attend_values<HKV>(p, ts, sm_v, wb, kv, rows, sc, my_o, reinterpret_cast<float2*>(my_o + G * 128));
        fstamp(p, 20);
        __syncthreads();
        // merge the blocks of the round (and, from the second round on, the partial written so far):
        // per head the new (max, sum) and the weights of the pieces, then the weighted outputs
        float* s_w = reinterpret_cast<float*>(sh.hist);               // [hq][kBlocks + 1] weights, then [hq][2] (max, sum)
        constexpr int kW = AG::kBlocks + 1;
        const bool more = r0 > 0;
        if (tid < hq) {
            const int h = tid, kvh = h / G, gg = h - kvh * G;
            const float2 prev = more ? g_ml[h] : make_float2(-INFINITY, 0.f);
            float mm = prev.x;
#pragma unroll 1
            for (int w = 0; w < nblk; ++w)
                mm = fmaxf(mm, reinterpret_cast<const float2*>(part + (size_t)(w * HKV + kvh) * G * 130 + G * 128)[gg].x);
            const float wp = (prev.x == -INFINITY) ? 0.f : ex2_ftz(fmaxf(prev.x - mm, -126.f));
            float ll = prev.y * wp;
            s_w[h * kW + AG::kBlocks] = wp;
#pragma unroll 1
            for (int w = 0; w < AG::kBlocks; ++w) {
                float wgt = 0.f;
                if (w < nblk) {
                    const float2 ml = reinterpret_cast<const float2*>(part + (size_t)(w * HKV + kvh) * G * 130 + G * 128)[gg];
                    wgt = (ml.x == -INFINITY) ? 0.f : ex2_ftz(fmaxf(ml.x - mm, -126.f));
                    ll += ml.y * wgt;
                }
                s_w[h * kW + w] = wgt;
            }
            s_w[hq * kW + 2 * h] = mm;
            s_w[hq * kW + 2 * h + 1] = ll;
        }
        __syncthreads();
#pragma unroll 1
        for (int idx = tid; idx < hq * 128; idx += kFusedThreads) {
            const int h = idx >> 7, e = idx & 127;
            const int kvh = h / G, gg = h - kvh * G;
            const float wp = s_w[h * kW + AG::kBlocks];
            float acc = wp > 0.f ? g_o[idx] * wp : 0.f;
#pragma unroll 1
            for (int w = 0; w < nblk; ++w) {
                const float wgt = s_w[h * kW + w];
                if (wgt > 0.f) acc += part[(size_t)(w * HKV + kvh) * G * 130 + gg * 128 + e] * wgt;
            }
            g_o[idx] = acc;
        }
        if (tid < hq) g_ml[tid] = make_float2(s_w[hq * kW + 2 * tid], s_w[hq * kW + 2 * tid + 1]);
        fstamp(p, 21);
        staged = false;                                    // only the first round can have been requested early
    }
    __syncthreads();
}

// Phases 4 and 5 for everything this CTA holds.
template <int HKV, bool ATTN>
__device__ __forceinline__ void resolve_and_attend(const LayerParams& p, FusedShared& sh, unsigned char* dyn, bool& dead) {
    constexpr bool attn = ATTN;
    using AG = AttnGeom<(HKV > 0 ? HKV : 1)>;
    TailScratch& ts = tail_scratch(sh);
    // members are staged where the rotation rows and the partial outputs go later (behind the K/V rows, which
    // may already be arriving), up to the copies of the own votes and pool rows, which the emission reads; the inline
    // members of all records (at most kMaxGrid * kRecInline) always fit
    constexpr int kOwnOff = kFusedDynSmem - 2 * kOwnCap * 4;
    static_assert(AG::kCsOff + kMaxGrid * kRecInline * 8 <= kOwnOff, "all records' inline members fit the staging area");
    uint2* cand_s = reinterpret_cast<uint2*>(dyn + (attn ? AG::kCsOff : 0));
    unsigned cand_cap = (unsigned)((kOwnOff - (attn ? AG::kCsOff : 0)) / 8);
    const bool prepared = ATTN && ts.fast != 0 && ts.pad == 1u;
    if constexpr (ATTN) {
        if (prepared) {
            // the attention's inputs were prepared before the barrier, where the members would be staged: they go
            // behind the partial outputs instead (into the shared-memory copies of the own votes, done with here)
            cand_s = reinterpret_cast<uint2*>(dyn + early_cand_offset<HKV>(p));
            cand_cap = (unsigned)((kFusedDynSmem - early_cand_offset<HKV>(p)) / 8);
        }
    }
#pragma unroll 1
    for (int s = 0; s < sh.nseg; ++s) {
        const Resolved r = resolve_segment(p, sh, s, cand_s, cand_cap);
        emit_segment(p, sh, dyn, s, r, ts.fast != 0 && s == 0);
        fstamp(p, 16);
    }
    if constexpr (ATTN) {
        uint32_t kv_parity = 0;
        // the staged row set first (its rows are already in flight), then every other request this CTA has a part in
        const int nb = p.batch;
#pragma unroll 1
        for (int it = 0; it < 2 * nb; ++it) {
            const int pass = it >= nb ? 1 : 0, b = it - pass * nb;
            const bool is_fast = ts.fast != 0 && b == ts.fast_b;
            if ((pass == 0) != is_fast) continue;
            int me, st0, st_cnt, own0 = 0, own_cnt = 0;
            if (is_fast) {
                // staged rows: the static ones, then the possible winners (those not selected carry rank -1)
                me = ts.fast_share;
                st0 = 0;
                st_cnt = ts.fast_static + ts.fast_pot;
            } else {
                const StaticShare ss = static_share(p, sh, b, AG::kRows);
                me = share_index(p, ss);
                if (me < 0) continue;
                st0 = me * ss.chunk;
                st_cnt = max(0, min(ss.total, st0 + ss.chunk) - st0);
#pragma unroll 1
                for (int s = 0; s < sh.nseg; ++s)
                    if (sh.seg[s].b == b) { own0 = (int)sh.seg_above[s]; own_cnt = (int)sh.seg_cnt[s]; }
            }
            attend_rowset<HKV>(p, sh, dyn, b, sh.pbase[b] + me, st0, st_cnt, own0, own_cnt, is_fast, is_fast && prepared, kv_parity,
                               dead);
        }
    }
}

// ------------------------------------------------------------------------------------------
// phase 6: merge of the partials; one (request, head, quarter of the head dimension) per CTA at a time
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ void merge_phase(const LayerParams& p, FusedShared& sh) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int hq = p.hq;
    float* s_acc = reinterpret_cast<float*>(sh.hist);          // [16 warps][32]
    float* s_red = s_acc + 16 * 32;                              // [2][16]
    const int items = p.batch * hq * 4;
    fstamp(p, 22);
#pragma unroll 1
    for (int item = blockIdx.x; item < items; item += gridDim.x) {
        const int b = item / (hq * 4), rem = item - b * hq * 4;
        const int h = rem >> 2, qd = rem & 3;
        const int np = sh.pbase[b + 1] - sh.pbase[b];
        if (np <= 0) continue;
        const float2* ml = p.part_ml + (size_t)sh.pbase[b] * hq + h;
        const float* o = p.part_o + ((size_t)sh.pbase[b] * hq + h) * 128 + qd * 32 + lane;
        float mm = -INFINITY, ll = 0.f, acc = 0.f;
#pragma unroll 1
        for (int c0 = 0; c0 < np; c0 += 16 * 10) {
            // (max, sum) of up to 160 partials, and this warp's share of their outputs, requested together
            const int c = c0 + tid;
            float2 mine = make_float2(-INFINITY, 0.f);
            if (c < np && tid < 16 * 10) mine = __ldcg(ml + (size_t)c * hq);
            constexpr int kPer = 10;                          // partials per warp and round: one round for grids up to 160
            float xo[kPer];
#pragma unroll
            for (int u = 0; u < kPer; ++u) {
                const int cc = c0 + warp + 16 * u;
                xo[u] = cc < np ? __ldcg(o + (size_t)cc * hq * 128) : 0.f;
            }
            float m2 = mine.x;
#pragma unroll
            for (int off = 16; off >= 1; off >>= 1) m2 = fmaxf(m2, __shfl_xor_sync(0xffffffffu, m2, off));
            __syncthreads();
            fstamp(p, 23);
            if (lane == 0) s_red[warp] = m2;
            __syncthreads();
            float mn = mm;
#pragma unroll
            for (int w = 0; w < 16; ++w) mn = fmaxf(mn, s_red[w]);
            const float wgt = (mine.x == -INFINITY) ? 0.f : exp2f(mine.x - mn);
            float l2 = mine.y * wgt;
#pragma unroll
            for (int off = 16; off >= 1; off >>= 1) l2 += __shfl_xor_sync(0xffffffffu, l2, off);
            if (lane == 0) s_red[16 + warp] = l2;
            // weights of the partials this warp holds: partial cc belongs to thread cc - c0
            float* s_w = reinterpret_cast<float*>(sh.hist) + 1024;   // [512]
            s_w[tid] = wgt;
            __syncthreads();
            const float rescale = (mm == -INFINITY) ? 0.f : exp2f(mm - mn);
            acc *= rescale;
            ll *= rescale;
#pragma unroll
            for (int w = 0; w < 16; ++w) ll += s_red[16 + w];
#pragma unroll
            for (int u = 0; u < kPer; ++u) {
                const int cl = warp + 16 * u;
                if (c0 + cl < np) {
                    const float w = s_w[cl];
                    acc += w > 0.f ? w * xo[u] : 0.f;
                }
            }
            mm = mn;
        }
        __syncthreads();
        s_acc[warp * 32 + lane] = acc;
        __syncthreads();
        if (warp == 0) {
            float r = 0.f;
#pragma unroll
            for (int w = 0; w < 16; ++w) r += s_acc[w * 32 + lane];
            reinterpret_cast<__nv_bfloat16*>(p.out)[((size_t)b * hq + h) * 128 + qd * 32 + lane] = __float2bfloat16_rn(ll > 0.f ? r / ll : 0.f);
        }
        __syncthreads();
    }
    fstamp(p, 24);
}

}  // namespace ts
