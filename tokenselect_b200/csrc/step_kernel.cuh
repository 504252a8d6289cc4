// The decode layer step as ONE lean kernel: K/V append, scoring, soft vote, exact top-k, sparse attention and
// the merge of its partials, for the shapes the staged tensor-core scoring handles (bf16, head_dim 128, 1/2/4/8
// KV heads per rank, no vote pooling), on one GPU or with the vote sum over ranks done inside the kernel.
// Included by fused.cu, whose general selection kernel keeps every other mode (fp32 check mode, plain and
// register scoring, the split tensor-parallel form, max-pooled votes, prefill chunks).
//
// Why a kernel of its own: every phase after the key stream runs ONCE per launch, and a phase that runs once
// costs what its instruction bytes cost to fetch (measured: a fraction of a microsecond per kilobyte, the
// instruction cache hit rate of the general kernel is ~40 %).  This kernel therefore carries no mode
// switches, keeps its cold loops rolled and calls the helpers that appear in several places out of line.
//
// Replaces patcher/token_retrieval.py:777-825 (store_kv_cache :844-854, retrieval_indices :375-449,
// get_topk_tokens :338-373 with paged_matmul :166-261, the decode attention call :815-823).
#pragma once

namespace ts {

template <int HKV>
__global__ void __launch_bounds__(kFusedThreads, 1) decode_step_kernel(const LayerParams p, const int tp_fused) {
    using T = __nv_bfloat16;
    extern __shared__ __align__(128) unsigned char ring[];
    __shared__ FusedShared sh;
    const int tid = threadIdx.x;
    bool dead = false;
    // Launched with programmatic serialization where the runtime accepts it: the CTAs may be placed while the
    // previous kernel drains; nothing is read or written before it has finished.
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (tp_fused && tid == 0) {
        const unsigned e = p.cta_epoch[blockIdx.x] + 1u;
        p.cta_epoch[blockIdx.x] = e;
        sh.epoch = e;
    }
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    stamp(p, 0);
    if (p.stamps) stamp_range_slow(p.phase_ts, 0);
    const int err0 = *(volatile int*)p.err;
    dead = err0 != 0;                   // a handle in error waits for nothing (its kernels do nothing either)
    unsigned bar_gen = tid == 0 ? grid_barrier_generation(p) : 0u;
    const int mode = tp_fused ? kModeTpFused : kModeAll;
    // Selection cache off: the flags follow from the lengths alone, so the plan is built first and the
    // per-request preparation runs on the multiplying warps while the first key rows are in flight.  With the
    // cache on, the decisions come first and a grid barrier publishes them.
    const bool side = p.query_cache == 0;
    if (!side) {
        // one decision for the CTA: the preparation has barriers, and another CTA's may set the error word meanwhile
        const bool stop = (int)blockIdx.x < p.batch && __syncthreads_or(err0 != 0);
#pragma unroll 1
        for (int b = blockIdx.x; b < p.batch && !stop; b += gridDim.x) {
            prepare_request_cached<T>(p, b, sh.prep, reinterpret_cast<float*>(ring));
        }
        grid_barrier(p, dead, bar_gen);
    }
    bool ok = side ? build_plan<true>(p, sh.plan) : build_plan<false>(p, sh.plan);
    ok = ok && err0 == 0;
    if (tid == 0) {
        plan_ownership(p, sh, ok, true, AttnGeom<HKV>::kRows, true);
        // below the own-candidate copies and, where it has been rotated already, the attention's query
        const int q_off = early_query_offset(p, kScoreStages * ScoreGeom<HKV>::kStageBytes);
        sh.vote_top = q_off ? q_off : kFusedDynSmem - 2 * kOwnCap * 4;
        mbar_init(smem_u32(&sh.row_bar[0]), 1);
        mbar_init(smem_u32(&sh.row_bar[1]), 1);
        mbar_init(smem_u32(&sh.part_bar), 1);
#pragma unroll 1
        for (int s = 0; s < kScoreStages; ++s) {
            mbar_init(smem_u32(&sh.full[s]), ScoreGeom<HKV>::kFullArrivals);
            mbar_init(smem_u32(&sh.empty[s]), 8);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    // raw votes of this rank: the workspace, or (exchange inside the kernel) this rank's peer-visible buffer
    float* votes_raw = tp_fused ? p.peer_votes[(sh.epoch & 1u) * kMaxTp + p.tp_rank] : p.votes;
    stamp(p, 1);
    const bool nothing_to_score = sh.tile_off[p.batch] == 0;
    if (side && (nothing_to_score || !ok)) side_work<T>(p, sh, mode, err0, ok, whole_cta());
    if (!side && ok) emit_windows(p, sh, whole_cta());
    if (!nothing_to_score) {
        if (ok) {
            if (!side) {
                // a CTA without candidates of request b still owes (-inf, 0) statistics for it
#pragma unroll 1
                for (int i = tid; i < p.batch * p.hq; i += kFusedThreads) {
                    const int b = i / p.hq, c = i - b * p.hq;
                    bool mine = false;
                    for (int s = 0; s < sh.nseg; ++s) mine |= sh.seg[s].b == b;
                    if (sh.plan.flag[b] == TS_FLAG_RECOMPUTE && !mine)
                        p.partials[(size_t)b * p.part_stride + (size_t)blockIdx.x * p.hq + c] = make_float2(-INFINITY, 0.f);
                }
            }
            score_phase_tma<T, HKV, (HKV > kBulkMinHkv), true>(p, sh, ring, dead, side, mode, err0);
            vote_prefetch(p, sh, ring);
        }
        stamp(p, 2);
        if (p.stamps) stamp_range_slow(p.phase_ts, 1);
        grid_barrier(p, dead, bar_gen);
        stamp(p, 3);
        if (ok) vote_phase(p, sh, ring, !tp_fused, dead, votes_raw);
        stamp(p, 4);
        if (tp_fused) tp_exchange_phase(p, sh, ring, ok, dead);
        stamp(p, 24);
        grid_barrier_arrive(p);
    } else if (side) {
        // every request attends to all its tokens: nothing but this barrier lies between the append of the new rows, by
        // the CTA that prepares the request, and their attention by another one (with the cache on, the decisions' barrier)
        grid_barrier_arrive(p);
    }
    tail_init(p, sh);
    if (nothing_to_score && side) grid_barrier_wait(p, dead, bar_gen);
    if (!nothing_to_score) {
        StaticRows st{0, 0, -1, -1};
        if (ok) st = look_up_static_rows<HKV>(p, sh);
        grid_barrier_wait(p, dead, bar_gen);
        stamp(p, 5);
        if (ok) classify_phase<HKV, true>(p, sh, ring, st);
        stamp(p, 6);
        grid_barrier_arrive(p);
        if (ok) {
            issue_staged_rows<HKV>(p, sh, ring);
            early_prepare<HKV>(p, sh, ring);
        }
        grid_barrier_wait(p, dead, bar_gen);
        stamp(p, 7);
    }
    if (ok) resolve_and_attend<HKV, true>(p, sh, ring, dead);
    stamp(p, 8);
    grid_barrier(p, dead, bar_gen);
    stamp(p, 15);
    if (ok) merge_phase(p, sh);
    stamp(p, 16);
    if (p.stamps) stamp_range_slow(p.phase_ts, 2);
}

}  // namespace ts
