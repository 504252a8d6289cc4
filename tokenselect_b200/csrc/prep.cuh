// Per-request preparation of one layer step, as device functions shared by the stand-alone
// prepare kernel (tensor-parallel form) and phase 0 of the fused selection kernel:
// K/V append, scoring-query rotation, cosine terms of the selection cache and the
// recompute / reuse / dense decision.
//
// Replaces store_kv_cache (token_retrieval.py:844-854), the query rotation at :380-388 with
// RotaryEmbedding.apply_rotary_pos_emb (:98-107), the guard at :376-378 and the (intended)
// selection-cache rule at :394-421.
#pragma once
#include "common.cuh"

namespace ts {

// Decision for one request given the three cosine terms.  Thread 0 of the block calls it.
// The request's flag, and the caller's copy of it when one was asked for (written by the kernel itself: a copy
// node between the kernels of a captured token would serialise them).
__device__ __forceinline__ void put_flag(const LayerParams& p, int b, int f) {
    p.flags[b] = f;
    if (p.flags_out != nullptr) p.flags_out[b] = f;
}

template <typename T>
__device__ __forceinline__ int decide(const LayerParams& p, int b, int req, float dot, float qq, float cc) {
    int flag = TS_FLAG_RECOMPUTE;
    if (p.query_cache) {
        int* valid = p.valid + (size_t)req * p.n_layers + p.layer;
        bool recompute = true;
        if (*valid) {
            // cos = dot / (sqrt(qq) * sqrt(cc)), every operation rounded to fp32
            float den = __fmul_rn(__fsqrt_rn(qq), __fsqrt_rn(cc));
            float c = (den == 0.f) ? 0.f : __fdiv_rn(dot, den);
            recompute = c < p.theta;                       // strict <, :397-400
        }
        flag = recompute ? TS_FLAG_RECOMPUTE : TS_FLAG_REUSE;
        atomicAdd(p.counters + 2 * (size_t)req, 1ULL);     // retrieval_count, :421
        if (!recompute) atomicAdd(p.counters + 2 * (size_t)req + 1, 1ULL);  // skip_count, :420
        if (recompute) *valid = 1;                         // is_first_query = False, :417
    }
    return flag;
}

struct PrepShared {
    int flag;
    float terms[3];
};

// A group of `nthr` consecutive threads of the CTA (all of them, or some of its warps) that synchronises
// on hardware barrier `bar`; `tid` is the thread's index inside the group.
struct ThreadGroup {
    int tid, nthr, bar;
    __device__ __forceinline__ void sync() const {
        asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(nthr) : "memory");
    }
};
__device__ __forceinline__ ThreadGroup whole_cta() { return ThreadGroup{(int)threadIdx.x, (int)blockDim.x, 0}; }

// All threads of the group call this for request b (uniformly).  kFusedDecide: the layer's own kernel with the selection
// cache off; otherwise (tensor-parallel form) also publish the cosine terms, which are summed over ranks first.
template <typename T, bool kFusedDecide>
__device__ __forceinline__ void prepare_request(const LayerParams& p, int b, const ThreadGroup& tg) {
    const int tid = tg.tid;
    const int n = p.seq_lens[b];
    const int req = p.req_pool_indices[b];
    const int hd = p.hq * p.d;
    if (n < 1 || n > p.max_ctx || req < 0 || req >= p.max_reqs) {
        if (tid == 0) { set_error(p.err, TS_ERR_BAD_LENGTH, n); put_flag(p, b, TS_FLAG_DENSE); }
        return;
    }

    // 1. append this step's K/V rows to the pools (:849-850)
    if (p.k_new != nullptr) {
        int loc = p.out_cache_loc[b];
        if (loc < 0 || loc >= p.pool_rows) {
            if (tid == 0) { set_error(p.err, TS_ERR_BAD_SLOT, loc); put_flag(p, b, TS_FLAG_DENSE); }
            return;
        }
        const int row_vec = p.hkv * p.d * (int)sizeof(T) / 16;
        const uint4* ks = reinterpret_cast<const uint4*>(p.k_new) + (size_t)b * row_vec;
        const uint4* vs = reinterpret_cast<const uint4*>(p.v_new) + (size_t)b * row_vec;
        uint4* kd = reinterpret_cast<uint4*>(p.k_pool) + (size_t)loc * row_vec;
        uint4* vd = reinterpret_cast<uint4*>(p.v_pool) + (size_t)loc * row_vec;
#pragma unroll 1
        for (int i = tid; i < row_vec; i += tg.nthr) { kd[i] = ks[i]; vd[i] = vs[i]; }
    }

    // 2. clear this request's first-level histogram and candidate counter
#pragma unroll 1
    for (int i = tid; i < kHistBins; i += tg.nthr) p.hist[(size_t)b * kHistBins + i] = 0u;
    if (tid == 0) p.cand_count[b] = 0u;

    // 3. guard (:376-378): short requests attend to everything
    if (p.n_sel >= n) {
        if (tid == 0) put_flag(p, b, TS_FLAG_DENSE);
        return;
    }

    // 4. rotate the scoring query at the fixed position and round to the model dtype (:98-107).
    //    out[i] = x[i]*cos + (-x[i+d/2])*sin ; out[i+d/2] = x[i+d/2]*cos + x[i]*sin, each product and
    //    the sum rounded separately, as eager tensor arithmetic does.
    const T* q = reinterpret_cast<const T*>(p.q) + (size_t)b * hd;
    T* qr = reinterpret_cast<T*>(p.q_rot) + (size_t)b * hd;
    const int half = p.d / 2;
#pragma unroll 1
    for (int e = tid; e < p.hq * half; e += tg.nthr) {
        int h = e / half, i = e % half;
        if (p.q_prerot) {                                  // a prefill chunk's fingerprint: copy
            qr[h * p.d + i] = q[h * p.d + i];
            qr[h * p.d + i + half] = q[h * p.d + i + half];
            continue;
        }
        float x1 = to_f32<T>(q[h * p.d + i]);
        float x2 = to_f32<T>(q[h * p.d + i + half]);
        float2 cs = p.score_cs[i];
        float r1 = __fadd_rn(__fmul_rn(x1, cs.x), __fmul_rn(-x2, cs.y));
        float r2 = __fadd_rn(__fmul_rn(x2, cs.x), __fmul_rn(x1, cs.y));
        qr[h * p.d + i] = from_f32<T>(r1);
        qr[h * p.d + i + half] = from_f32<T>(r2);
    }
    if (kFusedDecide) {                                    // (with the cache on: prepare_request_cached)
        if (tid == 0) put_flag(p, b, TS_FLAG_RECOMPUTE);
        return;
    }
    tg.sync();

    // 5. cosine terms against the cached query in a fixed order: lane j sums elements j + 32*i in
    //    ascending i, then an XOR butterfly (16, 8, 4, 2, 1) joins the 32 partial sums.
    const T* fp = reinterpret_cast<const T*>(p.fp_cache) + ((size_t)req * p.n_layers + p.layer) * hd;
    if (p.query_cache && tid < 32) {
        float dot = 0.f, qq = 0.f, cc = 0.f;
        const bool have = p.valid[(size_t)req * p.n_layers + p.layer] != 0;
        if (have) {
            // sixteen elements per lane are requested together (the sums stay in ascending order): this warp is
            // on the critical path of every layer when the cache is on, and one round trip per element would
            // cost it tens of microseconds
            constexpr int kBatch = 16;
#pragma unroll 1
            for (int e0 = tid; e0 < hd; e0 += 32 * kBatch) {
                float a[kBatch], c[kBatch];
#pragma unroll
                for (int u = 0; u < kBatch; ++u) {
                    const int e = e0 + 32 * u;
                    const bool in = e < hd;
                    a[u] = in ? to_f32<T>(qr[e]) : 0.f;
                    c[u] = in ? to_f32<T>(fp[e]) : 0.f;
                }
#pragma unroll
                for (int u = 0; u < kBatch; ++u) {
                    if (e0 + 32 * u < hd) {
                        dot = __fadd_rn(dot, __fmul_rn(a[u], c[u]));
                        qq = __fadd_rn(qq, __fmul_rn(a[u], a[u]));
                        cc = __fadd_rn(cc, __fmul_rn(c[u], c[u]));
                    }
                }
            }
#pragma unroll
            for (int o = 16; o >= 1; o >>= 1) {
                dot = __fadd_rn(dot, __shfl_xor_sync(0xffffffffu, dot, o));
                qq = __fadd_rn(qq, __shfl_xor_sync(0xffffffffu, qq, o));
                cc = __fadd_rn(cc, __shfl_xor_sync(0xffffffffu, cc, o));
            }
        }
        if (tid == 0) {
            p.cos_terms[4 * b + 0] = dot; p.cos_terms[4 * b + 1] = qq;
            p.cos_terms[4 * b + 2] = cc;  p.cos_terms[4 * b + 3] = 0.f;
        }
    }
    if (tid == 0) put_flag(p, b, TS_FLAG_RECOMPUTE);       // provisional: decide_request overwrites it
}

// The same for the selection cache's decision inside the layer's own kernel, by a whole CTA with 2*hq*d floats of scratch:
// everything every other CTA waits for at the barrier that follows.  So it takes two round trips: what only depends on
// the request's place in the batch is requested at once (lengths, slot, query, new rows), then the cached query and its
// valid flag; rotated and cached query meet in shared memory, and three warps sum the three cosine terms side by side,
// each in the fixed order of step 5.  (Step by step, with the rotated query written to global memory and read back by one
// warp, the decision took 12.5 us of a reusing step's 28.)
template <typename T>
__device__ __forceinline__ void prepare_request_cached(const LayerParams& p, int b, PrepShared& ps, float* scratch) {
    const int tid = threadIdx.x, nthr = blockDim.x, lane = tid & 31, warp = tid >> 5;
    const int hd = p.hq * p.d, half = p.d / 2, pairs = p.hq * half;
    const int n = p.seq_lens[b];
    const int req = p.req_pool_indices[b];
    const bool append = p.k_new != nullptr;
    const int loc = append ? p.out_cache_loc[b] : 0;
    const int row_vec = p.hkv * p.d * (int)sizeof(T) / 16;
    const uint4* ks = reinterpret_cast<const uint4*>(p.k_new) + (size_t)b * row_vec;
    const uint4* vs = reinterpret_cast<const uint4*>(p.v_new) + (size_t)b * row_vec;
    uint4 k0 = make_uint4(0u, 0u, 0u, 0u), v0 = k0;
    if (append && tid < row_vec) { k0 = ks[tid]; v0 = vs[tid]; }
    const T* q = reinterpret_cast<const T*>(p.q) + (size_t)b * hd;
    constexpr int kAhead = 4;                              // rotation pairs a thread requests together
    float x1[kAhead], x2[kAhead];
    float2 cs[kAhead];
    auto load_pairs = [&](int e0) {
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            const int e = min(e0 + u * nthr, pairs - 1), h = e / half, i = e - h * half;
            x1[u] = to_f32<T>(q[h * p.d + i]);
            x2[u] = to_f32<T>(q[h * p.d + i + half]);
            cs[u] = p.score_cs[i];
        }
    };
    load_pairs(tid);
    if (n < 1 || n > p.max_ctx || req < 0 || req >= p.max_reqs) {
        if (tid == 0) { set_error(p.err, TS_ERR_BAD_LENGTH, n); put_flag(p, b, TS_FLAG_DENSE); }
        return;
    }
    if (append) {
        if (loc < 0 || loc >= p.pool_rows) {
            if (tid == 0) { set_error(p.err, TS_ERR_BAD_SLOT, loc); put_flag(p, b, TS_FLAG_DENSE); }
            return;
        }
        uint4* kd = reinterpret_cast<uint4*>(p.k_pool) + (size_t)loc * row_vec;
        uint4* vd = reinterpret_cast<uint4*>(p.v_pool) + (size_t)loc * row_vec;
        if (tid < row_vec) { kd[tid] = k0; vd[tid] = v0; }
#pragma unroll 1
        for (int i = tid + nthr; i < row_vec; i += nthr) { kd[i] = ks[i]; vd[i] = vs[i]; }
    }
    if (p.n_sel >= n) {
        if (tid == 0) { p.cand_count[b] = 0u; put_flag(p, b, TS_FLAG_DENSE); }
        return;
    }
    const size_t entry = (size_t)req * p.n_layers + p.layer;
    T* fp = reinterpret_cast<T*>(p.fp_cache) + entry * hd;
    constexpr int kVec = 16 / (int)sizeof(T);              // hq*d is a multiple of 64
    const bool have = p.valid[entry] != 0;
    float* q_s = scratch;
    float* c_s = scratch + hd;
#pragma unroll 1
    for (int e = tid * kVec; e < hd; e += nthr * kVec) {
        alignas(16) T raw[kVec];
        *reinterpret_cast<uint4*>(raw) = *reinterpret_cast<const uint4*>(fp + e);
#pragma unroll
        for (int u = 0; u < kVec; ++u) c_s[e + u] = to_f32<T>(raw[u]);
    }
#pragma unroll 1
    for (int i = tid; i < kHistBins; i += nthr) p.hist[(size_t)b * kHistBins + i] = 0u;
    if (tid == 0) p.cand_count[b] = 0u;
    T* qr = reinterpret_cast<T*>(p.q_rot) + (size_t)b * hd;
#pragma unroll 1
    for (int e0 = tid; e0 < pairs; e0 += kAhead * nthr) {
        if (e0 != tid) load_pairs(e0);
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            const int e = e0 + u * nthr, h = e / half, i = e - h * half;
            if (e >= pairs) continue;
            T r1 = from_f32<T>(x1[u]), r2 = from_f32<T>(x2[u]);            // a prefill chunk's fingerprint: as it is
            if (!p.q_prerot) {
                r1 = from_f32<T>(__fadd_rn(__fmul_rn(x1[u], cs[u].x), __fmul_rn(-x2[u], cs[u].y)));
                r2 = from_f32<T>(__fadd_rn(__fmul_rn(x2[u], cs[u].x), __fmul_rn(x1[u], cs[u].y)));
            }
            qr[h * p.d + i] = r1;
            qr[h * p.d + i + half] = r2;
            q_s[h * p.d + i] = to_f32<T>(r1);
            q_s[h * p.d + i + half] = to_f32<T>(r2);
        }
    }
    __syncthreads();
    if (warp < 3) {
        const float* a = warp == 2 ? c_s : q_s;
        const float* c = warp == 1 ? q_s : c_s;
        float sum = 0.f;
        if (have) {
#pragma unroll 8
            for (int e = lane; e < hd; e += 32) sum = __fadd_rn(sum, __fmul_rn(a[e], c[e]));
#pragma unroll
            for (int o = 16; o >= 1; o >>= 1) sum = __fadd_rn(sum, __shfl_xor_sync(0xffffffffu, sum, o));
        }
        if (lane == 0) ps.terms[warp] = sum;
    }
    __syncthreads();
    if (tid == 0) {
        const int f = decide<T>(p, b, req, ps.terms[0], ps.terms[1], ps.terms[2]);
        put_flag(p, b, f);
        ps.flag = f;
    }
    __syncthreads();
    if (ps.flag == TS_FLAG_RECOMPUTE) {                    // query_fingerprints_cache[layer] = q (:416)
#pragma unroll 1
        for (int e = tid * kVec; e < hd; e += nthr * kVec) {
            alignas(16) T raw[kVec];
#pragma unroll
            for (int u = 0; u < kVec; ++u) raw[u] = from_f32<T>(q_s[e + u]);
            *reinterpret_cast<uint4*>(fp + e) = *reinterpret_cast<const uint4*>(raw);
        }
    }
    // The scratch lies in the ring, whose next writers are bulk copies of key rows (another proxy): their writes come after
    // the ones above only behind this fence.
    asm volatile("fence.proxy.async;" ::: "memory");
    __syncthreads();                                       // the scratch serves the CTA's next request
}

// Tensor-parallel form: the cosine terms were summed over ranks by the caller.
template <typename T>
__device__ __forceinline__ void decide_request(const LayerParams& p, int b, PrepShared& ps) {
    const int tid = threadIdx.x;
    int& s_flag = ps.flag;
    const int n = p.seq_lens[b];
    const int req = p.req_pool_indices[b];
    if (n < 1 || n > p.max_ctx || req < 0 || req >= p.max_reqs) return;
    if (p.n_sel >= n) return;                              // prep already wrote TS_FLAG_DENSE
    const int hd = p.hq * p.d;
    if (tid == 0) {
        int f = decide<T>(p, b, req, p.cos_terms[4 * b], p.cos_terms[4 * b + 1], p.cos_terms[4 * b + 2]);
        put_flag(p, b, f);
        s_flag = f;
    }
    __syncthreads();
    if (p.query_cache && s_flag == TS_FLAG_RECOMPUTE) {
        const T* qr = reinterpret_cast<const T*>(p.q_rot) + (size_t)b * hd;
        T* fpw = reinterpret_cast<T*>(p.fp_cache) + ((size_t)req * p.n_layers + p.layer) * hd;
#pragma unroll 1
        for (int e = tid; e < hd; e += blockDim.x) fpw[e] = qr[e];
    }
}

}  // namespace ts
