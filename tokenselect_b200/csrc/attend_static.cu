// ts_attend_rows_static: sparse paged decode attention over a caller-supplied list of pool rows, for
// callers that must not allocate.
//
// Who that is: code that runs where device allocation is forbidden or impossible -- a host callback or a
// latency-critical serving loop that is not allowed to touch the allocator (cudaMalloc can synchronise the
// device), or a process whose device memory was handed out in full at start-up (to the KV pool, say) and
// whose owner gives out no more.  Such a caller cannot use ts_create(), which makes one cudaMalloc for its
// workspace.  This entry point needs no handle: the split kernel's partial results go
// to a fixed array that is part of the library image, the caller passes only inputs and the output.
//
// The array is shared by every call in the process and keeps whatever the last call left in it.  Nothing
// in it has to start at zero (every partial that the merge reads is written by the split of the same
// call).  Two calls whose kernels overlap on the GPU (different streams, no ordering) race on it.
//
// The first call on a device looks up the array's device address (cudaGetSymbolAddress).  That first call
// should be made before any stream capture begins.
//
// Same arithmetic as csrc/attend.cu (query rotated at position count-1, j-th listed key at position j,
// rotate-half pairing, logits * sm_scale, optional soft cap, fp32 softmax, KV head = h / group), except
// that cos/sin are evaluated in the kernel instead of being read from the handle's tables.
#include <math.h>

#include "common.cuh"

namespace ts {

constexpr size_t kStaticScratchBytes = 4u << 20;       // 4 MiB, held by every GPU that loads the library
constexpr int kStaticChunkMax = 32, kStaticChunkMin = 16;   // listed rows per split CTA
constexpr int kStaticMaxDevices = 64;

static __device__ __align__(256) unsigned char g_static_scratch[kStaticScratchBytes];

struct StaticParams {
    const void* q;
    const void* k_pool;
    const void* v_pool;
    const int* rows;
    void* out;
    float* scratch;                 // [chunks][hq][d] unnormalised partial outputs
    float2* scratch_ml;             // [chunks][hq] (max in base-2 units, sum)
    long long pool_rows;
    int hq, hkv, d, count, chunk_rows, chunks;
    float sm_scale, logit_cap;
    double log2_base, rope_scale;
    int* status;                    // optional device int: set to TS_ERR_BAD_SLOT on a row outside the pool
};

// Split kernel.  One CTA = one chunk of listed rows for ALL heads; a warp = one KV head and up to four of its query
// heads, eight rows at a time; lane l holds elements [P*l, P*l+P) of both halves of a row (P = d/64), i.e. both
// members of each rotation pair.
//
// What bounds it: latency (11 MB at 2688 rows x 8 KV heads is 2 us of HBM time).  So the chunk's rotation angles are
// evaluated once per CTA and shared by every head (a CTA per KV head evaluated them eight times over, each warp
// again for each query head), before the kernel waits for its predecessor; a warp's eight K and V rows are all
// requested before the first is used; and the 32 partial dot products of eight rows x four heads are reduced over
// the lanes together, 31 shuffles instead of 160.
constexpr int kStaticThreads = 256;
constexpr int kStaticHeads = 4;                         // query heads per warp
constexpr int kStaticRows = 8;                          // rows per step of a warp

template <typename T, int P> struct LaneElems;          // P consecutive elements
template <> struct LaneElems<__nv_bfloat16, 2> { using type = uint32_t; };
template <> struct LaneElems<__nv_bfloat16, 1> { using type = __nv_bfloat16; };
template <> struct LaneElems<float, 2> { using type = float2; };
template <> struct LaneElems<float, 1> { using type = float; };
template <typename T, int P>
__device__ __forceinline__ void unpack(const T (&raw)[P], float (&x)[P]) {
#pragma unroll
    for (int e = 0; e < P; ++e) x[e] = to_f32<T>(raw[e]);
}

// WIDE: q and the pools are aligned to P elements, so a lane's elements come with one load; otherwise one by one.
template <typename T, int P, bool WIDE>
__device__ __forceinline__ void load_elems(const T* src, T (&raw)[P]) {
    if constexpr (WIDE) {
        using Raw = typename LaneElems<T, P>::type;
        *reinterpret_cast<Raw*>(raw) = *reinterpret_cast<const Raw*>(src);
    } else {
#pragma unroll
        for (int e = 0; e < P; ++e) raw[e] = src[e];
    }
}

template <typename T, int P, bool WIDE>
__global__ void __launch_bounds__(kStaticThreads) static_split_kernel(const StaticParams p) {
    constexpr int D = 64 * P, HALF = 32 * P;
    struct alignas(P * sizeof(T)) Elems { T x[P]; };
    __shared__ float2 sm_cs[kStaticChunkMax][HALF];     // (cos, sin) of the chunk's positions
    __shared__ float2 sm_qcs[HALF];                     // of the query's position
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int G = p.hq / p.hkv;
    const int base = blockIdx.x * p.chunk_rows;
    const int cnt = min(p.chunk_rows, p.count - base);
    static_assert(kStaticThreads % HALF == 0, "a thread evaluates one frequency");
    const int e = threadIdx.x % HALF;
    const float inv_freq = (float)(exp2(-p.log2_base * (double)(2 * e) / (double)D) / p.rope_scale);
    for (int r = threadIdx.x / HALF; r <= cnt; r += kStaticThreads / HALF) {
        const int pos = r < cnt ? base + r : p.count - 1;   // row cnt stands for the query
        float s, c;
        sincosf(__fmul_rn((float)pos, inv_freq), &s, &c);
        if (r < cnt) sm_cs[r][e] = make_float2(c, s);
        else sm_qcs[e] = make_float2(c, s);
    }
    // nothing above depends on the predecessor's results
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    __syncthreads();
    const T* kpool = reinterpret_cast<const T*>(p.k_pool);
    const T* vpool = reinterpret_cast<const T*>(p.v_pool);
    const T* q = reinterpret_cast<const T*>(p.q);
    const int nsub = (G + kStaticHeads - 1) / kStaticHeads;
    for (int unit = warp; unit < p.hkv * nsub; unit += kStaticThreads / 32) {
        const int kv = unit / nsub, g0 = (unit - kv * nsub) * kStaticHeads;
        const int ng = min(kStaticHeads, G - g0);
        const int h0 = kv * G + g0;
        float q1[kStaticHeads][P], q2[kStaticHeads][P];
#pragma unroll
        for (int g = 0; g < kStaticHeads; ++g) {
            float x1[P], x2[P];
            Elems a, b;
            const T* qh = q + (size_t)(h0 + min(g, ng - 1)) * D + P * lane;
            load_elems<T, P, WIDE>(qh, a.x);
            load_elems<T, P, WIDE>(qh + HALF, b.x);
            unpack(a.x, x1);
            unpack(b.x, x2);
#pragma unroll
            for (int e = 0; e < P; ++e) {
                const float2 cs = sm_qcs[P * lane + e];
                q1[g][e] = x1[e] * cs.x - x2[e] * cs.y;
                q2[g][e] = x2[e] * cs.x + x1[e] * cs.y;
            }
        }
        // running softmax of head lane & 3 (the same in the eight lanes that share a head), this lane's output elements
        float m = -INFINITY, l = 0.f, o1[kStaticHeads][P], o2[kStaticHeads][P];
#pragma unroll
        for (int g = 0; g < kStaticHeads; ++g)
#pragma unroll
            for (int e = 0; e < P; ++e) { o1[g][e] = 0.f; o2[g][e] = 0.f; }
        for (int r0 = 0; r0 < cnt; r0 += kStaticRows) {
            int my_row = 0;
            if (lane < kStaticRows && r0 + lane < cnt) {
                my_row = p.rows[base + r0 + lane];
                if ((unsigned long long)(long long)my_row >= (unsigned long long)p.pool_rows) {
                    if (p.status != nullptr) atomicCAS(p.status, 0, TS_ERR_BAD_SLOT);
                    my_row = 0;
                }
            }
            Elems k1[kStaticRows], k2[kStaticRows], v1[kStaticRows], v2[kStaticRows];
#pragma unroll
            for (int r = 0; r < kStaticRows; ++r) {
                const int row = __shfl_sync(0xffffffffu, my_row, min(r, cnt - r0 - 1));   // past the end: the last row again
                const size_t at = ((size_t)row * p.hkv + kv) * D + P * lane;
                load_elems<T, P, WIDE>(kpool + at, k1[r].x);
                load_elems<T, P, WIDE>(kpool + at + HALF, k2[r].x);
                load_elems<T, P, WIDE>(vpool + at, v1[r].x);
                load_elems<T, P, WIDE>(vpool + at + HALF, v2[r].x);
            }
            float s[kStaticRows * kStaticHeads];
#pragma unroll
            for (int r = 0; r < kStaticRows; ++r) {
                float x1[P], x2[P];
                unpack(k1[r].x, x1);
                unpack(k2[r].x, x2);
                float acc[kStaticHeads] = {0.f, 0.f, 0.f, 0.f};
                const int rr = min(r0 + r, cnt - 1);
#pragma unroll
                for (int e = 0; e < P; ++e) {
                    const float2 cs = sm_cs[rr][P * lane + e];
                    const float y1 = x1[e] * cs.x - x2[e] * cs.y, y2 = x2[e] * cs.x + x1[e] * cs.y;
#pragma unroll
                    for (int g = 0; g < kStaticHeads; ++g) acc[g] += q1[g][e] * y1 + q2[g][e] * y2;
                }
#pragma unroll
                for (int g = 0; g < kStaticHeads; ++g) s[r * kStaticHeads + g] = acc[g];
            }
            // lane r*4 + g ends up with the whole sum of (row r, head g)
#pragma unroll
            for (int off = 16; off >= 1; off >>= 1) {
                const bool up = (lane & off) != 0;
#pragma unroll
                for (int i = 0; i < off; ++i) {
                    const float keep = up ? s[i + off] : s[i], send = up ? s[i] : s[i + off];
                    s[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
                }
            }
            float x = s[0] * p.sm_scale;
            if (p.logit_cap > 0.f) x = p.logit_cap * tanhf(x / p.logit_cap);
            x = (r0 + (lane >> 2) < cnt) ? x * 1.4426950408889634f : -INFINITY;
            float mn = fmaxf(m, x);
#pragma unroll
            for (int off = 4; off <= 16; off <<= 1) mn = fmaxf(mn, __shfl_xor_sync(0xffffffffu, mn, off));
            const float pe = (x == -INFINITY) ? 0.f : exp2f(x - mn);
            const float sc = (m == -INFINITY) ? 0.f : exp2f(m - mn);
            float sum = pe;
#pragma unroll
            for (int off = 4; off <= 16; off <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
            l = l * sc + sum;
            m = mn;
#pragma unroll
            for (int g = 0; g < kStaticHeads; ++g) {
                const float scg = __shfl_sync(0xffffffffu, sc, g);
#pragma unroll
                for (int e = 0; e < P; ++e) { o1[g][e] *= scg; o2[g][e] *= scg; }
            }
#pragma unroll
            for (int r = 0; r < kStaticRows; ++r) {
                if (r0 + r >= cnt) break;                  // warp-uniform
                float x1[P], x2[P];
                unpack(v1[r].x, x1);
                unpack(v2[r].x, x2);
#pragma unroll
                for (int g = 0; g < kStaticHeads; ++g) {
                    const float pg = __shfl_sync(0xffffffffu, pe, r * kStaticHeads + g);
#pragma unroll
                    for (int e = 0; e < P; ++e) { o1[g][e] += pg * x1[e]; o2[g][e] += pg * x2[e]; }
                }
            }
        }
#pragma unroll
        for (int g = 0; g < kStaticHeads; ++g) {
            if (g < ng) {
                float* dst = p.scratch + ((size_t)blockIdx.x * p.hq + h0 + g) * D;
#pragma unroll
                for (int e = 0; e < P; ++e) { dst[P * lane + e] = o1[g][e]; dst[HALF + P * lane + e] = o2[g][e]; }
            }
        }
        if (lane < ng) p.scratch_ml[(size_t)blockIdx.x * p.hq + h0 + lane] = make_float2(m, l);
    }
}

// grid hq, 512 threads: warp w joins partials w, w+16, ...; lane i holds elements [VEC*i, VEC*i + VEC).  (One thread
// per element walking all partials twice was one dependent chain of 84 rounds at that size.)
constexpr int kStaticMergeThreads = 512;
template <typename T, int VEC>
__global__ void __launch_bounds__(kStaticMergeThreads) static_merge_kernel(const StaticParams p) {
    constexpr int D = 32 * VEC, NW = kStaticMergeThreads / 32, kAhead = 8;
    __shared__ float s_acc[NW][D];
    __shared__ float2 s_ml[NW];
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int h = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float m = -INFINITY, l = 0.f, acc[VEC];
#pragma unroll
    for (int v = 0; v < VEC; ++v) acc[v] = 0.f;
    for (int c0 = warp; c0 < p.chunks; c0 += NW * kAhead) {
        float x[kAhead][VEC];
        float2 ml[kAhead];
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            const int c = c0 + NW * u;
            ml[u] = make_float2(-INFINITY, 0.f);
#pragma unroll
            for (int v = 0; v < VEC; ++v) x[u][v] = 0.f;
            if (c < p.chunks) {
                ml[u] = __ldcg(p.scratch_ml + (size_t)c * p.hq + h);
                const float* src = p.scratch + ((size_t)c * p.hq + h) * D + VEC * lane;
                if constexpr (VEC == 4) {
                    const float4 t = __ldcg(reinterpret_cast<const float4*>(src));
                    x[u][0] = t.x; x[u][1] = t.y; x[u][2] = t.z; x[u][3] = t.w;
                } else {
                    const float2 t = __ldcg(reinterpret_cast<const float2*>(src));
                    x[u][0] = t.x; x[u][1] = t.y;
                }
            }
        }
        float mn = m;
#pragma unroll
        for (int u = 0; u < kAhead; ++u) mn = fmaxf(mn, ml[u].x);
        const float sc = (m == -INFINITY) ? 0.f : exp2f(m - mn);
        l *= sc;
#pragma unroll
        for (int v = 0; v < VEC; ++v) acc[v] *= sc;
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            const float w = (ml[u].x == -INFINITY) ? 0.f : exp2f(ml[u].x - mn);
            l += ml[u].y * w;
#pragma unroll
            for (int v = 0; v < VEC; ++v) acc[v] += x[u][v] * w;
        }
        m = mn;
    }
#pragma unroll
    for (int v = 0; v < VEC; ++v) s_acc[warp][VEC * lane + v] = acc[v];
    if (lane == 0) s_ml[warp] = make_float2(m, l);
    __syncthreads();
    for (int e = threadIdx.x; e < D; e += kStaticMergeThreads) {
        float mm = -INFINITY, r = 0.f, ll = 0.f;
#pragma unroll
        for (int w = 0; w < NW; ++w) mm = fmaxf(mm, s_ml[w].x);
#pragma unroll
        for (int w = 0; w < NW; ++w) {
            const float wgt = (s_ml[w].x == -INFINITY) ? 0.f : exp2f(s_ml[w].x - mm);
            r += s_acc[w][e] * wgt;
            ll += s_ml[w].y * wgt;
        }
        reinterpret_cast<T*>(p.out)[(size_t)h * D + e] = from_f32<T>(r / ll);
    }
}

template <typename T, int P, bool WIDE>
static cudaError_t launch_static_t(const StaticParams& p, cudaStream_t stream) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cfg.stream = stream;
    cfg.gridDim = dim3(p.chunks);
    cfg.blockDim = dim3(kStaticThreads);
    cudaError_t e = cudaLaunchKernelEx(&cfg, static_split_kernel<T, P, WIDE>, p);
    if (e != cudaSuccess) return e;
    cfg.gridDim = dim3(p.hq);
    cfg.blockDim = dim3(kStaticMergeThreads);
    return cudaLaunchKernelEx(&cfg, static_merge_kernel<T, 2 * P>, p);
}
// The entry point takes tensors at any element offset; rows are multiples of 128 bytes, so the bases decide.
template <typename T, int P>
static cudaError_t launch_static(const StaticParams& p, cudaStream_t stream) {
    const uintptr_t bits = reinterpret_cast<uintptr_t>(p.q) | reinterpret_cast<uintptr_t>(p.k_pool) | reinterpret_cast<uintptr_t>(p.v_pool);
    return bits % (P * sizeof(T)) == 0 ? launch_static_t<T, P, true>(p, stream) : launch_static_t<T, P, false>(p, stream);
}

}  // namespace ts

extern "C" int ts_attend_rows_static(const ts_attend_static_args* a) {
    using namespace ts;
    if (!a || a->struct_size != sizeof(ts_attend_static_args)) return TS_ERR_INVALID_ARG;
    if (!a->q || !a->k_pool || !a->v_pool || !a->rows || !a->out) return TS_ERR_INVALID_ARG;
    if (a->hq < 1 || a->hkv < 1 || a->hq % a->hkv != 0 || a->count < 1 || a->pool_rows < 1) return TS_ERR_INVALID_ARG;
    if (a->dtype != TS_DTYPE_BF16 && a->dtype != TS_DTYPE_F32) return TS_ERR_UNSUPPORTED;
    if (a->head_dim != 64 && a->head_dim != 128) return TS_ERR_UNSUPPORTED;
    if (a->hq / a->hkv > 8) return TS_ERR_UNSUPPORTED;
    if (!(a->rope_base > 0.0) || !(a->rope_scale > 0.0)) return TS_ERR_INVALID_ARG;
    // the fixed array bounds the list length: one partial of head_dim + 2 floats per chunk and head must fit
    const size_t per_chunk = (size_t)a->hq * (a->head_dim + 2) * sizeof(float);
    const auto chunks_of = [a](int rows) { return (a->count + rows - 1) / rows; };
    if (chunks_of(kStaticChunkMax) * per_chunk > kStaticScratchBytes) return TS_ERR_CAPACITY;
    // Small chunks while their partials fit: the kernel is bound by one CTA's latency, so a list is spread over as
    // many CTAs as the array allows.
    const int chunk_rows = chunks_of(kStaticChunkMin) * per_chunk <= kStaticScratchBytes ? kStaticChunkMin : kStaticChunkMax;
    const int chunks = chunks_of(chunk_rows);

    // One-time set-up per device, with that device current: the array's name is only a host-side handle
    // here; kernels need its device address.
    static float* scratch_of_device[kStaticMaxDevices] = {nullptr};
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kStaticMaxDevices) return TS_ERR_CUDA;
    if (scratch_of_device[dev] == nullptr) {
        void* ptr = nullptr;
        if (cudaGetSymbolAddress(&ptr, g_static_scratch) != cudaSuccess || ptr == nullptr) return TS_ERR_CUDA;
        scratch_of_device[dev] = static_cast<float*>(ptr);
    }

    StaticParams p;
    p.q = a->q; p.k_pool = a->k_pool; p.v_pool = a->v_pool; p.rows = a->rows; p.out = a->out;
    p.scratch = scratch_of_device[dev];
    p.scratch_ml = reinterpret_cast<float2*>(p.scratch + (size_t)chunks * a->hq * a->head_dim);
    p.pool_rows = a->pool_rows;
    p.hq = a->hq; p.hkv = a->hkv; p.d = a->head_dim; p.count = a->count;
    p.chunk_rows = chunk_rows; p.chunks = chunks;
    p.sm_scale = a->sm_scale; p.logit_cap = a->logit_cap;
    p.log2_base = log2(a->rope_base); p.rope_scale = a->rope_scale;
    p.status = a->status;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(a->stream);
    cudaError_t e;
    if (a->dtype == TS_DTYPE_BF16) e = a->head_dim == 128 ? launch_static<__nv_bfloat16, 2>(p, s) : launch_static<__nv_bfloat16, 1>(p, s);
    else e = a->head_dim == 128 ? launch_static<float, 2>(p, s) : launch_static<float, 1>(p, s);
    return e == cudaSuccess ? TS_OK : TS_ERR_CUDA;
}
