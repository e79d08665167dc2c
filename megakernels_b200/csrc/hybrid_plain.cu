// Prefill attention with 32-bit arithmetic: the float build's, and the bf16 build's for head sizes the tensor-core
// kernels do not take.  One CTA per kQueries neighbouring tokens and query head: 128 keys at a time, a thread per key
// for the scores (a key is read once for all queries), online softmax, a thread per value column for the outputs.  The
// keys are the union of what the queries see; a query leaves out the others' values (whatever they hold).
// Bound by reads of keys and values: one query per CTA read every key as scalars a row apart, and 300 tokens with
// 16 heads of 2 x 64 / 128 in float32 took 487 us; 95 here.
#include "hybrid_kernels.h"

#include <type_traits>

namespace mkbh {
namespace {

constexpr int kThreads = 128, kWarps = kThreads / 32;

template <typename T>
struct PlainArgs {
    MkbhLayer L;
    const float* proj;  // differential: the stacked projection
    int64_t ld;
    const T* query;  // rotary and latent
    int64_t ldq;
    KeySource<T> src;
    int n, pos0;
    float eps;
    T* out;
    int64_t ldo;
};

template <typename T> __device__ __forceinline__ float4 load4(const T* p, bool wide) {
    if constexpr (sizeof(T) == 4)
        if (wide) return *reinterpret_cast<const float4*>(p);
    return make_float4(to_f(p[0]), to_f(p[1]), to_f(p[2]), to_f(p[3]));
}

// kMaps 2: the differential mixer (a key is two halves, one per map), 1: rotary and latent; kE: value columns per thread
template <typename T, int kMaps, int kE>
__global__ void __launch_bounds__(kThreads) plain_attention_kernel(const PlainArgs<T> a) {
    constexpr int kQueries = kMaps == 2 ? 4 : 8, kRows = kMaps * kQueries;
    extern __shared__ __align__(16) float sm[];  // q [kRows][padded dim], p [kRows][128]; later o [kQueries][vdim]
    __shared__ float red[kRows * kWarps];
    __shared__ __align__(16) int rows[kThreads];
    const MkbhLayer& L = a.L;
    const int A = a.src.split, B = a.src.rest, D = A + B, DP = (D + 3) & ~3, E = L.vdim, H = L.heads;
    const int t0 = blockIdx.x * kQueries, h = blockIdx.y, g = h / a.src.per, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nq = min(kQueries, a.n - t0);
    float *q = sm, *p = sm + kRows * DP;
    for (int i = tid; i < kRows * DP; i += kThreads) {
        const int r = i / DP, d = i % DP, t = t0 + r % kQueries;
        float v = 0.f;
        if (r % kQueries < nq && d < D) {
            // (a query takes the precision of the activations it would have had as a stored tensor)
            if constexpr (kMaps == 2) v = to_f(from_f<T>(a.proj[(size_t)t * a.ld + (h * 2 + r / kQueries) * D + d]));
            else v = to_f(a.query[(size_t)t * a.ldq + h * D + d]);
        }
        q[i] = v;
    }
    // what the queries see: the kept positions, then first .. last
    int start[kQueries];
#pragma unroll
    for (int i = 0; i < kQueries; ++i) start[i] = KeyRange(a.pos0 + t0 + min(i, nq - 1), L.window, L.keep_first, L.chunk).start;
    const int first = start[0], last = a.pos0 + t0 + nq - 1, keep = L.chunk > 0 ? 0 : L.keep_first, sinks = min(keep, first);
    const int count = sinks + last + 1 - first;
    const float scale = L.scale * (kMaps == 1 && L.temp ? L.temp[h] : 1.f);
    const bool sink = kMaps == 1 && L.sink != nullptr;
    const bool wide = sizeof(T) == 4 && ((A | B | a.src.key_ld | a.src.shared_ld | a.src.key_head) & 3) == 0 &&
                      ((reinterpret_cast<uintptr_t>(a.src.keys) | reinterpret_cast<uintptr_t>(a.src.shared)) & 15) == 0;
    float m[kRows], l[kRows], acc[kRows][kE];
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
        m[r] = sink ? L.sink[h] : -INFINITY;
        l[r] = sink ? 1.f : 0.f;
#pragma unroll
        for (int e = 0; e < kE; ++e) acc[r][e] = 0.f;
    }
    __syncthreads();
    for (int c0 = 0; c0 < count; c0 += kThreads) {
        const int nk = min(kThreads, count - c0), j = c0 + tid, pos = j < sinks ? j : first + (j - sinks);
        auto seen = [&](int r) {
            const int i = r % kQueries;
            return tid < nk && i < nq && pos <= a.pos0 + t0 + i && (pos >= start[i] || pos < keep);
        };
        float s[kRows];
#pragma unroll
        for (int r = 0; r < kRows; ++r) s[r] = 0.f;
        rows[tid] = 0;
        if (tid < nk) {
            const int row = cache_row(pos, a.src.keep, a.src.ring);
            rows[tid] = row;
#pragma unroll
            for (int b = 0; b < kMaps; ++b) {
                const T* k = a.src.keys + (size_t)row * a.src.key_ld + g * a.src.key_head + b * D;
                auto span = [&](const T* x, int from, int size) {
                    int i = 0;
                    for (; i + 4 <= size && (from & 3) == 0; i += 4) {
                        const float4 v = load4(x + i, wide);
#pragma unroll
                        for (int r = b * kQueries; r < (b + 1) * kQueries; ++r) {
                            const float4 u = *reinterpret_cast<const float4*>(q + r * DP + from + i);
                            s[r] = fmaf(u.w, v.w, fmaf(u.z, v.z, fmaf(u.y, v.y, fmaf(u.x, v.x, s[r]))));
                        }
                    }
                    for (; i < size; ++i) {
                        const float v = to_f(x[i]);
#pragma unroll
                        for (int r = b * kQueries; r < (b + 1) * kQueries; ++r) s[r] = fmaf(q[r * DP + from + i], v, s[r]);
                    }
                };
                span(k, 0, A);
                if (B > 0) span(a.src.shared + (size_t)row * a.src.shared_ld, A, B);
            }
        }
#pragma unroll
        for (int r = 0; r < kRows; ++r) {
            s[r] = seen(r) ? s[r] * scale : -INFINITY;
            const float x = warp_max(s[r]);
            if (lane == 0) red[r * kWarps + warp] = x;
        }
        __syncthreads();
        float f[kRows];
#pragma unroll
        for (int r = 0; r < kRows; ++r) {
            float x = m[r];
#pragma unroll
            for (int w = 0; w < kWarps; ++w) x = fmaxf(x, red[r * kWarps + w]);
            const float off = x == -INFINITY ? 0.f : x;  // (nothing seen yet)
            f[r] = expf(m[r] - off);
            m[r] = x;
            s[r] = expf(s[r] - off);
            p[r * kThreads + tid] = seen(r) ? s[r] : -1.f;  // (weights are not negative)
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < kRows; ++r) {
            const float x = warp_sum(s[r]);
            if (lane == 0) red[r * kWarps + warp] = x;
        }
#pragma unroll
        for (int ei = 0; ei < kE; ++ei) {
            const int e = tid + ei * kThreads;
            if (e >= E) break;
            const T* v = a.src.values + g * a.src.value_head + e;
#pragma unroll
            for (int r = 0; r < kRows; ++r) acc[r][ei] *= f[r];
            auto add = [&](auto whole) {  // whole: every query sees every key of the chunk
                for (int k = 0; k < nk; k += 4) {
                    const int4 at = *reinterpret_cast<const int4*>(rows + k);
                    const float x0 = to_f(v[(size_t)at.x * a.src.value_ld]), x1 = to_f(v[(size_t)at.y * a.src.value_ld]);
                    const float x2 = to_f(v[(size_t)at.z * a.src.value_ld]), x3 = to_f(v[(size_t)at.w * a.src.value_ld]);
#pragma unroll
                    for (int r = 0; r < kRows; ++r) {
                        const float4 w = *reinterpret_cast<const float4*>(p + r * kThreads + k);
                        float y = acc[r][ei];
                        if (decltype(whole)::value || !(w.x < 0.f)) y = fmaf(w.x, x0, y);
                        if (decltype(whole)::value || !(w.y < 0.f)) y = fmaf(w.y, x1, y);
                        if (decltype(whole)::value || !(w.z < 0.f)) y = fmaf(w.z, x2, y);
                        if (decltype(whole)::value || !(w.w < 0.f)) y = fmaf(w.w, x3, y);
                        acc[r][ei] = y;
                    }
                }
            };
            const int low = first + (c0 - sinks);
            if (nk == kThreads && nq == kQueries && c0 >= sinks && low >= start[kQueries - 1] && low + kThreads - 1 <= a.pos0 + t0) add(std::true_type{});
            else add(std::false_type{});
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < kRows; ++r) {
            float x = 0.f;
#pragma unroll
            for (int w = 0; w < kWarps; ++w) x += red[r * kWarps + w];
            l[r] = l[r] * f[r] + x;
        }
        __syncthreads();
    }
    if constexpr (kMaps == 2) {
        float sq[kQueries];
#pragma unroll
        for (int i = 0; i < kQueries; ++i) {
            sq[i] = 0.f;
#pragma unroll
            for (int ei = 0; ei < kE; ++ei) {
                const float o = tid + ei * kThreads < E && i < nq ? acc[i][ei] / l[i] - L.lambda * (acc[kQueries + i][ei] / l[kQueries + i]) : 0.f;
                acc[i][ei] = o;
                sq[i] += o * o;
            }
        }
        block_sum<kQueries, kThreads>(sq, red);
#pragma unroll
        for (int i = 0; i < kQueries; ++i) {
            if (i >= nq) break;
            const float f = (1.f - L.diff) / sqrtf(sq[i] / E + a.eps);
            const float* gate = a.proj + (size_t)(t0 + i) * a.ld + H * 2 * D + h * E;
            T* dst = a.out + (size_t)(t0 + i) * a.ldo + h * E;
#pragma unroll
            for (int ei = 0; ei < kE; ++ei) {
                const int e = tid + ei * kThreads;
                if (e < E) dst[e] = from_f<T>(acc[i][ei] * f * sigmoid_f(gate[e]));
            }
        }
    } else {
        float* o = sm;  // (queries and weights have been read)
#pragma unroll
        for (int i = 0; i < kQueries; ++i)
#pragma unroll
            for (int ei = 0; ei < kE; ++ei)
                if (tid + ei * kThreads < E && i < nq) o[i * E + tid + ei * kThreads] = acc[i][ei] / l[i];
        __syncthreads();
        for (int i = 0; i < nq; ++i) {
            const float2* turn = L.value_rope ? reinterpret_cast<const float2*>(L.value_rope) + (size_t)(a.pos0 + t0 + i) * (E / 2) : nullptr;
            T* dst = a.out + (size_t)(t0 + i) * a.ldo + h * E;
            for (int e = tid; e < E; e += kThreads) {
                float y = o[i * E + e];
                if (turn != nullptr) {  // back by the query's angle
                    const float2 r = turn[e >> 1];
                    y = y * r.x + (e & 1 ? -r.y : r.y) * o[i * E + (e ^ 1)];
                }
                dst[e] = from_f<T>(y);
            }
        }
    }
    if (h == 0)
        for (int i = 0; i < nq; ++i)
            for (int e = H * E + tid; e < pad8(H * E); e += kThreads) a.out[(size_t)(t0 + i) * a.ldo + e] = from_f<T>(0.f);
}

template <typename T, int kMaps, int kE>
cudaError_t launch(const PlainArgs<T>& a, cudaStream_t s) {
    constexpr int kQueries = kMaps == 2 ? 4 : 8, kRows = kMaps * kQueries;
    const auto kernel = plain_attention_kernel<T, kMaps, kE>;
    const int dim = (a.src.split + a.src.rest + 3) & ~3;
    int floats = kRows * (dim + kThreads);
    if (floats < kQueries * a.L.vdim) floats = kQueries * a.L.vdim;
    if (floats * 4 > 47 * 1024) {  // (the kernel's own arrays are another kilobyte)
        // (the most there is, whatever this layer takes: another thread's call in between must not lower it)
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 226 * 1024);
        if (e != cudaSuccess) return e;
    }
    kernel<<<dim3((a.n + kQueries - 1) / kQueries, a.L.heads), kThreads, floats * 4, s>>>(a);
    return cudaGetLastError();
}
template <typename T, int kMaps>
cudaError_t choose(const PlainArgs<T>& a, cudaStream_t s) {
    const int per = (a.L.vdim + kThreads - 1) / kThreads;  // (vdim <= 512)
    return per <= 1 ? launch<T, kMaps, 1>(a, s) : per == 2 ? launch<T, kMaps, 2>(a, s) : launch<T, kMaps, 4>(a, s);
}

}  // namespace

template <typename T>
cudaError_t plain_attention(const MkbhGlobals& g, const MkbhLayer& L, T* out, int64_t ldo, cudaStream_t s) {
    PlainArgs<T> a{L, g.proj, pad8(L.in_rows), static_cast<const T*>(g.query), 0, {}, g.num_tokens, g.pos0, g.eps, out, ldo};
    if (L.mixer == MKBH_DIFF_ATTENTION) {
        const int rows = L.cache_keep + L.cache_ring, kw = L.kv_heads * 2 * L.dim, vw = L.kv_heads * L.vdim;
        a.src = {static_cast<const T*>(L.k_cache) + (size_t)g.slot * rows * kw, nullptr, static_cast<const T*>(L.v_cache) + (size_t)g.slot * rows * vw,
                 kw, 0, vw, 2 * L.dim, L.vdim, L.dim, 0, L.heads / L.kv_heads, L.cache_keep, L.cache_ring};
        return choose<T, 2>(a, s);
    }
    a.src = key_source<T>(g, L);
    a.ldq = pad8(L.heads * (a.src.split + a.src.rest));
    return choose<T, 1>(a, s);
}
template cudaError_t plain_attention<float>(const MkbhGlobals&, const MkbhLayer&, float*, int64_t, cudaStream_t);
template cudaError_t plain_attention<bf16>(const MkbhGlobals&, const MkbhLayer&, bf16*, int64_t, cudaStream_t);

}  // namespace mkbh
