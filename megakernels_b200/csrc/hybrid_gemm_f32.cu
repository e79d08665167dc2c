// 32-bit matrix product of the hybrid models' float build (true fp32 FMA, no reduced-precision matrix mode).
//
// Bound by the FMA rate (74 TFLOP/s at 1.96 GHz) and by shared-memory reads, four cycles per 16-byte read of a warp (300 x
// 8192 x 2048: 283 us, 36 TFLOP/s; 388 us with 64 x 64 tiles of 4 x 4 outputs): tiles of 16, 32 or 64 tokens x 128 features, 128 threads with up to
// 8 x 8 outputs each, two neighbouring features per instruction (fma.rn.f32x2, rounded like two fmaf), so that issue
// slots are left for the shared-memory reads; the next slice of operands is in registers while this one is multiplied.
// Where the tiles do not fill the SMs evenly, a cluster of up to eight CTAs shares a tile's inner dimension and adds
// the partial tiles through distributed shared memory, always in the same order.
// One or two tokens (the head): a warp per pair of features, bound by the weights' traffic.
#include "hybrid_kernels.h"

namespace mkbh {
namespace {

constexpr int kCols = 128, kDepth = 16, kThreads = 128;
constexpr int kColStride = kCols + 4;

__device__ __forceinline__ uint64_t twice(float x) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ void fma2(uint64_t& d, uint64_t a, uint64_t b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b)); }
__device__ __forceinline__ float2 both(uint64_t x) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(x));
    return r;
}

// columns n (even) and n + 1 of token t
__device__ __forceinline__ void put(const GemmEpilogue& e, int t, int n, int N, float x, float y) {
    if (n >= N) return;
    if (e.what == Result::kGlu) {  // (N is even: both columns are there)
        static_cast<float*>(e.cast)[(size_t)t * e.ld + n / 2] = clamped_glu(x, y, e.limit, e.alpha);
        return;
    }
    float* o = (e.what == Result::kCast ? static_cast<float*>(e.cast) : e.out) + (size_t)t * e.ld + n;
    if (e.what == Result::kAdd) {
        o[0] += (e.scale ? e.scale[n] : 1.f) * x;
        if (n + 1 < N) o[1] += (e.scale ? e.scale[n + 1] : 1.f) * y;
    } else {
        o[0] = x + (e.bias ? e.bias[n] : 0.f);
        if (n + 1 < N) o[1] = y + (e.bias ? e.bias[n + 1] : 0.f);
    }
}

// Four columns from k0 + c on of a row, zero beyond `limit` (rows are padded to 8: what lies beyond may be read).
__device__ __forceinline__ float4 slice(const float* row, bool live, int k, int limit) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (live && k < limit) {
        v = *reinterpret_cast<const float4*>(row + k);
        if (k + 1 >= limit) v.y = 0.f;
        if (k + 2 >= limit) v.z = 0.f;
        if (k + 3 >= limit) v.w = 0.f;
    }
    return v;
}

// R rows of tokens per thread; grid (features, tokens, clusters of gridDim.z)
template <int R>
__global__ void __launch_bounds__(kThreads, R == 8 ? 4 : 5)
gemm_f32_kernel(const float* __restrict__ A, int64_t lda, const float* __restrict__ W, int64_t ldw, int T, int N, int K, int per,
                const GemmEpilogue e) {
    constexpr int kRows = 8 * R, kRowStride = kRows + 4, kBuffer = kDepth * (kRowStride + kColStride);
    constexpr int kLoadsA = kRows * kDepth / 4 / kThreads > 0 ? kRows * kDepth / 4 / kThreads : 1, kLoadsW = kCols * kDepth / 4 / kThreads;
    constexpr int kFloats = 2 * kBuffer > kRows * kColStride ? 2 * kBuffer : kRows * kColStride;
    __shared__ __align__(16) float sm[kFloats];
    const int n0 = blockIdx.x * kCols, t0 = blockIdx.y * kRows, tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4, lr = tid >> 2, lc = (tid & 3) * 4;
    const int first = blockIdx.z * per, last = min(K, first + per);  // this CTA's part of the inner dimension
    uint64_t acc[R][4] = {};
    float4 a[kLoadsA], w[kLoadsW];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int i = 0; i < kLoadsA; ++i) {
            const int r = lr + 32 * i;
            a[i] = slice(A + (size_t)(t0 + r) * lda, r < kRows && t0 + r < T, k0 + lc, last);
        }
#pragma unroll
        for (int i = 0; i < kLoadsW; ++i) {
            const int r = lr + 32 * i;
            w[i] = slice(W + (size_t)(n0 + r) * ldw, n0 + r < N, k0 + lc, last);
        }
    };
    auto keep = [&](float* b) {
        float *sa = b, *sw = b + kDepth * kRowStride;
#pragma unroll
        for (int i = 0; i < kLoadsA; ++i) {
            const int r = lr + 32 * i;
            if (r >= kRows) break;
            sa[lc * kRowStride + r] = a[i].x; sa[(lc + 1) * kRowStride + r] = a[i].y;
            sa[(lc + 2) * kRowStride + r] = a[i].z; sa[(lc + 3) * kRowStride + r] = a[i].w;
        }
#pragma unroll
        for (int i = 0; i < kLoadsW; ++i) {
            const int r = lr + 32 * i;
            sw[lc * kColStride + r] = w[i].x; sw[(lc + 1) * kColStride + r] = w[i].y;
            sw[(lc + 2) * kColStride + r] = w[i].z; sw[(lc + 3) * kColStride + r] = w[i].w;
        }
    };
    fetch(first);
    keep(sm);
    __syncthreads();
    int buf = 0;
    for (int k0 = first; k0 < last; k0 += kDepth, buf ^= 1) {
        const bool more = k0 + kDepth < last;
        if (more) fetch(k0 + kDepth);
        const float *sa = sm + buf * kBuffer, *sw = sa + kDepth * kRowStride;
#pragma unroll
        for (int k = 0; k < kDepth; ++k) {
            float x[R];
            if constexpr (R == 2) {
                const float2 v = *reinterpret_cast<const float2*>(sa + k * kRowStride + ty * 2);
                x[0] = v.x; x[1] = v.y;
            } else {
#pragma unroll
                for (int i = 0; i < R / 4; ++i) {
                    const float4 v = *reinterpret_cast<const float4*>(sa + k * kRowStride + 32 * i + ty * 4);
                    x[4 * i] = v.x; x[4 * i + 1] = v.y; x[4 * i + 2] = v.z; x[4 * i + 3] = v.w;
                }
            }
            const ulonglong2 u = *reinterpret_cast<const ulonglong2*>(sw + k * kColStride + tx * 4);
            const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(sw + k * kColStride + 64 + tx * 4);
#pragma unroll
            for (int i = 0; i < R; ++i) {
                const uint64_t f = twice(x[i]);
                fma2(acc[i][0], f, u.x);
                fma2(acc[i][1], f, u.y);
                fma2(acc[i][2], f, v.x);
                fma2(acc[i][3], f, v.y);
            }
        }
        if (more) keep(sm + (buf ^ 1) * kBuffer);  // (that buffer was read before the last barrier)
        __syncthreads();
    }
    const auto row_of = [&](int i) { return R == 2 ? ty * 2 + i : (i / 4) * 32 + ty * 4 + i % 4; };
    const auto col_of = [&](int j) { return (j / 2) * 64 + tx * 4 + (j % 2) * 2; };
    if (gridDim.z == 1) {
#pragma unroll
        for (int i = 0; i < R; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float2 v = both(acc[i][j]);
                if (t0 + row_of(i) < T) put(e, t0 + row_of(i), n0 + col_of(j), N, v.x, v.y);
            }
        return;
    }
    // partial tiles side by side in the cluster; every CTA adds up its share of the rows, in the CTAs' order
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) *reinterpret_cast<uint64_t*>(sm + row_of(i) * kColStride + col_of(j)) = acc[i][j];
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    const uint32_t base = mkb::smem_u32(sm);
    const int parts = gridDim.z, rows = min(kRows, T - t0);
    for (int r = blockIdx.z + parts * (tid >> 6); r < rows; r += parts * (kThreads / 64)) {
        const int c = 2 * (tid & 63);
        float x = 0.f, y = 0.f;
        for (int z = 0; z < parts; ++z) {
            uint32_t at;
            float px, py;
            asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(base + (uint32_t)(r * kColStride + c) * 4), "r"(z));
            asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(px), "=f"(py) : "r"(at) : "memory");
            x += px;
            y += py;
        }
        put(e, t0 + r, n0 + c, N, x, y);
    }
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// A pair of features per warp, B tokens.
template <int B>
__global__ void __launch_bounds__(256) gemv_f32_kernel(const float* __restrict__ A, int64_t lda, const float* __restrict__ W, int64_t ldw, int N,
                                                       int K, const GemmEpilogue e) {
    const int n = 2 * (blockIdx.x * 8 + (threadIdx.x >> 5)), lane = threadIdx.x & 31;
    if (n >= N) return;
    const float *w0 = W + (size_t)n * ldw, *w1 = n + 1 < N ? w0 + ldw : w0;
    float s[2][B] = {};
#pragma unroll 4
    for (int k = 4 * lane; k < K; k += 128) {
        const float4 u = slice(w0, true, k, K), v = slice(w1, true, k, K);
#pragma unroll
        for (int b = 0; b < B; ++b) {
            const float4 x = slice(A + b * lda, true, k, K);
            s[0][b] = fmaf(u.x, x.x, fmaf(u.y, x.y, fmaf(u.z, x.z, fmaf(u.w, x.w, s[0][b]))));
            s[1][b] = fmaf(v.x, x.x, fmaf(v.y, x.y, fmaf(v.z, x.z, fmaf(v.w, x.w, s[1][b]))));
        }
    }
#pragma unroll
    for (int b = 0; b < B; ++b) {
        const float x = warp_sum(s[0][b]), y = warp_sum(s[1][b]);
        if (lane == 0) put(e, b, n, N, x, y);
    }
}

template <int R>
cudaError_t launch(const float* A, int64_t lda, const float* W, int64_t ldw, int T, int N, int K, const GemmEpilogue& e, int parts, cudaStream_t s) {
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3((N + kCols - 1) / kCols, (T + 8 * R - 1) / (8 * R), parts);
    c.blockDim = dim3(kThreads);
    c.stream = s;
    cudaLaunchAttribute cluster;
    cluster.id = cudaLaunchAttributeClusterDimension;
    cluster.val.clusterDim.x = cluster.val.clusterDim.y = 1;
    cluster.val.clusterDim.z = parts;
    c.attrs = &cluster;
    c.numAttrs = parts > 1 ? 1 : 0;
    const int per = ((K + parts - 1) / parts + kDepth - 1) / kDepth * kDepth;
    return cudaLaunchKernelEx(&c, gemm_f32_kernel<R>, A, lda, W, ldw, T, N, K, per, e);
}

}  // namespace

cudaError_t gemm_f32(const float* A, int64_t lda, const float* W, int64_t ldw, int T, int N, int K,
                     const GemmEpilogue& e, cudaStream_t s) {
    if (T <= 2) {
        const int blocks = (N + 15) / 16;
        if (T == 1) gemv_f32_kernel<1><<<blocks, 256, 0, s>>>(A, lda, W, ldw, N, K, e);
        else gemv_f32_kernel<2><<<blocks, 256, 0, s>>>(A, lda, W, ldw, N, K, e);
        return cudaGetLastError();
    }
    int sms = 0;
    if (const cudaError_t err = sm_count(&sms); err != cudaSuccess) return err;
    const int rows = T <= 16 ? 16 : T <= 32 ? 32 : 64, tiles = ((T + rows - 1) / rows) * ((N + kCols - 1) / kCols);
    // An SM works off its CTAs at one rate: the share of the inner dimension that leaves the fullest SM the least
    // work, a share's own cost (filling the pipeline, the exchange) counted as 64 of the inner dimension.
    int parts = 1;
    float least = 0.f;
    for (int p = 1; p <= 8; p *= 2) {
        if (p > 1 && K < p * 8 * kDepth) break;
        const float t = (float)((tiles * p + sms - 1) / sms) * ((float)K / p + 64.f);
        if (p == 1 || t < least) least = t, parts = p;
    }
    return rows == 16 ? launch<2>(A, lda, W, ldw, T, N, K, e, parts, s) : rows == 32 ? launch<4>(A, lda, W, ldw, T, N, K, e, parts, s)
                                                                       : launch<8>(A, lda, W, ldw, T, N, K, e, parts, s);
}

}  // namespace mkbh
