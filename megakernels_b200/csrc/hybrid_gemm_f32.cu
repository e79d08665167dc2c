// 32-bit matrix product of the hybrid models' float build, on the 5th-generation tensor cores without giving up 32 bits.
//
// An operand is split into a tf32 part (11 bits, rounded to nearest) and the exact remainder, of which the tensor core reads
// another 11 bits: x y = h(x) h(y) + h(x) l(y) + l(x) h(y), what is left out below 2^-23 of |x y|.  The tensor core cuts where an FMA
// rounds (measured: 2^-24 of the sum per instruction of 8, always towards zero: 4.8e-6 over 2048 of the inner dimension), so
// the accumulators of the first products are added up in registers every 64 of it (2.2e-7; fp32 FMA in order: 8.1e-7);
// the other two products, 2^-11 as large, have an accumulator of their own that is read once.
// Bound by the hand-over between the warps that copy, split, multiply and add up: a step of 32 of the inner dimension takes 0.75 us with
// 160 tokens, of which the MMAs are 0.51 (0.67 if hardly anything is split, and 0.42 with 32 tokens).  300 x 8192 x 2048: 66 us, 152
// TFLOP/s, against 283 us with FMA; 20 x 2048 x 8192: 37 us.
// Features are the M side (128 a tile), tokens the N side (16 to 160), so that few tokens pad little; where tiles are
// few, a cluster of up to four CTAs shares a tile's inner dimension and adds the parts through distributed shared memory, always in
// the same order.  An operand that is infinite (or rounds to it) has no remainder: such a tile is done over with FMA.
// One or two tokens (the head): a warp per pair of features, bound by the weights' traffic.
#include "hybrid_kernels.h"
#include "hybrid_tcgen05.cuh"

namespace mkbh {
namespace {

constexpr int kFeatures = 128, kStep = 32, kChunk = 2;  // steps whose products one accumulator takes
constexpr int kSplitWarps = 6, kSumWarps = 8;
constexpr int kThreads = 32 * (2 + kSplitWarps + kSumWarps);

template <int NT>
struct GeoF {
    // Either part of the weights goes to tensor memory: shared memory's traffic is a third less (300 x 8192 x 2048: 80 us with
    // all four parts there, 67 without).  So a stage of weights is free again once it is split, one of tokens, split in
    // place, when the MMAs have read it; their remainders are there only in between.
    static constexpr int kW = kFeatures * kStep * 4, kX = NT * kStep * 4;
    static constexpr int kRests = 3, kWStages = NT <= 64 ? 8 : NT <= 96 ? 6 : 4;
    static constexpr int kRoom = (227 * 1024 - 2048 - kWStages * kW) / kX - kRests, kXStages = kRoom < 8 ? kRoom : 8;
    static constexpr int kTokens = kWStages * kW, kRest = kTokens + kXStages * kX, kBars = kRest + kRests * kX;
    static constexpr int kNumBars = 2 * kWStages + 3 * kXStages + kRests + 4;
    static constexpr int kCtl = kBars + kNumBars * 8;
    static constexpr int kAlloc = kCtl + 16 + 1024;
    // tensor memory: the sums of a chunk, two of them where there is room, the remainders', the weights' parts
    static constexpr int kSums = NT <= 96 ? 2 : 1, kWeights = (kSums + 1) * NT, kColumns = kWeights + kRests * 2 * kStep;
    static constexpr int kTmem = kColumns <= 256 ? 256 : 512;
    static constexpr int kPieces = kX / 16, kEach = (kW / 16 + kPieces + 32 * kSplitWarps - 1) / (32 * kSplitWarps);  // 16-byte pieces of tokens; of both per thread
    static constexpr int kByWeights = kEach > kStep / 4 ? (kEach - kStep / 4) * kFeatures : 0;  // of the tokens' pieces, by the warps that split weights
    static_assert(kAlloc <= 227 * 1024 && kColumns <= 512, "");
    static_assert(NT * kFeatures * 4 <= kBars, "the parts of a cluster's tile go where the ring was");
};

struct ShapeF {
    int T, N, K, tokens, token_tiles, parts;  // tokens of a tile (the rest of its NT are padding)
    unsigned long long timeout_ns;
    int* status;
    bool early;
};

__device__ __forceinline__ void mma_tf32(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d),
        "r"(a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
}
// sum[0 .. 7] += 8 columns of the warp's 32 lanes
__device__ __forceinline__ void add8(uint32_t addr, float* sum) {
    uint32_t r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(addr));
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7])::"memory");
#pragma unroll
    for (int j = 0; j < 8; ++j) sum[j] += __uint_as_float(r[j]);
}
__device__ __forceinline__ void add16(uint32_t addr, float* sum) {
    uint32_t r[16];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
                   "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(addr));
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]),
                   "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])::"memory");
#pragma unroll
    for (int j = 0; j < 16; ++j) sum[j] += __uint_as_float(r[j]);
}
template <int C>
__device__ __forceinline__ void add_columns(uint32_t addr, float (&sum)[C]) {
    if constexpr (C == 8) {
        add8(addr, sum);
    } else {
#pragma unroll
        for (int c = 0; c < C; c += 16) add16(addr + c, sum + c);
    }
}
// High part in place of x, remainder in r; `odd` turns to not-a-number with any remainder that is not finite.
__device__ __forceinline__ void split(float& x, float& r, float& odd) {
    const float h = __uint_as_float((__float_as_uint(x) + 0x1000u) & 0xffffe000u);
    r = x - h;
    x = h;
    odd = fmaf(r, 0.f, odd);
}
__device__ __forceinline__ void split4(float4& x, float4& r, float& odd) {
    split(x.x, r.x, odd);
    split(x.y, r.y, odd);
    split(x.z, r.z, odd);
    split(x.w, r.w, odd);
}
__device__ __forceinline__ bool infinite(float h) { return (__float_as_uint(h) & 0x7fffffffu) == 0x7f800000u; }
__device__ __forceinline__ bool infinite4(const float4& h) { return infinite(h.x) | infinite(h.y) | infinite(h.z) | infinite(h.w); }

// columns n (even) and n + 1 of token t
__device__ __forceinline__ void put(const GemmEpilogue& e, int t, int n, int N, float x, float y) {
    if (n >= N) return;
    if (e.what == Result::kGlu) {  // (N is even: both columns are there)
        static_cast<float*>(e.cast)[(size_t)t * e.ld + n / 2] = clamped_glu(x, y, e.limit, e.alpha);
        return;
    }
    float* o = (e.what == Result::kCast ? static_cast<float*>(e.cast) : e.out) + (size_t)t * e.ld + n;
    if (e.what == Result::kAdd) {
        o[0] = fmaf(e.scale ? e.scale[n] : 1.f, x, o[0]);
        if (n + 1 < N) o[1] = fmaf(e.scale ? e.scale[n + 1] : 1.f, y, o[1]);
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

// A thread's pieces first + thread, + kStride, .. below kEnd: read, or split and written back.
template <int kCount, int kStride, int kEnd, int kRegs>
__device__ __forceinline__ void split_pieces(float4* v, float4* rest, int thread, int first, float4 (&x)[kRegs], float& odd, bool read) {
#pragma unroll
    for (int j = 0; j < kCount; ++j) {
        const int i = first + thread + j * kStride;
        if (i >= kEnd) break;
        if (read) {
            x[j] = v[i];
        } else {
            float4 r;
            split4(x[j], r, odd);
            v[i] = x[j];
            rest[i] = r;
        }
    }
}

template <int kCount, int kStride, int kEnd, int kRegs>
__device__ __forceinline__ bool any_infinite(const float4 (&h)[kRegs], int thread, int first) {
    bool any = false;
#pragma unroll
    for (int j = 0; j < kCount; ++j)
        if (first + thread + j * kStride < kEnd) any |= infinite4(h[j]);
    return any;
}

// A cluster of s.parts CTAs per tile, tiles of the same features side by side.
template <int NT>
__global__ void __launch_bounds__(kThreads, 1) gemm_f32_kernel(const __grid_constant__ CUtensorMap wmap, const __grid_constant__ CUtensorMap amap,
                                                               const float* __restrict__ A, int64_t lda, const float* __restrict__ W, int64_t ldw,
                                                               const ShapeF s, const GemmEpilogue e) {
    using G = GeoF<NT>;
    extern __shared__ uint8_t raw[];
    const uint32_t raw32 = mkb::smem_u32(raw), base = (raw32 + 1023u) & ~1023u;
    uint8_t* gbase = raw + (base - raw32);
    volatile int* ctl = reinterpret_cast<volatile int*>(gbase + G::kCtl);  // [0] dead, [1] tensor-memory base, [2] infinite operands
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    auto bar = [&](int i) { return base + G::kBars + i * 8; };
    auto w_full = [&](int i) { return bar(i); };
    auto w_empty = [&](int i) { return bar(G::kWStages + i); };
    auto full = [&](int i) { return bar(2 * G::kWStages + i); };
    auto ready = [&](int i) { return bar(2 * G::kWStages + G::kXStages + i); };
    auto empty = [&](int i) { return bar(2 * G::kWStages + 2 * G::kXStages + i); };
    auto rest_empty = [&](int i) { return bar(2 * G::kWStages + 3 * G::kXStages + i); };
    auto acc_full = [&](int i) { return bar(2 * G::kWStages + 3 * G::kXStages + G::kRests + i); };
    auto acc_empty = [&](int i) { return bar(2 * G::kWStages + 3 * G::kXStages + G::kRests + 2 + i); };
    auto wait = [&](uint32_t b, int use, int role) { return tc_wait(b, use & 1u, ctl, s.timeout_ns, s.status, role); };
    if (threadIdx.x == 0) {
        for (int i = 0; i < G::kWStages; ++i) {
            mkb::mbar_init(w_full(i), 1);
            mkb::mbar_init(w_empty(i), 4);
        }
        for (int i = 0; i < G::kXStages; ++i) {
            mkb::mbar_init(full(i), 1);
            mkb::mbar_init(ready(i), kSplitWarps);
            mkb::mbar_init(empty(i), 1);
        }
        for (int i = 0; i < G::kRests; ++i) mkb::mbar_init(rest_empty(i), 1);
        for (int i = 0; i < 2; ++i) {
            mkb::mbar_init(acc_full(i), 1);
            mkb::mbar_init(acc_empty(i), kSumWarps);
        }
        ctl[0] = ctl[2] = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(base + G::kCtl + 4), "r"((uint32_t)G::kTmem) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_before_sync();
    __syncthreads();
    tc_after_sync();
    const uint32_t tmem = (uint32_t)ctl[1];
    let_next();
    if (warp != 0) after_previous();
    const int tile = blockIdx.x / s.parts, part = blockIdx.x % s.parts;
    const int t0 = (tile % s.token_tiles) * s.tokens, n0 = (tile / s.token_tiles) * kFeatures;
    const int steps_all = (s.K + kStep - 1) / kStep, first = steps_all * part / s.parts, steps = steps_all * (part + 1) / s.parts - first;
    const int chunks = (steps + kChunk - 1) / kChunk;
    constexpr int C = NT / 2;  // columns of a thread that sums

    if (warp == 0) {
        const bool chosen = tc_elect();
        bool ok = true;
        int it = 0;
        auto weights = [&](int i) {
            const uint32_t b = w_full(i % G::kWStages);
            mkb::mbar_expect_tx(b, G::kW);
            tc_tma_2d(base + i % G::kWStages * G::kW, &wmap, (first + i) * kStep, n0, b);
        };
        // a ring of weights is on its way while the launch before this one ends
        const int before = s.early ? min(steps, G::kWStages) : 0;
        if (chosen)
            for (int i = 0; i < before; ++i) weights(i);
        after_previous();
        for (; it < steps; ++it) {
            const int ws = it % G::kWStages, xs = it % G::kXStages;
            ok = __all_sync(0xffffffffu, wait(w_empty(ws), it / G::kWStages + 1, 0) && wait(empty(xs), it / G::kXStages + 1, 0));
            if (!ok) break;
            if (!chosen) continue;
            if (it >= before) weights(it);
            mkb::mbar_expect_tx(full(xs), G::kX);
            tc_tma_2d(base + G::kTokens + xs * G::kX, &amap, (first + it) * kStep, t0, full(xs));
        }
        // no copy may be in flight when the CTA's shared memory goes away
        for (int i = it > G::kXStages ? it - G::kXStages : 0; i < it; ++i) {
            if (ok) wait(empty(i % G::kXStages), i / G::kXStages, 0);
            else tc_wait(full(i % G::kXStages), (i / G::kXStages) & 1u, nullptr, s.timeout_ns, s.status, 0);
        }
        for (int i = it > G::kWStages ? it - G::kWStages : 0; i < it; ++i) {
            if (ok) wait(w_empty(i % G::kWStages), i / G::kWStages, 0);
            else tc_wait(w_full(i % G::kWStages), (i / G::kWStages) & 1u, nullptr, s.timeout_ns, s.status, 0);
        }
    } else if (warp == 1) {
        const bool chosen = tc_elect();
        // tf32 x tf32 -> fp32, both K-major
        const uint32_t idesc = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(NT >> 3) << 17) | ((uint32_t)(kFeatures >> 4) << 24);
        for (int it = 0; it < steps; ++it) {
            const int st = it % G::kXStages, chunk = it / kChunk, buf = chunk % G::kSums;
            bool ok = wait(ready(st), it / G::kXStages, 1);
            if (!__all_sync(0xffffffffu, ok)) break;
            tc_after_sync();
            const uint32_t xh = base + G::kTokens + st * G::kX, xl = base + G::kRest + it % G::kRests * G::kX;
            const uint32_t wh = tmem + G::kWeights + it % G::kRests * 2 * kStep, wl = wh + kStep;
            if (chosen) {
#pragma unroll
                for (int k = 0; k < kStep / 8; ++k) {
                    mma_tf32(tmem + G::kSums * NT, wl + k * 8, tc_desc(xh + k * 32), idesc, (uint32_t)((it | k) != 0));
                    mma_tf32(tmem + G::kSums * NT, wh + k * 8, tc_desc(xl + k * 32), idesc, 1u);
                }
            }
            // (meanwhile the sums of the chunk before are read)
            if (it % kChunk == 0) {
                ok = wait(acc_empty(buf), chunk / G::kSums + 1, 1);
                if (!__all_sync(0xffffffffu, ok)) break;
                tc_after_sync();
            }
            if (!chosen) continue;
#pragma unroll
            for (int k = 0; k < kStep / 8; ++k)
                mma_tf32(tmem + buf * NT, wh + k * 8, tc_desc(xh + k * 32), idesc, (uint32_t)((it % kChunk | k) != 0));
            tc_commit(empty(st));
            tc_commit(rest_empty(it % G::kRests));
            if (it % kChunk == kChunk - 1 || it == steps - 1) tc_commit(acc_full(buf));
        }
    } else if (warp < 2 + kSplitWarps) {
        // warps 2 .. 5: 32 rows of weights each (the quarter of tensor memory's lanes a warp may write) and some of the tokens
        const bool weights = warp < 6;
        float odd = 0.f;
        for (int it = 0; it < steps; ++it) {
            const int st = it % G::kXStages, rs = it % G::kRests, ws = it % G::kWStages;
            const bool ok = (!weights || wait(w_full(ws), it / G::kWStages, 2)) && wait(full(st), it / G::kXStages, 2) &&
                            wait(rest_empty(rs), it / G::kRests + 1, 2);
            if (!__all_sync(0xffffffffu, ok)) break;
            float4 *v = reinterpret_cast<float4*>(gbase + G::kTokens + st * G::kX), *rest = reinterpret_cast<float4*>(gbase + G::kRest + rs * G::kX);
            // everything is read before anything is written, so that the reads are on their way together
            if (weights) {
                const int q = warp & 3, row = q * 32 + lane;
                const float4* w = reinterpret_cast<const float4*>(gbase + ws * G::kW + row * 128);
                const uint32_t to = tmem + ((uint32_t)(q * 32) << 16) + G::kWeights + rs * 2 * kStep;
                float4 x[8], y[G::kByWeights / kFeatures + 1];
#pragma unroll
                for (int c = 0; c < 8; ++c) x[c] = w[c ^ (row & 7)];  // (the copy's swizzle)
                split_pieces<G::kByWeights / kFeatures, kFeatures, G::kByWeights>(v, rest, threadIdx.x - 64, 0, y, odd, true);
                __syncwarp();
                if (lane == 0) mkb::mbar_arrive(w_empty(ws));
                tc_after_sync();
#pragma unroll
                for (int c = 0; c < 8; c += 4) {
                    uint32_t hi[16], lo[16];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        float4 r;
                        split4(x[c + j], r, odd);
                        hi[4 * j] = __float_as_uint(x[c + j].x), hi[4 * j + 1] = __float_as_uint(x[c + j].y);
                        hi[4 * j + 2] = __float_as_uint(x[c + j].z), hi[4 * j + 3] = __float_as_uint(x[c + j].w);
                        lo[4 * j] = __float_as_uint(r.x), lo[4 * j + 1] = __float_as_uint(r.y);
                        lo[4 * j + 2] = __float_as_uint(r.z), lo[4 * j + 3] = __float_as_uint(r.w);
                    }
                    tc_store16(to + 4 * c, hi);
                    tc_store16(to + kStep + 4 * c, lo);
                }
                split_pieces<G::kByWeights / kFeatures, kFeatures, G::kByWeights>(v, rest, threadIdx.x - 64, 0, y, odd, false);
                if (odd != odd) {  // (rare: is it an infinite operand, which has no remainder?)
                    bool any = any_infinite<G::kByWeights / kFeatures, kFeatures, G::kByWeights>(y, threadIdx.x - 64, 0);
#pragma unroll
                    for (int c = 0; c < 8; ++c) any |= infinite4(x[c]);
                    if (any) ctl[2] = 1;
                }
                tc_stored();
                tc_before_sync();
            } else {
                constexpr int kCount = (G::kPieces - G::kByWeights + 63) / 64;
                float4 y[kCount];
                split_pieces<kCount, 64, G::kPieces>(v, rest, threadIdx.x - 192, G::kByWeights, y, odd, true);
                split_pieces<kCount, 64, G::kPieces>(v, rest, threadIdx.x - 192, G::kByWeights, y, odd, false);
                if (odd != odd && any_infinite<kCount, 64, G::kPieces>(y, threadIdx.x - 192, G::kByWeights)) ctl[2] = 1;
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mkb::mbar_arrive(ready(st));
        }
    } else {
        const int q = warp & 3, half = (warp - 2 - kSplitWarps) >> 2;  // the quarter of tensor memory's lanes this warp may read
        const uint32_t at = tmem + ((uint32_t)(q * 32) << 16) + half * C;
        float sum[C] = {};
        bool ok = true;
        for (int chunk = 0; chunk < chunks; ++chunk) {
            const int buf = chunk % G::kSums;
            ok = __all_sync(0xffffffffu, wait(acc_full(buf), chunk / G::kSums, 3));
            if (!ok) break;
            tc_after_sync();
            add_columns<C>(at + buf * NT, sum);
            tc_before_sync();
            __syncwarp();
            if (lane == 0) mkb::mbar_arrive(acc_empty(buf));
        }
        if (ok) {
            add_columns<C>(at + G::kSums * NT, sum);  // (the last commit covers these too)
            // the ring's stages have been read: [token][feature], for the loop below (unrolled from registers, with its kinds of
            // results, it was 100 KB of code)
            float* o = reinterpret_cast<float*>(gbase) + half * C * kFeatures + q * 32 + lane;
#pragma unroll
            for (int j = 0; j < C; ++j) o[j * kFeatures] = sum[j];
        }
    }
    tc_before_sync();
    __syncthreads();
    if (*ctl) tc_settle();
    const int tokens = min(s.tokens, s.T - t0), c = 4 * lane;
    if (ctl[2]) {  // (behind the block's barrier: whichever warp found the operand)
        const int last = min(s.K, (first + steps) * kStep);
        for (int i = warp; i < tokens * kFeatures; i += kThreads / 32) {  // an element per warp, with FMA
            const int t = i / kFeatures, n = i % kFeatures;
            if (n0 + n >= s.N) continue;
            const float *w = W + (size_t)(n0 + n) * ldw, *v = A + (size_t)(t0 + t) * lda;
            float x = 0.f;
#pragma unroll 4
            for (int k = first * kStep + 4 * lane; k < last; k += 128) {
                const float4 a = slice(w, true, k, last), b = slice(v, true, k, last);
                x = fmaf(a.x, b.x, fmaf(a.y, b.y, fmaf(a.z, b.z, fmaf(a.w, b.w, x))));
            }
            x = warp_sum(x);
            if (lane == 0) reinterpret_cast<float*>(gbase)[t * kFeatures + n] = x;
        }
        __syncthreads();
    }
    if (s.parts > 1) tc_cluster_sync();
#pragma unroll 2
    for (int t = part + s.parts * warp; t < tokens; t += s.parts * (kThreads / 32)) {
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
        if (s.parts == 1) {
            x = *reinterpret_cast<const float4*>(gbase + (t * kFeatures + c) * 4);
        } else {
            for (int z = 0; z < s.parts; ++z) {
                const uint32_t at = tc_peer(base + (uint32_t)(t * kFeatures + c) * 4, z);
                const float2 u = tc_peer_load2(at), v = tc_peer_load2(at + 8);
                x.x += u.x, x.y += u.y, x.z += v.x, x.w += v.y;
            }
        }
        put(e, t0 + t, n0 + c, s.N, x.x, x.y);
        put(e, t0 + t, n0 + c + 2, s.N, x.z, x.w);
    }
    if (s.parts > 1) tc_cluster_sync();
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)G::kTmem) : "memory");
}

template <int NT>
cudaError_t launch(const float* A, int64_t lda, const float* W, int64_t ldw, ShapeF s, const GemmEpilogue& e, cudaStream_t st) {
    using G = GeoF<NT>;
    static bool set[64] = {};
    int dev = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err != cudaSuccess) return err;
    if (!set[dev & 63]) {
        err = cudaFuncSetAttribute(gemm_f32_kernel<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, G::kAlloc);
        if (err != cudaSuccess) return err;
        set[dev & 63] = true;
    }
    CUtensorMap wmap, amap;
    if ((err = tc_map(&wmap, W, s.K, s.N, ldw, kStep, kFeatures)) != cudaSuccess) return err;
    if ((err = tc_map(&amap, A, s.K, s.T, lda, kStep, NT)) != cudaSuccess) return err;
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3(s.token_tiles * ((s.N + kFeatures - 1) / kFeatures) * s.parts);
    c.blockDim = dim3(kThreads);
    c.dynamicSmemBytes = G::kAlloc;
    c.stream = st;
    cudaLaunchAttribute attrs[2] = {may_begin_early()};
    attrs[1].id = cudaLaunchAttributeClusterDimension;
    attrs[1].val.clusterDim.x = s.parts;
    attrs[1].val.clusterDim.y = attrs[1].val.clusterDim.z = 1;
    c.attrs = attrs;
    c.numAttrs = s.parts > 1 ? 2 : 1;
    return cudaLaunchKernelEx(&c, gemm_f32_kernel<NT>, wmap, amap, A, lda, W, ldw, s, e);
}

}  // namespace

cudaError_t gemm_f32(const float* A, int64_t lda, const float* W, int64_t ldw, int T, int N, int K,
                     const GemmEpilogue& e, int* status, cudaStream_t st, unsigned long long timeout_ns, bool early) {
    if (T <= 2) {
        const int blocks = (N + 15) / 16;
        if (T == 1) gemv_f32_kernel<1><<<blocks, 256, 0, st>>>(A, lda, W, ldw, N, K, e);
        else gemv_f32_kernel<2><<<blocks, 256, 0, st>>>(A, lda, W, ldw, N, K, e);
        return cudaGetLastError();
    }
    int sms = 0;
    if (const cudaError_t err = sm_count(&sms); err != cudaSuccess) return err;
    // Tokens of a tile and CTAs on it: waves of tiles, each so many steps (in cycles, as measured) and a beginning
    // and an end of its own; a cluster's exchange besides.  Clusters of eight wait for whole groups of SMs (20 x 2048 x 8192: 57 us, four
    // 49 us, when a step took as long).
    const int widths[] = {16, 32, 64, 96, 128, 160}, steps = (K + kStep - 1) / kStep, rows = (N + kFeatures - 1) / kFeatures;
    ShapeF s{T, N, K, 0, 0, 1, timeout_ns, status, early};
    int width = 0;
    float least = 0.f;
    for (int w : widths) {
        const int tiles = (T + w - 1) / w;
        for (int p = 1; p <= 4 && (p == 1 || steps >= 4 * p); p *= 2) {
            const int waves = (tiles * rows * p + sms - 1) / sms;
            if (p > 1 && waves > 1) break;
            const float t = waves * ((steps + p - 1) / p * (700.f + 4.6f * w) + 8000.f) + (p > 1 ? 4000.f + 20.f * w : 0.f);
            if (width == 0 || t < least) {
                least = t;
                width = w;
                s.parts = p;
                s.token_tiles = tiles;
            }
        }
    }
    s.tokens = (T + s.token_tiles - 1) / s.token_tiles;  // (even tiles; at most `width`)
    switch (width) {
        case 16: return launch<16>(A, lda, W, ldw, s, e, st);
        case 32: return launch<32>(A, lda, W, ldw, s, e, st);
        case 64: return launch<64>(A, lda, W, ldw, s, e, st);
        case 96: return launch<96>(A, lda, W, ldw, s, e, st);
        case 128: return launch<128>(A, lda, W, ldw, s, e, st);
        default: return launch<160>(A, lda, W, ldw, s, e, st);
    }
}

}  // namespace mkbh
