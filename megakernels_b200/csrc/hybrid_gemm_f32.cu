// 32-bit matrix product of the hybrid models' float build, on the 5th-generation tensor cores without giving up 32 bits.
//
// An operand is three bf16 parts, each what the parts before it leave, rounded to nearest (Henry, Tang, Heinecke, "Leveraging the bfloat16
// Artificial Intelligence Datatype For Higher-Precision Computations", 2019): together they are all of its 24 bits.  Six of the nine products of
// parts are formed; the others are 2^-24 of |x y| together at most.  The tensor core cuts a sum where an FMA rounds it, by up to 2^-23 of its size per
// instruction: the five small products of a step of 32 of the inner dimension go first, while the sum is small, and every step's sum
// is added up in registers, rounded to nearest.  Relative error against 64 bits (2-norm; FMA in order in the same tiles): N(0, 1) operands, inner
// dimension 64: 6.4e-8 (1.4e-7), 2048: 1.0e-7 (2.9e-7); of one sign 6.4e-8 (1.1e-7) and 7.0e-8 (9.0e-8); nowhere above it
// at 102 points of 1 to 8192, six distributions.  (Two tf32 parts lose a bit of every operand and drop 2^-22: 2.0e-7 and 2.1e-7, 2.7e-7 and 2.7e-7.)
// Below 16 FMA in order is no further off: a kernel of its own.  Parts of operands below 2^-109 are cut at 2^-133: error 8e-8 down to 2^-108,
// 2e-6 at 2^-116, where FMA keeps what a subnormal holds.
// Bound by the hand-over between the warps that copy, split, multiply and add up; the MMAs of a step of 160 tokens alone take 980
// cycles, 80 each.  300 x 8192 x 2048: 72 us, 140 TFLOP/s; 283 us with FMA, 68 us as two tf32 parts.  (Six warps that split both operands, tokens'
// parts exchanged by shuffles, 170 cycles per 16 bytes: 98 us; six warps for tokens instead of four: 75 us.)
// Features are the M side (128 a tile), tokens the N side (16 to 160), so that few tokens pad little; where tiles are
// few, a cluster of up to four CTAs shares a tile's inner dimension and adds the parts through distributed shared memory, always in
// the same order.  An operand that is infinite (or rounds to it) has no parts: its token's or feature's sums are done over with FMA.
// One or two tokens (the head): a warp per pair of features, bound by the weights' traffic.
#include "hybrid_kernels.h"
#include "hybrid_tcgen05.cuh"

namespace mkbh {
namespace {

constexpr int kFeatures = 128, kStep = 32;
constexpr int kWeightWarps = 4, kTokenWarps = 4, kSumWarps = 8;
constexpr int kThreads = 32 * (2 + kWeightWarps + kTokenWarps + kSumWarps);
constexpr int kDeep = 4;            // steps whose parts are there at a time
constexpr int kPartColumns = 3 * kStep / 2;

template <int NT>
struct GeoF {
    // The parts of the weights go to tensor memory, so that shared memory's traffic is a third less.  A stage of weights is free
    // again once it is split, one of tokens when the MMAs have read it: its first two parts take its place, row by row
    // [first | second], the third parts of two steps share the rows of a tile of their own.
    static constexpr int kW = kFeatures * kStep * 4, kX = NT * kStep * 4;
    static constexpr int kWStages = NT <= 64 ? 8 : NT <= 96 ? 6 : 4;
    static constexpr int kRoom = (227 * 1024 - 2048 - kWStages * kW) / kX - kDeep / 2, kXStages = kRoom < 8 ? kRoom : 8;
    static constexpr int kTokens = kWStages * kW, kRest = kTokens + kXStages * kX, kBars = kRest + kDeep / 2 * kX;
    static constexpr int kNumBars = 2 * kWStages + 3 * kXStages + kDeep + 4;
    static constexpr int kCtl = kBars + kNumBars * 8;  // control words, then which tokens and features have infinite operands
    static constexpr int kAlloc = kCtl + (4 + 8 + 4) * 4 + 1024;
    // tensor memory: the sums of two steps, the weights' parts
    static constexpr int kWeights = 2 * NT, kColumns = kWeights + kDeep * kPartColumns;
    static constexpr int kTmem = kColumns <= 256 ? 256 : 512;
    static_assert(kAlloc <= 227 * 1024 && kColumns <= 512 && kXStages >= kWStages && kDeep % 2 == 0, "");
    static_assert(NT * kFeatures * 4 <= kBars, "the parts of a cluster's tile go where the ring was");
};

struct ShapeF {
    int T, N, K, tokens, token_tiles, parts;  // tokens of a tile (the rest of its NT are padding)
    unsigned long long timeout_ns;
    int* status;
    bool early;
};

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
// The parts of x and y, packed; an entry of `odd` turns to not-a-number if one is infinite, rounds to infinity or is no number.
__device__ __forceinline__ uint64_t pair(uint32_t lo, uint32_t hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi));
    return r;
}
__device__ __forceinline__ float2 both(uint64_t x) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(x));
    return r;
}
__device__ __forceinline__ uint32_t take_part(uint64_t& v) {  // (what is left is exact)
    const float2 f = both(v);
    const uint32_t p = mkb::pack_bf16x2(f.x, f.y);
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(v) : "l"(pair(p << 16, p & 0xffff0000u)), "l"(pair(0xbf800000u, 0xbf800000u)));
    return p;
}
__device__ __forceinline__ void split2(float x, float y, uint32_t& p1, uint32_t& p2, uint32_t& p3, uint32_t& odd) {
    uint64_t v = pair(__float_as_uint(x), __float_as_uint(y));
    p1 = take_part(v);
    p2 = take_part(v);
    const float2 f = both(v);
    p3 = mkb::pack_bf16x2(f.x, f.y);
    asm("fma.rn.bf16x2 %0, %1, %2, %0;" : "+r"(odd) : "r"(p3), "r"(0));
}
__device__ __forceinline__ bool infinite(float x) { return (__float_as_uint(x) & 0x7fffffffu) - 0x7f7f8000u <= 0x8000u; }  // or rounds to it
__device__ __forceinline__ bool infinite4(const float4& x) { return infinite(x.x) | infinite(x.y) | infinite(x.z) | infinite(x.w); }

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

// Inner dimensions below kShort, where a sum that is cut is further off than FMA (of one sign, 8: 5.7e-8, FMA 4.7e-8; 16: 6.0e-8, 6.4e-8): two
// features and kFmaTokens tokens per thread, FMA in order.
constexpr int kShort = 16, kFmaTokens = 8;
__global__ void __launch_bounds__(256) fma_f32_kernel(const float* __restrict__ A, int64_t lda, const float* __restrict__ W, int64_t ldw, int T, int N, int K,
                                                      const GemmEpilogue e) {
    const int n = 2 * (blockIdx.x * 256 + threadIdx.x), t0 = blockIdx.y * kFmaTokens;
    const float *w0 = W + (size_t)min(n, N - 1) * ldw, *w1 = W + (size_t)min(n + 1, N - 1) * ldw;
    float2 sum[kFmaTokens] = {};
    for (int k = 0; k < K; ++k) {
        const float x = w0[k], y = w1[k];
#pragma unroll
        for (int j = 0; j < kFmaTokens; ++j) {
            const float a = A[(size_t)min(t0 + j, T - 1) * lda + k];
            sum[j].x = fmaf(x, a, sum[j].x);
            sum[j].y = fmaf(y, a, sum[j].y);
        }
    }
#pragma unroll
    for (int j = 0; j < kFmaTokens; ++j)
        if (t0 + j < T) put(e, t0 + j, n, N, sum[j].x, sum[j].y);
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
    volatile int* ctl = reinterpret_cast<volatile int*>(gbase + G::kCtl);  // [0] dead, [1] tensor-memory base
    uint32_t* flags = reinterpret_cast<uint32_t*>(gbase + G::kCtl) + 4;  // tokens, then features, with an infinite operand
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    auto bar = [&](int i) { return base + G::kBars + i * 8; };
    auto w_full = [&](int i) { return bar(i); };
    auto w_empty = [&](int i) { return bar(G::kWStages + i); };
    auto full = [&](int i) { return bar(2 * G::kWStages + i); };
    auto ready = [&](int i) { return bar(2 * G::kWStages + G::kXStages + i); };
    auto empty = [&](int i) { return bar(2 * G::kWStages + 2 * G::kXStages + i); };
    auto rest_empty = [&](int i) { return bar(2 * G::kWStages + 3 * G::kXStages + i); };
    auto acc_full = [&](int i) { return bar(2 * G::kWStages + 3 * G::kXStages + kDeep + i); };
    auto acc_empty = [&](int i) { return bar(2 * G::kWStages + 3 * G::kXStages + kDeep + 2 + i); };
    auto wait = [&](uint32_t b, int use, int role) { return tc_wait(b, use & 1u, ctl, s.timeout_ns, s.status, role); };
    if (threadIdx.x == 0) {
        for (int i = 0; i < G::kWStages; ++i) {
            mkb::mbar_init(w_full(i), 1);
            mkb::mbar_init(w_empty(i), 4);
        }
        for (int i = 0; i < G::kXStages; ++i) {
            mkb::mbar_init(full(i), 1);
            mkb::mbar_init(ready(i), kWeightWarps + kTokenWarps);
            mkb::mbar_init(empty(i), 1);
        }
        for (int i = 0; i < kDeep; ++i) mkb::mbar_init(rest_empty(i), 1);
        for (int i = 0; i < 2; ++i) {
            mkb::mbar_init(acc_full(i), 1);
            mkb::mbar_init(acc_empty(i), kSumWarps);
        }
        ctl[0] = 0;
        for (int i = 0; i < 12; ++i) flags[i] = 0;
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
        if (it < before) it = before;  // (weights that were read early)
        for (int i = it > G::kWStages ? it - G::kWStages : 0; i < it; ++i) {
            if (ok) wait(w_empty(i % G::kWStages), i / G::kWStages, 0);
            else tc_wait(w_full(i % G::kWStages), (i / G::kWStages) & 1u, nullptr, s.timeout_ns, s.status, 0);
        }
    } else if (warp == 1) {
        const bool chosen = tc_elect();
        const uint32_t idesc = tc_idesc(kFeatures, NT);
        for (int it = 0; it < steps; ++it) {
            const uint32_t sums = tmem + (it & 1) * NT;
            const bool ok = wait(acc_empty(it & 1), it / 2 + 1, 1) && wait(ready(it % G::kXStages), it / G::kXStages, 1);
            if (!__all_sync(0xffffffffu, ok)) break;
            tc_after_sync();
            if (!chosen) continue;
            const uint32_t x = base + G::kTokens + it % G::kXStages * G::kX, rest = base + G::kRest + it % kDeep / 2 * G::kX + (it & 1) * 64;
            const uint32_t w = tmem + G::kWeights + it % kDeep * kPartColumns;
            // what is small is added first, before the sum has a size that it could be cut at
            constexpr int kParts[6][2] = {{1, 1}, {2, 0}, {0, 2}, {1, 0}, {0, 1}, {0, 0}};  // of weights, of tokens
#pragma unroll
            for (int i = 0; i < 6; ++i)
#pragma unroll
                for (int k = 0; k < kStep / 16; ++k)
                    tc_mma_ts(sums, w + k * 24 + kParts[i][0] * 8, tc_desc((kParts[i][1] < 2 ? x + kParts[i][1] * 64 : rest) + k * 32), idesc, (uint32_t)((i | k) != 0));
            tc_commit(empty(it % G::kXStages));
            tc_commit(rest_empty(it % kDeep));
            tc_commit(acc_full(it & 1));
        }
    } else if (warp < 2 + kWeightWarps + kTokenWarps) {
        const bool weights = warp < 2 + kWeightWarps;
        uint32_t odd = 0;
        for (int it = 0; it < steps; ++it) {
            const int st = it % G::kXStages, rs = it % kDeep, ws = it % G::kWStages;
            const bool ok = (weights ? wait(w_full(ws), it / G::kWStages, 2) : wait(full(st), it / G::kXStages, 2)) && wait(rest_empty(rs), it / kDeep + 1, 2);
            if (!__all_sync(0xffffffffu, ok)) break;
            if (weights) {  // a row per thread
                const int q = warp & 3, row = q * 32 + lane;  // (the quarter of tensor memory's lanes a warp may write)
                const float4* w = reinterpret_cast<const float4*>(gbase + ws * G::kW + row * 128);
                const uint32_t to = tmem + ((uint32_t)(q * 32) << 16) + G::kWeights + rs * kPartColumns;
                float4 x[8];
#pragma unroll
                for (int c = 0; c < 8; ++c) x[c] = w[c ^ (row & 7)];  // (the copy's swizzle)
                __syncwarp();
                if (lane == 0) mkb::mbar_arrive(w_empty(ws));
                tc_after_sync();
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    uint32_t p[24];  // 16 of the inner dimension: first, second, third parts
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float4 v = x[4 * k + j];
                        split2(v.x, v.y, p[2 * j], p[8 + 2 * j], p[16 + 2 * j], odd);
                        split2(v.z, v.w, p[2 * j + 1], p[8 + 2 * j + 1], p[16 + 2 * j + 1], odd);
                    }
                    tc_store16(to + 24 * k, p);
                    tc_store8(to + 24 * k + 16, p + 16);
                }
                if (odd & 0x7fff7fffu) {  // (rare)
                    bool any = false;
#pragma unroll
                    for (int c = 0; c < 8; ++c) any |= infinite4(x[c]);
                    if (any) atomicOr(flags + 8 + q, 1u << lane);
                }
                tc_stored();
                tc_before_sync();
            } else {  // eight neighbours of a row per thread, of every 32nd row
                constexpr int kRows = (NT + 31) / 32;
                const int i = threadIdx.x - 32 * (2 + kWeightWarps), row = i >> 2, quarter = i & 3, turn = row & 7;
                if (NT >= 32 || row < NT) {  // (uniform over the warp)
                    uint8_t *stage = gbase + G::kTokens + st * G::kX + row * 128, *rest = gbase + G::kRest + rs / 2 * G::kX + row * 128;
                    float4 x[kRows][2];
#pragma unroll
                    for (int j = 0; j < kRows; ++j)
#pragma unroll
                        for (int h = 0; h < 2; ++h) x[j][h] = *reinterpret_cast<const float4*>(stage + j * 4096 + (((2 * quarter + h) ^ turn) << 4));
                    __syncwarp();  // (a row's parts take the place that its four lanes read from)
                    const bool swap = turn & 1;  // (which part is written first: odd rows the other one, so that no two rows meet in a bank)
                    const int to1 = (quarter ^ turn) << 4, to2 = ((4 + quarter) ^ turn) << 4, to3 = (((it & 1) * 4 + quarter) ^ turn) << 4;
#pragma unroll
                    for (int j = 0; j < kRows; ++j) {
                        uint32_t p1[4], p2[4], p3[4];
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            split2(x[j][h].x, x[j][h].y, p1[2 * h], p2[2 * h], p3[2 * h], odd);
                            split2(x[j][h].z, x[j][h].w, p1[2 * h + 1], p2[2 * h + 1], p3[2 * h + 1], odd);
                        }
                        const uint4 u = make_uint4(p1[0], p1[1], p1[2], p1[3]), v = make_uint4(p2[0], p2[1], p2[2], p2[3]);
                        *reinterpret_cast<uint4*>(stage + j * 4096 + (swap ? to2 : to1)) = swap ? v : u;
                        *reinterpret_cast<uint4*>(stage + j * 4096 + (swap ? to1 : to2)) = swap ? u : v;
                        *reinterpret_cast<uint4*>(rest + j * 4096 + to3) = make_uint4(p3[0], p3[1], p3[2], p3[3]);
                    }
                    if (odd & 0x7fff7fffu) {
#pragma unroll
                        for (int j = 0; j < kRows; ++j)
                            if (infinite4(x[j][0]) || infinite4(x[j][1])) atomicOr(flags + j, 1u << row);
                    }
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                }
            }
            __syncwarp();
            if (lane == 0) mkb::mbar_arrive(ready(st));
        }
    } else {
        const int q = warp & 3, half = (warp - 2 - kWeightWarps - kTokenWarps) >> 2;  // the quarter of tensor memory's lanes this warp may read
        const uint32_t at = tmem + ((uint32_t)(q * 32) << 16) + half * C;
        float sum[C] = {};
        bool ok = true;
        for (int it = 0; it < steps; ++it) {
            ok = __all_sync(0xffffffffu, wait(acc_full(it & 1), it / 2, 3));
            if (!ok) break;
            tc_after_sync();
            add_columns<C>(at + (it & 1) * NT, sum);
            tc_before_sync();
            __syncwarp();
            if (lane == 0) mkb::mbar_arrive(acc_empty(it & 1));
        }
        if (ok) {
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
    uint32_t any = 0;
    for (int i = 0; i < 12; ++i) any |= flags[i];
    if (any != 0) {
        // An infinite operand has no parts: its token's or feature's sums once more with FMA, a warp each (300 x 8192 x 2048 with one infinite
        // activation: 188 us instead of 68; one in every token: 2.1 ms).
        const int last = min(s.K, (first + steps) * kStep);
        for (int i = warp; i < tokens * kFeatures; i += kThreads / 32) {
            const int t = i / kFeatures, n = i % kFeatures;
            if (n0 + n >= s.N || ((flags[t >> 5] >> (t & 31) | flags[8 + (n >> 5)] >> (n & 31)) & 1) == 0) continue;
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
    if (K < kShort) {
        fma_f32_kernel<<<dim3((N + 511) / 512, (T + kFmaTokens - 1) / kFmaTokens), 256, 0, st>>>(A, lda, W, ldw, T, N, K, e);
        return cudaGetLastError();
    }
    int sms = 0;
    if (const cudaError_t err = sm_count(&sms); err != cudaSuccess) return err;
    // Tokens of a tile and CTAs on it: waves of tiles, each so many steps (in cycles, as measured with tf32 parts; of 78 shapes of 3 to
    // 2048 tokens x 512 to 10304 features x 512 to 8192 the choice misses the fastest of these kinds by more than 5 % in two, 2 us at most) and a beginning
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
