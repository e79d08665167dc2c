// bf16 matrix product of the hybrid models' prefill on the 5th-generation tensor cores:
// out[token, feature] = sum_k A[token, k] * W[feature, k], fp32 accumulation in tensor memory.
//
// Persistent, warp-specialised: one producer thread (TMA, 128-byte swizzle), one MMA thread
// (tcgen05.mma, M = 128 tokens per CTA, N = kBN features), four epilogue warps that read one of two
// accumulators back while the other is being filled.  The epilogue goes through shared memory so
// that stores are row segments: plus the bias, times the layer scale into the 32-bit residual stream,
// in bf16, the gated unit of neighbouring columns in bf16, the gated unit of two matrices (a tile is then
// as many rows of either), rotated into the queries and the key/value cache, or into a fixed-point residual stream.
#include "hybrid_kernels.h"
#include "hybrid_tcgen05.cuh"

namespace mkbh {
namespace {

constexpr int kBM = 128, kBK = 64;
constexpr int kGemmThreads = 192;
constexpr int kEpiStride = 33;  // floats per row of a warp's 32 x 32 transpose buffer

// kPair CTAs work on one tile: 128 tokens each, the features' operand halved between them.  One CTA's
// 128 x 256 tile takes in 94 bytes a cycle of MMA, more than L2 gives an SM (64); a pair's 256 x 256 takes 63 per SM:
// 2048 x 28672 x 4096 in 330 us alone, 307 in pairs.
template <int kBN, int kPair>
struct Geo {
    static constexpr int kRowsW = kBN / kPair;
    static constexpr int kStageBytes = (kBM + kRowsW) * kBK * 2;
    static constexpr int kStages = kRowsW == 256 ? 4 : kRowsW == 128 ? 6 : 8;
    static constexpr int kEpi = kStages * kStageBytes;
    static constexpr int kBars = kEpi + 4 * 32 * kEpiStride * 4;
    static constexpr int kNumBars = 2 * kStages + 4;
    static constexpr int kCtl = kBars + kNumBars * 8;
    static constexpr int kTotal = kCtl + 16;
    static constexpr int kAlloc = kTotal + 1024;
    static_assert(kAlloc <= 227 * 1024, "");
};

struct Shape {
    int T, N, K, tiles_m, tiles, parts, a_rows;  // parts: CTAs that share a tile's inner dimension; a_rows: tokens of a copy
    unsigned long long timeout_ns;
    int* status;
    bool early;  // begins before the launch before it has ended: weights may be read until then
};

// What the epilogue can do: a build per group of results, so that one group's code does not cost the others registers.
enum class Group { kPlain, kSilu, kRope, kFixed };  // kSilu: two weight matrices, kBN / 2 columns of each per tile
template <int kBN> constexpr int kPartRow = kBN + 4;  // floats of a row of partial sums
constexpr Group group_of(Result r) {
    return r == Result::kSilu ? Group::kSilu : r == Result::kRope ? Group::kRope : r == Result::kFixed ? Group::kFixed : Group::kPlain;
}
__device__ __forceinline__ long long fixed_of(float x) { return __float2ll_rn(x * mkb::kResidualScale); }

// Columns n (even) and n + 1 of token t, where a thread has just these.  kAdd: `before` is what they are added to, fetched while the
// sums are still on their way (as additions in L2, which nobody waits for, the scaled sum would be rounded first).
template <Group kGroup>
__device__ __forceinline__ float2 put_on(const GemmEpilogue& e, int N, int t, int n) {
    float2 v = make_float2(0.f, 0.f);
    if (kGroup != Group::kPlain || e.what != Result::kAdd || n >= N) return v;
    const float* o = e.out + (size_t)t * e.ld + n;
    v.x = __ldcg(o);
    if (n + 1 < N) v.y = __ldcg(o + 1);
    return v;
}
template <Group kGroup>
__device__ __forceinline__ void put(const GemmEpilogue& e, int N, int t, int n, float x, float y, float2 before) {
    if (n >= N) return;
    if constexpr (kGroup == Group::kRope) {
        const RopeTarget& p = e.rope;
        const int at = n - p.q_cols;  // column of [keys | values]
        if (at < p.k_cols) {
            const size_t z = (size_t)(p.pos0 + t) * p.dim + n % p.dim;
            const float2 c = __ldg(reinterpret_cast<const float2*>(p.cos + z)), d = __ldg(reinterpret_cast<const float2*>(p.sin + z));
            const float turned = x * c.x - y * d.x;
            y = y * c.y + x * d.y;
            x = turned;
        }
        bf16* o = at < 0 ? p.q + (size_t)t * p.q_cols + n : (at < p.k_cols ? p.k + at : p.v + (at - p.k_cols)) + (size_t)(p.pos0 + t) * p.k_cols;
        *reinterpret_cast<uint32_t*>(o) = mkb::pack_bf16x2(x, y);
    } else if constexpr (kGroup == Group::kFixed) {
        long long* o = static_cast<long long*>(e.cast) + (size_t)t * e.ld + n;
        mkb::red_add_u64(o, (unsigned long long)fixed_of(x));
        mkb::red_add_u64(o + 1, (unsigned long long)fixed_of(y));
    } else if (kGroup == Group::kSilu || e.what == Result::kCast) {
        bf16* o = static_cast<bf16*>(e.cast) + (size_t)t * e.ld + n;
        if (n + 1 < N) *reinterpret_cast<uint32_t*>(o) = mkb::pack_bf16x2(x, y);
        else *o = __float2bfloat16_rn(x);
    } else if (e.what == Result::kGlu) {  // (N is even)
        static_cast<bf16*>(e.cast)[(size_t)t * e.ld + n / 2] = __float2bfloat16_rn(clamped_glu(x, y, e.limit, e.alpha));
    } else {
        float* o = e.out + (size_t)t * e.ld + n;
        const bool two = n + 1 < N;
        if (e.what == Result::kAdd) {  // (no other thread writes these)
            o[0] = fmaf(e.scale ? __ldg(e.scale + n) : 1.f, x, before.x);
            if (two) o[1] = fmaf(e.scale ? __ldg(e.scale + n + 1) : 1.f, y, before.y);
        } else {
            o[0] = x + (e.bias ? __ldg(e.bias + n) : 0.f);
            if (two) o[1] = y + (e.bias ? __ldg(e.bias + n + 1) : 0.f);
        }
    }
}

// kMode 1: a CTA per tile; 2: a pair of CTAs (cta_group::2) per tile; 0: s.parts CTAs, a cluster, share a tile's
// inner dimension and add up their accumulators through distributed shared memory, always in the same order.
template <int kBN, int kMode, Group kGroup>
__global__ void __launch_bounds__(kGemmThreads, 1)
gemm_bf16_kernel(const __grid_constant__ CUtensorMap amap, const __grid_constant__ CUtensorMap wmap,
                 const __grid_constant__ CUtensorMap wmap2, const Shape s, const GemmEpilogue e) {
    constexpr int kPair = kMode == 2 ? 2 : 1;
    constexpr bool kShare = kMode == 0;
    using G = Geo<kBN, kPair>;
    extern __shared__ uint8_t raw[];
    const uint32_t raw32 = mkb::smem_u32(raw), base = (raw32 + 1023u) & ~1023u;
    uint8_t* gbase = raw + (base - raw32);
    volatile int* ctl = reinterpret_cast<volatile int*>(gbase + G::kCtl);  // [0] dead, [1] tensor-memory base
    // (uniform, and known to be: the roles' loops then run on the uniform datapath, which the copies and MMAs read from)
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const uint32_t rank = kPair == 2 ? tc_rank() : 0u;
    const int worker = blockIdx.x / (kShare ? s.parts : kPair), workers = gridDim.x / (kShare ? s.parts : kPair);  // (a pair's CTAs are neighbours)
    auto full = [&](int i) { return base + G::kBars + i * 8; };
    auto empty = [&](int i) { return base + G::kBars + (G::kStages + i) * 8; };
    auto acc_full = [&](int i) { return base + G::kBars + (2 * G::kStages + i) * 8; };
    auto acc_empty = [&](int i) { return base + G::kBars + (2 * G::kStages + 2 + i) * 8; };

    if (threadIdx.x == 0) {
        for (int i = 0; i < G::kStages; ++i) {
            mkb::mbar_init(full(i), 1);
            mkb::mbar_init(empty(i), 1);
        }
        for (int i = 0; i < 2; ++i) {
            mkb::mbar_init(acc_full(i), 1);
            mkb::mbar_init(acc_empty(i), 4 * kPair);
        }
        ctl[0] = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        if constexpr (kPair == 2) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(base + G::kCtl + 4),
                         "r"((uint32_t)(2 * kBN))
                         : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(base + G::kCtl + 4),
                         "r"((uint32_t)(2 * kBN))
                         : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if constexpr (kPair == 2) tc_cluster_sync();  // (the other CTA's barriers are there)
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = (uint32_t)ctl[1];
    let_next();
    if (warp != 0) after_previous();
    constexpr bool kDual = kGroup == Group::kSilu;
    constexpr int wide = kDual ? kBN / 2 : kBN;
    int ksteps = (s.K + kBK - 1) / kBK, kfirst = 0;
    if constexpr (kShare) {
        const int r = (int)tc_rank(), end = ksteps * (r + 1) / s.parts;  // (at least one step: parts <= steps)
        kfirst = ksteps * r / s.parts;
        ksteps = end - kfirst;
    }

    if (warp == 0) {
        const bool chosen = tc_elect();
        uint32_t it = 0;
        bool ok = true;
        auto weights = [&](int st, int k, int n0) {
            const uint32_t dw = base + st * G::kStageBytes + kBM * kBK * 2;
            if (rank == 0) mkb::mbar_expect_tx(full(st), kPair * (s.a_rows + G::kRowsW) * kBK * 2);
            if constexpr (kPair == 2) {  // both CTAs' copies count on the first one's barrier
                const uint32_t bar = tc_peer(full(st), 0);
                if (kDual) tc_tma_2d_pair(dw, rank ? &wmap2 : &wmap, k * kBK, n0, bar);
                else tc_tma_2d_pair(dw, &wmap, k * kBK, n0 + rank * G::kRowsW, bar);
            } else {
                tc_tma_2d(dw, &wmap, (kfirst + k) * kBK, n0, full(st));
                if (kDual) tc_tma_2d(dw + kBN / 2 * kBK * 2, &wmap2, (kfirst + k) * kBK, n0, full(st));
            }
        };
        // a ring of weights is on its way while the launch before this one ends (if it has ended, the tokens' copies
        // would only wait behind them)
        const int before = s.early ? min(ksteps, G::kStages) : 0;
        if (chosen)
            for (int k = 0; k < before; ++k) weights(k, k, (worker / s.tiles_m) * wide);
        after_previous();
        for (int tile = worker; tile < s.tiles && ok; tile += workers) {
            const int m0 = ((tile % s.tiles_m) * kPair + rank) * kBM, n0 = (tile / s.tiles_m) * wide;
            for (int k = 0; k < ksteps; ++k, ++it) {
                const int st = it % G::kStages;
                ok = __all_sync(0xffffffffu, tc_wait(empty(st), ((it / G::kStages) & 1u) ^ 1u, ctl, s.timeout_ns, s.status, 0));
                if (!ok) break;
                if (!chosen) continue;
                if (it >= (uint32_t)before) weights(st, k, n0);
                const uint32_t dst = base + st * G::kStageBytes;
                if constexpr (kPair == 2) tc_tma_2d_pair(dst, &amap, k * kBK, m0, tc_peer(full(st), 0));
                else tc_tma_2d(dst, &amap, (kfirst + k) * kBK, m0, full(st));
            }
        }
        // no copy may be in flight when the CTA's shared memory goes away, nor an arrival from the pair's first CTA
        const uint32_t last = it > (uint32_t)G::kStages ? it - G::kStages : 0u;
        for (uint32_t i = last; i < it; ++i) {
            if (ok) tc_wait(empty(i % G::kStages), (i / G::kStages) & 1u, ctl, s.timeout_ns, s.status, 0);
            else if (rank == 0) tc_wait(full(i % G::kStages), (i / G::kStages) & 1u, nullptr, s.timeout_ns, s.status, 0);
        }
    } else if (warp == 1 && rank == 0) {
        const bool chosen = tc_elect();
        const uint32_t idesc = tc_idesc(kPair * kBM, kBN);
        uint32_t it = 0, acc = 0;
        bool ok = true;
        for (int tile = worker; tile < s.tiles && ok; tile += workers, ++acc) {
            const uint32_t buf = acc & 1u;
            ok = __all_sync(0xffffffffu, tc_wait(acc_empty(buf), ((acc >> 1) & 1u) ^ 1u, ctl, s.timeout_ns, s.status, 1));
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            for (int k = 0; k < ksteps; ++k, ++it) {
                const int st = it % G::kStages;
                ok = __all_sync(0xffffffffu, tc_wait(full(st), (it / G::kStages) & 1u, ctl, s.timeout_ns, s.status, 1));
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if (!chosen) continue;
                const uint32_t a = base + st * G::kStageBytes, w = a + kBM * kBK * 2;
#pragma unroll
                for (int kk = 0; kk < kBK / 16; ++kk)
                    if constexpr (kPair == 2) tc_mma_pair(tmem + buf * kBN, tc_desc(a + kk * 32), tc_desc(w + kk * 32), idesc, (uint32_t)((k | kk) != 0));
                    else tc_mma(tmem + buf * kBN, tc_desc(a + kk * 32), tc_desc(w + kk * 32), idesc, (uint32_t)((k | kk) != 0));
                if constexpr (kPair == 2) tc_commit_pair(empty(st));
                else tc_commit(empty(st));
            }
            if (!ok) break;
            if (!chosen) continue;
            if constexpr (kPair == 2) tc_commit_pair(acc_full(buf));
            else tc_commit(acc_full(buf));
        }
    } else if (warp >= 2) {
        const int q = warp & 3;  // the quarter of tensor memory's lanes this warp may read
        float* tr = reinterpret_cast<float*>(gbase + G::kEpi) + (warp - 2) * 32 * kEpiStride;
        uint32_t acc = 0;
        for (int tile = worker; tile < s.tiles; tile += workers, ++acc) {
            const int m0 = ((tile % s.tiles_m) * kPair + rank) * kBM + q * 32, n0 = (tile / s.tiles_m) * wide;
            const uint32_t buf = acc & 1u;
            const bool ok = tc_wait(acc_full(buf), (acc >> 1) & 1u, ctl, s.timeout_ns, s.status, 2);
            if (!__all_sync(0xffffffffu, ok)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int rows = min(32, s.T - m0);
            if constexpr (kShare) {  // the ring's copies have arrived and been read: the accumulators take its place
                for (int c0 = 0; c0 < kBN; c0 += 32) {
                    uint32_t r[32];
                    tc_load32(tmem + ((uint32_t)(q * 32) << 16) + c0, r);
                    float4* o = reinterpret_cast<float4*>(gbase) + ((q * 32 + lane) * kPartRow<kBN> + c0) / 4;
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        o[j] = make_float4(__uint_as_float(r[4 * j]), __uint_as_float(r[4 * j + 1]), __uint_as_float(r[4 * j + 2]),
                                           __uint_as_float(r[4 * j + 3]));
                }
            } else for (int c0 = 0; c0 < wide; c0 += 32) {
                if (n0 + c0 >= s.N || rows <= 0) break;  // uniform over the warp
                uint32_t r[32];
                tc_load32(tmem + ((uint32_t)(q * 32) << 16) + buf * kBN + c0, r);
                if constexpr (kDual) {
                    uint32_t u[32];
                    tc_load32(tmem + ((uint32_t)(q * 32) << 16) + buf * kBN + kBN / 2 + c0, u);
#pragma unroll
                    for (int j = 0; j < 32; ++j) {
                        const float g = __uint_as_float(r[j]);
                        r[j] = __float_as_uint(g * sigmoid_f(g) * __uint_as_float(u[j]));
                    }
                }
#pragma unroll
                for (int j = 0; j < 32; ++j) tr[lane * kEpiStride + j] = __uint_as_float(r[j]);
                __syncwarp();
                if (kDual || (kGroup == Group::kPlain && e.what == Result::kCast)) {  // two rows at a time, two columns per lane
                    const int col = 2 * (lane & 15), n = n0 + c0 + col;
                    bf16* o = static_cast<bf16*>(e.cast) + (size_t)m0 * e.ld + n;
                    for (int i = lane >> 4; i < rows; i += 2) {
                        const float *v = tr + i * kEpiStride + col;
                        if (n + 1 < s.N) *reinterpret_cast<uint32_t*>(o + (size_t)i * e.ld) = mkb::pack_bf16x2(v[0], v[1]);
                        else if (n < s.N) o[(size_t)i * e.ld] = __float2bfloat16_rn(v[0]);
                    }
                } else if (kGroup == Group::kPlain && e.what == Result::kGlu) {  // 16 units of a row per half warp
                    const int col = 2 * (lane & 15), n = n0 + c0 + col;
                    bf16* o = static_cast<bf16*>(e.cast) + (size_t)m0 * e.ld + n / 2;
                    if (n < s.N)  // (N is even)
                        for (int i = lane >> 4; i < rows; i += 2) {
                            const float* v = tr + i * kEpiStride + col;
                            o[(size_t)i * e.ld] = __float2bfloat16_rn(clamped_glu(v[0], v[1], e.limit, e.alpha));
                        }
                } else if (kGroup == Group::kRope) {  // (boundaries are multiples of 64: a chunk has one target)
                    const int col = 2 * (lane & 15), n = n0 + c0 + col;
                    const RopeTarget& p = e.rope;
                    const int at = n - p.q_cols;  // column of [keys | values]
                    bf16* o = at < 0 ? p.q + n : at < p.k_cols ? p.k + at : p.v + (at - p.k_cols);
                    const int64_t ld = at < 0 ? p.q_cols : p.k_cols;
                    const int row0 = at < 0 ? m0 : p.pos0 + m0;
                    // (eight rows' angles are on their way together: a row at a time, each a round trip to L2, made 501 x 3072 x
                    // 2048 take 39 us of which the product is 17)
#pragma unroll 1
                    for (int i0 = lane >> 4; i0 < 32; i0 += 16) {
                        float2 c[8], d[8];
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            const size_t z = (size_t)(p.pos0 + m0 + min(i0 + 2 * j, rows - 1)) * p.dim + n % p.dim;
                            if (at >= p.k_cols) break;  // (values stay as they are)
                            c[j] = __ldg(reinterpret_cast<const float2*>(p.cos + z));
                            d[j] = __ldg(reinterpret_cast<const float2*>(p.sin + z));
                        }
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            const int i = i0 + 2 * j;
                            if (i >= rows) break;
                            const float x = tr[i * kEpiStride + col], y = tr[i * kEpiStride + col + 1];
                            *reinterpret_cast<uint32_t*>(o + (size_t)(row0 + i) * ld) =
                                at < p.k_cols ? mkb::pack_bf16x2(x * c[j].x - y * d[j].x, y * c[j].y + x * d[j].y) : mkb::pack_bf16x2(x, y);
                        }
                    }
                }
                const int n = n0 + c0 + lane;
                if (kGroup == Group::kFixed && n < s.N) {
                    long long* o = static_cast<long long*>(e.cast) + (size_t)m0 * e.ld + n;
                    for (int i = 0; i < rows; ++i) mkb::red_add_u64(o + (size_t)i * e.ld, (unsigned long long)fixed_of(tr[i * kEpiStride + lane]));
                }
                if (kGroup == Group::kPlain && n < s.N && e.what <= Result::kAdd) {
                    float* o = e.out + (size_t)m0 * e.ld + n;
                    if (e.what == Result::kAdd) {
                        const float f = e.scale ? __ldg(e.scale + n) : 1.f;
                        // (this tile is the only writer of these elements: one addition each, in L2)
                        for (int i = 0; i < rows; ++i)
                            asm volatile("red.global.add.f32 [%0], %1;" ::"l"(o + (size_t)i * e.ld), "f"(f * tr[i * kEpiStride + lane])
                                         : "memory");
                    } else {
                        const float b = e.bias ? __ldg(e.bias + n) : 0.f;
                        for (int i = 0; i < rows; ++i) o[(size_t)i * e.ld] = tr[i * kEpiStride + lane] + b;
                    }
                }
                __syncwarp();
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) {
                if constexpr (kPair == 2) tc_arrive_cluster(tc_peer(acc_empty(buf), 0));
                else mkb::mbar_arrive(acc_empty(buf));
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (*ctl) tc_settle();  // (the roles leave one by one then, the drain above too)
    if constexpr (kShare) {
        tc_cluster_sync();
        const int m0 = (worker % s.tiles_m) * kBM, n0 = (worker / s.tiles_m) * wide, rows = min(kBM, s.T - m0);
        const uint32_t me = tc_rank(), parts = s.parts;
        // Four rows of a warp at a time: a row's parts, another SM's shared memory, take most of a microsecond to arrive.
        constexpr int kRowsAtOnce = 4, kWarps = kGemmThreads / 32;
        const int next = (int)parts * kWarps;
        for (int i0 = (int)me + (int)parts * warp; i0 < rows; i0 += kRowsAtOnce * next)
#pragma unroll 1
            for (int c = 2 * lane; c < wide; c += 64) {
                float2 sum[kRowsAtOnce], up[kRowsAtOnce], before[kRowsAtOnce];
#pragma unroll
                for (int r = 0; r < kRowsAtOnce; ++r) {
                    sum[r] = up[r] = make_float2(0.f, 0.f);
                    before[r] = put_on<kGroup>(e, s.N, m0 + min(i0 + r * next, rows - 1), n0 + c);
                }
                for (uint32_t z = 0; z < parts; z += 2) {  // (two or four parts)
                    float2 v[2][kRowsAtOnce], u[2][kRowsAtOnce];
#pragma unroll
                    for (int y = 0; y < 2; ++y)
#pragma unroll
                        for (int r = 0; r < kRowsAtOnce; ++r) {
                            const uint32_t at = tc_peer(base + (uint32_t)(min(i0 + r * next, rows - 1) * kPartRow<kBN> + c) * 4, z + y);
                            v[y][r] = tc_peer_load2(at);
                            if constexpr (kDual) u[y][r] = tc_peer_load2(at + wide * 4);
                        }
#pragma unroll
                    for (int y = 0; y < 2; ++y)
#pragma unroll
                        for (int r = 0; r < kRowsAtOnce; ++r) {
                            sum[r].x += v[y][r].x;
                            sum[r].y += v[y][r].y;
                            if constexpr (kDual) {
                                up[r].x += u[y][r].x;
                                up[r].y += u[y][r].y;
                            }
                        }
                }
#pragma unroll
                for (int r = 0; r < kRowsAtOnce; ++r) {
                    if (i0 + r * next >= rows) break;
                    float x = sum[r].x, y = sum[r].y;
                    if constexpr (kDual) x *= sigmoid_f(x) * up[r].x, y *= sigmoid_f(y) * up[r].y;
                    put<kGroup>(e, s.N, m0 + i0 + r * next, n0 + c, x, y, before[r]);
                }
            }
        tc_cluster_sync();
    }
    if constexpr (kPair == 2) {
        tc_cluster_sync();
        if (warp == 1)
            asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)(2 * kBN)) : "memory");
    } else if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)(2 * kBN)) : "memory");
    }
}

template <int kBN, int kMode, Group kGroup>
cudaError_t launch(const bf16* A, int64_t lda, const bf16* W, const bf16* W2, int64_t ldw, Shape s, const GemmEpilogue& e,
                   int sms, cudaStream_t st) {
    constexpr int kPair = kMode == 2 ? 2 : 1;
    using G = Geo<kBN, kPair>;
    static_assert(kMode != 0 || kBM * kPartRow<kBN> * 4 <= G::kEpi, "");
    static bool set[64] = {};
    const auto kernel = gemm_bf16_kernel<kBN, kMode, kGroup>;
    int dev = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err != cudaSuccess) return err;
    if (!set[dev & 63]) {
        err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, G::kAlloc);
        if (err != cudaSuccess) return err;
        set[dev & 63] = true;
    }
    CUtensorMap amap, wmap, wmap2;
    constexpr bool kDual = kGroup == Group::kSilu;
    constexpr int wide = kDual ? kBN / 2 : kBN, box = kPair == 2 ? kBN / 2 : wide;
    // (rows of the tile that no copy fills hold anything: they only reach accumulators that nobody reads)
    s.a_rows = s.T < kBM ? (s.T + 7) / 8 * 8 : kBM;
    if ((err = tc_map(&amap, A, s.K, s.T, lda, kBK, s.a_rows)) != cudaSuccess) return err;
    if ((err = tc_map(&wmap, W, s.K, s.N, ldw, kBK, box)) != cudaSuccess) return err;
    wmap2 = wmap;
    if (kDual && (err = tc_map(&wmap2, W2, s.K, s.N, ldw, kBK, box)) != cudaSuccess) return err;
    s.tiles_m = (s.T + kPair * kBM - 1) / (kPair * kBM);
    s.tiles = s.tiles_m * ((s.N + wide - 1) / wide);
    const int workers = kMode == 0 || s.tiles < sms / kPair ? s.tiles : sms / kPair, ctas = kMode == 0 ? s.parts : kPair;
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3(workers * ctas);
    c.blockDim = dim3(kGemmThreads);
    c.dynamicSmemBytes = G::kAlloc;
    c.stream = st;
    cudaLaunchAttribute attrs[2] = {may_begin_early()};
    attrs[1].id = cudaLaunchAttributeClusterDimension;
    attrs[1].val.clusterDim.x = ctas;
    attrs[1].val.clusterDim.y = attrs[1].val.clusterDim.z = 1;
    c.attrs = attrs;
    c.numAttrs = ctas > 1 ? 2 : 1;
    return cudaLaunchKernelEx(&c, kernel, amap, wmap, wmap2, s, e);
}

template <Group kGroup>
cudaError_t choose(const bf16* A, int64_t lda, const bf16* W, const bf16* W2, int64_t ldw, Shape s, const GemmEpilogue& e, int sms,
                   cudaStream_t st) {
    // The kind of tile with the smallest estimate, fitted in us to 48 shapes of 16..2048 tokens x 2048..28672 features x
    // 512..14336 (cold caches): waves of tiles, each so many steps of the inner dimension, and the last epilogue.  It ranks the
    // kinds and is no time: what all kinds pay alike (the launch, the weights' way from memory) is left out.  One row of
    // a head of 128256 x 2048 takes 101 - 108 us whatever the kind (80 us of bytes), 61 x 16384 x 2048 27.6 us as tiles of 128
    // and of 64 and 29.8 - 33.8 as wider ones or pairs.  A step costs what an SM takes in from L2 (24 KB: 0.19 us, 32 KB:
    // 0.23 us), so few narrow tiles with a long inner dimension are shared, 61 x 2048 x 8192 in us: 38.0 as 16 tiles of
    // 128, 33.8 as 32 of 64, 23.6 with two CTAs on each of these, 19.5 with four.  A cluster's exchange costs what its rows
    // do, and clusters beyond one wave wait for whole groups of SMs, as do clusters of eight.  Of 25 shapes of 1 to 2048 tokens
    // the choice missed the fastest kind by more than 5 % in two: 61 x 3072 x 2048 (17.4 us, 15.4) and 200 x 16384 x 2048
    // (33.8, 31.7).
    const int steps = (s.K + kBK - 1) / kBK;
    auto tiles_of = [&](int bn, int pair) {
        const int wide = kGroup == Group::kSilu ? bn / 2 : bn;
        return ((s.T + pair * kBM - 1) / (pair * kBM)) * ((s.N + wide - 1) / wide);
    };
    auto alone = [&](int bn, int pair, float step, float epilogue) {
        const int workers = sms / pair;
        return epilogue + (tiles_of(bn, pair) + workers - 1) / workers * steps * step;
    };
    auto shared = [&](int bn, int parts, float step, float epilogue) {
        if (tiles_of(bn, 1) * parts > sms || steps < 2 * parts) return INFINITY;
        return epilogue + (steps + parts - 1) / parts * step + 2.7f + (s.T < kBM ? s.T : kBM) * bn * 0.00027f;
    };
    const float costs[] = {alone(256, 2, 0.35f, 5.f),   alone(128, 2, 0.205f, 3.5f), alone(256, 1, 0.38f, 3.6f), alone(128, 1, 0.232f, 1.f),
                           alone(64, 1, 0.19f, 1.f),    shared(128, 2, 0.232f, 1.f), shared(128, 4, 0.232f, 1.f), shared(64, 2, 0.19f, 1.f),
                           shared(64, 4, 0.19f, 1.f)};
    int best = 0;
    for (int i = 1; i < 9; ++i)
        if (costs[i] < costs[best]) best = i;
    s.parts = best == 5 || best == 7 ? 2 : 4;
    switch (best) {
        case 0: return launch<256, 2, kGroup>(A, lda, W, W2, ldw, s, e, sms, st);
        case 1: return launch<128, 2, kGroup>(A, lda, W, W2, ldw, s, e, sms, st);
        case 2: return launch<256, 1, kGroup>(A, lda, W, W2, ldw, s, e, sms, st);
        case 3: return launch<128, 1, kGroup>(A, lda, W, W2, ldw, s, e, sms, st);
        case 4: return launch<64, 1, kGroup>(A, lda, W, W2, ldw, s, e, sms, st);
        case 5:
        case 6: return launch<128, 0, kGroup>(A, lda, W, W2, ldw, s, e, sms, st);
        default: return launch<64, 0, kGroup>(A, lda, W, W2, ldw, s, e, sms, st);
    }
}

}  // namespace

cudaError_t gemm_bf16(const bf16* A, int64_t lda, const bf16* W, int64_t ldw, int T, int N, int K, const GemmEpilogue& e,
                      int* status, cudaStream_t st, const bf16* W2, unsigned long long timeout_ns, bool early) {
    int sms = 0;
    if (const cudaError_t err = sm_count(&sms); err != cudaSuccess) return err;
    const Shape s{T, N, K, 0, 0, 1, 0, timeout_ns, status, early};
    switch (group_of(e.what)) {
        case Group::kSilu: return choose<Group::kSilu>(A, lda, W, W2, ldw, s, e, sms, st);
        case Group::kRope: return choose<Group::kRope>(A, lda, W, W2, ldw, s, e, sms, st);
        case Group::kFixed: return choose<Group::kFixed>(A, lda, W, W2, ldw, s, e, sms, st);
        default: return choose<Group::kPlain>(A, lda, W, W2, ldw, s, e, sms, st);
    }
}

}  // namespace mkbh
