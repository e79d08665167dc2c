// A prompt of a llama model, all tokens at once: the layers' matrix products on the 5th-generation tensor
// cores with the rotation, the cache append and the gated unit as epilogues, attention over the cache.
// Seven launches a layer.  501 tokens at the 1B widths (16 layers): 354.6 ms as a decode step per token, bound by the
// weights that every token streams again; 2.1 ms at once, bound by the products and the 118 launches' hand-over.  
// The residual stream is the embedding and a fixed-point sum of what the layers add to it (exact, whatever the order),
// operands of the products are bf16, both as in decoding.
#include "llama_prompt.h"

#include "hybrid_kernels.h"

namespace mkb {
namespace {

using mkbh::bf16;
using mkbh::GemmEpilogue;

constexpr int kNormThreads = 256, kKept = 8;  // float4s of a row per thread: widths up to 8192

// out = x / rms(x) * w, a block per row, x = hidden + sums.  `first`: the sums are cleared instead; `last`: they are copied there.
__global__ void __launch_bounds__(kNormThreads) prompt_norm_kernel(const bf16* hidden, long long* sums, bool first, long long* last, int width,
                                                                   float eps, const bf16* __restrict__ w, bf16* out) {
    __shared__ float red[kNormThreads / 32];
    mkbh::let_next();
    mkbh::after_previous();
    const size_t row = (size_t)blockIdx.x * width;
    float4 v[kKept];
    float square[1] = {0.f};
#pragma unroll
    for (int k = 0; k < kKept; ++k) {
        const int i = 4 * (threadIdx.x + k * kNormThreads);
        v[k] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (i >= width) continue;
        const uint2 e = *reinterpret_cast<const uint2*>(hidden + row + i);
        v[k] = make_float4(bf16_lo(e.x), bf16_hi(e.x), bf16_lo(e.y), bf16_hi(e.y));
        uint4* s = reinterpret_cast<uint4*>(sums + row + i);
        if (first) {
            s[0] = s[1] = make_uint4(0, 0, 0, 0);
        } else {
            const uint4 a = s[0], b = s[1];
            v[k].x += q32_to_float(a.x, a.y);
            v[k].y += q32_to_float(a.z, a.w);
            v[k].z += q32_to_float(b.x, b.y);
            v[k].w += q32_to_float(b.z, b.w);
            if (last != nullptr) {
                reinterpret_cast<uint4*>(last + i)[0] = a;
                reinterpret_cast<uint4*>(last + i)[1] = b;
            }
        }
        square[0] += v[k].x * v[k].x + v[k].y * v[k].y + v[k].z * v[k].z + v[k].w * v[k].w;
    }
    mkbh::block_sum<1, kNormThreads>(square, red);
    const float inv = 1.f / sqrtf(square[0] / width + eps);
#pragma unroll
    for (int k = 0; k < kKept; ++k) {
        const int i = 4 * (threadIdx.x + k * kNormThreads);
        if (i >= width) continue;
        const uint2 g = *reinterpret_cast<const uint2*>(w + i);
        *reinterpret_cast<uint2*>(out + row + i) = make_uint2(pack_bf16x2(v[k].x * inv * bf16_lo(g.x), v[k].y * inv * bf16_hi(g.x)),
                                                              pack_bf16x2(v[k].z * inv * bf16_lo(g.y), v[k].w * inv * bf16_hi(g.y)));
    }
}

}  // namespace

#define MKB_TRY(call)                             \
    do {                                          \
        const cudaError_t e_ = (call);            \
        if (e_ != cudaSuccess) return e_;         \
    } while (0)

cudaError_t prompt_launch(const MkbGlobals& g, const MkbPrompt& p, int* status, cudaStream_t s) {
    const PromptBuffers b(g, p.tokens, p.workspace);
    const int n = p.tokens, H = g.hidden_size, F = g.intermediate_size, D = g.head_dim, Q = g.num_attention_heads * D, KV = g.num_kv_heads * D;
    const unsigned long long wait = g.wait_timeout_ms ? g.wait_timeout_ms * 1000000ull : mkbh::kWaitNs;
    auto at = [](const void* w, size_t elements) { return static_cast<const bf16*>(w) + elements; };
    auto norm = [&](int row0, int rows, bool first, long long* last, const bf16* w) {
        cudaLaunchConfig_t c = {};
        c.gridDim = dim3(rows);
        c.blockDim = dim3(kNormThreads);
        c.stream = s;
        cudaLaunchAttribute early = mkbh::may_begin_early();
        c.attrs = &early;
        c.numAttrs = first ? 0 : 1;  // (the first launch waits for all that came before, the weights' arrival among it)
        return cudaLaunchKernelEx(&c, prompt_norm_kernel, static_cast<const bf16*>(p.hidden) + (size_t)row0 * H, b.sums + (size_t)row0 * H, first, last,
                                  H, g.rms_norm_eps, w, b.act);
    };
    auto gemm = [&](const bf16* A, const bf16* W, int rows, int N, int K, const GemmEpilogue& e, const bf16* W2 = nullptr) {
        return mkbh::gemm_bf16(A, K, W, K, rows, N, K, e, status, s, W2, wait);
    };
    for (size_t i = 0; i < (size_t)g.num_layers; ++i) {
        const size_t cache = i * g.kv_batch * g.kv_max_len * KV;
        bf16 *k = static_cast<bf16*>(g.k_cache) + cache, *v = static_cast<bf16*>(g.v_cache) + cache;
        MKB_TRY(norm(0, n, i == 0, nullptr, at(g.attn_ln_weights, i * H)));
        MKB_TRY(gemm(b.act, at(g.qkv_weights, i * (Q + 2 * KV) * H), n, Q + 2 * KV, H,
                     GemmEpilogue::rotate({b.q, k, v, Q, KV, D, p.pos0, static_cast<const float*>(g.rope_cos), static_cast<const float*>(g.rope_sin)})));
        MKB_TRY(mkbh::flash_cache({b.q, k, v, b.act, n, p.pos0, g.num_attention_heads, g.num_kv_heads, D, g.attn_scale, status, wait}, s));
        MKB_TRY(gemm(b.act, at(g.o_proj_weights, i * H * Q), n, H, Q, GemmEpilogue::add_fixed(b.sums, H)));
        MKB_TRY(norm(0, n, false, nullptr, at(g.mlp_ln_weights, i * H)));
        MKB_TRY(gemm(b.act, at(g.gate_proj_weights, i * F * H), n, F, H, GemmEpilogue::silu(b.ffn, F), at(g.up_proj_weights, i * F * H)));
        MKB_TRY(gemm(b.ffn, at(g.down_proj_weights, i * H * F), n, H, F, GemmEpilogue::add_fixed(b.sums, H)));
    }
    if (p.want_logits) {
        MKB_TRY(norm(n - 1, 1, false, reinterpret_cast<long long*>(g.residual_acc), at(g.lm_head_norm_weights, 0)));
        MKB_TRY(gemm(b.act, at(g.lm_head_weights, 0), 1, g.vocab_size, H, GemmEpilogue::to(g.logits, g.vocab_size)));
    }
    return cudaSuccess;
}

}  // namespace mkb
