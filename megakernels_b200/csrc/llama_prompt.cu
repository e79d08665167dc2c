// A prompt of a llama model, all tokens at once: the layers' matrix products on the 5th-generation tensor
// cores with the rotation, the cache append and the gated unit as epilogues, attention over the cache.
// Seven launches a layer.  501 tokens at the 1B widths (16 layers): 354.6 ms as a decode step per token, bound by the
// weights that every token streams again; 2.1 ms at once, bound by the products and the 118 launches' hand-over.  The residual stream is 32-bit; operands of the products are bf16, as in decoding.
#include "llama_prompt.h"

#include "hybrid_kernels.h"

namespace mkb {
namespace {

using mkbh::bf16;
using mkbh::GemmEpilogue;

constexpr int kNormThreads = 256, kKept = 8;  // float4s of a row per thread: widths up to 8192

// out = x / rms(x) * w, a block per row.  `first`: the rows of x are taken from the embeddings and stored.
__global__ void __launch_bounds__(kNormThreads) prompt_norm_kernel(const bf16* first, float* x, int width, float eps, const bf16* __restrict__ w,
                                                                   bf16* out) {
    __shared__ float red[kNormThreads / 32];
    mkbh::let_next();
    mkbh::after_previous();
    const size_t row = (size_t)blockIdx.x * width;
    float4 v[kKept];
    float s[1] = {0.f};
#pragma unroll
    for (int k = 0; k < kKept; ++k) {
        const int i = 4 * (threadIdx.x + k * kNormThreads);
        v[k] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (i >= width) continue;
        if (first != nullptr) {
            const uint2 e = *reinterpret_cast<const uint2*>(first + row + i);
            v[k] = make_float4(bf16_lo(e.x), bf16_hi(e.x), bf16_lo(e.y), bf16_hi(e.y));
            *reinterpret_cast<float4*>(x + row + i) = v[k];
        } else {
            v[k] = *reinterpret_cast<const float4*>(x + row + i);
        }
        s[0] += v[k].x * v[k].x + v[k].y * v[k].y + v[k].z * v[k].z + v[k].w * v[k].w;
    }
    mkbh::block_sum<1, kNormThreads>(s, red);
    const float inv = 1.f / sqrtf(s[0] / width + eps);
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
    auto at = [](const void* w, size_t elements) { return static_cast<const bf16*>(w) + elements; };
    auto norm = [&](const bf16* first, int rows, const bf16* w, float* x) {
        cudaLaunchConfig_t c = {};
        c.gridDim = dim3(rows);
        c.blockDim = dim3(kNormThreads);
        c.stream = s;
        cudaLaunchAttribute early = mkbh::may_begin_early();
        c.attrs = &early;
        c.numAttrs = 1;
        return cudaLaunchKernelEx(&c, prompt_norm_kernel, first, x, H, g.rms_norm_eps, w, b.act);
    };
    auto gemm = [&](const bf16* A, const bf16* W, int rows, int N, int K, const GemmEpilogue& e, const bf16* W2 = nullptr) {
        return mkbh::gemm_bf16(A, K, W, K, rows, N, K, e, status, s, W2);
    };
    for (size_t i = 0; i < (size_t)g.num_layers; ++i) {
        const size_t cache = i * g.kv_batch * g.kv_max_len * KV;
        bf16 *k = static_cast<bf16*>(g.k_cache) + cache, *v = static_cast<bf16*>(g.v_cache) + cache;
        MKB_TRY(norm(i == 0 ? static_cast<const bf16*>(p.hidden) : nullptr, n, at(g.attn_ln_weights, i * H), b.x));
        MKB_TRY(gemm(b.act, at(g.qkv_weights, i * (Q + 2 * KV) * H), n, Q + 2 * KV, H,
                     GemmEpilogue::rotate({b.q, k, v, Q, KV, D, p.pos0, static_cast<const float*>(g.rope_cos), static_cast<const float*>(g.rope_sin)})));
        MKB_TRY(mkbh::flash_cache({b.q, k, v, b.act, n, p.pos0, g.num_attention_heads, g.num_kv_heads, D, g.attn_scale, status}, s));
        MKB_TRY(gemm(b.act, at(g.o_proj_weights, i * H * Q), n, H, Q, GemmEpilogue::add(b.x, H, nullptr)));
        MKB_TRY(norm(nullptr, n, at(g.mlp_ln_weights, i * H), b.x));
        MKB_TRY(gemm(b.act, at(g.gate_proj_weights, i * F * H), n, F, H, GemmEpilogue::silu(b.ffn, F), at(g.up_proj_weights, i * F * H)));
        MKB_TRY(gemm(b.ffn, at(g.down_proj_weights, i * H * F), n, H, F, GemmEpilogue::add(b.x, H, nullptr)));
    }
    if (p.want_logits) {
        MKB_TRY(norm(nullptr, 1, at(g.lm_head_norm_weights, 0), b.x + (size_t)(n - 1) * H));
        MKB_TRY(gemm(b.act, at(g.lm_head_weights, 0), 1, g.vocab_size, H, GemmEpilogue::to(g.logits, g.vocab_size)));
    }
    return cudaSuccess;
}

}  // namespace mkb
