// Prompts of llama models: tokens at once (llama_prompt.cu).
#pragma once
#include "mk_common.cuh"

namespace mkb {

// Layout of a prompt's workspace, every part 256-byte aligned.
struct PromptBuffers {
    long long* sums;  // what the layers have added to the embeddings, in the decode kernel's fixed-point format
    __nv_bfloat16 *act, *q, *ffn;
    size_t total = 0;
    PromptBuffers(const MkbGlobals& g, int tokens, void* base) {
        char* b = static_cast<char*>(base);
        auto take = [&](size_t row_bytes) {
            char* at = b ? b + total : nullptr;
            total += ((size_t)tokens * row_bytes + 255) / 256 * 256;
            return at;
        };
        const size_t heads = (size_t)g.num_attention_heads * g.head_dim, hidden = g.hidden_size;
        sums = reinterpret_cast<long long*>(take(hidden * 8));
        act = reinterpret_cast<__nv_bfloat16*>(take((hidden > heads ? hidden : heads) * 2));
        q = reinterpret_cast<__nv_bfloat16*>(take(heads * 2));
        ffn = reinterpret_cast<__nv_bfloat16*>(take((size_t)g.intermediate_size * 2));
    }
};

cudaError_t prompt_launch(const MkbGlobals& g, const MkbPrompt& p, int* status, cudaStream_t stream);

}  // namespace mkb
