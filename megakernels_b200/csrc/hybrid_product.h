// One matrix product of the prefill by itself, for the tests: not part of the library's interface (include/mkb200_hybrid.h), it
// may change with the kernels.
#pragma once
#include <stdint.h>

extern "C" {

/*
 * One matrix product of the prefill: out[t, n] = sum_k a[t, k] w[n, k], rows 16-byte aligned, in both dtypes.
 * MKBH_STORE: out (float) = sum + bias[n]; MKBH_ADD: out (float) += scale[n] * sum; MKBH_CAST: out = sum in the
 * dtype; MKBH_GLU: out[t, n / 2] = the clamped gated unit of columns n (gate, even) and n + 1; MKBH_SILU (bf16):
 * out = silu(sum) times the product with w2.  bias and scale may be NULL.
 */
enum { MKBH_STORE = 0, MKBH_ADD = 1, MKBH_CAST = 2, MKBH_GLU = 3, MKBH_SILU = 4 };
typedef struct MkbhProduct {
    uint32_t struct_bytes;
    int32_t dtype, result, tokens, features, inner;
    int64_t lda, ldw, ldo; /* elements between rows */
    const void *a, *w, *w2;
    const float *bias, *scale;
    float limit, alpha;
    void *out;
    int32_t *status; /* MKBH_STATUS_WORDS */
} MkbhProduct;
int mkb_hybrid_product(const MkbhProduct *p, void *cuda_stream);

}  // extern "C"
