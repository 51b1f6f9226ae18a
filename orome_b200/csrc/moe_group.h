// moe_group.h -- expert products of token batches, tokens grouped by expert (defined in moe_group.cu).
#pragma once
#include "ctx.h"

bool orome_moe_group_supported(int fmt, uint32_t in_dim);
// Gate/up (+ SwiGLU) into act [t][K][inter] and / or down + weighted sum into out.  Requires 16-byte aligned x and act,
// ldx a multiple of 4.  OROME_ENOTSUP: there is no memory for the call's scratch; nothing was launched.
int orome_moe_group(orome_cuda_ctx *c, const OromeExpertLayerRef *L, int layout, bool gate_up, bool down, const float *x, int n_tokens, int ldx,
                    const uint32_t *idx, const float *w, uint32_t K, uint32_t hidden, uint32_t inter, float *act, float *out, int ldo, cudaStream_t st);
