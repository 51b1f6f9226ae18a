// gemm.h -- the batched form's launches (defined in gemm.cu).
#pragma once
#include "ctx.h"

#include "gemv_pipe.cuh"

namespace orome {
constexpr int TC_MAX_N = 64;         // input vectors per launch of the staged form, and of a row-split product on several GPUs

// Row-split form on several GPUs (the batched counterpart of the publish fields of PipeArgs): every Y value also
// goes, as a {value, tag} slot, into this rank's and every peer's copy of the gather arena.
struct TcPub {
    int npeers;                               // 0: single GPU, nothing is published
    long long peer_delta[PIPE_MAX_PEERS];
    const uint8_t *arena_base;
    uint8_t *ll_origin;
    unsigned int *pub_gen, *pub_arrived;
};
}  // namespace orome

// Partial sums that the tensor-memory form's shares of a product leave (at most 256 vectors; 0: no tile is cut), and the most that any
// leave: two tiles of 256 x 256 per pair of SMs.
size_t orome_tc_part_floats(const orome_cuda_ctx *c, int fmt, uint32_t out_dim, uint32_t in_dim, int batch);
inline size_t tp_part_usual(const orome_cuda_ctx *c) { return (size_t)(c->sm_count < 2 ? 1 : c->sm_count / 2) * 2 * 256 * 256; }

bool orome_tc_supported(const orome_cuda_ctx *c, int fmt, uint32_t in_dim);
// Y[b][r] for b < batch.  pub / x_ll / wait_gen: the row-split form on several GPUs (batch <= TC_MAX_N, one launch): Y is
// published to every rank's arena by the kernel that writes it, a gathered X is read from its slots by the packing kernel.
// x_packed (never with pub; the tensor-memory form is then the one taken): in, X is the one the previous call on the stream packed; out,
// all of it lies packed in scratch.
int orome_launch_tc(orome_cuda_ctx *c, int fmt, const uint8_t *data, uint32_t out_dim, uint32_t in_dim, int layout, const float *x,
                    int batch, int ldx, float *y, int ldy, cudaStream_t st, const orome::TcPub *pub = nullptr, const uint2 *x_ll = nullptr,
                    const unsigned int *wait_gen = nullptr, bool *x_packed = nullptr);

// Few vectors (gemm_few.cuh): Y, or with w1 (at most eight vectors) silu(W0 x) * (W1 x), in one launch behind the packing of X.  packed: X
// is the one the previous launch on the stream has packed.  OROME_ENOTSUP: no scratch for X.
bool orome_few_supported(const orome_cuda_ctx *c, int fmt, uint32_t out_dim, uint32_t in_dim, int batch, bool fused);      // ... and the faster form there
int orome_launch_few(orome_cuda_ctx *c, int fmt, const uint8_t *w0, const uint8_t *w1, uint32_t out_dim, uint32_t in_dim, int layout, const float *x,
                     int batch, int ldx, float *y, int ldy, cudaStream_t st, bool packed = false);
