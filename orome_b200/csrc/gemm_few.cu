// gemm_few.cu -- host side of the batched form for few vectors.
#include "gemm.h"

#include <algorithm>
#include <cstring>

#include "gemm_few.cuh"

using namespace orome;
#define fail orome_fail

template <int FMT, int NT, bool SWIGLU>
static int launch_inst(orome_cuda_ctx *c, const GfArgs &a, int grid, size_t smem, cudaStream_t st)
{
    auto kern = gemm_few_kernel<FMT, NT, SWIGLU>;
    static bool configured[64] = {false};
    if (!configured[c->device]) {
        cudaFuncAttributes fa;
        CU(cudaFuncGetAttributes(&fa, kern));
        CU(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, c->smem_optin - (int)fa.sharedSizeBytes));
        configured[c->device] = true;
    }
    return orome_launch_pdl_smem(c, "gemm_few", kern, dim3(grid), dim3((a.rt * a.kp + gf_loaders(NT) + 1) * 32), smem, st, a);
}
template <int FMT, bool SWIGLU>
static int launch_nt(orome_cuda_ctx *c, const GfArgs &a, uint32_t nt, int grid, size_t smem, cudaStream_t st)
{
    switch (nt) {
    case 1: return launch_inst<FMT, 1, SWIGLU>(c, a, grid, smem, st);
    case 2: return launch_inst<FMT, 2, SWIGLU>(c, a, grid, smem, st);
    case 3: return launch_inst<FMT, 3, SWIGLU>(c, a, grid, smem, st);
    default: return launch_inst<FMT, 4, SWIGLU>(c, a, grid, smem, st);
    }
}
template <int FMT>
static int launch_fmt(orome_cuda_ctx *c, const GfArgs &a, uint32_t nt, int grid, size_t smem, cudaStream_t st)
{
    return a.w1 ? launch_nt<FMT, true>(c, a, nt, grid, smem, st) : launch_nt<FMT, false>(c, a, nt, grid, smem, st);
}

// CTAs take equal row ranges; a pass covers up to eight row tiles (16 rows; fused: 8 of gate and 8 of up).
static uint32_t few_grid(const orome_cuda_ctx *c, uint32_t out_dim, uint32_t trows) { return std::max(1u, std::min((uint32_t)c->sm_count, (out_dim + trows - 1) / trows)); }
static uint32_t few_tiles(const orome_cuda_ctx *c, uint32_t out_dim, uint32_t trows)
{
    const uint32_t grid = few_grid(c, out_dim, trows);
    return ((out_dim + grid - 1) / grid + trows - 1) / trows;
}

// Where this form is the faster one: a cost model in us, fitted to 136 products (4 formats, 0.5 to 85 million weights, 4 to 32 vectors).
// This form: ~3.5 and so much a piece (row tile x chunk) of the busiest CTA, by format and groups of eight vectors; the
// tensor-memory form: ~7 and so much per 2^20 weights, which hardly depends on the vectors here; fused, it is two products and a
// pass.  Measured, this form / the other: Q4_K 1024x2560 at 12 vectors 4.4 / 6.8, 9728x2560 at 32 11.8 / 13.9, 17408x5120 at 4 20.9 /
// 22.0 and at 32 27.3 / 22.5, Q8_0 12288x4096 at 8 15.0 / 19.6, gate/up 512x2048 at 12 5.3 / 16.8, 9728x2560 at 12 20.5 / 31.6.
// (5 % margin: where the two are that close it does not matter.)
static bool few_faster(const orome_cuda_ctx *c, int fmt, uint32_t out_dim, uint32_t in_dim, uint32_t nt, bool fused)
{
    const double piece = fmt == FMT_Q8_0 ? 0.110 + 0.018 * nt : fmt == FMT_Q4_K ? 0.095 + 0.0145 * nt : fmt == FMT_Q5_K ? 0.100 + 0.019 * nt : 0.155 + 0.016 * nt;
    const double mega = fmt == FMT_Q8_0 ? 0.24 : fmt == FMT_Q4_K ? 0.21 : fmt == FMT_Q5_K ? 0.235 : 0.335;
    const double few = 3.5 + piece * few_tiles(c, out_dim, fused ? 8u : 16u) * (in_dim / TC_KC), pair = 7.0 + mega * ((double)out_dim * in_dim / 1048576.0);
    return 1.05 * few < (fused ? 2.0 * pair + 3.0 : pair);
}

bool orome_few_supported(const orome_cuda_ctx *c, int fmt, uint32_t out_dim, uint32_t in_dim, int batch, bool fused)
{
    if (fused && batch > 8) return false;
    return batch <= GF_MAX_VECTORS && !c->tc_slabs && !c->tc_split && orome_tc_supported(c, fmt, in_dim) &&
           few_faster(c, fmt, out_dim, in_dim, ((uint32_t)batch + 7) / 8, fused);
}

int orome_launch_few(orome_cuda_ctx *c, int fmt, const uint8_t *w0, const uint8_t *w1, uint32_t out_dim, uint32_t in_dim, int layout, const float *x,
                     int batch, int ldx, float *y, int ldy, cudaStream_t st, bool packed)
{
    const uint32_t nt = ((uint32_t)batch + 7) / 8, chunks = in_dim / TC_KC, trows = w1 ? 8u : 16u;
    const size_t xp_floats = (size_t)in_dim * nt * 4 + 64;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    CU(cudaStreamIsCapturing(st, &cap));
    // no room for X, or none to be had during a capture: the form that slices its X finds its own way
    if (cap != cudaStreamCaptureStatusNone && c->tc_xp.cap < xp_floats) return OROME_ENOTSUP;
    int rc = orome_ensure(c, c->tc_xp, xp_floats, st, (size_t)8 << 20);
    if (rc) return rc == OROME_ENOMEM ? OROME_ENOTSUP : rc;
    if (cap == cudaStreamCaptureStatusNone && !c->tc_part.cap) {
        rc = orome_reserve(c, c->tc_part, orome_tc_part_floats(c, fmt, out_dim, in_dim, batch), st, tp_part_usual(c));
        if (rc) return rc;
    }
    GfArgs a;
    memset(&a, 0, sizeof a);
    // the warps that a pass's row tiles leave split the chunks of a row
    const uint32_t grid = few_grid(c, out_dim, trows), tiles = few_tiles(c, out_dim, trows), passes = (tiles + 7) / 8;
    a.rt = (tiles + passes - 1) / passes;
    const size_t room = (size_t)c->smem_optin - 1024;
    for (uint32_t kp = std::min((uint32_t)GF_MAX_WARPS / a.rt, chunks);; --kp) {
        const uint32_t steps = (chunks + kp - 1) / kp;
        a.kp = (chunks + steps - 1) / steps;
        a.stage_bytes = a.rt * 16 * a.kp * gf_pitch(fmt) + a.kp * nt * GF_X_CHUNK;
        a.stage_base = (a.kp > 1 ? a.rt * a.kp * nt * 512u : 0u);
        a.nstages = a.stage_base + (size_t)a.stage_bytes <= room ? (uint32_t)std::min<size_t>(GF_MAX_STAGES, (room - a.stage_base) / a.stage_bytes) : 0u;
        a.nstages = std::min(a.nstages, steps * passes);
        if (a.nstages >= std::min(2u, steps * passes) || kp == 1) break;      // two stages at least, so that loads and products overlap
    }
    if (!a.nstages) return OROME_ENOTSUP;
    if (!packed) {
        rc = orome_launch_pdl(c, "pack_x_few", pack_x_few_kernel, dim3((in_dim / 8 + 255) / 256, nt * 8), dim3(256), st, x, (uint32_t)batch, (uint32_t)ldx, in_dim, nt,
                              reinterpret_cast<uint4 *>(c->tc_xp.p));
        if (rc) return rc;
    }
    a.w0 = w0; a.w1 = w1; a.xp = reinterpret_cast<const uint8_t *>(c->tc_xp.p); a.y = y;
    a.rows = out_dim; a.row_bytes = (uint32_t)row_bytes_of(fmt, in_dim); a.w_bytes = (uint64_t)a.row_bytes * out_dim;
    a.batch = (uint32_t)batch; a.ldy = (uint32_t)ldy; a.chunks = chunks;
    a.layout = layout; a.status = c->status_dev;
    const size_t smem = a.stage_base + (size_t)a.nstages * a.stage_bytes;
    switch (fmt) {
    case FMT_Q8_0: return launch_fmt<FMT_Q8_0>(c, a, nt, (int)grid, smem, st);
    case FMT_Q4_K: return launch_fmt<FMT_Q4_K>(c, a, nt, (int)grid, smem, st);
    case FMT_Q5_K: return launch_fmt<FMT_Q5_K>(c, a, nt, (int)grid, smem, st);
    default: return launch_fmt<FMT_Q6_K>(c, a, nt, (int)grid, smem, st);
    }
}
