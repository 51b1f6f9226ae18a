// gemm_few.cu -- host side of the batched form for few vectors.
#include "gemm.h"

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
template <int FMT>
static int launch_nt(orome_cuda_ctx *c, const GfArgs &a, uint32_t nt, int grid, size_t smem, cudaStream_t st)
{
    switch (nt) {
    case 1: return launch_inst<FMT, 1, false>(c, a, grid, smem, st);
    case 2: return launch_inst<FMT, 2, false>(c, a, grid, smem, st);
    case 3: return launch_inst<FMT, 3, false>(c, a, grid, smem, st);
    default: return launch_inst<FMT, 4, false>(c, a, grid, smem, st);
    }
}
template <int FMT>
static int launch_fmt(orome_cuda_ctx *c, const GfArgs &a, uint32_t nt, int grid, size_t smem, cudaStream_t st)
{
    return a.w1 ? launch_inst<FMT, 1, true>(c, a, grid, smem, st) : launch_nt<FMT>(c, a, nt, grid, smem, st);
}

static FewShape few_shape(const orome_cuda_ctx *c, int fmt, uint32_t out_dim, uint32_t in_dim, int batch, bool fused)
{
    return FewShape{fmt, out_dim, in_dim, (uint32_t)batch, fused, (uint32_t)c->sm_count, (size_t)c->smem_optin};
}

bool orome_few_supported(const orome_cuda_ctx *c, int fmt, uint32_t out_dim, uint32_t in_dim, int batch, bool fused)
{
    if (fused && batch > 8) return false;        // the fused form exists for one group of eight
    return batch <= GF_MAX_VECTORS && !c->tc_slabs && !c->tc_split && orome_tc_supported(c, fmt, in_dim) &&
           few_faster(few_shape(c, fmt, out_dim, in_dim, batch, fused));
}

int orome_launch_few(orome_cuda_ctx *c, int fmt, const uint8_t *w0, const uint8_t *w1, uint32_t out_dim, uint32_t in_dim, int layout, const float *x,
                     int batch, int ldx, float *y, int ldy, cudaStream_t st, bool packed)
{
    const uint32_t nt = few_groups((uint32_t)batch);
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
    FewPlan p;
    if (!few_plan(few_shape(c, fmt, out_dim, in_dim, batch, w1 != nullptr), p)) return OROME_ENOTSUP;
    a.rt = p.rt; a.kp = p.kp; a.nstages = p.nstages; a.red_base = 0; a.stage_base = p.stage_base; a.stage_bytes = p.stage_bytes;
    if (!packed) {
        rc = orome_launch_pdl(c, "pack_x_few", pack_x_few_kernel, dim3((in_dim / 8 + 255) / 256, nt * 8), dim3(256), st, x, (uint32_t)batch, (uint32_t)ldx, in_dim, nt,
                              reinterpret_cast<uint4 *>(c->tc_xp.p));
        if (rc) return rc;
    }
    a.w0 = w0; a.w1 = w1; a.xp = reinterpret_cast<const uint8_t *>(c->tc_xp.p); a.y = y;
    a.rows = out_dim; a.row_bytes = (uint32_t)row_bytes_of(fmt, in_dim); a.w_bytes = (uint64_t)a.row_bytes * out_dim;
    a.batch = (uint32_t)batch; a.ldy = (uint32_t)ldy; a.chunks = in_dim / GF_KC;
    a.layout = layout; a.status = c->status_dev;
    switch (fmt) {
    case FMT_Q8_0: return launch_fmt<FMT_Q8_0>(c, a, nt, (int)p.grid, p.bytes, st);
    case FMT_Q4_K: return launch_fmt<FMT_Q4_K>(c, a, nt, (int)p.grid, p.bytes, st);
    case FMT_Q5_K: return launch_fmt<FMT_Q5_K>(c, a, nt, (int)p.grid, p.bytes, st);
    default: return launch_fmt<FMT_Q6_K>(c, a, nt, (int)p.grid, p.bytes, st);
    }
}
