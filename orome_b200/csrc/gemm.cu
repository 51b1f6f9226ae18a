// gemm.cu -- host side of the batched (prefill) form: packing X, the tensor-core product, the reduction of cut tiles.
#include "gemm.h"

#include <algorithm>
#include <cstring>

#include "gemm_pair.cuh"
#include "gemm_tc.cuh"

using namespace orome;
#define fail orome_fail

// Q6_K (rows only 2-byte aligned, no tensor map possible) exists in the tensor-memory form only.
bool orome_tc_supported(const orome_cuda_ctx *c, int fmt, uint32_t in_dim)
{
    if (in_dim % TC_KC != 0) return false;
    return fmt == FMT_Q8_0 || fmt == FMT_Q4_K || fmt == FMT_Q5_K || (fmt == FMT_Q6_K && !c->tc_slabs);
}

template <typename K>
static int allow_smem(orome_cuda_ctx *c, K kern, bool (&configured)[64])
{
    if (configured[c->device]) return OROME_OK;
    cudaFuncAttributes fa;
    CU(cudaFuncGetAttributes(&fa, kern));
    CU(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, c->smem_optin - (int)fa.sharedSizeBytes));
    configured[c->device] = true;
    return OROME_OK;
}

template <int FMT, bool BIG, bool PUB>
static int launch_pair_inst(orome_cuda_ctx *c, const TpArgs &a, size_t smem, cudaStream_t st)
{
    static bool configured[64] = {false};
    int rc = allow_smem(c, gemm_pair_kernel<FMT, BIG, PUB>, configured);
    if (rc) return rc;
    return orome_launch_pdl_smem(c, "gemm_pair", gemm_pair_kernel<FMT, BIG, PUB>, dim3(2 * a.clusters), dim3(TP_THREADS), smem, st, a);
}
template <int FMT>
static int launch_pair_fmt(orome_cuda_ctx *c, const TpArgs &a, size_t smem, cudaStream_t st)
{
    static_assert(TC_MAX_N <= 128, "a published product fits the smaller tiles");
    if (a.pub.npeers > 0) return launch_pair_inst<FMT, false, true>(c, a, smem, st);
    return a.nt_rows > 128 ? launch_pair_inst<FMT, true, false>(c, a, smem, st) : launch_pair_inst<FMT, false, false>(c, a, smem, st);
}

template <int FMT>
static int launch_tc_fmt(orome_cuda_ctx *c, const TcArgs &a, int grid, size_t smem, cudaStream_t st)
{
    static bool configured[64] = {false};
    int rc = allow_smem(c, gemm_tc_kernel<FMT>, configured);
    if (rc) return rc;
    return orome_launch_pdl_smem(c, "gemm_tc", gemm_tc_kernel<FMT>, dim3(grid), dim3(TC_THREADS), smem, st, a);
}

static uint32_t tc_chunk_bytes(int fmt) { return fmt == FMT_Q8_0 ? 272u : fmt == FMT_Q4_K ? 144u : fmt == FMT_Q5_K ? 176u : 210u; }

static int launch_pack(orome_cuda_ctx *c, const float *x, int nb, int ldx, uint32_t in_dim, uint32_t nt_rows, uint32_t ntiles, const uint2 *x_ll,
                       const unsigned int *wait_gen, cudaStream_t st)
{
    return orome_launch_pdl(c, "pack_x_f16", pack_x_f16_kernel, dim3((in_dim / 8 + 255) / 256, nt_rows * ntiles), dim3(256), st, x, nb, ldx, in_dim, nt_rows,
                            reinterpret_cast<__half *>(c->tc_xp.p), x_ll, wait_gen, orome_wait_cycles(c), c->status_dev);
}

// The form staged in shared memory (OROME_OPT_TC_SLABS): slices of TC_MAX_N vectors, each of which reads the weights again.
static int launch_staged(orome_cuda_ctx *c, int fmt, const uint8_t *data, uint32_t out_dim, uint32_t in_dim, int layout, const float *x,
                         int batch, int ldx, float *y, int ldy, cudaStream_t st, const TcPub *pub, const uint2 *x_ll, const unsigned int *wait_gen)
{
    const uint32_t chunk_bytes = tc_chunk_bytes(fmt), chunks = in_dim / TC_KC, tiles = (out_dim + TC_M - 1) / TC_M;
    // Split K so that the SMs stay busy: a CTA costs about one time unit per chunk plus about five to set up (TMEM,
    // barriers, pipeline fill -- measured: three parts in two waves were slower than one part on 96 of 148 SMs), the
    // grid runs in waves of sm_count CTAs, a split adds a reduction pass.  Parts may be uneven.
    uint32_t split = 1;
    double best = 1e30;
    for (uint32_t s = c->tc_split ? (uint32_t)c->tc_split : 1u; s <= (c->tc_split ? (uint32_t)c->tc_split : 12u) && s <= chunks; ++s) {
        const uint32_t ctas = tiles * s, waves = (ctas + c->sm_count - 1) / c->sm_count;
        const double cost = (double)waves * ((double)((chunks + s - 1) / s) + 5.0) + (s > 1 ? 1.0 + 0.25 * s : 0.0);
        if (cost < best) { best = cost; split = s; }
    }
    for (int b0 = 0; b0 < batch; b0 += TC_MAX_N) {
        const int nb = std::min(batch - b0, TC_MAX_N);
        const uint32_t npad = (uint32_t)(nb + 15) / 16 * 16;
        int rc = orome_ensure(c, c->tc_xp, (size_t)in_dim * npad / 2 + 64, st);
        if (rc) return rc;
        if (split > 1) { rc = orome_ensure(c, c->tc_part, (size_t)split * nb * out_dim, st); if (rc) return rc; }
        rc = launch_pack(c, x + (size_t)b0 * ldx, nb, ldx, in_dim, npad, 1, x_ll, wait_gen, st);
        if (rc) return rc;
        TcArgs a;
        memset(&a, 0, sizeof a);
        EncodeTiledFn enc = orome_encode_tiled_fn();      // packed weights arrive by tensor copies
        if (!enc) return fail(OROME_ECUDA, "gemm_tc: cuTensorMapEncodeTiled is not available");
        const cuuint64_t dims[2] = {(cuuint64_t)row_bytes_of(fmt, in_dim) / 4, out_dim};
        const cuuint64_t strides[1] = {(cuuint64_t)row_bytes_of(fmt, in_dim)};
        const cuuint32_t box[2] = {chunk_bytes / 4, (cuuint32_t)TC_M}, estr[2] = {1, 1};
        CUresult r = enc(&a.wmap, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, const_cast<uint8_t *>(data), dims, strides, box, estr,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) return fail(OROME_ECUDA, "gemm_tc: cuTensorMapEncodeTiled failed (%d)", (int)r);
        a.w = data; a.xp = reinterpret_cast<__half *>(c->tc_xp.p); a.y = split == 1 ? y + (size_t)b0 * ldy : c->tc_part.p;
        a.rows = out_dim; a.in_dim = in_dim; a.row_bytes = (uint32_t)row_bytes_of(fmt, in_dim); a.chunk_bytes = chunk_bytes;
        a.batch = (uint32_t)nb; a.npad = npad; a.ldy = (uint32_t)ldy; a.split = split; a.chunks = chunks;
        a.layout = layout; a.status = c->status_dev;
        a.pub = *pub;
        // Shared memory: one chunk's worth of fp16 slab buffers, two X tile stages, two packed-weight stages (169 KB for
        // Q4_K at batch 64); deeper rings measured slower (35-41 us against 34 us on Q4_K 12288x4096, batch 64).
        const size_t pk_stage = (TC_M * chunk_bytes + 127) & ~127u, b_tile = (size_t)npad * 128 * TC_SLABS;
        const size_t smem = 1024 + (size_t)TC_MAX_RING * 16384 + (size_t)TC_B_STAGES * b_tile + 512 + (size_t)tc_pk_stages(fmt) * pk_stage;
        if (smem > (size_t)c->smem_optin - 1024) return fail(OROME_ENOTSUP, "gemm_tc: batch %d does not fit shared memory", nb);
        const int grid = (int)(tiles * split);
        switch (fmt) {
        case FMT_Q8_0: rc = launch_tc_fmt<FMT_Q8_0>(c, a, grid, smem, st); break;
        case FMT_Q4_K: rc = launch_tc_fmt<FMT_Q4_K>(c, a, grid, smem, st); break;
        default: rc = launch_tc_fmt<FMT_Q5_K>(c, a, grid, smem, st); break;
        }
        if (rc) return rc;
        if (split > 1) {
            const size_t n = (size_t)nb * out_dim;
            rc = orome_launch_pdl(c, "splitk_reduce", splitk_reduce_kernel, dim3((unsigned)std::min<size_t>((n + 255) / 256, 1184)), dim3(256), st,
                                  (const float *)c->tc_part.p, split, (uint32_t)nb, out_dim, y + (size_t)b0 * ldy, (uint32_t)ldy, *pub);
            if (rc) return rc;
        }
    }
    return OROME_OK;
}

// How many clusters share the (tile, chunk) units.  In clocks: a unit costs the longest of its MMAs (8 a vector), its dequant
// (~1100) and its packed bytes at an SM's share of memory (~22 a clock); a share costs ~5000 to set up, fill and drain; cut
// tiles are written and read back at ~2000 bytes a clock and cost one more launch (~4000).  (896 products with their number of clusters
// swept: the choice is 5 % slower than the best count on average.  Equal parts of a tile are cheaper than this says, 4096 x 4096 at 128
// vectors 20.1 us as whole tiles, 15.3 in halves; models that know it made others slower, 12288 x 4096 at 2048 164 -> 180.)
static uint32_t tp_clusters(const orome_cuda_ctx *c, int fmt, uint32_t tiles, uint32_t chunks, uint32_t nt_rows, bool may_cut)
{
    const uint32_t pairs = std::max(1u, (uint32_t)c->sm_count / 2), units = tiles * chunks;
    if (c->tc_split) return tiles * std::min<uint32_t>((uint32_t)c->tc_split, chunks);
    const double unit = std::max({8.0 * nt_rows, 1100.0, 128.0 * tc_chunk_bytes(fmt) / 22.0});
    uint32_t pick = tiles;
    double best = (double)((tiles + pairs - 1) / pairs) * (chunks * unit + 5000.0);       // whole tiles, in waves
    if (!may_cut) return pick;
    for (uint32_t g = 1; g <= std::min(pairs, units); ++g) {
        const bool cut = ((uint64_t)units % g) != 0 || (units / g) % chunks != 0;
        const double slots = std::min<double>(2.0 * g, (double)g + tiles);
        const double cost = (double)((units + g - 1) / g) * unit + 5000.0 + (cut ? 4000.0 + slots * nt_rows * TP_ROWS * 8.0 / 2000.0 : 0.0);
        if (cost < best) { best = cost; pick = g; }
    }
    return pick;
}

size_t orome_tc_part_floats(const orome_cuda_ctx *c, int fmt, uint32_t out_dim, uint32_t in_dim, int batch)
{
    const uint32_t chunks = in_dim / TC_KC, tiles = (out_dim + TP_ROWS - 1) / TP_ROWS, nt_rows = ((uint32_t)batch + 15) / 16 * 16;
    const uint32_t units = tiles * chunks, clusters = tp_clusters(c, fmt, tiles, chunks, nt_rows, true);
    return units % clusters != 0 || (units / clusters) % chunks != 0 ? (size_t)clusters * 2 * nt_rows * TP_ROWS : 0;
}

int orome_launch_tc(orome_cuda_ctx *c, int fmt, const uint8_t *data, uint32_t out_dim, uint32_t in_dim, int layout, const float *x,
                    int batch, int ldx, float *y, int ldy, cudaStream_t st, const TcPub *pub, const uint2 *x_ll, const unsigned int *wait_gen, bool *x_packed)
{
    TcPub no_pub;
    memset(&no_pub, 0, sizeof no_pub);
    const bool single = !pub && !x_ll;
    if (!pub) pub = &no_pub;
    if (single && !x_packed && orome_few_supported(c, fmt, out_dim, in_dim, batch, false)) {
        const int rc = orome_launch_few(c, fmt, data, nullptr, out_dim, in_dim, layout, x, batch, ldx, y, ldy, st);
        if (rc != OROME_ENOTSUP) return rc;
    }
    if (c->tc_slabs) return launch_staged(c, fmt, data, out_dim, in_dim, layout, x, batch, ldx, y, ldy, st, pub, x_ll, wait_gen);
    const uint32_t chunks = in_dim / TC_KC, mtiles = (out_dim + TP_ROWS - 1) / TP_ROWS;
    // At most 4096 vectors a launch (bounds the packed X), fewer where the packed X of that many has no room: while a graph is
    // being captured, where no scratch can grow, as many as what is there holds; else half as many until there is room, down to
    // 64.  Tiles are not cut if their partial sums have no room.  A row-split product is never sliced: a launch publishes one
    // generation of the whole Y, and reads the gathered X from row 0 on.
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    CU(cudaStreamIsCapturing(st, &cap));
    const bool capturing = cap != cudaStreamCaptureStatusNone, one_launch = pub->npeers > 0 || x_ll;
    // A fixed number of parts cuts every tile, at most twelve ways: 64 vectors then bound the partial sums.
    int slice = std::min(batch, c->tc_split ? 64 : 4096), rc;
    auto padded = [](uint32_t nb) { const uint32_t nt = (nb + TP_MAX_N - 1) / TP_MAX_N; return ((nb + nt - 1) / nt + 15) / 16 * 16 * nt; };
    auto xp_floats = [&](int nb) { return (size_t)in_dim * padded((uint32_t)nb) / 2 + 64; };
    if (capturing && !one_launch && c->tc_xp.cap < xp_floats(slice) && c->tc_xp.cap >= xp_floats(16)) {
        const int most = slice;
        slice = 16;
        while (slice < most && xp_floats(slice + 16) <= c->tc_xp.cap) slice += 16;
    }
    // (first sizes: 32 MiB of packed X, 960 vectors of 17408, and all the partial sums that shares can leave, so that the products of
    // a layer do not each outgrow the one before)
    while ((rc = orome_ensure(c, c->tc_xp, xp_floats(slice), st, (size_t)8 << 20)) == OROME_ENOMEM && !capturing && !one_launch && slice > 64) slice = (slice / 2 + 63) / 64 * 64;
    if (rc) return rc;
    const bool packed = x_packed && *x_packed && slice >= batch;
    if (x_packed) *x_packed = slice >= batch;
    for (int b0 = 0; b0 < batch; b0 += slice) {
        const uint32_t nb = (uint32_t)std::min(batch - b0, slice);
        const uint32_t ntiles = (nb + TP_MAX_N - 1) / TP_MAX_N, nt_rows = ((nb + ntiles - 1) / ntiles + 15) / 16 * 16;
        TpArgs a;
        memset(&a, 0, sizeof a);
        a.slots = c->tc_split ? 1 : 2;      // a fixed number of parts never crosses a tile's end
        auto part_floats = [&](uint32_t clusters) { return (size_t)clusters * a.slots * nt_rows * TP_ROWS; };
        a.chunks = chunks;
        a.units = chunks * mtiles * ntiles;
        a.clusters = tp_clusters(c, fmt, mtiles * ntiles, chunks, nt_rows, true);
        auto is_cut = [&]() { return a.units % a.clusters != 0 || (a.units / a.clusters) % chunks != 0; };
        if (is_cut()) {
            rc = capturing && part_floats(a.clusters) > c->tc_part.cap ? OROME_ENOMEM : orome_ensure(c, c->tc_part, part_floats(a.clusters), st, tp_part_usual(c));
            if (rc == OROME_ENOMEM) {
                a.clusters = tp_clusters(c, fmt, mtiles * ntiles, chunks, nt_rows, false);
                rc = is_cut() ? orome_ensure(c, c->tc_part, part_floats(a.clusters), st) : OROME_OK;      // (a fixed number of parts)
            }
            if (rc) return rc;
        }
        const bool cut = is_cut();
        if (!packed) {
            rc = launch_pack(c, x + (size_t)b0 * ldx, (int)nb, ldx, in_dim, nt_rows / 2, 2 * ntiles, x_ll, wait_gen, st);      // a CTA's half of a tile lies together
            if (rc) return rc;
        }
        a.w = data; a.xp = reinterpret_cast<const __half *>(c->tc_xp.p); a.y = y + (size_t)b0 * ldy; a.part = c->tc_part.p;
        a.rows = out_dim; a.row_bytes = (uint32_t)row_bytes_of(fmt, in_dim); a.w_bytes = (uint64_t)a.row_bytes * out_dim;
        a.batch = nb; a.nt_rows = nt_rows; a.ntiles = ntiles; a.ldy = (uint32_t)ldy;
        a.publish_done = !cut;
        a.layout = layout; a.status = c->status_dev;
        a.pub = *pub;
        // Rings: four X stages of 128 k (256 up to 128 vectors), 128 KiB from 128 vectors on, more of them below, at least 32 KiB;
        // the rest for packed weights (two 34-KiB stages of Q8_0 at 256 vectors, five of Q4_K; six of anything where there is
        // room).  At least half an SM's shared memory, so that two CTAs (each takes all of tensor memory) never share an SM.
        const size_t x_stage = (size_t)nt_rows * 64 * (nt_rows > 128 ? 2 : 4), stage = tp_stage_bytes(fmt), room = (size_t)c->smem_optin - 1024 - 1024 - 512;
        a.bs = (uint32_t)std::max<size_t>(4, std::min<size_t>(8, 65536 / x_stage));
        a.ws = (uint32_t)std::min<size_t>(TP_MAX_WS, (room - a.bs * x_stage) / stage);
        const size_t smem = std::max<size_t>(1024 + a.bs * x_stage + a.ws * stage + 512, 120 * 1024);
        switch (fmt) {
        case FMT_Q8_0: rc = launch_pair_fmt<FMT_Q8_0>(c, a, smem, st); break;
        case FMT_Q4_K: rc = launch_pair_fmt<FMT_Q4_K>(c, a, smem, st); break;
        case FMT_Q5_K: rc = launch_pair_fmt<FMT_Q5_K>(c, a, smem, st); break;
        default: rc = launch_pair_fmt<FMT_Q6_K>(c, a, smem, st); break;
        }
        if (rc) return rc;
        if (cut) {
            rc = orome_launch_pdl(c, "tile_reduce", tile_reduce_kernel, dim3(mtiles * ntiles, nt_rows / 4), dim3(256), st, a);
            if (rc) return rc;
        }
    }
    return OROME_OK;
}
