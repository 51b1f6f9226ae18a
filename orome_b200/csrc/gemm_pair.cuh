// gemm_pair.cuh -- the batched (prefill) form: dequantized weights in TENSOR MEMORY, two SMs on one tile.
//
//   Y[b][r] = sum_c W[r][c] * X[b][c], W block-quantized, X rounded to fp16 once (pack_x_f16_kernel), fp32 accumulators.
//
// A cluster of two CTAs computes 256 rows x up to 256 input vectors with tcgen05.mma.cta_group::2 (each CTA: 128 rows of the
// weights, half of the vectors), so a packed weight is read and dequantized once per 256 vectors instead of once per 64, and
// an X tile crosses the L2 once per 256 rows.  Roles of a CTA:
//
//   4 loader warps     packed weights, 128 rows x 256 weights a stage, as 16-byte cp.async in row order: consecutive lanes
//                      copy consecutive pieces of a row (a warp touches two or three rows).  Reading the pieces where they
//                      are converted (lane = row) costs one L1 line per lane and load: that form needed ~3600 clocks a
//                      stage and set its pace (12288 x 4096 Q8_0, 8 vectors: 31 us on 96 SMs); a tensor copy of the same
//                      box took ~2100.  Stage rows are an odd number of 16-byte pieces apart, so that the per-row reads
//                      below are free of bank conflicts.
//   16 dequant warps   lane = row: 64 weights a thread, shared memory -> fp16 (bias removed exactly, one HFMA2 per two
//                      weights) -> tensor memory (two weights per column, stages of 128 columns).  ~650 issue slots per SM
//                      sub-partition and stage, against 2048 clocks of MMA at 256 vectors.
//   1 X producer       bulk copies of this CTA's half of the X tile, 256 k (128 in tiles of more than 128 vectors) at a time
//   1 MMA warp         rank 0: issues 16 x (M256 x N x K16) per stage, A from both CTAs' tensor memory, B from both CTAs'
//                      shared memory.  Rank 1: passes "my half of X has landed" on to rank 0.
//
// Work: the (tile, 256-weight chunk) units of the whole product, tile-major, are cut into equal contiguous shares, one per
// cluster (one cluster per pair of SMs), so that no wave is left nearly empty whatever the shape.  A cluster whose share
// starts or ends inside a tile leaves that tile's partial sums in scratch (at most two a cluster) and tile_reduce_kernel adds
// them up in cluster order.  Every barrier wait is bounded (status code 4 on expiry).
#pragma once
#include "gemm_tc.cuh"

namespace orome {

constexpr int TP_LOADERS = 4;
constexpr int TP_W_MMA = TC_DEQ_WARPS, TP_W_X = TC_DEQ_WARPS + 1, TP_W_LOAD = TC_DEQ_WARPS + 2;
constexpr int TP_THREADS = (TC_DEQ_WARPS + 2 + TP_LOADERS) * 32;
constexpr int TP_MAX_N = 256;            // input vectors of a tile
constexpr int TP_MAX_WS = 6, TP_MAX_BS = 8, TP_MAX_AS = 3;
constexpr int TP_ROWS = 2 * TC_M;        // rows of a tile (a cluster)

// Pieces between rows: odd.
__host__ __device__ constexpr uint32_t tp_pitch(int fmt) { return 16u * (tp_pieces(fmt) | 1u); }
__host__ __device__ constexpr uint32_t tp_stage_bytes(int fmt) { return TC_M * tp_pitch(fmt); }

struct TpArgs {
    const uint8_t *w;
    const __half *xp;             // packed X: [half of an n tile][k slab of 64][nt_rows / 2][64] fp16, swizzled
    float *y;                     // [batch][ldy]
    float *part;                  // [cluster][slots][nt_rows][256]
    uint32_t slots;               // partial tiles a cluster may leave: 2, or 1 where every share lies inside one tile
    uint32_t rows, row_bytes;
    uint64_t w_bytes;
    uint32_t batch, nt_rows, ntiles, ldy;      // vectors of a tile (a multiple of 16), tiles of vectors
    uint32_t chunks, units, clusters;          // 256-weight chunks of a row; chunks * tiles; shares of the units
    uint32_t ws, bs;                           // ring sizes: weight stages, X stages
    uint32_t publish_done;                     // this kernel is the last writer of Y
    int layout;
    int *status;
    TcPub pub;
};

// Share c of the units starts here; the inverse gives the share a unit belongs to.
__host__ __device__ __forceinline__ uint32_t tp_share_lo(uint32_t units, uint32_t clusters, uint32_t c) { return (uint32_t)((uint64_t)units * c / clusters); }
__host__ __device__ __forceinline__ uint32_t tp_share_of(uint32_t units, uint32_t clusters, uint32_t u) { return (uint32_t)((((uint64_t)u + 1) * clusters - 1) / units); }

__device__ __forceinline__ uint32_t cluster_rank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ void cluster_sync_all()
{
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t map_rank(uint32_t saddr, uint32_t rank)
{
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(rank));
    return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t mapped)      // an address from map_rank
{
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(mapped) : "memory");
}
__device__ __forceinline__ bool elect_one()      // one lane of the (whole) warp, always the same
{
    uint32_t p;
    asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(p));
    return p != 0;
}
__device__ __forceinline__ void tp_commit(uint32_t bar)      // both CTAs' barrier at this offset
{
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(bar), "h"((unsigned short)3) : "memory");
}
__device__ __forceinline__ void tp_mma(uint32_t tmem_d, uint32_t tmem_a, uint64_t db, uint32_t idesc, uint32_t accumulate)
{
    asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
                 " tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n}\n"
                 ::"r"(tmem_d), "r"(tmem_a), "l"(db), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tc_st16(uint32_t taddr, const uint4 (&v)[4])
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
                 ::"r"(taddr), "r"(v[0].x), "r"(v[0].y), "r"(v[0].z), "r"(v[0].w), "r"(v[1].x), "r"(v[1].y), "r"(v[1].z), "r"(v[1].w),
                   "r"(v[2].x), "r"(v[2].y), "r"(v[2].z), "r"(v[2].w), "r"(v[3].x), "r"(v[3].y), "r"(v[3].z), "r"(v[3].w) : "memory");
}

// The packed bytes one dequant thread needs for its 64 weights (sub-blocks 2kq, 2kq+1 of a K-quant superblock, blocks
// 2kq, 2kq+1 of a Q8_0 chunk) of one row, as 16-byte pieces.
//   Q4_K: header (d, dmin, 12 scale bytes), 32 quant bytes (low nibbles = sub-block 2kq, high = 2kq+1).
//   Q5_K: the same plus the 32 bytes of fifth bits (all eight sub-blocks share them).
//   Q8_0: the 80 bytes from the 16-byte boundary at or below byte 68*kq of the chunk; the thread's 68 bytes start kq words in.
//   Q6_K (210-byte superblocks, 2-byte aligned): thread kq takes half n = kq / 2 of the superblock and the elements
//   l = 16 (kq % 2) .. + 15 of that half's four 32-groups (weights 128 n + 32 j + l, j = 0..3): 16 bytes of ql[l],
//   16 of ql[32 + l], 16 of qh[l], the half's eight scale bytes and d.  (Taking 64 consecutive weights instead would
//   need all 64 ql bytes for one of their nibbles each.)
template <int FMT> struct TcPacked { uint4 p[FMT == FMT_Q4_K ? 3 : 5]; };
template <> struct TcPacked<FMT_Q6_K> { uint32_t qa[4], qb[4], qh[4], sc[2], d; };

// row: shared address of the row's chunk (Q6_K: of its first byte, 2-byte aligned).
template <int FMT>
__device__ __forceinline__ void tc_load_packed(uint32_t row, uint32_t kq, TcPacked<FMT> &d)
{
    if constexpr (FMT == FMT_Q6_K) {
        const uint32_t n = kq >> 1, l0 = 16u * (kq & 1u);
        lds_words_a2<4>(row + 64u * n + l0, d.qa);
        lds_words_a2<4>(row + 64u * n + 32u + l0, d.qb);
        lds_words_a2<4>(row + 128u + 32u * n + l0, d.qh);
        lds_words_a2<2>(row + 192u + 8u * n, d.sc);
        d.d = lds16<208>(row);
    } else if constexpr (FMT == FMT_Q8_0) {
        const uint32_t a = row + ((kq * 68u) & ~15u);
        d.p[0] = lds128<0>(a); d.p[1] = lds128<16>(a); d.p[2] = lds128<32>(a); d.p[3] = lds128<48>(a); d.p[4] = lds128<64>(a);
    } else {
        constexpr uint32_t QOFF = FMT == FMT_Q4_K ? 16u : 48u;
        d.p[0] = lds128<0>(row);
        d.p[1] = lds128<QOFF>(row + 32u * kq);
        d.p[2] = lds128<QOFF + 16>(row + 32u * kq);
        if constexpr (FMT == FMT_Q5_K) { d.p[3] = lds128<16>(row); d.p[4] = lds128<32>(row); }
    }
}

// 32 weights (half h of the thread's 64) from the packed pieces -> four 16-byte fp16 pieces, element order.
template <int FMT, int KQ>
__device__ __forceinline__ void tc_dequant_half(const TcPacked<FMT> &d, uint32_t h, int layout, uint4 (&out)[4])
{
    uint32_t w[8];
    __half2 scale, bias, addend;
    if constexpr (FMT == FMT_Q8_0) {
        // words KQ .. KQ+16 of the 20 loaded: block A = fp16 scale in the low half of word KQ, quants from its upper half
        // on; block B = scale in the upper half of word KQ+8, quants = words KQ+9 .. KQ+16
        const uint32_t v[20] = {d.p[0].x, d.p[0].y, d.p[0].z, d.p[0].w, d.p[1].x, d.p[1].y, d.p[1].z, d.p[1].w, d.p[2].x, d.p[2].y,
                                d.p[2].z, d.p[2].w, d.p[3].x, d.p[3].y, d.p[3].z, d.p[3].w, d.p[4].x, d.p[4].y, d.p[4].z, d.p[4].w};
        uint32_t dbits;
        if (h == 0) {
            dbits = v[KQ] & 0xffffu;
#pragma unroll
            for (int i = 0; i < 8; ++i) w[i] = __byte_perm(v[KQ + i], v[KQ + i + 1], 0x5432u) ^ 0x80808080u;
        } else {
            dbits = v[KQ + 8] >> 16;
#pragma unroll
            for (int i = 0; i < 8; ++i) w[i] = v[KQ + 9 + i] ^ 0x80808080u;
        }
        const float dd = __half2float(__ushort_as_half((unsigned short)dbits));
        scale = __float2half2_rn(dd); bias = __float2half2_rn(1152.0f); addend = __float2half2_rn(0.0f);   // bytes are q + 128
    } else {
        const uint4 hd = d.p[0];
        uint32_t scA, scB, mnA, mnB;
        pair_scales(hd.y, hd.z, hd.w, layout, KQ, scA, scB, mnA, mnB);
        const uint32_t sc = h ? scB : scA, mn = h ? mnB : mnA;
        const float dd = __half2float(__ushort_as_half((unsigned short)(hd.x & 0xffffu)));
        const float dmin = __half2float(__ushort_as_half((unsigned short)(hd.x >> 16)));
        w[0] = d.p[1].x; w[1] = d.p[1].y; w[2] = d.p[1].z; w[3] = d.p[1].w; w[4] = d.p[2].x; w[5] = d.p[2].y; w[6] = d.p[2].z; w[7] = d.p[2].w;
        const uint32_t shift = h * 4u;
#pragma unroll
        for (int i = 0; i < 8; ++i) w[i] = (w[i] >> shift) & 0x0F0F0F0Fu;
        if constexpr (FMT == FMT_Q5_K) {
            const uint32_t hb[8] = {d.p[3].x, d.p[3].y, d.p[3].z, d.p[3].w, d.p[4].x, d.p[4].y, d.p[4].z, d.p[4].w};
            const uint32_t g32 = 2u * KQ + h;
#pragma unroll
            for (int i = 0; i < 8; ++i) w[i] |= ((hb[i] >> g32) & 0x01010101u) << 4;
        }
        scale = __float2half2_rn(dd * (float)sc); bias = __float2half2_rn(1024.0f); addend = __float2half2_rn(-(dmin * (float)mn));
    }
#pragma unroll
    for (int p = 0; p < 4; ++p) {
        out[p].x = h2_bits(two_weights(w[2 * p], 0x5140u, bias, scale, addend));
        out[p].y = h2_bits(two_weights(w[2 * p], 0x7362u, bias, scale, addend));
        out[p].z = h2_bits(two_weights(w[2 * p + 1], 0x5140u, bias, scale, addend));
        out[p].w = h2_bits(two_weights(w[2 * p + 1], 0x7362u, bias, scale, addend));
    }
}

__device__ __forceinline__ void tc_st8(uint32_t taddr, const uint32_t (&v)[8])
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                 ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]) : "memory");
}

// Q6_K, 32-group J of the thread's half: its 16 weights (q - 32) * d * scale as fp16, two per word (format.m:131-174:
// ql nibble | two qh bits << 4, scale 8 n + 2 J + l / 16).
template <int KQ, int J>
__device__ __forceinline__ void tc_dequant_q6_group(const TcPacked<FMT_Q6_K> &d, uint32_t (&out)[8])
{
    constexpr int SI = (KQ & 1) + 2 * J;             // scale byte inside the half's eight
    const int sc = (int)(signed char)((d.sc[SI >> 2] >> (8 * (SI & 3))) & 0xffu);
    const float dd = __half2float(__ushort_as_half((unsigned short)d.d));
    const __half2 scale = __float2half2_rn(dd * (float)sc), bias = __float2half2_rn(1056.0f), addend = __float2half2_rn(0.0f);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t ql = (J & 1) ? d.qb[i] : d.qa[i];
        const uint32_t lo = (J < 2 ? ql : ql >> 4) & 0x0F0F0F0Fu;
        const uint32_t w = lo | (((d.qh[i] >> (2 * J)) & 0x03030303u) << 4);
        out[2 * i] = h2_bits(two_weights(w, 0x5140u, bias, scale, addend));
        out[2 * i + 1] = h2_bits(two_weights(w, 0x7362u, bias, scale, addend));
    }
}

// taddr: the thread's lane and the stage's column 32 * KQ (two weights per column).
template <int FMT, int KQ>
__device__ __forceinline__ void tc_convert_unit(const TcPacked<FMT> &d, int layout, uint32_t taddr)
{
    if constexpr (FMT == FMT_Q6_K) {
        // group J, elements 16 (KQ % 2) ..: weights 128 (KQ / 2) + 32 J + 16 (KQ % 2) .., i.e. column 64 (KQ / 2) + 16 J + 8 (KQ % 2)
        const uint32_t col = taddr - 24u * (KQ & 1);
        uint32_t v[8];
        tc_dequant_q6_group<KQ, 0>(d, v); tc_st8(col, v);
        tc_dequant_q6_group<KQ, 1>(d, v); tc_st8(col + 16u, v);
        tc_dequant_q6_group<KQ, 2>(d, v); tc_st8(col + 32u, v);
        tc_dequant_q6_group<KQ, 3>(d, v); tc_st8(col + 48u, v);
    } else {
#pragma unroll
        for (uint32_t h = 0; h < 2; ++h) {
            uint4 v[4];
            tc_dequant_half<FMT, KQ>(d, h, layout, v);
            tc_st16(taddr + h * 16u, v);
        }
    }
}

// BIG: tiles of more than 128 vectors.  The accumulator then takes half of tensor memory (two A stages are left instead of
// three) and an X stage holds 128 k instead of 256.
template <bool BIG> struct TpShape {
    static constexpr uint32_t AS = BIG ? 2 : 3, ACC_COL = BIG ? 256 : 384, SL = BIG ? 2 : 4;      // A stages, accumulator column, slabs of an X stage
};

// PUB: Y is published to the peers (a row-split product, at most 64 vectors).  Its code, inlined behind every store, is not in the other
// instances: a launch starts with cold instruction caches.
template <int FMT, bool BIG, bool PUB>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(TP_THREADS, 1)
gemm_pair_kernel(const __grid_constant__ TpArgs a)
{
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    // layout: [X stages bs x SL slabs x nt_rows / 2 x 128][weight stages][barriers]; the two CTAs' layouts are the same
    constexpr uint32_t AS = TpShape<BIG>::AS, ACC_COL = TpShape<BIG>::ACC_COL, SL = TpShape<BIG>::SL, XPU = TC_SLABS / SL;   // X stages per unit
    const uint32_t slab_bytes = a.nt_rows * 64u, x_bytes = SL * slab_bytes, WS = a.ws, BS = a.bs;
    constexpr uint32_t STAGE = tp_stage_bytes(FMT), PITCH = tp_pitch(FMT), PPR = tp_pieces(FMT);
    uint8_t *x_stages = smem, *w_stages = smem + BS * x_bytes;
    uint64_t *bars = reinterpret_cast<uint64_t *>(w_stages + WS * STAGE);
    uint64_t *b_full = bars, *b_empty = b_full + TP_MAX_BS, *w_full = b_empty + TP_MAX_BS, *w_empty = w_full + TP_MAX_WS;
    uint64_t *a_full = w_empty + TP_MAX_WS, *a_empty = a_full + TP_MAX_AS, *acc_full = a_empty + TP_MAX_AS, *acc_empty = acc_full + 1;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(acc_empty + 1);
    __shared__ volatile int s_abort;

    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const uint32_t rank = cluster_rank(), cl = blockIdx.x >> 1;
    const uint32_t u_lo = tp_share_lo(a.units, a.clusters, cl), n_units = tp_share_lo(a.units, a.clusters, cl + 1) - u_lo;
    const uint32_t tile0 = u_lo / a.chunks, chunk0 = u_lo - tile0 * a.chunks;
    // Positions along the share advance by counters: the loops below hand units on every ~1500 clocks, and a division in one
    // of them (or a shared-memory read of the abort flag in the issuing thread) showed up whole in that interval.

    if (tid == 0) {
        s_abort = 0;
        for (uint32_t s = 0; s < BS; ++s) { mbar_init(smem_u32(b_full + s), rank == 0 ? 2 : 1); mbar_init(smem_u32(b_empty + s), 1); }
        for (uint32_t s = 0; s < WS; ++s) { mbar_init(smem_u32(w_full + s), TP_LOADERS * 32); mbar_init(smem_u32(w_empty + s), TC_DEQ_WARPS); }
        for (uint32_t s = 0; s < AS; ++s) { mbar_init(smem_u32(a_full + s), 2 * TC_DEQ_WARPS); mbar_init(smem_u32(a_empty + s), 1); }
        mbar_init(smem_u32(acc_full), 1);
        mbar_init(smem_u32(acc_empty), 2 * TC_DEQ_WARPS);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 0) {   // all 512 columns of both CTAs: one CTA per SM (its shared memory request sees to that)
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();          // both CTAs' barriers exist and both tensor memories are allocated
    tc_fence_after();
    const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t *>(tmem_slot);
    pdl_launch_dependents();

    // false: the wait ran out, here or earlier in this CTA; every loop ends then
    auto wait = [&](uint64_t *bar, uint32_t parity) -> bool {
        if (mbar_try_wait(smem_u32(bar), parity)) return true;
        if (!s_abort && mbar_wait_bounded(smem_u32(bar), parity)) return true;
        if (!s_abort) { s_abort = 1; atomicExch(a.status, 4); }
        return false;
    };

    if (warp >= (uint32_t)TP_W_LOAD) {
        // ---- loaders: packed weights of this CTA's 128 rows, independent of the previous kernel ----
        const uint32_t lw = warp - TP_W_LOAD;
        constexpr uint32_t CB = FMT == FMT_Q8_0 ? 272u : FMT == FMT_Q4_K ? 144u : FMT == FMT_Q5_K ? 176u : 210u;
        const uint8_t *w_end = a.w + a.w_bytes;
        uint32_t s = 0, ph = 1, tile = tile0, chunk = chunk0, live = 0;
        const uint8_t *rows0 = nullptr;
        for (uint32_t i = 0; i < n_units; ++i) {
            if (i == 0 || chunk == 0) {      // a new tile
                const uint32_t row0 = (tile / a.ntiles) * TP_ROWS + rank * TC_M + lw * 32u;
                live = a.rows > row0 ? a.rows - row0 : 0u;
                rows0 = a.w + (size_t)row0 * a.row_bytes;
            }
            if (i >= WS && !wait(w_empty + s, ph)) break;
            const uint8_t *src0 = rows0 + chunk * CB;
            const uint32_t dst0 = smem_u32(w_stages + s * STAGE) + lw * 32u * PITCH;
#pragma unroll
            for (uint32_t j = 0; j < PPR; ++j) {
                const uint32_t q = lane + 32u * j, r = q / PPR, p = q - r * PPR;
                const uint8_t *src = src0 + r * a.row_bytes;
                if constexpr (FMT == FMT_Q6_K) src = reinterpret_cast<const uint8_t *>(reinterpret_cast<uintptr_t>(src) & ~(uintptr_t)15);
                src += p * 16u;
                uint32_t bytes = r < live ? 16u : 0u;
                if constexpr (FMT == FMT_Q6_K) {      // the tensor may end inside or before a row's last piece
                    if (bytes && src + 16 > w_end) bytes = src < w_end ? (uint32_t)(w_end - src) : 0u;
                }
                cp_async16(dst0 + r * PITCH + p * 16u, bytes ? src : a.w, bytes);
            }
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(w_full + s)) : "memory");
            if (++s == WS) { s = 0; ph ^= 1u; }
            if (++chunk == a.chunks) { chunk = 0; ++tile; }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else if (warp == (uint32_t)TP_W_X) {
        // ---- X producer: this CTA's half of the tile's vectors, a stage of SL slabs at a time ----
        if (lane == 0) {
            pdl_wait();          // the packed X is the previous kernel's output
            uint32_t s = 0, ph = 1, n = 0, nt = tile0 % a.ntiles, chunk = chunk0;
            bool ok = true;
            for (uint32_t i = 0; i < n_units && ok; ++i) {
                const uint8_t *src = reinterpret_cast<const uint8_t *>(a.xp) + ((size_t)(2 * nt + rank) * a.chunks + chunk) * (TC_SLABS * slab_bytes);
                for (uint32_t j = 0; j < XPU; ++j, ++n) {
                    if (n >= BS) { ok = wait(b_empty + s, ph); if (!ok) break; }      // only MMAs and bulk copies touch X: no proxy to order
                    mbar_expect_tx(smem_u32(b_full + s), x_bytes);
                    bulk_g2s(smem_u32(x_stages + s * x_bytes), src + j * x_bytes, x_bytes, smem_u32(b_full + s));
                    if (++s == BS) { s = 0; ph ^= 1u; }
                }
                if (++chunk == a.chunks) { chunk = 0; if (++nt == a.ntiles) nt = 0; }
            }
            if (!ok) {           // copies still in flight get a bounded time to land (rank 0's barriers also wait for the relay, so by time)
                const long long t0 = clock64();
                while (clock64() - t0 < 200000) { }
            }
        }
    } else if (warp == (uint32_t)TP_W_MMA) {
        if (lane == 0 && rank == 1) {
            // ---- relay: this CTA's half of X has landed ----
            const uint32_t peer = map_rank(smem_u32(b_full), 0);
            uint32_t s = 0, ph = 0;
            for (uint32_t n = 0; n < n_units * XPU; ++n) {
                if (!wait(b_full + s, ph)) break;
                mbar_arrive_cluster(peer + 8u * s);
                if (++s == BS) { s = 0; ph ^= 1u; }
            }
        } else if (rank == 0) {
            // ---- MMA issue ----
            // The whole warp walks the loop and one elected lane issues: descriptors and columns then stay in uniform registers.  As
            // the body of `if (lane == 0)` every operand of every MMA had to be moved there, and with the dequant warps competing for
            // issue slots the 16 MMAs of a unit took ~600-900 clocks longer (12288 x 4096 Q8_0 at 2048 vectors 3180 -> 2580 clocks a
            // unit, 17408 x 5120 Q4_K at 333 2680 -> 1830, 12288 x 4096 Q4_K at 64 2200 -> 1420).
            const uint32_t idesc = (1u << 4) | ((a.nt_rows >> 3) << 17) | ((uint32_t)(TP_ROWS >> 4) << 24);   // fp32 accumulate, fp16 x fp16, K-major both
            const uint32_t slab_step = slab_bytes >> 4, acc = tmem_base + ACC_COL;
            uint32_t sa = 0, pa = 0, sb = 0, pb = 0, seg = 0, chunk = chunk0;
            bool ok = true;
            for (uint32_t i = 0; i < n_units && ok; ++i) {
                const bool first = i == 0 || chunk == 0;
                if (first && seg > 0 && !__all_sync(0xffffffffu, wait(acc_empty, (seg - 1) & 1u))) break;      // the previous tile's sums have been read
                if (!__all_sync(0xffffffffu, wait(a_full + sa, pa))) break;
                const uint32_t a_col = tmem_base + sa * 128u;
#pragma unroll
                for (uint32_t j = 0; j < XPU; ++j) {
                    if (!__all_sync(0xffffffffu, wait(b_full + sb, pb))) { ok = false; break; }
                    tc_fence_after();
                    if (elect_one()) {
                        const uint64_t db0 = tc_desc_sw128(smem_u32(x_stages + sb * x_bytes));
#pragma unroll
                        for (uint32_t k16 = 0; k16 < 4 * SL; ++k16)      // a step of 32 bytes is 2 in the descriptor
                            tp_mma(acc, a_col + (j * 4 * SL + k16) * 8u, db0 + (k16 >> 2) * slab_step + (k16 & 3u) * 2u, idesc, j == 0 && k16 == 0 ? !first : 1u);
                        tp_commit(smem_u32(b_empty + sb));
                    }
                    __syncwarp();
                    if (++sb == BS) { sb = 0; pb ^= 1u; }
                }
                if (!ok) break;
                if (elect_one()) tp_commit(smem_u32(a_empty + sa));
                __syncwarp();
                if (++sa == AS) { sa = 0; pa ^= 1u; }
                if (++chunk == a.chunks) chunk = 0;
                if (chunk == 0 || i + 1 == n_units) {
                    if (elect_one()) tp_commit(smem_u32(acc_full));
                    __syncwarp();
                    ++seg;
                }
            }
        }
    } else {
        // ---- dequant warps: packed stage -> fp16 in tensor memory; then the tile's sums ----
        const uint32_t quad = warp & 3u, kq = warp >> 2, r = quad * 32u + lane, lane_addr = (quad * 32u) << 16;
        const uint32_t a_full0 = map_rank(smem_u32(a_full), 0), acc_empty0 = map_rank(smem_u32(acc_empty), 0);
        const uint32_t tmem_a = tmem_base + lane_addr + kq * 32u;
        uint32_t s = 0, pw = 0, sa = 0, pa = 1, seg = 0, tile = tile0, chunk = chunk0;
        uint32_t row_off = 0;        // Q6_K: the row's first byte inside its 16-byte piece, before the chunk's offset
        // s_abort may be set between two lanes' looks at it, but what follows a wait (__syncwarp, tensor memory accesses) needs the
        // warp together: the lanes vote, where they have to meet anyway, and give up as a whole.
        for (uint32_t i = 0; i < n_units; ++i) {
            if (FMT == FMT_Q6_K && (i == 0 || chunk == 0))
                row_off = (uint32_t)reinterpret_cast<uintptr_t>(a.w) + ((tile / a.ntiles) * TP_ROWS + rank * TC_M + r) * a.row_bytes;
            bool ok = wait(w_full + s, pw);
            TcPacked<FMT> pk;
            uint32_t row_s = smem_u32(w_stages + s * STAGE) + r * PITCH;
            if constexpr (FMT == FMT_Q6_K) row_s += (row_off + chunk * 210u) & 15u;
            tc_load_packed<FMT>(row_s, kq, pk);
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(w_empty + s));
            if (++s == WS) { s = 0; pw ^= 1u; }
            if (ok && i >= AS) ok = wait(a_empty + sa, pa);
            if (!__all_sync(0xffffffffu, ok)) break;
            tc_fence_after();
            const uint32_t taddr = tmem_a + sa * 128u;
            switch (kq) {                         // warp-uniform; the sub-block index is a compile-time constant inside
            case 0: tc_convert_unit<FMT, 0>(pk, a.layout, taddr); break;
            case 1: tc_convert_unit<FMT, 1>(pk, a.layout, taddr); break;
            case 2: tc_convert_unit<FMT, 2>(pk, a.layout, taddr); break;
            default: tc_convert_unit<FMT, 3>(pk, a.layout, taddr); break;
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(a_full0 + 8u * sa);
            if (++sa == AS) { sa = 0; pa ^= 1u; }
            if (++chunk < a.chunks && i + 1 < n_units) continue;
            // the last unit of this tile (or of the share): a warp takes 16 columns in four, lane = row
            const uint32_t t_lo = tile * a.chunks;
            const bool whole = u_lo <= t_lo && u_lo + n_units >= t_lo + a.chunks;
            const uint32_t grow = (tile / a.ntiles) * TP_ROWS + rank * TC_M + r, n_base = (tile % a.ntiles) * a.nt_rows;
            float *part = a.part + ((size_t)cl * a.slots + (u_lo <= t_lo ? a.slots - 1 : 0)) * a.nt_rows * TP_ROWS + rank * TC_M + r;   // 0: the share starts inside the tile
            const bool done = __all_sync(0xffffffffu, wait(acc_full, seg & 1u));
            tc_fence_after();
            for (uint32_t n0 = kq * 16u; n0 < a.nt_rows; n0 += 64u) {
                uint32_t v[16];
                __syncwarp();
                asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                             : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
                               "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
                             : "r"(tmem_base + lane_addr + ACC_COL + n0));
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (!done) continue;
                if (!whole) {
#pragma unroll
                    for (uint32_t q = 0; q < 16; ++q) part[(size_t)(n0 + q) * TP_ROWS] = __uint_as_float(v[q]);
                } else if (grow < a.rows) {
                    float *dst = a.y + (size_t)(n_base + n0) * a.ldy + grow;
#pragma unroll
                    for (uint32_t q = 0; q < 16; ++q) {
                        if (n_base + n0 + q < a.batch) {
                            dst[(size_t)q * a.ldy] = __uint_as_float(v[q]);
                            if (PUB && a.pub.npeers > 0) tc_publish(a.pub, dst + (size_t)q * a.ldy, __uint_as_float(v[q]), *reinterpret_cast<const volatile unsigned int *>(a.pub.pub_gen) + 1u);
                        }
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (!done) break;
            if (lane == 0) mbar_arrive_cluster(acc_empty0);
            ++seg;
            if (chunk == a.chunks) { chunk = 0; ++tile; }
        }
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();          // neither CTA leaves while the other may still reach into it
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
    }
    if (PUB && tid == 0 && a.publish_done && a.pub.npeers > 0)
        tc_publish_done(a.pub, *reinterpret_cast<const volatile unsigned int *>(a.pub.pub_gen) + 1u);
}

// Tiles that were cut over several clusters: Y = the sum of their partial sums, in cluster order.  blockIdx.x = tile,
// blockIdx.y = four of its vectors; a thread adds up four rows of one vector, so that a tile cut six ways is one round of
// independent 16-byte loads (with 16 vectors a thread in turn this pass took longer than the product it follows).
__global__ void __launch_bounds__(256)
tile_reduce_kernel(const __grid_constant__ TpArgs a)
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const uint32_t tile = blockIdx.x, t_lo = tile * a.chunks, t_hi = t_lo + a.chunks;
    const uint32_t c_lo = tp_share_of(a.units, a.clusters, t_lo), c_hi = tp_share_of(a.units, a.clusters, t_hi - 1);
    const uint32_t row = (threadIdx.x & 63u) * 4u, n = blockIdx.y * 4u + (threadIdx.x >> 6);
    const uint32_t grow = (tile / a.ntiles) * TP_ROWS + row, gn = (tile % a.ntiles) * a.nt_rows + n;
    const unsigned int tag = a.pub.npeers > 0 ? *reinterpret_cast<const volatile unsigned int *>(a.pub.pub_gen) + 1u : 0u;
    if (c_lo != c_hi && grow < a.rows && gn < a.batch) {
        const size_t slot = (size_t)a.nt_rows * TP_ROWS, step = a.slots * slot;
        const float *src = a.part + (size_t)c_lo * step + (size_t)n * TP_ROWS + row;
        // the tile's first cluster has it as its last tile (the last slot); the others start inside it (slot 0)
        float4 acc = __ldcg(reinterpret_cast<const float4 *>(src + (a.slots - 1) * slot));
#pragma unroll 8
        for (uint32_t c = c_lo + 1; c <= c_hi; ++c) {
            src += step;
            const float4 v = __ldcg(reinterpret_cast<const float4 *>(src));
            acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
        }
        float *dst = a.y + (size_t)gn * a.ldy + grow;
        const float o[4] = {acc.x, acc.y, acc.z, acc.w};
        if (grow + 4 <= a.rows && !(reinterpret_cast<uintptr_t>(dst) & 15)) *reinterpret_cast<float4 *>(dst) = acc;
        else {
            for (uint32_t q = 0; q < 4 && grow + q < a.rows; ++q) dst[q] = o[q];
        }
        if (a.pub.npeers > 0) {
            for (uint32_t q = 0; q < 4 && grow + q < a.rows; ++q) tc_publish(a.pub, dst + q, o[q], tag);
        }
    }
    if (a.pub.npeers > 0) {
        __syncthreads();
        if (threadIdx.x == 0 && atomicAdd(a.pub.pub_arrived, 1u) == gridDim.x * gridDim.y - 1) {
            *reinterpret_cast<volatile unsigned int *>(a.pub.pub_arrived) = 0;
            *reinterpret_cast<volatile unsigned int *>(a.pub.pub_gen) = tag;
        }
    }
}

}  // namespace orome
