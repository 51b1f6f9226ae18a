// moe_group.cuh -- routed experts for token batches, tokens grouped by expert.
//
// Token by token, an expert that n tokens chose is streamed, unpacked and multiplied n times (300 tokens, top-8 of 128:
// ~19 times each).  Here the (token, slot) pairs are sorted by expert first and an expert's weights are unpacked once per 32
// of its tokens:
//
//   moe_prepare_kernel   block 0: pairs -> blocks of at most `cap` pairs of one expert; the others: x -> byte planes
//   moe_group_kernel     fused gate/up over (pair block, 128 rows) items
//   moe_quantize_kernel  activations -> byte planes
//   moe_group_kernel     down over (pair block, 256 rows) items
//   moe_sum_kernel       out[t] = sum over a token's slots, in slot order, of weight * result
//
// Arithmetic: that of gemv_mma.cuh -- x as 24-bit fixed point per superblock (three balanced byte planes), integer mma, exact
// integer sums per superblock, one float step per superblock -- with the columns of the B operand used differently: eight
// TOKENS a plane, three mma (one per plane) against the same A operand, instead of the three planes of one token.  So all
// eight columns work, A is unpacked once for up to 32 tokens, and a token's planes meet in one thread.  The order of the
// sums of a pair does not depend on its neighbours: results do not depend on what else is in the batch.
//
// What bounds it: the integer multiply-adds that apply the six-bit scales (96 a warp, 16 rows x 256 weights x 8 tokens, half
// rate), the mma (27 a piece at one per two clocks) and the B fragments (48 shared-memory wavefronts) each need ~50 clocks a
// piece and SM.  Sixteen warps with one 16-row tile each hide the latencies between them: eight warps with two tiles, which
// read a B fragment once for both, had 0.8 eligible warps a scheduler and half the issue slots idle.
#pragma once
#include "gemv_mma.cuh"

namespace orome {

constexpr int MG_WARPS = 16, MG_LOADERS = 4, MG_THREADS = (MG_WARPS + MG_LOADERS) * 32;
constexpr int MG_MAX_CAP = 32;                    // pairs of an item
constexpr int MG_BINS = 1024;                     // experts that are sorted; pairs of experts beyond become items of their own
constexpr uint32_t MG_REC = 800;                  // a superblock of x: 8 sub-blocks x 3 planes x 32 B, 3 x 8 sum bytes, two scales; = 32 (mod 128)
constexpr uint32_t MG_MAX_STAGES = 6;
__host__ __device__ constexpr uint32_t mg_unit(int fmt) { return fmt == FMT_Q4_K ? 144u : 176u; }
__host__ __device__ constexpr uint32_t mg_pitch(int fmt) { return fmt == FMT_Q4_K ? 160u : 224u; }      // = 32 or 96 (mod 128): rows g .. g + 3 of a fragment load hit different banks
__host__ __device__ constexpr uint32_t mg_stage_bytes(int fmt, uint32_t cap) { return 16 * MG_WARPS * mg_pitch(fmt) + cap * MG_REC; }

struct MgBlock { uint32_t expert, start, count, pad; };     // pairs order[start .. start + count) of one expert

struct MgArgs {
    const uint8_t *w0, *w1;        // gate and up; down: w0
    uint64_t stride;               // bytes between experts
    uint32_t rows, units, row_bytes;
    uint32_t K, cap;
    const uint8_t *xq;             // [vector][units] records
    uint32_t x_per_token;          // gate/up: pairs of a token share its vector; down: every pair has its own
    const uint32_t *order;         // t * 8 + slot
    const MgBlock *blocks;
    const uint32_t *n_blocks;
    float *out;                    // [t * K + slot][rows]
    uint32_t nstages;
    int layout;
    int *status;
};

// One superblock of x (eight elements a lane) -> its record in global memory.
__device__ __forceinline__ void mg_quantize(const float *__restrict__ src, uint8_t *__restrict__ rec, uint32_t lane)
{
    constexpr int QMAXI = 127 * 65536 + 127 * 256 + 127;
    constexpr float QMAX = (float)QMAXI;
    const float4 v0 = __ldcg(reinterpret_cast<const float4 *>(src) + 2 * lane), v1 = __ldcg(reinterpret_cast<const float4 *>(src) + 2 * lane + 1);
    float amax = fmaxf(fmaxf(fmaxf(fabsf(v0.x), fabsf(v0.y)), fmaxf(fabsf(v0.z), fabsf(v0.w))),
                       fmaxf(fmaxf(fabsf(v1.x), fabsf(v1.y)), fmaxf(fabsf(v1.z), fabsf(v1.w))));
    float sum = ((v0.x + v0.y) + (v0.z + v0.w)) + ((v1.x + v1.y) + (v1.z + v1.w));
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) { amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o)); sum += __shfl_xor_sync(0xffffffffu, sum, o); }
    float smax = fabsf(sum);
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) { amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o)); smax = fmaxf(smax, __shfl_xor_sync(0xffffffffu, smax, o)); }
    const float inv = amax > 0.0f ? QMAX / amax : 0.0f, sinv = smax > 0.0f ? QMAX / smax : 0.0f;
    const float v[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
    uint32_t uq[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) uq[i] = (uint32_t)max(-QMAXI, min(QMAXI, __float2int_rn(v[i] * inv))) + digit_bias<3>();
#pragma unroll
    for (int p = 0; p < 3; ++p)
        *reinterpret_cast<uint2 *>(rec + (lane >> 2) * 96 + p * 32 + (lane & 3u) * 8) =
            make_uint2(plane_word(uq[0], uq[1], uq[2], uq[3], p), plane_word(uq[4], uq[5], uq[6], uq[7], p));
    const uint32_t us = (uint32_t)max(-QMAXI, min(QMAXI, __float2int_rn(sum * sinv))) + digit_bias<3>();
    if ((lane & 3u) == 0) {
#pragma unroll
        for (int p = 0; p < 3; ++p) rec[768 + p * 8 + (lane >> 2)] = (uint8_t)(((us >> (8 * p)) & 255u) ^ 0x80u);
    }
    if (lane == 0) *reinterpret_cast<float2 *>(rec + 792) = make_float2(amax / QMAX, smax / QMAX);
}

// A warp per superblock; blockIdx.y = vector.
__global__ void __launch_bounds__(256)
moe_quantize_kernel(const float *__restrict__ x, uint32_t ldx, uint32_t units, uint8_t *__restrict__ xq)
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const uint32_t u = blockIdx.x * 8u + (threadIdx.x >> 5);
    if (u < units) mg_quantize(x + (size_t)blockIdx.y * ldx + u * 256u, xq + ((size_t)blockIdx.y * units + u) * MG_REC, threadIdx.x & 31u);
}

// Block 0 sorts the pairs: a histogram over experts, its running sums, the pairs in expert order and blocks of at most `cap`
// pairs, the ones with more groups of eight first: CTAs take items in turn, so every round then has items of one cost.
// Which of an expert's pairs (and which of equal blocks) comes first is left to the atomics; no result depends on it.
// Blocks 1.. quantize x.
__global__ void __launch_bounds__(1024)
moe_prepare_kernel(const uint32_t *__restrict__ idx, uint32_t n_tokens, uint32_t K, uint32_t cap, uint32_t *__restrict__ order,
                   MgBlock *__restrict__ blocks, uint32_t *__restrict__ n_blocks, const float *__restrict__ x, uint32_t ldx, uint32_t units,
                   uint8_t *__restrict__ xq)
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    if (blockIdx.x > 0) {
        for (uint32_t i = (blockIdx.x - 1) * 32u + warp; i < n_tokens * units; i += (gridDim.x - 1) * 32u) {
            const uint32_t t = i / units, u = i - t * units;
            mg_quantize(x + (size_t)t * ldx + u * 256u, xq + (size_t)i * MG_REC, lane);
        }
        return;
    }
    __shared__ uint32_t s_count[MG_BINS], s_warp[32], s_class[MG_MAX_CAP / 8], s_extra, s_far;
    s_count[tid] = 0;
    if (tid < MG_MAX_CAP / 8) s_class[tid] = 0;
    if (tid == 0) s_far = 0;
    __syncthreads();
    const uint32_t n = n_tokens * K;
    for (uint32_t i = tid; i < n; i += 1024u) {
        const uint32_t e = __ldcg(idx + (i / K) * 8u + i % K);
        if (e < (uint32_t)MG_BINS) atomicAdd(&s_count[e], 1u);
    }
    __syncthreads();
    const uint32_t count = s_count[tid], whole = count / cap, rest = count % cap;
    if (whole) atomicAdd(&s_class[(cap + 7) / 8 - 1], whole);
    if (rest) atomicAdd(&s_class[(rest + 7) / 8 - 1], 1u);
    uint32_t ps = count;                           // inclusive sum over the warp, then over the block
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t a = __shfl_up_sync(0xffffffffu, ps, o);
        if (lane >= (uint32_t)o) ps += a;
    }
    if (lane == 31) s_warp[warp] = ps;
    __syncthreads();
    if (warp == 0) {
        uint32_t a = s_warp[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t aa = __shfl_up_sync(0xffffffffu, a, o);
            if (lane >= (uint32_t)o) a += aa;
        }
        s_warp[lane] = a;
    }
    if (tid == 32) {                               // the classes' first positions, the costliest first
        uint32_t at = 0;
        for (int k = MG_MAX_CAP / 8 - 1; k >= 0; --k) { const uint32_t m = s_class[k]; s_class[k] = at; at += m; }
        s_extra = at;
    }
    __syncthreads();
    const uint32_t sorted = s_warp[31], start = ps - count + (warp ? s_warp[warp - 1] : 0u);
    if (whole) {
        const uint32_t at = atomicAdd(&s_class[(cap + 7) / 8 - 1], whole);
        for (uint32_t b = 0; b < whole; ++b) blocks[at + b] = MgBlock{tid, start + b * cap, cap, 0u};
    }
    if (rest) blocks[atomicAdd(&s_class[(rest + 7) / 8 - 1], 1u)] = MgBlock{tid, start + whole * cap, rest, 0u};
    s_count[tid] = start;                          // from here on: where the expert's next pair goes
    __syncthreads();
    for (uint32_t i = tid; i < n; i += 1024u) {
        const uint32_t t = i / K, k = i - t * K, e = __ldcg(idx + t * 8u + k);
        uint32_t pos;
        if (e < (uint32_t)MG_BINS) pos = atomicAdd(&s_count[e], 1u);
        else {
            pos = sorted + atomicAdd(&s_far, 1u);
            blocks[atomicAdd(&s_extra, 1u)] = MgBlock{e, pos, 1u, 0u};
        }
        order[pos] = t * 8u + k;
    }
    __syncthreads();
    if (tid == 0) *n_blocks = s_extra;
}

// SWIGLU: a warp's 16-row tile is rows 8 w .. 8 w + 7 of gate and the same rows of up, so that both halves of an output meet in
// one thread; an item covers 128 rows.  Else rows 16 w .. of down, an item covers 256.  Loader warps stream one superblock of
// all those rows and of the item's vectors a stage, across items.
template <int FMT, bool SWIGLU>
__global__ void __launch_bounds__(MG_THREADS, 1)
moe_group_kernel(const __grid_constant__ MgArgs a)
{
    extern __shared__ __align__(128) uint8_t smem[];
    constexpr uint32_t UNIT = mg_unit(FMT), PITCH = mg_pitch(FMT), PPR = UNIT / 16, W_BYTES = 16 * MG_WARPS * PITCH;
    constexpr uint32_t ROWS = SWIGLU ? 8 * MG_WARPS : 16 * MG_WARPS;
    constexpr int QOFF = FMT == FMT_Q4_K ? 16 : 48;
    __shared__ uint64_t full[MG_MAX_STAGES], empty[MG_MAX_STAGES];
    __shared__ uint32_t s_order[8][MG_MAX_CAP];     // the pairs of the last eight items (the ring holds stages of fewer)
    __shared__ volatile int s_abort;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const uint32_t stage_bytes = W_BYTES + a.cap * MG_REC, U = a.units;
    if (tid == 0) {
        s_abort = 0;
        for (uint32_t s = 0; s < a.nstages; ++s) { mbar_init(smem_u32(full + s), MG_LOADERS * 32 + 1); mbar_init(smem_u32(empty + s), MG_WARPS); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    pdl_launch_dependents();
    pdl_wait();                     // the blocks and the vectors are the previous kernels' output
    const uint32_t row_blocks = (a.rows + ROWS - 1) / ROWS, n_items = __ldcg(a.n_blocks) * row_blocks;

    auto block_of = [&](uint32_t item) { return item < n_items ? __ldcg(reinterpret_cast<const uint4 *>(a.blocks + item / row_blocks)) : make_uint4(0u, 0u, 0u, 0u); };
    if (warp >= (uint32_t)MG_WARPS) {
        const uint32_t lt = tid - MG_WARPS * 32;
        uint32_t s = 0, ph = 1, fill = 0, slot = 0;
        // `dead`: a wait ran out somewhere in this CTA.  A loader that finds out stops waiting and copying but keeps coming to the
        // barrier below, since the others may not have found out yet and count on it; without waits the items left over are brief.
        bool dead = false;
        uint4 bq = block_of(blockIdx.x);
        uint32_t ord = lt < bq.z ? __ldcg(a.order + bq.y + lt) : 0u;
        for (uint32_t item = blockIdx.x; item < n_items; item += gridDim.x, slot = (slot + 1) & 7u) {
            const uint32_t row0 = item % row_blocks * ROWS;
            const uint8_t *e0 = a.w0 + bq.x * a.stride + (size_t)row0 * a.row_bytes, *e1 = SWIGLU ? a.w1 + bq.x * a.stride + (size_t)row0 * a.row_bytes : e0;
            const uint32_t live = min(ROWS, a.rows - row0), pieces = bq.z * (MG_REC / 16);
            if (lt < bq.z) s_order[slot][lt] = ord;
            __syncwarp();
            named_bar_sync(PIPE_BAR_CONSUMERS, MG_LOADERS * 32);
            // the next item's block and pairs are on their way while this one's stages are filled
            const uint4 nq = block_of(item + gridDim.x);
            for (uint32_t u = 0; u < U && !dead; ++u, ++fill) {
                if (fill >= a.nstages && !mbar_wait_bounded(smem_u32(empty + s), ph)) { if (!s_abort) { s_abort = 1; atomicExch(a.status, 2); } }
                if (s_abort) { dead = true; break; }
                const uint32_t st = smem_u32(smem + (size_t)s * stage_bytes);
#pragma unroll
                for (uint32_t j = 0; j < 16 * MG_WARPS * PPR / (MG_LOADERS * 32); ++j) {
                    const uint32_t q = lt + j * (MG_LOADERS * 32), r = q / PPR, p = q - r * PPR;      // stage rows: gate, then up; else rows in order
                    const uint32_t row = SWIGLU ? r % ROWS : r;
                    const uint8_t *src = (SWIGLU && r >= ROWS ? e1 : e0) + row * a.row_bytes + (u * UNIT + p * 16u);
                    const uint32_t ok = row < live ? 16u : 0u;
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(st + r * PITCH + p * 16u), "l"(ok ? src : a.w0), "r"(ok) : "memory");
                }
#pragma unroll 4
                for (uint32_t q = lt; q < pieces; q += MG_LOADERS * 32) {
                    const uint32_t v = q / (MG_REC / 16), p = q - v * (MG_REC / 16);
                    const uint32_t o = s_order[slot][v], vec = a.x_per_token ? o >> 3 : (o >> 3) * a.K + (o & 7u);
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(st + W_BYTES + q * 16u), "l"(a.xq + ((size_t)vec * U + u) * MG_REC + p * 16u) : "memory");
                }
                asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(full + s)) : "memory");
                if (lt == 0) mbar_arrive(smem_u32(full + s));      // and, in order with the barrier above, the item's pairs
                if (++s == a.nstages) { s = 0; ph ^= 1u; }
                if (u == 0) ord = lt < nq.z ? __ldcg(a.order + nq.y + lt) : 0u;
            }
            bq = nq;
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        return;
    }

    const uint32_t g = lane >> 2, t = lane & 3u;
    uint32_t s = 0, ph = 0, slot = 0;
    uint4 bq = block_of(blockIdx.x), nq;
    for (uint32_t item = blockIdx.x; item < n_items; item += gridDim.x, slot = (slot + 1) & 7u, bq = nq) {
        const uint32_t row0 = item % row_blocks * ROWS;
        nq = block_of(item + gridDim.x);
        float y[MG_MAX_CAP / 8][4];
#pragma unroll
        for (int c = 0; c < MG_MAX_CAP / 8; ++c) y[c][0] = y[c][1] = y[c][2] = y[c][3] = 0.0f;
        for (uint32_t u = 0; u < U; ++u) {
            if (!mbar_wait_bounded(smem_u32(full + s), ph)) { if (!s_abort) { s_abort = 1; atomicExch(a.status, 1); } }
            if (__any_sync(0xffffffffu, s_abort)) return;      // the whole warp, ahead of its mma
            const uint32_t st = smem_u32(smem + (size_t)s * stage_bytes);
            const uint32_t h0 = st + (SWIGLU ? warp * 8u + g : warp * 16u + g) * PITCH, h1 = h0 + (SWIGLU ? 8 * MG_WARPS : 8) * PITCH;
            uint32_t A[8][4], sl0, sh0, sl1, sh1, ml0, mh0, ml1, mh1;
            const uint4 hd0 = lds128<0>(h0), hd1 = lds128<0>(h1);
            unpack_scales4(hd0.y, hd0.z, hd0.w, a.layout, sl0, sh0, ml0, mh0);
            unpack_scales4(hd1.y, hd1.z, hd1.w, a.layout, sl1, sh1, ml1, mh1);
            const uint32_t mn0 = t == 0 ? ml0 : (t == 1 ? mh0 : 0u), mn1 = t == 0 ? ml1 : (t == 1 ? mh1 : 0u);
            uint2 q0 = make_uint2(0u, 0u), q1 = q0;
            if constexpr (FMT == FMT_Q5_K) { q0 = lds64<16>(h0 + 8u * t); q1 = lds64<16>(h1 + 8u * t); }
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                const uint2 w0 = lds64<QOFF>(h0 + 8u * t + 32u * b), w1 = lds64<QOFF>(h1 + 8u * t + 32u * b);
                const uint32_t w[4] = {w0.x, w1.x, w0.y, w1.y}, hb[4] = {q0.x, q1.x, q0.y, q1.y};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    A[2 * b][i] = w[i] & 0x0F0F0F0Fu;
                    A[2 * b + 1][i] = (w[i] >> 4) & 0x0F0F0F0Fu;
                    if constexpr (FMT == FMT_Q5_K) {
                        A[2 * b][i] |= ((hb[i] >> (2 * b)) & 0x01010101u) << 4;
                        A[2 * b + 1][i] |= ((hb[i] >> (2 * b + 1)) & 0x01010101u) << 4;
                    }
                }
            }
            const __half2 dd0 = *reinterpret_cast<const __half2 *>(&hd0.x), dd1 = *reinterpret_cast<const __half2 *>(&hd1.x);
            const float d[2] = {__low2float(dd0), __low2float(dd1)}, dm[2] = {__high2float(dd0), __high2float(dd1)};
            const uint32_t xb = st + W_BYTES + g * MG_REC + 8u * t;
#pragma unroll
            for (int c = 0; c < MG_MAX_CAP / 8; ++c) {
                if (c * 8u >= bq.z) continue;
                const uint32_t x0 = xb + c * 8u * MG_REC;
                int acc[3][4];
#pragma unroll
                for (int i = 0; i < 12; ++i) acc[i / 4][i & 3] = 0;
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const int s0 = (int)__byte_perm(j < 4 ? sl0 : sh0, 0u, 0x4440u + (j & 3)), s1 = (int)__byte_perm(j < 4 ? sl1 : sh1, 0u, 0x4440u + (j & 3));
#pragma unroll
                    for (int p = 0; p < 3; ++p) {
                        uint2 b;
                        asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(b.x), "=r"(b.y) : "r"(x0 + 96u * j + 32u * p));
                        int r[4];
                        mma_u8s8_k32(r, A[j], b.x, b.y);
                        acc[p][0] += s0 * r[0]; acc[p][1] += s0 * r[1]; acc[p][2] += s1 * r[2]; acc[p][3] += s1 * r[3];
                    }
                }
                // the vectors' sums against the mins, and the two columns' scales
                const uint32_t sx = x0 - 8u * t + 768u + (t & 1u) * 4u, cx = st + W_BYTES + (c * 8u + 2u * t) * MG_REC + 792u;
                int m0[4], m1[4], m2[4];
                mma_u8s8_k16(m0, mn0, mn1, lds32<0>(sx));
                mma_u8s8_k16(m1, mn0, mn1, lds32<8>(sx));
                mma_u8s8_k16(m2, mn0, mn1, lds32<16>(sx));
                const uint2 xsa = lds64<0>(cx), xsb = lds64<MG_REC>(cx);
                const float xs[2] = {__uint_as_float(xsa.x), __uint_as_float(xsb.x)}, sxs[2] = {__uint_as_float(xsa.y), __uint_as_float(xsb.y)};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float f = fmaf(65536.0f, (float)acc[2][i], fmaf(256.0f, (float)acc[1][i], (float)acc[0][i]));
                    const float fm = fmaf(65536.0f, (float)m2[i], fmaf(256.0f, (float)m1[i], (float)m0[i]));
                    y[c][i] = fmaf(d[i >> 1] * xs[i & 1], f, y[c][i]);
                    y[c][i] = fmaf(-(dm[i >> 1] * sxs[i & 1]), fm, y[c][i]);
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(empty + s));
            if (++s == a.nstages) { s = 0; ph ^= 1u; }
        }
        // a thread holds rows g, g + 8 of columns 2t, 2t + 1
#pragma unroll
        for (int c = 0; c < MG_MAX_CAP / 8; ++c) {
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const uint32_t col = c * 8u + 2u * t + q;
                if (col >= bq.z) continue;
                const uint32_t o = s_order[slot][col];
                float *dst = a.out + (size_t)((o >> 3) * a.K + (o & 7u)) * a.rows;
                if constexpr (SWIGLU) {
                    const uint32_t row = row0 + warp * 8u + g;
                    if (row < a.rows) dst[row] = silu_mul(y[c][q], y[c][2 + q]);
                } else {
                    const uint32_t row = row0 + warp * 16u + g;
                    if (row < a.rows) dst[row] = y[c][q];
                    if (row + 8u < a.rows) dst[row + 8u] = y[c][2 + q];
                }
            }
        }
    }
}

// out[t][h] = sum over slots k = 0 .. K - 1 of w[t][k] * r[t * K + k][h]
__global__ void __launch_bounds__(256)
moe_sum_kernel(const float *__restrict__ r, const float *__restrict__ w, uint32_t K, uint32_t hidden, float *__restrict__ out, uint32_t ldo)
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const uint32_t t = blockIdx.y, h = blockIdx.x * 256u + threadIdx.x;
    if (h >= hidden) return;
    float v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = (uint32_t)k < K ? __ldcg(r + ((size_t)t * K + k) * hidden + h) : 0.0f;
    float acc = 0.0f;
#pragma unroll
    for (int k = 0; k < 8; ++k) if ((uint32_t)k < K) acc = fmaf(__ldcg(w + (size_t)t * 8 + k), v[k], acc);
    out[(size_t)t * ldo + h] = acc;
}

}  // namespace orome
