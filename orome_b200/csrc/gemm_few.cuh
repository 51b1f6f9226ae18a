// gemm_few.cuh -- the batched form for few vectors (up to 32): fp16 mma.sync, weights read and dequantized once for all of them.
//
//   Y[b][r] = sum_c W[r][c] * X[b][c]   or, fused gate/up,   silu(Wg x) * (Wu x)
//
// Same operands as the tensor-memory form (gemm_pair.cuh): weights and X rounded to fp16 once, fp32 sums.  With so few vectors that
// form is mostly its own overhead -- tensor memory and cluster set-up, partial sums of cut tiles and a kernel to add them up, MMAs
// that take the time of 128 vectors (12288 x 4096 Q8_0, 8 vectors: 7 of 20 us stream weights).  Here a CTA owns whole rows, like
// the decode kernels: no partial sums leave it, one launch behind the packing of X, and gate, up and SwiGLU are one launch.
//
//   warps 0 .. rt * kp - 1   warp = row tile (16 rows; fused: 8 of gate and the same 8 of up) x share of the 256-weight chunks;
//                            a chunk of a tile: fragments from shared memory, fp16 in registers, 16 mma (m16n8k16) per 8 vectors
//   8 (7) loader warps       packed weights as 16-byte cp.async, rows 32 or 96 bytes apart (mod 128): rows g .. g + 3 of a fragment
//                            load hit different banks
//   1 X warp                 the chunks' packed X, one bulk copy a stage
//
// A stage is kp chunks of rt * 16 rows.  The shares' sums meet in shared memory at the end of a pass over the CTA's rows (one
// pass up to 128 rows).  The mma's k slots are dealt out so that a thread's eight k of a 32-group are eight consecutive ones, in
// the weights (two packed words) as in X (16 bytes).
// What bounds it: the conversion.  12288 x 4096 at 8 vectors (83 pieces of 16 x 256 weights an SM): Q8_0 16.5 us, Q4_K 14.7, where
// memory needs 8.2 and 4.3; issue slots 0.6 used, the ALU pipe 44 and 52 %, the tensor pipe 12 %, ~740 issued instructions a piece
// with its loads and waits.  With four groups of vectors the reads of X (32 wavefronts a group and piece) and the mma come on top:
// 22.2 and 19.9 us.
#pragma once
#include "few_plan.h"
#include "gemm_common.cuh"
#include "gemv_mma.cuh"

namespace orome {

// Four groups: one fewer, for 80 registers a thread instead of 72 (17408 x 5120 Q4_K 31.4 -> 30.1 us, Q5_K 37.2 -> 34.4); with fewer groups the
// loads are what a stage waits for (three: 28.2 -> 28.5, 5120 x 5120 12.5 -> 14.2).
constexpr int gf_loaders(int nt) { return nt == 4 ? 7 : 8; }

struct GfArgs {
    const uint8_t *w0, *w1;        // the tensor; fused: gate and up
    const uint8_t *xp;             // [chunk][8 vectors][32-group][vector][32] fp16
    float *y;
    uint32_t rows, row_bytes;
    uint64_t w_bytes;
    uint32_t batch, ldy, chunks;
    uint32_t rt, kp, nstages;      // row tiles of a pass, chunks of a stage; warps = rt * kp
    // Shared memory: the shares' sums, then the stages.  The sums begin at its start, but as an address that is known when the kernel is
    // compiled it made two 9B layers at eight vectors slower (Q8_0, 138.8 -> 139.7 us): other registers, another order.
    uint32_t red_base, stage_base, stage_bytes;
    int layout;
    int *status;
};

// One superblock of 32 Q6_K rows, by a warp: half a warp per row, its 14 pieces from the 16-byte boundary at or below the row (rows
// are only 2-byte aligned).  INTERLEAVED: eight rows of `src`, eight of `src2`, and so on.  CHECK: near the tensor's end, past
// which nothing is read.  (Pieces dealt out 32 in a row, as in the other formats, cost a row's address and
// the end's comparison for every piece: 5120 x 17408 at 16 vectors 43.5 us, 39.4 like this.)
template <bool CHECK, bool INTERLEAVED>
__device__ __forceinline__ void load_q6_rows(uint32_t dst, uint32_t pitch, const uint8_t *src, const uint8_t *src2, uint32_t row_bytes, uint32_t rows_left,
                                             uint32_t stage_rows_left, const uint8_t *end, const uint8_t *end2, uint32_t lane)
{
    const uint32_t hw = lane >> 4, p = lane & 15u;
    src += hw * row_bytes;
    if constexpr (INTERLEAVED) src2 += hw * row_bytes;
    dst += hw * pitch + p * 16u;
#pragma unroll
    for (uint32_t i = 0; i < 16; ++i) {
        const bool second = INTERLEAVED && ((i >> 2) & 1u);
        const uint32_t out = INTERLEAVED ? (i >> 3) * 8u + ((2u * i) & 7u) : 2u * i;       // + hw
        if (p < 14u && out + hw < rows_left && 2u * i + hw < stage_rows_left) {
            const uint8_t *a = reinterpret_cast<const uint8_t *>(reinterpret_cast<uintptr_t>((second ? src2 : src) + out * row_bytes) & ~(uintptr_t)15) + p * 16u;
            uint32_t bytes = 16u;
            if constexpr (CHECK) {
                const uint8_t *e = second ? end2 : end;
                if (a + 16 > e) bytes = a < e ? (uint32_t)(e - a) : 0u;
                if (!bytes) a = reinterpret_cast<const uint8_t *>(reinterpret_cast<uintptr_t>(second ? src2 : src) & ~(uintptr_t)15);
            }
            cp_async16(dst + 2u * i * pitch, a, bytes);
        }
    }
}

// X fp32 [batch][ldx] -> the layout above; vectors >= batch are zero.  One thread per eight elements.
__global__ void __launch_bounds__(256)
pack_x_few_kernel(const float *__restrict__ x, uint32_t batch, uint32_t ldx, uint32_t in_dim, uint32_t nt, uint4 *__restrict__ xp)
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const uint32_t piece = blockIdx.x * 256u + threadIdx.x, n = blockIdx.y;
    if (piece >= in_dim / 8) return;
    __half2 h[4];
    h[0] = h[1] = h[2] = h[3] = __floats2half2_rn(0.f, 0.f);
    if (n < batch) {
        const float4 *src = reinterpret_cast<const float4 *>(x + (size_t)n * ldx + (size_t)piece * 8);
        const float4 a = __ldcg(src), b = __ldcg(src + 1);
        h[0] = __floats2half2_rn(a.x, a.y); h[1] = __floats2half2_rn(a.z, a.w);
        h[2] = __floats2half2_rn(b.x, b.y); h[3] = __floats2half2_rn(b.z, b.w);
    }
    const uint32_t c = piece >> 5, j = (piece >> 2) & 7u, t = piece & 3u;
    xp[((c * nt + (n >> 3)) * 8u + j) * 32u + (n & 7u) * 4u + t] = *reinterpret_cast<const uint4 *>(h);
}

__device__ __forceinline__ void mma_f16_k16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1)
{
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// What a thread holds of a row's chunk at shared address `h` besides its quants (bytes 8t .. 8t + 7 of every 32-group): d and -dmin in both
// halves, the K-quants' eight scales and minimums as bytes, Q5_K's fifth bits (Q6_K: the half's upper bits), Q6_K's scales.
struct GfRow { uint32_t h; __half2 d, dmin; uint32_t scl, sch, mnl, mnh; uint2 qh; uint32_t sc[4]; };

__device__ __forceinline__ __half2 gf_byte_pair(uint32_t w, int j, float bias)       // bytes j, j + 1 of a word as fp16, less bias
{
    const uint32_t b = __byte_perm(w, 0x64646464u, 0x4040u | (uint32_t)j | ((uint32_t)(j + 1) << 8));
    return __hsub2(*reinterpret_cast<const __half2 *>(&b), __float2half2_rn(1024.0f + bias));
}

template <int FMT>
__device__ __forceinline__ void gf_row(uint32_t h, uint32_t t, int layout, GfRow &r)
{
    r.h = h;
    if constexpr (FMT == FMT_Q4_K || FMT == FMT_Q5_K) {
        const uint4 hd = lds128<0>(h);
        unpack_scales4(hd.y, hd.z, hd.w, layout, r.scl, r.sch, r.mnl, r.mnh);
        const __half2 dd = *reinterpret_cast<const __half2 *>(&hd.x);
        r.d = __low2half2(dd);
        r.dmin = __hneg2(__high2half2(dd));
        if constexpr (FMT == FMT_Q5_K) r.qh = lds64<16>(h + 8u * t);
    } else if constexpr (FMT == FMT_Q6_K) {
        lds_words_a2<4>(h + 192u, r.sc);
        r.d = __half2half2(__ushort_as_half((unsigned short)lds16<208>(h)));
    }
}

// Two words of a row at a 2-byte aligned address.
__device__ __forceinline__ uint2 gf_words_a2(uint32_t a)
{
    uint32_t w[2];
    lds_words_a2<2>(a, w);
    return make_uint2(w[0], w[1]);
}

// Quants of groups J0 and J0 + 1 (Q6_K: J0 and J0 + 2, which share their low-nibble words) of one row as bytes, and the groups' factors.
template <int FMT, int P>
__device__ __forceinline__ void gf_pair_words(const GfRow &r, uint32_t t, uint2 &wa, uint2 &wb, __half2 &sa, __half2 &sb, __half2 &ma, __half2 &mb)
{
    ma = mb = __float2half2_rn(0.0f);
    if constexpr (FMT == FMT_Q8_0) {
        // blocks 2P, 2P + 1: fp16 scale, 32 bytes, fp16 scale, 32 bytes; the first block's words are two bytes off
        const uint32_t u = r.h + 68u * P, a = u + 8u * t;
        const uint32_t v0 = lds32<0>(a), v1 = lds32<4>(a), v2 = lds32<8>(a);
        wa = make_uint2(__byte_perm(v0, v1, 0x5432) ^ 0x80808080u, __byte_perm(v1, v2, 0x5432) ^ 0x80808080u);
        wb = make_uint2(lds32<36>(a) ^ 0x80808080u, lds32<40>(a) ^ 0x80808080u);
        const uint32_t d0 = lds32<0>(u), d1 = lds32<32>(u);
        sa = __low2half2(*reinterpret_cast<const __half2 *>(&d0));
        sb = __high2half2(*reinterpret_cast<const __half2 *>(&d1));
    } else if constexpr (FMT == FMT_Q6_K) {
        constexpr int H = P >> 1, J = P & 1;             // half of the superblock; groups J and J + 2 of it
        const uint2 ql = gf_words_a2(r.h + 64u * H + 32u * J + 8u * t), qh = r.qh;
        auto low = [](uint32_t q, uint32_t h) { return (q & 0x0F0F0F0Fu) | (((h >> (2 * J)) & 0x03030303u) << 4); };
        auto high = [](uint32_t q, uint32_t h) { return ((q >> 4) & 0x0F0F0F0Fu) | (((h >> (2 * J + 4)) & 0x03030303u) << 4); };
        wa = make_uint2(low(ql.x, qh.x), low(ql.y, qh.y));
        wb = make_uint2(high(ql.x, qh.x), high(ql.y, qh.y));
        // scale 8 H + 2 (group) + (second 16 of the group)
        const uint32_t sel = 0x8880u + (2u * J + (t >> 1)) * 0x1111u;      // one byte, sign-extended
        const int s0 = prmt_sext(r.sc[2 * H], sel), s1 = prmt_sext(r.sc[2 * H + 1], sel);
        sa = __hmul2(r.d, __half2half2(__int2half_rn(s0)));
        sb = __hmul2(r.d, __half2half2(__int2half_rn(s1)));
    } else {
        constexpr int QOFF = FMT == FMT_Q4_K ? 16 : 48;
        const uint2 q = lds64<QOFF + 32 * P>(r.h + 8u * t);
        wa = make_uint2(q.x & 0x0F0F0F0Fu, q.y & 0x0F0F0F0Fu);
        wb = make_uint2((q.x >> 4) & 0x0F0F0F0Fu, (q.y >> 4) & 0x0F0F0F0Fu);
        if constexpr (FMT == FMT_Q5_K) {
            wa.x |= ((r.qh.x >> (2 * P)) & 0x01010101u) << 4;     wa.y |= ((r.qh.y >> (2 * P)) & 0x01010101u) << 4;
            wb.x |= ((r.qh.x >> (2 * P + 1)) & 0x01010101u) << 4; wb.y |= ((r.qh.y >> (2 * P + 1)) & 0x01010101u) << 4;
        }
        const __half2 s = __hmul2(r.d, gf_byte_pair(P < 2 ? r.scl : r.sch, 2 * (P & 1), 0.0f));
        const __half2 m = __hmul2(r.dmin, gf_byte_pair(P < 2 ? r.mnl : r.mnh, 2 * (P & 1), 0.0f));
        sa = __low2half2(s); sb = __high2half2(s);
        ma = __low2half2(m); mb = __high2half2(m);
    }
}

// NA = 2 NT: even and odd k steps in sums of their own, so that one group of vectors is not one chain of 16 mma.
template <int FMT, int NT, int NA>
__device__ __forceinline__ void gf_group(const uint2 &w0, const uint2 &w1, __half2 s0, __half2 m0, __half2 s1, __half2 m1, uint32_t xa, float (&acc)[NA][4])
{
    const __half2 bias = __float2half2_rn(FMT == FMT_Q8_0 ? 1152.0f : FMT == FMT_Q6_K ? 1056.0f : 1024.0f);
    uint32_t a[2][4];
#pragma unroll
    for (int s = 0; s < 2; ++s) {
        const uint32_t q0 = s ? w0.y : w0.x, q1 = s ? w1.y : w1.x;
        a[s][0] = h2_bits(two_weights(q0, 0x5140u, bias, s0, m0)); a[s][1] = h2_bits(two_weights(q1, 0x5140u, bias, s1, m1));
        a[s][2] = h2_bits(two_weights(q0, 0x7362u, bias, s0, m0)); a[s][3] = h2_bits(two_weights(q1, 0x7362u, bias, s1, m1));
    }
#pragma unroll
    for (int n = 0; n < NT; ++n) {
        uint4 b;
        asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(b.x), "=r"(b.y), "=r"(b.z), "=r"(b.w) : "r"(xa + n * GF_X_CHUNK));
        mma_f16_k16(acc[n], a[0][0], a[0][1], a[0][2], a[0][3], b.x, b.y);
        mma_f16_k16(acc[NA == 2 * NT ? NT + n : n], a[1][0], a[1][1], a[1][2], a[1][3], b.z, b.w);
    }
}

template <int FMT, int NT, int NA, int P>
__device__ __forceinline__ void gf_pair(GfRow &r0, GfRow &r1, uint32_t t, uint32_t xl, float (&acc)[NA][4])
{
    constexpr int JA = FMT == FMT_Q6_K ? 4 * (P >> 1) + (P & 1) : 2 * P, JB = FMT == FMT_Q6_K ? JA + 2 : JA + 1;
    if constexpr (FMT == FMT_Q6_K && (P & 1) == 0) { r0.qh = gf_words_a2(r0.h + 128u + 16u * P + 8u * t); r1.qh = gf_words_a2(r1.h + 128u + 16u * P + 8u * t); }
    uint2 wa0, wb0, wa1, wb1;
    __half2 sa0, sb0, ma0, mb0, sa1, sb1, ma1, mb1;
    gf_pair_words<FMT, P>(r0, t, wa0, wb0, sa0, sb0, ma0, mb0);
    gf_pair_words<FMT, P>(r1, t, wa1, wb1, sa1, sb1, ma1, mb1);
    gf_group<FMT, NT, NA>(wa0, wa1, sa0, ma0, sa1, ma1, xl + JA * 512u, acc);
    gf_group<FMT, NT, NA>(wb0, wb1, sb0, mb0, sb1, mb1, xl + JB * 512u, acc);
}

template <int FMT, int NT, bool SWIGLU>
__global__ void __launch_bounds__((GF_MAX_WARPS + gf_loaders(NT) + 1) * 32, 1)
gemm_few_kernel(const __grid_constant__ GfArgs a)
{
    extern __shared__ __align__(128) uint8_t smem[];
    constexpr uint32_t PITCH = gf_pitch(FMT), PPR = tp_pieces(FMT);
    constexpr uint32_t CB = FMT == FMT_Q8_0 ? 272u : FMT == FMT_Q4_K ? 144u : FMT == FMT_Q5_K ? 176u : 210u;
    constexpr uint32_t TROWS = SWIGLU ? 8u : 16u;        // output rows of a tile
    constexpr uint32_t LOADERS = gf_loaders(NT);
    __shared__ uint64_t full[GF_MAX_STAGES], empty[GF_MAX_STAGES];
    __shared__ volatile int s_abort;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const uint32_t RT = a.rt, KP = a.kp, CW = RT * KP, SR = RT * 16u;        // stage rows
    const uint32_t lo = (uint32_t)((uint64_t)blockIdx.x * a.rows / gridDim.x), hi = (uint32_t)((uint64_t)(blockIdx.x + 1) * a.rows / gridDim.x);
    const uint32_t steps = (a.chunks + KP - 1) / KP, x_off = SR * KP * PITCH;
    if (tid == 0) {
        s_abort = 0;
        for (uint32_t s = 0; s < a.nstages; ++s) { mbar_init(smem_u32(full + s), LOADERS * 32 + 1); mbar_init(smem_u32(empty + s), CW); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncthreads();
    pdl_launch_dependents();
    // false: the wait ran out, here or earlier in this CTA; every loop ends then
    auto wait = [&](uint64_t *bar, uint32_t parity) -> bool {
        if (mbar_try_wait(smem_u32(bar), parity)) return true;
        if (!s_abort && mbar_wait_bounded(smem_u32(bar), parity)) return true;
        if (!s_abort) { s_abort = 1; atomicExch(a.status, 4); }
        return false;
    };

    if (warp >= CW + LOADERS) {
        // ---- X: one bulk copy a stage ----
        if (lane == 0) {
            pdl_wait();          // the packed X is the previous kernel's output
            uint32_t s = 0, ph = 1, fill = 0;
            bool ok = true;
            for (uint32_t row = lo; row < hi && ok; row += RT * TROWS) {
                for (uint32_t k = 0; k < steps; ++k, ++fill) {
                    if (fill >= a.nstages && !(ok = wait(empty + s, ph))) break;
                    const uint32_t n = min(KP, a.chunks - k * KP), bytes = n * NT * GF_X_CHUNK;
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    mbar_expect_tx(smem_u32(full + s), bytes);
                    bulk_g2s(smem_u32(smem + a.stage_base + s * a.stage_bytes + x_off), a.xp + (size_t)k * KP * NT * GF_X_CHUNK, bytes, smem_u32(full + s));
                    if (++s == a.nstages) { s = 0; ph ^= 1u; }
                }
            }
            if (!ok) {           // copies still in flight get a bounded time to land
                const long long t0 = clock64();
                while (clock64() - t0 < 200000) { }
            }
        }
        return;
    }
    if (warp >= CW) {
        // ---- loaders: packed weights, independent of the previous kernel ----
        // A warp takes 32 stage rows of a chunk at a time, consecutive lanes consecutive pieces of a row; unrolled, so that the address
        // arithmetic of a piece does not wait for the one before (as a plain loop 350 clocks a piece and lane, a third of memory's rate).
        const uint32_t lw = warp - CW, blocks = (SR + 31u) / 32u;
        uint32_t s = 0, ph = 1, fill = 0;
        bool ok = true;
        for (uint32_t row = lo; row < hi && ok; row += RT * TROWS) {
            for (uint32_t k = 0; k < steps; ++k, ++fill) {
                if (fill >= a.nstages && !(ok = wait(empty + s, ph))) break;
                const uint32_t st = smem_u32(smem + a.stage_base + s * a.stage_bytes), n = min(KP, a.chunks - k * KP);
                uint32_t j = 0, b = lw;
                for (;; b += LOADERS) {
                    while (b >= blocks) { b -= blocks; ++j; }
                    if (j >= n) break;
                    const uint32_t first = row + b * 2u * TROWS, rows_left = first < hi ? hi - first : 0u, dst0 = st + (j * SR + b * 32u) * PITCH;
                    const uint8_t *src0 = a.w0 + (size_t)first * a.row_bytes + (k * KP + j) * CB;
                    const ptrdiff_t up = SWIGLU ? a.w1 - a.w0 : 0;
                    if constexpr (FMT == FMT_Q6_K) {
                        const uint32_t stage_left = SR - b * 32u;
                        const uint8_t *end = a.w0 + a.w_bytes, *src1 = src0 + up;
                        if (src0 + (size_t)2 * TROWS * a.row_bytes + 16 <= end) load_q6_rows<false, SWIGLU>(dst0, PITCH, src0, src1, a.row_bytes, rows_left, stage_left, end, end + up, lane);
                        else load_q6_rows<true, SWIGLU>(dst0, PITCH, src0, src1, a.row_bytes, rows_left, stage_left, end, end + up, lane);
                    } else {
#pragma unroll
                        for (uint32_t i = 0; i < PPR; ++i) {
                            const uint32_t q = lane + 32u * i, r = q / PPR, p = q - r * PPR;
                            const uint32_t out = SWIGLU ? (r >> 4) * 8u + (r & 7u) : r;          // row of the tensor, from `first`
                            if (out >= rows_left || b * 32u + r >= SR) continue;                 // its sums are not stored
                            cp_async16(dst0 + r * PITCH + p * 16u, src0 + out * a.row_bytes + (SWIGLU && (r & 8u) ? up : 0) + p * 16u, 16u);
                        }
                    }
                }
                asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(full + s)) : "memory");
                if (++s == a.nstages) { s = 0; ph ^= 1u; }
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        return;
    }

    // ---- products ----
    const uint32_t g = lane >> 2, t = lane & 3u, tile = warp % RT, kph = warp / RT;
    float *red = reinterpret_cast<float *>(smem + a.red_base);
    uint32_t s = 0, ph = 0;
    for (uint32_t row = lo; row < hi; row += RT * TROWS) {
        const uint32_t row0 = row + tile * TROWS;            // this warp's output rows
        // The mma truncates where it adds: from two groups on a chunk's 16 have sums of their own, added up as fp32 (one chain over a warp's
        // chunks: 1024 x 4096 at 32 vectors 1.3e-6 off the exact product of the same operands, 3.5e-7 like this and in the tensor-memory
        // form; a single group has two chains, and more warps for its chunks: 2e-7, and 1 % slower like this).
        constexpr int NA = NT == 1 ? 2 : NT;
        float acc[NA][4], sum[NT][4];
#pragma unroll
        for (int n = 0; n < NA; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.0f;
        if constexpr (NT > 1) {
#pragma unroll
            for (int n = 0; n < NT; ++n) sum[n][0] = sum[n][1] = sum[n][2] = sum[n][3] = 0.0f;
        }
        for (uint32_t k = 0; k < steps; ++k) {
            const bool ok = wait(full + s, ph);
            const uint32_t c = k * KP + kph;
            if (__all_sync(0xffffffffu, ok) && c < a.chunks && row0 < hi) {
                const uint32_t st = smem_u32(smem + a.stage_base + s * a.stage_bytes);
                uint32_t h0 = st + (kph * SR + tile * 16u + g) * PITCH, h1 = h0 + 8u * PITCH;
                if constexpr (FMT == FMT_Q6_K) {             // where the rows start inside their first 16-byte piece
                    h0 += ((uint32_t)reinterpret_cast<uintptr_t>(a.w0) + (row0 + g) * a.row_bytes + c * CB) & 15u;
                    h1 += ((uint32_t)reinterpret_cast<uintptr_t>(SWIGLU ? a.w1 : a.w0) + (row0 + (SWIGLU ? g : g + 8u)) * a.row_bytes + c * CB) & 15u;
                }
                const uint32_t xl = st + x_off + kph * (NT * GF_X_CHUNK) + lane * 16u;
                GfRow r0, r1;
                gf_row<FMT>(h0, t, a.layout, r0);
                gf_row<FMT>(h1, t, a.layout, r1);
                gf_pair<FMT, NT, NA, 0>(r0, r1, t, xl, acc);
                gf_pair<FMT, NT, NA, 1>(r0, r1, t, xl, acc);
                gf_pair<FMT, NT, NA, 2>(r0, r1, t, xl, acc);
                gf_pair<FMT, NT, NA, 3>(r0, r1, t, xl, acc);
                if constexpr (NT > 1) {
#pragma unroll
                    for (int n = 0; n < NT; ++n) {
                        sum[n][0] += acc[n][0]; sum[n][1] += acc[n][1]; sum[n][2] += acc[n][2]; sum[n][3] += acc[n][3];
                        acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.0f;
                    }
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(empty + s));
            if (++s == a.nstages) { s = 0; ph ^= 1u; }
        }
        if constexpr (NT == 1) {
#pragma unroll
            for (int i = 0; i < 4; ++i) sum[0][i] = acc[0][i] + acc[1][i];
        }
        // the shares of a tile meet: all but the first leave theirs, the first adds them up in order
        if (KP > 1) {
            if (row != lo) named_bar_sync(PIPE_BAR_CONSUMERS, (int)(CW * 32u));      // the last pass's have been read
            if (kph > 0) {
#pragma unroll
                for (int n = 0; n < NT; ++n) *reinterpret_cast<float4 *>(red + ((size_t)(warp * NT + n) * 32u + lane) * 4u) = make_float4(sum[n][0], sum[n][1], sum[n][2], sum[n][3]);
            }
            named_bar_sync(PIPE_BAR_CONSUMERS, (int)(CW * 32u));
            if (kph > 0) continue;
            for (uint32_t o = 1; o < KP; ++o) {
#pragma unroll
                for (int n = 0; n < NT; ++n) {
                    const float4 v = *reinterpret_cast<const float4 *>(red + ((size_t)((o * RT + tile) * NT + n) * 32u + lane) * 4u);
                    sum[n][0] += v.x; sum[n][1] += v.y; sum[n][2] += v.z; sum[n][3] += v.w;
                }
            }
        }
        if (s_abort) continue;
        // a thread holds rows g, g + 8 (fused: gate and up of row g) of vectors 8n + 2t, 8n + 2t + 1
#pragma unroll
        for (int n = 0; n < NT; ++n) {
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const uint32_t v = n * 8u + 2u * t + q;
                if (v >= a.batch) continue;
                float *dst = a.y + (size_t)v * a.ldy + row0 + g;
                if constexpr (SWIGLU) {
                    if (row0 + g < hi) *dst = silu_mul(sum[n][q], sum[n][2 + q]);
                } else {
                    if (row0 + g < hi) dst[0] = sum[n][q];
                    if (row0 + g + 8u < hi) dst[8] = sum[n][2 + q];
                }
            }
        }
    }
}

}  // namespace orome
