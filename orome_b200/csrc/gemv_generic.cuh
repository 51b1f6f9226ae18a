// gemv_generic.cuh -- shape-agnostic kernels: row decode, warp-per-row matvec for
// any format / batch, SwiGLU epilogue.  They take every shape the formats allow;
// the pipelined kernels in gemv_pipe.cuh take over for the decode-sized ones.
#pragma once
#include "decode.cuh"

namespace orome {

// One thread per 32-weight group: out[(r - row0) * in_dim + 32*b .. +32].  The unquantized formats.
// Device counterpart of format_decode_row_f32 (format.m:176-218).
template <int FMT>
__global__ void dequant_rows_kernel(const uint8_t *__restrict__ data, size_t row_bytes, uint32_t row0, uint32_t nrows,
                                    uint32_t in_dim, int layout, float *__restrict__ out)
{
    static_assert(FMT >= FMT_F16, "quantized rows: dequant_flat_kernel");
    uint32_t groups = in_dim / 32;
    size_t gid = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (gid >= (size_t)nrows * groups) return;
    uint32_t r = (uint32_t)(gid / groups), b = (uint32_t)(gid % groups);
    float w[32];
    decode32<FMT>(data + (size_t)(row0 + r) * row_bytes, b, layout, w);
    float4 *o = reinterpret_cast<float4 *>(out + (size_t)r * in_dim + (size_t)b * 32);
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] = make_float4(w[4 * j], w[4 * j + 1], w[4 * j + 2], w[4 * j + 3]);
}

// Eight bytes from a 2-byte aligned address, as two words.  Stays inside [p - 2, p + 8).
__device__ __forceinline__ uint2 ld8_a2(const uint8_t *p)
{
    const bool odd = (reinterpret_cast<uintptr_t>(p) & 2u) != 0;
    const uint32_t *q = reinterpret_cast<const uint32_t *>(reinterpret_cast<uintptr_t>(p) & ~(uintptr_t)3);
    const uint32_t a = __ldcg(q), b = __ldcg(q + 1), c = odd ? (uint32_t)__ldcg(reinterpret_cast<const unsigned short *>(p + 6)) : 0u, sh = odd ? 16u : 0u;
    return make_uint2(__funnelshift_r(a, b, sh), __funnelshift_r(b, c, sh));
}

// Byte `b` of a word less `bias` (an integer), exactly, as a float: on top of the bits of 2^23 the byte is a float that much too large.  I2F
// runs at an eighth of the rate of the permute and the subtraction.
__device__ __forceinline__ float byte_float(uint32_t v, int b, float bias)
{
    return __uint_as_float(__byte_perm(v, 0x4B000000u, 0x7440u + (uint32_t)b)) - (8388608.0f + bias);
}

// Rows of a quantized tensor lie one behind the other without gaps, so a range of rows is one run of 8-weight pieces: thread i
// decodes pieces i, i + 32, .. of its warp's 1024 weights and stores 32 bytes a piece, so that a warp's stores are whole lines
// and its loads fall into a few (a thread per 32-weight block, loading bytes and storing 128 bytes apart, ran at a third of the
// memory rate: 5120 x 4096 Q6_K 47 us).  Bit-exact like decode32: the same rounded operations on the same integers.
constexpr uint32_t DQ_PIECES = 4;            // pieces a thread has in flight
template <int FMT>
__global__ void __launch_bounds__(256)
dequant_flat_kernel(const uint8_t *__restrict__ blocks, uint64_t pieces, int layout, float *__restrict__ out)
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t base = ((uint64_t)blockIdx.x * 8u + (threadIdx.x >> 5)) * (32u * DQ_PIECES) + lane;
    // The packed rows may be what the kernel before has written: nothing of them is loaded before the wait (nor without coherence
    // after it), but their lines may come to the L2, where that kernel's writes go too (5120 x 4096 Q6_K, back to back: 29.8 us
    // without, 25.7 with).
    constexpr uint32_t GROUP = FMT == FMT_Q8_0 ? 4u : 32u, BLOCK = FMT == FMT_Q8_0 ? 34u : FMT == FMT_Q4_K ? 144u : FMT == FMT_Q5_K ? 176u : 210u;
    const uint64_t first = (base - lane) / GROUP * BLOCK + 128u * lane;
    if (128u * lane < 32u * DQ_PIECES / GROUP * BLOCK && first < pieces / GROUP * BLOCK) asm volatile("prefetch.global.L2 [%0];" ::"l"(blocks + first));
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const bool whole = (reinterpret_cast<uintptr_t>(out) & 31) == 0;      // a piece in one store: whole lines a warp
    uint2 q[DQ_PIECES], h[DQ_PIECES];
    uint4 hd[DQ_PIECES];
    uint32_t d[DQ_PIECES];
    int sc[DQ_PIECES];
#pragma unroll
    for (uint32_t k = 0; k < DQ_PIECES; ++k) {
        const uint64_t i = base + 32u * k;
        if (i >= pieces) continue;
        if constexpr (FMT == FMT_Q8_0) {
            const uint8_t *blk = blocks + (i >> 2) * 34u;
            d[k] = __ldcg(reinterpret_cast<const unsigned short *>(blk));
            q[k] = ld8_a2(blk + 2 + 8u * (i & 3u));
        } else if constexpr (FMT == FMT_Q6_K) {
            const uint8_t *sb = blocks + (i >> 5) * 210u;
            const uint32_t p = (uint32_t)i & 31u, half = p >> 4, j = (p >> 2) & 3u, l = 8u * (p & 3u);
            q[k] = ld8_a2(sb + 64u * half + 32u * (j & 1u) + l);
            h[k] = ld8_a2(sb + 128u + 32u * half + l);
            sc[k] = (int)(signed char)__ldcg(sb + 192u + 8u * half + 2u * j + (l >> 4));
            d[k] = __ldcg(reinterpret_cast<const unsigned short *>(sb + 208));
        } else {
            constexpr uint32_t UNIT = FMT == FMT_Q4_K ? 144u : 176u, QOFF = FMT == FMT_Q4_K ? 16u : 48u;
            const uint8_t *sb = blocks + (i >> 5) * UNIT;
            const uint32_t p = (uint32_t)i & 31u;
            hd[k] = __ldcg(reinterpret_cast<const uint4 *>(sb));
            q[k] = __ldcg(reinterpret_cast<const uint2 *>(sb + QOFF + 32u * (p >> 3) + 8u * (p & 3u)));
            if constexpr (FMT == FMT_Q5_K) h[k] = __ldcg(reinterpret_cast<const uint2 *>(sb + 16u + 8u * (p & 3u)));
        }
    }
#pragma unroll
    for (uint32_t k = 0; k < DQ_PIECES; ++k) {
        const uint64_t i = base + 32u * k;
        if (i >= pieces) continue;
        const uint32_t p = (uint32_t)i & 31u;
        float w[8];
        if constexpr (FMT == FMT_Q8_0) {
            const float dd = half_bits_to_float(d[k]);
#pragma unroll
            for (int b = 0; b < 8; ++b) w[b] = __fmul_rn(dd, byte_float((b < 4 ? q[k].x : q[k].y) ^ 0x80808080u, b & 3, 128.0f));
        } else if constexpr (FMT == FMT_Q6_K) {
            const uint32_t j = (p >> 2) & 3u;
            const float a = __fmul_rn(half_bits_to_float(d[k]), (float)sc[k]);
            const uint32_t lo0 = (q[k].x >> (4u * (j >> 1))) & 0x0F0F0F0Fu, lo1 = (q[k].y >> (4u * (j >> 1))) & 0x0F0F0F0Fu;
            const uint32_t v0 = lo0 | (((h[k].x >> (2u * j)) & 0x03030303u) << 4), v1 = lo1 | (((h[k].y >> (2u * j)) & 0x03030303u) << 4);
#pragma unroll
            for (int b = 0; b < 8; ++b) w[b] = __fmul_rn(a, byte_float(b < 4 ? v0 : v1, b & 3, 32.0f));
        } else {
            const uint32_t sub = p >> 2, shift = 4u * (sub & 1u), w0 = hd[k].y, w1 = hd[k].z, w2 = hd[k].w;
            auto byte = [](uint32_t v, uint32_t n) { return (v >> (8u * n)) & 255u; };
            uint32_t s, m;                       // kq_scale_min on words: w0 = bytes 0-3, w1 = 4-7, w2 = 8-11
            if (sub < 4) { s = byte(w0, sub) & 63u; m = byte(w1, sub) & 63u; }
            else if (layout == LAYOUT_A) {
                const uint32_t u = (sub - 4) >> 1, hi = sub & 1u, sp = byte(w2, u), mp = byte(w2, 2 + u);
                s = (hi ? (sp >> 4) : (sp & 15u)) | ((byte(w0, 2 * u + hi) >> 6) << 4);
                m = (hi ? (mp >> 4) : (mp & 15u)) | ((byte(w1, 2 * u + hi) >> 6) << 4);
            } else {
                s = (byte(w2, sub - 4) & 15u) | ((byte(w0, sub - 4) >> 6) << 4);
                m = (byte(w2, sub - 4) >> 4) | ((byte(w1, sub - 4) >> 6) << 4);
            }
            const float a = __fmul_rn(half_bits_to_float(hd[k].x & 0xffffu), (float)s), mm = __fmul_rn(half_bits_to_float(hd[k].x >> 16), (float)m);
            uint32_t v0 = (q[k].x >> shift) & 0x0F0F0F0Fu, v1 = (q[k].y >> shift) & 0x0F0F0F0Fu;
            if constexpr (FMT == FMT_Q5_K) { v0 |= ((h[k].x >> sub) & 0x01010101u) << 4; v1 |= ((h[k].y >> sub) & 0x01010101u) << 4; }
#pragma unroll
            for (int b = 0; b < 8; ++b) w[b] = __fsub_rn(__fmul_rn(a, byte_float(b < 4 ? v0 : v1, b & 3, 0.0f)), mm);
        }
        float4 *o = reinterpret_cast<float4 *>(out + i * 8u);
        if (whole) asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                                ::"l"(o), "f"(w[0]), "f"(w[1]), "f"(w[2]), "f"(w[3]), "f"(w[4]), "f"(w[5]), "f"(w[6]), "f"(w[7]) : "memory");
        else {
            o[0] = make_float4(w[0], w[1], w[2], w[3]);
            o[1] = make_float4(w[4], w[5], w[6], w[7]);
        }
    }
}

// Tail of an unquantized row whose length is not a multiple of 32 (F32/F16/BF16 only).
template <int FMT>
__device__ __forceinline__ float plain_elem(const uint8_t *row, uint32_t c)
{
    if constexpr (FMT == FMT_F32) return reinterpret_cast<const float *>(row)[c];
    else if constexpr (FMT == FMT_F16) return half_bits_to_float(ld16(row + 2 * (size_t)c));
    else return __uint_as_float(ld16(row + 2 * (size_t)c) << 16);
}

// y[b][r] = sum_c W[r][c] x[b][c]; one warp per row, lanes stride over 32-weight
// groups, NB batch columns per pass (the weights are decoded once per pass).
template <int FMT, int NB>
__global__ void __launch_bounds__(256)
gemv_generic_kernel(const uint8_t *__restrict__ data, size_t row_bytes, uint32_t out_dim, uint32_t in_dim, int layout,
                    const float *__restrict__ x, int batch, int ldx, float *__restrict__ y, int ldy)
{
    uint32_t row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    uint32_t lane = threadIdx.x & 31;
    if (row >= out_dim) return;
    const uint8_t *rp = data + (size_t)row * row_bytes;
    uint32_t groups = in_dim / 32;
    for (int b0 = 0; b0 < batch; b0 += NB) {
        float acc[NB];
#pragma unroll
        for (int i = 0; i < NB; ++i) acc[i] = 0.0f;
        for (uint32_t g = lane; g < groups; g += 32) {
            float w[32];
            decode32<FMT>(rp, g, layout, w);
#pragma unroll
            for (int i = 0; i < NB; ++i) {
                if (b0 + i < batch) {
                    const float *xb = x + (size_t)(b0 + i) * ldx + (size_t)g * 32;
                    float a = 0.0f;
#pragma unroll
                    for (int j = 0; j < 32; ++j) a = fmaf(w[j], xb[j], a);
                    acc[i] += a;
                }
            }
        }
        if constexpr (FMT == FMT_F32 || FMT == FMT_F16 || FMT == FMT_BF16) {
            for (uint32_t c = groups * 32 + lane; c < in_dim; c += 32) {
                float wv = plain_elem<FMT>(rp, c);
#pragma unroll
                for (int i = 0; i < NB; ++i)
                    if (b0 + i < batch) acc[i] = fmaf(wv, x[(size_t)(b0 + i) * ldx + c], acc[i]);
            }
        }
#pragma unroll
        for (int i = 0; i < NB; ++i) {
            float s = warp_sum(acc[i]);
            if (lane == 0 && b0 + i < batch) y[(size_t)(b0 + i) * ldy + row] = s;
        }
    }
}

// fp32 weights (the MoE router, shaders.metal:1342-1366): one warp per row, lanes take consecutive float4s so every
// load is coalesced; up to 4 input vectors per pass.  Waits for the previous kernel first (it may produce x).
// With W1 set, one more output row (index out_dim) comes from that single-row tensor: the router logits and the
// shared-expert gate logit in one launch, as matvec_f32_pair does (shaders.metal:1368-1392).
__global__ void __launch_bounds__(128)
gemv_f32_kernel(const float *__restrict__ W, uint32_t out_dim, uint32_t in_dim, const float *__restrict__ x, int batch, int ldx,
                float *__restrict__ y, int ldy, const float *__restrict__ W1 = nullptr)
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");   // the next kernel may set itself up; it waits for this one's results itself
    asm volatile("griddepcontrol.wait;" ::: "memory");
    // One CTA of four warps per row: a 2048-wide row is then one round of four 16-byte loads per thread, all in flight
    // together (a warp per row needed four dependent rounds, and a 128-row router matrix kept only 33 CTAs busy).
    const uint32_t row = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const float4 *w4 = reinterpret_cast<const float4 *>(row < out_dim ? W + (size_t)row * in_dim : W1);
    const uint32_t n4 = in_dim / 4;
    // grid.y cuts the batch into groups of four vectors
    const int b0 = (int)blockIdx.y * 4;
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    for (uint32_t c0 = tid; c0 < n4; c0 += 512) {
        float4 w[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) w[u] = c0 + 128 * u < n4 ? __ldg(w4 + c0 + 128 * u) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (b0 + i < batch) {
                const float4 *x4 = reinterpret_cast<const float4 *>(x + (size_t)(b0 + i) * ldx);
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    if (c0 + 128 * u < n4) {
                        const float4 xv = __ldcg(x4 + c0 + 128 * u);
                        acc[i] = fmaf(w[u].x, xv.x, fmaf(w[u].y, xv.y, fmaf(w[u].z, xv.z, fmaf(w[u].w, xv.w, acc[i]))));
                    }
                }
            }
        }
    }
    __shared__ float red[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float s = warp_sum(acc[i]);
        if (lane == 0) red[warp][i] = s;
    }
    __syncthreads();
    if (tid < 4 && b0 + (int)tid < batch) y[(size_t)(b0 + tid) * ldy + row] = (red[0][tid] + red[1][tid]) + (red[2][tid] + red[3][tid]);
}

// out = silu(gate) * up, elementwise (shaders.metal:1018-1030); used after two products when the fused kernel does not take the
// shape.  Bound by memory: four elements a thread, 16-byte accesses where rows and pointers allow; blockIdx.y strides over rows.
__global__ void __launch_bounds__(256)
swiglu_kernel(const float *__restrict__ gate, const float *__restrict__ up, float *__restrict__ out, uint32_t n, int batch, int ldg, int ldo)
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const uint32_t c = (blockIdx.x * 256u + threadIdx.x) * 4u;
    if (c >= n) return;
    const bool wide = c + 4 <= n && !((reinterpret_cast<uintptr_t>(gate) | reinterpret_cast<uintptr_t>(up) | reinterpret_cast<uintptr_t>(out)) & 15) &&
                      !((ldg | ldo) & 3);
    for (int b = blockIdx.y; b < batch; b += gridDim.y) {
        const float *g = gate + (size_t)b * ldg + c, *u = up + (size_t)b * ldg + c;
        float *o = out + (size_t)b * ldo + c;
        if (wide) {
            const float4 gv = __ldcg(reinterpret_cast<const float4 *>(g)), uv = __ldcg(reinterpret_cast<const float4 *>(u));
            *reinterpret_cast<float4 *>(o) = make_float4(silu_mul(gv.x, uv.x), silu_mul(gv.y, uv.y), silu_mul(gv.z, uv.z), silu_mul(gv.w, uv.w));
        } else {
            for (uint32_t q = 0; q < 4 && c + q < n; ++q) o[q] = silu_mul(__ldcg(g + q), __ldcg(u + q));
        }
    }
}

// Index of the largest element: argmax_kernel (shaders.metal:1249-1305), dispatched after the lm_head at
// engine.m:1036-1046 so that a token costs the host a 4-byte read.  The reference runs one threadgroup of 1024
// threads; one CTA reading 600 KB takes tens of microseconds here, so the vector is cut over up to 148 CTAs.
// Candidates are compared as {value key, ~tie rank} (argmax_rank), a total order in which equal values resolve
// exactly as the reference's strided scan and shuffle-down trees do, so the cut changes nothing; NaN and -inf never
// win, an input without candidates gives index 0.  state[0]: running best (atomicMax), state[1]: CTAs done; the last
// CTA writes the result and clears both for the next call.
__global__ void __launch_bounds__(256)
argmax_kernel(const float *__restrict__ data, uint32_t count, uint32_t *__restrict__ result, unsigned long long *__restrict__ state)
{
    __shared__ unsigned long long s_best[8];
    asm volatile("griddepcontrol.wait;" ::: "memory");
    unsigned long long best = 0ull;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
        const float v = __ldcg(data + i);
        if (v > -INFINITY) {
            const unsigned long long cand = ((unsigned long long)float_key(v) << 32) | (uint32_t)~argmax_rank(i);
            if (cand > best) best = cand;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long other = __shfl_xor_sync(0xffffffffu, best, o);
        if (other > best) best = other;
    }
    if ((threadIdx.x & 31u) == 0) s_best[threadIdx.x >> 5] = best;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w) if (s_best[w] > best) best = s_best[w];
        if (best) atomicMax(state, best);
        __threadfence();
        if (atomicAdd(state + 1, 1ull) == gridDim.x - 1) {
            __threadfence();
            const unsigned long long m = atomicExch(state, 0ull);
            *result = m ? argmax_unrank(~(uint32_t)m) : 0u;
            atomicExch(state + 1, 0ull);
        }
    }
}

}  // namespace orome
