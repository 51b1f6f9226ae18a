// gemm_common.cuh -- what the batched forms share: fetching packed rows, packed bytes to fp16 pairs.
#pragma once
#include <cuda_fp16.h>

#include "gemm.h"

namespace orome {

// 16-byte pieces a chunk of a row is fetched as.  Q6_K rows are only 2-byte aligned: the 210 bytes of a superblock lie in 14 pieces
// from the boundary below.
__host__ __device__ constexpr uint32_t tp_pieces(int fmt) { return fmt == FMT_Q8_0 ? 17 : fmt == FMT_Q4_K ? 9 : fmt == FMT_Q5_K ? 11 : 14; }

__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src, uint32_t bytes)      // bytes < 16: the rest is zero-filled
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

// N consecutive 32-bit words of shared memory from a 2-byte aligned address.
template <int N>
__device__ __forceinline__ void lds_words_a2(uint32_t a, uint32_t (&out)[N])
{
    const uint32_t q = a & ~3u, sh = (a & 2u) * 8u;
    uint32_t w[N + 1];
#pragma unroll
    for (int i = 0; i <= N; ++i) w[i] = lds32<0>(q + 4u * i);
#pragma unroll
    for (int i = 0; i < N; ++i) out[i] = __funnelshift_r(w[i], w[i + 1], sh);
}

__device__ __forceinline__ uint32_t h2_bits(__half2 v) { return *reinterpret_cast<uint32_t *>(&v); }

// Two byte lanes of `w` (selected by `sel`) -> fp16 pair (byte - bias) * scale + addend.  0x6400 | byte is the
// fp16 number 1024 + byte exactly, so the bias comes off exactly before the one rounded multiply-add.
__device__ __forceinline__ __half2 two_weights(uint32_t w, uint32_t sel, __half2 bias, __half2 scale, __half2 addend)
{
    const uint32_t bits = __byte_perm(w, 0x64646464u, sel);
    return __hfma2(__hsub2(*reinterpret_cast<const __half2 *>(&bits), bias), scale, addend);
}

}  // namespace orome
