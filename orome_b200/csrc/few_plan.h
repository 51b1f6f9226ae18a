// few_plan.h -- how the batched form for few vectors (gemm_few.cuh) cuts a product over CTAs, warps and stages, and where it is the faster
// form.  Host arithmetic only, so that it can be checked without a GPU.
#pragma once
#include <algorithm>
#include <cstddef>
#include <cstdint>

#include "../../include/orome_cuda.h"

namespace orome {

constexpr int GF_MAX_VECTORS = 32, GF_MAX_WARPS = 16, GF_MAX_STAGES = 8;
constexpr uint32_t GF_KC = 256;              // weights of a chunk
constexpr uint32_t GF_X_CHUNK = 4096;        // packed X of one chunk and eight vectors
constexpr uint32_t gf_pitch(int fmt) { return fmt == OROME_QFMT_GGUF_Q8_0 ? 288u : fmt == OROME_QFMT_GGUF_Q4_K ? 160u : 224u; }

struct FewShape {
    int fmt;
    uint32_t out_dim, in_dim, batch;
    bool fused;                    // gate, up and SwiGLU in one launch
    uint32_t sm_count;
    size_t smem_optin;             // shared memory a CTA may ask for
};

struct FewPlan {
    uint32_t grid, tiles;          // CTAs take equal row ranges; row tiles (16 rows; fused: 8 of gate and 8 of up) of the busiest one
    uint32_t passes, rt;           // a pass covers rt row tiles, at most eight
    uint32_t kp, steps;            // the warps that a pass's row tiles leave split the chunks of a row: kp of them a stage, steps stages a pass
    uint32_t nstages, stage_base, stage_bytes, bytes;      // shared memory: the sums of a row's shares, then the stages; all of it
};

inline uint32_t few_tile_rows(bool fused) { return fused ? 8u : 16u; }
inline uint32_t few_groups(uint32_t batch) { return (batch + 7) / 8; }

inline void few_rows(const FewShape &in, FewPlan &p)
{
    const uint32_t trows = few_tile_rows(in.fused);
    p.grid = std::max(1u, std::min(in.sm_count, (in.out_dim + trows - 1) / trows));
    p.tiles = ((in.out_dim + p.grid - 1) / p.grid + trows - 1) / trows;
    p.passes = (p.tiles + 7) / 8;
    p.rt = (p.tiles + p.passes - 1) / p.passes;
}

// false: not even one stage fits
inline bool few_plan(const FewShape &in, FewPlan &p)
{
    few_rows(in, p);
    const uint32_t chunks = in.in_dim / GF_KC, nt = few_groups(in.batch);
    const size_t room = in.smem_optin - 1024;
    for (uint32_t kp = std::min((uint32_t)GF_MAX_WARPS / p.rt, chunks);; --kp) {
        p.steps = (chunks + kp - 1) / kp;
        p.kp = (chunks + p.steps - 1) / p.steps;
        p.stage_bytes = p.rt * 16 * p.kp * gf_pitch(in.fmt) + p.kp * nt * GF_X_CHUNK;
        p.stage_base = p.kp > 1 ? p.rt * p.kp * nt * 512 : 0;
        p.nstages = p.stage_base + (size_t)p.stage_bytes <= room ? (uint32_t)std::min<size_t>(GF_MAX_STAGES, (room - p.stage_base) / p.stage_bytes) : 0u;
        p.nstages = std::min(p.nstages, p.steps * p.passes);
        p.bytes = p.stage_base + p.nstages * p.stage_bytes;
        if (p.nstages >= std::min(2u, p.steps * p.passes) || kp == 1) break;      // two stages at least, so that loads and products overlap
    }
    return p.nstages > 0;
}

// Where this form is the faster one: a cost model in us.  This form: 3.5 and so much a piece (row tile x chunk) of the busiest CTA, by format
// and groups of eight vectors; the tensor-memory form: 7 and so much per 2^20 weights; fused, it is two products and a pass.  1800 random
// products (4 formats, 4 to 32 vectors): 0.5 % slower than the better form on average, 4 % of them by more than 5 %, Q6_K by up to 1.33x
// where its tiles in the other form stay whole.  Fitting the constants anew to half of them, or stages, shares and cuts as terms, gained
// nothing on the other half.  Measured, this form / the other: Q4_K 1024x4096 at 24 vectors 6.4 / 8.8, 12288x4096 at 8 14.7 / 17.2 and at
// 32 20.3 / 18.5, Q8_0 4096x4096 at 16 8.8 / 9.8, 17408x5120 at 8 27.1 / 25.3, Q6_K 12288x4096 at 24 22.1 / 29.0, 2560x9728 at 8 17.2 /
// 14.0; gate/up of 9728x2560 at 8 Q8_0 19.1 / 26.5.  (5 % margin: where the two are that close it does not matter.)
inline bool few_faster(const FewShape &in)
{
    const bool q8 = in.fmt == OROME_QFMT_GGUF_Q8_0, q4 = in.fmt == OROME_QFMT_GGUF_Q4_K, q5 = in.fmt == OROME_QFMT_GGUF_Q5_K;
    const uint32_t nt = few_groups(in.batch);
    const double piece = q8 ? 0.110 + 0.018 * nt : q4 ? 0.095 + 0.0145 * nt : q5 ? 0.100 + 0.019 * nt : 0.155 + 0.016 * nt;
    const double mega = q8 ? 0.24 : q4 ? 0.21 : q5 ? 0.235 : 0.335;
    FewPlan p;
    few_rows(in, p);
    const double few = 3.5 + piece * p.tiles * (in.in_dim / GF_KC), pair = 7.0 + mega * ((double)in.out_dim * in.in_dim / 1048576.0);
    return 1.05 * few < (in.fused ? 2.0 * pair + 3.0 : pair);
}

}  // namespace orome
