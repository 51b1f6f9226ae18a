// mma_plan.h -- how the K-quant mma kernel (gemv_mma.cuh) cuts rows into stages and lays its ring out in shared memory.  Host
// arithmetic only, so that it can be checked without a GPU.
#pragma once
#include <algorithm>
#include <cstddef>
#include <cstdint>

namespace orome {

constexpr int MMA_TILE_ROWS = 16;
constexpr int MMA_MAX_WARPS = 8;                  // consumer warps of a group
constexpr int MMA_MAX_GROUPS = 5;
constexpr int MMA_MAX_CONSUMER_WARPS = 16;        // groups * warps per group
constexpr int MMA_MAX_PRODUCERS = 2;              // producer warps (two where every row is its own copy)
constexpr int MMA_MAX_STAGES = 16;

struct MmaRingShape {
    bool q6;                       // 210-byte superblocks: rows arrive by their own copies, issued by two producer warps
    uint32_t unit, units_row;      // bytes of a superblock, superblocks of a row
    uint32_t nvec;                 // combine form: input vectors of a row (0: plain)
    uint32_t share;                // rows of the busiest CTA
    bool swiglu, two;              // gate and up rows side by side; two input vectors at once
    size_t xq_sb, smem_optin;      // bytes of quantized x per superblock; shared memory a CTA may ask for
    uint32_t stage_kb;             // KiB of a stage (0: chosen here)
};

struct MmaRing {
    uint32_t units, nchunks, kc;             // superblocks per row (of all vectors), stages per row tile, superblocks per stage
    uint32_t nwarps, ngroups, nstages;
    uint32_t pitch, half_stride, stage_stride;
    uint32_t red_base, red_rows, xs_base, stage_base;
};

enum { MMA_RING_OK = 0, MMA_RING_SHALLOW = 1, MMA_RING_NO_ROOM = 2 };

// A stage of at most `want` bytes: 16 rows (x2 in the fused gate/up form) of kc superblocks.
inline int mma_lay_out(const MmaRingShape &in, uint32_t want, bool odd, MmaRing &a)
{
    const uint32_t kc_max = std::max(1u, std::min(in.units_row, want / (MMA_TILE_ROWS * in.unit * (in.swiglu ? 2u : 1u))));
    a.units = in.units_row * std::max(1u, in.nvec);
    if (in.nvec > 0) {
        if (in.units_row > kc_max) return MMA_RING_NO_ROOM;
        a.nchunks = in.nvec;
        a.kc = in.units_row;
    } else {
        a.nchunks = (a.units + kc_max - 1) / kc_max;
        a.kc = (a.units + a.nchunks - 1) / a.nchunks;
    }
    const uint32_t rounds = (a.kc + MMA_MAX_WARPS - 1) / MMA_MAX_WARPS;
    a.nwarps = (a.kc + rounds - 1) / rounds;
    // stages (row tiles x chunks) go round the groups: as many groups as the warp budget and the CTA's stage count allow
    const uint32_t row_tiles = (in.share + MMA_TILE_ROWS - 1) / MMA_TILE_ROWS, cta_stages = row_tiles * a.nchunks;
    a.ngroups = std::max(1u, std::min(std::min<uint32_t>(MMA_MAX_GROUPS, MMA_MAX_CONSUMER_WARPS / a.nwarps), cta_stages));
    // box width in superblocks: the smallest kb >= kc with kb = 2 (mod 4), which makes the row pitch 32 or 96 (mod 128)
    a.pitch = (a.kc + ((6 - a.kc % 4) % 4)) * in.unit;
    if (in.q6) {
        // rows are widened to 16-byte boundaries (up to 15 bytes before and after the chunk)
        a.pitch = (a.kc * in.unit + 30 + 15) / 16 * 16;
        while (a.pitch % 128 != 16) a.pitch += 16;      // the quads of the eight rows of a load then read eight different four-bank groups
    }
    a.half_stride = MMA_TILE_ROWS * a.pitch;
    a.stage_stride = a.half_stride * (in.swiglu ? 2 : 1);
    a.red_base = 2 * 8 * MMA_MAX_STAGES;
    a.red_rows = std::max<uint32_t>(MMA_TILE_ROWS, std::min<uint32_t>(row_tiles * MMA_TILE_ROWS, 128u));
    const size_t red_bytes = (size_t)2 * a.red_rows * a.nwarps * a.ngroups * (in.swiglu || in.two ? 2 : 1) * sizeof(float);
    a.xs_base = (uint32_t)((a.red_base + red_bytes + 127) / 128 * 128);
    const size_t xq_bytes = (size_t)a.units * in.xq_sb + (size_t)a.units * 8 * (in.two ? 2 : 1) + 768;   // planes and sums, two scales per superblock and vector, a block of zeros
    a.stage_base = (uint32_t)((a.xs_base + xq_bytes + 127) / 128 * 128);
    const size_t budget = std::min<size_t>(228 * 1024 - 1024 - 256, in.smem_optin - 256);
    if (budget < (size_t)a.stage_base + a.stage_stride) return MMA_RING_NO_ROOM;
    a.nstages = (uint32_t)std::min<size_t>(std::min<size_t>(MMA_MAX_STAGES, (row_tiles + 1) * a.nchunks), (budget - a.stage_base) / a.stage_stride);
    // A whole number of ring slots per group, so that every use of a slot belongs to the same group.  A wait by parity tells
    // only the last two phases apart: a group waiting for use k of a slot whose use k - 1 is another group's, and has not
    // landed yet, would take phase k - 2 for phase k and read the stage too early.
    a.ngroups = std::min(a.ngroups, a.nstages);
    // `odd`: three or more slots for two groups, where the kernel makes a group wait for the slot's other user first.  That needs
    // ONE producer: it fills the slots in order, so a warp that has read its group's stage i - 2 knows that stage i - nstages was
    // issued, hence that its whole group is through with the slot's use before.  Two producers (Q6_K) are not ordered with each
    // other: a warp whose neighbour lags would pass both waits on the use two back and read an old stage.
    if (!(odd && !in.q6 && a.ngroups == 2 && a.nstages >= 3)) a.nstages -= a.nstages % a.ngroups;
    return a.nstages >= std::min(2 * a.ngroups, cta_stages) ? MMA_RING_OK : MMA_RING_SHALLOW;
}

// 40-KiB stages, or smaller ones where that leaves a consumer group fewer than two ring slots: with one, a group waits out every
// copy into the slot it has just read.  27B shapes, one slot a group / the largest stage that leaves two: gate/up 32.6 / 23.4 us,
// fused down 36.5 / 28.6, lm_head 155 / 131.
inline int mma_plan_ring(const MmaRingShape &in, MmaRing &a)
{
    if (in.stage_kb || in.nvec > 0) return mma_lay_out(in, (in.stage_kb ? in.stage_kb : 40u) * 1024u, true, a);
    int fit = MMA_RING_NO_ROOM;
    for (uint32_t kb = 40; kb >= 16 && fit != MMA_RING_OK; kb -= 4) {
        fit = mma_lay_out(in, kb * 1024u, false, a);
        if (fit == MMA_RING_OK && kb < 40 && a.nwarps * a.ngroups < 12) fit = MMA_RING_SHALLOW;      // narrow stages that leave warps idle cost more (7-superblock rows: 3 %)
    }
    return fit == MMA_RING_SHALLOW ? mma_lay_out(in, 40u * 1024u, true, a) : fit;      // shallow at every size: the largest stage
}

}  // namespace orome
