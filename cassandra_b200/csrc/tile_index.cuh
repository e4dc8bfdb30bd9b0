// The indexers as a matrix product on the tensor cores.
//
// Every column index is a combination of digit lists sum_i 3^i cell(sq_i),
// and the lists of all slots are linear in the 64 cells: (rows x 64 cells)
// times (64 x lists weights).  A warp takes 32 rows and multiplies them by
// tiles of 8 lists with mma.sync m16n8k32 (bytes in, 32-bit integers out, so
// every step is exact):
//
//   A  cell values 0, 1, 2 as bytes: the bits of a position's words masked
//      into place are the operand, four cells a register.  A lane's
//      registers are squares 2t + s + {0, 8, 16, 24} of a word (t the lane
//      in its quad, s the k-step); the weights are stored in that order
//      (append_tile).
//   B  weights 3^i up to 3^10 as a low and a high byte; tiles of short lists
//      have no high bytes and take half the instructions.
//
// The general kernel reads digit boards: a shared-memory load and a
// multiply-add per square, 570 squares a row of the 8-pattern expanded set,
// bound by instruction issue.  Here 16 such rows take 32 tensor instructions
// (8.3 cycles each per SM quarter, measured; the m16n8k16 form on halves
// runs at the same rate and needs twice as many) and the kernel is bound by
// the write of the indices.  A product this small has no use for tcgen05:
// its operand would have to be expanded into shared memory first, where
// mma.sync takes it from the registers that made it.
#pragma once
#include <cstdint>

#include "tile_index.h"

namespace cas {

constexpr int kTileRows = 32;      // rows of a warp's step
constexpr int kTileThreads = 256;  // threads of a CTA of the tile indexers

// A fragments of 32 rows: [16-row half][k-step][register].
struct CellFragments {
    uint32_t a[2][2][4];
};

// The cells of rows g, g + 8, g + 16, g + 24 (g = lane / 4) of a position
// block; load(row) gives a row's record.
template <typename Load>
__device__ __forceinline__ void load_cells(CellFragments& f, Load&& load)
{
    const int lane = threadIdx.x & 31, g = lane >> 2, sh = 2 * (lane & 3);
    ulonglong2 po[2][2];
#pragma unroll
    for (int m = 0; m < 2; m++)
#pragma unroll
        for (int r = 0; r < 2; r++) po[m][r] = load(16 * m + 8 * r + g);
#pragma unroll
    for (int m = 0; m < 2; m++)
#pragma unroll
        for (int r = 0; r < 2; r++)
#pragma unroll
            for (int w = 0; w < 2; w++) {
                const uint32_t p = static_cast<uint32_t>(po[m][r].x >> (32 * w)) >> sh;
                const uint32_t o = static_cast<uint32_t>(po[m][r].y >> (32 * w)) >> sh;
#pragma unroll
                for (int s = 0; s < 2; s++)
                    f.a[m][s][2 * w + r] = ((p >> s) & 0x01010101u) | (((o << 1) >> s) & 0x02020202u);
            }
}

__device__ __forceinline__ void mma_u8(uint32_t (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
    asm volatile(
        "mma.sync.aligned.m16n8k32.row.col.s32.u8.u8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
        "{%0, %1, %2, %3};"
        : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// The digits of a tile's lists 2t and 2t + 1 for the lane's four rows:
// v[m][2 r + j] is list 2t + j of row 16 m + 8 r + g.
__device__ __forceinline__ void tile_digits(const uint32_t* __restrict__ tile, bool high, const CellFragments& f,
                                            uint32_t (&v)[2][4])
{
    const uint4* b = reinterpret_cast<const uint4*>(tile) + (threadIdx.x & 31);
    const uint4 lo = b[0];
#pragma unroll
    for (int m = 0; m < 2; m++) {
#pragma unroll
        for (int i = 0; i < 4; i++) v[m][i] = 0;
        mma_u8(v[m], f.a[m][0], lo.x, lo.y);
        mma_u8(v[m], f.a[m][1], lo.z, lo.w);
    }
    if (high) {
        const uint4 hi = b[32];
#pragma unroll
        for (int m = 0; m < 2; m++) {
            uint32_t h[4] = {};
            mma_u8(h, f.a[m][0], hi.x, hi.y);
            mma_u8(h, f.a[m][1], hi.z, hi.w);
#pragma unroll
            for (int i = 0; i < 4; i++) v[m][i] += h[i] << 8;
        }
    }
}

// Column of an unordered pair of half-board digits.
__device__ __forceinline__ uint32_t pair_index(uint32_t a, uint32_t b, uint32_t half_size)
{
    const uint32_t lo = min(a, b), hi = max(a, b);
    return lo * half_size + hi - (lo * (lo + 1) / 2);
}

// The columns (without the pattern's offset) of a unit's slots for the
// lane's rows.  two(m, r, c0, c1): slots 2t and 2t + 1 of row 16 m + 8 r + g
// (kDirect, kTable; slots past the unit's are 0); one(m, r, c): slot t
// (kPair, kDiagPair; t below the unit's slots).
template <typename Two, typename One>
__device__ __forceinline__ void unit_columns(const IndexUnit& u, const uint32_t* __restrict__ s_tiles,
                                             const uint32_t* __restrict__ tables, const CellFragments& f, Two&& two,
                                             One&& one)
{
    const int t = threadIdx.x & 3;
    const uint32_t* tile = s_tiles + u.tile0 * kTileWords;
    uint32_t v[2][4];
    tile_digits(tile, u.high[0] != 0, f, v);
    if (u.kind == kDirect) {
#pragma unroll
        for (int m = 0; m < 2; m++)
#pragma unroll
            for (int r = 0; r < 2; r++) two(m, r, v[m][2 * r], v[m][2 * r + 1]);
    } else if (u.kind == kTable) {
#pragma unroll
        for (int m = 0; m < 2; m++)
#pragma unroll
            for (int r = 0; r < 2; r++) {
                const uint32_t c0 = 2 * t < u.slots ? __ldg(tables + u.table_offset + v[m][2 * r]) : 0u;
                const uint32_t c1 = 2 * t + 1 < u.slots ? __ldg(tables + u.table_offset + v[m][2 * r + 1]) : 0u;
                two(m, r, c0, c1);
            }
    } else {
        uint32_t c[2][2];
#pragma unroll
        for (int m = 0; m < 2; m++)
#pragma unroll
            for (int r = 0; r < 2; r++) c[m][r] = pair_index(v[m][2 * r], v[m][2 * r + 1], u.half_size);
        if (u.kind == kDiagPair) {
            tile_digits(tile + kTileWords, u.high[1] != 0, f, v);
#pragma unroll
            for (int m = 0; m < 2; m++)
#pragma unroll
                for (int r = 0; r < 2; r++) c[m][r] = c[m][r] * u.diag_size + v[m][2 * r];
        }
        if (t < u.slots) {
#pragma unroll
            for (int m = 0; m < 2; m++)
#pragma unroll
                for (int r = 0; r < 2; r++) one(m, r, c[m][r]);
        }
    }
}

// Copies a chunk's tiles into shared memory (all threads of the CTA; ends
// with a barrier).
__device__ __forceinline__ void stage_tiles(const uint32_t* __restrict__ tiles, int t0, int t1,
                                            uint32_t* __restrict__ s_tiles)
{
    const uint4* src = reinterpret_cast<const uint4*>(tiles + static_cast<int64_t>(t0) * kTileWords);
    uint4* dst = reinterpret_cast<uint4*>(s_tiles);
    for (int i = threadIdx.x; i < (t1 - t0) * (kTileWords / 4); i += blockDim.x) dst[i] = __ldg(src + i);
    __syncthreads();
}

}  // namespace cas
