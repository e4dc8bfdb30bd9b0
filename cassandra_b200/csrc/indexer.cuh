// Device evaluation of the indexer recipes built by patterns.cpp: the
// ternary digits of a square list and the per-kind combination of
// Pattern/Indexer.cpp:17-317.
#pragma once
#include <cstdint>

#include "patterns.h"

namespace cas {

__device__ __forceinline__ uint32_t digits(const uint8_t* sq, int n, uint32_t plo, uint32_t phi, uint32_t olo,
                                           uint32_t ohi)
{
    uint32_t idx = 0;
    for (int i = n - 1; i >= 0; i--) {
        const int t = sq[i];
        const uint32_t pw = t < 32 ? plo : phi, ow = t < 32 ? olo : ohi;
        const int sh = t & 31;
        idx = idx * 3 + ((pw >> sh) & 1u) + (((ow >> sh) & 1u) << 1);
    }
    return idx;
}

// The digits of a square list read from a row's digit board in shared
// memory: board[t * STRIDE] = cell(pos, t) for the 64 squares, one byte each.
template <int STRIDE>
__device__ __forceinline__ uint32_t board_digits(const uint8_t* sq, int n, const uint8_t* board)
{
    uint32_t idx = 0;
    for (int i = n - 1; i >= 0; i--) idx = idx * 3 + board[sq[i] * STRIDE];
    return idx;
}

// The per-kind combination of an instance's square lists; dig(list, n)
// gives the digits of one list.
template <typename Digits>
__device__ __forceinline__ uint32_t combine_slot(const Instance& in, const uint32_t* __restrict__ tables, Digits&& dig)
{
    uint32_t r;
    if (in.kind == kDirect) {
        r = dig(in.sq[0], in.n0);
    } else if (in.kind == kTable) {
        r = __ldg(tables + in.table_offset + dig(in.sq[0], in.n0));
    } else {
        uint32_t a = dig(in.sq[0], in.n0);
        uint32_t b = dig(in.sq[1], in.n1);
        const uint32_t lo = min(a, b), hi = max(a, b);
        r = lo * in.half_size + hi - (lo * (lo + 1) / 2);
        if (in.kind == kDiagPair) r = r * in.diag_size + dig(in.sq[2], in.n2);
    }
    return in.offset + r;
}

__device__ __forceinline__ uint32_t eval_slot(const Instance& in, const uint32_t* __restrict__ tables, uint32_t plo,
                                              uint32_t phi, uint32_t olo, uint32_t ohi)
{
    return combine_slot(in, tables,
                        [&](const uint8_t* sq, int n) { return digits(sq, n, plo, phi, olo, ohi); });
}

// eval_slot from the row's digit board.
template <int STRIDE>
__device__ __forceinline__ uint32_t eval_slot_board_all(const Instance& in, const uint32_t* __restrict__ tables,
                                                        const uint8_t* board)
{
    return combine_slot(in, tables, [&](const uint8_t* sq, int n) { return board_digits<STRIDE>(sq, n, board); });
}

}  // namespace cas
