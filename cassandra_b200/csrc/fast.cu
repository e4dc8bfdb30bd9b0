// Blocked pattern layout: build (indexing straight into the layout, a
// per-block column sort for the transposed copy, chunk pointers, diag(A'A))
// and the two products.  See fast.cuh for the layout.
//
// A x   one row a thread, its index words (2 B per entry, 16 B per row and
//       pattern) loaded first, then its entries of x gathered: from a table
//       in shared memory for the patterns whose slices fit one, through L1
//       and L2 for the others.  HBM traffic: 2 B per entry + the output.
// A'y   one CTA per work item (a column chunk of one pattern x a range of row
//       blocks).  Per block the CTA stages y's block slice in shared memory,
//       streams the chunk's column-sorted entries (4 B each, coalesced),
//       gathers y from shared memory and reduces each run of equal columns
//       with a deterministic segmented scan into a shared-memory accumulator
//       of the chunk.  Items write partial column sums that the caller adds
//       in a fixed order: no atomics anywhere, bitwise reproducible.
#include <algorithm>
#include <cstring>
#include <cstdio>
#include <cstdlib>
#include <map>
#include <mutex>
#include <string>
#include <vector>

#include "common.cuh"
#include "fast.cuh"
#include "tile_index.cuh"

namespace cas {

namespace {

constexpr int kSortThreads = 256;  // a sort pass's round is kSortThreads items (at least 256: one thread per digit)
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kSortCtasPerSm = 4;  // groups sorted at once per SM: their barriers and scans overlap
// The A'y accumulator of a work item holds at most kMaxSc column chunks
// (with the y tile, the FP32 kernel's dynamic shared memory: 192 KB).  The
// build-time autotuner picks the schedule (accumulator width, items per SM,
// packing of narrow patterns, persistent CTAs).
constexpr int kMaxSc = 4;
constexpr int64_t kBatchItemBlocks = 4;  // most row blocks of one A'y work item in a batched layout
constexpr int64_t kBatchSmallBlocks = 8;  // batched problems this small get one block per A'y item

unsigned fgrid(int64_t work, int per)
{
    const int64_t want = (work + per - 1) / per;
    return static_cast<unsigned>(std::max<int64_t>(1, std::min<int64_t>(want, static_cast<int64_t>(sm_count()) * 4)));
}

// ---------------------------------------------------------------------------
// Indexing into the blocked layout, by the matrix form (tile_index.cuh): the
// layout's patterns have at most 65536 columns, so no digit list exceeds 11
// squares.  A warp takes 32 rows; a quad of lanes writes a row's slots of a
// pattern, so 8 rows of 8 slots are 128 consecutive bytes of A16.  5M rows of
// the 8-pattern expanded set: 250 us, 2.9 TB/s (883 us by digit boards).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kTileThreads, 3) fast_index_kernel(const uint32_t* __restrict__ tiles,
                                                                     const IndexUnit* __restrict__ units,
                                                                     const int32_t* __restrict__ chunk_unit,
                                                                     const int32_t* __restrict__ chunk_tile,
                                                                     const uint32_t* __restrict__ tables,
                                                                     const ulonglong2* __restrict__ pos,
                                                                     FastGeometry g, uint16_t* __restrict__ a16,
                                                                     int64_t r_begin, int64_t r_end)
{
    extern __shared__ __align__(16) uint32_t s_tiles[];
    const int u0 = chunk_unit[blockIdx.y], u1 = chunk_unit[blockIdx.y + 1];
    stage_tiles(tiles, chunk_tile[blockIdx.y], chunk_tile[blockIdx.y + 1], s_tiles);
    const int lane = threadIdx.x & 31, grp = lane >> 2, t = lane & 3;
    const int64_t step = static_cast<int64_t>(gridDim.x) * (kTileThreads / 32) * kTileRows;
    for (int64_t base = r_begin + (static_cast<int64_t>(blockIdx.x) * (kTileThreads / 32) + (threadIdx.x >> 5)) * kTileRows;
         base < r_end; base += step) {
        const int64_t end = min(base + kTileRows, r_end);
        // one pass unless the rows lie in several blocks (at block and
        // problem bounds only); everything but the lane's place is uniform
        for (int64_t r0 = base, r1; r0 < end; r0 = r1) {
            int64_t b, rl;
            g.locate_row(r0, b, rl);
            r1 = min(end, r0 + g.block_rows(b) - rl);
            const int cnt = static_cast<int>(r1 - r0) - grp;  // row 16 m + 8 r + grp is one of these if 16 m + 8 r < cnt
            CellFragments f;
            load_cells(f, [&](int r) { return r0 + r < r1 ? __ldg(pos + r0 + r) : make_ulonglong2(0, 0); });
            uint16_t* blk0 = a16 + b * static_cast<int64_t>(kBlockRows) * g.k;
            const int pad = static_cast<int>(g.padded_rows(b));
            for (int i = u0; i < u1; i++) {
                const IndexUnit u = units[i];
                uint16_t* dst = blk0 + pad * static_cast<int>(u.slot0) + (static_cast<int>(rl) + grp) * u.slots;
                unit_columns(
                    u, s_tiles, tables, f,
                    [&](int m, int r, uint32_t c0, uint32_t c1) {
                        const int row = 16 * m + 8 * r;
                        if (row >= cnt || 2 * t >= u.slots) return;
                        if (u.slots == 1)
                            dst[row] = static_cast<uint16_t>(c0);
                        else
                            *reinterpret_cast<uint32_t*>(dst + row * u.slots + 2 * t) = c0 | (c1 << 16);
                    },
                    [&](int m, int r, uint32_t c) {
                        const int row = 16 * m + 8 * r;
                        if (row < cnt) dst[row * u.slots + t] = static_cast<uint16_t>(c);
                    });
            }
        }
    }
}

// ---------------------------------------------------------------------------
// Per-(block, pattern) stable sort of entries by local column: two 8-bit LSD
// passes inside one CTA, the first into a per-CTA scratch slice.  Items are
// (column << 16) | (row-in-block << 2) | end, end (bit 0) set on the last
// entry of each column; the input order is row-major (row, slot), so equal
// columns keep ascending rows.
//
// A pass moves its items in tiles of kSortTile: each warp ranks its 512
// items by digit (peers from ballots, in item order, counts per digit in shared
// memory), one scan per tile turns the warps' counts into offsets, the tile
// is scattered digit by digit into a shared buffer and written out from
// there, so that consecutive threads write the consecutive output positions
// of a digit's run.  The final pass writes G32's round order and the end
// flags: an entry ends its run when the next entry of its digit in the tile
// has another column; the last entry of a digit in a tile waits (position
// and column kept per digit) for the digit's first entry in a later tile,
// or for the pass's end (the next entry then has another digit).
// ---------------------------------------------------------------------------
constexpr int kSortPerThread = 16;                           // items per thread and tile
constexpr int kSortTile = kSortThreads * kSortPerThread;     // items per tile
constexpr int kSortWarpItems = 32 * kSortPerThread;          // items a warp ranks per tile
constexpr uint32_t kNoPend = 0xFFFFFFFFu;
constexpr int kSortPrefetchPieces = kSortTile * 4 / 4096;  // 4 KB pieces of a tile of 4-byte items

struct SortSmem {
    uint32_t hist[256];   // digit counts of the first pass (counted from the input)
    uint32_t hist2[256];  // digit counts of the final pass (counted by the first pass's write-out)
    uint32_t dst[256];    // output position of the tile buffer's slot 0 for the digit (mod 2^32)
    uint32_t wtot[kSortWarps];
    uint16_t wcnt[kSortWarps][256];  // a warp's items of a digit, then their first slot in the tile buffer
    uint32_t buf[kSortTile];
};
static_assert(kSortThreads == 256, "one thread per digit");

// Exclusive scan over the CTA's threads of v.  Ends with a barrier behind the
// reads of wtot's previous use only: the caller has one before the next.
__device__ __forceinline__ uint32_t sort_scan(uint32_t v, uint32_t* wtot)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t u = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += u;
    }
    if (lane == 31) wtot[warp] = incl;
    __syncthreads();
    uint32_t pre = 0;
#pragma unroll
    for (int w = 0; w < kSortWarps; w++) pre += w < warp ? wtot[w] : 0;
    return pre + incl - v;
}

// The lanes of the warp whose 8-bit digit equals this lane's, from eight
// ballots.
__device__ __forceinline__ unsigned digit_peers(uint32_t d)
{
    unsigned peers = 0xffffffffu;
#pragma unroll
    for (int b = 0; b < 8; b++) {
        const bool bit = (d >> b) & 1u;
        const unsigned m = __ballot_sync(0xffffffffu, bit);
        peers &= bit ? m : ~m;
    }
    return peers;
}

// What a thread keeps of its digit (thread t: digit t) over a pass's tiles.
struct SortDigit {
    uint32_t next;      // output position of the digit's next entry
    uint32_t pend_pos;  // final pass: the digit's last entry so far (kNoPend: none)
    uint32_t pend_col;  //   and its column
};

// One tile of a pass: count items (all kSortTile of them if WHOLE) from item
// t0 of the group on.
template <bool FROM_A16, bool WHOLE>
__device__ __forceinline__ void sort_tile(const uint16_t* __restrict__ a16_in, const uint32_t* __restrict__ in, int t0,
                                          int count, int slots_log2, uint32_t* __restrict__ out, SortDigit& dig,
                                          SortSmem& sm)
{
    constexpr bool FINAL = !FROM_A16;
    constexpr int kShift = FROM_A16 ? 16 : 24;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const unsigned lt_mask = (1u << lane) - 1;
    uint16_t* mine = sm.wcnt[warp];
    {
        uint32_t* z = reinterpret_cast<uint32_t*>(mine);
#pragma unroll
        for (int i = 0; i < 128; i += 32) z[i + lane] = 0;
    }
    __syncwarp();
    // 1. rank: the warp's items warp * 512 + 32 k + lane of the tile, in item
    // order; items past the end take the last digit and rank behind it
    const int i0 = warp * kSortWarpItems + lane;
    uint32_t item[kSortPerThread];
    uint16_t rk[kSortPerThread];  // rank among the warp's items of the same digit
#pragma unroll
    for (int k = 0; k < kSortPerThread; k++) {  // all loads first: one memory latency per tile
        const int i = i0 + 32 * k;
        item[k] = 0xFFFFFFFFu;
        if (WHOLE || i < count)
            item[k] = FROM_A16 ? static_cast<uint32_t>(a16_in[t0 + i]) << 16 |
                                     static_cast<uint32_t>((t0 + i) >> slots_log2) << 2
                               : in[t0 + i];
    }
#pragma unroll
    for (int k = 0; k < kSortPerThread; k++) {
        const uint32_t d = (item[k] >> kShift) & 255u;
        const unsigned peers = digit_peers(d);
        const uint32_t before = __popc(peers & lt_mask), c = mine[d];
        __syncwarp();
        if (before == 0) mine[d] = static_cast<uint16_t>(c + __popc(peers));
        __syncwarp();
        rk[k] = static_cast<uint16_t>(c + before);
    }
    __syncthreads();
    // 2. digit t: the tile's entries, their first slot, each warp's first
    uint32_t total = 0, cnt[kSortWarps];
#pragma unroll
    for (int w = 0; w < kSortWarps; w++) {
        cnt[w] = total;
        total += sm.wcnt[w][t];
    }
    const uint32_t start = sort_scan(total, sm.wtot);
#pragma unroll
    for (int w = 0; w < kSortWarps; w++) sm.wcnt[w][t] = static_cast<uint16_t>(start + cnt[w]);
    sm.dst[t] = dig.next - start;
    if (!WHOLE && t == 255) total -= kSortTile - count;
    __syncthreads();
    // 3. the tile into the buffer, digit by digit
#pragma unroll
    for (int k = 0; k < kSortPerThread; k++) sm.buf[mine[(item[k] >> kShift) & 255u] + rk[k]] = item[k];
    __syncthreads();
    // 4. out: consecutive buffer slots of a digit are consecutive positions
#pragma unroll 4
    for (int j = t; j < (WHOLE ? kSortTile : count); j += kSortThreads) {
        uint32_t it = sm.buf[j];
        const uint32_t pos = sm.dst[(it >> kShift) & 255u] + static_cast<uint32_t>(j);
        if (FINAL) {
            // an entry whose next one in the tile is of its digit ends its run
            // if the columns differ; the digit's last one in the tile waits
            const uint32_t nx = j + 1 < count ? sm.buf[j + 1] : ~it;
            if ((nx >> 24) == (it >> 24) && (nx >> 16) != (it >> 16)) it |= 1u;
            out[round_phys(pos)] = it;
        } else {
            out[pos] = it;
            atomicAdd(&sm.hist2[it >> 24], 1u);
        }
    }
    if (FINAL && total > 0) {
        // the digit's entry waiting from an earlier tile ends its run unless
        // this tile's first entry of the digit continues its column
        const uint32_t first = sm.buf[start];
        if (dig.pend_pos != kNoPend && (first >> 16) != dig.pend_col) out[round_phys(dig.pend_pos)] |= 1u;
        dig.pend_pos = dig.next + total - 1;
        dig.pend_col = sm.buf[start + total - 1] >> 16;
    }
    dig.next += total;
    __syncthreads();
}

// One stable 8-bit counting-sort pass of a group's n items.  FROM_A16: the
// first pass, by the low byte of the column, items made from the A16 segment
// (local column << 16 | row << 2), written to out in sorted order while the
// final pass's digit counts are gathered.  !FROM_A16: the final pass, by the
// high byte, items read from `in`, written in G32's round order (round_phys of
// the sorted position; out starts on a round boundary) with their end flags.
//
// Bound by instructions, the eight ballots of a ranked item first: whole tiles
// run without bounds, a digit's counts and places stay with its thread, and
// every lane reads its digit's count itself.  320M entries (5M rows of eight
// expanded patterns): 4,230 us with bounds, divisions and a leader that hands
// the count out, 3,240 us so.
template <bool FROM_A16>
__device__ __forceinline__ void sort_pass(const uint16_t* __restrict__ a16_in, const uint32_t* __restrict__ in, int n,
                                          int slots, uint32_t* __restrict__ out, SortSmem& sm)
{
    constexpr bool FINAL = !FROM_A16;
    const int t = threadIdx.x;
    if (FROM_A16) {
        // the digits (low column bytes) of the group, 8 columns per 16-byte
        // load (segments start on 1024-entry rounds), the last n % 8 one by
        // one
        sm.hist[t] = 0;
        __syncthreads();
        const uint4* v = reinterpret_cast<const uint4*>(a16_in);
        for (int e = (n & ~7) + t; e < n; e += kSortThreads) atomicAdd(&sm.hist[a16_in[e] & 255u], 1u);
        for (int i = t; i < n / 8; i += kSortThreads) {
            const uint4 u = __ldcs(v + i);
            const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
            for (int q = 0; q < 8; q++) atomicAdd(&sm.hist[(w[q >> 1] >> (16 * (q & 1))) & 255u], 1u);
        }
        __syncthreads();
    }
    SortDigit dig{sort_scan(FROM_A16 ? sm.hist[t] : sm.hist2[t], sm.wtot), kNoPend, 0};
    if (FROM_A16) sm.hist2[t] = 0;
    __syncthreads();
    const int slots_log2 = 31 - __clz(slots);  // 1, 2, 4 or 8
    for (int t0 = 0; t0 < n; t0 += kSortTile) {
        // the next tile's input into L2 while this one is ranked, in 4 KB
        // pieces rounded up to 16 bytes (inside the group's room: whole
        // rounds of A16, whole tiles of the scratch slice)
        if (t < kSortPrefetchPieces) {
            const int nt = t0 + kSortTile;
            const int64_t bytes = static_cast<int64_t>(min(kSortTile, n - nt)) * (FROM_A16 ? 2 : 4);
            const int64_t lo = static_cast<int64_t>(t) * 4096;
            if (nt < n && lo < bytes) {
                const char* src = FROM_A16 ? reinterpret_cast<const char*>(a16_in + nt)
                                           : reinterpret_cast<const char*>(in + nt);
                const int64_t piece = bytes - lo < 4096 ? bytes - lo : 4096;
                const unsigned len = static_cast<unsigned>((piece + 15) & ~int64_t(15));
                asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src + lo), "r"(len) : "memory");
            }
        }
        if (n - t0 >= kSortTile)
            sort_tile<FROM_A16, true>(a16_in, in, t0, kSortTile, slots_log2, out, dig, sm);
        else
            sort_tile<FROM_A16, false>(a16_in, in, t0, n - t0, slots_log2, out, dig, sm);
    }
    // the last entry of every digit ends its run (the next has another digit)
    if (FINAL && dig.pend_pos != kNoPend) out[round_phys(dig.pend_pos)] |= 1u;
    __syncthreads();
}

__global__ void __launch_bounds__(kSortThreads, kSortCtasPerSm) fast_sort_kernel(FastGeometry g,
                                                                                const uint16_t* __restrict__ a16,
                                                                   uint32_t* __restrict__ g32,
                                                                   uint32_t* __restrict__ scratch)
{
    __shared__ SortSmem sm;
    uint32_t* mine = scratch + static_cast<int64_t>(blockIdx.x) * kBlockRows * 8;
    const int64_t groups = g.nblocks * g.npat;
    for (int64_t grp = blockIdx.x; grp < groups; grp += gridDim.x) {
        const int64_t b = grp / g.npat;
        const int p = static_cast<int>(grp - b * g.npat);
        const int n = static_cast<int>(g.seg_len(b, p));
        const int64_t seg = g.seg(b, p);
        sort_pass<true>(a16 + seg, nullptr, n, g.slots[p], mine, sm);
        sort_pass<false>(nullptr, mine, n, g.slots[p], g32 + seg, sm);
    }
}

// First entry of every (block, column sub-chunk) in G32: lower bound of the
// sub-chunk's first column in the sorted group (sub-chunks past the end of
// a pattern's columns get the group's end).
__global__ void fast_sub_kernel(FastGeometry g, const uint32_t* __restrict__ g32, uint32_t* __restrict__ sub_start)
{
    const int nsub = g.nchunks * kSubPerChunk;
    const int64_t total = g.nblocks * nsub;
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const int64_t b = i / nsub;
        const int j = static_cast<int>(i - b * nsub);
        const int ch = j / kSubPerChunk;
        int p = 0;
        while (p + 1 < g.npat && g.chunk0[p + 1] <= ch) p++;
        const uint32_t c0 = static_cast<uint32_t>(j - g.chunk0[p] * kSubPerChunk) * kSubCols;
        const int64_t seg = g.seg(b, p);
        int64_t lo = 0, hi = g.seg_len(b, p);
        while (lo < hi) {
            const int64_t mid = (lo + hi) >> 1;
            if ((g32[seg + round_phys(static_cast<uint32_t>(mid))] >> 16) < c0)
                lo = mid + 1;
            else
                hi = mid;
        }
        sub_start[i] = static_cast<uint32_t>(seg + lo);
    }
}

// Entries of every (block, chunk): the distance between the chunk's first
// sub-chunk start and the next chunk's (or the group's end).
__global__ void fast_chunk_entries_kernel(FastGeometry g, const uint32_t* __restrict__ sub_start,
                                          uint32_t* __restrict__ out)
{
    const int64_t total = g.nblocks * g.nchunks;
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const int64_t b = i / g.nchunks;
        const int ch = static_cast<int>(i - b * g.nchunks);
        int p = 0;
        while (p + 1 < g.npat && g.chunk0[p + 1] <= ch) p++;
        const int c_end = p + 1 < g.npat ? g.chunk0[p + 1] : g.nchunks;
        const int64_t lo = sub_start[i * kSubPerChunk];
        const int64_t hi = ch + 1 < c_end ? static_cast<int64_t>(sub_start[(i + 1) * kSubPerChunk])
                                          : g.seg(b, p) + g.seg_len(b, p);
        out[i] = static_cast<uint32_t>(hi - lo);
    }
}

// diag(A'A)_c = sum over rows of m^2: inside a sorted group equal
// (column, row) pairs are adjacent, so the j-th copy contributes 2j+1.
__global__ void fast_diag_kernel(FastGeometry g, const uint32_t* __restrict__ g32, uint64_t* __restrict__ diag)
{
    const int lane = threadIdx.x & 31;
    const int64_t groups = g.nblocks * g.npat;
    for (int64_t grp = blockIdx.x; grp < groups; grp += gridDim.x) {
        const int64_t b = grp / g.npat;
        const int p = static_cast<int>(grp - b * g.npat);
        const int64_t seg = g.seg(b, p), n = g.seg_len(b, p);
        for (int64_t e0 = 0; e0 < n; e0 += blockDim.x) {
            const int64_t e = e0 + threadIdx.x;
            uint32_t col = 0xFFFFFFFFu, contrib = 0;
            if (e < n) {
                const uint32_t v = g32[seg + round_phys(static_cast<uint32_t>(e))];
                int64_t j = 0;
                while (e - j - 1 >= 0 &&
                       (g32[seg + round_phys(static_cast<uint32_t>(e - j - 1))] >> 2) == (v >> 2))
                    j++;  // same (column, row)
                col = v >> 16;
                contrib = static_cast<uint32_t>(2 * j + 1);
            }
            const unsigned peers = __match_any_sync(0xffffffffu, col);
            const uint32_t sum = __reduce_add_sync(peers, contrib);
            if (e < n && lane == __ffs(peers) - 1)
                atomicAdd(reinterpret_cast<unsigned long long*>(diag + g.col_base(b) + g.off[p] + col), sum);
        }
    }
}

// The column counts A'1 from the FP32 A'y partials of a vector of ones:
// every partial (and every sum the A'y kernel forms on the way) counts
// entries of one column inside one item, so it is an exact float integer
// while the item holds fewer than 2^24 entries; the column sums add the
// partials in FP64.
__global__ void fast_count_kernel(FastCols fc, const float* __restrict__ partial, uint64_t* __restrict__ diag)
{
    for (int64_t c = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; c < fc.g.cols;
         c += static_cast<int64_t>(gridDim.x) * blockDim.x)
        diag[c] = static_cast<uint64_t>(fast_col_sum<float>(fc, partial, c));
}

constexpr int kRepeatRounds = 16;  // G32 rounds of one warp's stretch

// One G32 round (4 KB, on a 16-byte boundary) into L2.
__device__ __forceinline__ void prefetch_round(const uint32_t* round)
{
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(round),
                 "r"(static_cast<unsigned>(kRound * sizeof(uint32_t)))
                 : "memory");
}

// The repeats' share of diag(A'A): a row holding a column m times adds
// m^2 = m + 2 (1 + 2 + ... + (m - 1)), and the count A'1 holds the m.
// Equal (column, row) pairs are adjacent in a sorted group and number at
// most the pattern's slots (<= 8).  A warp takes a stretch of kRepeatRounds
// rounds of one group; per round each lane holds its 32 consecutive sorted
// entries (the lane run of the round: eight 16-byte words 512 bytes apart)
// and counts copies along them, starting from the entry before its run and
// the number of equal entries that end there (the previous lane's, carried
// from lane 31 across rounds, and walked back in G32 at the stretch's
// start).  A lane adds a column's repeats once per run of that column.
__global__ void __launch_bounds__(256, 4) fast_repeat_kernel(FastGeometry g, const uint32_t* __restrict__ g32,
                                                             uint64_t* __restrict__ diag, int stretches)
{
    const int lane = threadIdx.x & 31;
    const int64_t nwarps = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
    const int64_t units = g.nblocks * g.npat * stretches;
    for (int64_t u = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; u < units; u += nwarps) {
        const int64_t grp = u / stretches;
        const int st = static_cast<int>(u - grp * stretches);
        const int64_t b = grp / g.npat;
        const int p = static_cast<int>(grp - b * g.npat);
        const int64_t seg = g.seg(b, p), n = g.seg_len(b, p);
        const int64_t r_begin = static_cast<int64_t>(st) * kRepeatRounds * kRound;
        if (r_begin >= n) continue;  // uniform over the warp
        const int64_t r_end = n < r_begin + kRepeatRounds * kRound ? n : r_begin + kRepeatRounds * kRound;
        uint64_t* dcol = diag + g.col_base(b) + g.off[p];
        if (lane == 0 && r_begin + kRound < r_end) prefetch_round(g32 + seg + r_begin + kRound);
        // the entry before the stretch and the equal entries ending there
        uint32_t carry_last = 0;
        int carry_tail = 0;  // 0: none before
        if (r_begin > 0) {
            carry_last = g32[seg + round_phys(static_cast<uint32_t>(r_begin - 1))];
            carry_tail = 1;
            while (carry_tail < r_begin &&
                   (g32[seg + round_phys(static_cast<uint32_t>(r_begin - 1 - carry_tail))] >> 2) == (carry_last >> 2))
                carry_tail++;
        }
        for (int64_t r0 = r_begin; r0 < r_end; r0 += kRound) {
            // the round after next into L2 (whole rounds: the segment's room
            // ends on a round)
            if (lane == 0 && r0 + 2 * kRound < r_end) prefetch_round(g32 + seg + r0 + 2 * kRound);
            const int64_t lb = r0 + kLaneRun * lane;  // the lane's first sorted position
            const int64_t rem = r_end - lb;
            const int cnt = rem <= 0 ? 0 : (rem >= kLaneRun ? kLaneRun : static_cast<int>(rem));
            uint32_t e[kLaneRun];
            const uint4* src = reinterpret_cast<const uint4*>(g32 + seg + r0) + lane;
#pragma unroll
            for (int q = 0; q < kLaneRun / 4; q++) {
                uint4 w = make_uint4(0, 0, 0, 0);
                if (4 * q < cnt) w = src[32 * q];
                e[4 * q] = w.x, e[4 * q + 1] = w.y, e[4 * q + 2] = w.z, e[4 * q + 3] = w.w;
            }
            // the run's last entry and the equal entries ending it (a full
            // run holds more than 8 entries, so this needs nothing before it)
            int tail = 0;
            uint32_t last = 0;
#pragma unroll
            for (int k = 0; k < kLaneRun; k++) {
                if (k < cnt) {
                    tail = (k > 0 && (e[k] >> 2) == (e[k - 1] >> 2)) ? tail + 1 : 1;
                    last = e[k];
                }
            }
            uint32_t before = __shfl_up_sync(0xffffffffu, last, 1);
            int m = __shfl_up_sync(0xffffffffu, tail, 1);
            if (lane == 0) before = carry_last, m = carry_tail;
            carry_last = __shfl_sync(0xffffffffu, last, 31);
            carry_tail = __shfl_sync(0xffffffffu, tail, 31);
            uint64_t acc = 0;
            uint32_t acc_col = cnt > 0 ? e[0] >> 16 : 0;
#pragma unroll
            for (int k = 0; k < kLaneRun; k++) {
                if (k < cnt) {
                    const uint32_t col = e[k] >> 16;
                    if (col != acc_col) {
                        if (acc) atomicAdd(reinterpret_cast<unsigned long long*>(dcol + acc_col), acc);
                        acc = 0;
                        acc_col = col;
                    }
                    if (m > 0 && (e[k] >> 2) == (before >> 2)) {  // copy number m (from 0) of (column, row)
                        acc += 2 * static_cast<uint64_t>(m);
                        m++;
                    } else {
                        m = 1;
                    }
                    before = e[k];
                }
            }
            if (acc) atomicAdd(reinterpret_cast<unsigned long long*>(dcol + acc_col), acc);
        }
    }
}

// ---------------------------------------------------------------------------
// A x on the blocked layout.
// ---------------------------------------------------------------------------
template <typename T>
struct AccOf {
    using type = float;
};
template <>
struct AccOf<double> {
    using type = double;
};

// Asks L2 to fetch [p, p + bytes) (the 16-byte words wholly inside it), in
// 4 KB bulk prefetches spread over the CTA's threads.  A hint: the data is
// read later with ordinary loads.
__device__ __forceinline__ void prefetch_l2(const void* p, int64_t bytes)
{
    if (bytes <= 0) return;
    const uintptr_t a = (reinterpret_cast<uintptr_t>(p) + 15) & ~uintptr_t(15);
    const uintptr_t e = (reinterpret_cast<uintptr_t>(p) + static_cast<uintptr_t>(bytes)) & ~uintptr_t(15);
    for (uintptr_t c = a + static_cast<uintptr_t>(threadIdx.x) * 4096; c < e;
         c += static_cast<uintptr_t>(blockDim.x) * 4096) {
        const unsigned n = static_cast<unsigned>(min(static_cast<uint64_t>(e - c), static_cast<uint64_t>(4096)));
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(c), "r"(n) : "memory");
    }
}

// Prefix sums over an active list of a per-problem count (cnt(q)) into
// pref[0..n] in shared memory, by warp 0; every thread returns the total.
template <typename F>
__device__ __forceinline__ int active_prefix(const FastActive* __restrict__ act, int* pref, F cnt)
{
    const int n = act->n;
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        int carry = 0;
        for (int base = 0; base < n; base += 32) {
            const int t = base + lane;
            int v = t < n ? cnt(act->list[t]) : 0;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int u = __shfl_up_sync(0xffffffffu, v, d);
                if (lane >= d) v += u;
            }
            if (t < n) pref[t + 1] = carry + v;
            carry += __shfl_sync(0xffffffffu, v, 31);
        }
        if (lane == 0) pref[0] = 0;
    }
    __syncthreads();
    return pref[n];
}

// Slot k of the active list with pref[k] <= i < pref[k + 1] (0 <= i < pref[n]).
__device__ __forceinline__ int active_slot(const int* pref, int n, int i)
{
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (pref[mid] <= i)
            lo = mid;
        else
            hi = mid - 1;
    }
    return lo;
}

// The index words of one row of a pattern (slots 16-bit columns).  STREAM:
// past L1, whose lines stay with x.
template <bool STREAM>
__device__ __forceinline__ uint4 load_words(const uint16_t* __restrict__ src, int slots)
{
    uint4 w = make_uint4(0, 0, 0, 0);
    if (slots == 8) {
        if (STREAM)
            asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
                         : "=r"(w.x), "=r"(w.y), "=r"(w.z), "=r"(w.w)
                         : "l"(src));
        else
            w = *reinterpret_cast<const uint4*>(src);
    } else if (slots == 4) {
        if (STREAM) {
            asm volatile("ld.global.nc.L1::no_allocate.v2.u32 {%0, %1}, [%2];" : "=r"(w.x), "=r"(w.y) : "l"(src));
        } else {
            const uint2 u = *reinterpret_cast<const uint2*>(src);
            w.x = u.x, w.y = u.y;
        }
    } else if (slots == 2) {
        w.x = *reinterpret_cast<const uint32_t*>(src);
    } else {
        w.x = *src;
    }
    return w;
}

// The entries of a row's words gathered from src (x or a table of it) into
// acc, in slot order.
template <typename T, bool ALL8, bool SHARED>
__device__ __forceinline__ void gather_words(const uint4& u, int slots, const T* __restrict__ src,
                                             typename AccOf<T>::type& acc)
{
    using Acc = typename AccOf<T>::type;
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int s = 0; s < 8; s++) {
        if (ALL8 || s < slots) {
            const uint32_t c = (s & 1) ? w[s >> 1] >> 16 : w[s >> 1] & 0xFFFFu;
            acc += static_cast<Acc>(SHARED ? src[c] : __ldg(src + c));
        }
    }
}

constexpr int kRowPatterns = 8;  // most patterns whose index words a thread holds at once

// Row r of block blk times x: the index words of AHEAD patterns first, then
// their gathers, so that they are in flight together.  TABLE: the patterns of
// tab have their slice of x in table.
template <typename T, bool ALL8, bool TABLE, int AHEAD = kRowPatterns>
__device__ __forceinline__ typename AccOf<T>::type row_sum(const FastGeometry& g, const uint16_t* __restrict__ a16,
                                                           int64_t blk, int r, const T* __restrict__ x,
                                                           const FastTable& tab, const T* __restrict__ table)
{
    const uint16_t* bp = a16 + blk * static_cast<int64_t>(kBlockRows) * g.k;
    const int pad = static_cast<int>(g.padded_rows(blk));
    typename AccOf<T>::type acc = 0;
    for (int p0 = 0; p0 < g.npat; p0 += AHEAD) {
        uint4 w[AHEAD];
#pragma unroll
        for (int i = 0; i < AHEAD; i++) {
            const int p = p0 + i;
            if (p < g.npat) {
                const int ns = ALL8 ? 8 : g.slots[p];
                w[i] = load_words<TABLE>(bp + pad * g.slot0[p] + r * ns, ns);
            }
        }
#pragma unroll
        for (int i = 0; i < AHEAD; i++) {
            const int p = p0 + i;
            if (p < g.npat) {
                const int ns = ALL8 ? 8 : g.slots[p];
                if (TABLE && tab.base[p] >= 0)
                    gather_words<T, ALL8, true>(w[i], ns, table + tab.base[p], acc);
                else
                    gather_words<T, ALL8, false>(w[i], ns, x + g.off[p], acc);
            }
        }
    }
    return acc;
}

// The value of a row from its product v (MODE as fast_spmv's mode), stored;
// returns the stored value.
template <typename Y, int MODE>
__device__ __forceinline__ double store_row(double v, Y* __restrict__ y, const double* __restrict__ b, double c,
                                            int64_t row)
{
    if (MODE == 1) v = static_cast<double>(y[row]) * -c + v;
    if (MODE == 2) v = (b ? b[row] : 0.0) - v;
    const Y yv = static_cast<Y>(v);
    y[row] = yv;
    return static_cast<double>(yv);
}

// A x with the slices of x that fit kept in shared memory (FastTable: the
// patterns with the most entries a row per column first) and the others
// gathered through L1 and L2.  One CTA per SM runs over a contiguous share
// of the rows, one row a thread; the table is staged once per CTA (once per
// problem of a batch), so nothing waits on a barrier between rows.
//
// Bound by the gathers: 32 random words of shared memory take 3.5 wavefronts,
// the same through L1 about 8 tag wavefronts at a 79 % hit rate.  The table
// ends at 140 KB because L1 holds the other patterns' popular columns: on the
// 8-pattern expanded set, 610 blocks, FP32, tables of 0, 64, 115, 195 and 224
// KB gave 744, 629, 543, 630 and 630 us (FP64 876, 870, 862, 1015, 1590), and
// keeping the index words out of L1 another 3 to 7 % (without a table, where
// L1 is large, 5 % the other way).
//
// The kernel before this one staged every pattern's slice for every block of
// rows (42 us of the 143 us a block took: 665 KB a block and 16 barriers).
// us before and now, FP32 / FP64:
//   8 patterns expanded   200 blocks 262 / 461 -> 192 / 294   610: 625 / 1136 -> 524 / 878
//   8 patterns reference  200 blocks 330 / 420 -> 136 / 166   610: 781 / 1032 -> 371 / 463
// Up to kAxDirectBlocks blocks the rows are done before a table pays (8
// patterns expanded, FP32, us without and with it: 16 blocks 26.8 and 28.9,
// 48 64.1 and 64.0, 74 92.7 and 83).  Of the other sets and FP64 the line lies
// between 49 and 75 blocks where a table is staged at all (table_plan), and the
// two are within 5 % of one another there (a call of eight reference patterns,
// FP32 / FP64, 60 blocks 78 / 87 and 76 / 85, 80 96 / 108 and 87 / 100; five
// expanded ones, FP64, 60 88.7 and 89.3, 80 108.1 and 106.7).
//
// A unit is 1/kAxTableSplit of a block.  part (optional): compensated
// partials of ||y||^2, one per CTA without act, else per unit laid out
// [block][kAxSplitMax] (the rest 0).  With act only the listed problems'
// blocks run, and none when fast_spmv_direct_kernel's launch does them.
template <typename T, typename Y, int MODE, bool ALL8>
__global__ void __launch_bounds__(kAxThreads, 1) fast_spmv_table_kernel(FastGeometry g, FastTable tab,
                                                                         const uint16_t* __restrict__ a16,
                                                                         const T* __restrict__ x, Y* __restrict__ y,
                                                                         const double* __restrict__ b,
                                                                         const double* __restrict__ coef,
                                                                         double* __restrict__ part,
                                                                         const int* __restrict__ done,
                                                                         const int* __restrict__ pdone,
                                                                         const FastActive* __restrict__ act)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* table = reinterpret_cast<T*>(smem_raw);
    __shared__ double red[64];
    __shared__ int pref[kMaxProblems + 1];
    if (done && *(volatile const int*)done) return;
    const double c = MODE == 1 ? *coef : 0.0;
    int64_t nblk = g.nblocks;
    if (act) {
        nblk = active_prefix(act, pref, [&](int q) { return g.pblk0[q + 1] - g.pblk0[q]; });
        if (nblk <= kAxDirectBlocks) return;
    }
    const int64_t units = nblk * kAxTableSplit;
    const int64_t u0 = units * blockIdx.x / gridDim.x, u1 = units * (blockIdx.x + 1) / gridDim.x;
    int staged = -1;  // problem whose x the table holds
    Comp mine;
    for (int64_t u = u0; u < u1; u++) {
        const int sp = static_cast<int>(u % kAxTableSplit);
        int64_t blk = u / kAxTableSplit;
        if (act) {
            const int i = static_cast<int>(blk);
            const int slot = active_slot(pref, act->n, i);
            blk = g.pblk0[act->list[slot]] + (i - pref[slot]);
        }
        const int q = g.prob_of_block(blk);
        double* pu = part && act ? part + 2 * (blk * kAxSplitMax + sp) : nullptr;
        if (pu && sp == 0 && static_cast<int>(threadIdx.x) < 2 * (kAxSplitMax - kAxTableSplit))
            pu[2 * kAxTableSplit + threadIdx.x] = 0;
        if (pdone && pdone[q]) {
            if (pu && threadIdx.x == 0) {
                pu[0] = 0;
                pu[1] = 0;
            }
            continue;
        }
        const T* xq = x + q * g.pcols;
        if (q != staged) {
            __syncthreads();
            for (int p = 0; p < g.npat; p++) {
                if (tab.base[p] < 0) continue;
                T* dst = table + tab.base[p];
                const T* src = xq + g.off[p];
#pragma unroll 8
                for (int i = threadIdx.x; i < g.space[p]; i += kAxThreads) dst[i] = __ldg(src + i);
            }
            __syncthreads();
            staged = q;
        }
        const int rows_b = static_cast<int>(g.block_rows(blk));
        const int r0 = rows_b * sp / kAxTableSplit, nb = rows_b * (sp + 1) / kAxTableSplit - r0;
        if (static_cast<int>(threadIdx.x) < nb) {
            const int r = r0 + threadIdx.x;
            const double v = static_cast<double>(row_sum<T, ALL8, true>(g, a16, blk, r, xq, tab, table));
            const double yv = store_row<Y, MODE>(v, y, b, c, g.block_row0(blk) + r);
            mine.add(yv * yv);
        }
        if (pu) {
            const Comp r = block_sum_comp<kAxThreads>(mine, red);
            if (threadIdx.x == 0) {
                pu[0] = r.s;
                pu[1] = r.c;
            }
            mine = Comp{};
        }
    }
    if (part && !act) {
        const Comp r = block_sum_comp<kAxThreads>(mine, red);
        if (threadIdx.x == 0) {
            part[2 * blockIdx.x] = r.s;
            part[2 * blockIdx.x + 1] = r.c;
        }
    }
}

// A x on at most kAxDirectBlocks blocks (a small fit, the last small problems
// of a batch): units of 1/kAxSplitMax of a block, one row a thread, all
// gathers through L1 and L2, in the order of the table kernel, so both give
// the same values.  So few rows are done before a table would be staged.
// Without act it runs when the host chose it; with act it decides on the
// device, as the table kernel (launched beside it) does, and exactly one of
// the two does the work.  Partials [block][kAxSplitMax].
//
// Bound by latency, so a row's index words are loaded ahead of its gathers: all
// of them where every pattern has 8 slots; four patterns' where the loads are
// predicated by the slots (five reference patterns, 3,000 rows, FP64 LSQR's
// product: 10.4 us with all ahead, 7.4 so).
template <typename T, typename Y, int MODE, bool ALL8>
__global__ void __launch_bounds__(kAxDirectRows) fast_spmv_direct_kernel(FastGeometry g,
                                                                         const uint16_t* __restrict__ a16,
                                                                         const T* __restrict__ x, Y* __restrict__ y,
                                                                         const double* __restrict__ b,
                                                                         const double* __restrict__ coef,
                                                                         double* __restrict__ part,
                                                                         const int* __restrict__ done,
                                                                         const int* __restrict__ pdone,
                                                                         const FastActive* __restrict__ act)
{
    constexpr int kAhead = ALL8 ? kRowPatterns : 4;
    __shared__ double red[64];
    __shared__ int pref[kMaxProblems + 1];
    if (done && *(volatile const int*)done) return;
    const double c = MODE == 1 ? *coef : 0.0;
    int64_t nblk = g.nblocks;
    if (act) {
        nblk = active_prefix(act, pref, [&](int q) { return g.pblk0[q + 1] - g.pblk0[q]; });
        if (nblk > kAxDirectBlocks) return;  // the table kernel's work
    }
    const int64_t units = nblk * kAxSplitMax;
    for (int64_t u = blockIdx.x; u < units; u += gridDim.x) {
        const int sp = static_cast<int>(u % kAxSplitMax);
        int64_t blk = u / kAxSplitMax;
        if (act) {
            const int i = static_cast<int>(blk);
            const int slot = active_slot(pref, act->n, i);
            blk = g.pblk0[act->list[slot]] + (i - pref[slot]);
        }
        const int q = g.prob_of_block(blk);
        double* pu = part ? part + 2 * (blk * kAxSplitMax + sp) : nullptr;
        if (pdone && pdone[q]) {
            if (pu && threadIdx.x == 0) {
                pu[0] = 0;
                pu[1] = 0;
            }
            continue;
        }
        const int rows_b = static_cast<int>(g.block_rows(blk));
        const int r0 = rows_b * sp / kAxSplitMax, nb = rows_b * (sp + 1) / kAxSplitMax - r0;
        Comp mine;
        if (static_cast<int>(threadIdx.x) < nb) {
            const int r = r0 + threadIdx.x;
            const double v = static_cast<double>(
                row_sum<T, ALL8, false, kAhead>(g, a16, blk, r, x + q * g.pcols, FastTable{}, nullptr));
            const double yv = store_row<Y, MODE>(v, y, b, c, g.block_row0(blk) + r);
            mine.add(yv * yv);
        }
        if (pu) {
            const Comp rs = block_sum_comp<kAxDirectRows>(mine, red);
            if (threadIdx.x == 0) {
                pu[0] = rs.s;
                pu[1] = rs.c;
            }
        }
    }
}

// ---------------------------------------------------------------------------
// A'y on the blocked layout.
// ---------------------------------------------------------------------------
struct TView {
    const int* item_sc;
    const int* item_b0;
    const int* item_b1;
    const int64_t* item_part;
    const int* sc_piece0;
    const int* piece_pat;
    const int* piece_ch0;
    const int* piece_ch1;
    const int* piece_acc;
    const uint32_t* units;
    int nunits;
    int nsc;
    int npieces;
};

// The units of a list of one item per (block, chunk): splits of each chunk
// (0: the list has its own units).
struct BlockUnits {
    int per_block = 0;
    uint8_t splits[kMaxChunks];
};

// Column-sorted entries are reduced lane by lane.  For one block of an item,
// the entry ranges of all the item's pieces (their shares of columns) are
// cut into G32 rounds: piece k covers the rounds that overlap its range
// [lo_k, hi_k), and the pieces' round lists, one after another, form the
// block's list of virtual rounds, which the 32 warps split into contiguous
// stretches of nearly equal length.  In a round each lane owns 32
// consecutive entries (one round is read with 8 coalesced 16-byte loads per
// lane; entries outside the piece's range are masked).  An entry's bit 0
// marks the last entry of its column, so a lane sums y over its entries and
// closes a run at every flagged entry, with no column comparisons.  A
// column's entries of a block are one run, so only the lane where a run ends
// touches its column, and the order of the adds is fixed by the data: the
// result is bitwise reproducible.
//   1. at every run end the lane adds its own part of the run to acc[col];
//   2. the parts of a run in the lanes before (their open tails) are combined
//      by a segmented scan over the warp's lanes (shuffles; the run still
//      open at the end of the warp's previous round enters as `carry`) and
//      added by the lane where the run ends;
//   3. the run still open at the end of a warp's stretch goes to the warp's
//      record;
//   4. after the block, warp 0 combines the 32 records with the same
//      segmented scan (one lane per warp) and adds each chain to the column
//      where it ends.
// A run never crosses pieces (a piece holds whole columns), so the chain is
// reset where a warp's stretch moves on to the next piece.

constexpr int kMaxPieces = kMaxFastPatterns;  // pieces of one super-chunk: at most one per pattern

// The pieces of one (item, block): logical entry ranges, the accumulator
// index of column field 0, and the first virtual round of each piece.
struct BlockPieces {
    uint32_t lo[kMaxPieces];
    uint32_t hi[kMaxPieces];
    int acc_off[kMaxPieces];
    int round0[kMaxPieces + 1];
    int n;
};

// What a warp leaves for the runs that cross warp boundaries.
template <typename T>
struct WarpRec {
    T ls;        // open sum of the warp's last run (0 when that run ends in the warp)
    int fc;      // accumulator index of the warp's first entry's column
    int valid;   // the warp's stretch is non-empty
    int cp;      // the first run continues the previous warp's last run
    int single;  // no run ends in the warp's stretch
};

// y of an entry: its row, already scaled by 4, sits in bits 2..15.
template <typename T>
__device__ __forceinline__ T y_of(const T* __restrict__ ytile, uint32_t e)
{
    if constexpr (sizeof(T) == 4)
        return *reinterpret_cast<const T*>(reinterpret_cast<const char*>(ytile) + (e & 0xFFFCu));
    else
        return ytile[(e & 0xFFFCu) >> 2];
}

// Segmented inclusive scan over the 32 lanes of the open run sums ts.  A
// chain starts at a lane that ends a run (its tail) or whose first entry
// starts a column; a lane with no run end that continues the run from its
// left (single && cont_prev) extends the chain.  The lane whose first run
// continues from the left and ends in it gets the chain of the lanes before
// it (carry before lane 0) through `sink`.  Lanes without entries pass the
// chain through.  Returns the chain leaving lane 31.
template <typename T, typename Sink>
__device__ __forceinline__ T lane_chain(bool any, bool single, bool cont_prev, int hc, T ts, T carry, Sink&& sink)
{
    const int lane = threadIdx.x & 31;
    T v = any ? ts : T(0);
    bool f = any && !(single && cont_prev);
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const T vu = __shfl_up_sync(0xffffffffu, v, d);
        const bool fu = __shfl_up_sync(0xffffffffu, f, d);
        if (lane >= d) {
            if (!f) v += vu;
            f = f || fu;
        }
    }
    const T X = f ? v : v + carry;  // chain value ending at this lane
    T Xprev = __shfl_up_sync(0xffffffffu, X, 1);
    if (lane == 0) Xprev = carry;
    if (any && !single && cont_prev) sink(hc, Xprev);
    return __shfl_sync(0xffffffffu, X, 31);
}

__device__ __forceinline__ uint32_t word_of(const uint4& u, int j)
{
    return j == 0 ? u.x : (j == 1 ? u.y : (j == 2 ? u.z : u.w));
}

// A lane's entries of one round: slots [k0, k1) of its 32 (all of them when
// FULL), read from src (the lane's first 16-byte word of the round) in two
// halves of 16.  Runs that end here are added to accc (indexed by an entry's
// column field); returns the open tail, the OR of the entries (bit 0: some
// run ended) and the first and last entries in range.
template <typename T, bool FULL>
__device__ __forceinline__ T lane_entries(const uint4* __restrict__ src, int k0, int k1, const T* __restrict__ ytile,
                                          T* __restrict__ accc, uint32_t& eor, uint32_t& first_e, uint32_t& last_e)
{
    T sum = 0;
    uint32_t o = 0, fe = 1u, le = 1u;
#pragma unroll
    for (int h = 0; h < 2; h++) {
        uint4 u[4];
#pragma unroll
        for (int q = 0; q < 4; q++) u[q] = __ldcs(src + 32 * (4 * h + q));
#pragma unroll
        for (int t = 0; t < kLaneRun / 2; t++) {
            const int s = (kLaneRun / 2) * h + t;
            const uint32_t e = word_of(u[t >> 2], t & 3);
            if (FULL || (s >= k0 && s < k1)) {
                sum += y_of<T>(ytile, e);
                o |= e;
                if (e & 1u) {  // the run ends here: this lane's part of it
                    accc[e >> 16] += sum;
                    sum = T(0);
                }
                if (FULL) {
                    if (s == 0) fe = e;
                } else if (s == k0) {
                    fe = e;
                }
                le = e;
            }
        }
    }
    eor = o;
    first_e = fe;
    last_e = le;
    return sum;
}

// Lane w asks L2 for the first round of warp w's stretch in the block whose
// table is bp.
__device__ __forceinline__ void prefetch_first_rounds(const uint32_t* __restrict__ g32, const BlockPieces& bp)
{
    constexpr int kWarps = kFastThreads / 32;
    static_assert(kWarps == 32, "a lane per warp");
    const int w = threadIdx.x & 31;
    const int nrounds = bp.round0[bp.n];
    const int v = nrounds * w / kWarps;
    if (v >= nrounds * (w + 1) / kWarps) return;  // no stretch
    int k = 0;
    while (bp.round0[k + 1] <= v) k++;
    const uint32_t rbase = ((bp.lo[k] / kRound) + static_cast<uint32_t>(v - bp.round0[k])) * kRound;
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(g32 + rbase),
                 "r"(static_cast<unsigned>(kRound * sizeof(uint32_t)))
                 : "memory");
}

// The reduction of one block's entries of every piece in `bp` into acc.
// Ends with a block barrier and warp 0's record combination; the next block
// may restage ytile after the next barrier.
template <typename T>
__device__ __forceinline__ void reduce_block(const uint32_t* __restrict__ g32, const BlockPieces& bp,
                                             const T* __restrict__ ytile,
                                             T* __restrict__ acc, WarpRec<T>* recs)
{
    constexpr int kWarps = kFastThreads / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nrounds = bp.round0[bp.n];
    const int vr0 = nrounds * warp / kWarps, vr1 = nrounds * (warp + 1) / kWarps;
    T carry = 0;
    bool prev_end = true;
    bool w_end = false, w_cp = false;
    int w_fc = 0;
    int k = 0;
    while (k < bp.n && bp.round0[k + 1] <= vr0) k++;
    for (int vr = vr0; vr < vr1; vr++) {
        if (vr >= bp.round0[k + 1]) {  // the stretch moves on to the next piece
            do {
                k++;
            } while (vr >= bp.round0[k + 1]);
            carry = T(0);
            prev_end = true;
        }
        const uint32_t lo = bp.lo[k], hi = bp.hi[k];
        const uint32_t rbase = ((lo / kRound) + static_cast<uint32_t>(vr - bp.round0[k])) * kRound;
        T* accc = acc + bp.acc_off[k];
        if (lane == 0 && vr + 1 < bp.round0[k + 1]) {
            // the next round of this piece into L2 while this one is reduced
            asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(g32 + rbase + kRound),
                         "r"(static_cast<unsigned>(kRound * sizeof(uint32_t)))
                         : "memory");
        }
        const uint4* src = reinterpret_cast<const uint4*>(g32 + rbase) + lane;
        const uint32_t lb = rbase + kLaneRun * lane;  // the lane's first slot
        const int k0 = lo > lb ? static_cast<int>(min(lo - lb, static_cast<uint32_t>(kLaneRun))) : 0;
        const int k1 = hi > lb ? static_cast<int>(min(hi - lb, static_cast<uint32_t>(kLaneRun))) : 0;
        const bool any = k0 < k1;
        uint32_t eor, first_e, last_e;
        T sum;
        if (__all_sync(0xffffffffu, k0 == 0 && k1 == kLaneRun))
            sum = lane_entries<T, true>(src, 0, kLaneRun, ytile, accc, eor, first_e, last_e);
        else
            sum = lane_entries<T, false>(src, k0, k1, ytile, accc, eor, first_e, last_e);
        // no run ends in the lane: one column, its last entry not flagged
        const bool single = any && !(eor & 1u);
        const int hc = static_cast<int>(first_e >> 16);  // the lane's first run
        // the lane continues the run of the entry before it unless that entry
        // ended its run (previous lane's last entry; at lane 0 the warp's
        // previous round, and none in the warp's first round: the record
        // chain joins runs across warps)
        const uint32_t f = lb + static_cast<uint32_t>(k0);
        const uint32_t prev_last = __shfl_up_sync(0xffffffffu, last_e, 1);
        const bool cont_prev = any && f > lo && (lane == 0 ? (vr != vr0 && !prev_end) : !(prev_last & 1u));
        auto sink = [&](int col, T val) { accc[col] += val; };
        const unsigned anyb = __ballot_sync(0xffffffffu, any);
        const int lastl = 31 - __clz(anyb);  // a round holds at least one entry of its piece
        if (__ballot_sync(0xffffffffu, single && cont_prev) == 0) {
            // no lane extends a run from its left: a chain is one lane's tail
            T prev_ts = __shfl_up_sync(0xffffffffu, sum, 1);
            if (lane == 0) prev_ts = carry;
            if (any && !single && cont_prev) sink(hc, prev_ts);
            carry = __shfl_sync(0xffffffffu, sum, lastl);
        } else {
            carry = lane_chain<T>(any, single, cont_prev, hc, sum, carry, sink);
        }
        prev_end = (__shfl_sync(0xffffffffu, last_e, lastl) & 1u) != 0;
        if (vr == vr0) {
            // the stretch's first entry: its column, and whether it continues
            // the run that ends the previous warp's stretch
            const int fl = __ffs(anyb) - 1;
            const uint32_t f0 = __shfl_sync(0xffffffffu, f, fl);
            w_fc = bp.acc_off[k] + static_cast<int>(__shfl_sync(0xffffffffu, first_e, fl) >> 16);
            w_cp = f0 > lo && !(g32[round_phys(f0 - 1)] & 1u);
        }
        const bool ended = __ballot_sync(0xffffffffu, any && !single) != 0;  // every lane votes, every round
        w_end = w_end || ended;
    }
    if (lane == 0) {
        WarpRec<T>& rec = recs[warp];
        rec.valid = vr0 < vr1;
        rec.ls = carry;  // the chain still open at the stretch's end (0 if its last run ended)
        rec.fc = w_fc;
        rec.cp = w_cp;
        rec.single = !w_end;
    }
    __syncthreads();
    if (warp == 0) {
        WarpRec<T> r{};  // lanes past the CTA's warps carry no stretch
        if (lane < kWarps) r = recs[lane];
        lane_chain<T>(r.valid != 0, r.single != 0, r.cp != 0, r.fc, r.ls, T(0),
                      [&](int col, T val) { acc[col] += val; });
    }
}

// ---------------------------------------------------------------------------
// The same reduction for items whose blocks hold few rounds (the FP64
// products, whose accumulator holds one chunk): each (block, piece) entry
// range is cut into 32 nearly equal stretches of whole 4-entry words, one
// per warp, so every warp works whatever the number of rounds; a warp's
// stretch is reduced in steps of kStretchRun entries per lane (consecutive
// in the sorted order, two 16-byte words of G32 each), with the same lane
// chain and warp records.
// ---------------------------------------------------------------------------
constexpr int kStretchRun = 16;                 // entries per lane and step
constexpr int kStretchVecs = kStretchRun / 4;   // 16-byte words per lane and step

// The 16-byte word of G32 that holds sorted positions e .. e+3 (e a
// multiple of 4).
__device__ __forceinline__ uint4 word_at(const uint32_t* __restrict__ g32, uint32_t e)
{
    return __ldcs(reinterpret_cast<const uint4*>(g32 + round_phys(e)));
}

// A lane's entries of a step are all inside the warp's stretch.
__device__ __forceinline__ bool lane_full(uint32_t e_first, uint32_t w_lo, uint32_t w_hi)
{
    return e_first >= w_lo && e_first + kStretchRun <= w_hi;
}

__device__ __forceinline__ void load_lane(const uint32_t* __restrict__ g32, uint32_t e_first,
                                          uint4 (&u)[kStretchVecs])
{
#pragma unroll
    for (int q = 0; q < kStretchVecs; q++) u[q] = word_at(g32, e_first + 4 * q);
}

// One step of a warp over [w_lo, w_hi): lanes take kStretchRun entries
// each from step_start (a multiple of 4).  A lane whose entries are all in
// range gets them in `cur` (loaded ahead by the caller); edge lanes load
// theirs one by one.  accc: the accumulator shifted so that an entry's
// column field indexes it.  carry: the run open before the step (updated);
// prev_end: the last entry before this step ended its run (updated).
template <typename T>
__device__ __forceinline__ void stretch_step(const uint32_t* __restrict__ g32, uint32_t step_start, uint32_t w_lo,
                                             uint32_t w_hi, const T* __restrict__ ytile, T* __restrict__ accc,
                                             T& carry, bool& prev_end, const uint4 (&cur)[kStretchVecs], bool full)
{
    const int lane = threadIdx.x & 31;
    const uint32_t e_first = step_start + lane * kStretchRun;
    T sum = 0;
    uint32_t ends = 0;
    auto step = [&](uint32_t e) {
        sum += y_of<T>(ytile, e);
        ends |= e;
        if (e & 1u) {  // the run ends here: this lane's part of it
            accc[e >> 16] += sum;
            sum = T(0);
        }
    };
    bool any = false;
    uint32_t first_ent = 1u, last_ent = 1u;  // an empty lane looks like a closed run
    if (full) {
        first_ent = cur[0].x;
#pragma unroll
        for (int q = 0; q < kStretchVecs; q++) {
            step(cur[q].x);
            step(cur[q].y);
            step(cur[q].z);
            step(cur[q].w);
        }
        any = true;
        last_ent = cur[kStretchVecs - 1].w;
    } else {
        const uint32_t lo = max(e_first, w_lo), hi = min(e_first + kStretchRun, w_hi);
        if (lo < hi) {
            for (uint32_t e = lo; e < hi; e++) step(g32[round_phys(e)]);
            any = true;
            first_ent = g32[round_phys(lo)];
            last_ent = g32[round_phys(hi - 1)];
        }
    }
    const bool single = any && !(ends & 1u);
    const int hc = static_cast<int>(first_ent >> 16);
    const uint32_t first_valid = max(e_first, w_lo);
    const uint32_t prev_last = __shfl_up_sync(0xffffffffu, last_ent, 1);
    const bool cont_prev = any && first_valid > w_lo && (lane == 0 ? !prev_end : !(prev_last & 1u));
    auto sink = [&](int col, T val) { accc[col] += val; };
    if (__ballot_sync(0xffffffffu, single && cont_prev) == 0) {
        T prev_ts = __shfl_up_sync(0xffffffffu, sum, 1);
        if (lane == 0) prev_ts = carry;
        if (any && !single && cont_prev) sink(hc, prev_ts);
        const int last = min(31, static_cast<int>((w_hi - 1 - step_start) / kStretchRun));  // last lane with entries
        carry = __shfl_sync(0xffffffffu, sum, last);
    } else {
        carry = lane_chain<T>(any, single, cont_prev, hc, sum, carry, sink);
    }
    prev_end = (__shfl_sync(0xffffffffu, last_ent, 31) & 1u) != 0;
}

// The stretch reduction of one block's entries [e_lo, e_hi) of one piece
// into accc (indexed by column field).  Ends with a block barrier; warp 0
// then combines the records (recs: the set of this piece; the caller
// alternates two sets so that the next piece may start meanwhile).
template <typename T>
__device__ __forceinline__ void reduce_stretch(const uint32_t* __restrict__ g32, uint32_t e_lo, uint32_t e_hi,
                                               const T* __restrict__ ytile, T* __restrict__ accc, WarpRec<T>* recs)
{
    constexpr int kWarps = kFastThreads / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t n = e_hi - e_lo;
    auto cut = [&](int w) -> uint32_t {
        if (w == 0) return e_lo;
        if (w == kWarps) return e_hi;
        return max(e_lo, (e_lo + static_cast<uint32_t>(n * w / kWarps)) & ~3u);
    };
    const uint32_t w_lo = cut(warp), w_hi = cut(warp + 1);
    T carry = 0;
    bool prev_end = true;
    const uint32_t step_len = 32 * kStretchRun;
    const uint32_t rs0 = w_lo & ~3u;
    if (w_lo < w_hi) {
        // two register buffers that swap roles every step: the next step's
        // entries load while this one is reduced
        uint4 ba[kStretchVecs], bb[kStretchVecs];
        uint32_t rs = rs0;
        bool fa = rs < w_hi && lane_full(rs + lane * kStretchRun, w_lo, w_hi);
        if (fa) load_lane(g32, rs + lane * kStretchRun, ba);
        while (rs < w_hi) {
            uint32_t rn = rs + step_len;
            const bool fb = rn < w_hi && lane_full(rn + lane * kStretchRun, w_lo, w_hi);
            if (fb) load_lane(g32, rn + lane * kStretchRun, bb);
            stretch_step<T>(g32, rs, w_lo, w_hi, ytile, accc, carry, prev_end, ba, fa);
            rs = rn;
            if (rs >= w_hi) break;
            rn = rs + step_len;
            fa = rn < w_hi && lane_full(rn + lane * kStretchRun, w_lo, w_hi);
            if (fa) load_lane(g32, rn + lane * kStretchRun, ba);
            stretch_step<T>(g32, rs, w_lo, w_hi, ytile, accc, carry, prev_end, bb, fb);
            rs = rn;
        }
    }
    if (lane == 0) {
        WarpRec<T>& rec = recs[warp];
        rec.valid = w_lo < w_hi;
        rec.ls = carry;  // the chain still open at the stretch's end (0 if its last run ended)
        rec.fc = rec.cp = rec.single = 0;
        if (w_lo < w_hi) {
            const uint32_t ef = g32[round_phys(w_lo)], el = g32[round_phys(w_hi - 1)];
            rec.fc = static_cast<int>(ef >> 16);
            rec.cp = w_lo > e_lo && !(g32[round_phys(w_lo - 1)] & 1u);
            rec.single = ((ef ^ el) >> 16) == 0 && !(el & 1u);
        }
    }
    __syncthreads();
    if (warp == 0) {
        WarpRec<T> r{};  // lanes past the CTA's warps carry no stretch
        if (lane < kWarps) r = recs[lane];
        lane_chain<T>(r.valid != 0, r.single != 0, r.cp != 0, r.fc, r.ls, T(0),
                      [&](int col, T val) { accc[col] += val; });
    }
}

// A piece in shared memory (loaded once by each CTA).
struct PieceMeta {
    int pat;
    int sub0;  // first column sub-chunk
    int w;     // columns
    int acc;   // accumulator offset of the first column
};

// First entry of column sub-chunk j (in the pattern's own count of the
// layout) of a block, the group's end past the pattern's last.
__device__ __forceinline__ uint32_t sub_entry(const FastGeometry& g, const uint32_t* __restrict__ sub_start, int p,
                                              int j, int64_t blk)
{
    const int end = (p + 1 < g.npat ? g.chunk0[p + 1] : g.nchunks) * kSubPerChunk;
    return j < end ? sub_start[blk * (static_cast<int64_t>(g.nchunks) * kSubPerChunk) + j]
                   : static_cast<uint32_t>(g.seg(blk, p) + g.seg_len(blk, p));
}

// The columns of every piece that split `split` of K covers, by one warp: the
// item's sub-chunks in piece order are cut where the entries of block blk
// pass s / K of the item's.  (Cut by column counts, the columns that hold
// most entries stayed in one unit: 1,024 columns hold up to 77% of a
// pattern's entries, 64 up to 15%.)
__device__ __forceinline__ void unit_share(const FastGeometry& g, const PieceMeta* pm, int npc,
                                           const uint32_t* __restrict__ sub_start, int64_t blk, int split, int K,
                                           int2* share)
{
    const int lane = threadIdx.x & 31;
    int w = 0, ns = 0;
    if (lane < npc) w = pm[lane].w;
    int ck[2] = {0, npc}, cc[2] = {0, 0};  // first and end cut: piece, column
    if (K > 1) {
        uint32_t start = 0, len = 0;
        if (lane < npc) {
            ns = (w + kSubCols - 1) / kSubCols;
            start = sub_entry(g, sub_start, pm[lane].pat, pm[lane].sub0, blk);
            len = sub_entry(g, sub_start, pm[lane].pat, pm[lane].sub0 + ns, blk) - start;
        }
        uint32_t incl = len;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t u = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= d) incl += u;
        }
        const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
        // half a warp for each cut
        const int e = lane >> 4, l = lane & 15;
        const int sp = split + e;
        const uint32_t tgt = sp < K ? static_cast<uint32_t>(static_cast<uint64_t>(total) * sp / K) : 0;
        int k = 0;  // the piece where the entries pass the target
        for (int t = 0; t < npc; t++) k += __shfl_sync(0xffffffffu, incl, t) <= tgt;
        const bool inside = sp > 0 && sp < K && k < npc;
        const int kk = min(k, npc - 1);
        const uint32_t goal = __shfl_sync(0xffffffffu, start, kk) + (tgt - __shfl_sync(0xffffffffu, incl - len, kk));
        const int p = pm[kk].pat, sub0 = pm[kk].sub0;
        // first sub-chunk that starts at or after the goal
        int lo = 0, hi = __shfl_sync(0xffffffffu, ns, kk);
        if (!inside) hi = 0;
        while (__any_sync(0xffffffffu, lo < hi)) {
            const int step = (hi - lo + 15) / 16, j = lo + l * step;
            const unsigned at = __ballot_sync(0xffffffffu, j >= hi || sub_entry(g, sub_start, p, sub0 + j, blk) >= goal) >>
                                (16 * e) & 0xFFFFu;
            const int f = at ? __ffs(at) - 1 : 16;
            const int nlo = f == 0 ? lo : lo + (f - 1) * step + 1;
            if (f < 16) hi = min(hi, lo + f * step);
            lo = min(nlo, hi);
        }
        // a cut past the last entry is the end (no entries: the first split covers all)
        const int cut = sp == 0 ? 0 : (inside ? k : npc), col = inside ? lo * kSubCols : 0;
        ck[0] = __shfl_sync(0xffffffffu, cut, 0);
        cc[0] = __shfl_sync(0xffffffffu, col, 0);
        ck[1] = __shfl_sync(0xffffffffu, cut, 16);
        cc[1] = __shfl_sync(0xffffffffu, col, 16);
    }
    if (lane < npc) {
        const int a0 = lane < ck[0] ? w : (lane == ck[0] ? min(w, cc[0]) : 0);
        const int a1 = lane < ck[1] ? w : (lane == ck[1] ? min(w, cc[1]) : 0);
        share[lane] = make_int2(a0, a1);
    }
    __syncwarp();
}

// The table of one block's pieces (entry ranges of their shares, the
// accumulator offsets, the virtual rounds), by one warp.
__device__ __forceinline__ void fill_pieces(const FastGeometry& g, const PieceMeta* pm, int npc,
                                            const uint32_t* __restrict__ sub_start, const int2* share, int64_t blk,
                                            BlockPieces& bp)
{
    const int lane = threadIdx.x & 31;
    uint32_t lo = 0, hi = 0;
    int off = 0, nr = 0;
    if (lane < npc) {
        const PieceMeta m = pm[lane];
        const int a0 = share[lane].x, a1 = share[lane].y;
        if (a0 < a1) {
            lo = sub_entry(g, sub_start, m.pat, m.sub0 + a0 / kSubCols, blk);
            hi = sub_entry(g, sub_start, m.pat, m.sub0 + (a1 + kSubCols - 1) / kSubCols, blk);
            off = m.acc - (m.sub0 * kSubCols - g.chunk0[m.pat] * kChunkCols);
            if (lo < hi) nr = static_cast<int>((hi - 1) / kRound - lo / kRound) + 1;
        }
    }
    int incl = nr;  // inclusive scan of the rounds over the pieces
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += v;
    }
    if (lane < npc) {
        bp.lo[lane] = lo;
        bp.hi[lane] = hi;
        bp.acc_off[lane] = off;
        bp.round0[lane + 1] = incl;
    }
    if (lane == 0) {
        bp.round0[0] = 0;
        bp.n = npc;
    }
    __syncwarp();
}

template <typename T>
struct AtyShared {
    // two record sets: the stretch reduction alternates them per piece, so
    // that warp 0 may still combine one piece's records while the other
    // warps start on the next piece
    WarpRec<T> recs[2][kFastThreads / 32];
    BlockPieces bp[2];  // this block's piece table and the next one's
    PieceMeta pm[kMaxChunks];
    int sc_piece0[kMaxChunks + 1];
    // the unit: what its loop over blocks needs.  In shared memory, because
    // the reductions need all 64 registers: with these held or spilled, the
    // FP64 A'y of 610 blocks took 3,020 us, 2,570 so.  (The FP64 reduction
    // still spills 116 bytes a thread, the FP32 one none.)
    int64_t out;             // offset of its partials
    const T* yb;             // y of its first block
    int b0, nblk;
    int full, rest;          // blocks from the first one on that are whole (at most nblk), rows of the next one
    int pc0, npc;            // its pieces
    int2 share[kMaxPieces];  // columns of the unit in each piece
    int unit;                // the CTA's next unit (persistent schedules)
    uint32_t pack;           // the unit of a block list
};

// Stages y of `nb` rows into the tile by asynchronous copies, 16 bytes each
// where the slice is aligned (a batch's problems start at any row); the caller
// waits for them (stage_wait) before its barrier.
template <typename T>
__device__ __forceinline__ void stage_y(const T* __restrict__ yb, int nb, T* __restrict__ ytile)
{
    if (!yb) {  // no y: a vector of ones (the column counts A'1)
        for (int i = threadIdx.x; i < nb; i += kFastThreads) ytile[i] = T(1);
        return;
    }
    constexpr int kPer = 16 / sizeof(T);
    constexpr unsigned kSize = sizeof(T);
    const bool aligned = (reinterpret_cast<uintptr_t>(yb) & 15) == 0;
    const int nvec = aligned ? nb / kPer : 0;
    const unsigned dst = static_cast<unsigned>(__cvta_generic_to_shared(ytile));
    for (int i = threadIdx.x; i < nvec; i += kFastThreads)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 16u * i), "l"(yb + kPer * i) : "memory");
    for (int i = nvec * kPer + threadIdx.x; i < nb; i += kFastThreads)
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(dst + kSize * i), "l"(yb + i), "n"(kSize) : "memory");
}

__device__ __forceinline__ void stage_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// One work unit: split `split` of K of item `item`, i.e. the partial column
// sums of its share of super-chunk item_sc[item]'s columns (unit_share by the
// item's first block) over the blocks [item_b0, item_b1), written to those
// columns of partial + item_part[item] - item_part[item_base].  A column's
// entries of a block are one run of the sorted group, so splitting at
// sub-chunk bounds splits no run.
// STRETCH: each (block, piece) range is reduced on its own by the stretch
// reduction (the FP64 items); else the block's pieces share one round list.
//
// A unit of a small product is a chain of dependent loads, so the chain is
// short: the item's fields at once, then the first block's y (asynchronous
// copies) beside the unit's share and the table of the block's pieces, whose
// fields the CTA has in shared memory.
template <typename T, bool STRETCH>
__device__ __forceinline__ void aty_item(const FastGeometry& g, const TView& tv, const uint32_t* __restrict__ g32,
                                         const uint32_t* __restrict__ sub_start, const T* __restrict__ y,
                                         T* __restrict__ partial, int item, int item_base, int64_t y_block0,
                                         int split, int K, T* __restrict__ acc, T* __restrict__ ytile,
                                         AtyShared<T>& sh, const int* __restrict__ pdone)
{
    const int warp = threadIdx.x >> 5;
    {
        const int sc = tv.item_sc[item];
        const int b0 = tv.item_b0[item], b1 = tv.item_b1[item];
        const int64_t out = tv.item_part[item] - tv.item_part[item_base];
        const int q = g.prob_of_block(b0);  // items never span problems
        if (pdone && pdone[q]) return;      // retired problem: partials unused
        const int64_t row0 = g.prow0[q] + static_cast<int64_t>(b0 - g.pblk0[q]) * kBlockRows;
        // the problem's rows from here on: 2^31 and more with one entry a row
        const int64_t left = g.prow0[q + 1] - row0;
        const int full = static_cast<int>(min(left / kBlockRows, static_cast<int64_t>(b1 - b0)));
        const int rest = static_cast<int>(left % kBlockRows);
        const T* yb = y ? y + (row0 - g.block_row0(y_block0)) : nullptr;
        stage_y(yb, full > 0 ? kBlockRows : rest, ytile);
        if (warp == 0) {
            const int pc0 = sh.sc_piece0[sc], npc = sh.sc_piece0[sc + 1] - pc0;
            if (threadIdx.x == 0) {
                sh.out = out;
                sh.yb = yb;
                sh.b0 = b0;
                sh.nblk = b1 - b0;
                sh.full = full;
                sh.rest = rest;
                sh.pc0 = pc0;
                sh.npc = npc;
            }
            unit_share(g, sh.pm + pc0, npc, sub_start, b0, split, K, sh.share);
            fill_pieces(g, sh.pm + pc0, npc, sub_start, sh.share, b0, sh.bp[0]);
            if (!STRETCH) prefetch_first_rounds(g32, sh.bp[0]);
        }
    }
    __syncthreads();
    for (int k = 0; k < sh.npc; k++) {
        T* ap = acc + sh.pm[sh.pc0 + k].acc;
        for (int i = sh.share[k].x + threadIdx.x; i < sh.share[k].y; i += kFastThreads) ap[i] = 0;
    }
    for (int i = 0; i < sh.nblk; i++) {
        if (i > 0) {
            __syncthreads();  // the tile is free
            stage_y(sh.yb ? sh.yb + static_cast<int64_t>(i) * kBlockRows : nullptr,
                    i < sh.full ? kBlockRows : sh.rest, ytile);
        }
        if (i + 1 < sh.nblk) {
            if (sh.yb)  // the next block's y slice into L2
                prefetch_l2(sh.yb + static_cast<int64_t>(i + 1) * kBlockRows,
                            (i + 1 < sh.full ? kBlockRows : sh.rest) * static_cast<int64_t>(sizeof(T)));
            if (warp == 0) {  // and its table, a block ahead
                fill_pieces(g, sh.pm + sh.pc0, sh.npc, sub_start, sh.share, sh.b0 + i + 1, sh.bp[(i + 1) & 1]);
                if (!STRETCH) prefetch_first_rounds(g32, sh.bp[(i + 1) & 1]);
            }
        }
        stage_wait();
        __syncthreads();
        const BlockPieces& bp = sh.bp[i & 1];
        if constexpr (STRETCH) {
            int flip = 0;
            for (int k = 0; k < bp.n; k++) {
                const uint32_t lo = bp.lo[k], hi = bp.hi[k];
                if (lo >= hi) continue;
                reduce_stretch<T>(g32, lo, hi, ytile, acc + bp.acc_off[k], sh.recs[flip]);
                flip ^= 1;
            }
        } else {
            reduce_block<T>(g32, bp, ytile, acc, sh.recs[0]);
        }
    }
    __syncthreads();
    T* out = partial + sh.out;
    for (int k = 0; k < sh.npc; k++) {
        const int o = sh.pm[sh.pc0 + k].acc;
        for (int i = sh.share[k].x + threadIdx.x; i < sh.share[k].y; i += kFastThreads) out[o + i] = acc[o + i];
    }
}

// A'y over a work list's units (unit_pack), or over those of the active
// list's problems.  With ctr (persistent schedule: one CTA per SM) the CTAs
// take units in order, the first by their index and the next from the counter
// ctr[0], until the list is done, so no SM idles while units of uneven
// duration remain; which CTA runs a unit does not change its output, so
// results stay bitwise reproducible.  The last CTA to finish resets the
// counters for the next launch (launches on one work list must therefore be
// stream-ordered).  Without ctr, CTA i runs unit i.  bu.per_block set: the
// units of a list of one item per (block, chunk), block by block from item
// item_base on.
template <typename T>
__global__ void __launch_bounds__(kFastThreads, 1) fast_spmv_t_kernel(FastGeometry g, TView tv,
                                                                       const uint32_t* __restrict__ g32,
                                                                       const uint32_t* __restrict__ sub_start,
                                                                       const T* __restrict__ y,
                                                                       T* __restrict__ partial,
                                                                       const int* __restrict__ done, int item_base,
                                                                       int64_t y_block0, int* __restrict__ ctr,
                                                                       const int* __restrict__ pdone,
                                                                       const FastActive* __restrict__ act,
                                                                       BlockUnits bu)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ AtyShared<T> sh;
    constexpr bool kStretch = sizeof(T) == 8;  // FP64 items hold one chunk: few rounds per block
    if (done && *(volatile const int*)done) return;
    T* ytile = reinterpret_cast<T*>(smem_raw);  // first: its entries' byte offsets address it directly
    T* acc = ytile + kBlockRows;
    for (int i = threadIdx.x; i < tv.npieces; i += kFastThreads) {
        const int p = tv.piece_pat[i], c0 = tv.piece_ch0[i], c1 = tv.piece_ch1[i];
        const int cl0 = (c0 - g.chunk0[p]) * kChunkCols;
        sh.pm[i] = PieceMeta{p, c0 * kSubPerChunk, min(g.space[p], (c1 - g.chunk0[p]) * kChunkCols) - cl0, tv.piece_acc[i]};
    }
    for (int i = threadIdx.x; i <= tv.nsc; i += kFastThreads) sh.sc_piece0[i] = tv.sc_piece0[i];
    if (!ctr) {
        const int u = static_cast<int>(blockIdx.x);
        if (bu.per_block && threadIdx.x < 32) {
            const int b = u / bu.per_block, r = u - b * bu.per_block, lane = threadIdx.x;
            for (int c0 = 0, at = 0; c0 < g.nchunks; c0 += 32) {
                const int K = c0 + lane < g.nchunks ? bu.splits[c0 + lane] : 0;
                int incl = K;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const int v = __shfl_up_sync(0xffffffffu, incl, d);
                    if (lane >= d) incl += v;
                }
                const int split = r - (at + incl - K);
                if (split >= 0 && split < K) sh.pack = unit_pack(item_base + b * g.nchunks + c0 + lane, split, K);
                at += __shfl_sync(0xffffffffu, incl, 31);
            }
        }
        __syncthreads();
        const uint32_t un = bu.per_block ? sh.pack : tv.units[u];
        aty_item<T, kStretch>(g, tv, g32, sub_start, y, partial, static_cast<int>(un >> 8), item_base, y_block0,
                              static_cast<int>(un >> 4 & 15u), static_cast<int>(un & 15u) + 1, acc, ytile, sh, pdone);
        return;
    }
    __syncthreads();
    constexpr int kType = sizeof(T) == 4 ? 0 : 1;
    const int units = act ? act->nunits[kType] : tv.nunits;
    for (int u = static_cast<int>(blockIdx.x); u < units;) {
        const uint32_t un = act ? act->units[kType][u] : tv.units[u];
        aty_item<T, kStretch>(g, tv, g32, sub_start, y, partial, static_cast<int>(un >> 8), 0, 0,
                              static_cast<int>(un >> 4 & 15u), static_cast<int>(un & 15u) + 1, acc, ytile, sh, pdone);
        if (threadIdx.x == kFastThreads - 1) sh.unit = static_cast<int>(gridDim.x) + atomicAdd(ctr, 1);
        __syncthreads();
        u = sh.unit;
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(ctr + 1, 1) == static_cast<int>(gridDim.x) - 1) {
            ctr[0] = 0;
            ctr[1] = 0;
            __threadfence();
        }
    }
}

// Evaluator forward on a row range: score[r - row0] = sum_j w[col_rj], one
// thread per row (row_sum), gathers of w through L1/L2 (the range is a
// minibatch, too short to amortise staging w in shared memory).
//
// How many patterns' index words a thread loads ahead of its gathers depends
// on what a range is bound by.  Rows that are resident at once are bound by
// their chains of loads: all words ahead.  Longer ranges are bound by the
// gathers' L1 lookups and want as many warps as possible: a pattern at a time,
// in few registers (all words ahead leave 7 CTAs an SM).  Forward, us, all
// words ahead and a pattern at a time: eight expanded patterns, 16,384 rows 9.4
// and 11.6, 131,072 15.0 and 15.5, 163,840 26.3 and 17.2, 3.9M 330 and 290.
// Without the expanded layout's 8 slots everywhere the loads ahead are
// predicated and pay less: the forward takes a pattern at a time (five reference
// patterns, 16,384 rows 9.0 and 8.3, 3.9M 169 and 115), the loss kernel four
// (1, 4 and 8 ahead: 16,384 rows 11.0, 7.0, 6.7; 3.9M 137, 126, 141).
constexpr int kEvalRows = 128;                      // threads of a CTA
constexpr int kEvalCtas = 28;                       // most CTAs per SM of a launch
constexpr int64_t kEvalResident = 7 * kEvalRows;    // rows per SM at once with all words ahead

template <bool ALL8, int AHEAD>
__device__ __forceinline__ float eval_row(const FastGeometry& g, const uint16_t* __restrict__ a16,
                                          const float* __restrict__ w, int64_t r)
{
    int64_t b, rb;
    g.locate_row(r, b, rb);
    return row_sum<float, ALL8, false, AHEAD>(g, a16, b, static_cast<int>(rb), w + g.col_base(b), FastTable{}, nullptr);
}

template <bool ALL8, int AHEAD>
__global__ void __launch_bounds__(kEvalRows) fast_rows_forward_kernel(FastGeometry g, const uint16_t* __restrict__ a16,
                                                                      const float* __restrict__ w, int64_t row0,
                                                                      int64_t row1, float* __restrict__ out)
{
    for (int64_t r = row0 + static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; r < row1;
         r += static_cast<int64_t>(gridDim.x) * blockDim.x)
        out[r - row0] = eval_row<ALL8, AHEAD>(g, a16, w, r);
}

// Dense column sums of per-block partials laid out [block][cols].
__global__ void block_partial_sum_kernel(const float* __restrict__ partial, int nb, int64_t cols,
                                         float* __restrict__ out)
{
    for (int64_t c = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; c < cols;
         c += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        float acc = 0;
        for (int j = 0; j < nb; j++) acc += partial[static_cast<int64_t>(j) * cols + c];
        out[c] = acc;
    }
}

// Forward of a training step fused with its loss: per row the score (as in
// fast_rows_forward_kernel), d = score - target, the Huber loss of d summed
// per CTA into red[blockIdx.x] (FP64, deterministic tree), and the loss
// gradient dscore = clamp(d, -delta, delta) / n for the adjoint.
template <bool ALL8, int AHEAD>
__global__ void __launch_bounds__(kEvalRows) eval_loss_grad_kernel(FastGeometry g, const uint16_t* __restrict__ a16,
                                                                   const float* __restrict__ w,
                                                                   const float* __restrict__ target, int64_t row0,
                                                                   int64_t row1, float delta, float inv_n,
                                                                   float* __restrict__ dscore, double* __restrict__ red)
{
    __shared__ double smem[32];
    double hs = 0;
    for (int64_t r = row0 + static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; r < row1;
         r += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const float tg = target[r - row0];
        const float d = eval_row<ALL8, AHEAD>(g, a16, w, r) - tg;
        const float ad = fabsf(d);
        hs += ad < delta ? 0.5f * d * d : delta * (ad - 0.5f * delta);
        dscore[r - row0] = fminf(fmaxf(d, -delta), delta) * inv_n;
    }
    const double t = block_sum<kEvalRows>(hs, smem);
    if (threadIdx.x == 0) red[blockIdx.x] = t;
}

// Epilogue of a training step, per column c: the gradient g = sum of the
// adjoint's block partials (block order) + 2 l2 w, then Adam on w, m, v with
// the step t = *step + 1 (torch.optim.Adam's update: m += (1 - b1)(g - m),
// v = b2 v + (1 - b2) g^2, w -= lr / (1 - b1^t) * m / (sqrt(v) / sqrt(1 -
// b2^t) + eps)).  ||w||^2 before the update is summed per CTA; the last CTA
// (integer counter) adds the step's loss, sum(Huber)/n + l2 ||w||^2, to
// *loss_sum, stores t and resets the counter.  The step's two powers are one
// thread's work each, behind the loads of the first columns (166,212
// columns, 4 blocks: 9.9 us with both in every thread, 8.5 us so).
__global__ void __launch_bounds__(256) eval_adam_kernel(const float* __restrict__ partial, int nb, int64_t cols,
                                                        float* __restrict__ w, float* __restrict__ m,
                                                        float* __restrict__ v, int64_t* __restrict__ step,
                                                        double* __restrict__ loss_sum, double* __restrict__ red,
                                                        int nred, int* __restrict__ ctr, EvalAdam o, double inv_n)
{
    __shared__ double smem[32];
    __shared__ int last;
    __shared__ float s_step, s_bc2;
    const int64_t t = *step + 1;  // read by every CTA before the last one stores t
    if (threadIdx.x == 0)
        s_step = static_cast<float>(o.lr / (1.0 - pow(static_cast<double>(o.beta1), static_cast<double>(t))));
    if (threadIdx.x == 32)
        s_bc2 = static_cast<float>(sqrt(1.0 - pow(static_cast<double>(o.beta2), static_cast<double>(t))));
    double wsq = 0;
    bool powers = false;
    const int64_t c0 = static_cast<int64_t>(blockIdx.x) * blockDim.x;
    for (int64_t b = c0; b < cols; b += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const int64_t c = b + threadIdx.x;
        float gc = 0, wc = 0, mc = 0, vc = 0;
        if (c < cols) {
            wc = w[c];
            mc = m[c];
            vc = v[c];
            // the partials ahead of their adds, which keep their order (240
            // blocks of 105,543 columns: 86 us with one in flight, 34 so)
            const float* at = partial + c;
            int left = nb;
            for (; left >= 16; left -= 16) sum_ahead<float, 16>(at, cols, gc);
            if (left & 8) sum_ahead<float, 8>(at, cols, gc);
            if (left & 4) sum_ahead<float, 4>(at, cols, gc);
            if (left & 2) sum_ahead<float, 2>(at, cols, gc);
            if (left & 1) sum_ahead<float, 1>(at, cols, gc);
        }
        if (!powers) __syncthreads();  // behind the first columns' loads
        powers = true;
        if (c >= cols) continue;
        const float step_size = s_step, bc2_sqrt = s_bc2;
        wsq += static_cast<double>(wc) * wc;
        gc += (2.0f * o.l2) * wc;
        mc += (1.0f - o.beta1) * (gc - mc);
        vc = o.beta2 * vc + (1.0f - o.beta2) * gc * gc;
        const float denom = sqrtf(vc) / bc2_sqrt + o.eps;
        w[c] = wc - step_size * (mc / denom);
        m[c] = mc;
        v[c] = vc;
    }
    const double s = block_sum<256>(wsq, smem);
    if (threadIdx.x == 0) {
        red[kEvalRedMax + blockIdx.x] = s;
        __threadfence();
        last = atomicAdd(ctr, 1) == static_cast<int>(gridDim.x) - 1;
    }
    __syncthreads();
    if (last) {  // the whole last CTA: strided sums, then the fixed block tree
        __threadfence();
        double h = 0, q = 0;
        for (int i0 = threadIdx.x; i0 < nred; i0 += 8 * 256) {
            double v[8];
#pragma unroll
            for (int u = 0; u < 8; u++) v[u] = i0 + u * 256 < nred ? __ldcg(red + i0 + u * 256) : 0.0;
#pragma unroll
            for (int u = 0; u < 8; u++) h += v[u];
        }
        for (int i = threadIdx.x; i < static_cast<int>(gridDim.x); i += blockDim.x) q += __ldcg(red + kEvalRedMax + i);
        h = block_sum<256>(h, smem);
        q = block_sum<256>(q, smem);
        if (threadIdx.x == 0) {
            *loss_sum += h * inv_n + static_cast<double>(o.l2) * q;
            *step = t;
            *ctr = 0;
            __threadfence();
        }
    }
}

template <typename T>
__global__ void fast_col_sum_kernel(FastCols fc, const T* __restrict__ partial, T* __restrict__ x)
{
    for (int64_t c = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; c < fc.g.cols;
         c += static_cast<int64_t>(gridDim.x) * blockDim.x)
        x[c] = static_cast<T>(fast_col_sum<T, 32>(fc, partial, c));
}

// The small arrays of a work list, gathered on the host and sent to the
// device as one block: one allocation and one copy instead of one each, so
// that building a layout makes few driver calls.
struct MetaPack {
    std::vector<unsigned char> host;
    std::vector<std::pair<size_t, void**>> fields;

    template <typename V>
    void add(const std::vector<V>& v, V** field)
    {
        const size_t off = (host.size() + 15) & ~size_t(15);
        host.resize(off + sizeof(V) * std::max<size_t>(v.size(), 1), 0);
        if (!v.empty()) std::memcpy(host.data() + off, v.data(), sizeof(V) * v.size());
        fields.emplace_back(off, reinterpret_cast<void**>(field));
    }
    // Uploads the block into *base and points every field into it.
    cas_status upload(void** base)
    {
        CAS_CUDA(dmalloc(base, std::max<size_t>(host.size(), 16)));
        if (!host.empty()) CAS_CUDA(cudaMemcpy(*base, host.data(), host.size(), cudaMemcpyHostToDevice));
        for (auto& f : fields) *f.second = static_cast<unsigned char*>(*base) + f.first;
        return CAS_OK;
    }
};

// Columns of a global chunk (the last chunk of a pattern may be partial).
int chunk_width(const FastGeometry& g, int ch)
{
    int p = 0;
    while (p + 1 < g.npat && g.chunk0[p + 1] <= ch) p++;
    return std::min(kChunkCols, g.space[p] - (ch - g.chunk0[p]) * kChunkCols);
}

int pattern_of_chunk(const FastGeometry& g, int ch)
{
    int p = 0;
    while (p + 1 < g.npat && g.chunk0[p + 1] <= ch) p++;
    return p;
}

// Super-chunk pieces, host side.
struct Pieces {
    std::vector<int> sc_piece0, sc_width, pat, ch0, ch1, acc, chunk_sc, chunk_acc;
};

// Packs the chunks, in pattern order, into accumulators of cap columns: a
// chunk joins the current super-chunk while it fits, and consecutive chunks
// of one pattern in one super-chunk form one piece.
Pieces pack_chunks(const FastGeometry& g, int cap, bool across_patterns)
{
    Pieces pc;
    pc.chunk_sc.resize(g.nchunks);
    pc.chunk_acc.resize(g.nchunks);
    int w = 0;
    for (int ch = 0; ch < g.nchunks; ch++) {
        const int p = pattern_of_chunk(g, ch);
        const int cw = chunk_width(g, ch);
        const bool new_pattern = !pc.pat.empty() && pc.pat.back() != p;
        if (pc.sc_piece0.empty() || w + cw > cap || (new_pattern && !across_patterns)) {
            if (!pc.sc_piece0.empty()) pc.sc_width.push_back(w);
            pc.sc_piece0.push_back(static_cast<int>(pc.pat.size()));
            w = 0;
        }
        const bool extend = !pc.pat.empty() && pc.sc_piece0.back() < static_cast<int>(pc.pat.size()) &&
                            pc.pat.back() == p && pc.ch1.back() == ch;
        if (extend) {
            pc.ch1.back() = ch + 1;
        } else {
            pc.pat.push_back(p);
            pc.ch0.push_back(ch);
            pc.ch1.push_back(ch + 1);
            pc.acc.push_back(w);
        }
        pc.chunk_sc[ch] = static_cast<int>(pc.sc_piece0.size()) - 1;
        pc.chunk_acc[ch] = w;
        w += cw;
    }
    if (!pc.sc_piece0.empty()) pc.sc_width.push_back(w);
    pc.sc_piece0.push_back(static_cast<int>(pc.pat.size()));
    return pc;
}

void pack_pieces(const Pieces& pc, FastTranspose& t, MetaPack& mp)
{
    t.nsc = static_cast<int>(pc.sc_width.size());
    t.npieces = static_cast<int>(pc.pat.size());
    mp.add(pc.sc_piece0, &t.sc_piece0);
    mp.add(pc.pat, &t.piece_pat);
    mp.add(pc.ch0, &t.piece_ch0);
    mp.add(pc.ch1, &t.piece_ch1);
    mp.add(pc.acc, &t.piece_acc);
    mp.add(pc.chunk_sc, &t.chunk_sc);
    mp.add(pc.chunk_acc, &t.chunk_acc);
}

// The G32 entries of every item: its super-chunk's chunks over its blocks.
std::vector<int64_t> item_entries(const FastGeometry& g, const std::vector<int64_t>& entries_bc, const Pieces& pc,
                                  const std::vector<int>& item_sc, const std::vector<int>& item_b0,
                                  const std::vector<int>& item_b1)
{
    const int nsc = pc.sc_width.empty() ? 0 : static_cast<int>(pc.sc_width.size());
    // prefix over blocks of every super-chunk's entries
    std::vector<int64_t> pre(static_cast<size_t>(g.nblocks + 1) * nsc, 0);
    for (int64_t b = 0; b < g.nblocks; b++) {
        for (int sc = 0; sc < nsc; sc++) pre[(b + 1) * nsc + sc] = pre[b * nsc + sc];
        for (int ch = 0; ch < g.nchunks; ch++) pre[(b + 1) * nsc + pc.chunk_sc[ch]] += entries_bc[b * g.nchunks + ch];
    }
    std::vector<int64_t> out(item_sc.size());
    for (size_t i = 0; i < item_sc.size(); i++)
        out[i] = pre[static_cast<size_t>(item_b1[i]) * nsc + item_sc[i]] -
                 pre[static_cast<size_t>(item_b0[i]) * nsc + item_sc[i]];
    return out;
}

// The splits of n items, each there `copies` times (fixed cost and entries
// each), on the GPU: none from kPlanWaves items a CTA on, else those of the
// best limit.
std::vector<int> plan_splits(const float* fixed, const float* entries, size_t n, size_t copies)
{
    const float ctas = static_cast<float>(sm_count());
    std::vector<int> K(n, 1);
    if (n * copies >= static_cast<size_t>(kPlanWaves) * sm_count()) return K;
    float top = 0, best = 0, best_limit = 0;
    for (size_t i = 0; i < n; i++) top = std::max(top, fixed[i] + entries[i]);
    for (int j = 0; j < kPlanLimits; j++) {
        const float limit = top * std::exp2(-0.25f * static_cast<float>(j));
        float load = 0, longest = 0, units = 0;
        for (size_t i = 0; i < n; i++) {
            const int k = unit_split(fixed[i], entries[i], limit);
            load += k * fixed[i] + entries[i];
            longest = std::max(longest, fixed[i] + entries[i] / static_cast<float>(k));
            units += static_cast<float>(k);
        }
        units *= static_cast<float>(copies);
        load *= static_cast<float>(copies);
        // items that fit one wave are not cut into two: the second pays the
        // fixed cost of its units once more, and an SM runs one unit at a time
        // (us, whole and cut: a training step's 6 blocks of eight reference
        // patterns 17 and 24, FP64 A'y of 80 blocks of two 64 and 80)
        if (j > 0 && units > ctas && static_cast<float>(n * copies) <= ctas) break;
        const float est = plan_estimate(units, load, longest, ctas);
        if (j == 0 || est < best) {
            best = est;
            best_limit = limit;
        }
    }
    for (size_t i = 0; i < n; i++) K[i] = unit_split(fixed[i], entries[i], best_limit);
    return K;
}

// Units of a work list without an active list: in item order, and where
// items are split, the most expensive first.
void pack_units(const std::vector<int>& item_b0, const std::vector<int>& item_b1, const std::vector<int64_t>& entries,
                bool fp64, FastTranspose& t, MetaPack& mp)
{
    const size_t n = entries.size();
    std::vector<float> fixed(n), en(n);
    for (size_t i = 0; i < n; i++) {
        fixed[i] = unit_fixed(fp64, item_b1[i] - item_b0[i]);
        en[i] = static_cast<float>(entries[i]);
    }
    const std::vector<int> K = plan_splits(fixed.data(), en.data(), n, 1);
    std::vector<int> order(n);
    for (size_t i = 0; i < n; i++) order[i] = static_cast<int>(i);
    if (n < static_cast<size_t>(kPlanWaves) * sm_count())
        std::stable_sort(order.begin(), order.end(), [&](int a, int b) {
            return fixed[a] + en[a] / static_cast<float>(K[a]) > fixed[b] + en[b] / static_cast<float>(K[b]);
        });
    std::vector<uint32_t> units;
    for (int i : order)
        for (int k = 0; k < K[i]; k++) units.push_back(unit_pack(i, k, K[i]));
    t.nunits = static_cast<int>(units.size());
    mp.add(units, &t.units);
}

// Builds the work list of one A'y variant from the entry counts per (block,
// chunk): super-chunks of at most per_sc chunks of columns, each split into
// block ranges so that items carry about equal numbers of entries.
cas_status build_items(const FastGeometry& g, const std::vector<int64_t>& entries_bc, int per_sc, int items_per_sm,
                       bool range_major, bool pack, bool persistent, size_t elem, FastTranspose& t)
{
    t.per_sc = per_sc;
    t.range_major = range_major;
    t.items_per_sm = items_per_sm;
    t.pack = pack;
    t.persistent = persistent;
    const Pieces pc = pack_chunks(g, per_sc * kChunkCols, pack);
    MetaPack mp;
    pack_pieces(pc, t, mp);
    const int nsc = t.nsc;
    // entries per (problem, super-chunk); items never span problems
    std::vector<int64_t> sc_entries(static_cast<size_t>(g.nprob) * nsc, 0);
    int64_t total = 0;
    for (int q = 0; q < g.nprob; q++)
        for (int64_t b = g.pblk0[q]; b < g.pblk0[q + 1]; b++)
            for (int ch = 0; ch < g.nchunks; ch++) {
                sc_entries[static_cast<size_t>(q) * nsc + pc.chunk_sc[ch]] += entries_bc[b * g.nchunks + ch];
                total += entries_bc[b * g.nchunks + ch];
            }
    const int64_t target_items = static_cast<int64_t>(sm_count()) * items_per_sm;
    const double per_item = std::max<double>(1.0, static_cast<double>(total) / target_items);
    std::vector<int> item_sc, item_b0, item_b1, sc_item0;
    std::vector<int64_t> item_part;
    int64_t part_elems = 0;
    if (range_major && g.nprob == 1 && nsc > 1 && g.nblocks > 0) {
        // One fit: every super-chunk shares one partition of the blocks into
        // ranges, and the items run range by range (within a range the
        // heaviest super-chunks first), so that the CTAs at work at one time
        // stage the y slices of the same few blocks: a slice comes from HBM
        // once and from L2 for the other super-chunks.  Items of one
        // super-chunk stay contiguous in the partial buffer, in range order,
        // which is the order its column sums add them in.
        const int64_t nb = g.pblk0[1] - g.pblk0[0];
        const int64_t nr = std::max<int64_t>(1, std::min<int64_t>(nb, (target_items + nsc - 1) / nsc));
        std::vector<int> order(nsc);
        for (int sc = 0; sc < nsc; sc++) order[sc] = sc;
        std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return sc_entries[a] > sc_entries[b]; });
        // partials in item order; each super-chunk's items listed for the
        // column sums in range order
        std::vector<std::vector<int64_t>> by_sc(nsc);
        for (int64_t r = 0; r < nr; r++)
            for (int sc : order) {
                item_sc.push_back(sc);
                item_b0.push_back(static_cast<int>(g.pblk0[0] + nb * r / nr));
                item_b1.push_back(static_cast<int>(g.pblk0[0] + nb * (r + 1) / nr));
                item_part.push_back(part_elems);
                by_sc[sc].push_back(part_elems);
                part_elems += pc.sc_width[sc];
            }
        std::vector<int64_t> part_by_sc;
        part_by_sc.reserve(item_sc.size());
        for (int sc = 0; sc < nsc; sc++) {
            sc_item0.push_back(static_cast<int>(part_by_sc.size()));
            part_by_sc.insert(part_by_sc.end(), by_sc[sc].begin(), by_sc[sc].end());
        }
        sc_item0.push_back(static_cast<int>(part_by_sc.size()));
        t.nitems = static_cast<int>(item_sc.size());
        const std::vector<int64_t> ie = item_entries(g, entries_bc, pc, item_sc, item_b0, item_b1);
        t.max_item_entries = ie.empty() ? 0 : *std::max_element(ie.begin(), ie.end());
        pack_units(item_b0, item_b1, ie, elem == sizeof(double), t, mp);
        mp.add(item_sc, &t.item_sc);
        mp.add(item_b0, &t.item_b0);
        mp.add(item_b1, &t.item_b1);
        mp.add(item_part, &t.item_part);
        mp.add(sc_item0, &t.sc_item0);
        mp.add(part_by_sc, &t.sc_part);
        mp.add(std::vector<int>{0, 0}, &t.ctr);
        CAS_TRY(mp.upload(&t.meta));
        CAS_CUDA(dmalloc(&t.partial, elem * std::max<int64_t>(part_elems, 1)));
        return CAS_OK;
    }
    for (int q = 0; q < g.nprob; q++) {
        const int64_t qb0 = g.pblk0[q], qnb = g.pblk0[q + 1] - g.pblk0[q];
        for (int sc = 0; sc < nsc; sc++) {
            sc_item0.push_back(static_cast<int>(item_sc.size()));
            if (qnb == 0) continue;
            int64_t n = static_cast<int64_t>(std::llround(sc_entries[static_cast<size_t>(q) * nsc + sc] / per_item));
            // batched layouts: at most kBatchItemBlocks blocks per item, and
            // one block per item for problems of at most kBatchSmallBlocks
            // blocks (the small stages that iterate longest), so that a
            // problem left alone (or with few others) still has short units:
            // a unit's blocks run one after another in one CTA
            if (g.nprob > 1)
                n = std::max<int64_t>(n, qnb <= kBatchSmallBlocks ? qnb
                                                                  : (qnb + kBatchItemBlocks - 1) / kBatchItemBlocks);
            n = std::max<int64_t>(1, std::min<int64_t>(n, qnb));
            for (int64_t i = 0; i < n; i++) {
                item_sc.push_back(sc);
                item_b0.push_back(static_cast<int>(qb0 + qnb * i / n));
                item_b1.push_back(static_cast<int>(qb0 + qnb * (i + 1) / n));
                item_part.push_back(part_elems);
                part_elems += pc.sc_width[sc];
            }
        }
    }
    sc_item0.push_back(static_cast<int>(item_sc.size()));
    t.nitems = static_cast<int>(item_sc.size());
    const std::vector<int64_t> ie = item_entries(g, entries_bc, pc, item_sc, item_b0, item_b1);
    t.max_item_entries = ie.empty() ? 0 : *std::max_element(ie.begin(), ie.end());
    pack_units(item_b0, item_b1, ie, elem == sizeof(double), t, mp);
    if (g.nprob > 1) {
        std::vector<float> grp_entries(static_cast<size_t>(g.nprob) * nsc, 0.0f);
        std::vector<int> grp_blocks(grp_entries.size(), 0);
        for (size_t grp = 0; grp < grp_entries.size(); grp++)
            for (int i = sc_item0[grp]; i < sc_item0[grp + 1]; i++) {
                grp_entries[grp] = std::max(grp_entries[grp], static_cast<float>(ie[i]));
                grp_blocks[grp] = std::max(grp_blocks[grp], item_b1[i] - item_b0[i]);
            }
        mp.add(grp_entries, &t.grp_entries);
        mp.add(grp_blocks, &t.grp_blocks);
    }
    mp.add(item_sc, &t.item_sc);
    mp.add(item_b0, &t.item_b0);
    mp.add(item_b1, &t.item_b1);
    mp.add(item_part, &t.item_part);
    mp.add(sc_item0, &t.sc_item0);
    mp.add(item_part, &t.sc_part);  // items are listed super-chunk by super-chunk already
    mp.add(std::vector<int>{0, 0}, &t.ctr);
    CAS_TRY(mp.upload(&t.meta));
    CAS_CUDA(dmalloc(&t.partial, elem * std::max<int64_t>(part_elems, 1)));
    return CAS_OK;
}

// Work list of one item per (block, chunk), block-major, for adjoints over a
// block range (minibatches): item b * nchunks + ch, one piece per chunk;
// partial offsets give the layout [block][global column] relative to the
// first item of the range.
cas_status build_block_items(const FastGeometry& g, FastTranspose& t)
{
    t.per_sc = 1;
    Pieces pc;
    for (int ch = 0; ch < g.nchunks; ch++) {
        pc.sc_piece0.push_back(ch);
        pc.sc_width.push_back(chunk_width(g, ch));
        pc.pat.push_back(pattern_of_chunk(g, ch));
        pc.ch0.push_back(ch);
        pc.ch1.push_back(ch + 1);
        pc.acc.push_back(0);
        pc.chunk_sc.push_back(ch);
        pc.chunk_acc.push_back(0);
    }
    pc.sc_piece0.push_back(g.nchunks);
    MetaPack mp;
    pack_pieces(pc, t, mp);
    const int64_t n = g.nblocks * g.nchunks;
    t.nitems = static_cast<int>(n);
    std::vector<int> isc(n), ib0(n), ib1(n);
    std::vector<int64_t> ipart(n);
    for (int64_t b = 0; b < g.nblocks; b++)
        for (int ch = 0; ch < g.nchunks; ch++) {
            const int p = pattern_of_chunk(g, ch);
            const int64_t i = b * g.nchunks + ch;
            isc[i] = ch;
            ib0[i] = static_cast<int>(b);
            ib1[i] = static_cast<int>(b + 1);
            ipart[i] = b * g.cols + g.off[p] + static_cast<int64_t>(ch - g.chunk0[p]) * kChunkCols;
        }
    mp.add(isc, &t.item_sc);
    mp.add(ib0, &t.item_b0);
    mp.add(ib1, &t.item_b1);
    mp.add(ipart, &t.item_part);
    return mp.upload(&t.meta);
}

TView tview(const FastTranspose& t)
{
    TView v;
    v.npieces = t.npieces;
    v.item_sc = t.item_sc;
    v.item_b0 = t.item_b0;
    v.item_b1 = t.item_b1;
    v.item_part = t.item_part;
    v.sc_piece0 = t.sc_piece0;
    v.piece_pat = t.piece_pat;
    v.piece_ch0 = t.piece_ch0;
    v.piece_ch1 = t.piece_ch1;
    v.piece_acc = t.piece_acc;
    v.units = t.units;
    v.nunits = t.nunits;
    v.nsc = t.nsc;
    return v;
}

template <typename T>
const FastTranspose& transpose_of(const FastLayout& f)
{
    return sizeof(T) == 4 ? f.t32 : f.t64;
}

template <typename T>
size_t spmv_t_smem(int per_sc)
{
    return sizeof(T) * (static_cast<size_t>(kChunkCols) * per_sc + kBlockRows);
}

void free_transpose(FastTranspose& t)
{
    dfree(t.meta);
    dfree(t.partial);
    t = FastTranspose{};
}

// Opt-in shared memory for every product kernel (set outside any stream
// capture, at the first build on each device).
cas_status fast_set_attributes_now();
cas_status fast_set_attributes()
{
    static std::mutex mu;
    static std::vector<char> done;
    int dev = 0;
    CAS_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lk(mu);
    if (static_cast<int>(done.size()) <= dev) done.resize(dev + 1, 0);
    if (done[dev]) return CAS_OK;
    CAS_TRY(fast_set_attributes_now());
    done[dev] = 1;
    return CAS_OK;
}
cas_status fast_set_attributes_now()
{
    const int tbl = kTableBytes;
    const int t32 = static_cast<int>(spmv_t_smem<float>(kMaxSc));
    const int t64 = static_cast<int>(spmv_t_smem<double>(1));
    const auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
    CAS_CUDA(cudaFuncSetAttribute(fast_spmv_table_kernel<float, float, 0, true>, attr, tbl));
    CAS_CUDA(cudaFuncSetAttribute(fast_spmv_table_kernel<float, float, 0, false>, attr, tbl));
    CAS_CUDA(cudaFuncSetAttribute(fast_spmv_table_kernel<float, float, 1, true>, attr, tbl));
    CAS_CUDA(cudaFuncSetAttribute(fast_spmv_table_kernel<float, float, 1, false>, attr, tbl));
    CAS_CUDA(cudaFuncSetAttribute(fast_spmv_table_kernel<float, float, 2, true>, attr, tbl));
    CAS_CUDA(cudaFuncSetAttribute(fast_spmv_table_kernel<float, float, 2, false>, attr, tbl));
    CAS_CUDA(cudaFuncSetAttribute(fast_spmv_table_kernel<double, double, 0, true>, attr, tbl));
    CAS_CUDA(cudaFuncSetAttribute(fast_spmv_table_kernel<double, double, 0, false>, attr, tbl));
    CAS_CUDA(cudaFuncSetAttribute(fast_spmv_table_kernel<double, double, 1, true>, attr, tbl));
    CAS_CUDA(cudaFuncSetAttribute(fast_spmv_table_kernel<double, double, 1, false>, attr, tbl));
    CAS_CUDA(cudaFuncSetAttribute(fast_spmv_table_kernel<double, double, 2, true>, attr, tbl));
    CAS_CUDA(cudaFuncSetAttribute(fast_spmv_table_kernel<double, double, 2, false>, attr, tbl));
    CAS_CUDA(cudaFuncSetAttribute(fast_spmv_table_kernel<double, float, 0, true>, attr, tbl));
    CAS_CUDA(cudaFuncSetAttribute(fast_spmv_table_kernel<double, float, 0, false>, attr, tbl));
    CAS_CUDA(cudaFuncSetAttribute(fast_spmv_table_kernel<double, float, 1, true>, attr, tbl));
    CAS_CUDA(cudaFuncSetAttribute(fast_spmv_table_kernel<double, float, 1, false>, attr, tbl));
    CAS_CUDA(cudaFuncSetAttribute(fast_spmv_table_kernel<double, float, 2, true>, attr, tbl));
    CAS_CUDA(cudaFuncSetAttribute(fast_spmv_table_kernel<double, float, 2, false>, attr, tbl));
    CAS_CUDA(cudaFuncSetAttribute(fast_spmv_t_kernel<float>, attr, t32));
    CAS_CUDA(cudaFuncSetAttribute(fast_spmv_t_kernel<double>, attr, t64));
    return CAS_OK;
}

// ---------------------------------------------------------------------------
// Build-time autotuner of the FP32 A'y schedule.  Every candidate work list
// is built and timed (partials + column sums, CUDA events, one warm-up
// launch) on this layout; the fastest is kept and remembered per geometry
// for the rest of the process, so later builds of the same shape skip the
// timing.  CAS_ATY_SCHEDULE="chunks,range_major,items_per_sm,pack,persistent"
// forces a schedule.
// ---------------------------------------------------------------------------
struct Sched {
    int per_sc;
    bool range_major;
    int ips;
    bool pack;
    bool persistent;
};
constexpr Sched kSchedDefault = {4, false, 2, false, false};
constexpr Sched kSchedCandidates[] = {
    {4, false, 2, false, false}, {4, false, 3, false, false}, {4, false, 2, true, true}, {4, false, 4, true, true},
    {4, false, 4, false, true},  {2, false, 4, true, true},   {4, false, 6, false, true}, {4, true, 2, false, false},
    {4, true, 4, false, true},   {4, true, 6, false, true},   {4, true, 4, true, true},   {2, true, 4, true, true}};
static_assert(sizeof(kSchedCandidates) / sizeof(Sched) <= kMaxTune, "tune table");
constexpr int64_t kTuneMinBlocks = 64;  // smaller layouts take the default schedule

std::mutex g_tune_mu;
std::map<std::string, Sched> g_tune_cache;

std::string tune_key(const FastGeometry& g)
{
    std::string k = std::to_string(g.k) + "/" + std::to_string(g.nblocks) + "/" + std::to_string(g.rows);
    for (int p = 0; p < g.npat; p++) k += "/" + std::to_string(g.space[p]) + "x" + std::to_string(g.slots[p]);
    for (int q = 0; q <= g.nprob; q++) k += ":" + std::to_string(g.pblk0[q]);
    return k;
}

bool valid_sched(const Sched& c)
{
    return c.per_sc >= 1 && c.per_sc <= kMaxSc && c.ips >= 1 && c.ips <= 16;
}

cas_status tune_transpose(FastLayout& f, const std::vector<int64_t>& entries, cudaStream_t s)
{
    const FastGeometry& g = f.g;
    f.ntune = 0;
    f.tune_cached = 0;
    auto build = [&](const Sched& c) {
        return build_items(g, entries, c.per_sc, c.ips, c.range_major, c.pack, c.persistent, sizeof(float), f.t32);
    };
    if (const char* env = std::getenv("CAS_ATY_SCHEDULE")) {
        int a = 0, b = 0, c = 0, d = 0, e = 0;
        const int n = std::sscanf(env, "%d,%d,%d,%d,%d", &a, &b, &c, &d, &e);
        const Sched forced{a, b != 0, c, d != 0, e != 0};
        CAS_REQUIRE(n == 5 && valid_sched(forced), CAS_ERR_INVALID_ARGUMENT,
                    "CAS_ATY_SCHEDULE must be \"chunks,range_major,items_per_sm,pack,persistent\" within limits");
        return build(forced);
    }
    if (g.nblocks < kTuneMinBlocks) return build(kSchedDefault);
    const std::string key = tune_key(g);
    {
        std::lock_guard<std::mutex> lk(g_tune_mu);
        auto it = g_tune_cache.find(key);
        if (it != g_tune_cache.end()) {
            f.tune_cached = 1;
            return build(it->second);
        }
    }
    float* y = nullptr;
    float* x = nullptr;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    cas_status st = CAS_OK;
    auto fail = [&](cudaError_t e) {
        if (e != cudaSuccess && st == CAS_OK) {
            set_error(std::string("autotuner: ") + cudaGetErrorString(e));
            st = CAS_ERR_CUDA;
        }
    };
    fail(dmalloc(&y, sizeof(float) * g.rows));
    fail(dmalloc(&x, sizeof(float) * std::max<int64_t>(g.cols, 1)));
    fail(cudaEventCreate(&e0));
    fail(cudaEventCreate(&e1));
    if (st == CAS_OK) fail(cudaMemsetAsync(y, 0, sizeof(float) * g.rows, s));
    Sched best = kSchedDefault;
    float best_ms = 1e30f;
    for (const Sched& c : kSchedCandidates) {
        if (st != CAS_OK) break;
        st = build(c);
        if (st == CAS_OK) st = fast_spmv_t<float>(f, y, x, s);  // warm-up
        if (st == CAS_OK) fail(cudaEventRecord(e0, s));
        for (int r = 0; r < 2 && st == CAS_OK; r++) st = fast_spmv_t<float>(f, y, x, s);
        if (st == CAS_OK) fail(cudaEventRecord(e1, s));
        if (st == CAS_OK) fail(cudaEventSynchronize(e1));
        float ms = 0;
        if (st == CAS_OK) fail(cudaEventElapsedTime(&ms, e0, e1));
        free_transpose(f.t32);
        if (st != CAS_OK) break;
        ms *= 0.5f;
        f.tune[f.ntune++] =
            FastTuneEntry{c.per_sc, c.range_major ? 1 : 0, c.ips, c.pack ? 1 : 0, c.persistent ? 1 : 0, ms};
        if (ms < best_ms) {
            best_ms = ms;
            best = c;
        }
    }
    dfree(y);
    dfree(x);
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    if (st != CAS_OK) return st;
    {
        std::lock_guard<std::mutex> lk(g_tune_mu);
        g_tune_cache[key] = best;
    }
    return build(best);
}

// The patterns whose slices of x the table kernel keeps in shared memory: by
// entries a row per column, while they fit, and of those the ones that a CTA
// gathers from as often as the slice has bytes between two stagings (one per
// CTA, and one more per problem of a batch), or half as often for a slice of up
// to kTableSmall, which leaves L1 to the others.  Below that, staging takes
// longer than its gathers save: one pattern of 29,646 columns and 4 slots, FP32,
// us staged and not, 49 blocks 39 and 29, 200 66 and 59, 300 83 and 80; five
// reference patterns with 65 KB for 10 slots, 49 blocks 56 and 50, 80 68 and 70.
// A slice of 26 KB with 2 slots of eight reference patterns, FP64, 92 blocks,
// saves 4 of 95 us.
constexpr int kTableSmall = 32 * 1024;

FastTable table_plan(const FastGeometry& g, size_t elem)
{
    FastTable t;
    std::vector<int> order(g.npat);
    for (int p = 0; p < g.npat; p++) order[p] = p;
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) {
        return static_cast<int64_t>(g.slots[a]) * g.space[b] > static_cast<int64_t>(g.slots[b]) * g.space[a];
    });
    for (int p = 0; p < kMaxFastPatterns; p++) t.base[p] = -1;
    const int room = static_cast<int>(kTableBytes / elem);
    const int64_t rows = g.rows / (sm_count() + g.nprob - 1);  // of a staging
    for (int p : order) {
        const int64_t bytes = static_cast<int64_t>(elem) * g.space[p];
        if (t.elems + g.space[p] <= room && rows * g.slots[p] >= (bytes <= kTableSmall ? bytes / 2 : bytes)) {
            t.base[p] = t.elems;
            t.elems += g.space[p];
        }
    }
    return t;
}

}  // namespace

bool fast_supported(const PatternSet& ps)
{
    if (ps.indexers.empty() || static_cast<int>(ps.indexers.size()) > kMaxFastPatterns) return false;
    for (const IndexerInfo& in : ps.indexers) {
        if (in.space > 65536) return false;
        if (in.order != 1 && in.order != 2 && in.order != 4 && in.order != 8) return false;
    }
    // 65536 columns a pattern keep every digit list within the tile indexer's
    for (const Instance& in : ps.instances)
        if (in.n0 > kTileSquares || in.n1 > kTileSquares || in.n2 > kTileSquares) return false;
    return true;
}

void fast_free(FastLayout& f)
{
    dfree(f.a16);
    dfree(f.g32);
    dfree(f.sub_start);
    free_transpose(f.t32);
    free_transpose(f.t64);
    free_transpose(f.tb);
    dfree(f.eval_partial);
    dfree(f.eval_dscore);
    dfree(f.eval_red);
    dfree(f.eval_ctr);
    f = FastLayout{};
}

cas_status fast_build(const DevicePatterns& dp, const PatternSet& ps, const uint64_t* d_pos, int64_t rows,
                      const int64_t* prob_rows, int nprob, uint64_t* diag_int, FastLayout& f, cudaStream_t s,
                      const PositionChunks* chunks)
{
    cas::NvtxRange nvtx_range("blocked layout build");
    CAS_REQUIRE(fast_supported(ps), CAS_ERR_INVALID_ARGUMENT, "pattern set does not fit the blocked layout");
    CAS_REQUIRE(nprob >= 1 && nprob <= kMaxProblems, CAS_ERR_INVALID_ARGUMENT,
                "blocked layout: 1 to 64 problems per batch");
    CAS_TRY(fast_set_attributes());
    FastGeometry& g = f.g;
    g = FastGeometry{};
    g.npat = static_cast<int>(ps.indexers.size());
    g.k = dp.k;
    g.rows = rows;
    g.nprob = nprob;
    g.pcols = ps.cols;
    g.cols = ps.cols * nprob;
    // problem table: rows and whole blocks of each problem
    int64_t r0 = 0, b0 = 0;
    for (int q = 0; q < nprob; q++) {
        const int64_t rq = prob_rows ? prob_rows[q] : rows;
        CAS_REQUIRE(rq >= 0, CAS_ERR_INVALID_ARGUMENT, "blocked layout: negative problem size");
        g.prow0[q] = r0;
        g.pblk0[q] = static_cast<int>(b0);
        r0 += rq;
        b0 += (rq + kBlockRows - 1) / kBlockRows;
    }
    g.prow0[nprob] = r0;
    g.pblk0[nprob] = static_cast<int>(b0);
    CAS_REQUIRE(r0 == rows, CAS_ERR_SIZE_MISMATCH, "blocked layout: problem sizes do not add up to the rows");
    g.nblocks = b0;
    int slot = 0, chunk = 0;
    for (int p = 0; p < g.npat; p++) {
        g.slot0[p] = slot;
        g.slots[p] = ps.indexers[p].order;
        g.off[p] = ps.indexers[p].offset;
        g.space[p] = static_cast<int>(ps.indexers[p].space);
        g.chunk0[p] = chunk;
        slot += g.slots[p];
        chunk += (g.space[p] + kChunkCols - 1) / kChunkCols;
    }
    g.nchunks = chunk;
    f.tab32 = table_plan(g, sizeof(float));
    f.tab64 = table_plan(g, sizeof(double));
    CAS_REQUIRE(g.total_elems() < 0xFFFFFFFFLL, CAS_ERR_INVALID_ARGUMENT,
                "blocked layout: 2^32 or more entries (with block padding) are not supported");
    const int64_t elems = std::max<int64_t>(g.total_elems(), 8);
    CAS_CUDA(dmalloc(&f.a16, sizeof(uint16_t) * elems));
    CAS_CUDA(dmalloc(&f.g32, sizeof(uint32_t) * elems));
    const int64_t nsub = g.nblocks * g.nchunks * kSubPerChunk;
    CAS_CUDA(dmalloc(&f.sub_start, sizeof(uint32_t) * std::max<int64_t>(nsub, 1)));
    if (rows > 0) {
        // one launch over all rows, or one per arriving chunk behind its copy
        // (and one over the rows past the last chunk)
        auto index_rows = [&](int64_t r0, int64_t r1) -> cas_status {
            if (r1 <= r0) return CAS_OK;
            const int64_t steps = (r1 - r0 + kTileThreads - 1) / kTileThreads;  // a CTA step: one row a thread
            const dim3 grid(static_cast<unsigned>(std::min<int64_t>(steps, static_cast<int64_t>(sm_count()) * 3)),
                            static_cast<unsigned>(dp.chunks));
            { fast_index_kernel<<<grid, kTileThreads, dp.tile_bytes, s>>>(
                dp.tiles, dp.units, dp.chunk_unit, dp.chunk_tile, dp.tables,
                reinterpret_cast<const ulonglong2*>(d_pos), g, f.a16, r0, r1); cas::count_launch(); }
            CAS_CHECK_LAUNCH();
            return CAS_OK;
        };
        int64_t r0 = 0;
        for (int c = 0; chunks && c < chunks->n; c++) {
            const int64_t r1 = std::min(chunks->row_end[c], rows);
            CAS_CUDA(cudaStreamWaitEvent(s, chunks->ready[c], 0));
            CAS_TRY(index_rows(r0, r1));
            r0 = std::max(r0, r1);
        }
        CAS_TRY(index_rows(r0, rows));
        const int64_t groups = g.nblocks * g.npat;
        const unsigned sgrid =
            static_cast<unsigned>(std::min<int64_t>(groups, static_cast<int64_t>(sm_count()) * kSortCtasPerSm));
        uint32_t* scratch = nullptr;
        CAS_CUDA(dmalloc(&scratch, sizeof(uint32_t) * kBlockRows * 8 * sgrid));
        { fast_sort_kernel<<<sgrid, kSortThreads, 0, s>>>(g, f.a16, f.g32, scratch); cas::count_launch(); }
        CAS_CHECK_LAUNCH();
        dfree(scratch);
        { fast_sub_kernel<<<fgrid(nsub, 256), 256, 0, s>>>(g, f.g32, f.sub_start); cas::count_launch(); }
        CAS_CHECK_LAUNCH();
    }
    // entries per (block, chunk) -> work items
    std::vector<int64_t> entries(static_cast<size_t>(g.nblocks * g.nchunks), 0);
    if (!entries.empty() && rows > 0) {
        std::vector<uint32_t> ce(entries.size());
        uint32_t* d_ce = nullptr;
        CAS_CUDA(dmalloc(&d_ce, sizeof(uint32_t) * ce.size()));
        { fast_chunk_entries_kernel<<<fgrid(static_cast<int64_t>(ce.size()), 256), 256, 0, s>>>(g, f.sub_start, d_ce); cas::count_launch(); }
        CAS_CHECK_LAUNCH();
        CAS_CUDA(cudaMemcpyAsync(ce.data(), d_ce, sizeof(uint32_t) * ce.size(), cudaMemcpyDeviceToHost, s));
        CAS_CUDA(cudaStreamSynchronize(s));
        dfree(d_ce);
        for (size_t i = 0; i < ce.size(); i++) entries[i] = ce[i];
    }
    for (int ch = 0; ch < g.nchunks; ch++) {
        double sum = 0;
        for (int64_t b = 0; b < g.nblocks; b++) sum += static_cast<double>(entries[b * g.nchunks + ch]);
        f.chunk_entries[ch] = g.nblocks ? static_cast<float>(sum / static_cast<double>(g.nblocks)) : 0.0f;
    }
    if (g.nblocks > 0) {
        CAS_TRY(tune_transpose(f, entries, s));
        // FP64 items hold one chunk, so the y slices would be read once per
        // chunk: always range by range
        CAS_TRY(build_items(g, entries, 1, 2, true, true, false, sizeof(double), f.t64));
        if (g.nprob == 1) CAS_TRY(build_block_items(g, f.tb));  // evaluator minibatches: single fits only
        if (diag_int && rows > 0) CAS_TRY(fast_diag(f, diag_int, s));
    } else {
        // no items, but the column sums of a solve read the lists' tables
        const Sched& c = kSchedDefault;
        CAS_TRY(build_items(g, entries, c.per_sc, c.ips, c.range_major, c.pack, c.persistent, sizeof(float), f.t32));
        CAS_TRY(build_items(g, entries, 1, 2, false, true, false, sizeof(double), f.t64));
    }
    return CAS_OK;
}

cas_status fast_diag(const FastLayout& f, uint64_t* diag, cudaStream_t s)
{
    const int64_t groups = f.g.nblocks * f.g.npat;
    if (f.g.cols == 0) return CAS_OK;
    if (groups == 0) {
        CAS_CUDA(cudaMemsetAsync(diag, 0, sizeof(uint64_t) * f.g.cols, s));
        return CAS_OK;
    }
    const unsigned grid = std::min<unsigned>(static_cast<unsigned>(groups), sm_count() * 8);
    int max_slots = 0;
    for (int p = 0; p < f.g.npat; p++) max_slots = std::max(max_slots, f.g.slots[p]);
    // a column's count inside an item is at most the item's entries;
    // CAS_DIAG_FROM_G32=1 takes the direct count whatever the items
    const char* direct = std::getenv("CAS_DIAG_FROM_G32");
    const bool exact32 = f.t32.nitems > 0 && f.t32.partial && !(direct && std::strcmp(direct, "1") == 0) &&
                         f.t32.max_item_entries < (int64_t(1) << 24);
    if (!exact32) {
        CAS_CUDA(cudaMemsetAsync(diag, 0, sizeof(uint64_t) * f.g.cols, s));
        { fast_diag_kernel<<<grid, 256, 0, s>>>(f.g, f.g32, diag); cas::count_launch(); }
        CAS_CHECK_LAUNCH();
        return CAS_OK;
    }
    CAS_TRY(fast_spmv_t_partials<float>(f, nullptr, nullptr, s));  // no y: ones
    { fast_count_kernel<<<fgrid(f.g.cols, 256), 256, 0, s>>>(fast_cols<float>(f), static_cast<const float*>(f.t32.partial), diag); cas::count_launch(); }
    CAS_CHECK_LAUNCH();
    const int stretches = (kBlockRows * max_slots + kRepeatRounds * kRound - 1) / (kRepeatRounds * kRound);
    const int64_t warps = groups * stretches;
    const unsigned rgrid = static_cast<unsigned>(std::max<int64_t>(1, std::min<int64_t>((warps + 7) / 8, sm_count() * 8)));
    { fast_repeat_kernel<<<rgrid, 256, 0, s>>>(f.g, f.g32, diag, stretches); cas::count_launch(); }
    CAS_CHECK_LAUNCH();
    return CAS_OK;
}

static bool all_slots_8(const FastGeometry& g)
{
    bool all8 = true;
    for (int p = 0; p < g.npat; p++) all8 = all8 && g.slots[p] == 8;
    return all8;
}

int fast_ax_parts(int64_t nblocks)
{
    return static_cast<int>(nblocks <= kAxDirectBlocks ? nblocks * kAxSplitMax : sm_count());
}

template <typename T, typename Y>
cas_status fast_spmv(const FastLayout& f, const T* x, Y* y, const double* b, const double* coef, double* part,
                     int* done_flag, int mode, cudaStream_t s, int* n_parts, const int* pdone, const FastActive* act)
{
    const FastGeometry& g = f.g;
    if (n_parts) *n_parts = fast_ax_parts(g.nblocks);
    if (g.nblocks == 0) return CAS_OK;
    const bool all8 = all_slots_8(g);
    if (act || g.nblocks <= kAxDirectBlocks) {
        const unsigned grid = static_cast<unsigned>(std::min<int64_t>(g.nblocks * kAxSplitMax, 4LL * sm_count()));
        auto kd = all8 ? (mode == 0 ? fast_spmv_direct_kernel<T, Y, 0, true>
                                    : (mode == 1 ? fast_spmv_direct_kernel<T, Y, 1, true>
                                                 : fast_spmv_direct_kernel<T, Y, 2, true>))
                       : (mode == 0 ? fast_spmv_direct_kernel<T, Y, 0, false>
                                    : (mode == 1 ? fast_spmv_direct_kernel<T, Y, 1, false>
                                                 : fast_spmv_direct_kernel<T, Y, 2, false>));
        { kd<<<grid, kAxDirectRows, 0, s>>>(g, f.a16, x, y, b, coef, part, done_flag, pdone, act); cas::count_launch(); }
        CAS_CHECK_LAUNCH();
    }
    if (g.nblocks > kAxDirectBlocks) {
        const FastTable& tab = sizeof(T) == 4 ? f.tab32 : f.tab64;
        auto kt = all8 ? (mode == 0 ? fast_spmv_table_kernel<T, Y, 0, true>
                                    : (mode == 1 ? fast_spmv_table_kernel<T, Y, 1, true>
                                                 : fast_spmv_table_kernel<T, Y, 2, true>))
                       : (mode == 0 ? fast_spmv_table_kernel<T, Y, 0, false>
                                    : (mode == 1 ? fast_spmv_table_kernel<T, Y, 1, false>
                                                 : fast_spmv_table_kernel<T, Y, 2, false>));
        { kt<<<sm_count(), kAxThreads, sizeof(T) * static_cast<size_t>(tab.elems), s>>>(
            g, tab, f.a16, x, y, b, coef, part, done_flag, pdone, act); cas::count_launch(); }
        CAS_CHECK_LAUNCH();
    }
    return CAS_OK;
}

template <typename T>
cas_status fast_spmv_t_partials(const FastLayout& f, const T* y, int* done_flag, cudaStream_t s, const int* pdone,
                                const FastActive* act)
{
    const FastTranspose& t = transpose_of<T>(f);
    if (t.nitems == 0) return CAS_OK;
    const size_t smem = spmv_t_smem<T>(t.per_sc);
    const bool persistent = t.persistent || act;
    const unsigned grid = static_cast<unsigned>(
        act ? sm_count() : (persistent ? std::min(t.nunits, sm_count()) : t.nunits));
    { fast_spmv_t_kernel<T><<<grid, kFastThreads, smem, s>>>(f.g, tview(t), f.g32, f.sub_start, y,
                                                             static_cast<T*>(t.partial), done_flag, 0, 0,
                                                             persistent ? t.ctr : nullptr, pdone, act,
                                                             BlockUnits{}); cas::count_launch(); }
    CAS_CHECK_LAUNCH();
    return CAS_OK;
}

template <typename T>
FastPlanView fast_plan_view(const FastLayout& f)
{
    const FastTranspose& t = transpose_of<T>(f);
    const bool one = f.g.nprob == 1;
    return FastPlanView{one ? t.units : nullptr, one ? t.nunits : 0, t.sc_item0, t.grp_entries, t.grp_blocks, t.nsc,
                        sizeof(T) == 8};
}

int64_t fast_plan_room(const FastLayout& f)
{
    return std::max<int64_t>(std::max(f.t32.nitems, f.t64.nitems),
                             static_cast<int64_t>(kPlanWaves) * sm_count() * kAtySplitMax);
}

template <typename T>
FastCols fast_cols(const FastLayout& f)
{
    const FastTranspose& t = transpose_of<T>(f);
    FastCols c;
    c.g = f.g;
    c.nsc = t.nsc;
    c.chunk_sc = t.chunk_sc;
    c.chunk_acc = t.chunk_acc;
    c.sc_item0 = t.sc_item0;
    c.sc_part = t.sc_part;
    return c;
}

template <typename T>
cas_status fast_spmv_t(const FastLayout& f, const T* y, T* x, cudaStream_t s)
{
    CAS_TRY(fast_spmv_t_partials<T>(f, y, nullptr, s));
    const FastTranspose& t = transpose_of<T>(f);
    if (f.g.cols == 0) return CAS_OK;
    if (t.nitems == 0) {
        CAS_CUDA(cudaMemsetAsync(x, 0, sizeof(T) * f.g.cols, s));
        return CAS_OK;
    }
    { fast_col_sum_kernel<T><<<fgrid(f.g.cols, 256), 256, 0, s>>>(fast_cols<T>(f), static_cast<const T*>(t.partial), x); cas::count_launch(); }
    CAS_CHECK_LAUNCH();
    return CAS_OK;
}

static bool eval_resident(int64_t n) { return n <= kEvalResident * sm_count(); }
static unsigned eval_grid(int64_t n)
{
    return static_cast<unsigned>(std::min<int64_t>(
        {(n + kEvalRows - 1) / kEvalRows, static_cast<int64_t>(kEvalCtas) * sm_count(), int64_t(kEvalRedMax)}));
}

cas_status fast_eval_forward(const FastLayout& f, int64_t row0, int64_t row1, const float* w, float* score,
                             cudaStream_t s)
{
    if (row1 <= row0) return CAS_OK;
    const int64_t n = row1 - row0;
    auto kernel = !all_slots_8(f.g) ? fast_rows_forward_kernel<false, 1>
                                    : (eval_resident(n) ? fast_rows_forward_kernel<true, kRowPatterns>
                                                        : fast_rows_forward_kernel<true, 1>);
    { kernel<<<eval_grid(n), kEvalRows, 0, s>>>(f.g, f.a16, w, row0, row1, score); cas::count_launch(); }
    CAS_CHECK_LAUNCH();
    return CAS_OK;
}

// The evaluator's per-call buffers for adjoints over nb blocks (grown, never
// shrunk).  A call made while `s` is capturing marks them as held by a CUDA
// graph: from then on a call that would grow them (and so free the buffers
// the graph's kernels use) is refused, captured or not, and so is growing
// during a capture.  Growing waits for the whole device, since eager work
// on other streams may still use the old buffers.
static cas_status eval_buffers(FastLayout& f, int64_t nb, cudaStream_t s)
{
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    CAS_CUDA(cudaStreamIsCapturing(s, &cap));
    const bool capturing = cap != cudaStreamCaptureStatusNone;
    if (nb > f.eval_blocks) {
        CAS_REQUIRE(!capturing, CAS_ERR_INVALID_ARGUMENT,
                    "evaluator step: a captured call may not grow the matrix's evaluator scratch; make one call of "
                    "the largest minibatch before capturing");
        CAS_REQUIRE(!f.eval_captured, CAS_ERR_INVALID_ARGUMENT,
                    "evaluator step: the matrix's evaluator scratch is held by captured CUDA graphs; a call over "
                    "more blocks than they were captured with would reallocate it (use a new matrix)");
        if (f.eval_partial || f.eval_dscore) {
            CAS_CUDA(cudaDeviceSynchronize());
            dfree(f.eval_partial);
            dfree(f.eval_dscore);
            f.eval_partial = nullptr;
            f.eval_dscore = nullptr;
            f.eval_blocks = 0;
        }
        CAS_CUDA(dmalloc(&f.eval_partial, sizeof(float) * nb * f.g.cols));
        CAS_CUDA(dmalloc(&f.eval_dscore, sizeof(float) * nb * kBlockRows));
        f.eval_blocks = nb;
    }
    if (!f.eval_red) {
        CAS_REQUIRE(!capturing, CAS_ERR_INVALID_ARGUMENT,
                    "evaluator step: make one call of the largest minibatch before capturing");
        CAS_CUDA(dmalloc(&f.eval_red, sizeof(double) * 2 * kEvalRedMax));
        CAS_CUDA(dmalloc(&f.eval_ctr, sizeof(int)));
        CAS_CUDA(cudaMemsetAsync(f.eval_ctr, 0, sizeof(int), s));
    }
    if (capturing) f.eval_captured = true;
    return CAS_OK;
}

// The adjoint's per-block partials of blocks [b0, b1) on g into eval_partial.
// The (block, chunk) items of a short range are split (plan_splits) by the
// chunks' mean entries in a block, the same in every block: the plan is made
// anew in each call, from one block's chunks (4 blocks of eight expanded
// patterns: the kernel takes 25 us with whole items, 18 so; planned over all
// items, 24 blocks cost the host 30 us a call).
static cas_status eval_adjoint_partials(FastLayout& f, int64_t b0, int64_t b1, const float* g, cudaStream_t s)
{
    const size_t smem = spmv_t_smem<float>(1);
    const int nch = f.g.nchunks;
    float fixed[kMaxChunks];
    std::fill_n(fixed, nch, unit_fixed(false, 1));
    const std::vector<int> K = plan_splits(fixed, f.chunk_entries, nch, static_cast<size_t>(b1 - b0));
    BlockUnits bu;
    for (int ch = 0; ch < nch; ch++) {
        bu.splits[ch] = static_cast<uint8_t>(K[ch]);
        bu.per_block += K[ch];
    }
    const int units = static_cast<int>(b1 - b0) * bu.per_block;
    { fast_spmv_t_kernel<float><<<units, kFastThreads, smem, s>>>(f.g, tview(f.tb), f.g32, f.sub_start, g,
                                                                  f.eval_partial, nullptr,
                                                                  static_cast<int>(b0 * nch), b0, nullptr, nullptr,
                                                                  nullptr, bu); cas::count_launch(); }
    CAS_CHECK_LAUNCH();
    return CAS_OK;
}

cas_status fast_eval_backward(FastLayout& f, int64_t b0, int64_t b1, const float* g, float* grad, cudaStream_t s)
{
    const int64_t nb = b1 - b0;
    if (f.g.cols == 0) return CAS_OK;
    if (nb <= 0) {
        CAS_CUDA(cudaMemsetAsync(grad, 0, sizeof(float) * f.g.cols, s));
        return CAS_OK;
    }
    CAS_TRY(eval_buffers(f, nb, s));
    CAS_TRY(eval_adjoint_partials(f, b0, b1, g, s));
    { block_partial_sum_kernel<<<fgrid(f.g.cols, 256), 256, 0, s>>>(f.eval_partial, static_cast<int>(nb), f.g.cols,
                                                                  grad); cas::count_launch(); }
    CAS_CHECK_LAUNCH();
    return CAS_OK;
}

cas_status fast_eval_adam_step(FastLayout& f, int64_t row0, int64_t row1, const float* target, float* w, float* m,
                               float* v, int64_t* step, double* loss_sum, const EvalAdam& o, cudaStream_t s)
{
    const int64_t n = row1 - row0;
    const int64_t b0 = row0 / kBlockRows, b1 = (row1 + kBlockRows - 1) / kBlockRows;
    if (f.g.cols == 0 || n <= 0) return CAS_OK;
    CAS_TRY(eval_buffers(f, b1 - b0, s));
    const unsigned g1 = eval_grid(n);
    auto loss = !all_slots_8(f.g) ? eval_loss_grad_kernel<false, 4>
                                  : (eval_resident(n) ? eval_loss_grad_kernel<true, kRowPatterns>
                                                      : eval_loss_grad_kernel<true, 1>);
    { loss<<<g1, kEvalRows, 0, s>>>(f.g, f.a16, w, target, row0, row1, o.delta, 1.0f / static_cast<float>(n),
                                    f.eval_dscore, f.eval_red); cas::count_launch(); }
    CAS_CHECK_LAUNCH();
    CAS_TRY(eval_adjoint_partials(f, b0, b1, f.eval_dscore, s));
    const unsigned g3 = static_cast<unsigned>(std::min<int64_t>((f.g.cols + 255) / 256, kEvalRedMax));  // a column a thread
    { eval_adam_kernel<<<g3, 256, 0, s>>>(f.eval_partial, static_cast<int>(b1 - b0), f.g.cols, w, m, v, step,
                                          loss_sum, f.eval_red, static_cast<int>(g1), f.eval_ctr, o,
                                          1.0 / static_cast<double>(n)); cas::count_launch(); }
    CAS_CHECK_LAUNCH();
    return CAS_OK;
}

template cas_status fast_spmv<float, float>(const FastLayout&, const float*, float*, const double*, const double*,
                                            double*, int*, int, cudaStream_t, int*, const int*, const FastActive*);
template cas_status fast_spmv<double, double>(const FastLayout&, const double*, double*, const double*,
                                              const double*, double*, int*, int, cudaStream_t, int*, const int*,
                                              const FastActive*);
template cas_status fast_spmv<double, float>(const FastLayout&, const double*, float*, const double*, const double*,
                                             double*, int*, int, cudaStream_t, int*, const int*, const FastActive*);
template cas_status fast_spmv_t_partials<float>(const FastLayout&, const float*, int*, cudaStream_t, const int*,
                                                const FastActive*);
template cas_status fast_spmv_t_partials<double>(const FastLayout&, const double*, int*, cudaStream_t, const int*,
                                                 const FastActive*);
template FastPlanView fast_plan_view<float>(const FastLayout&);
template FastPlanView fast_plan_view<double>(const FastLayout&);
template FastCols fast_cols<float>(const FastLayout&);
template FastCols fast_cols<double>(const FastLayout&);
template cas_status fast_spmv_t<float>(const FastLayout&, const float*, float*, cudaStream_t);
template cas_status fast_spmv_t<double>(const FastLayout&, const double*, double*, cudaStream_t);

}  // namespace cas
