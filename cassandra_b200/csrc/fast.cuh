// The blocked layout of a pattern CSR and its products (fast.cu).
//
// Rows are cut into blocks of kBlockRows.  Inside a block the entries of each
// pattern (indexer) are stored together:
//
//   A16  uint16  [block][pattern][row][slot]   local column of every entry
//   G32  uint32  [block][pattern][entry]       (local column << 16) |
//                                              (row in block << 2) | end,
//                                              sorted by column then row (the
//                                              transposed copy); end marks the
//                                              last entry of each column
//
// G32 is stored in rounds of kRound entries: the sorted order is cut into
// rounds from each group's start (every group starts on a round boundary),
// and inside a round the 32 consecutive entries a lane reduces (lane L:
// entries 32L .. 32L+31) lie in 8 rows of 512 bytes, one 16-byte word per
// lane and row, so that a warp reads a round with 8 coalesced loads.
// round_phys() maps an entry's position in the sorted order to its place.
//
// Both copies group a block's entries by pattern.  A x gathers a row's
// entries of x from a table of the patterns' slices (see FastTable) or
// through the caches; A'y stages the block's slice of y in shared memory and
// reduces the column-sorted entries of one column chunk into a shared-memory
// accumulator.  Local columns must fit 16 bits (index space per pattern <=
// 65536).
#pragma once
#include <cstdint>

#include "internal.cuh"

namespace cas {

constexpr int kBlockRows = 16384;        // rows per block (and per A'y tile)
constexpr int kRound = 1024;             // G32 entries of one A'y round (32 lanes x 32)
constexpr int kLaneRun = kRound / 32;    // consecutive entries a lane reduces per round
constexpr int kFastThreads = 1024;       // threads of the A'y kernel
constexpr int kAxThreads = 1024;         // threads of the A x kernel
constexpr int kChunkCols = 8192;         // column chunk of the A'y accumulators
constexpr int kSubCols = 64;             // column sub-chunk: the finest split of an A'y item
constexpr int kSubPerChunk = kChunkCols / kSubCols;
constexpr int kEvalRedMax = 4096;        // CTAs of each reduction of an evaluator training step
constexpr int kAxSplitMax = 32;          // units of a block in the direct A x, and A x partials per block of a batch
constexpr int kAxDirectRows = kBlockRows / kAxSplitMax;  // rows of such a unit, one a thread
constexpr int kAxDirectBlocks = 48;      // most blocks that A x does without a table (see fast_spmv_table_kernel)
constexpr int kAxTableSplit = kBlockRows / kAxThreads;   // units of a block in the table A x, one row a thread
static_assert(kAxTableSplit < kAxSplitMax, "a table unit's partials share the layout of the direct units'");
constexpr int kAtySplitMax = 16;         // most CTAs sharing one A'y item's columns
constexpr int kMaxFastPatterns = 32;
constexpr int kMaxChunks = kMaxFastPatterns * (65536 / kChunkCols);  // of a layout; pieces and super-chunks are no more
constexpr int kTableBytes = 140 * 1024;  // most shared memory of the A x table; the rest of the SM's 256 KB is L1

constexpr int kMaxProblems = 64;         // independent fits in one batched layout

// Per-pattern geometry, passed to kernels by value.
//
// A layout may hold several independent problems (a batch of fits over the
// same patterns): problem q owns rows [prow0[q], prow0[q+1]) and blocks
// [pblk0[q], pblk0[q+1]) -- blocks never straddle problems, so a problem's
// last block may be partial -- and columns [q * pcols, (q + 1) * pcols).
// The matrix is block diagonal.  A single fit is the case nprob == 1.
struct FastGeometry {
    int npat = 0;
    int k = 0;                           // entries per row (sum of slots)
    int64_t rows = 0, cols = 0;          // cols = nprob * pcols
    int64_t nblocks = 0;
    int slot0[kMaxFastPatterns];
    int slots[kMaxFastPatterns];
    int64_t off[kMaxFastPatterns];       // column offset of the pattern inside a problem
    int space[kMaxFastPatterns];         // columns of the pattern
    int chunk0[kMaxFastPatterns];        // first global chunk of the pattern
    int nchunks = 0;
    int nprob = 1;
    int64_t pcols = 0;                   // columns per problem
    int64_t prow0[kMaxProblems + 1];     // first row of each problem
    int pblk0[kMaxProblems + 1];         // first block of each problem

    __host__ __device__ int prob_of_block(int64_t b) const
    {
        int lo = 0, hi = nprob - 1;  // largest q with pblk0[q] <= b
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (pblk0[mid] <= b)
                lo = mid;
            else
                hi = mid - 1;
        }
        return lo;
    }
    __host__ __device__ int prob_of_row(int64_t r) const
    {
        int lo = 0, hi = nprob - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (prow0[mid] <= r)
                lo = mid;
            else
                hi = mid - 1;
        }
        return lo;
    }
    __host__ __device__ int64_t block_row0(int64_t b) const
    {
        const int q = prob_of_block(b);
        return prow0[q] + (b - pblk0[q]) * kBlockRows;
    }
    __host__ __device__ int64_t block_rows(int64_t b) const
    {
        const int q = prob_of_block(b);
        const int64_t r = prow0[q + 1] - (prow0[q] + (b - pblk0[q]) * kBlockRows);
        return r < kBlockRows ? r : kBlockRows;
    }
    // First column of the problem that owns block b.
    __host__ __device__ int64_t col_base(int64_t b) const { return prob_of_block(b) * pcols; }
    // Block and row inside the block of row r.
    __host__ __device__ void locate_row(int64_t r, int64_t& b, int64_t& rb) const
    {
        const int q = prob_of_row(r);
        const int64_t local = r - prow0[q];
        b = pblk0[q] + local / kBlockRows;
        rb = local - (local / kBlockRows) * kBlockRows;
    }
    // Rows of a block rounded up to kRound, so that every (block, pattern)
    // segment starts on a G32 round (and on a 16-byte boundary).
    __host__ __device__ int64_t padded_rows(int64_t b) const
    {
        return (block_rows(b) + kRound - 1) & ~int64_t(kRound - 1);
    }
    // Element offset of (block, pattern) in A16 / G32.
    __host__ __device__ int64_t seg(int64_t b, int p) const
    {
        return b * int64_t(kBlockRows) * k + padded_rows(b) * slot0[p];
    }
    __host__ __device__ int64_t seg_len(int64_t b, int p) const { return block_rows(b) * slots[p]; }
    __host__ __device__ int64_t total_elems() const
    {
        return nblocks == 0 ? 0 : (nblocks - 1) * int64_t(kBlockRows) * k + padded_rows(nblocks - 1) * k;
    }
};

// Place in G32 of the entry at position i of the sorted order (i counted
// from any round boundary): offset o = 32 L + 4 q + j inside the round goes
// to 128 q + 4 L + j.
__host__ __device__ __forceinline__ uint32_t round_phys(uint32_t i)
{
    return (i & ~uint32_t(kRound - 1)) | ((i & 0x1Cu) << 5) | ((i & 0x3E0u) >> 3) | (i & 3u);
}
static_assert(kRound == 1024 && kLaneRun == 32, "round_phys assumes 32 lanes x 32 entries");

// The problems a batched step works on (those not retired), in problem
// order, rebuilt on the device before each iteration.  Given to the
// products, it lets a few remaining small problems still fill the GPU: A x
// and A'y split their work units (a block's rows, an item's columns) over
// more CTAs the fewer units the listed problems have.  The A'y units of the
// list are laid out when it changes (fast_plan_active).
struct FastActive {
    int n;
    int list[kMaxProblems];
    int pos[kMaxProblems];  // slot of each problem in list, -1 if absent
    int nunits[2];          // A'y units of the listed problems: FP32, FP64
    uint32_t* units[2];     // (unit_pack), room for fast_plan_room() each
};

// A'y work units.  An item of a work list (a super-chunk's columns over a
// block range) is one unit or is split by columns into up to kAtySplitMax.
// What a unit takes is a fixed part (its fields, its share, its columns
// cleared and written: 12,000 cycles), a part per block (y staged, the table,
// barriers: 8,000) and its entries (280 cycles a round of 1,024 in FP32 and
// 700 in FP64, which is the shared-memory bandwidth that y gathers and
// accumulator updates at random banks leave), so it is counted in entries.
// With fewer items than kPlanWaves a CTA, the items that cost more than a limit
// are split; of kPlanLimits limits the one with the shortest estimate is taken.
// A list without an active list whose items fit one wave is not split past it
// (plan_splits).  Items differ by a factor of 100 (the columns of an edge or
// corner pattern that random play reaches, and those it does not), so a few
// large ones set the time of a small product that does not split them.
// A'y of the eight expanded patterns, us, FP32 / FP64, items whole or split by
// column counts -> these units: 8 blocks 35 / 66 -> 29 / 49, 32 blocks
// 68 / 199 -> 64 / 156, 64 blocks 126 / 335 -> 117 / 285; a training step's
// 4 blocks 25 -> 17; a batch's iteration with 24 blocks left in three problems
// 81 -> 59, with 15 left 43 -> 30.
constexpr int kPlanWaves = 4;
constexpr int kPlanLimits = 16;  // the most expensive item's cost, down in steps of 2^(1/4)

// The fixed cost of a unit of `blocks` blocks, in entries.
__host__ __device__ inline float unit_fixed(bool fp64, int blocks)
{
    return fp64 ? 18000.0f + 12000.0f * blocks : 40000.0f + 30000.0f * blocks;
}

__host__ __device__ inline uint32_t unit_pack(int item, int split, int K)
{
    return static_cast<uint32_t>(item) << 8 | static_cast<uint32_t>(split) << 4 | static_cast<uint32_t>(K - 1);
}
static_assert(kAtySplitMax == 16, "unit_pack: 4 bits for the split and its number");

// Splits of an item of `entries` entries and fixed cost `fixed` that bring a
// unit's cost to limit (at least two rounds a unit).
__host__ __device__ inline int unit_split(float fixed, float entries, float limit)
{
    const float most = entries / (2.0f * kRound);
    float k = limit > fixed ? ceilf(entries / (limit - fixed)) : static_cast<float>(kAtySplitMax);
    k = k < most ? k : floorf(most);
    return k < 1 ? 1 : (k > kAtySplitMax ? kAtySplitMax : static_cast<int>(k));
}

// What a schedule of `units` units takes on `ctas` CTAs: the longest unit in
// one wave, else the mean load and a quarter of the longest.
__host__ __device__ inline float plan_estimate(float units, float load, float longest, float ctas)
{
    return units <= ctas ? longest : (load / ctas > longest ? load / ctas : longest) + 0.25f * longest;
}

// Work list of one A'y variant.  Columns are grouped into "super-chunks":
// sets of column pieces (whole 8192-column chunks of one pattern, or a
// pattern's last partial chunk) packed into one shared-memory accumulator of
// per_sc chunks, so several narrow patterns share one pass over a block's y
// slice.  An item is (super-chunk, block range); every item writes the
// partial sums of its super-chunk's columns, and a column's value is the sum
// of its super-chunk's items in item order.
struct FastTranspose {
    int per_sc = 1;        // accumulator capacity in chunks
    bool range_major = false;  // single fits: items run block range by block range (y slices shared in L2)
    int items_per_sm = 2;  // work items per SM the entries are balanced over
    bool pack = true;      // super-chunks may hold pieces of several patterns
    bool persistent = false;  // one CTA per SM taking items from a counter (else one CTA per item)
    int nsc = 0;
    int npieces = 0;
    int nitems = 0;
    int64_t max_item_entries = 0;  // most G32 entries any item reduces
    int* sc_piece0 = nullptr;  // [nsc + 1] first piece of each super-chunk
    int* piece_pat = nullptr;  // [npieces] pattern of the piece
    int* piece_ch0 = nullptr;  // [npieces] first global chunk
    int* piece_ch1 = nullptr;  // [npieces] one past the last global chunk (same pattern)
    int* piece_acc = nullptr;  // [npieces] accumulator offset of the piece's first column
    int* chunk_sc = nullptr;   // [nchunks] super-chunk of every chunk
    int* chunk_acc = nullptr;  // [nchunks] accumulator offset of the chunk's first column
    int* item_sc = nullptr;    // [nitems]
    int* item_b0 = nullptr;    // [nitems]
    int* item_b1 = nullptr;    // [nitems]
    int64_t* item_part = nullptr;  // [nitems] offset of the item's partials
    int* sc_item0 = nullptr;       // [nprob * nsc + 1] first entry of each (problem, super-chunk) in sc_part
    uint32_t* units = nullptr;     // [nunits] the work units without an active list (unit_pack)
    int nunits = 0;
    float* grp_entries = nullptr;  // [nprob * nsc] most entries of an item of the (problem, super-chunk); null for
                                   // one problem, whose active list takes `units`
    int* grp_blocks = nullptr;     // [nprob * nsc] most blocks of one, likewise
    int64_t* sc_part = nullptr;    // [nitems] partial offsets of the items, listed super-chunk by super-chunk
                                   // (block ranges in order): the order the column sums add them in
    void* partial = nullptr;       // float or double partials
    int* ctr = nullptr;            // [2] work counter and finished CTAs of the persistent schedule (reset by the kernel)
    void* meta = nullptr;          // one device block holding every array above except partial
};

// The patterns whose slices of x the A x kernel keeps in shared memory.
struct FastTable {
    int base[kMaxFastPatterns];  // first table element of the pattern's slice, -1: not in the table
    int elems = 0;
};

// One measured A'y schedule of the build-time autotuner.
struct FastTuneEntry {
    int per_sc;
    int range_major;
    int items_per_sm;
    int pack;
    int persistent;
    float ms;  // mean time of one FP32 A'y (partials + column sums) on this layout
};
constexpr int kMaxTune = 12;

struct FastLayout {
    FastGeometry g;
    FastTable tab32, tab64;
    FastTuneEntry tune[kMaxTune];      // candidates timed at build (empty: default schedule)
    int ntune = 0;
    int tune_cached = 0;               // schedule taken from the per-process cache
    uint16_t* a16 = nullptr;
    uint32_t* g32 = nullptr;
    float chunk_entries[kMaxChunks];   // mean entries of each chunk in a block
    uint32_t* sub_start = nullptr;     // [nblocks][nchunks * kSubPerChunk] absolute index in G32 of the
                                       // first entry of every column sub-chunk (a chunk starts at its first)
    FastTranspose t32, t64;            // A'y work lists of the solvers (FP32, FP64)
    FastTranspose tb;                  // one item per (block, chunk): adjoints over block ranges
    float* eval_partial = nullptr;     // [blocks][cols] partials of the last adjoint
    float* eval_dscore = nullptr;      // [blocks * kBlockRows] loss gradient of a training step's rows
    int64_t eval_blocks = 0;           // blocks the two buffers above hold
    bool eval_captured = false;        // a CUDA graph captured a call that uses them: they never move again
    double* eval_red = nullptr;        // [2 * kEvalRedMax] per-CTA loss partials of a training step
    int* eval_ctr = nullptr;           // last-CTA counter of the training step's epilogue
};

// Hyperparameters of one training step of the evaluator (Adam as
// torch.optim.Adam without weight decay; mean Huber loss plus l2 ||w||^2).
struct EvalAdam {
    float lr, beta1, beta2, eps, l2, delta;
};

// Device view of a work list for fast_plan_active.  One problem is listed or
// not, so its plan is the one made at build (units); several problems' units
// are laid out from the costs of their (problem, super-chunk) groups, whose
// items sc_item0 numbers (in a list of one problem sc_item0 counts sc_part's
// entries, which are not the items when those run range by range).
struct FastPlanView {
    const uint32_t* units;
    int nunits;
    const int* sc_item0;
    const float* grp_entries;
    const int* grp_blocks;
    int nsc;
    bool fp64;
    // every array that fast_plan_active reads is there
    bool complete() const { return nsc == 0 || units || (sc_item0 && grp_entries && grp_blocks); }
};
template <typename T>
FastPlanView fast_plan_view(const FastLayout& f);
int64_t fast_plan_room(const FastLayout& f);  // units of either list at most

// Lays out the units of the listed problems' items in units / *nunits; every
// thread of one CTA calls (whole warps).  Items expensive under the chosen
// limit come first.
__device__ inline void fast_plan_active(const FastPlanView& pv, const FastActive* al, uint32_t* units, int* nunits,
                                        float ctas)
{
    if (pv.units) {
        const int n = al->n > 0 ? pv.nunits : 0;
        for (int i = threadIdx.x; i < n; i += blockDim.x) units[i] = pv.units[i];
        if (threadIdx.x == 0) *nunits = n;
        __syncthreads();
        return;
    }
    __shared__ float s_est[kPlanLimits], s_long[kPlanLimits], s_limit[kPlanLimits];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const int ng = al->n * pv.nsc;
    auto group = [&](int i, int& it0, int& nit, float& fixed, float& entries) {
        const int grp = al->list[i / pv.nsc] * pv.nsc + i % pv.nsc;
        it0 = pv.sc_item0[grp];
        nit = pv.sc_item0[grp + 1] - it0;
        fixed = unit_fixed(pv.fp64, pv.grp_blocks[grp]);
        entries = pv.grp_entries[grp];
    };
    int it0, nit;
    float fixed, entries;
    float top = 0, items = 0;
    for (int i = lane; i < ng; i += 32) {
        group(i, it0, nit, fixed, entries);
        if (nit > 0) top = fmaxf(top, fixed + entries);
        items += nit;
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
        top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, d));
        items += __shfl_xor_sync(0xffffffffu, items, d);
    }
    const int limits = items < kPlanWaves * ctas ? kPlanLimits : 1;  // the first limit splits nothing
    for (int j = warp; j < limits; j += warps) {
        const float limit = top * exp2f(-0.25f * j);
        float load = 0, longest = 0, n = 0;
        for (int i = lane; i < ng; i += 32) {
            group(i, it0, nit, fixed, entries);
            if (nit == 0) continue;
            const int K = unit_split(fixed, entries, limit);
            load += nit * (K * fixed + entries);
            longest = fmaxf(longest, fixed + entries / K);
            n += nit * K;
        }
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) {
            load += __shfl_xor_sync(0xffffffffu, load, d);
            n += __shfl_xor_sync(0xffffffffu, n, d);
            longest = fmaxf(longest, __shfl_xor_sync(0xffffffffu, longest, d));
        }
        if (lane == 0) {
            s_est[j] = plan_estimate(n, load, longest, ctas);
            s_long[j] = longest;
            s_limit[j] = limit;
        }
    }
    __syncthreads();
    if (warp == 0) {
        int best = 0;
        for (int j = 1; j < limits; j++)
            if (s_est[j] < s_est[best]) best = j;
        int at = 0;
        for (int small = 0; small < 2; small++)
            for (int i0 = 0; i0 < ng; i0 += 32) {
                int K = 0;
                nit = 0;
                if (i0 + lane < ng) {
                    group(i0 + lane, it0, nit, fixed, entries);
                    K = unit_split(fixed, entries, s_limit[best]);
                    if ((fixed + entries / K < 0.6f * s_long[best]) != (small != 0)) nit = 0;
                }
                int incl = nit * K;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const int u = __shfl_up_sync(0xffffffffu, incl, d);
                    if (lane >= d) incl += u;
                }
                int o = at + incl - nit * K;
                for (int it = 0; it < nit; it++)
                    for (int k = 0; k < K; k++) units[o++] = unit_pack(it0 + it, k, K);
                at += __shfl_sync(0xffffffffu, incl, 31);
            }
        if (lane == 0) *nunits = at;
    }
    __syncthreads();
}

// Device view used by the column reductions of the solver.
struct FastCols {
    FastGeometry g;
    int nsc;                 // super-chunks per problem
    const int* chunk_sc;
    const int* chunk_acc;
    const int* sc_item0;
    const int64_t* sc_part;
};

// Builds the blocked layout from positions (indexes them itself).  Returns
// CAS_ERR_INVALID_ARGUMENT without touching `out` if the pattern set does
// not fit the layout (a pattern wider than 16-bit columns, too many patterns
// or a slot count other than 1, 2, 4, 8).
// prob_rows (host, nprob entries) splits the rows into independent problems
// (a batch of fits, in row order); null with nprob == 1 is a single fit.
// chunks (may be null): positions still arriving, indexed chunk by chunk.
cas_status fast_build(const DevicePatterns& dp, const PatternSet& ps, const uint64_t* d_pos, int64_t rows,
                      const int64_t* prob_rows, int nprob, uint64_t* diag_int, FastLayout& out, cudaStream_t s,
                      const PositionChunks* chunks = nullptr);
bool fast_supported(const PatternSet& ps);
void fast_free(FastLayout& f);

// y = A x on the blocked layout; also writes compensated partials of
// ||y||^2 (part may be null; *n_parts = their number, fast_ax_parts).  mode
// 0: y = A x; 1: y = A x - coef * y (coef read from *coef); 2: y = b - A x
// (b may be null: y = -A x).  done_flag set: nothing runs; pdone[q] set: the
// rows of problem q are skipped (their partials are 0).
//
// With act only the listed problems' blocks run, and the partials are laid
// out [block][kAxSplitMax] (those not used are 0): problem q's are the
// 2 * kAxSplitMax * (pblk0[q+1] - pblk0[q]) doubles from part + 2 *
// kAxSplitMax * pblk0[q].
template <typename T, typename Y>
cas_status fast_spmv(const FastLayout& f, const T* x, Y* y, const double* b, const double* coef, double* part,
                     int* done_flag, int mode, cudaStream_t s, int* n_parts, const int* pdone = nullptr,
                     const FastActive* act = nullptr);
// Norm partials of A x without an active list.
int fast_ax_parts(int64_t nblocks);

// Partials of A' y on the blocked layout (FP32: float partials, FP64:
// double partials; a null y stands for a vector of ones); columns are
// summed by fast_col_sum().  Items of
// problems whose pdone flag is set are skipped.  An item's columns may be
// split over several CTAs (column sub-chunks), each writing its columns of
// the item's partials, so the partial layout does not depend on the split.
// With act only the listed problems' items run (one CTA per SM taking
// units from the work counter).
template <typename T>
cas_status fast_spmv_t_partials(const FastLayout& f, const T* y, int* done_flag, cudaStream_t s,
                                const int* pdone = nullptr, const FastActive* act = nullptr);

template <typename T>
FastCols fast_cols(const FastLayout& f);

// acc += the next N partials, all loaded before the adds, in their order.  (An
// unrolled loop leaves it to the compiler how many loads it issues ahead, and
// it chose otherwise in each kernel: the FP32 LSQR step of one pattern's 148
// partials a column, 786,432 rows, took 14.5 us instead of 8.8, where the PCG
// step took 8.2 instead of 10.7; 5.9 and 5.7 so.  Remainders go by halves, as
// a predicated batch costs as much as a full one.)
template <typename T, int N, typename Acc>
__device__ __forceinline__ void sum_ahead(const T*& at, int64_t stride, Acc& acc)
{
    T v[N];
#pragma unroll
    for (int u = 0; u < N; u++) {
        v[u] = *at;
        at += stride;
    }
#pragma unroll
    for (int u = 0; u < N; u++) acc += static_cast<Acc>(v[u]);
}

// Column c of A'y, TOP partials ahead: 32 where the sum is all the kernel does
// (fast_col_sum_kernel, us, 16 and 32 ahead: FP64, 4.9M rows of two patterns, 148
// partials a column, 36 and 21; FP32, 9.8M rows of eight expanded ones 24 and
// 18), 16 where its registers are shared (32 take the steps of the solvers past
// 64 and a quarter of their CTAs: the PCG step of 786,432 rows of five expanded
// patterns 8.8 and 12.0).
template <typename T, int TOP = 16>
__device__ __forceinline__ double fast_col_sum(const FastCols& fc, const T* partial, int64_t c)
{
    int64_t q = 0;
    if (fc.g.nprob > 1) {
        q = c / fc.g.pcols;
        c -= q * fc.g.pcols;
    }
    int p = 0;
    while (p + 1 < fc.g.npat && fc.g.off[p + 1] <= c) p++;
    const int local = static_cast<int>(c - fc.g.off[p]);
    const int ch = fc.g.chunk0[p] + local / kChunkCols;
    const int sc = static_cast<int>(q) * fc.nsc + fc.chunk_sc[ch];
    const int pos = fc.chunk_acc[ch] + local % kChunkCols;
    const int i0 = fc.sc_item0[sc], n = fc.sc_item0[sc + 1] - i0;
    if (n == 0) return 0;
    // A super-chunk's items have their partials at equal distances, so no
    // address waits for a load.
    const T* at = partial + fc.sc_part[i0] + pos;
    const int64_t stride = n > 1 ? fc.sc_part[i0 + 1] - fc.sc_part[i0] : 0;
    double acc = 0;
    int left = n;
    if constexpr (TOP == 32)
        for (; left >= 32; left -= 32) sum_ahead<T, 32>(at, stride, acc);
    for (; left >= 16; left -= 16) sum_ahead<T, 16>(at, stride, acc);
    if (left & 8) sum_ahead<T, 8>(at, stride, acc);
    if (left & 4) sum_ahead<T, 4>(at, stride, acc);
    if (left & 2) sum_ahead<T, 2>(at, stride, acc);
    if (left & 1) sum_ahead<T, 1>(at, stride, acc);
    return acc;
}

// Where the partials of a chunk's columns lie: column j of the chunk is the
// sum over i < n of partial[at + j + i * stride] (a super-chunk's items have
// their partials at equal distances).
struct ChunkPartials {
    int64_t at;
    int n;
    int stride;
};

// Those of problem q's chunks into ref[0..nchunks) (shared memory), by a CTA.
__device__ __forceinline__ void fast_chunk_partials(const FastCols& fc, int q, ChunkPartials* ref)
{
    for (int ch = threadIdx.x; ch < fc.g.nchunks; ch += blockDim.x) {
        const int sc = q * fc.nsc + fc.chunk_sc[ch];
        const int i0 = fc.sc_item0[sc], n = fc.sc_item0[sc + 1] - i0;
        const int64_t at = n > 0 ? fc.sc_part[i0] : 0;
        ref[ch] = ChunkPartials{at + fc.chunk_acc[ch], n, n > 1 ? static_cast<int>(fc.sc_part[i0 + 1] - at) : 0};
    }
}

// Sums of U columns (local to the problem) from their chunks' references,
// their partials' loads in flight together; a column not below P gives 0.
template <typename T, int U>
__device__ __forceinline__ void fast_col_sums(const FastGeometry& g, const ChunkPartials* ref,
                                              const T* __restrict__ partial, const int64_t (&c)[U], double (&sum)[U])
{
    const T* at[U];
    int n[U], stride[U], most = 0;
#pragma unroll
    for (int u = 0; u < U; u++) {
        n[u] = 0;
        stride[u] = 0;
        at[u] = partial;
        sum[u] = 0;
        if (c[u] < g.pcols) {
            int p = 0;
            while (p + 1 < g.npat && g.off[p + 1] <= c[u]) p++;
            const int local = static_cast<int>(c[u] - g.off[p]);
            const ChunkPartials r = ref[g.chunk0[p] + local / kChunkCols];
            at[u] = partial + r.at + local % kChunkCols;
            n[u] = r.n;
            stride[u] = r.stride;
        }
        most = max(most, n[u]);
    }
#pragma unroll 4
    for (int i = 0; i < most; i++)
#pragma unroll
        for (int u = 0; u < U; u++)
            if (i < n[u]) sum[u] += static_cast<double>(at[u][static_cast<int64_t>(i) * stride[u]]);
}

// Jacobi diagonal diag(A'A) as integers (deterministic), written over diag:
// the column counts from the FP32 A'y of a vector of ones (exact while every
// item holds fewer than 2^24 entries, else counted from G32 directly) plus
// the share of rows that hold a column more than once.  Needs the FP32 work
// list.
cas_status fast_diag(const FastLayout& f, uint64_t* diag, cudaStream_t s);

// Evaluator forward over rows [row0, row1) (FP32 scores) and its adjoint
// grad = A' g over the rows of blocks [b0, b1) (deterministic; grad has cols
// entries and is overwritten).
cas_status fast_eval_forward(const FastLayout& f, int64_t row0, int64_t row1, const float* w, float* score,
                             cudaStream_t s);
cas_status fast_eval_backward(FastLayout& f, int64_t b0, int64_t b1, const float* g, float* grad, cudaStream_t s);
// One training step on rows [row0, row1) (block bounds; row1 may be the last
// row): three kernels — forward with the Huber loss and its gradient, the
// adjoint's partials, and the epilogue with the L2 term and Adam (w, m, v
// updated; *step advanced; the step's loss added to *loss_sum).
cas_status fast_eval_adam_step(FastLayout& f, int64_t row0, int64_t row1, const float* target, float* w, float* m,
                               float* v, int64_t* step, double* loss_sum, const EvalAdam& o, cudaStream_t s);

// Full A'y into a dense vector (standalone product).
template <typename T>
cas_status fast_spmv_t(const FastLayout& f, const T* y, T* x, cudaStream_t s);

}  // namespace cas
