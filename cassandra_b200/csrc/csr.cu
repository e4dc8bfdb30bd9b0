// The device-resident CSR: construction (indexing, the sort-built transposed
// copy, column statistics) and the products A x, A' y and the Jacobi diagonal.
//
// Layout in HBM for rows R, K entries per row, cols C, nnz = R K:
//   idx       R*K  uint32   row-major column indices (the reference's MatrixCSR)
//   row_idx   nnz  uint32   rows of each entry, sorted by (column, row)
//   col_ptr   C+1  int64    start of each column in row_idx
//   unit_*                  A' y work units (<= kUnit entries of one column)
//   diag_int  C    uint64   diag(A'A), exact integers
#include <algorithm>
#include <vector>

#include "common.cuh"
#include "fast.cuh"
#include "internal.cuh"

namespace cas {

namespace {

// ---------------------------------------------------------------------------
// Exclusive scan of uint32 (totals must stay below 2^32).
// ---------------------------------------------------------------------------
constexpr int kScanThreads = 256;
constexpr int kScanItems = 16;
constexpr int kScanTile = kScanThreads * kScanItems;

__global__ void scan_reduce_kernel(const uint32_t* __restrict__ in, int64_t n, uint32_t* __restrict__ sums)
{
    __shared__ uint32_t s[kScanThreads / 32];
    const int64_t base = static_cast<int64_t>(blockIdx.x) * kScanTile;
    uint32_t acc = 0;
    for (int i = threadIdx.x; i < kScanTile; i += kScanThreads)
        if (base + i < n) acc += in[base + i];
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t t = 0;
        for (int w = 0; w < kScanThreads / 32; w++) t += s[w];
        sums[blockIdx.x] = t;
    }
}

// Exclusive scan of one tile, plus a per-tile carry-in.
__global__ void scan_tile_kernel(const uint32_t* __restrict__ in, int64_t n, const uint32_t* __restrict__ carry,
                                 uint32_t* __restrict__ out)
{
    __shared__ uint32_t s[kScanThreads];
    const int64_t base = static_cast<int64_t>(blockIdx.x) * kScanTile + static_cast<int64_t>(threadIdx.x) * kScanItems;
    uint32_t v[kScanItems];
    uint32_t local = 0;
#pragma unroll
    for (int i = 0; i < kScanItems; i++) {
        v[i] = base + i < n ? in[base + i] : 0;
        local += v[i];
    }
    s[threadIdx.x] = local;
    __syncthreads();
    for (int o = 1; o < kScanThreads; o <<= 1) {
        uint32_t t = threadIdx.x >= o ? s[threadIdx.x - o] : 0;
        __syncthreads();
        s[threadIdx.x] += t;
        __syncthreads();
    }
    uint32_t run = s[threadIdx.x] - local + (carry ? carry[blockIdx.x] : 0);
#pragma unroll
    for (int i = 0; i < kScanItems; i++) {
        if (base + i < n) out[base + i] = run;
        run += v[i];
    }
}

// Values of scratch an exclusive scan of n needs: its tiles' sums, theirs,
// and so on.
int64_t scan_scratch(int64_t n)
{
    int64_t total = 0;
    while (n > kScanTile) {
        n = (n + kScanTile - 1) / kScanTile;
        total += n;
    }
    return total;
}

// Exclusive scan of n uint32 values into out (may alias in).
cas_status exclusive_scan(const uint32_t* in, uint32_t* out, int64_t n, uint32_t* scratch, cudaStream_t s)
{
    if (n <= 0) return CAS_OK;
    const int64_t tiles = (n + kScanTile - 1) / kScanTile;
    if (tiles == 1) {
        { scan_tile_kernel<<<1, kScanThreads, 0, s>>>(in, n, nullptr, out); cas::count_launch(); }
        CAS_CHECK_LAUNCH();
        return CAS_OK;
    }
    { scan_reduce_kernel<<<static_cast<unsigned>(tiles), kScanThreads, 0, s>>>(in, n, scratch); cas::count_launch(); }
    CAS_CHECK_LAUNCH();
    CAS_TRY(exclusive_scan(scratch, scratch, tiles, scratch + tiles, s));
    { scan_tile_kernel<<<static_cast<unsigned>(tiles), kScanThreads, 0, s>>>(in, n, scratch, out); cas::count_launch(); }
    CAS_CHECK_LAUNCH();
    return CAS_OK;
}

// ---------------------------------------------------------------------------
// Stable LSD radix sort of (key, value) uint32 pairs, up to 9 bits per pass:
// two passes sort the columns of every pattern set of up to 2^18 columns.
// Pass 0 may take its values implicitly as entry / k (the CSR row), which is
// how the transposed copy is built straight from the row-major indices.
// ---------------------------------------------------------------------------
constexpr int kSortThreads = 512;
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kSortItems = 16;  // per thread
constexpr int kSortTile = kSortThreads * kSortItems;
constexpr int kRadixBits = 9;
constexpr int kRadix = 1 << kRadixBits;
static_assert(kRadix == kSortThreads, "one thread per digit");

// counts[digit * tiles + tile].  Bound by memory: 16 keys a thread are loaded
// before their shared-memory atomics (34M keys: 71 us a pass when each was
// counted before the next was loaded, 34 us).
__global__ void __launch_bounds__(kSortThreads) radix_hist_kernel(const uint32_t* __restrict__ keys, int64_t n,
                                                                  int shift, int bits, int64_t tiles,
                                                                  uint32_t* __restrict__ counts)
{
    __shared__ uint32_t h[kRadix];
    const uint32_t mask = (1u << bits) - 1;
    for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        h[threadIdx.x] = 0;
        __syncthreads();
        const int64_t base = tile * kSortTile + threadIdx.x;
        uint32_t key[kSortItems];
#pragma unroll
        for (int r = 0; r < kSortItems; r++) {
            const int64_t i = base + r * kSortThreads;
            key[r] = i < n ? keys[i] : 0;
        }
#pragma unroll
        for (int r = 0; r < kSortItems; r++)
            if (base + r * kSortThreads < n) atomicAdd(&h[(key[r] >> shift) & mask], 1u);
        __syncthreads();
        if (threadIdx.x <= mask) counts[static_cast<int64_t>(threadIdx.x) * tiles + tile] = h[threadIdx.x];
        __syncthreads();
    }
}

// The lanes whose digit equals this lane's: one ballot a bit.
template <int BITS>
__device__ __forceinline__ unsigned digit_peers(uint32_t d)
{
    unsigned peers = 0xffffffffu;
#pragma unroll
    for (int b = 0; b < BITS; b++) {
        const bool one = (d >> b) & 1;
        const unsigned m = __ballot_sync(0xffffffffu, one);
        peers &= one ? m : ~m;
    }
    return peers;
}

// The value of an item without values: its row, item / k, from the row and
// place in it of the warp's first item.  inv = 2^32 / k rounded up (k up to
// kImplicitMagic, where the quotients of rem + 8,192 are exact), else 0.
constexpr uint32_t kImplicitMagic = 32768;

__device__ __forceinline__ uint32_t implicit_row(uint32_t row0, uint32_t rem, uint32_t k, uint32_t inv)
{
    if (k == 1) return row0 + rem;
    return row0 + (inv ? __umulhi(rem, inv) : rem / k);
}

// One tile's items ranked once: a warp takes 512 consecutive items, 32 at a
// time, and counts them by digit in its own row of wcount (ballots give the
// rank among equals); the rows and the digits are then scanned across the
// CTA, the tile is put in digit order in shared memory and leaves in runs of
// a digit (16 items on average, 64 bytes).  Bound by instructions, a ballot a
// bit first of all: with bounds checks and divisions by k a warp took 156 for
// 32 pairs and 320 us a pass, so whole tiles run without checks, and rows
// without divisions.  34M pairs of 17 bits: three passes of 445 us when 256
// items at a time were ranked, with two scans, and scattered from registers;
// 230 + 243 us now (544 MB a pass: 83 us at the copy rate).
struct ScatterSmem {
    uint32_t key[kSortTile], val[kSortTile];
    uint32_t base[kRadix];               // first place of the tile's items of a digit, less their place in the tile
    uint16_t wcount[kSortWarps][kRadix];  // a warp's items of a digit, then the tile's before them
    uint32_t wsum[kSortWarps];
};

template <int BITS, bool WHOLE>
__device__ __forceinline__ void scatter_tile(ScatterSmem& sm, const uint32_t* __restrict__ keys_in,
                                             const uint32_t* __restrict__ vals_in, uint32_t k, uint32_t inv,
                                             int64_t first, int count, int shift, uint32_t base,
                                             uint32_t* __restrict__ keys_out, uint32_t* __restrict__ vals_out)
{
    constexpr uint32_t kMask = (1u << BITS) - 1;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const unsigned lt_mask = (1u << lane) - 1;
    const int i0 = warp * (32 * kSortItems) + lane;  // item r of the lane: i0 + 32 r
    const uint32_t* kp = keys_in + first + i0;
    uint32_t key[kSortItems];
    uint16_t rank[kSortItems];
#pragma unroll
    for (int r = 0; r < kSortItems; r++) key[r] = WHOLE || i0 + 32 * r < count ? kp[32 * r] : 0xFFFFFFFFu;
    uint16_t* mine = sm.wcount[warp];
#pragma unroll
    for (int r = 0; r < kSortItems; r++) {
        // items past the end share the last digit with the tile's last items
        // and rank behind them
        const uint32_t d = (key[r] >> shift) & kMask;
        const unsigned peers = digit_peers<BITS>(d);
        const uint32_t c = mine[d], before = __popc(peers & lt_mask);
        __syncwarp();
        if (before == 0) mine[d] = static_cast<uint16_t>(c + __popc(peers));
        __syncwarp();
        rank[r] = static_cast<uint16_t>(c + before);
    }
    __syncthreads();
    // digit t: the tile's items of it, and where they start in the tile
    uint32_t total = 0;
#pragma unroll
    for (int w = 0; w < kSortWarps; w++) {
        const uint32_t c = sm.wcount[w][t];
        sm.wcount[w][t] = static_cast<uint16_t>(total);
        total += c;
    }
    uint32_t incl = total;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t u = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += u;
    }
    if (lane == 31) sm.wsum[warp] = incl;
    __syncthreads();
    uint32_t start = incl - total;
#pragma unroll
    for (int w = 0; w < kSortWarps; w++)
        if (w < warp) start += sm.wsum[w];
    sm.base[t] = base - start;
#pragma unroll
    for (int w = 0; w < kSortWarps; w++) sm.wcount[w][t] += static_cast<uint16_t>(start);
    __syncthreads();
    if (vals_in) {
        const uint32_t* vp = vals_in + first + i0;
#pragma unroll
        for (int r = 0; r < kSortItems; r++) {
            const uint32_t at = mine[(key[r] >> shift) & kMask] + rank[r];
            sm.key[at] = key[r];
            if (WHOLE || i0 + 32 * r < count) sm.val[at] = vp[32 * r];
        }
    } else {
        const int64_t w0 = first + warp * (32 * kSortItems);  // the warp's first item
        const int64_t row0 = w0 / k;
        const uint32_t rem = static_cast<uint32_t>(w0 - row0 * k) + lane;
#pragma unroll
        for (int r = 0; r < kSortItems; r++) {
            const uint32_t at = mine[(key[r] >> shift) & kMask] + rank[r];
            sm.key[at] = key[r];
            sm.val[at] = implicit_row(static_cast<uint32_t>(row0), rem + 32 * r, k, inv);
        }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kSortItems; r++) {
        const int i = t + r * kSortThreads;
        if (!WHOLE && i >= count) break;
        const uint32_t v = sm.key[i];
        const uint32_t pos = sm.base[(v >> shift) & kMask] + static_cast<uint32_t>(i);
        keys_out[pos] = v;
        vals_out[pos] = sm.val[i];
    }
    __syncthreads();
}

template <int BITS>
__global__ void __launch_bounds__(kSortThreads, 2) radix_scatter_kernel(
    const uint32_t* __restrict__ keys_in, const uint32_t* __restrict__ vals_in, uint32_t k, uint32_t inv, int64_t n,
    int shift, int64_t tiles, const uint32_t* __restrict__ offsets, uint32_t* __restrict__ keys_out,
    uint32_t* __restrict__ vals_out)
{
    extern __shared__ __align__(16) unsigned char scatter_raw[];
    ScatterSmem& sm = *reinterpret_cast<ScatterSmem*>(scatter_raw);
    const int t = threadIdx.x;
    for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const uint32_t base = t < (1 << BITS) ? offsets[static_cast<int64_t>(t) * tiles + tile] : 0;
        uint32_t* z = reinterpret_cast<uint32_t*>(sm.wcount);
#pragma unroll
        for (int i = 0; i < kSortWarps * kRadix / 2; i += kSortThreads) z[i + t] = 0;
        __syncthreads();
        const int64_t first = tile * kSortTile, left = n - first;
        if (left >= kSortTile)
            scatter_tile<BITS, true>(sm, keys_in, vals_in, k, inv, first, kSortTile, shift, base, keys_out, vals_out);
        else
            scatter_tile<BITS, false>(sm, keys_in, vals_in, k, inv, first, static_cast<int>(left), shift, base,
                                      keys_out, vals_out);
    }
}

using ScatterKernel = void (*)(const uint32_t*, const uint32_t*, uint32_t, uint32_t, int64_t, int, int64_t,
                               const uint32_t*, uint32_t*, uint32_t*);

// The kernel of a pass of `bits` bits: a ballot a bit is most of a pair's
// work, so few bits have their own.
ScatterKernel scatter_kernel(int bits)
{
    return bits <= 5 ? radix_scatter_kernel<5> : (bits <= 8 ? radix_scatter_kernel<8> : radix_scatter_kernel<9>);
}

// Sorts keys/values stably by the low `bits` bits of the key.  keys_in is not
// modified.  The result ends in (*keys_res, *vals_res), which point into
// bufA/bufB.  scratch holds radix_scratch(n) values.
int64_t radix_scratch(int64_t n)
{
    const int64_t counts = kRadix * ((n + kSortTile - 1) / kSortTile);
    return counts + scan_scratch(counts);
}

cas_status radix_sort_pairs(const uint32_t* keys_in, const uint32_t* vals_in, int implicit_k, int64_t n, int bits,
                            uint32_t* keysA, uint32_t* valsA, uint32_t* keysB, uint32_t* valsB,
                            uint32_t** keys_res, uint32_t** vals_res, uint32_t* scratch, cudaStream_t s)
{
    const int64_t tiles = (n + kSortTile - 1) / kSortTile;
    const int passes = std::max(1, (bits + kRadixBits - 1) / kRadixBits);
    uint32_t* counts = scratch;
    uint32_t* sums = scratch + kRadix * tiles;
    const unsigned grid = static_cast<unsigned>(std::min<int64_t>(tiles, static_cast<int64_t>(sm_count()) * 8));
    const uint32_t k = static_cast<uint32_t>(implicit_k);
    const uint32_t inv = k > 1 && k <= kImplicitMagic ? static_cast<uint32_t>(((uint64_t(1) << 32) + k - 1) / k) : 0;
    const uint32_t* kin = keys_in;
    const uint32_t* vin = vals_in;
    for (int pass = 0; pass < passes && n > 0; pass++) {
        // the bits in equal shares, as the kernels take them (bits past the
        // key's are zero)
        const int shift = bits * pass / passes, share = bits * (pass + 1) / passes - shift;
        const int b = share <= 5 ? 5 : (share <= 8 ? 8 : 9);
        const ScatterKernel scatter = scatter_kernel(b);
        CAS_CUDA(cudaFuncSetAttribute(scatter, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      static_cast<int>(sizeof(ScatterSmem))));
        uint32_t* kout = (pass % 2 == 0) ? keysA : keysB;
        uint32_t* vout = (pass % 2 == 0) ? valsA : valsB;
        { radix_hist_kernel<<<grid, kSortThreads, 0, s>>>(kin, n, shift, b, tiles, counts); cas::count_launch(); }
        CAS_CHECK_LAUNCH();
        CAS_TRY(exclusive_scan(counts, counts, (int64_t(1) << b) * tiles, sums, s));
        { scatter<<<grid, kSortThreads, sizeof(ScatterSmem), s>>>(kin, vin, k, inv, n, shift, tiles, counts, kout, vout); cas::count_launch(); }
        CAS_CHECK_LAUNCH();
        kin = kout;
        vin = vout;
        *keys_res = kout;
        *vals_res = vout;
    }
    return CAS_OK;
}

// ---------------------------------------------------------------------------
// Column structure from the sorted keys.
// ---------------------------------------------------------------------------
// col_ptr, and diag(A'A)_c = sum over rows of m^2 (m = multiplicity of c in
// the row), accumulated as sum over entries of 2j+1 where j is the entry's
// position in its (column, row) run.  Integer sums: any order gives the same
// result.  One pass over the sorted pairs, bound by memory: two kernels, with
// a match across the warp in the second, took 210 us for 34M, this 155 us.
__global__ void column_kernel(const uint32_t* __restrict__ keys, const uint32_t* __restrict__ rows, uint32_t nnz,
                              int64_t cols, int64_t* __restrict__ col_ptr, uint64_t* __restrict__ diag)
{
    const int lane = threadIdx.x & 31;
    for (int64_t e0 = static_cast<int64_t>(blockIdx.x) * blockDim.x; e0 <= nnz;
         e0 += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const uint32_t e = static_cast<uint32_t>(e0) + threadIdx.x;  // nnz < 2^32 - 1; past it in the last warps only
        const bool valid = e0 + threadIdx.x < nnz;
        const uint32_t c = valid ? keys[e] : 0xFFFFFFFFu, r = valid ? rows[e] : 0;
        uint32_t cb = __shfl_up_sync(0xffffffffu, c, 1), rb = __shfl_up_sync(0xffffffffu, r, 1);
        if (lane == 0 && e0 + threadIdx.x > 0 && e0 + threadIdx.x <= nnz) {
            cb = keys[e - 1];
            rb = rows[e - 1];
        }
        const bool head = e0 + threadIdx.x == 0 || (e0 + threadIdx.x <= nnz && cb != c);
        if (head) {
            const int64_t to = valid ? static_cast<int64_t>(c) : cols;
            for (int64_t k = e > 0 ? static_cast<int64_t>(cb) + 1 : 0; k <= to && k <= cols; k++) col_ptr[k] = e;
        }
        const bool repeat = valid && !head && rb == r;
        // a column's entries are consecutive: the last lane of each run adds
        // the run's sum
        const unsigned heads = __ballot_sync(0xffffffffu, head || lane == 0);
        const int first = 31 - __clz(heads & (0xffffffffu >> (31 - lane)));
        uint32_t run = static_cast<uint32_t>(lane - first + 1);
        if (__any_sync(0xffffffffu, repeat)) {
            uint32_t twice = 0;  // 2j, summed over the run
            if (repeat) {
                uint32_t j = 1;
                while (e > j && keys[e - j - 1] == c && rows[e - j - 1] == r) j++;
                twice = 2 * j;
            }
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t u = __shfl_up_sync(0xffffffffu, twice, o);
                if (lane >= o) twice += u;
            }
            const uint32_t rest = __shfl_sync(0xffffffffu, twice, first > 0 ? first - 1 : 0);
            run += twice - (first > 0 ? rest : 0);
        }
        const unsigned tail = __shfl_down_sync(0xffffffffu, static_cast<unsigned>(head || !valid), 1);
        if (valid && (lane == 31 || tail)) atomicAdd(reinterpret_cast<unsigned long long*>(diag + c), run);
    }
}

__global__ void unit_count_kernel(const int64_t* __restrict__ col_ptr, int64_t cols, uint32_t* __restrict__ cnt)
{
    for (int64_t c = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; c < cols;
         c += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const int64_t len = col_ptr[c + 1] - col_ptr[c];
        cnt[c] = static_cast<uint32_t>(len == 0 ? 1 : (len + kUnit - 1) / kUnit);
    }
}

__global__ void unit_fill_kernel(const uint32_t* __restrict__ unit_ptr, int64_t cols, int32_t* __restrict__ unit_col)
{
    for (int64_t c = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; c < cols;
         c += static_cast<int64_t>(gridDim.x) * blockDim.x)
        for (uint32_t u = unit_ptr[c]; u < unit_ptr[c + 1]; u++) unit_col[u] = static_cast<int32_t>(c);
}

__global__ void bound_check_kernel(const uint32_t* __restrict__ idx, int64_t n, uint32_t cols,
                                   unsigned int* __restrict__ bad)
{
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x)
        if (idx[i] >= cols) atomicOr(bad, 1u);
}

// ---------------------------------------------------------------------------
// Products.
// ---------------------------------------------------------------------------

// y = A x: a warp takes ROWS rows at a time, its lanes stride over each row's K
// indices (coalesced 4K-byte streams), gathers of x summed in FP64,
// warp-shuffle trees.  Bound by the gathers' L1 lookups, one line a cycle and
// SM (2M rows of 32 at random: 227 us), once the rows' chains of index, gather
// and tree overlap: a row at a time 281 us (FP64 307), four 237 (261).  A part
// of x in shared memory (64 to 180 KB, one CTA an SM) took 281 to 482.
//
// A row of more than kSpmvShortRow entries has loads enough in flight by
// itself, and four of them are a chain as long as the kernel when rows are few:
// us, FP32, a row at a time and four: 148 rows of 8,192 50 and 366, 5,000 of
// 3,000 88 and 156, 60,000 of 1,000 98 and 147, 30,000 of 100 29 and 32; the
// other way 300,000 of 100 146 and 138, 100,000 of 8 27 and 23.
constexpr int kSpmvRows = 4;
constexpr int kSpmvShortRow = 64;

template <typename T, int ROWS>
__global__ void __launch_bounds__(256) spmv_kernel(const uint32_t* __restrict__ idx, int64_t rows, int k,
                                                   const T* __restrict__ x, T* __restrict__ y)
{
    const int lane = threadIdx.x & 31;
    const int64_t warps = static_cast<int64_t>(gridDim.x) * (blockDim.x >> 5);
    for (int64_t r = (static_cast<int64_t>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5)) * ROWS; r < rows;
         r += warps * ROWS) {
        const uint32_t* row = idx + r * k;
        const int n = static_cast<int>(min(rows - r, static_cast<int64_t>(ROWS)));
        double acc[ROWS] = {};
        if constexpr (ROWS == 1) {
            for (int j = lane; j < k; j += 32) acc[0] += static_cast<double>(__ldg(x + __ldg(row + j)));
        } else {
            for (int j = lane; j < k; j += 32) {
                uint32_t c[ROWS];
                T v[ROWS];
#pragma unroll
                for (int i = 0; i < ROWS; i++)
                    if (i < n) c[i] = __ldg(row + static_cast<int64_t>(i) * k + j);
#pragma unroll
                for (int i = 0; i < ROWS; i++)
                    if (i < n) v[i] = __ldg(x + c[i]);
#pragma unroll
                for (int i = 0; i < ROWS; i++)
                    if (i < n) acc[i] += static_cast<double>(v[i]);
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int i = 0; i < ROWS; i++) acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], o);
        double mine = acc[0];
#pragma unroll
        for (int i = 1; i < ROWS; i++)
            if (lane == i) mine = acc[i];
        if (lane < n) y[r + lane] = static_cast<T>(mine);
    }
}

// Partial sums of A' y: one warp per work unit.
template <typename T>
__global__ void __launch_bounds__(256) spmv_t_units_kernel(CsrView a, const T* __restrict__ y,
                                                           double* __restrict__ partial)
{
    const int lane = threadIdx.x & 31;
    const int64_t warps = static_cast<int64_t>(gridDim.x) * (blockDim.x >> 5);
    for (int64_t u = static_cast<int64_t>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5); u < a.units;
         u += warps) {
        const int32_t c = a.unit_col[u];
        const int64_t begin = a.col_ptr[c] + static_cast<int64_t>(u - a.unit_ptr[c]) * kUnit;
        const int64_t end = min(a.col_ptr[c + 1], begin + kUnit);
        double acc = 0;
        for (int64_t e = begin + lane; e < end; e += 32) acc += static_cast<double>(__ldg(y + __ldg(a.row_idx + e)));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (lane == 0) partial[u] = acc;
    }
}

template <typename T>
__global__ void spmv_t_finalize_kernel(CsrView a, const double* __restrict__ partial, T* __restrict__ x)
{
    for (int64_t c = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; c < a.cols;
         c += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        double acc = 0;
        for (uint32_t u = a.unit_ptr[c]; u < a.unit_ptr[c + 1]; u++) acc += partial[u];
        x[c] = static_cast<T>(acc);
    }
}

template <typename T>
__global__ void jacobi_kernel(const uint64_t* __restrict__ diag, int64_t cols, T* __restrict__ out)
{
    for (int64_t c = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; c < cols;
         c += static_cast<int64_t>(gridDim.x) * blockDim.x)
        out[c] = static_cast<T>(1) / static_cast<T>(diag[c]);
}

unsigned grid_for(int64_t work, int per_block)
{
    const int64_t want = (work + per_block - 1) / per_block;
    return static_cast<unsigned>(std::max<int64_t>(1, std::min<int64_t>(want, static_cast<int64_t>(sm_count()) * 16)));
}

}  // namespace

template <typename T>
cas_status spmv(const CsrView& a, const T* x, T* y, cudaStream_t s)
{
    if (a.rows == 0) return CAS_OK;
    const bool several = a.k <= kSpmvShortRow;
    auto kernel = several ? spmv_kernel<T, kSpmvRows> : spmv_kernel<T, 1>;
    { kernel<<<grid_for(a.rows, several ? 8 * kSpmvRows : 8), 256, 0, s>>>(a.idx, a.rows, a.k, x, y); cas::count_launch(); }
    CAS_CHECK_LAUNCH();
    return CAS_OK;
}

template <typename T>
cas_status spmv_t(const CsrView& a, const T* y, double* unit_partial, T* x, cudaStream_t s)
{
    if (a.cols == 0) return CAS_OK;
    { spmv_t_units_kernel<T><<<grid_for(a.units, 8), 256, 0, s>>>(a, y, unit_partial); cas::count_launch(); }
    CAS_CHECK_LAUNCH();
    { spmv_t_finalize_kernel<T><<<grid_for(a.cols, 256), 256, 0, s>>>(a, unit_partial, x); cas::count_launch(); }
    CAS_CHECK_LAUNCH();
    return CAS_OK;
}

template <typename T>
cas_status jacobi(const CsrView& a, T* out, cudaStream_t s)
{
    if (a.cols == 0) return CAS_OK;
    { jacobi_kernel<T><<<grid_for(a.cols, 256), 256, 0, s>>>(a.diag_int, a.cols, out); cas::count_launch(); }
    CAS_CHECK_LAUNCH();
    return CAS_OK;
}

template cas_status spmv<float>(const CsrView&, const float*, float*, cudaStream_t);
template cas_status spmv<double>(const CsrView&, const double*, double*, cudaStream_t);
template cas_status spmv_t<float>(const CsrView&, const float*, double*, float*, cudaStream_t);
template cas_status spmv_t<double>(const CsrView&, const double*, double*, double*, cudaStream_t);
template cas_status jacobi<float>(const CsrView&, float*, cudaStream_t);
template cas_status jacobi<double>(const CsrView&, double*, cudaStream_t);

// Builds the transposed copy, column pointers, work units and diag(A'A) for a
// CSR whose idx array is in place.
cas_status build_structure(cas_csr* a, cudaStream_t s)
{
    const int64_t nnz = a->rows * a->k;
    CAS_REQUIRE(nnz < 0xFFFFFFFFLL, CAS_ERR_INVALID_ARGUMENT,
                "CSR with 2^32 or more entries is not supported (uint32 entry offsets)");
    CAS_REQUIRE(a->rows < 0xFFFFFFFFLL, CAS_ERR_INVALID_ARGUMENT, "rows must fit uint32");
    const int64_t cols = a->cols;
    CAS_CUDA(dmalloc(&a->col_ptr, sizeof(int64_t) * (cols + 1)));
    if (!a->diag_int) {
        CAS_CUDA(dmalloc(&a->diag_int, sizeof(uint64_t) * std::max<int64_t>(cols, 1)));
        CAS_CUDA(cudaMemsetAsync(a->diag_int, 0, sizeof(uint64_t) * std::max<int64_t>(cols, 1), s));
    }

    // scratch of the whole build: the check's flag, then the sort's or the
    // scan's
    struct Scratch {
        uint32_t* p = nullptr;
        ~Scratch() { dfree(p); }
    } scratch;
    CAS_CUDA(dmalloc(&scratch.p, sizeof(uint32_t) * (1 + std::max(radix_scratch(nnz), scan_scratch(cols + 1)))));
    if (nnz > 0) {
        unsigned int* bad = scratch.p;
        CAS_CUDA(cudaMemsetAsync(bad, 0, sizeof(unsigned int), s));
        { bound_check_kernel<<<grid_for(nnz, 1024), 256, 0, s>>>(a->idx, nnz, static_cast<uint32_t>(cols), bad); cas::count_launch(); }
        CAS_CHECK_LAUNCH();
        unsigned int hbad = 0;
        CAS_CUDA(cudaMemcpyAsync(&hbad, bad, sizeof hbad, cudaMemcpyDeviceToHost, s));
        CAS_CUDA(cudaStreamSynchronize(s));
        CAS_REQUIRE(hbad == 0, CAS_ERR_INVALID_ARGUMENT, "column index >= cols in CSR indices");
    }

    int bits = 1;
    while (bits < 32 && (1LL << bits) < cols) bits++;
    uint32_t *kA = nullptr, *vA = nullptr, *kB = nullptr, *vB = nullptr;
    const size_t bytes = sizeof(uint32_t) * std::max<int64_t>(nnz, 1);
    CAS_CUDA(dmalloc(&kA, bytes));
    CAS_CUDA(dmalloc(&vA, bytes));
    CAS_CUDA(dmalloc(&kB, bytes));
    CAS_CUDA(dmalloc(&vB, bytes));
    uint32_t *keys = kA, *vals = vA;
    cas_status st = CAS_OK;
    if (nnz > 0) st = radix_sort_pairs(a->idx, nullptr, a->k, nnz, bits, kA, vA, kB, vB, &keys, &vals, scratch.p + 1, s);
    if (st == CAS_OK) {
        { column_kernel<<<grid_for(nnz + 1, 256), 256, 0, s>>>(keys, vals, static_cast<uint32_t>(nnz), cols, a->col_ptr, a->diag_int); cas::count_launch(); }
        if (cudaGetLastError() != cudaSuccess) st = CAS_ERR_CUDA;
    }
    // keep the sorted rows, release the rest
    a->row_idx = vals;
    for (uint32_t* p : {kA, vA, kB, vB})
        if (p != vals) dfree(p);
    if (st != CAS_OK) return st;

    // A'y work units
    CAS_CUDA(dmalloc(&a->unit_ptr, sizeof(uint32_t) * (cols + 1)));
    if (cols > 0) {
        { unit_count_kernel<<<grid_for(cols, 256), 256, 0, s>>>(a->col_ptr, cols, a->unit_ptr); cas::count_launch(); }
        CAS_CHECK_LAUNCH();
    }
    CAS_CUDA(cudaMemsetAsync(a->unit_ptr + cols, 0, sizeof(uint32_t), s));
    CAS_TRY(exclusive_scan(a->unit_ptr, a->unit_ptr, cols + 1, scratch.p + 1, s));
    uint32_t units = 0;
    CAS_CUDA(cudaMemcpyAsync(&units, a->unit_ptr + cols, sizeof units, cudaMemcpyDeviceToHost, s));
    CAS_CUDA(cudaStreamSynchronize(s));
    a->units = units;
    CAS_CUDA(dmalloc(&a->unit_col, sizeof(int32_t) * std::max<int64_t>(units, 1)));
    CAS_CUDA(dmalloc(&a->unit_partial, sizeof(double) * std::max<int64_t>(units, 1)));
    if (cols > 0) {
        { unit_fill_kernel<<<grid_for(cols, 256), 256, 0, s>>>(a->unit_ptr, cols, a->unit_col); cas::count_launch(); }
        CAS_CHECK_LAUNCH();
    }
    return CAS_OK;
}

}  // namespace cas

using namespace cas;

namespace {
void free_csr(cas_csr* a)
{
    if (!a) return;
    int cur = 0;
    cudaGetDevice(&cur);
    if (a->device >= 0) cudaSetDevice(a->device);
    dfree(a->idx);
    dfree(a->col_ptr);
    dfree(a->row_idx);
    dfree(a->unit_col);
    dfree(a->unit_ptr);
    dfree(a->diag_int);
    dfree(a->unit_partial);
    if (a->fast) {
        fast_free(*a->fast);
        delete a->fast;
    }
    cudaSetDevice(cur);
    delete a;
}

cas_status finish_create(cas_csr* a, cudaStream_t s, cas_csr** out)
{
    cas_status st = build_structure(a, s);
    if (st == CAS_OK) {
        cudaError_t e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) {
            set_error(std::string("CSR build: ") + cudaGetErrorString(e));
            st = CAS_ERR_CUDA;
        }
    }
    if (st != CAS_OK) {
        free_csr(a);
        return st;
    }
    *out = a;
    return CAS_OK;
}
}  // namespace

extern "C" {

CAS_API cas_status cas_csr_from_positions_layout(const cas_patterns* p, const uint64_t* d_positions, int64_t rows,
                                                 int layouts, void* stream, cas_csr** out)
{
    return cas::csr_from_positions(p, d_positions, rows, layouts, static_cast<cudaStream_t>(stream), out, nullptr);
}
}  // extern "C"

cas_status cas::csr_from_positions(const cas_patterns* p, const uint64_t* d_positions, int64_t rows, int layouts,
                                   cudaStream_t s, cas_csr** out, const PositionChunks* chunks)
{
    cas::NvtxRange nvtx_range("cas_csr_from_positions");
    CAS_REQUIRE(p && out && rows >= 0, CAS_ERR_INVALID_ARGUMENT, "cas_csr_from_positions: bad argument");
    CAS_REQUIRE(rows == 0 || d_positions, CAS_ERR_INVALID_ARGUMENT, "cas_csr_from_positions: null positions");
    CAS_REQUIRE((reinterpret_cast<uintptr_t>(d_positions) & 15) == 0, CAS_ERR_INVALID_ARGUMENT,
                "cas_csr_from_positions: position records must be 16-byte aligned");
    CAS_REQUIRE(layouts > 0 && (layouts & ~(CAS_LAYOUT_ROWS | CAS_LAYOUT_BLOCKED)) == 0, CAS_ERR_INVALID_ARGUMENT,
                "cas_csr_from_positions: layouts must be a non-empty mask of cas_layout");
    CAS_REQUIRE(!(layouts & CAS_LAYOUT_BLOCKED) || fast_supported(pattern_set(p)), CAS_ERR_INVALID_ARGUMENT,
                "cas_csr_from_positions: the blocked layout needs index spaces <= 65536 per pattern");
    CAS_REQUIRE(rows * static_cast<int64_t>(cas_patterns_nnz_per_row(p)) < 0xFFFFFFFFLL, CAS_ERR_INVALID_ARGUMENT,
                "cas_csr_from_positions: 2^32 or more entries are not supported");
    *out = nullptr;
    const DevicePatterns* dp = nullptr;
    CAS_TRY(patterns_on_device(p, &dp));
    auto* a = new cas_csr;
    CAS_CUDA(cudaGetDevice(&a->device));
    a->rows = rows;
    a->cols = dp->cols;
    a->k = dp->k;
    a->layouts = layouts;
    cudaError_t e = dmalloc(&a->diag_int, sizeof(uint64_t) * std::max<int64_t>(a->cols, 1));
    if (e == cudaSuccess) e = cudaMemsetAsync(a->diag_int, 0, sizeof(uint64_t) * std::max<int64_t>(a->cols, 1), s);
    if (e != cudaSuccess) {
        free_csr(a);
        set_error("cas_csr_from_positions: cannot allocate the column statistics");
        return CAS_ERR_OUT_OF_MEMORY;
    }
    cas_status st = CAS_OK;
    if (layouts & CAS_LAYOUT_BLOCKED) {
        a->fast = new FastLayout;
        // diag(A'A) comes from the blocked copy unless the row layout builds it
        st = fast_build(*dp, pattern_set(p), d_positions, rows, nullptr, 1,
                        (layouts & CAS_LAYOUT_ROWS) ? nullptr : a->diag_int, *a->fast, s, chunks);
        if (st != CAS_OK) {
            free_csr(a);
            return st;
        }
    }
    if (layouts & CAS_LAYOUT_ROWS) {
        e = dmalloc(&a->idx, sizeof(uint32_t) * std::max<int64_t>(rows * a->k, 1));
        if (e != cudaSuccess) {
            free_csr(a);
            set_error("cas_csr_from_positions: cannot allocate the index array");
            return CAS_ERR_OUT_OF_MEMORY;
        }
        if (chunks && !(layouts & CAS_LAYOUT_BLOCKED))  // the row layout indexes all rows at once
            for (int c = 0; c < chunks->n; c++) CAS_CUDA(cudaStreamWaitEvent(s, chunks->ready[c], 0));
        st = launch_index(*dp, d_positions, rows, a->idx, s);
        if (st != CAS_OK) {
            free_csr(a);
            return st;
        }
        return finish_create(a, s, out);
    }
    e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) {
        free_csr(a);
        set_error(std::string("CSR build: ") + cudaGetErrorString(e));
        return CAS_ERR_CUDA;
    }
    *out = a;
    return CAS_OK;
}

extern "C" {

CAS_API cas_status cas_csr_from_positions_batched(const cas_patterns* p, const uint64_t* d_positions,
                                                  const int64_t* h_problem_rows, int problems, void* stream,
                                                  cas_csr** out)
{
    cas::NvtxRange nvtx_range("cas_csr_from_positions_batched");
    CAS_REQUIRE(p && out && h_problem_rows && problems >= 1 && problems <= kMaxProblems, CAS_ERR_INVALID_ARGUMENT,
                "cas_csr_from_positions_batched: bad argument (1 to 64 problems)");
    CAS_REQUIRE(fast_supported(pattern_set(p)), CAS_ERR_INVALID_ARGUMENT,
                "cas_csr_from_positions_batched: the blocked layout needs index spaces <= 65536 per pattern");
    int64_t rows = 0;
    for (int q = 0; q < problems; q++) {
        CAS_REQUIRE(h_problem_rows[q] >= 0, CAS_ERR_INVALID_ARGUMENT,
                    "cas_csr_from_positions_batched: negative problem size");
        rows += h_problem_rows[q];
    }
    CAS_REQUIRE(rows == 0 || d_positions, CAS_ERR_INVALID_ARGUMENT, "cas_csr_from_positions_batched: null positions");
    CAS_REQUIRE((reinterpret_cast<uintptr_t>(d_positions) & 15) == 0, CAS_ERR_INVALID_ARGUMENT,
                "cas_csr_from_positions_batched: position records must be 16-byte aligned");
    *out = nullptr;
    const DevicePatterns* dp = nullptr;
    CAS_TRY(patterns_on_device(p, &dp));
    auto s = static_cast<cudaStream_t>(stream);
    auto* a = new cas_csr;
    CAS_CUDA(cudaGetDevice(&a->device));
    a->rows = rows;
    a->cols = dp->cols * problems;
    a->k = dp->k;
    a->layouts = CAS_LAYOUT_BLOCKED;
    cudaError_t e = dmalloc(&a->diag_int, sizeof(uint64_t) * std::max<int64_t>(a->cols, 1));
    if (e == cudaSuccess) e = cudaMemsetAsync(a->diag_int, 0, sizeof(uint64_t) * std::max<int64_t>(a->cols, 1), s);
    if (e != cudaSuccess) {
        free_csr(a);
        set_error("cas_csr_from_positions_batched: cannot allocate the column statistics");
        return CAS_ERR_OUT_OF_MEMORY;
    }
    a->fast = new FastLayout;
    cas_status st = fast_build(*dp, pattern_set(p), d_positions, rows, h_problem_rows, problems, a->diag_int,
                               *a->fast, s);
    if (st == CAS_OK) {
        e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) {
            set_error(std::string("batched CSR build: ") + cudaGetErrorString(e));
            st = CAS_ERR_CUDA;
        }
    }
    if (st != CAS_OK) {
        free_csr(a);
        return st;
    }
    *out = a;
    return CAS_OK;
}

CAS_API int cas_csr_problems(const cas_csr* a, int64_t* h_row0)
{
    if (!a) return -1;
    if (!a->fast) {
        if (h_row0) {
            h_row0[0] = 0;
            h_row0[1] = a->rows;
        }
        return 1;
    }
    const FastGeometry& g = a->fast->g;
    if (h_row0)
        for (int q = 0; q <= g.nprob; q++) h_row0[q] = g.prow0[q];
    return g.nprob;
}

CAS_API cas_status cas_csr_from_positions(const cas_patterns* p, const uint64_t* d_positions, int64_t rows,
                                          void* stream, cas_csr** out)
{
    CAS_REQUIRE(p, CAS_ERR_INVALID_ARGUMENT, "cas_csr_from_positions: null pattern set");
    const int layouts = CAS_LAYOUT_ROWS | (fast_supported(pattern_set(p)) ? CAS_LAYOUT_BLOCKED : 0);
    return cas_csr_from_positions_layout(p, d_positions, rows, layouts, stream, out);
}

CAS_API int cas_csr_layouts(const cas_csr* a) { return a ? a->layouts : 0; }

CAS_API int64_t cas_block_rows(void) { return kBlockRows; }

CAS_API int cas_csr_schedules(const cas_csr* a, cas_schedule* out, int max, cas_schedule* in_use)
{
    if (!a || !a->fast) return -1;
    const FastLayout& f = *a->fast;
    if (in_use) {
        in_use->chunks_per_item = f.t32.per_sc;
        in_use->range_major = f.t32.range_major ? 1 : 0;
        in_use->items_per_sm = f.t32.items_per_sm;
        in_use->pack = f.t32.pack ? 1 : 0;
        in_use->persistent = f.t32.persistent ? 1 : 0;
        in_use->ms = 0;
        for (int i = 0; i < f.ntune; i++)
            if (f.tune[i].per_sc == f.t32.per_sc && f.tune[i].range_major == in_use->range_major &&
                f.tune[i].items_per_sm == f.t32.items_per_sm && f.tune[i].pack == in_use->pack &&
                f.tune[i].persistent == in_use->persistent)
                in_use->ms = f.tune[i].ms;
    }
    int n = 0;
    for (int i = 0; i < f.ntune && out && n < max; i++, n++)
        out[n] = cas_schedule{f.tune[i].per_sc, f.tune[i].range_major, f.tune[i].items_per_sm, f.tune[i].pack,
                              f.tune[i].persistent, f.tune[i].ms};
    return n;
}

CAS_API cas_status cas_eval_forward(const cas_csr* a, int64_t row0, int64_t row1, const float* d_w, float* d_score,
                                    void* stream)
{
    CAS_REQUIRE(a && a->fast, CAS_ERR_INVALID_ARGUMENT, "cas_eval_forward: the CSR needs the blocked layout");
    CAS_REQUIRE(0 <= row0 && row0 <= row1 && row1 <= a->rows, CAS_ERR_SIZE_MISMATCH,
                "cas_eval_forward: row range outside the matrix");
    CAS_REQUIRE(row1 == row0 || (d_w && d_score), CAS_ERR_INVALID_ARGUMENT, "cas_eval_forward: null buffer");
    return fast_eval_forward(*a->fast, row0, row1, d_w, d_score, static_cast<cudaStream_t>(stream));
}

CAS_API cas_status cas_eval_backward(const cas_csr* a, int64_t row0, int64_t row1, const float* d_g, float* d_grad,
                                     void* stream)
{
    CAS_REQUIRE(a && a->fast, CAS_ERR_INVALID_ARGUMENT, "cas_eval_backward: the CSR needs the blocked layout");
    CAS_REQUIRE(a->fast->g.nprob == 1, CAS_ERR_INVALID_ARGUMENT,
                "cas_eval_backward: needs the layout of a single fit, not a batch");
    CAS_REQUIRE(0 <= row0 && row0 <= row1 && row1 <= a->rows, CAS_ERR_SIZE_MISMATCH,
                "cas_eval_backward: row range outside the matrix");
    CAS_REQUIRE(row0 % kBlockRows == 0 && (row1 % kBlockRows == 0 || row1 == a->rows), CAS_ERR_INVALID_ARGUMENT,
                "cas_eval_backward: the row range must start and end on block boundaries (cas_block_rows())");
    CAS_REQUIRE(d_grad && (row1 == row0 || d_g), CAS_ERR_INVALID_ARGUMENT, "cas_eval_backward: null buffer");
    const int64_t b0 = row0 / kBlockRows, b1 = (row1 + kBlockRows - 1) / kBlockRows;
    return fast_eval_backward(*a->fast, b0, b1, d_g, d_grad, static_cast<cudaStream_t>(stream));
}

CAS_API cas_status cas_eval_adam_step(const cas_csr* a, int64_t row0, int64_t row1, const float* d_target,
                                      float* d_w, float* d_m, float* d_v, int64_t* d_step, double* d_loss_sum,
                                      const cas_adam_opts* opts, void* stream)
{
    CAS_REQUIRE(a && a->fast, CAS_ERR_INVALID_ARGUMENT, "cas_eval_adam_step: the CSR needs the blocked layout");
    CAS_REQUIRE(a->fast->g.nprob == 1, CAS_ERR_INVALID_ARGUMENT,
                "cas_eval_adam_step: needs the layout of a single fit, not a batch");
    CAS_REQUIRE(0 <= row0 && row0 <= row1 && row1 <= a->rows, CAS_ERR_SIZE_MISMATCH,
                "cas_eval_adam_step: row range outside the matrix");
    CAS_REQUIRE(row0 % kBlockRows == 0 && (row1 % kBlockRows == 0 || row1 == a->rows), CAS_ERR_INVALID_ARGUMENT,
                "cas_eval_adam_step: the row range must start and end on block boundaries (cas_block_rows())");
    CAS_REQUIRE(opts, CAS_ERR_INVALID_ARGUMENT, "cas_eval_adam_step: null options");
    CAS_REQUIRE(row1 == row0 || (d_target && d_w && d_m && d_v && d_step && d_loss_sum), CAS_ERR_INVALID_ARGUMENT,
                "cas_eval_adam_step: null buffer");
    CAS_REQUIRE(opts->lr >= 0 && opts->beta1 >= 0 && opts->beta1 < 1 && opts->beta2 >= 0 && opts->beta2 < 1 &&
                    opts->eps > 0 && opts->l2 >= 0 && opts->delta > 0,
                CAS_ERR_INVALID_ARGUMENT, "cas_eval_adam_step: bad options");
    const EvalAdam o{opts->lr, opts->beta1, opts->beta2, opts->eps, opts->l2, opts->delta};
    return fast_eval_adam_step(*a->fast, row0, row1, d_target, d_w, d_m, d_v, d_step, d_loss_sum, o,
                               static_cast<cudaStream_t>(stream));
}

CAS_API cas_status cas_csr_from_indices(const uint32_t* d_indices, int nnz_per_row, int64_t rows, int64_t cols,
                                        void* stream, cas_csr** out)
{
    CAS_REQUIRE(out && nnz_per_row > 0 && rows >= 0 && cols >= 0, CAS_ERR_INVALID_ARGUMENT,
                "cas_csr_from_indices: bad argument");
    CAS_REQUIRE(rows == 0 || d_indices, CAS_ERR_INVALID_ARGUMENT, "cas_csr_from_indices: null indices");
    CAS_REQUIRE(cols < 0xFFFFFFFFLL, CAS_ERR_INVALID_ARGUMENT, "cas_csr_from_indices: cols must fit uint32");
    *out = nullptr;
    CAS_TRY(require_device());
    auto s = static_cast<cudaStream_t>(stream);
    auto* a = new cas_csr;
    CAS_CUDA(cudaGetDevice(&a->device));
    a->rows = rows;
    a->cols = cols;
    a->k = nnz_per_row;
    a->layouts = CAS_LAYOUT_ROWS;
    const size_t bytes = sizeof(uint32_t) * rows * nnz_per_row;
    cudaError_t e = dmalloc(&a->idx, std::max<size_t>(bytes, 4));
    if (e == cudaSuccess && bytes) e = cudaMemcpyAsync(a->idx, d_indices, bytes, cudaMemcpyDefault, s);
    if (e != cudaSuccess) {
        free_csr(a);
        set_error(std::string("cas_csr_from_indices: ") + cudaGetErrorString(e));
        return e == cudaErrorMemoryAllocation ? CAS_ERR_OUT_OF_MEMORY : CAS_ERR_CUDA;
    }
    return finish_create(a, s, out);
}

CAS_API void cas_csr_destroy(cas_csr* a) { free_csr(a); }
CAS_API int64_t cas_csr_rows(const cas_csr* a) { return a ? a->rows : -1; }
CAS_API int64_t cas_csr_cols(const cas_csr* a) { return a ? a->cols : -1; }
CAS_API int cas_csr_nnz_per_row(const cas_csr* a) { return a ? a->k : -1; }
CAS_API const uint32_t* cas_csr_indices(const cas_csr* a) { return a ? a->idx : nullptr; }

CAS_API cas_status cas_csr_transposed(const cas_csr* a, const int64_t** d_col_ptr, const uint32_t** d_row_idx)
{
    CAS_REQUIRE(a, CAS_ERR_INVALID_ARGUMENT, "cas_csr_transposed: null handle");
    if (d_col_ptr) *d_col_ptr = a->col_ptr;
    if (d_row_idx) *d_row_idx = a->row_idx;
    return CAS_OK;
}

CAS_API cas_status cas_spmv(const cas_csr* a, cas_dtype dtype, const void* d_x, void* d_y, void* stream)
{
    CAS_REQUIRE(a, CAS_ERR_INVALID_ARGUMENT, "cas_spmv: null handle");
    CAS_REQUIRE((d_x || a->cols == 0) && (d_y || a->rows == 0), CAS_ERR_INVALID_ARGUMENT, "cas_spmv: null vector");
    auto s = static_cast<cudaStream_t>(stream);
    if (a->fast && (dtype == CAS_F32 || dtype == CAS_F64)) {
        if (dtype == CAS_F32)
            return fast_spmv<float, float>(*a->fast, static_cast<const float*>(d_x), static_cast<float*>(d_y), nullptr,
                                           nullptr, nullptr, nullptr, 0, s, nullptr);
        return fast_spmv<double, double>(*a->fast, static_cast<const double*>(d_x), static_cast<double*>(d_y), nullptr,
                                         nullptr, nullptr, nullptr, 0, s, nullptr);
    }
    if (dtype == CAS_F32) return spmv<float>(a->view(), static_cast<const float*>(d_x), static_cast<float*>(d_y), s);
    if (dtype == CAS_F64)
        return spmv<double>(a->view(), static_cast<const double*>(d_x), static_cast<double*>(d_y), s);
    set_error("cas_spmv: unknown dtype");
    return CAS_ERR_INVALID_ARGUMENT;
}

CAS_API cas_status cas_spmv_t(const cas_csr* a, cas_dtype dtype, const void* d_y, void* d_x, void* stream)
{
    CAS_REQUIRE(a, CAS_ERR_INVALID_ARGUMENT, "cas_spmv_t: null handle");
    CAS_REQUIRE((d_y || a->rows == 0) && (d_x || a->cols == 0), CAS_ERR_INVALID_ARGUMENT, "cas_spmv_t: null vector");
    auto s = static_cast<cudaStream_t>(stream);
    if (a->fast && dtype == CAS_F32)
        return fast_spmv_t<float>(*a->fast, static_cast<const float*>(d_y), static_cast<float*>(d_x), s);
    if (a->fast && dtype == CAS_F64)
        return fast_spmv_t<double>(*a->fast, static_cast<const double*>(d_y), static_cast<double*>(d_x), s);
    if (dtype == CAS_F32)
        return spmv_t<float>(a->view(), static_cast<const float*>(d_y), a->unit_partial, static_cast<float*>(d_x), s);
    if (dtype == CAS_F64)
        return spmv_t<double>(a->view(), static_cast<const double*>(d_y), a->unit_partial, static_cast<double*>(d_x),
                              s);
    set_error("cas_spmv_t: unknown dtype");
    return CAS_ERR_INVALID_ARGUMENT;
}

CAS_API cas_status cas_jacobi(const cas_csr* a, cas_dtype dtype, void* d_out, void* stream)
{
    CAS_REQUIRE(a && (d_out || a->cols == 0), CAS_ERR_INVALID_ARGUMENT, "cas_jacobi: null argument");
    auto s = static_cast<cudaStream_t>(stream);
    if (dtype == CAS_F32) return jacobi<float>(a->view(), static_cast<float*>(d_out), s);
    if (dtype == CAS_F64) return jacobi<double>(a->view(), static_cast<double*>(d_out), s);
    set_error("cas_jacobi: unknown dtype");
    return CAS_ERR_INVALID_ARGUMENT;
}

}  // extern "C"
