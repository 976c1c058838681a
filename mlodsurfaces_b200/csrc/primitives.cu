// primitives.cu -- device exclusive scan and stable LSD radix sort.
//
// Tiles of 2048 items per 256-thread block, grids sized by the input; small
// sorts run in one block.
#include <utility>

#include "primitives.cuh"
#include "mlods_internal.cuh"

namespace mlods
{
namespace
{
constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;
constexpr int64_t kScanRawSums = 4096;  // block sums a block adds up itself (at most 16 a thread)

constexpr int kSortThreads = 256;
constexpr int kSortWarps = kSortThreads / 32;

inline size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t v)
{
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t n = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += n;
    }
    return v;
}

// Block-wide exclusive scan of one value per thread (blockDim.x == kScanThreads).
__device__ __forceinline__ uint32_t block_excl_scan(uint32_t v, uint32_t* s_warp, uint32_t* block_total)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t incl = warp_incl_scan(v);
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = lane < kScanThreads / 32 ? s_warp[lane] : 0u;
        uint32_t wi = warp_incl_scan(w);
        if (lane < kScanThreads / 32) s_warp[lane] = wi - w;
        if (lane == kScanThreads / 32 - 1) s_warp[kScanThreads / 32] = wi;
    }
    __syncthreads();
    const uint32_t r = s_warp[warp] + incl - v;
    *block_total = s_warp[kScanThreads / 32];
    __syncthreads();
    return r;
}

__global__ void scan_reduce_kernel(const uint32_t* __restrict__ in, int64_t n, uint32_t* __restrict__ block_sums)
{
    __shared__ uint32_t s_warp[kScanThreads / 32 + 1];
    const int64_t base = int64_t(blockIdx.x) * kScanTile;
    uint32_t sum = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        int64_t i = base + int64_t(k) * kScanThreads + threadIdx.x;
        if (i < n) sum += in[i];
    }
    uint32_t total;
    block_excl_scan(sum, s_warp, &total);
    if (threadIdx.x == 0) block_sums[blockIdx.x] = total;
}

// block_offs: the blocks' exclusive offsets, or (raw_sums) their sums, which the
// block adds up itself: fewer launches while the sums are few.
__global__ void scan_apply_kernel(const uint32_t* in, uint32_t* out, int64_t n, const uint32_t* __restrict__ block_offs,
                                  bool raw_sums, uint32_t* total_out)
{
    __shared__ uint32_t s_warp[kScanThreads / 32 + 1];
    uint32_t off = 0;
    if (raw_sums) {
        uint32_t before = 0;
        for (unsigned b = threadIdx.x; b < blockIdx.x; b += kScanThreads) before += __ldg(block_offs + b);
        block_excl_scan(before, s_warp, &off);
    } else if (block_offs) {
        off = block_offs[blockIdx.x];
    }
    const int64_t base = int64_t(blockIdx.x) * kScanTile + int64_t(threadIdx.x) * kScanItems;
    uint32_t v[kScanItems];
    uint32_t sum = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        int64_t i = base + k;
        v[k] = i < n ? in[i] : 0u;
        sum += v[k];
    }
    uint32_t total;
    uint32_t run = block_excl_scan(sum, s_warp, &total);
    run += off;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        int64_t i = base + k;
        if (i < n) out[i] = run;
        run += v[k];
    }
    if (total_out && blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) *total_out = off + total;
}

// ---------------------------------------------------------------- radix sort
//
// Latency bounds the small sorts and HBM the large ones.  Up to kSmallItems
// one block keeps all items in registers and shared memory and runs every pass
// in one launch.  Above that a pass is a per-tile histogram and a scatter;
// with at most kColumnTiles tiles every scatter block adds up the tiles before
// its own itself (64 columns of L2-resident counts), beyond that a scan of the
// counts does.  Keys are ranked a warp at a time (each warp holds a contiguous
// run of its tile, so no block synchronisation between the runs of 32) and
// leave the tile through shared memory in sorted order, so that a digit's keys
// go to consecutive addresses.  Against 256-thread blocks that ranked 16 runs
// one after another (a 4096-item tile in 13 us, 12 launches a sort of 30 bits):
// a 1,000-query projection 428 -> 381 us, ten one-iteration projections of 50k
// queries 4.57 -> 3.52 ms; tiles of 2048 keep a 100k sort on 49 SMs instead of 25.

constexpr int kSmallThreads = 1024;
constexpr int kSmallWarps = kSmallThreads / 32;
constexpr int64_t kSmallItems = 8 * kSmallThreads;
constexpr int64_t kColumnTiles = 128;
constexpr int kSortItems = 8;
constexpr int kSortTile = kSortThreads * kSortItems;

__device__ __forceinline__ uint32_t lane_lt()
{
    return (1u << (threadIdx.x & 31)) - 1u;
}

// Rank of each of the warp's items (ITEMS runs of 32, in that order) among the
// warp's items of the same digit; the warp's digit counts in cnt (zeroed).
template <int ITEMS>
__device__ __forceinline__ void warp_rank(const uint32_t (&digit)[ITEMS], uint32_t (&rank)[ITEMS], uint32_t* cnt)
{
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        const uint32_t peers = __match_any_sync(0xffffffffu, digit[k]);
        const uint32_t before = cnt[digit[k]];
        const uint32_t lower = __popc(peers & lane_lt());
        __syncwarp();
        if (lower == 0) cnt[digit[k]] = before + __popc(peers);
        __syncwarp();
        rank[k] = before + lower;
    }
}

// The whole sort of n <= ITEMS * kSmallThreads items in one block, the result
// in place.  Digits in which no two keys differ are skipped.  Slots beyond n
// hold the largest key and, being last in a stable sort, stay last.
template <typename K, bool PAIRS, int ITEMS>
__global__ void __launch_bounds__(kSmallThreads) radix_small_kernel(K* __restrict__ keys, uint32_t* __restrict__ vals,
                                                                    int n, int nbits)
{
    extern __shared__ __align__(16) unsigned char smem[];
    K* s_key = reinterpret_cast<K*>(smem);
    uint32_t* s_val = reinterpret_cast<uint32_t*>(s_key + ITEMS * kSmallThreads);
    uint32_t* s_cnt = PAIRS ? s_val + ITEMS * kSmallThreads : s_val;  // [warp][digit]
    __shared__ uint32_t s_base[256], s_sum[8];
    __shared__ unsigned long long s_diff;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int at = warp * 32 * ITEMS + lane;
    K key[ITEMS];
    uint32_t val[ITEMS];
    if (threadIdx.x == 0) s_diff = 0ull;
    const K k0 = keys[0];
    K diff = 0;
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        const int i = at + 32 * k;
        key[k] = i < n ? keys[i] : ~K(0);
        if (PAIRS) val[k] = i < n ? vals[i] : 0u;
        if (i < n) diff |= key[k] ^ k0;
    }
    __syncthreads();
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) diff |= __shfl_xor_sync(0xffffffffu, diff, o);
    if (lane == 0 && diff) atomicOr(&s_diff, (unsigned long long)diff);
    __syncthreads();
    const unsigned long long all_diff = s_diff;
    for (int shift = 0; shift < nbits; shift += 8) {
        if (((all_diff >> shift) & 255ull) == 0ull) continue;
        for (int k = threadIdx.x; k < kSmallWarps * 256; k += kSmallThreads) s_cnt[k] = 0;
        __syncthreads();
        uint32_t digit[ITEMS], rank[ITEMS];
#pragma unroll
        for (int k = 0; k < ITEMS; ++k) digit[k] = uint32_t(key[k] >> shift) & 255u;
        warp_rank<ITEMS>(digit, rank, s_cnt + warp * 256);
        __syncthreads();
        // each digit's counts over the warps -> exclusive prefixes, then a
        // scan of the digit totals
        uint32_t run = 0, incl = 0;
        if (threadIdx.x < 256) {
#pragma unroll 8
            for (int w = 0; w < kSmallWarps; ++w) {
                const uint32_t c = s_cnt[w * 256 + threadIdx.x];
                s_cnt[w * 256 + threadIdx.x] = run;
                run += c;
            }
            incl = warp_incl_scan(run);
            if (lane == 31) s_sum[warp] = incl;
        }
        __syncthreads();
        if (threadIdx.x < 256) {
            uint32_t off = 0;
            for (int w = 0; w < warp; ++w) off += s_sum[w];
            s_base[threadIdx.x] = off + incl - run;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < ITEMS; ++k) {
            const uint32_t pos = s_base[digit[k]] + s_cnt[warp * 256 + digit[k]] + rank[k];
            s_key[pos] = key[k];
            if (PAIRS) s_val[pos] = val[k];
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < ITEMS; ++k) {
            key[k] = s_key[at + 32 * k];
            if (PAIRS) val[k] = s_val[at + 32 * k];
        }
    }
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        const int i = at + 32 * k;
        if (i < n) {
            keys[i] = key[k];
            if (PAIRS) vals[i] = val[k];
        }
    }
}

// counts[tile * 256 + digit] (by_tile) or counts[digit * tiles + tile].
template <typename K>
__global__ void __launch_bounds__(kSortThreads) radix_hist_kernel(const K* __restrict__ keys, int64_t n, int shift,
                                                                  int tiles, bool by_tile, uint32_t* __restrict__ counts)
{
    __shared__ uint32_t hist[256];
    const int64_t base = int64_t(blockIdx.x) * kSortTile + threadIdx.x;
    K key[kSortItems];
#pragma unroll
    for (int k = 0; k < kSortItems; ++k) {
        const int64_t i = base + k * kSortThreads;
        key[k] = i < n ? keys[i] : K(0);
    }
    hist[threadIdx.x] = 0;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kSortItems; ++k)
        if (base + k * kSortThreads < n) atomicAdd(&hist[uint32_t(key[k] >> shift) & 255u], 1u);
    __syncthreads();
    counts[by_tile ? int64_t(blockIdx.x) * 256 + threadIdx.x : int64_t(threadIdx.x) * tiles + blockIdx.x] =
        hist[threadIdx.x];
}

// BY_TILE: counts as the histogram left them, by tile; else their exclusive
// scan in (digit, tile) order.
template <typename K, bool PAIRS, bool BY_TILE>
__global__ void __launch_bounds__(kSortThreads)
    radix_scatter_kernel(const K* __restrict__ keys, const uint32_t* __restrict__ vals, int64_t n, int shift, int tiles,
                         const uint32_t* __restrict__ counts, K* __restrict__ keys_out, uint32_t* __restrict__ vals_out)
{
    __shared__ K s_key[kSortTile];
    __shared__ uint32_t s_val[PAIRS ? kSortTile : 1];
    __shared__ uint32_t s_cnt[kSortWarps][256];
    __shared__ uint32_t s_base[256];  // first place of the digit in the tile
    __shared__ int64_t s_out[256];    // its place in the output less that
    __shared__ uint32_t s_warp[kSortWarps + 1];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t tile0 = int64_t(blockIdx.x) * kSortTile;
    const int at = warp * 32 * kSortItems + lane;
    K key[kSortItems];
    uint32_t val[kSortItems];
#pragma unroll
    for (int k = 0; k < kSortItems; ++k) {
        const int64_t i = tile0 + at + 32 * k;
        key[k] = i < n ? keys[i] : ~K(0);
        if (PAIRS) val[k] = i < n ? vals[i] : 0u;
    }
    // the digit's place in the output: the tiles before this one
    uint32_t before = 0, all = 0;
    if (BY_TILE) {
#pragma unroll 16
        for (int t = 0; t < tiles; ++t) {
            const uint32_t c = __ldg(counts + int64_t(t) * 256 + threadIdx.x);
            all += c;
            if (t < int(blockIdx.x)) before += c;
        }
        uint32_t total;
        before += block_excl_scan(all, s_warp, &total);
    } else {
        before = __ldg(counts + int64_t(threadIdx.x) * tiles + blockIdx.x);
    }
#pragma unroll
    for (int w = 0; w < kSortWarps; ++w) s_cnt[w][threadIdx.x] = 0;
    __syncthreads();
    uint32_t digit[kSortItems], rank[kSortItems];
#pragma unroll
    for (int k = 0; k < kSortItems; ++k) digit[k] = uint32_t(key[k] >> shift) & 255u;
    warp_rank<kSortItems>(digit, rank, s_cnt[warp]);
    __syncthreads();
    {
        uint32_t run = 0;
#pragma unroll
        for (int w = 0; w < kSortWarps; ++w) {
            const uint32_t c = s_cnt[w][threadIdx.x];
            s_cnt[w][threadIdx.x] = run;
            run += c;
        }
        uint32_t total;
        const uint32_t excl = block_excl_scan(run, s_warp, &total);
        s_base[threadIdx.x] = excl;
        s_out[threadIdx.x] = int64_t(before) - int64_t(excl);
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kSortItems; ++k) {
        const uint32_t pos = s_base[digit[k]] + s_cnt[warp][digit[k]] + rank[k];
        s_key[pos] = key[k];
        if (PAIRS) s_val[pos] = val[k];
    }
    __syncthreads();
    const int m = n - tile0 < kSortTile ? int(n - tile0) : kSortTile;  // the padding sorts last
#pragma unroll
    for (int k = 0; k < kSortItems; ++k) {
        const int i = k * kSortThreads + int(threadIdx.x);
        if (i >= m) break;
        const K v = s_key[i];
        const int64_t o = s_out[uint32_t(v >> shift) & 255u] + i;
        keys_out[o] = v;
        if (PAIRS) vals_out[o] = s_val[i];
    }
}

template <typename K, bool PAIRS, int ITEMS>
cudaError_t launch_small(K* keys, uint32_t* vals, int64_t n, int nbits, cudaStream_t s)
{
    const size_t smem = size_t(ITEMS) * kSmallThreads * (sizeof(K) + (PAIRS ? 4 : 0)) + kSmallWarps * 256 * 4;
    auto kern = radix_small_kernel<K, PAIRS, ITEMS>;
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
    if (e != cudaSuccess) return e;
    kern<<<1, kSmallThreads, smem, s>>>(keys, vals, int(n), nbits);
    note_launch();
    return cudaGetLastError();
}

template <typename K, bool PAIRS>
cudaError_t radix_sort(K* keys, uint32_t* vals, K* keys_alt, uint32_t* vals_alt, int64_t n, int nbits,
                       bool* result_in_alt, void* temp, cudaStream_t s)
{
    *result_in_alt = false;
    if (n <= 1 || nbits <= 0) return cudaSuccess;
    if (n <= kSmallThreads) return launch_small<K, PAIRS, 1>(keys, vals, n, nbits, s);
    if (n <= 2 * kSmallThreads) return launch_small<K, PAIRS, 2>(keys, vals, n, nbits, s);
    if (n <= 4 * kSmallThreads) return launch_small<K, PAIRS, 4>(keys, vals, n, nbits, s);
    if (n <= kSmallItems) return launch_small<K, PAIRS, 8>(keys, vals, n, nbits, s);
    const int64_t tiles = (n + kSortTile - 1) / kSortTile;
    const bool by_tile = tiles <= kColumnTiles;
    const int64_t nc = tiles * 256;
    uint32_t* counts = static_cast<uint32_t*>(temp);
    void* scan_tmp = static_cast<char*>(temp) + align_up(size_t(nc) * 4, 256);
    K *kin = keys, *kout = keys_alt;
    uint32_t *vin = vals, *vout = vals_alt;
    bool alt = false;
    for (int shift = 0; shift < nbits; shift += 8) {
        radix_hist_kernel<K><<<unsigned(tiles), kSortThreads, 0, s>>>(kin, n, shift, int(tiles), by_tile, counts);
        note_launch();
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
        if (by_tile) {
            radix_scatter_kernel<K, PAIRS, true>
                <<<unsigned(tiles), kSortThreads, 0, s>>>(kin, vin, n, shift, int(tiles), counts, kout, vout);
        } else {
            e = exclusive_scan_u32(counts, counts, nc, nullptr, scan_tmp, s);
            if (e != cudaSuccess) return e;
            radix_scatter_kernel<K, PAIRS, false>
                <<<unsigned(tiles), kSortThreads, 0, s>>>(kin, vin, n, shift, int(tiles), counts, kout, vout);
        }
        note_launch();
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
        std::swap(kin, kout);
        std::swap(vin, vout);
        alt = !alt;
    }
    *result_in_alt = alt;
    return cudaSuccess;
}

}  // namespace

size_t scan_temp_bytes(int64_t n)
{
    if (n <= kScanTile) return 256;
    const int64_t nb = (n + kScanTile - 1) / kScanTile;
    return align_up(size_t(nb) * 4, 256) + scan_temp_bytes(nb);
}

cudaError_t exclusive_scan_u32(const uint32_t* in, uint32_t* out, int64_t n, uint32_t* total, void* temp,
                               cudaStream_t s)
{
    if (n <= 0) {
        if (total) return cudaMemsetAsync(total, 0, sizeof(uint32_t), s);
        return cudaSuccess;
    }
    if (n <= kScanTile) {
        scan_apply_kernel<<<1, kScanThreads, 0, s>>>(in, out, n, nullptr, false, total);
        note_launch();
        return cudaGetLastError();
    }
    const int64_t nb = (n + kScanTile - 1) / kScanTile;
    uint32_t* sums = static_cast<uint32_t*>(temp);
    void* sub = static_cast<char*>(temp) + align_up(size_t(nb) * 4, 256);
    scan_reduce_kernel<<<unsigned(nb), kScanThreads, 0, s>>>(in, n, sums);
    note_launch();
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    const bool raw = nb <= kScanRawSums;
    if (!raw) {
        e = exclusive_scan_u32(sums, sums, nb, nullptr, sub, s);
        if (e != cudaSuccess) return e;
    }
    scan_apply_kernel<<<unsigned(nb), kScanThreads, 0, s>>>(in, out, n, sums, raw, total);
    note_launch();
    return cudaGetLastError();
}

bool radix_sort_is_small(int64_t n) { return n <= kSmallItems; }

size_t radix_temp_bytes(int64_t n)
{
    const int64_t nb = (n + kSortTile - 1) / kSortTile;
    const int64_t nc = nb * 256;
    return align_up(size_t(nc) * 4, 256) + scan_temp_bytes(nc);
}

cudaError_t radix_sort_pairs_u64(uint64_t* keys, uint32_t* vals, uint64_t* keys_alt, uint32_t* vals_alt, int64_t n,
                                 int nbits, bool* result_in_alt, void* temp, cudaStream_t s)
{
    if (vals) return radix_sort<uint64_t, true>(keys, vals, keys_alt, vals_alt, n, nbits, result_in_alt, temp, s);
    return radix_sort<uint64_t, false>(keys, nullptr, keys_alt, nullptr, n, nbits, result_in_alt, temp, s);
}

cudaError_t radix_sort_pairs_u32(uint32_t* keys, uint32_t* vals, uint32_t* keys_alt, uint32_t* vals_alt, int64_t n,
                                 int nbits, bool* result_in_alt, void* temp, cudaStream_t s)
{
    if (vals) return radix_sort<uint32_t, true>(keys, vals, keys_alt, vals_alt, n, nbits, result_in_alt, temp, s);
    return radix_sort<uint32_t, false>(keys, nullptr, keys_alt, nullptr, n, nbits, result_in_alt, temp, s);
}

}  // namespace mlods
