// radix_sort.cu -- stable LSD radix sort of (key, value) pairs and an exclusive scan, on the device.
//
// One kernel counts every pass' 8-bit digits, and each pass is then a single kernel after Adinets and
// Merrill's "Onesweep" (2022): a tile ranks its keys by digit (inside a warp with __match_any_sync, across the
// tile's warps through shared memory), learns how many equal digits the tiles before it hold by looking back
// over their published counts, scans the digit counts for itself (a kernel of its own for that cost 4 us a
// sort) and writes its keys in runs. Keys and values cross memory twice a pass, in one launch and one per
// pass: a pass of histogram, table scan (three launches) and scatter read the keys twice and moved a 256-entry
// table per 256 keys. 30-bit keys, us before -> after: 4,000,000 450 -> 256, 500,003 92 -> 45. Used by the BVH
// builder (30-bit Morton keys), the pseudo-normal pass (vertex ids, 64-bit edge keys) and point lists.
#include <cuda_runtime.h>

#include "internal.h"

namespace ssdf_b200 {

namespace {

constexpr int kSortThreads = 256;  // one per digit value
constexpr int kSortItems = 8;      // keys a thread takes
constexpr int kSortTile = kSortThreads * kSortItems;
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kScanThreads = 1024;
constexpr int kScanItems = 4;
constexpr int kScanBlock = kScanThreads * kScanItems;

// Digit counts of every pass (counts[pass * 256 + digit], zeroed before).
template <typename K>
__global__ void __launch_bounds__(kSortThreads) k_digit_counts(const K *__restrict__ keys, int n, int passes,
                                                               unsigned *__restrict__ counts) {
    __shared__ unsigned hist[8][256];
    for (int p = 0; p < passes; p++) hist[p][threadIdx.x] = 0;
    __syncthreads();
    for (long long i = blockIdx.x * (long long)kSortThreads + threadIdx.x; i < n; i += (long long)gridDim.x * kSortThreads) {
        const K key = keys[i];
        for (int p = 0; p < passes; p++) atomicAdd(&hist[p][int((key >> (8 * p)) & 0xff)], 1u);
    }
    __syncthreads();
    for (int p = 0; p < passes; p++) {
        const unsigned c = hist[p][threadIdx.x];
        if (c) atomicAdd(&counts[p * 256 + threadIdx.x], c);
    }
}

// Exclusive scan of one value per thread over the block of kSortThreads (warp_tot: kSortWarps words of shared memory).
__device__ __forceinline__ unsigned block_exclusive(unsigned v, unsigned *warp_tot) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) warp_tot[warp] = incl;
    __syncthreads();
    unsigned before = 0;
    for (int w = 0; w < warp; w++) before += warp_tot[w];
    return before + incl - v;
}

// A tile's published word for a digit: state in the low two bits (0: nothing yet), count above.
constexpr unsigned long long kTileOwn = 1;   // the tile's own count
constexpr unsigned long long kTileUpTo = 2;  // the count of all tiles up to this one
// Polls of a word before the tile counts its predecessors' keys itself. Tiles are numbered in the order they
// start, so a predecessor is always running and the wait is short; the bound only makes that unconditional.
constexpr int kMaxPolls = 1 << 16;

// One pass. tile_words: [tile * 256 + digit], zeroed before; next_tile: zeroed before. ALONE: tiles look at no word
// and count for themselves (SSDF_B200_SORT_ALONE=1, for tests; an instantiation of its own, since polls given as
// an argument cost 15 us of 5,285 on 4,000,000 points).
template <typename K, bool ALONE>
__global__ void __launch_bounds__(kSortThreads) k_sort_pass(const K *__restrict__ kin, const int *__restrict__ vin,
                                                            K *__restrict__ kout, int *__restrict__ vout, int n,
                                                            int shift, const unsigned *__restrict__ counts,
                                                            unsigned long long *tile_words, int *next_tile) {
    __shared__ unsigned cnt[kSortWarps][256];
    __shared__ unsigned tile_start[256], to_global[256];
    __shared__ unsigned warp_tot[kSortWarps], digit_tot[kSortWarps];
    __shared__ int s_tile;
    __shared__ K s_key[kSortTile];
    __shared__ int s_val[kSortTile];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, digit = threadIdx.x;
    if (threadIdx.x == 0) s_tile = atomicAdd(next_tile, 1);
    const unsigned digit_count = counts[digit];
    for (int w = 0; w < kSortWarps; w++) cnt[w][digit] = 0;
    __syncthreads();
    const int tile = s_tile;
    const long long base = (long long)tile * kSortTile;
    // a warp's keys are consecutive, an item a row of 32: the ranks below keep their order
    K key[kSortItems];
    int val[kSortItems];
    unsigned rank[kSortItems];
#pragma unroll
    for (int k = 0; k < kSortItems; k++) {
        const long long i = base + warp * (32 * kSortItems) + k * 32 + lane;
        key[k] = i < n ? kin[i] : K(0);
        val[k] = i < n ? vin[i] : 0;
    }
    const unsigned lt = (1u << lane) - 1u;
#pragma unroll
    for (int k = 0; k < kSortItems; k++) {
        const bool valid = base + warp * (32 * kSortItems) + k * 32 + lane < n;
        const int d = int((key[k] >> shift) & 0xff);
        const unsigned peers = __match_any_sync(0xffffffffu, valid ? d : 256 + lane);
        const unsigned before = valid ? cnt[warp][d] : 0;
        rank[k] = before + __popc(peers & lt);
        __syncwarp();
        if (valid && (__ffs(peers) - 1) == lane) cnt[warp][d] = before + __popc(peers);
        __syncwarp();
    }
    __syncthreads();
    unsigned total = 0;  // thread = digit: the warps' offsets inside the tile's digit
    for (int w = 0; w < kSortWarps; w++) {
        const unsigned c = cnt[w][digit];
        cnt[w][digit] = total;
        total += c;
    }
    volatile unsigned long long *const mine = tile_words + (long long)tile * 256 + digit;
    *mine = (unsigned long long)total << 2 | (tile == 0 ? kTileUpTo : kTileOwn);
    tile_start[digit] = block_exclusive(total, warp_tot);
    const unsigned digit_start = block_exclusive(digit_count, digit_tot);
    __syncthreads();
    // the tile's keys in digit order, while the words travel
#pragma unroll
    for (int k = 0; k < kSortItems; k++) {
        if (base + warp * (32 * kSortItems) + k * 32 + lane < n) {
            const int d = int((key[k] >> shift) & 0xff);
            const unsigned at = tile_start[d] + cnt[warp][d] + rank[k];
            s_key[at] = key[k];
            s_val[at] = val[k];
        }
    }
    // how many keys of this digit the tiles before hold
    unsigned long long prev = 0;
    for (int t = tile - 1; t >= 0; t--) {
        volatile const unsigned long long *const word = tile_words + (long long)t * 256 + digit;
        unsigned long long w = ALONE ? 0 : *word;
        if (!ALONE)
            for (int poll = 0; (w & 3) == 0 && poll < kMaxPolls; poll++) w = *word;
        if ((w & 3) == 0) {  // count tile t's keys
            const long long end = (long long)(t + 1) * kSortTile;
            for (long long i = (long long)t * kSortTile; i < end; i++) prev += int((kin[i] >> shift) & 0xff) == digit;
            continue;
        }
        prev += w >> 2;
        if ((w & 3) == kTileUpTo) break;
    }
    if (tile > 0) *mine = (prev + total) << 2 | kTileUpTo;
    to_global[digit] = digit_start + unsigned(prev) - tile_start[digit];
    __syncthreads();
    const int m = int(n - base < kSortTile ? n - base : kSortTile);
    for (int i = threadIdx.x; i < m; i += kSortThreads) {
        const K k = s_key[i];
        const unsigned pos = to_global[int((k >> shift) & 0xff)] + unsigned(i);
        kout[pos] = k;
        vout[pos] = s_val[i];
    }
}

// Block-local exclusive scan of kScanBlock items; block totals to `sums` (if not null).
__global__ void __launch_bounds__(kScanThreads) k_scan_block(const int *__restrict__ in, int *__restrict__ out,
                                                             int n, int *__restrict__ sums) {
    __shared__ int warp_tot[kScanThreads / 32];
    const int base = blockIdx.x * kScanBlock + threadIdx.x * kScanItems;
    int v[kScanItems];
    int tsum = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; k++) {
        v[k] = (base + k < n) ? in[base + k] : 0;
        tsum += v[k];
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int incl = tsum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) warp_tot[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        int w = warp_tot[lane];
        int wi = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, wi, o);
            if (lane >= o) wi += t;
        }
        warp_tot[lane] = wi - w;
        if (lane == 31 && sums) sums[blockIdx.x] = wi;
    }
    __syncthreads();
    int run = warp_tot[warp] + incl - tsum;
#pragma unroll
    for (int k = 0; k < kScanItems; k++) {
        if (base + k < n) out[base + k] = run;
        run += v[k];
    }
}

__global__ void k_add_block_offsets(int *__restrict__ out, int n, const int *__restrict__ offs) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] += offs[i / kScanBlock];
}

}  // namespace

// Exclusive scan of n ints (out may alias in). Scratch is stream-ordered.
int exclusive_scan_i32(const int *in, int *out, int n, cudaStream_t stream) {
    if (n <= 0) return SSDF_OK;
    const int nblocks = (n + kScanBlock - 1) / kScanBlock;
    if (nblocks == 1) {
        k_scan_block<<<1, kScanThreads, 0, stream>>>(in, out, n, nullptr);
        SSDF_CUDA(cudaGetLastError());
        return SSDF_OK;
    }
    int *sums = nullptr;
    SSDF_CUDA(cudaMallocAsync(&sums, sizeof(int) * nblocks, stream));
    k_scan_block<<<nblocks, kScanThreads, 0, stream>>>(in, out, n, sums);
    SSDF_CUDA(cudaGetLastError());
    int st = exclusive_scan_i32(sums, sums, nblocks, stream);
    if (st == SSDF_OK) {
        k_add_block_offsets<<<grid_blocks(n, 256), 256, 0, stream>>>(out, n, sums);
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) st = cuda_fail(e, "k_add_block_offsets", __FILE__, __LINE__);
    }
    cudaFreeAsync(sums, stream);
    return st;
}

template <typename K>
static int radix_sort_pairs(K *keys, int *vals, int n, int key_bits, cudaStream_t stream) {
    if (n <= 1) return SSDF_OK;
    const int ntiles = int(((long long)n + kSortTile - 1) / kSortTile);
    const int passes = (key_bits + 7) / 8;
    const bool alone = env_int("SSDF_B200_SORT_ALONE", 0) != 0;
    // scratch: the second keys and values, then (zeroed) the tile words, the digit counts and the tile tickets
    const size_t words = size_t(passes) * ntiles * 256 * sizeof(unsigned long long);
    const size_t zeroed = words + size_t(passes) * 256 * sizeof(unsigned) + size_t(passes) * sizeof(int);
    const size_t kb = (sizeof(K) * size_t(n) + 15) / 16 * 16, vb = (sizeof(int) * size_t(n) + 15) / 16 * 16;
    char *scratch = nullptr;
    if (cudaMallocAsync(&scratch, kb + vb + zeroed, stream) != cudaSuccess)
        return fail(SSDF_ERR_OUT_OF_MEMORY, "radix sort scratch");
    K *k2 = reinterpret_cast<K *>(scratch);
    int *v2 = reinterpret_cast<int *>(scratch + kb);
    auto *tile_words = reinterpret_cast<unsigned long long *>(scratch + kb + vb);
    auto *counts = reinterpret_cast<unsigned *>(scratch + kb + vb + words);
    int *tickets = reinterpret_cast<int *>(counts + passes * 256);
    cudaError_t e = cudaMemsetAsync(tile_words, 0, zeroed, stream);
    if (e == cudaSuccess) {
        const int blocks = ntiles < 148 * 4 ? ntiles : 148 * 4;  // at most four an SM
        k_digit_counts<K><<<blocks, kSortThreads, 0, stream>>>(keys, n, passes, counts);
        e = cudaGetLastError();
    }
    K *kin = keys, *kout = k2;
    int *vin = vals, *vout = v2;
    for (int p = 0; p < passes && e == cudaSuccess; p++) {
        unsigned long long *const pass_words = tile_words + size_t(p) * ntiles * 256;
        if (alone)
            k_sort_pass<K, true><<<ntiles, kSortThreads, 0, stream>>>(kin, vin, kout, vout, n, 8 * p, counts + p * 256,
                                                                      pass_words, tickets + p);
        else
            k_sort_pass<K, false><<<ntiles, kSortThreads, 0, stream>>>(kin, vin, kout, vout, n, 8 * p, counts + p * 256,
                                                                       pass_words, tickets + p);
        e = cudaGetLastError();
        K *tk = kin;
        kin = kout;
        kout = tk;
        int *tv = vin;
        vin = vout;
        vout = tv;
    }
    if (e == cudaSuccess && kin != keys) {
        e = cudaMemcpyAsync(keys, kin, sizeof(K) * size_t(n), cudaMemcpyDeviceToDevice, stream);
        if (e == cudaSuccess) e = cudaMemcpyAsync(vals, vin, sizeof(int) * size_t(n), cudaMemcpyDeviceToDevice, stream);
    }
    cudaFreeAsync(scratch, stream);
    return e == cudaSuccess ? SSDF_OK : cuda_fail(e, "radix sort", __FILE__, __LINE__);
}

int radix_sort_pairs_u32(uint32_t *keys, int *vals, int n, int key_bits, cudaStream_t stream) {
    return radix_sort_pairs<uint32_t>(keys, vals, n, key_bits, stream);
}
int radix_sort_pairs_u64(uint64_t *keys, int *vals, int n, int key_bits, cudaStream_t stream) {
    return radix_sort_pairs<uint64_t>(keys, vals, n, key_bits, stream);
}

}  // namespace ssdf_b200
