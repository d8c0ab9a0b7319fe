// Device-wide exclusive scan (int32) and stable LSD radix sort of 64-bit
// Morton codes with int32 payloads.  Integer work for the tree build: the
// sort fixes the point order every later kernel reads, so it must be stable
// (equal codes keep caller order) to give lists identical to the CPU oracle,
// which sorts by (code, index).
#include "tagi_internal.h"

#include <algorithm>

namespace tagi {

namespace {

constexpr int SCAN_THREADS = 1024;
constexpr int SCAN_ITEMS = 4;
constexpr int SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;

__device__ __forceinline__ int warp_incl_scan(int v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

// Exclusive scan of one tile per block; writes the tile total to sums[block].
__global__ void __launch_bounds__(SCAN_THREADS) scan_tiles(const int *__restrict__ in,
                                                           int *__restrict__ out, int n,
                                                           int *__restrict__ sums) {
    __shared__ int warp_tot[SCAN_THREADS / 32];
    const long base = (long)blockIdx.x * SCAN_TILE + (long)threadIdx.x * SCAN_ITEMS;
    int v[SCAN_ITEMS];
    int tsum = 0;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; k++) {
        long i = base + k;
        v[k] = (i < n) ? in[i] : 0;
        tsum += v[k];
    }
    int incl = warp_incl_scan(tsum);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 31) warp_tot[wid] = incl;
    __syncthreads();
    if (wid == 0) {
        int w = warp_tot[lane];
        int wi = warp_incl_scan(w);
        warp_tot[lane] = wi - w;
        if (lane == 31) sums[blockIdx.x] = wi;
    }
    __syncthreads();
    int run = warp_tot[wid] + incl - tsum;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; k++) {
        long i = base + k;
        if (i < n) out[i] = run;
        run += v[k];
    }
}

__global__ void add_tile_offsets(int *__restrict__ out, int n, const int *__restrict__ offs) {
    const long base = (long)blockIdx.x * SCAN_TILE;
    const int add = offs[blockIdx.x];
    for (int k = threadIdx.x; k < SCAN_TILE; k += blockDim.x) {
        long i = base + k;
        if (i < n) out[i] += add;
    }
}

// Exclusive scan by one block, a tile at a time, total included: up to SCAN_SMALL
// elements one launch is quicker than tiles, their sums and the offsets (5,104
// cells: 4 launches of 2-3 us each before).
constexpr int SCAN_SMALL = 4 * SCAN_TILE;
__global__ void __launch_bounds__(SCAN_THREADS) scan_small(const int *__restrict__ in, int *__restrict__ out, int n,
                                                           int *__restrict__ total) {
    __shared__ int warp_tot[SCAN_THREADS / 32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int carry = 0;
    for (int base = 0; base < n; base += SCAN_TILE) {
        int v[SCAN_ITEMS], tsum = 0;
#pragma unroll
        for (int k = 0; k < SCAN_ITEMS; k++) {
            const int i = base + threadIdx.x * SCAN_ITEMS + k;
            v[k] = i < n ? in[i] : 0;
            tsum += v[k];
        }
        const int incl = warp_incl_scan(tsum);
        __syncthreads();   // the previous tile's warp totals are no longer read
        if (lane == 31) warp_tot[wid] = incl;
        __syncthreads();
        int before = 0, all = 0;
        const int wt = warp_tot[lane], ws = warp_incl_scan(wt);
        all = __shfl_sync(0xffffffffu, ws, 31);
        before = __shfl_sync(0xffffffffu, ws - wt, wid);
        int run = carry + before + incl - tsum;
#pragma unroll
        for (int k = 0; k < SCAN_ITEMS; k++) {
            const int i = base + threadIdx.x * SCAN_ITEMS + k;
            if (i < n) out[i] = run;
            run += v[k];
        }
        carry += all;
    }
    if (total && threadIdx.x == 0) *total = carry;
}

}  // namespace

int exclusive_scan(const int *in, int *out, int n, int *d_total, Arena &ar, cudaStream_t s) {
    if (n <= 0) {
        if (d_total) TAGI_CUDA(cudaMemsetAsync(d_total, 0, sizeof(int), s));
        return TAGI_OK;
    }
    if (n <= SCAN_SMALL) {
        launch(scan_small, 1, SCAN_THREADS, 0, s, in, out, n, d_total);
        TAGI_LAUNCH_CHECK();
        return TAGI_OK;
    }
    int nb = (n + SCAN_TILE - 1) / SCAN_TILE;
    int *sums = nullptr;
    TAGI_TRY(ar.alloc(&sums, nb + 1));
    launch(scan_tiles, nb, SCAN_THREADS, 0, s, in, out, n, sums);
    TAGI_LAUNCH_CHECK();
    int *offs = nullptr;
    TAGI_TRY(ar.alloc(&offs, nb));
    TAGI_TRY(exclusive_scan(sums, offs, nb, d_total, ar, s));
    launch(add_tile_offsets, nb, 256, 0, s, out, n, offs);
    TAGI_LAUNCH_CHECK();
    return TAGI_OK;
}

namespace {

// Radix passes: two chained launches per digit.  Bound: launch latency up to some
// 200,000 keys, then L2 (12 bytes in, 12 out, scattered).  A block of the scatter adds up
// where its tile's digits go from the tiles' counts, those of whole groups of tiles
// first, so no scan runs between the two kernels: at 1.5M keys (367 tiles) a block reads
// 23 rows of group sums and up to 15 rows of its group's tiles, 512 counts each.  Nine-bit digits: 63-bit Morton codes take seven passes; 512 counters for
// each of eight warps are 16 KB of shared memory.  Digits of eight bits with a scan
// between took 24 launches (40 above 130,000 keys).  44,000 keys: 60 us.
constexpr int RS_THREADS = 256, RS_WARPS = RS_THREADS / 32, RS_BITS = 9, RS_DIGITS = 1 << RS_BITS;

// counts[tile][digit], and their sums over groups of `group` tiles (zeroed before)
template <int ROUNDS>
__global__ void __launch_bounds__(RS_THREADS) rs_histogram(const uint64_t *keys, int n, int shift, int group,
                                                           int *counts, int *sums) {
    __shared__ int cnt[RS_DIGITS];
    for (int d = threadIdx.x; d < RS_DIGITS; d += RS_THREADS) cnt[d] = 0;
    chain_begin();
    __syncthreads();
    const long base = (long)blockIdx.x * ROUNDS * RS_THREADS;
#pragma unroll
    for (int r = 0; r < ROUNDS; r++) {
        const long i = base + (long)r * RS_THREADS + threadIdx.x;
        if (i < n) atomicAdd(&cnt[(int)(keys[i] >> shift) & (RS_DIGITS - 1)], 1);
    }
    __syncthreads();
    for (int d = threadIdx.x; d < RS_DIGITS; d += RS_THREADS) {
        const int c = cnt[d];
        counts[(long)blockIdx.x * RS_DIGITS + d] = c;
        if (c) atomicAdd(sums + (long)(blockIdx.x / group) * RS_DIGITS + d, c);
    }
}

// Stable scatter.  Each warp owns 32 ROUNDS consecutive keys of the tile and ranks them
// in order with its own counters; a column scan over the warps and the tile's start
// of each digit turn the ranks into places.
template <int ROUNDS>
__global__ void __launch_bounds__(RS_THREADS) rs_scatter(const uint64_t *kin, const int *vin,
                                                         uint64_t *kout, int *vout, int n,
                                                         int shift, int group, int ngroups,
                                                         const int *counts, const int *sums) {
    __shared__ int wcnt[RS_WARPS][RS_DIGITS];
    __shared__ int wtot[RS_WARPS];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, tile = blockIdx.x;
    for (int d = tid; d < RS_WARPS * RS_DIGITS; d += RS_THREADS) (&wcnt[0][0])[d] = 0;
    chain_begin();
    // digits 2 tid and 2 tid + 1: keys before this tile, and keys in all
    int2 before = make_int2(0, 0), all = make_int2(0, 0);
    const int mine = tile / group;
#pragma unroll 8
    for (int g = 0; g < ngroups; g++) {
        const int2 c = reinterpret_cast<const int2 *>(sums + (long)g * RS_DIGITS)[tid];
        all.x += c.x;
        all.y += c.y;
        if (g < mine) before.x += c.x, before.y += c.y;
    }
#pragma unroll 8
    for (int t = mine * group; t < tile; t++) {
        const int2 c = reinterpret_cast<const int2 *>(counts + (long)t * RS_DIGITS)[tid];
        before.x += c.x;
        before.y += c.y;
    }
    const int incl = warp_incl_scan(all.x + all.y);
    if (lane == 31) wtot[wid] = incl;
    __syncthreads();
    int first = incl - all.x - all.y;
    for (int w = 0; w < wid; w++) first += wtot[w];
    uint64_t k[ROUNDS];
    int place[ROUNDS];
    const long base = (long)tile * ROUNDS * RS_THREADS + (long)wid * ROUNDS * 32 + lane;
#pragma unroll
    for (int r = 0; r < ROUNDS; r++) k[r] = base + 32 * r < n ? kin[base + 32 * r] : 0;
#pragma unroll
    for (int r = 0; r < ROUNDS; r++) {
        const bool valid = base + 32 * r < n;
        const int d = (int)(k[r] >> shift) & (RS_DIGITS - 1);
        const unsigned peers = __match_any_sync(0xffffffffu, valid ? d : RS_DIGITS + lane);   // invalid lanes stay alone
        const int rank = __popc(peers & ((1u << lane) - 1u)), c = valid ? wcnt[wid][d] : 0;
        place[r] = c + rank;
        __syncwarp();
        if (valid && rank == 0) wcnt[wid][d] = c + __popc(peers);
        __syncwarp();
    }
    __syncthreads();
    int2 run = make_int2(first + before.x, first + all.x + before.y);
#pragma unroll
    for (int w = 0; w < RS_WARPS; w++) {
        int2 *p = reinterpret_cast<int2 *>(&wcnt[w][2 * tid]);
        const int2 c = *p;
        *p = run;
        run.x += c.x;
        run.y += c.y;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < ROUNDS; r++) {
        const long i = base + 32 * r;
        if (i < n) {
            const int p = place[r] + wcnt[wid][(int)(k[r] >> shift) & (RS_DIGITS - 1)];
            kout[p] = k[r];
            vout[p] = vin[i];
        }
    }
}

template <int ROUNDS>
int rs_pass(const uint64_t *kin, const int *vin, uint64_t *kout, int *vout, int n, int shift, int nb, int group,
            int *counts, int *sums, cudaStream_t s) {
    TAGI_CUDA(launch_chained(rs_histogram<ROUNDS>, nb, RS_THREADS, 0, s, kin, n, shift, group, counts, sums));
    TAGI_CUDA(launch_chained(rs_scatter<ROUNDS>, nb, RS_THREADS, 0, s, kin, vin, kout, vout, n, shift, group,
                             (nb + group - 1) / group, counts, sums));
    return TAGI_OK;
}

// Up to SORT_SMALL pairs by counting: an element's place is the number of smaller
// keys plus the equal keys before it.  n^2 comparisons over the whole chip: 16 us at
// 6,022 keys, 47 at 15,336 (the radix passes 60 at 44,000; at 16,384 they are even); a
// bitonic network in one block took 124 at 6,022.  Counts are whole numbers:
// the order of the atomic additions does not matter.
constexpr int SORT_SMALL = 16384, CNT_THREADS = 256;
__global__ void __launch_bounds__(CNT_THREADS) count_smaller(const uint64_t *keys,
                                                             int n, int span, int *rank) {
    __shared__ __align__(16) uint64_t s_key[CNT_THREADS];
    chain_begin();
    const int i0 = blockIdx.x * CNT_THREADS, i = i0 + threadIdx.x;
    const uint64_t k = i < n ? keys[i] : 0;
    const int j0 = blockIdx.y * span, j1 = min(j0 + span, n);
    int c = 0;
    for (int t = j0; t < j1; t += CNT_THREADS) {
        const int m = min(CNT_THREADS, j1 - t);
        __syncthreads();
        if (threadIdx.x < m) s_key[threadIdx.x] = keys[t + threadIdx.x];
        __syncthreads();
        // equal keys count where they lie before this one: all or none of a tile that lies
        // before or after the block's keys, which leaves one comparison
        if (t + m <= i0) {
#pragma unroll 8
            for (int j = 0; j < m; j++) c += s_key[j] <= k;
        } else if (t >= i0 + CNT_THREADS) {
#pragma unroll 8
            for (int j = 0; j < m; j++) c += s_key[j] < k;
        } else {
#pragma unroll 4
            for (int j = 0; j < m; j++) {
                const uint64_t q = s_key[j];
                c += q < k || (q == k && t + j < i);
            }
        }
    }
    if (i < n && c) atomicAdd(rank + i, c);
}
__global__ void place_sorted(const uint64_t *kin, const int *vin, const int *rank,
                             int n, uint64_t *kout, int *vout) {
    chain_begin();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int r = rank[i];
    kout[r] = kin[i];
    vout[r] = vin[i];
}

}  // namespace

int radix_sort_u64(uint64_t *kin, int *vin, uint64_t *kout, int *vout, int n, int bits, Arena &ar, cudaStream_t s) {
    if (n <= 0) return TAGI_OK;
    if (n <= SORT_SMALL) {
        int *rank = nullptr;
        TAGI_TRY(ar.alloc(&rank, n));
        TAGI_CUDA(cudaMemsetAsync(rank, 0, sizeof(int) * n, s));
        const int bx = (n + CNT_THREADS - 1) / CNT_THREADS;
        const int by = std::min(bx, ((int)GPU_SMS * 8 + bx - 1) / bx);   // about eight blocks per SM
        const int span = (n + by - 1) / by;
        launch(count_smaller, dim3(bx, (n + span - 1) / span), CNT_THREADS, 0, s, kin, n, span, rank);
        TAGI_CUDA(launch_chained(place_sorted, bx, CNT_THREADS, 0, s, kin, vin, rank, n, kout, vout));
        TAGI_LAUNCH_CHECK();
        return TAGI_OK;
    }
    // one or two tiles per SM, so that the chain of one tile is short; larger ones mean fewer rows of counts
    const int rounds = n > 1 << 18 ? 16 : n > 1 << 17 ? 8 : 2, tile = RS_THREADS * rounds;
    const int nb = (int)(((long)n + tile - 1) / tile);
    const int group = nb <= 1024 ? 16 : 64, ngroups = (nb + group - 1) / group, passes = (bits + RS_BITS - 1) / RS_BITS;
    int *counts = nullptr, *sums = nullptr;
    const long row = (long)ngroups * RS_DIGITS;
    TAGI_TRY(ar.alloc(&counts, (long)nb * RS_DIGITS));
    TAGI_TRY(ar.alloc(&sums, passes * row));
    TAGI_CUDA(cudaMemsetAsync(sums, 0, sizeof(int) * passes * row, s));
    for (int p = 0; p < passes; p++) {
        const bool odd = p & 1;
        TAGI_TRY((rounds == 16 ? rs_pass<16> : rounds == 8 ? rs_pass<8> : rs_pass<2>)(odd ? kout : kin, odd ? vout : vin, odd ? kin : kout, odd ? vin : vout, n,
                                                    RS_BITS * p, nb, group, counts, sums + p * row, s));
    }
    TAGI_LAUNCH_CHECK();
    if (passes % 2 == 0) {
        TAGI_CUDA(cudaMemcpyAsync(kout, kin, sizeof(uint64_t) * n, cudaMemcpyDeviceToDevice, s));
        TAGI_CUDA(cudaMemcpyAsync(vout, vin, sizeof(int) * n, cudaMemcpyDeviceToDevice, s));
    }
    return TAGI_OK;
}

}  // namespace tagi
