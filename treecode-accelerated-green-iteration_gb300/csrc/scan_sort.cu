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

constexpr int RS_THREADS = 256;
constexpr int RS_ROUNDS = 8;
constexpr int RS_TILE = RS_THREADS * RS_ROUNDS;
constexpr int RS_WARPS = RS_THREADS / 32;

__global__ void __launch_bounds__(RS_THREADS) rs_histogram(const uint64_t *__restrict__ keys,
                                                           int n, int shift,
                                                           int *__restrict__ hist, int nblocks) {
    __shared__ int cnt[256];
    cnt[threadIdx.x] = 0;
    __syncthreads();
    const long base = (long)blockIdx.x * RS_TILE;
    for (int r = 0; r < RS_ROUNDS; r++) {
        long i = base + (long)r * RS_THREADS + threadIdx.x;
        if (i < n) atomicAdd(&cnt[(int)((keys[i] >> shift) & 255u)], 1);
    }
    __syncthreads();
    hist[(long)threadIdx.x * nblocks + blockIdx.x] = cnt[threadIdx.x];
}

// Stable scatter: elements of a tile are ranked in index order, warp by warp,
// round by round; ties between tiles follow block order via the scanned
// digit-major histogram.
__global__ void __launch_bounds__(RS_THREADS) rs_scatter(const uint64_t *__restrict__ kin,
                                                         const int *__restrict__ vin,
                                                         uint64_t *__restrict__ kout,
                                                         int *__restrict__ vout, int n, int shift,
                                                         const int *__restrict__ offs,
                                                         int nblocks) {
    __shared__ int base[256];
    __shared__ int wcnt[RS_WARPS][256];
    base[threadIdx.x] = offs[(long)threadIdx.x * nblocks + blockIdx.x];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const unsigned lt = (1u << lane) - 1u;
    const long tile = (long)blockIdx.x * RS_TILE;
    for (int r = 0; r < RS_ROUNDS; r++) {
#pragma unroll
        for (int w = 0; w < RS_WARPS; w++) wcnt[w][threadIdx.x] = 0;
        __syncthreads();
        long i = tile + (long)r * RS_THREADS + threadIdx.x;
        bool valid = i < n;
        uint64_t k = valid ? kin[i] : 0;
        int v = valid ? vin[i] : 0;
        int d = valid ? (int)((k >> shift) & 255u) : 256 + lane;  // invalid lanes stay alone
        unsigned peers = __match_any_sync(0xffffffffu, d);
        int rank = __popc(peers & lt);
        if (valid && rank == 0) wcnt[wid][d] = __popc(peers);
        __syncthreads();
        {
            int dd = threadIdx.x;
            int run = base[dd];
#pragma unroll
            for (int w = 0; w < RS_WARPS; w++) {
                int c = wcnt[w][dd];
                wcnt[w][dd] = run;
                run += c;
            }
            base[dd] = run;
        }
        __syncthreads();
        if (valid) {
            int pos = wcnt[wid][d] + rank;
            kout[pos] = k;
            vout[pos] = v;
        }
        __syncthreads();
    }
}

// Up to SORT_SMALL pairs by counting: an element's place is the number of smaller
// keys plus the equal keys before it.  n^2 comparisons over the whole chip take
// 3 us at 6,000 keys and 25 at 16,384, where the radix passes are 40 launches (about
// 100 us) and a bitonic network in one block took 124.  Counts are whole numbers:
// the order of the atomic additions does not matter.
constexpr int SORT_SMALL = 16384, CNT_THREADS = 256;
__global__ void __launch_bounds__(CNT_THREADS) count_smaller(const uint64_t *__restrict__ keys,
                                                             const int *__restrict__ vals, int n, int span,
                                                             int *__restrict__ rank, uint64_t *__restrict__ kcopy,
                                                             int *__restrict__ vcopy) {
    __shared__ uint64_t s_key[CNT_THREADS];
    const int i = blockIdx.x * CNT_THREADS + threadIdx.x;
    const uint64_t k = i < n ? keys[i] : 0;
    const int j0 = blockIdx.y * span, j1 = min(j0 + span, n);
    int c = 0;
    for (int t = j0; t < j1; t += CNT_THREADS) {
        const int m = min(CNT_THREADS, j1 - t);
        __syncthreads();
        if (threadIdx.x < m) s_key[threadIdx.x] = keys[t + threadIdx.x];
        __syncthreads();
#pragma unroll 8
        for (int j = 0; j < m; j++) {
            const uint64_t q = s_key[j];
            c += q < k || (q == k && t + j < i);
        }
    }
    if (i >= n) return;
    if (c) atomicAdd(rank + i, c);
    if (blockIdx.y == 0) {
        kcopy[i] = k;
        vcopy[i] = vals[i];
    }
}
__global__ void place_sorted(const uint64_t *__restrict__ kcopy, const int *__restrict__ vcopy,
                             const int *__restrict__ rank, int n, uint64_t *__restrict__ keys, int *__restrict__ vals) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int r = rank[i];
    keys[r] = kcopy[i];
    vals[r] = vcopy[i];
}

}  // namespace

int radix_sort_u64(uint64_t *keys, int *vals, int n, Arena &ar, cudaStream_t s) {
    if (n <= 1) return TAGI_OK;
    if (n <= SORT_SMALL) {
        uint64_t *kc = nullptr;
        int *vc = nullptr, *rank = nullptr;
        TAGI_TRY(ar.alloc(&kc, n));
        TAGI_TRY(ar.alloc(&vc, n));
        TAGI_TRY(ar.alloc(&rank, n));
        TAGI_CUDA(cudaMemsetAsync(rank, 0, sizeof(int) * n, s));
        const int bx = (n + CNT_THREADS - 1) / CNT_THREADS;
        const int by = std::min(bx, (152 * 8 + bx - 1) / bx);   // about eight blocks per SM
        const int span = (n + by - 1) / by;
        launch(count_smaller, dim3(bx, (n + span - 1) / span), CNT_THREADS, 0, s, keys, vals, n, span, rank, kc, vc);
        launch(place_sorted, bx, CNT_THREADS, 0, s, kc, vc, rank, n, keys, vals);
        TAGI_LAUNCH_CHECK();
        return TAGI_OK;
    }
    int nb = (n + RS_TILE - 1) / RS_TILE;
    uint64_t *k2 = nullptr;
    int *v2 = nullptr, *hist = nullptr, *offs = nullptr;
    TAGI_TRY(ar.alloc(&k2, n));
    TAGI_TRY(ar.alloc(&v2, n));
    TAGI_TRY(ar.alloc(&hist, 256L * nb));
    TAGI_TRY(ar.alloc(&offs, 256L * nb));
    uint64_t *ka = keys, *kb = k2;
    int *va = vals, *vb = v2;
    for (int shift = 0; shift < 64; shift += 8) {
        launch(rs_histogram, nb, RS_THREADS, 0, s, ka, n, shift, hist, nb);
        TAGI_LAUNCH_CHECK();
        TAGI_TRY(exclusive_scan(hist, offs, 256 * nb, nullptr, ar, s));
        launch(rs_scatter, nb, RS_THREADS, 0, s, ka, va, kb, vb, n, shift, offs, nb);
        TAGI_LAUNCH_CHECK();
        uint64_t *kt = ka; ka = kb; kb = kt;
        int *vt = va; va = vb; vb = vt;
    }
    // 8 passes: the result is back in the caller's buffers.
    return TAGI_OK;
}

}  // namespace tagi
