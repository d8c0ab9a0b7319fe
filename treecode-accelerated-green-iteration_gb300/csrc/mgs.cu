// Subsystem (e), part 1: quadrature-weighted Gram-Schmidt of one orbital,
// the device counterpart of modifiedGramSchmidt_singleWavefunction
// (3D-GreenIteration/src/utilities/Orthogonalization.c:14-119), one GPU, FP64:
//   r_i = sum_j V_ij U_j W_j          (i < target)         :44-54
//   U_j -= sum_i r_i V_ij  (i in order, per point)         :71-79
//   U  /= sqrt(sum_j U_j^2 W_j);  V[target] = U            :85-106
// The projections use the incoming U (classical order inside one call), as the
// reference does.  V's rows are read twice (dots, then subtract).
//
// Bound: one FP64 operation per element read would take the FP64 pipe (527 G
// DFMA/s measured) 8 bytes x 527 G = 4.2 TB/s, below the HBM rate, so FP64
// instructions are what is saved: fused multiply-adds, per-block sums that halve
// the rows at each shuffle (9 additions per warp for 8 rows instead of 40), a
// reciprocal refined by two fused multiply-adds in place of a division.  Three
// kernels whose launches overlap; the sums over blocks are formed by every block
// that needs them, in block order, so results do not depend on scheduling.
// 32 orbitals x 1M points, orbital after orbital: 8.26 -> 3.58 ms.
#include "tagi_internal.h"

#include <algorithm>
#include <cstdint>
#include <mutex>

namespace tagi {

namespace {

constexpr int MT = 256;
constexpr int MW = MT / 32;
constexpr int RB = 8;   // rows per thread in the dot kernel

// A point's value, or two neighbours' where every row is 16-byte aligned.
template <bool VEC>
struct Pts;
template <>
struct Pts<true> {
    typedef double2 T;
    static __device__ __forceinline__ double2 ld(const double *p, long i) { return reinterpret_cast<const double2 *>(p)[i]; }
    static __device__ __forceinline__ void st(double *p, long i, double2 v) { reinterpret_cast<double2 *>(p)[i] = v; }
    static __device__ __forceinline__ double2 mul(double2 a, double2 b) { return make_double2(a.x * b.x, a.y * b.y); }
    // u - r v
    static __device__ __forceinline__ double2 sub(double2 u, double r, double2 v) {
        return make_double2(__fma_rn(-r, v.x, u.x), __fma_rn(-r, v.y, u.y));
    }
    static __device__ __forceinline__ double dot(double2 a, double2 b, double acc) {
        return __fma_rn(a.y, b.y, __fma_rn(a.x, b.x, acc));
    }
};
template <>
struct Pts<false> {
    typedef double T;
    static __device__ __forceinline__ double ld(const double *p, long i) { return p[i]; }
    static __device__ __forceinline__ void st(double *p, long i, double v) { p[i] = v; }
    static __device__ __forceinline__ double mul(double a, double b) { return a * b; }
    static __device__ __forceinline__ double sub(double u, double r, double v) { return __fma_rn(-r, v, u); }
    static __device__ __forceinline__ double dot(double a, double b, double acc) { return __fma_rn(a, b, acc); }
};

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// partial[row][block] for the rows of this block's row group.  n: points (VEC:
// pairs of points), chunk: of them per block.
template <bool VEC>
__global__ void __launch_bounds__(MT) mgs_dots(const double *V, const double *U,
                                               const double *W, int target, long npts, long n, long chunk,
                                               double *partial) {
    typedef Pts<VEC> P;
    __shared__ double sh[RB][MW];
    chain_begin();
    const int r0 = blockIdx.y * RB, nr = min(RB, target - r0);
    const long j0 = (long)blockIdx.x * chunk, j1 = min(j0 + chunk, n);
    double acc[RB];
#pragma unroll
    for (int r = 0; r < RB; r++) acc[r] = 0.0;
    const double *v0 = V + (long)r0 * npts;
    if (nr == RB) {
        for (long j = j0 + threadIdx.x; j < j1; j += MT) {
            typename P::T v[RB];
#pragma unroll
            for (int r = 0; r < RB; r++) v[r] = P::ld(v0 + (long)r * npts, j);
            const typename P::T uw = P::mul(P::ld(U, j), P::ld(W, j));
#pragma unroll
            for (int r = 0; r < RB; r++) acc[r] = P::dot(v[r], uw, acc[r]);
        }
    } else {
        for (long j = j0 + threadIdx.x; j < j1; j += MT) {
            const typename P::T uw = P::mul(P::ld(U, j), P::ld(W, j));
#pragma unroll
            for (int r = 0; r < RB; r++)
                if (r < nr) acc[r] = P::dot(P::ld(v0 + (long)r * npts, j), uw, acc[r]);
        }
    }
    // the warp's sums of 8 rows: at each of three steps a lane keeps half of its rows,
    // then lanes of one row (equal lane & 7) are added
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int h = RB / 2, o = 4; h > 0; h >>= 1, o >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int r = 0; r < h; r++) {
            const double give = up ? acc[r] : acc[r + h], keep = up ? acc[r + h] : acc[r];
            acc[r] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
    }
    double s = acc[0];   // row: bit 2 of the lane chose the half of 4, bit 1 of 2, bit 0 of 1
    s += __shfl_xor_sync(0xffffffffu, s, 8);
    s += __shfl_xor_sync(0xffffffffu, s, 16);
    if (lane < RB) sh[lane][wid] = s;
    __syncthreads();
    if (threadIdx.x < nr) {
        double t = 0.0;
        for (int w = 0; w < MW; w++) t += sh[threadIdx.x][w];
        partial[(long)(r0 + threadIdx.x) * gridDim.x + blockIdx.x] = t;
    }
}

// U -= sum_i r_i V_i with r_i from the dot kernel's partials; norm partials.
constexpr int SROWS = 128;   // projections held in shared memory at a time
template <bool VEC>
__global__ void __launch_bounds__(MT) mgs_subtract(const double *V, double *U,
                                                   const double *W, const double *partial,
                                                   int nblk, int target, long npts, long n, long chunk,
                                                   double *npart) {
    typedef Pts<VEC> P;
    __shared__ double s_r[SROWS], sh[MW];
    chain_begin();
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const long j0 = (long)blockIdx.x * chunk, j1 = min(j0 + chunk, n);
    double acc = 0.0;
    for (int i0 = 0; i0 == 0 || i0 < target; i0 += SROWS) {
        const int ni = min(SROWS, target - i0);
        __syncthreads();
        for (int i = wid; i < ni; i += MW) {
            const double *p = partial + (long)(i0 + i) * nblk;
            double t = 0.0;
            for (int b = lane; b < nblk; b += 32) t += p[b];
            t = warp_sum(t);
            if (lane == 0) s_r[i] = t;
        }
        __syncthreads();
        const double *v0 = V + (long)i0 * npts;
        const bool last = i0 + SROWS >= target;
        for (long j = j0 + threadIdx.x; j < j1; j += MT) {
            typename P::T u = P::ld(U, j);
            int i = 0;
            for (; i + 8 <= ni; i += 8) {
                typename P::T v[8];
#pragma unroll
                for (int q = 0; q < 8; q++) v[q] = P::ld(v0 + (long)(i + q) * npts, j);
#pragma unroll
                for (int q = 0; q < 8; q++) u = P::sub(u, s_r[i + q], v[q]);
            }
#pragma unroll 4
            for (; i < ni; i++) u = P::sub(u, s_r[i], P::ld(v0 + (long)i * npts, j));
            P::st(U, j, u);
            if (last) acc = P::dot(u, P::mul(u, P::ld(W, j)), acc);
        }
    }
    acc = warp_sum(acc);
    if (lane == 0) sh[wid] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < MW; w++) t += sh[w];
        npart[blockIdx.x] = t;
    }
}

// u / norm to the last place from the reciprocal: q = u inv, then one correction by
// the exact remainder (P. W. Markstein, IBM J. Res. Dev. 34, 1990; q itself where it is not finite).
__device__ __forceinline__ double divide(double u, double norm, double inv) {
    const double q = __dmul_rn(u, inv);
    const double c = __fma_rn(__fma_rn(-q, norm, u), inv, q);
    return ((unsigned)__double2hiint(q) & 0x7ff00000u) == 0x7ff00000u ? q : c;
}

template <bool VEC>
__global__ void __launch_bounds__(MT) mgs_normalize(double *V, double *U,
                                                    const double *npart, int nblk, int target, long npts,
                                                    long n, long chunk) {
    typedef Pts<VEC> P;
    __shared__ double s_norm;
    chain_begin();
    if (threadIdx.x < 32) {
        double s = 0.0;
        for (int b = threadIdx.x; b < nblk; b += 32) s += npart[b];
        s = warp_sum(s);
        if (threadIdx.x == 0) s_norm = sqrt(s);
    }
    __syncthreads();
    const double nrm = s_norm, inv = 1.0 / nrm;
    const bool plain = !(nrm > 1e-290 && nrm < 1e290);   // zero, tiny, huge or NaN: the division itself
    const long j0 = (long)blockIdx.x * chunk, j1 = min(j0 + chunk, n);
    double *vt = V + (long)target * npts;
    for (long j = j0 + threadIdx.x; j < j1; j += MT) {
        typename P::T u = P::ld(U, j);
        if constexpr (VEC)
            u = plain ? make_double2(u.x / nrm, u.y / nrm) : make_double2(divide(u.x, nrm, inv), divide(u.y, nrm, inv));
        else
            u = plain ? u / nrm : divide(u, nrm, inv);
        P::st(U, j, u);
        P::st(vt, j, u);
    }
}

// Blocks of the dot kernel (per row group) and of the point-wise kernels: enough
// for a few per SM, in whole turns of a block.
struct MgsGrid {
    bool vec;
    long n, dchunk, chunk;   // points or pairs; per block
    int dblk, groups, nblk;
};
MgsGrid mgs_grid(const double *V, const double *U, const double *W, int target, long npts, int sms) {
    MgsGrid g;
    auto aligned = [](const void *p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; };
    g.vec = npts % 2 == 0 && aligned(V) && aligned(U) && aligned(W);
    g.n = g.vec ? npts / 2 : npts;
    g.groups = std::max(1, (target + RB - 1) / RB);
    auto cut = [&](long blocks, long &chunk) {
        chunk = (g.n + blocks - 1) / blocks;
        chunk = (chunk + MT - 1) / MT * MT;
        return (int)((g.n + chunk - 1) / chunk);
    };
    g.dblk = cut(std::max(1L, 3L * sms / g.groups), g.dchunk);
    g.nblk = cut(4L * sms, g.chunk);
    return g;
}
// Doubles of scratch: the dot partials, then the norm partials.
size_t mgs_scratch(const MgsGrid &g, int target) { return (size_t)g.dblk * target + g.nblk; }

template <bool VEC>
int mgs_launch(double *V, double *U, const double *W, int target, long npts, const MgsGrid &g, double *scratch,
               cudaStream_t s) {
    double *partial = scratch, *npart = scratch + (size_t)g.dblk * target;
    if (target > 0)
        TAGI_CUDA(launch_chained(mgs_dots<VEC>, dim3(g.dblk, g.groups), MT, 0, s, V, U, W, target, npts, g.n, g.dchunk,
                                 partial));
    TAGI_CUDA(launch_chained(mgs_subtract<VEC>, g.nblk, MT, 0, s, V, U, W, partial, g.dblk, target, npts, g.n, g.chunk,
                             npart));
    TAGI_CUDA(launch_chained(mgs_normalize<VEC>, g.nblk, MT, 0, s, V, U, npart, g.nblk, target, npts, g.n, g.chunk));
    return TAGI_OK;
}
int mgs_run(double *V, double *U, const double *W, int target, long npts, const MgsGrid &g, double *scratch,
            cudaStream_t s) {
    return g.vec ? mgs_launch<true>(V, U, W, target, npts, g, scratch, s)
                 : mgs_launch<false>(V, U, W, target, npts, g, scratch, s);
}

int sm_count(int *sms) {
    int dev = 0;
    TAGI_CUDA(cudaGetDevice(&dev));
    TAGI_CUDA(cudaDeviceGetAttribute(sms, cudaDevAttrMultiProcessorCount, dev));
    return TAGI_OK;
}

}  // namespace

int mgs_device(double *V, double *U, const double *W, int target, int npts, int nwave,
               cudaStream_t s) {
    if (npts <= 0) return TAGI_OK;
    if (target < 0 || target >= nwave)
        return set_error(TAGI_ERR_ARG, "targetWavefunction %d outside [0, %d)", target, nwave);
    int sms = 0;
    TAGI_TRY(sm_count(&sms));
    const MgsGrid g = mgs_grid(V, U, W, target, npts, sms);
    Arena tmp;
    tmp.stream = s;
    double *scratch = nullptr;
    TAGI_TRY(tmp.alloc(&scratch, mgs_scratch(g, target)));
    const int rc = mgs_run(V, U, W, target, npts, g, scratch, s);
    tmp.release();
    return rc;
}

}  // namespace tagi

// ---------------------------------------------------------------------------
// Weighted Gram-Schmidt without any device allocation.
//
// Some callers cannot allocate device memory while they run: a process whose
// device memory is handed entirely to another allocator (a framework's caching
// pool, a fixed per-job budget), or a latency-critical Green-iteration loop in
// which a cudaMalloc/cudaFree would synchronize the device and stall other
// streams.  tagi_mgs_dev_noalloc does the same work as tagi_mgs_dev with its
// scratch (per-block partial sums, projection coefficients, norm partials) in
// the fixed device array below instead of freshly allocated memory.
//
// * The array is MGS_NOALLOC_BLOCKS x (MGS_NOALLOC_ROWS + 1) + MGS_NOALLOC_ROWS
//   doubles (about 1.06 MB): at most 768 blocks' dot partials of 128 rows (fewer
//   blocks per row the more rows) and 1024 norm partials; every GPU that loads this library holds it until
//   the process exits.  Requests with targetWavefunction > MGS_NOALLOC_ROWS are
//   rejected with TAGI_ERR_ARG.
// * Host code cannot use the array's name as a device address: the first call
//   on each device (with that device current) looks the address up with
//   cudaGetSymbolAddress and keeps it.  Make that first call before any stream
//   capture.
// * All calls share the array and it keeps the last call's contents.  Every
//   entry a call reads is written earlier in the same call, so nothing needs
//   clearing; two calls that overlap on the GPU (different streams, or
//   different host threads on one device) race on it.
// ---------------------------------------------------------------------------
namespace tagi {
namespace {

constexpr int MGS_NOALLOC_BLOCKS = 1024;
constexpr int MGS_NOALLOC_ROWS = 128;
constexpr long MGS_NOALLOC_DOUBLES =
    (long)MGS_NOALLOC_BLOCKS * (MGS_NOALLOC_ROWS + 1) + MGS_NOALLOC_ROWS;

static __device__ __align__(256) double g_mgs_noalloc_scratch[MGS_NOALLOC_DOUBLES];

std::mutex g_mgs_noalloc_mu;
double *g_mgs_noalloc_ptr[64] = {};

int mgs_noalloc_scratch(double **out) {
    int dev = 0;
    TAGI_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return set_error(TAGI_ERR_DEVICE, "device ordinal %d out of range", dev);
    std::lock_guard<std::mutex> lk(g_mgs_noalloc_mu);
    if (!g_mgs_noalloc_ptr[dev]) {
        void *p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_mgs_noalloc_scratch);
        if (e != cudaSuccess || !p)
            return set_error(TAGI_ERR_CUDA, "cudaGetSymbolAddress of the MGS scratch array failed: %s",
                             cudaGetErrorString(e));
        g_mgs_noalloc_ptr[dev] = static_cast<double *>(p);
    }
    *out = g_mgs_noalloc_ptr[dev];
    return TAGI_OK;
}

}  // namespace

}  // namespace tagi

extern "C" int tagi_mgs_dev_noalloc(double *V, double *U, const double *W, int targetWavefunction,
                                    int numPoints, int numWavefunctions, void *stream) {
    using namespace tagi;
    if (numPoints < 0 || numWavefunctions < 1) return set_error(TAGI_ERR_ARG, "bad MGS sizes");
    if (targetWavefunction < 0 || targetWavefunction >= numWavefunctions)
        return set_error(TAGI_ERR_ARG, "targetWavefunction %d outside [0, %d)", targetWavefunction,
                         numWavefunctions);
    if (targetWavefunction > MGS_NOALLOC_ROWS)
        return set_error(TAGI_ERR_ARG,
                         "tagi_mgs_dev_noalloc handles targetWavefunction <= %d (got %d); use tagi_mgs_dev",
                         MGS_NOALLOC_ROWS, targetWavefunction);
    if (numPoints == 0) return TAGI_OK;
    if (!V || !U || !W) return set_error(TAGI_ERR_ARG, "null device pointer");
    cudaStream_t s = (cudaStream_t)stream;
    double *scratch = nullptr;
    TAGI_TRY(mgs_noalloc_scratch(&scratch));
    int sms = 0;
    TAGI_TRY(sm_count(&sms));
    // at most 256 SMs' worth of blocks, so that both partials fit the array
    const MgsGrid g = mgs_grid(V, U, W, targetWavefunction, numPoints, std::min(sms, MGS_NOALLOC_BLOCKS / 4));
    return mgs_run(V, U, W, targetWavefunction, numPoints, g, scratch, s);
}

