// Subsystem (b): upward pass.  For every far-field cluster ("slot") the
// modified charges on its (n+1)^3 Chebyshev 2nd-kind proxy grid,
//     qhat_k = sum_{j in cluster} L_k1(u_jx) L_k2(u_jy) L_k3(u_jz) q_j ,
// with the barycentric Lagrange basis on nodes cos(m pi / n) and weights
// (-1)^m (halved at both ends), u = (y - c) / h in the slot's proxy box.
// k = (k1 * (n+1) + k2) * (n+1) + k3, x-major like the reference's cells.
//
// Work items are (slot, chunk of sorted sources); each item writes FP64 partial
// sums and a second kernel adds the partials of a slot in item order, so results
// do not depend on scheduling.  The weight charges (q = w) are built once per plan;
// charge vectors are done per call, in FP32 products summed over a tile of 64
// sources, the tiles' sums then accumulated to about 72 bits (mixed), or all in
// FP64.
//
// Bound (mixed): FP32 issue.  A tile's sums were added in FP64, whose pipe (1/64 of
// the FP32 rate) took three quarters of the kernel; they now go into three FP32
// words by two-sums (72 bits, 13 FP32 operations, two at a time in packed form,
// in place of one FP64 addition), and a CTA shares a tile's basis values between
// P2M_OB orbitals.  32 orbitals x 1M points 29.3 -> 14.8 ms; 6k points, one charge
// vector, chunks of 256 sources instead of 2048 157 -> 28 us.
#include "tagi_internal.h"

namespace tagi {

namespace {

constexpr int P2M_THREADS = 256;
constexpr int P2M_TILE = 64;

template <typename T>
struct P2MArgs {
    const int *item_slot, *item_begin, *item_end;
    int nitems;
    const double *geom;          // [slot][6]
    const double *xs, *ys, *zs;  // sorted sources
    const T *q;                  // [norb][ns] sorted charges
    long q_stride;
    const T *w;                  // the last vector, if it lies elsewhere (weights)
    double *part;                // [norb][nitems][P]
    int n1, P, norb;
    T tn[MAX_DEGREE + 1];
};

template <typename T>
__device__ __forceinline__ const T *charges(const P2MArgs<T> &a, int orb) {
    return a.w && orb == a.norb - 1 ? a.w : a.q + (long)orb * a.q_stride;
}

template <typename T>
__device__ __forceinline__ T bary_weight(int m, int n1) {
    T w = (m & 1) ? T(-1) : T(1);
    if (m == 0 || m == n1 - 1) w *= T(0.5);
    return w;
}

// A sum of floats in three words, each the rounding error of the one before.
struct Sum3 {
    float2 hi, mid, lo;
};
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __fadd2_rn(a, make_float2(-b.x, -b.y)); }
__device__ __forceinline__ float2 two_sum(float2 &s, float2 v) {   // s += v; returns the error (Knuth)
    const float2 t = __fadd2_rn(s, v), w = sub2(t, s);
    const float2 e = __fadd2_rn(sub2(s, sub2(t, w)), sub2(v, w));
    s = t;
    return e;
}
__device__ __forceinline__ void add(Sum3 &a, float2 v) {
    a.lo = __fadd2_rn(a.lo, two_sum(a.mid, two_sum(a.hi, v)));
}
// The words' sum.  An infinite first word has NaN errors: it is the sum, as in FP64.
__device__ __forceinline__ double total(float hi, float mid, float lo) {
    return fabsf(hi) < INFINITY ? (double)hi + ((double)mid + (double)lo) : (double)hi;
}

// a / h from inv = 1 / h: the product corrected by its exact remainder, which gives the rounded
// quotient (P. W. Markstein, IBM J. Res. Dev. 34, 1990).  The product alone can fall on the other
// side of a tie when it is rounded to FP32.
__device__ __forceinline__ double quotient(double a, double h, double inv) {
    if (!(h > 1e-290 && h < 1e290)) return a / h;
    const double q = __dmul_rn(a, inv);
    return __fma_rn(__fma_rn(-q, h, a), inv, q);
}

// Barycentric basis values of the coordinate that lies at u in the slot's box ([-1, 1]) along one
// axis, into L[0..n1-1].
template <typename T>
__device__ __forceinline__ void basis(T u, const T *tn, int n1, T *L) {
    int exact = -1;
    for (int m = 0; m < n1; m++)
        if (u - tn[m] == T(0)) exact = m;
    if (exact >= 0) {
        for (int m = 0; m < n1; m++) L[m] = (m == exact) ? T(1) : T(0);
    } else {
        T s = T(0);
        for (int m = 0; m < n1; m++) {
            T l = bary_weight<T>(m, n1) / (u - tn[m]);
            L[m] = l;
            s += l;
        }
        for (int m = 0; m < n1; m++) L[m] = L[m] / s;
    }
}

// Mixed: OB orbitals of one item.  Thread (g, k1, k2) sums the sources g, g + G, ...
// of each tile for its row of the grid.
constexpr int P2M_OB = 3;   // upward pass of 32 orbitals x 1M points at 2, 3, 4: 18.3, 14.8, 25.0 ms (registers)
// Resident CTAs per SM: one orbital needs few registers, and 50k points are 6 us quicker with four CTAs
// than with three.
template <int MAXN1, int OB>
__global__ void __launch_bounds__(P2M_THREADS, OB > 1 ? 2 : (MAXN1 <= 8 ? 4 : 3)) p2m_mixed(const __grid_constant__ P2MArgs<float> a) {
    constexpr int MH = (MAXN1 + 1) / 2, LP = 2 * MH;
    extern __shared__ double red[];  // [G][P]
    __shared__ __align__(8) float sL[3][P2M_TILE][LP];
    __shared__ float sq[OB][P2M_TILE];
    const int item = blockIdx.x, orb0 = blockIdx.y * OB, no = min(OB, a.norb - orb0);
    const int n1 = a.n1, pairs = n1 * n1, P = a.P;
    const int G = P2M_THREADS / pairs;
    const int tid = threadIdx.x;
    const int g = tid / pairs, pr = tid % pairs;
    const int k1 = pr / n1, k2 = pr % n1;
    const bool active = g < G;
    chain_begin();
    const int b = a.item_begin[item], e = a.item_end[item];
    const double *gm = a.geom + 6L * a.item_slot[item];
    const int axis = tid % 3;   // thread 3 p + d does source p along axis d
    const double *xs = axis == 0 ? a.xs : (axis == 1 ? a.ys : a.zs);
    const double center = gm[axis], width = gm[3 + axis], inv = 1.0 / width;
    Sum3 acc[OB][MH];
#pragma unroll
    for (int o = 0; o < OB; o++)
#pragma unroll
        for (int m = 0; m < MH; m++) acc[o][m].hi = acc[o][m].mid = acc[o][m].lo = make_float2(0.f, 0.f);
    for (int t0 = b; t0 < e; t0 += P2M_TILE) {
        const int cnt = min(P2M_TILE, e - t0);
        __syncthreads();   // the previous tile is no longer read
        if (tid < 3 * cnt) {
            float *L = sL[axis][tid / 3];
            basis<float>((float)quotient(xs[t0 + tid / 3] - center, width, inv), a.tn, n1, L);
            if (n1 & 1) L[n1] = 0.f;   // the second lane of the last pair
        }
        for (int k = tid; k < OB * P2M_TILE; k += P2M_THREADS) {
            const int o = k / P2M_TILE, p = k % P2M_TILE;
            if (o < no && p < cnt) sq[o][p] = charges(a, orb0 + o)[t0 + p];
        }
        __syncthreads();
        if (!active) continue;
#pragma unroll
        for (int o = 0; o < OB; o++) {
            if (o >= no) break;
            float2 t[MH];
#pragma unroll
            for (int m = 0; m < MH; m++) t[m] = make_float2(0.f, 0.f);
            for (int p = g; p < cnt; p += G) {
                const float axy = sL[0][p][k1] * sL[1][p][k2] * sq[o][p];
                const float2 ax = make_float2(axy, axy);
#pragma unroll
                for (int m = 0; m < MH; m++)
                    if (2 * m < n1) t[m] = __ffma2_rn(ax, *reinterpret_cast<const float2 *>(&sL[2][p][2 * m]), t[m]);
            }
#pragma unroll
            for (int m = 0; m < MH; m++)
                if (2 * m < n1) add(acc[o][m], t[m]);
        }
    }
#pragma unroll
    for (int o = 0; o < OB; o++) {
        if (o >= no) break;
        __syncthreads();   // red of the previous orbital is no longer read
        if (active) {
            double *r = red + (long)g * P + (long)pr * n1;
#pragma unroll
            for (int m = 0; m < MH; m++) {
                const Sum3 &v = acc[o][m];
                if (2 * m < n1) r[2 * m] = total(v.hi.x, v.mid.x, v.lo.x);
                if (2 * m + 1 < n1) r[2 * m + 1] = total(v.hi.y, v.mid.y, v.lo.y);
            }
        }
        __syncthreads();
        double *out = a.part + ((long)(orb0 + o) * a.nitems + item) * P;
        for (int k = tid; k < P; k += P2M_THREADS) {
            double s = 0.0;
            for (int gg = 0; gg < G; gg++) s += red[(long)gg * P + k];
            out[k] = s;
        }
    }
}

template <int MAXN1>
__global__ void __launch_bounds__(P2M_THREADS) p2m_f64(const __grid_constant__ P2MArgs<double> a) {
    extern __shared__ double red[];  // [G][P]
    __shared__ double sL[3][P2M_TILE][MAXN1];
    __shared__ double sq[P2M_TILE];
    const int item = blockIdx.x, orb = blockIdx.y;
    const int n1 = a.n1, pairs = n1 * n1, P = a.P;
    const int G = P2M_THREADS / pairs;
    const int tid = threadIdx.x;
    const int g = tid / pairs, pr = tid % pairs;
    const int k1 = pr / n1, k2 = pr % n1;
    const bool active = g < G;
    chain_begin();
    const int slot = a.item_slot[item];
    const int b = a.item_begin[item], e = a.item_end[item];
    const double *gm = a.geom + 6L * slot;
    const double *q = charges(a, orb);

    double acc[MAXN1];
#pragma unroll
    for (int m = 0; m < MAXN1; m++) acc[m] = 0.0;

    for (int t0 = b; t0 < e; t0 += P2M_TILE) {
        const int cnt = min(P2M_TILE, e - t0);
        if (tid < 3 * cnt) {
            const int p = tid / 3, d = tid - 3 * (tid / 3);
            const double *src = d == 0 ? a.xs : (d == 1 ? a.ys : a.zs);
            basis<double>((src[t0 + p] - gm[d]) / gm[3 + d], a.tn, n1, sL[d][p]);
        }
        if (tid < cnt) sq[tid] = q[t0 + tid];
        __syncthreads();
        if (active) {
            for (int p = g; p < cnt; p += G) {
                const double axy = sL[0][p][k1] * sL[1][p][k2] * sq[p];
#pragma unroll
                for (int m = 0; m < MAXN1; m++)
                    if (m < n1) acc[m] += axy * sL[2][p][m];
            }
        }
        __syncthreads();
    }
    if (active) {
#pragma unroll
        for (int m = 0; m < MAXN1; m++)
            if (m < n1) red[(long)g * P + (k1 * n1 + k2) * n1 + m] = acc[m];
    }
    __syncthreads();
    double *out = a.part + ((long)orb * a.nitems + item) * P;
    for (int k = tid; k < P; k += P2M_THREADS) {
        double s = 0.0;
        for (int gg = 0; gg < G; gg++) s += red[(long)gg * P + k];
        out[k] = s;
    }
}

template <typename TO>
__global__ void p2m_reduce(const double *part, const int *slot_item_off,
                           int nslots, int nitems, int P, TO *out, TO *wout) {
    const int slot = blockIdx.x, orb = blockIdx.y;
    chain_begin();
    const int i0 = slot_item_off[slot], i1 = slot_item_off[slot + 1];
    const double *pp = part + (long)orb * nitems * P;
    TO *o = wout && orb == (int)gridDim.y - 1 ? wout + (long)slot * P : out + ((long)orb * nslots + slot) * P;
    // a thread per grid point: its sum over the items is a chain, whose loads go out eight at
    // a time (50k points, degree 7: 19 us behind the sums with 256 threads per slot, now 5)
    const int k = blockIdx.z * blockDim.x + threadIdx.x;
    if (k < P) {
        double s = 0.0;
#pragma unroll 8
        for (int it = i0; it < i1; it++) s += pp[(long)it * P + k];
        o[k] = (TO)s;
    }
}

template <typename T>
int launch_p2m(Plan &p, const T *q, long q_stride, int norb, double *part, cudaStream_t s, const T *w = nullptr) {
    P2MArgs<T> a;
    a.item_slot = p.item_slot;
    a.item_begin = p.item_begin;
    a.item_end = p.item_end;
    a.nitems = p.nitems;
    a.geom = p.slot_geom;
    a.xs = p.src.x;
    a.ys = p.src.y;
    a.zs = p.src.z;
    a.q = q;
    a.q_stride = q_stride;
    a.w = w;
    a.part = part;
    a.n1 = p.n1;
    a.P = p.P;
    for (int m = 0; m <= MAX_DEGREE; m++) a.tn[m] = (T)(m <= p.degree ? p.cheb[m] : 0.0);
    const int G = P2M_THREADS / (p.n1 * p.n1);
    const size_t smem = sizeof(double) * (size_t)G * p.P;
    a.norb = norb;
    auto go = [&](auto kern, int ob) {
        if (smem > 32 * 1024) cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        return launch_chained(kern, dim3(p.nitems, (norb + ob - 1) / ob), P2M_THREADS, smem, s, a);
    };
    cudaError_t e;
    if constexpr (sizeof(T) == 8) {
        if (p.n1 <= 8) e = go(p2m_f64<8>, 1);
        else e = go(p2m_f64<MAX_DEGREE + 1>, 1);
    } else if (p.n1 <= 8) {
        if (norb == 1) e = go(p2m_mixed<8, 1>, 1);
        else e = go(p2m_mixed<8, P2M_OB>, P2M_OB);
    } else {   // 11 sums of three words per orbital: two orbitals fill the registers
        if (norb == 1) e = go(p2m_mixed<MAX_DEGREE + 1, 1>, 1);
        else e = go(p2m_mixed<MAX_DEGREE + 1, 2>, 2);
    }
    TAGI_CUDA(e);
    return TAGI_OK;
}

template <typename TO>
cudaError_t launch_reduce(const Plan &p, int rows, const double *part, TO *out, TO *wout, cudaStream_t s) {
    return launch_chained(p2m_reduce<TO>, dim3(p.nslots, rows, (p.P + 63) / 64), 64, 0, s, part, p.slot_item_off, p.nslots, p.nitems, p.P,
                          out, wout);
}

}  // namespace

// Weight modified charges (q = w).  The mixed path uses charges built with
// the same FP32 products as its charge vectors, so qhat - f_i what keeps the
// subtraction's structure; the FP64 set is built on first use by an FP64 call.
int build_weight_charges(Plan &p, cudaStream_t s) {
    TAGI_TRY(p.arena.alloc(&p.what32, (size_t)p.nslots * p.P));
    p.what64_ready = false;
    if (p.nslots == 0) return TAGI_OK;
    Arena tmp;
    tmp.stream = s;
    double *part = nullptr;
    int rc = tmp.alloc(&part, (size_t)p.nitems * p.P);
    if (!rc) rc = launch_p2m<float>(p, p.sw32, p.src.n, 1, part, s);
    if (!rc) {
        if (launch_reduce<float>(p, 1, part, p.what32, nullptr, s) != cudaSuccess) rc = set_error(TAGI_ERR_CUDA, "weight charge kernels");
    }
    tmp.release();
    return rc;
}

int ensure_weight_charges64(Plan &p, cudaStream_t s) {
    if (p.what64_ready) return TAGI_OK;
    if (!p.what64) {
        const size_t count = (size_t)p.nslots * p.P + 1;
        // plain cudaMalloc: the first FP64 call may run on another stream than the plan's
        void *v = nullptr;
        TAGI_CUDA(device_malloc(&v, sizeof(double) * count));
        p.arena.ptrs.push_back(v);
        p.what64 = static_cast<double *>(v);
    }
    if (p.nslots) {
        Arena tmp;
        tmp.stream = s;
        double *part = nullptr;
        int rc = tmp.alloc(&part, (size_t)p.nitems * p.P);
        if (!rc) rc = launch_p2m<double>(p, p.sw64, p.src.n, 1, part, s);
        if (!rc) {
            if (launch_reduce<double>(p, 1, part, p.what64, nullptr, s) != cudaSuccess) rc = set_error(TAGI_ERR_CUDA, "weight charge kernels");
        }
        tmp.release();
        if (rc) return rc;
    }
    p.what64_ready = true;
    return TAGI_OK;
}

// Charges for norb sorted charge vectors already in p.q32 / p.q64.  A one-shot plan has
// no weight charges yet: they ride along as one more vector (two launches and a chain of
// 23 us less at 6,000 points).
template <typename T>
static int charges_with_weights(Plan &p, const T *q, const T *w, int norb, T *qhat, T **what, cudaStream_t s) {
    if (p.one_shot && !*what) TAGI_TRY(p.arena.alloc(what, (size_t)p.nslots * p.P));
    T *const wout = p.one_shot ? *what : nullptr;
    const int rows = norb + (wout ? 1 : 0);
    TAGI_TRY(launch_p2m<T>(p, q, p.src.n, rows, p.part, s, wout ? w : nullptr));
    TAGI_CUDA(launch_reduce<T>(p, rows, p.part, qhat, wout, s));
    return TAGI_OK;
}

int modified_charges(Plan &p, int precision, int norb, cudaStream_t s) {
    if (p.nslots == 0) return TAGI_OK;
    if (precision == PREC_MIXED) return charges_with_weights<float>(p, p.q32, p.sw32, norb, p.qhat32, &p.what32, s);
    TAGI_TRY(charges_with_weights<double>(p, p.q64, p.sw64, norb, p.qhat64, &p.what64, s));
    if (p.one_shot) p.what64_ready = true;
    return TAGI_OK;
}

}  // namespace tagi
