// Subsystem (e), part 2: cell-wise Chebyshev interpolation between two
// meshes, the device counterpart of InterpolateBetweenTwoMeshes /
// interapolateBetweenTwoMeshesSingleCell
// (3D-GreenIteration/src/utilities/TwoMeshInterpolation.c:12-153,163-234), FP64.
//
// Semantics kept from the reference:
//  * coarseN == fineN: fineF = coarseF (overwrite) and nothing else   :175-180
//  * a cell whose coarse and fine counts match adds coarseF to fineF  :202-205,228-230
//  * otherwise fineF += barycentric interpolant of the coarse cell      :147
//  * nodes are read from the coarse cell assuming x-major order        :40-44
//  * first-kind weights (-1)^i sin((2i+1) pi / (2p+2))                 :49-51
//  * exact-node guard |t - node| < DBL_MIN; as in the reference, the x and z
//    exact-node tests compare against the z and x loop indices (:127,:139)
// Two to eight CTAs per cell share its children, each with the coarse values in shared
// memory; fine points on tensor grids (the mesh builders' layout) take a sum-factorised
// path, any other point the reference's per-point formula (see interp_cells).
#include "tagi_internal.h"

#include <cfloat>
#include <cmath>

namespace tagi {

namespace {

constexpr int IT = 128;
constexpr int MAXP1 = 12;

struct Weights {
    double w[MAXP1];
};

// One fine point by the reference's formula (TwoMeshInterpolation.c:59-147):
// per-axis barycentric terms w_k / (t - node_k), the exact-node guard with its
// swapped x/z index tests, the tensor sum with y innermost, times the
// product of the inverse sums.
template <int MAXP>
__device__ __noinline__ double interp_point(double tx, double ty, double tz, const double *s_c, const double *s_nx,
                                            const double *s_ny, const double *s_nz, const double *s_w) {
    constexpr int p1 = MAXP;
    double sx = 0.0, sy = 0.0, sz = 0.0;
    int eix = -1, eiy = -1, eiz = -1;
    double ax[MAXP], ay[MAXP], az[MAXP];
    for (int k = 0; k < p1; k++) {
        const double dx = tx - s_nx[k], dy = ty - s_ny[k], dz = tz - s_nz[k];
        if (fabs(dx) < DBL_MIN) eix = k;
        if (fabs(dy) < DBL_MIN) eiy = k;
        if (fabs(dz) < DBL_MIN) eiz = k;
        ax[k] = s_w[k] / dx;
        ay[k] = s_w[k] / dy;
        az[k] = s_w[k] / dz;
        sx += ax[k];
        sy += ay[k];
        sz += az[k];
    }
    double den = 1.0;
    if (eix == -1) den /= sx;
    if (eiy == -1) den /= sy;
    if (eiz == -1) den /= sz;
    // y factor depends on k2 only; x and z factors as in the reference.
    for (int k = 0; k < p1; k++) ay[k] = (eiy == -1) ? ay[k] : (eiy == k ? 1.0 : 0.0);
    double temp = 0.0;
    for (int k3 = 0; k3 < p1; k3++) {
        for (int k1 = 0; k1 < p1; k1++) {
            const double fx = (eix == -1) ? ax[k3] : (eix == k1 ? 1.0 : 0.0);
            const double fz = (eiz == -1) ? az[k1] : (eiz == k3 ? 1.0 : 0.0);
            const double fxz = fx * fz;
            if (fxz == 0.0) continue;
            const double *col = s_c + k3 * p1 * p1 + k1;
            double g = 0.0;
            for (int k2 = 0; k2 < p1; k2++) g += ay[k2] * col[k2 * p1];
            temp += fxz * g;
        }
    }
    return temp * den;
}

// Two to eight CTAs per cell.  A cell's fine points come in blocks of (p+1)^3 (one block
// per child cell), each CTA's following one another.  When a block is a tensor grid in
// x-major order (x depends on the block index i only, y on j, z on k -- the
// layout the mesh builders write) and none of its 1-D coordinates sits on a
// coarse node, the interpolant is the sum-factorised product
//     out[a][b][c] = sum_i Lx[a][i] sum_j Ly[b][j] sum_k Lz[c][k] F[i][j][k],
//     Lx[a][i] = (w_i / (x_a - xn_i)) / sum_i' (w_i' / (x_a - xn_i'))
// (three 1-D contractions: 3 (p+1)^4 multiply-adds per block instead of
// ~(p+1)^6); otherwise every point of the block takes the reference's
// per-point formula (interp_point).  Both agree to rounding.
//
// The kernel is bound by the FP64 pipe.  The children of a cell come x-major, so
// consecutive blocks share their x coordinates (and pairs of them x and y): the x
// contraction is formed once per change of x, the y contraction once per change
// of x or y, bit patterns compared -- 14 (p+1) multiply-adds per 8 points of 8
// children instead of 24, 39 instead of 81 per 27 points of 27.  The rows of 1-D
// weights are divided out by all threads: in one thread per row the divisions of a
// single warp held up the block as long as its contractions.  Ring molecule, 14.3M fine
// points, order 7: 1184 -> 571 us a call.
template <int p1>
__global__ void __launch_bounds__(IT, 10) interp_cells(
    const double *__restrict__ cX, const double *__restrict__ cY, const double *__restrict__ cZ,
    const double *__restrict__ cF, const int *__restrict__ ppc_c, const int *__restrict__ off_c,
    const double *__restrict__ fX, const double *__restrict__ fY, const double *__restrict__ fZ,
    double *__restrict__ fF, const int *__restrict__ ppc_f, const int *__restrict__ off_f,
    int ncells, int coarseN, int fineN, const __grid_constant__ Weights wts, int *__restrict__ err) {
    constexpr int p2 = p1 * p1, p3 = p2 * p1;
    __shared__ double s_c[p3];
    __shared__ double s_t[2][p3];                // contracted over x; over x and y
    __shared__ double s_f0[2][p1];               // the x and y coordinates that they belong to
    __shared__ double s_L[3][p2];        // Lx, Ly, Lz: [fine index][node]
    __shared__ double s_sum[3][p1], s_inv[3][p1];   // sums of their rows, reciprocals
    __shared__ double s_f[3][p1];                // the block's 1-D fine coordinates
    __shared__ double s_nx[p1], s_ny[p1], s_nz[p1], s_w[p1];
    // the cells' points must fit the arrays: nothing is read or written otherwise
    if (off_c[ncells] > coarseN || off_f[ncells] > fineN) {
        if (threadIdx.x == 0) atomicOr(err, 2);
        return;
    }
    const int cell = blockIdx.x;
    const int nc = ppc_c[cell], nf = ppc_f[cell];
    const int c0 = off_c[cell], f0 = off_f[cell];
    const int tid = threadIdx.x;
    const int part = blockIdx.y, parts = gridDim.y;
    if (nc == nf) {
        if (part) return;
        for (int j = tid; j < nf; j += IT) fF[f0 + j] = fF[f0 + j] + cF[c0 + j];
        return;
    }
    if (nc != p3) {  // a coarse cell must hold the full (p+1)^3 grid
        if (tid == 0) atomicOr(err, 1);
        return;
    }
    for (int j = tid; j < nc; j += IT) s_c[j] = cF[c0 + j];
    if (tid < p1) {
        const int i = tid;
        s_nx[i] = cX[c0 + i * p2];
        s_ny[i] = cY[c0 + i * p1];
        s_nz[i] = cZ[c0 + i];
        s_w[i] = wts.w[i];
    }
    __syncthreads();
    const int nblk = nf / p3, rest = nf - nblk * p3;
    bool have = false;   // s_t, s_f0 hold an earlier block's contractions
    for (int blk = (int)((long)nblk * part / parts), end = (int)((long)nblk * (part + 1) / parts); blk < end; blk++) {
        const int b0 = f0 + blk * p3;
        // tensor-grid check (bitwise) and exact-node check on the 1-D coordinates
        if (tid < 3 * p1) {
            const int d = tid / p1, m = tid - d * p1;
            s_f[d][m] = d == 0 ? fX[b0 + m * p2] : (d == 1 ? fY[b0 + m * p1] : fZ[b0 + m]);
        }
        __syncthreads();
        int bad = 0, newx = 0, newy = 0;
        if (tid < 2 * p1) {
            const int d = tid / p1, m = tid - d * p1;
            const bool differs = !have || __double_as_longlong(s_f[d][m]) != __double_as_longlong(s_f0[d][m]);
            (d == 0 ? newx : newy) = differs;
        }
#pragma unroll 1
        for (int q = tid; q < p3; q += IT) {
            const int i = q / p2, j = (q / p1) % p1, k = q % p1;
            bad |= __double_as_longlong(fX[b0 + q]) != __double_as_longlong(s_f[0][i]);
            bad |= __double_as_longlong(fY[b0 + q]) != __double_as_longlong(s_f[1][j]);
            bad |= __double_as_longlong(fZ[b0 + q]) != __double_as_longlong(s_f[2][k]);
        }
        if (tid < 3 * p1) {
            const int d = tid / p1, m = tid - d * p1;
            const double *nodes = d == 0 ? s_nx : (d == 1 ? s_ny : s_nz);
            for (int k = 0; k < p1; k++) bad |= fabs(s_f[d][m] - nodes[k]) < DBL_MIN;
        }
        const int general = __syncthreads_or(bad);   // not a tensor grid, or a point on a node
        newx = __syncthreads_or(newx);
        newy = __syncthreads_or(newy) || newx;
        if (general) {
#pragma unroll 1
            for (int q = tid; q < p3; q += IT)
                fF[b0 + q] = fF[b0 + q] + interp_point<p1>(fX[b0 + q], fY[b0 + q], fZ[b0 + q], s_c, s_nx, s_ny,
                                                           s_nz, s_w);
            __syncthreads();
            continue;
        }
        // normalised 1-D barycentric rows
#pragma unroll 1
        for (int q = tid; q < 3 * p2; q += IT) {
            const int d = q / p2, mk = q - d * p2, m = mk / p1, k = mk - m * p1;
            if (d == 2 || (d == 0 ? newx : newy)) {
                const double *nodes = d == 0 ? s_nx : (d == 1 ? s_ny : s_nz);
                s_L[d][mk] = s_w[k] / (s_f[d][m] - nodes[k]);
            }
        }
        __syncthreads();
#pragma unroll 1
        for (int q = tid; q < 3 * p1; q += IT) {
            const int d = q / p1, m = q - d * p1;
            if (d == 2 || (d == 0 ? newx : newy)) {
                double sum = 0.0;
#pragma unroll
                for (int k = 0; k < p1; k++) sum += s_L[d][m * p1 + k];
                s_sum[d][m] = sum;
                s_inv[d][m] = 1.0 / sum;
                if (d < 2) s_f0[d][m] = s_f[d][m];
            }
        }
        __syncthreads();
#pragma unroll 1
        for (int q = tid; q < 3 * p2; q += IT) {
            const int d = q / p2, mk = q - d * p2;
            if (d == 2 || (d == 0 ? newx : newy)) {
                // a quotient from the reciprocal and its remainder (Markstein, 1990): a product alone would give
                // a whole row the reciprocal's rounding error (4.3e-16 instead of 4.2e-16
                // from 64-bit results in the largest case)
                const int m = mk / p1;
                const double v = s_L[d][mk], inv = s_inv[d][m], qt = v * inv;
                s_L[d][mk] = fma(fma(-qt, s_sum[d][m], v), inv, qt);
            }
        }
        __syncthreads();
        if (newx) {   // T1[a][j][k] = sum_i Lx[a][i] F[i][j][k]
#pragma unroll 1
            for (int q = tid; q < p3; q += IT) {
                const int aa = q / p2, jk = q - aa * p2;
                double v = 0.0;
                for (int i = 0; i < p1; i++) v += s_L[0][aa * p1 + i] * s_c[i * p2 + jk];
                s_t[0][q] = v;
            }
            __syncthreads();
        }
        if (newy) {   // T2[a][b][k] = sum_j Ly[b][j] T1[a][j][k]
#pragma unroll 1
            for (int q = tid; q < p3; q += IT) {
                const int aa = q / p2, bk = q - aa * p2, bb = bk / p1, k = bk - bb * p1;
                double v = 0.0;
                for (int j = 0; j < p1; j++) v += s_L[1][bb * p1 + j] * s_t[0][aa * p2 + j * p1 + k];
                s_t[1][q] = v;
            }
            __syncthreads();
        }
        have = true;
        // out[a][b][c] = sum_k Lz[c][k] T2[a][b][k]
#pragma unroll 1
        for (int q = tid; q < p3; q += IT) {
            const int ab = q / p1, c = q - ab * p1;
            double v = 0.0;
            for (int k = 0; k < p1; k++) v += s_L[2][c * p1 + k] * s_t[1][ab * p1 + k];
            fF[b0 + q] = fF[b0 + q] + v;
        }
        __syncthreads();
    }
    // points past the last whole block (a cell whose fine count is not a multiple of (p+1)^3)
#pragma unroll 1
    for (int q = part == parts - 1 ? tid : rest; q < rest; q += IT) {
        const int g = f0 + nblk * p3 + q;
        fF[g] = fF[g] + interp_point<p1>(fX[g], fY[g], fZ[g], s_c, s_nx, s_ny, s_nz, s_w);
    }
}

__global__ void copy_all(const double *__restrict__ a, double *__restrict__ b, long n) {
    long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) b[i] = a[i];
}

}  // namespace

int interp_device(const double *cX, const double *cY, const double *cZ, const double *cF,
                  const int *ppc_c, int coarseN, const double *fX, const double *fY,
                  const double *fZ, double *fF, const int *ppc_f, int fineN, int ncells,
                  int order, const int *h_ppc_c, const int *h_ppc_f, cudaStream_t s) {
    (void)h_ppc_c;
    (void)h_ppc_f;
    if (coarseN == fineN) {
        if (coarseN > 0) launch(copy_all, (coarseN + 255) / 256, 256, 0, s, cF, fF, coarseN);
        TAGI_LAUNCH_CHECK();
        return TAGI_OK;
    }
    const int p1 = order + 1;
    if (p1 < 1 || p1 > MAXP1)
        return set_error(TAGI_ERR_UNSUPPORTED, "interpolation order %d outside [0, %d]", order, MAXP1 - 1);
    if (ncells <= 0) return TAGI_OK;
    Weights w{};
    for (int i = 0; i < p1; i++)
        w.w[i] = pow(-1, i) * sin((2 * i + 1) * M_PI / (2 * (p1 - 1) + 2));
    Arena tmp;
    tmp.stream = s;
    int *off_c = nullptr, *off_f = nullptr, *err = nullptr;
    int rc = TAGI_OK;
    do {
        if ((rc = tmp.alloc(&off_c, ncells + 1)) || (rc = tmp.alloc(&off_f, ncells + 1)) ||
            (rc = tmp.alloc(&err, 1)))
            break;
        cudaMemsetAsync(err, 0, sizeof(int), s);
        if ((rc = exclusive_scan(ppc_c, off_c, ncells, off_c + ncells, tmp, s))) break;
        if ((rc = exclusive_scan(ppc_f, off_f, ncells, off_f + ncells, tmp, s))) break;
        // A cell's children go to several CTAs where the cells alone would not fill the chip; each
        // CTA stages the cell and forms its own contractions.  Us a call for 1, 2, 4, 8 parts, a
        // fifth of the cells with 8 children of order 7: 624 cells 127, 99, 91, 89; 1,400 180, 136,
        // 118, 121; 3,900 257, 199, 200, 240; 8,000 357, 323, 336, 435; 12,000 457, 436, 462, 612;
        // order 3: 624 cells 76, 64, 58, 57; 12,000 139, 130, 143, 164.  Points off the tensor
        // grid or on a node would take 4 parts above 4,000 cells as well (20,000 cells, order 5: 2
        // parts 2196 us, 4 parts 2007, 8 parts 1899).
        const dim3 grid(ncells, ncells < 1500 ? 8 : (ncells < 4000 ? 4 : 2));
        switch (p1) {   // every loop over nodes known at compile time
#define TAGI_INTERP(N)                                                                                             \
    case N: launch(interp_cells<N>, grid, IT, 0, s, cX, cY, cZ, cF, ppc_c, off_c, fX, fY, fZ, fF, ppc_f, off_f,    \
                   ncells, coarseN, fineN, w, err);                                                                \
        break;
            TAGI_INTERP(1) TAGI_INTERP(2) TAGI_INTERP(3) TAGI_INTERP(4) TAGI_INTERP(5) TAGI_INTERP(6)
            TAGI_INTERP(7) TAGI_INTERP(8) TAGI_INTERP(9) TAGI_INTERP(10) TAGI_INTERP(11) TAGI_INTERP(12)
#undef TAGI_INTERP
        }
        int h_err = 0;
        if (cudaGetLastError() != cudaSuccess ||
            cudaMemcpyAsync(&h_err, err, sizeof(int), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
            cudaStreamSynchronize(s) != cudaSuccess) {
            rc = set_error(TAGI_ERR_CUDA, "interpolation kernel failed");
            break;
        }
        if (h_err & 2) {
            int tot[2] = {0, 0};
            if (cudaMemcpyAsync(&tot[0], off_c + ncells, sizeof(int), cudaMemcpyDeviceToHost, s) ||
                cudaMemcpyAsync(&tot[1], off_f + ncells, sizeof(int), cudaMemcpyDeviceToHost, s) ||
                cudaStreamSynchronize(s))
                rc = set_error(TAGI_ERR_CUDA, "interpolation offsets copy failed");
            else
                rc = set_error(TAGI_ERR_ARG, "points per cell sum to %d coarse / %d fine, arrays hold %d / %d", tot[0],
                               tot[1], coarseN, fineN);
            break;
        }
        if (h_err) rc = set_error(TAGI_ERR_ARG, "an interpolated coarse cell does not hold (order+1)^3 points");
    } while (0);
    tmp.release();
    return rc;
}

}  // namespace tagi
