// Device mesh generation: the reference's cell refinement for the
// "coarsenedUniformTwoLevel" divide criterion and the first-kind Chebyshev
// quadrature meshes built on the resulting cells (coarse and two-level fine).
//
// Follows, in 3D-GreenIteration/src:
//   divide rule     dataStructures/CellStruct_CC.py:2344-2439
//                   (refineCoarseningUniform_TwoLevel)
//   recursion       dataStructures/TreeStruct_CC.py:1049-1131 (recursiveDivide:
//                   level < minDepth divides; midpoint split,
//                   CellStruct_CC.py:3060-3100)
//   cell order      depth first, children x-major (the uniqueID order of the
//                   tree's masterList, CellStruct_CC.py:220-221,
//                   TreeStruct_CC.py:2387), base cells in their given order
//   cell table      TreeStruct_CC.py:2390-2406 (centre, width, points per cell)
//   coarse points   utilities/mpiMeshBuilding.py:725-752
//   fine points     utilities/mpiMeshBuilding.py:755-840
//
// GPU layout.  Refinement is level-synchronous, one launch per level: eight lanes per
// cell of the current level decide divide / leaf and write its children into the next
// level or the leaf into the list of leaves.  Every cell carries a 64-bit path key (base cell
// index in bits 48-63, then 3 bits per level, child digit 4i+2j+k), so one
// radix sort of the leaf keys gives the depth-first order.  Point generation
// is one thread per output point (32 bytes written: x, y, z, w); fine points
// find their cell by binary search over the per-cell offsets.  All arithmetic
// is FP64 with explicit round-to-nearest intrinsics in the order the
// reference's numpy expressions evaluate, so the cells and points are
// bit-identical to the reference's on the same 1-D node and weight tables.
// Ring molecule, 5,104 cells, 16.9M points, build_mesh 2.37 -> 0.58 ms: the nearest corner
// of a cell from the smallest square along each axis with one root per cell (eight
// corners, a root each, per atom before: 92 us a level), no counts read back between levels,
// leaves sorted in two launches, and one refinement instead of a counting one first.
#include "tagi_internal.h"

#include <algorithm>
#include <cmath>
#include <type_traits>

namespace tagi {
namespace {

constexpr int MESH_MAX_DEPTH = 16;          // 3 bits per level below bit 48
constexpr int MESH_MAX_BASE = 1 << 16;      // base cell index in bits 48..63
constexpr long MESH_MAX_CELLS = 1L << 24;   // cells per level / leaves in total
constexpr int MESH_MAX_P1 = 16;             // order <= 15
constexpr int MT = 256;

struct Rule {
    double h, H, r;
    int ge2, ge1, fine;  // level >= 2, level >= 1, level < -1
    int nsub;            // -int(level): fine children per side
    int min_depth, max_depth;
    // distances and sides of the cascade, each rounded as the reference's expression
    double far, r4, r2, h4th, h2th, h2, h4, h8, a1, a2, a3, r15;
};

struct Tables {
    double u[MESH_MAX_P1];  // first-kind nodes cos(theta_i) on [-1, 1], ascending
    double w[MESH_MAX_P1];  // unscaled first-kind weights
};

__device__ __forceinline__ double half_of(double a) { return __dmul_rn(a, 0.5); }

// Counters of a refinement, on the device.
struct Progress {
    unsigned long long fine;            // children (or 1) per leaf, summed
    int err;                            // 1: refines below maxDepth; 2: a level or the leaves do not fit
    int leaves;
    int count[MESH_MAX_DEPTH + 2];      // cells of each level
};

__global__ void mesh_start(Progress *p, int nbase) {
    const int i = threadIdx.x;
    if (i < MESH_MAX_DEPTH + 2) p->count[i] = i ? 0 : nbase;
    if (i == 0) {
        p->fine = 0;
        p->err = p->leaves = 0;
    }
}

// One level: divide flag and fine children of each cell (CellStruct_CC.py:2344-2439), the
// children of a dividing cell into the next level, a leaf into the leaf list.  Eight lanes a
// cell: they share the atoms, then a lane writes a child.  Places are taken from the
// counters as warps come, one addition a warp and counter: the leaves are sorted by their
// keys afterwards, so the order within a level does not matter, and the host reads no
// count between levels.  A level was a classification of one thread per cell (14 us: 12
// atoms in turn on the FP64 pipe), a scan, a copy to the host and eight allocations, 85 us in all.
constexpr int CELL_LANES = 8, LEVEL_THREADS = 128;
__global__ void __launch_bounds__(LEVEL_THREADS) mesh_level(
    const double *cells, const uint64_t *keys, int depth, const double *atoms,
    int natoms, const __grid_constant__ Rule p, Progress *prog, double *next_cells,
    uint64_t *next_keys, int next_cap, double *leaf_cells, uint64_t *leaf_keys,
    int *leaf_fine, int leaf_cap) {
    chain_begin();
    const int n = prog->count[depth];
    if (prog->err & 2) return;
    const int lane = threadIdx.x & 31, q = lane & (CELL_LANES - 1);
    const int group = (blockIdx.x * LEVEL_THREADS + threadIdx.x) / CELL_LANES, groups = gridDim.x * LEVEL_THREADS / CELL_LANES;
    const int warp_first = group - lane / CELL_LANES;
    for (int base = warp_first; base < n; base += groups) {   // the same for all of a warp
        const int i = base + lane / CELL_LANES;
        const bool valid = i < n;
        const double *c = cells + 6L * (valid ? i : 0);
        const double xmin = c[0], xmax = c[1], ymin = c[2], ymax = c[3], zmin = c[4], zmax = c[5];
        int div = 0, nf = 1;
        if (depth < p.min_depth) {
            div = 1;
        } else {
            // The distance to the nearest corner: rounded squares, sums and roots are
            // monotone, so the smallest square along each axis gives the smallest
            // rounded distance of the eight corners, and one root serves all atoms.
            double d2 = __longlong_as_double(0x7ff0000000000000LL);
            int inside = 0;
            for (int a = q; a < natoms; a += CELL_LANES) {
                const double ax = atoms[3 * a], ay = atoms[3 * a + 1], az = atoms[3 * a + 2];
                if (ax < xmax && ay < ymax && az < zmax && ax > xmin && ay > ymin && az > zmin) {
                    inside = 1;
                    continue;
                }
                const double x0 = __dsub_rn(xmin, ax), x1 = __dsub_rn(xmax, ax), y0 = __dsub_rn(ymin, ay),
                             y1 = __dsub_rn(ymax, ay), z0 = __dsub_rn(zmin, az), z1 = __dsub_rn(zmax, az);
                const double x = fmin(fabs(x0), fabs(x1)), y = fmin(fabs(y0), fabs(y1)), z = fmin(fabs(z0), fabs(z1));
                const double s = __dadd_rn(__dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y)), __dmul_rn(z, z));
                if (s < d2) d2 = s;
            }
            // d2 >= +0 and no NaN got in: its bit pattern orders as an integer does
            long long b2 = __double_as_longlong(d2);
#pragma unroll
            for (int o = CELL_LANES / 2; o > 0; o >>= 1) {
                b2 = min(b2, __shfl_xor_sync(0xffffffffu, b2, o));
                inside |= __shfl_xor_sync(0xffffffffu, inside, o);
            }
            double dist = p.far;
            const double dc = __dsqrt_rn(__longlong_as_double(b2));
            if (dc < dist) dist = dc;
            if (inside) dist = 0.0;
            const double sz = __dsub_rn(zmax, zmin), sx = __dsub_rn(xmax, xmin), sy = __dsub_rn(ymax, ymin);
            double side = sz;
            if (sx > side) side = sx;
            if (sy > side) side = sy;
            if (side > p.H)
                div = 1;
            else if (p.ge2 && dist < p.r4)
                div = side > p.h4th;
            else if (p.ge1 && dist < p.r2)
                div = side > p.h2th;
            else if (dist < p.r)
                div = side > p.h;
            else if (dist < p.a1)
                div = side > p.h2;
            else if (dist < p.a2)
                div = side > p.h4;
            else if (dist < p.a3)
                div = side > p.h8;
            if (!div && p.fine && dist < p.r15) nf = p.nsub * p.nsub * p.nsub;
        }
        if (div && depth >= p.max_depth) {
            if (valid && q == 0) atomicOr(&prog->err, 1);
            div = 0;
        }
        // places: one bit per cell in each mask
        const unsigned first = 0x01010101u;
        const unsigned md = __ballot_sync(0xffffffffu, valid && div) & first, ml = __ballot_sync(0xffffffffu, valid && !div) & first;
        const int fine = __reduce_add_sync(0xffffffffu, valid && !div && q == 0 ? nf : 0);
        int at_d = 0, at_l = 0;
        if (lane == 0) {
            if (md) at_d = atomicAdd(&prog->count[depth + 1], 8 * __popc(md));
            if (ml) {
                at_l = atomicAdd(&prog->leaves, __popc(ml));
                atomicAdd(&prog->fine, (unsigned long long)fine);
            }
        }
        const unsigned before = (1u << (lane & ~(CELL_LANES - 1))) - 1u;
        at_d = __shfl_sync(0xffffffffu, at_d, 0) + 8 * __popc(md & before);
        at_l = __shfl_sync(0xffffffffu, at_l, 0) + __popc(ml & before);
        if (!valid) continue;
        const uint64_t key = keys ? keys[i] : (uint64_t)i << 48;
        if (div) {
            if (at_d > next_cap - 8) {
                if (q == 0) atomicOr(&prog->err, 2);
                continue;
            }
            // child q = 4 ii + 2 jj + kk; xdiv = (xmax + xmin)/2 (TreeStruct_CC.py:1129-1131)
            const double xm = half_of(__dadd_rn(xmax, xmin)), ym = half_of(__dadd_rn(ymax, ymin)),
                         zm = half_of(__dadd_rn(zmax, zmin));
            double *o = next_cells + 6L * (at_d + q);
            o[0] = q & 4 ? xm : xmin;
            o[1] = q & 4 ? xmax : xm;
            o[2] = q & 2 ? ym : ymin;
            o[3] = q & 2 ? ymax : ym;
            o[4] = q & 1 ? zm : zmin;
            o[5] = q & 1 ? zmax : zm;
            next_keys[at_d + q] = key | ((uint64_t)q << (3 * (MESH_MAX_DEPTH - 1 - depth)));
        } else if (at_l >= leaf_cap) {
            if (q == 0) atomicOr(&prog->err, 2);
        } else {
            if (q < 6) leaf_cells[6L * at_l + q] = c[q];
            if (q == 6) leaf_keys[at_l] = key;
            if (q == 7) leaf_fine[at_l] = nf;
        }
    }
}

__global__ void mesh_iota(int *__restrict__ v, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) v[i] = i;
}

// Leaves in key order -> the reference's cell table (TreeStruct_CC.py:2390-2406).
__global__ void __launch_bounds__(MT) mesh_cell_table(const int *__restrict__ order_idx, int n,
                                                      const double *__restrict__ leaf_cells,
                                                      const int *__restrict__ leaf_fine, int p3,
                                                      double *__restrict__ cx, double *__restrict__ cy,
                                                      double *__restrict__ cz, double *__restrict__ dx,
                                                      double *__restrict__ dy, double *__restrict__ dz,
                                                      int *__restrict__ ppc_c,
                                                      int *__restrict__ ppc_f) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int s = order_idx[i];
    const double *c = leaf_cells + 6L * s;
    cx[i] = half_of(__dadd_rn(c[0], c[1]));
    cy[i] = half_of(__dadd_rn(c[2], c[3]));
    cz[i] = half_of(__dadd_rn(c[4], c[5]));
    dx[i] = __dsub_rn(c[1], c[0]);
    dy[i] = __dsub_rn(c[3], c[2]);
    dz[i] = __dsub_rn(c[5], c[4]);
    if (ppc_c) ppc_c[i] = p3;
    if (ppc_f) ppc_f[i] = leaf_fine[s] * p3;
}

// x/2 and x/4 are written as products with 0.5 and 0.25: the same correctly
// rounded value as the reference's divisions, without a division sequence.

// One cell's bounds from centre and width: xl = cx - dx/2, xh = cx + dx/2
// (mpiMeshBuilding.py:519-527).
__device__ __forceinline__ void cell_bounds(const double *cx, const double *cy, const double *cz,
                                            const double *dx, const double *dy, const double *dz,
                                            long c, double lo[3], double hi[3]) {
    const double ctr[3] = {cx[c], cy[c], cz[c]};
    const double wid[3] = {dx[c], dy[c], dz[c]};
#pragma unroll
    for (int d = 0; d < 3; d++) {
        const double hw = __dmul_rn(wid[d], 0.5);
        lo[d] = __dsub_rn(ctr[d], hw);
        hi[d] = __dadd_rn(ctr[d], hw);
    }
}

// Interior split points of [lo, hi] into m equal parts, as
// fineQuadraturePointsSingleCell writes them (mpiMeshBuilding.py:766-800).
__device__ __forceinline__ double split_point(double lo, double hi, int m, int s) {
    if (s == 0) return lo;
    if (s == m) return hi;
    if (m == 2) return __dmul_rn(__dadd_rn(lo, hi), 0.5);
    if (m == 3)
        return s == 1 ? __ddiv_rn(__dadd_rn(__dmul_rn(2.0, lo), hi), 3.0)
                      : __ddiv_rn(__dadd_rn(__dmul_rn(2.0, hi), lo), 3.0);
    // m == 4
    if (s == 2) return __dmul_rn(__dadd_rn(lo, hi), 0.5);
    return s == 1 ? __dmul_rn(__dadd_rn(__dmul_rn(3.0, lo), hi), 0.25)
                  : __dmul_rn(__dadd_rn(__dmul_rn(3.0, hi), lo), 0.25);
}

// m (children per side) and m^3 per cell from the fine point counts.
__global__ void mesh_fine_counts(const int *__restrict__ ppc_f, int n, int p3, int *__restrict__ sub,
                                 int *__restrict__ nsub, int *__restrict__ err) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int v = ppc_f[i];
    int m = 0;
    if (v == p3) m = 1;
    else if (v == 8 * p3) m = 2;
    else if (v == 27 * p3) m = 3;
    else if (v == 64 * p3) m = 4;
    if (!m) atomicOr(err, 2);
    sub[i] = m;
    nsub[i] = m * m * m;
}

constexpr int PW = 8;  // warps per CTA in mesh_points_warp

// One warp per sub-cell: a coarse cell (sub_off == nullptr), or child
// (ii, jj, kk) of a fine cell.  Every sub-cell holds (order+1)^3 points, so
// sub-cell s writes points [s p3, (s+1) p3).  Lanes < order+1 evaluate the
// 1-D nodes x = lo + (hi-lo)/2 (u+1) and scaled weights (hi-lo)/2 W of each
// axis once (meshUtilities.py:857-883), then the (order+1)^2 products
// wx_i wy_j; every point is then four shared loads, w = (wx_i wy_j) wz_k
// (the same two roundings in the same order as the reference's tensor
// product, one of them shared by a row of points) and four coalesced stores.
__global__ void __launch_bounds__(PW * 32) mesh_points_warp(const double *__restrict__ cx,
                                                            const double *__restrict__ cy,
                                                            const double *__restrict__ cz,
                                                            const double *__restrict__ dx,
                                                            const double *__restrict__ dy,
                                                            const double *__restrict__ dz,
                                                            const int *__restrict__ sub_off,
                                                            const int *__restrict__ sub, int ncells,
                                                            long nsubcells, int p1, unsigned m1,
                                                            unsigned m2, const __grid_constant__ Tables t,
                                                            double *__restrict__ X, double *__restrict__ Y,
                                                            double *__restrict__ Z, double *__restrict__ W) {
    __shared__ double sh[PW][6][MESH_MAX_P1];
    __shared__ double sh_wxy[PW][MESH_MAX_P1 * MESH_MAX_P1];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int p3 = p1 * p1 * p1;
    double(*nd)[MESH_MAX_P1] = sh[wid];
    double *wxy = sh_wxy[wid];
    for (long s = (long)blockIdx.x * PW + wid; s < nsubcells; s += (long)gridDim.x * PW) {
        int c = (int)s, m = 1, child = 0;
        if (sub_off) {
            // last cell whose first sub-cell is <= s (every cell has >= 1)
            int a = 0, b = ncells - 1;
            while (a < b) {
                const int mid = (a + b + 1) >> 1;
                if ((long)sub_off[mid] <= s) a = mid;
                else b = mid - 1;
            }
            c = a;
            m = sub[c];
            child = (int)(s - sub_off[c]);
        }
        if (lane < p1) {
            double lo[3], hi[3];
            cell_bounds(cx, cy, cz, dx, dy, dz, c, lo, hi);
            const int ch[3] = {child / (m * m), (child / m) % m, child % m};
#pragma unroll
            for (int d = 0; d < 3; d++) {
                const double l = split_point(lo[d], hi[d], m, ch[d]);
                const double h = split_point(lo[d], hi[d], m, ch[d] + 1);
                const double hw = __dmul_rn(__dsub_rn(h, l), 0.5);
                nd[d][lane] = __dadd_rn(l, __dmul_rn(hw, __dadd_rn(t.u[lane], 1.0)));
                nd[3 + d][lane] = __dmul_rn(hw, t.w[lane]);
            }
        }
        __syncwarp();
        for (int ij = lane; ij < p1 * p1; ij += 32) {
            const int i = ij / p1, j = ij - i * p1;
            wxy[ij] = __dmul_rn(nd[3][i], nd[4][j]);
        }
        __syncwarp();
        const long base = s * p3;
        for (int q = lane; q < p3; q += 32) {
            // i = q / p2, j = (q / p1) % p1, k = q % p1 by high multiplies with
            // m = ceil(2^32 / d): exact for q d < 2^32 (q < 4096, d <= 256)
            const unsigned uq = (unsigned)q, tq = __umulhi(uq, m1);
            const int i = (int)__umulhi(uq, m2);
            const int j = (int)(tq - __umulhi(tq, m1) * (unsigned)p1);
            const int k = (int)(uq - tq * (unsigned)p1);
            X[base + q] = nd[0][i];
            Y[base + q] = nd[1][j];
            Z[base + q] = nd[2][k];
            W[base + q] = __dmul_rn(wxy[i * p1 + j], nd[5][k]);
        }
        __syncwarp();
    }
}

int grid_for(long n) {
    long g = (n + MT - 1) / MT;
    return (int)(g < 1 ? 1 : (g > (1L << 30) ? (1L << 30) : g));
}

// Host copies of small device counters, on the call's stream.
int read_ints(const int *d, int *h, int n, cudaStream_t s) {
    TAGI_CUDA(cudaMemcpyAsync(h, d, sizeof(int) * n, cudaMemcpyDeviceToHost, s));
    TAGI_CUDA(cudaStreamSynchronize(s));
    return TAGI_OK;
}

// u_i and W_i of meshUtilities.py:835-883 from libm, for callers that pass
// no tables.  A caller that needs the bit pattern of a particular numpy
// build passes its own.
void default_tables(int order, Tables &t) {
    const int n1 = order + 1;
    const double pi = 3.141592653589793;
    // theta_i = (e_{i+1} + e_i)/2 with e_i = i * (-pi/(order+1)) + pi, e_{order+1} = 0
    const double step = -pi / n1;
    for (int i = 0; i < n1; i++) {
        const double e0 = i * step + pi, e1 = (i + 1 == n1) ? 0.0 : (i + 1) * step + pi;
        t.u[i] = std::cos((e1 + e0) / 2);
    }
    double Wv[MESH_MAX_P1] = {};
    for (int i = 0; i < n1; i++) Wv[i] = i == 0 ? 1.0 : (i % 2 == 0 ? 2.0 / (1.0 - (double)i * i) : 0.0);
    for (int j = 0; j < n1; j++) {
        double s = 0.0;
        for (int i = 0; i < n1; i++) s += 2.0 / n1 * std::cos(i * (j + 0.5) * pi / n1) * Wv[i];
        t.w[j] = s;
    }
}

}  // namespace
}  // namespace tagi

extern "C" {

int tagi_mesh_refine(const double *baseCells, int numBase, const double *atomXYZ, int numAtoms, int order,
                     double h, double H, double r, double level, int minDepth, int maxDepth, double *cellX,
                     double *cellY, double *cellZ, double *cellDX, double *cellDY, double *cellDZ,
                     int *ptsPerCellCoarse, int *ptsPerCellFine, int capacity, int *numCells,
                     long long *numCoarsePoints, long long *numFinePoints, void *stream) {
    using namespace tagi;
    if (!numCells) return set_error(TAGI_ERR_ARG, "numCells is null");
    *numCells = 0;
    if (numCoarsePoints) *numCoarsePoints = 0;
    if (numFinePoints) *numFinePoints = 0;
    if (numBase < 1 || numBase > MESH_MAX_BASE)
        return set_error(TAGI_ERR_ARG, "numBase %d outside [1, %d]", numBase, MESH_MAX_BASE);
    if (!baseCells) return set_error(TAGI_ERR_ARG, "baseCells is null");
    if (numAtoms < 0 || (numAtoms > 0 && !atomXYZ)) return set_error(TAGI_ERR_ARG, "bad atom array");
    if (order < 0 || order + 1 > MESH_MAX_P1)
        return set_error(TAGI_ERR_UNSUPPORTED, "order %d outside [0, %d]", order, MESH_MAX_P1 - 1);
    if (!std::isfinite(h) || !std::isfinite(H) || !std::isfinite(r) || !std::isfinite(level))
        return set_error(TAGI_ERR_ARG, "divide parameters must be finite");
    if (maxDepth < 0 || maxDepth > MESH_MAX_DEPTH || minDepth < 0)
        return set_error(TAGI_ERR_ARG, "maxDepth %d outside [0, %d] or minDepth %d < 0", maxDepth,
                         MESH_MAX_DEPTH, minDepth);
    if (capacity < 0) return set_error(TAGI_ERR_ARG, "capacity < 0");
    const bool query = cellX == nullptr;
    if (!query && (!cellY || !cellZ || !cellDX || !cellDY || !cellDZ))
        return set_error(TAGI_ERR_ARG, "cell table arrays must all be given (or cellX null to count)");
    Rule p;
    p.h = h;
    p.H = H;
    p.r = r;
    p.ge2 = level >= 2;
    p.ge1 = level >= 1;
    p.fine = level < -1;
    p.nsub = p.fine ? -(int)level : 1;
    p.min_depth = minDepth;
    p.max_depth = maxDepth;
    if (p.fine && p.nsub > 4)
        return set_error(TAGI_ERR_UNSUPPORTED, "fine mesh of %d^3 children per cell (1, 8, 27 or 64 supported)",
                         p.nsub);
    // host and device round these alike: the factors are powers of two but for r 1.5
    p.far = 10.0 + H;
    p.r4 = r / 4.0;
    p.r2 = r / 2.0;
    p.h4th = h / 4.0;
    p.h2th = h / 2.0;
    p.h2 = 2.0 * h;
    p.h4 = 4.0 * h;
    p.h8 = 8.0 * h;
    p.a1 = r + p.h2;
    p.a2 = r + (p.h2 + p.h4);
    p.a3 = r + ((p.h2 + p.h4) + p.h8);
    p.r15 = r * 1.5;
    const int p1 = order + 1, p3 = p1 * p1 * p1;
    cudaStream_t s = (cudaStream_t)stream;
    Arena tmp;
    tmp.stream = s;
    int rc = TAGI_OK;
    do {
        Progress *prog = nullptr, h_prog;
        double *cells[2] = {}, *leaf_cells = nullptr;
        uint64_t *keys[2] = {}, *leaf_keys = nullptr;
        int *leaf_fine = nullptr;
        if ((rc = tmp.alloc(&prog, 1))) break;
        // Room for the usual counts; a mesh that needs more starts again with more.
        long level_cap = std::max(32768L, 16L * numBase), leaf_cap = std::max(16384L, 16L * numBase);
        long total = 0;
        for (;;) {
            char *block = nullptr;   // two levels and the leaves
            const long cell = 6 * sizeof(double) + sizeof(uint64_t);
            if ((rc = tmp.alloc(&block, 2 * level_cap * cell + leaf_cap * (cell + (long)sizeof(int))))) break;
            char *at = block;
            auto take = [&](auto *&ptr, long count) {
                ptr = reinterpret_cast<std::remove_reference_t<decltype(ptr)>>(at);
                at += count * sizeof(*ptr);
            };
            for (int k = 0; k < 2; k++) take(cells[k], 6 * level_cap);
            take(leaf_cells, 6 * leaf_cap);
            for (int k = 0; k < 2; k++) take(keys[k], level_cap);
            take(leaf_keys, leaf_cap);
            take(leaf_fine, leaf_cap);
            launch(mesh_start, 1, 32, 0, s, prog, numBase);
            // LEVELS levels are launched at a time: one more costs 2 us where it has no cells
            constexpr int LEVELS = 6;
            for (int depth = 0; !rc;) {
                for (int k = 0; k < LEVELS && depth <= MESH_MAX_DEPTH && !rc; k++, depth++) {
                    const int from = depth & 1, to = from ^ 1;
                    // a level holds at most 8 times the cells of the one before
                    const long most = std::min(level_cap, depth < 10 ? (long)numBase << (3 * depth) : level_cap);
                    const int grid = (int)std::min(GPU_SMS * 8, (most * CELL_LANES + LEVEL_THREADS - 1) / LEVEL_THREADS);
                    if (launch_chained(mesh_level, grid, LEVEL_THREADS, 0, s, depth ? cells[from] : baseCells,
                                       depth ? keys[from] : (const uint64_t *)nullptr, depth, atomXYZ, numAtoms, p, prog,
                                       cells[to], keys[to], (int)level_cap, leaf_cells, leaf_keys, leaf_fine,
                                       (int)leaf_cap) != cudaSuccess)
                        rc = set_error(TAGI_ERR_CUDA, "mesh_level launch failed");
                }
                if (rc) break;
                if (cudaMemcpyAsync(&h_prog, prog, sizeof(Progress), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
                    cudaStreamSynchronize(s) != cudaSuccess) {
                    rc = set_error(TAGI_ERR_CUDA, "mesh refinement failed: %s", cudaGetErrorString(cudaGetLastError()));
                    break;
                }
                if (h_prog.err & 2 || depth > MESH_MAX_DEPTH || h_prog.count[depth] == 0) break;
            }
            if (rc || !(h_prog.err & 2)) break;
            long most = 0;
            for (int d = 1; d <= MESH_MAX_DEPTH + 1; d++) most = std::max(most, (long)h_prog.count[d]);
            // blocks that start after the overflow count nothing more: the next try may need still more room
            if (most > MESH_MAX_CELLS || h_prog.leaves > MESH_MAX_CELLS) {
                rc = set_error(TAGI_ERR_ARG, "refinement exceeds %ld cells", MESH_MAX_CELLS);
                break;
            }
            if (most > level_cap) level_cap = std::min(MESH_MAX_CELLS, std::max(2 * most, 4 * level_cap));
            else leaf_cap = std::min(MESH_MAX_CELLS, std::max(2L * h_prog.leaves, 4 * leaf_cap));
            tmp.release();
            if ((rc = tmp.alloc(&prog, 1))) break;
        }
        if (rc) break;
        if (h_prog.err) {
            rc = set_error(TAGI_ERR_ARG, "the divide rule refines below maxDepth %d", maxDepth);
            break;
        }
        total = h_prog.leaves;
        *numCells = (int)total;
        if (numCoarsePoints) *numCoarsePoints = (long long)total * p3;
        if (numFinePoints) *numFinePoints = (long long)h_prog.fine * p3;
        if (query) break;
        if (capacity < total) {
            rc = set_error(TAGI_ERR_ARG, "capacity %d < %ld cells (numCells holds the count)", capacity, total);
            break;
        }
        int *idx = nullptr;
        if ((rc = tmp.alloc(&idx, total))) break;
        launch(mesh_iota, grid_for(total), MT, 0, s, idx, (int)total);
        uint64_t *keys_out = nullptr;
        int *order_of = nullptr;
        if ((rc = tmp.alloc(&keys_out, total)) || (rc = tmp.alloc(&order_of, total)) ||
            (rc = radix_sort_u64(leaf_keys, idx, keys_out, order_of, (int)total, 64, tmp, s)))
            break;
        launch(mesh_cell_table, grid_for(total), MT, 0, s, order_of, (int)total, leaf_cells, leaf_fine, p3, cellX, cellY,
               cellZ, cellDX, cellDY, cellDZ, ptsPerCellCoarse, ptsPerCellFine);
        if (cudaGetLastError() != cudaSuccess || cudaStreamSynchronize(s) != cudaSuccess)
            rc = set_error(TAGI_ERR_CUDA, "mesh cell table failed");
    } while (0);
    tmp.release();
    return rc;
}

int tagi_mesh_points(const double *cellX, const double *cellY, const double *cellZ, const double *cellDX,
                     const double *cellDY, const double *cellDZ, const int *ptsPerCellFine, int numCells,
                     int order, const double *unitNodes, const double *unitWeights, double *X, double *Y,
                     double *Z, double *W, long long numCoarsePoints, double *Xf, double *Yf, double *Zf,
                     double *Wf, long long numFinePoints, void *stream) {
    using namespace tagi;
    if (numCells < 0) return set_error(TAGI_ERR_ARG, "numCells < 0");
    if (order < 0 || order + 1 > MESH_MAX_P1)
        return set_error(TAGI_ERR_UNSUPPORTED, "order %d outside [0, %d]", order, MESH_MAX_P1 - 1);
    const int p1 = order + 1, p3 = p1 * p1 * p1;
    if (numCoarsePoints != (long long)numCells * p3)
        return set_error(TAGI_ERR_ARG, "numCoarsePoints %lld != numCells * (order+1)^3 = %lld", numCoarsePoints,
                         (long long)numCells * p3);
    if (numCells == 0) return TAGI_OK;
    if (!cellX || !cellY || !cellZ || !cellDX || !cellDY || !cellDZ || !X || !Y || !Z || !W)
        return set_error(TAGI_ERR_ARG, "null cell table or coarse point array");
    const bool fine = Xf || Yf || Zf || Wf;
    if (fine && (!Xf || !Yf || !Zf || !Wf || !ptsPerCellFine))
        return set_error(TAGI_ERR_ARG, "fine mesh needs Xf, Yf, Zf, Wf and ptsPerCellFine");
    if (fine && (numFinePoints < 0 || numFinePoints > 0x7fffffffLL))
        return set_error(TAGI_ERR_ARG, "numFinePoints %lld outside [0, 2^31)", numFinePoints);
    Tables t;
    if (unitNodes && unitWeights) {
        for (int i = 0; i < p1; i++) {
            t.u[i] = unitNodes[i];
            t.w[i] = unitWeights[i];
        }
    } else if (!unitNodes && !unitWeights) {
        default_tables(order, t);
    } else {
        return set_error(TAGI_ERR_ARG, "give both unitNodes and unitWeights, or neither");
    }
    for (int i = p1; i < MESH_MAX_P1; i++) t.u[i] = t.w[i] = 0.0;
    cudaStream_t s = (cudaStream_t)stream;
    const int p2 = p1 * p1;
    const unsigned m1 = p1 > 1 ? (unsigned)((0x100000000ULL + p1 - 1) / p1) : 0u;
    const unsigned m2 = p2 > 1 ? (unsigned)((0x100000000ULL + p2 - 1) / p2) : 0u;
    auto warp_grid = [](long nsubcells) {
        long g = (nsubcells + PW - 1) / PW;
        return (int)(g < 1 ? 1 : (g > GPU_SMS * 32 ? GPU_SMS * 32 : g));
    };
    launch(mesh_points_warp, warp_grid(numCells), PW * 32, 0, s, cellX, cellY, cellZ, cellDX, cellDY, cellDZ,
           (const int *)nullptr, (const int *)nullptr, numCells, (long)numCells, p1, m1, m2, t, X, Y, Z, W);
    TAGI_LAUNCH_CHECK();
    if (!fine) return TAGI_OK;
    Arena tmp;
    tmp.stream = s;
    int rc = TAGI_OK;
    do {
        // off[numCells] receives the sub-cell total, off[numCells + 1] the error flag
        int *sub = nullptr, *nsub = nullptr, *off = nullptr;
        if ((rc = tmp.alloc(&sub, numCells)) || (rc = tmp.alloc(&nsub, numCells)) ||
            (rc = tmp.alloc(&off, numCells + 2)))
            break;
        int *err = off + numCells + 1;
        if (cudaMemsetAsync(err, 0, sizeof(int), s) != cudaSuccess) {
            rc = set_error(TAGI_ERR_CUDA, "mesh memset failed");
            break;
        }
        launch(mesh_fine_counts, grid_for(numCells), MT, 0, s, ptsPerCellFine, numCells, p3, sub, nsub, err);
        if ((rc = exclusive_scan(nsub, off, numCells, off + numCells, tmp, s))) break;
        int h[2] = {0, 0};
        if ((rc = read_ints(off + numCells, h, 2, s))) break;
        if (h[1]) {
            rc = set_error(TAGI_ERR_ARG, "a fine cell holds a point count other than 1, 8, 27 or 64 x (order+1)^3");
            break;
        }
        const long long fine_pts = (long long)h[0] * p3;
        if (fine_pts != numFinePoints) {
            rc = set_error(TAGI_ERR_ARG, "ptsPerCellFine sums to %lld, numFinePoints is %lld", fine_pts,
                           numFinePoints);
            break;
        }
        if (numFinePoints == 0) break;
        launch(mesh_points_warp, warp_grid(h[0]), PW * 32, 0, s, cellX, cellY, cellZ, cellDX, cellDY, cellDZ,
               (const int *)off, (const int *)sub, numCells, (long)h[0], p1, m1, m2, t, Xf, Yf, Zf, Wf);
        if (cudaGetLastError() != cudaSuccess) rc = set_error(TAGI_ERR_CUDA, "mesh_points_warp launch failed");
    } while (0);
    tmp.release();
    return rc;
}

}  // extern "C"
