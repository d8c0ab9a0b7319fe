// Subsystems (c) far field and (d) near field, plus the per-call glue.
//
// One CTA works on one (target chunk of a batch, orbital) item at a time,
// pulled from a global counter in heaviest-first order (persistent launch,
// grid = resident CTAs).  In the single-orbital kernels the CTA's warps form G
// groups of targets times S splits of each target's sources (Fields::split, set
// per plan by field_split).  Each target's sum is formed in
// a fixed order (list order, then source order), so results do not depend on
// scheduling; in mixed precision not on the split either: the splits' FP32
// partials go through shared memory to one thread per target, which adds them
// in list order.
//
// Mixed precision (default fast path):
//   * coordinates are taken relative to the batch center, then rounded to FP32: targets (and
//     proxy points) in FP64; sources from FP32 hi/lo splits, to 2^-49 of their distance from
//     the the origin (neg_relative), or in FP64 too in plans so far from the origin that this would
//     show (WIDE kernels).  Close ranges use the splits themselves;
//   * coordinates are also multiplied by a per-orbital scale sc, so that with
//     r' = sc r the kernels need no multiply for the exp2 argument:
//       Yukawa       sc = k log2(e):          e^{-k r}/r     = sc 2^{-r'} / r'
//       Coulomb SS   sc = a sqrt(log2(e)):    e^{-a^2 r^2}   = 2^{-r'^2},  1/r = sc / r'
//       Coulomb skip sc = 1
//     and the factor sc multiplies each target's sum once at the end;
//   * pair terms and per-tile sums in FP32, rsqrt and exp2 on the MUFU pipe;
//   * pair terms are summed in FP32 runs of 64 (near) or one (n+1)^2 slab
//     (far) and the runs are added with Kahan compensation;
//   * the singularity-subtraction term f_i * 4pi/k^2 (Yukawa) or
//     f_i * 2pi/a^2 (Coulomb) is added in FP64 in the epilogue.
// FP64 mode: identical structure, FP64 results: 1/r by a Newton step from the FP32 estimate,
// the exponential from a table and a short polynomial (inv_root, exp_root).
//
// Pair terms (targets i, sources j, r = |x_i - y_j| > 0):
//   Yukawa  SS  w_j (f_j - f_i) e^{-k r}/r        skip  w_j f_j e^{-k r}/r
//   Coulomb SS  w_j (f_j - f_i e^{-a^2 r^2})/r    skip  w_j f_j / r
// (TreeStruct_CC.py:2782,2795,2931; greenIterationFixedPoint.py:314-324;
//  scfFixedPoint.py:297-303).  Far field: the same with (y_j, w_j f_j, w_j)
// replaced by (proxy point s_k, qhat_k, what_k).
#include "tagi_internal.h"

#include <algorithm>
#include <cmath>
#include <functional>
#include <type_traits>

namespace tagi {

namespace {

constexpr int FT = 256;        // threads per CTA of the FP64 kernels
constexpr int SLOT = 64;       // sources per slot of a tile: one FP32 run per lane pair
constexpr int NTILE = 4 * SLOT;  // sources per tile of the loop ceiling
constexpr double LOG2E = 1.4426950408889634;

__device__ __forceinline__ float rsqrt_mufu(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float ex2_mufu(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float lg2_mufu(float x) {
    float y;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

struct Fields {
    // target side (sorted order)
    const double *tx, *ty, *tz;
    const double *tcenter, *tradius;
    const int *batch_node;
    int nt, norb;
    // near side
    const int *rng_off;
    const int2 *rng;
    const float *rng_dmin;
    const double *sx, *sy, *sz;
    const float4 *shi, *slo, *thi, *tlo;  // FP32 hi/lo splits of absolute coordinates
    int ns;
    const float *q32, *w32;       // [norb][ns] charges f*w, [ns] weights
    const double *f64, *w64;      // [norb][ns] values f, [ns] weights
    // far side
    const int *far_off, *far_list, *node_slot;
    const double *geom;
    const float *qhat32, *what32; // [norb][nslots][P], [nslots][P]
    const double *qhat64, *what64;
    int nslots, n1, P, split;     // split: warps that share a target's sources (1, 2, 4 or 8)
    double tn[MAX_DEGREE + 1];
    // per orbital
    const float *ft32;            // [norb][nt] sorted target values
    const double *ft64;
    const float *kc32;            // [norb] coordinate scale sc (orbital_constants)
    const double *kp64;           // [norb] kernel parameter k or a
    double *out;                  // [norb][nt] sorted order
};

// Argument of every persistent field kernel: the work list of this pass and
// up to MAX_SYSTEMS systems' fields.  It is a __grid_constant__ parameter, so
// a CTA reads the fields of its current item's system straight from the
// parameter bank (dynamic index, no local copy).
struct Work {
    const int4 *items;            // {batch, sys << 16 | first orbital, target begin, end}, heaviest first
    int nitems;
    int *queue;                   // this pass's work counter
    int turn;                     // FP64: which of an item's CTAs' worth of targets
    const double *exp_table;      // FP64 passes: 2^{i / EXP_N}
    Fields sys[MAX_SYSTEMS];
};
static_assert(sizeof(Work) <= 4096, "field-kernel parameter block above 4 KB");

__device__ __forceinline__ int next_item(int *queue, int *s_item) {
    __syncthreads();
    if (threadIdx.x == 0) *s_item = atomicAdd(queue, 1);
    __syncthreads();
    return *s_item;
}

// The field passes of a call (near, close, far) only read what earlier kernels
// wrote and write separate outputs, so each pass may start on the SMs that the
// one before has run out of items for: programmatic dependent launch.  A pass
// lets its successor start as soon as it runs (pass_begin), and one CTA of each
// pass ends only after the pass before has ended (pass_end), so that whatever
// follows the last pass in the stream follows all of them.  Both are no-ops
// where the launches are not programmatic.
__device__ __forceinline__ void pass_begin() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pass_end() {
    if (blockIdx.x == 0) asm volatile("griddepcontrol.wait;" ::: "memory");
}

// The place of a warp in its CTA: target group g of G, source split sp of S.
struct Place {
    int S, G, g, sp, lane, wid;
    __device__ __forceinline__ Place(int split, int warps)
        : S(split), G(warps / split), lane(threadIdx.x & 31), wid(threadIdx.x >> 5) {
        g = wid & (G - 1);
        sp = wid / G;
    }
};

// Adds the S splits' values v of each of a CTA's targets in split order; the
// result is valid in split 0.  red: FT doubles of shared memory that no warp
// still reads (the barrier here orders it after the last tile).
__device__ __forceinline__ double add_splits(double v, const Place &pl, double *red) {
    if (pl.S == 1) return v;
    __syncthreads();
    red[threadIdx.x] = v;   // threadIdx.x = sp * 32 G + (target group, lane)
    __syncthreads();
    if (pl.sp) return 0.0;
    for (int s = 1; s < pl.S; s++) v += red[threadIdx.x + s * 32 * pl.G];
    return v;
}

// The near ranges of one pass in list order, up to a CTA's THREADS of them at a
// time, cut into chunks of SLOT sources: first[i] = chunks before range i.  A
// tile holds the next chunks whatever ranges they come from (one slot per warp,
// which stages it), so the warps of a CTA stay evenly loaded where ranges are
// short or end inside a tile.
template <int THREADS>
struct RangeTable {
    int begin[THREADS], end[THREADS], first[THREADS];
    int wsum[THREADS / 32], wkeep[THREADS / 32];
};

// Fills t with the kept ranges of e0 .. e0 + THREADS - 1; returns their number and
// the number of chunks.  keep(range, dmin) decides; it leaves in range.x the
// begin, with bit 31 free for its own use.
template <int THREADS, typename Keep>
__device__ __forceinline__ int2 load_ranges(const Fields &a, int e0, int r1, RangeTable<THREADS> &t, Keep keep) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int e = e0 + threadIdx.x;
    int2 r = make_int2(0, 0);
    bool k = false;
    if (e < r1) {
        r = a.rng[e];
        k = keep(r, a.rng_dmin[e]);
    }
    const int n = k ? (r.y - (r.x & 0x7fffffff) + SLOT - 1) / SLOT : 0;
    const unsigned m = __ballot_sync(0xffffffffu, k);
    int incl = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    __syncthreads();   // the table's previous contents are no longer read
    if (lane == 31) {
        t.wsum[wid] = incl;
        t.wkeep[wid] = __popc(m);
    }
    __syncthreads();
    int first = incl - n, pos = __popc(m & ((1u << lane) - 1u)), nr = 0, nch = 0;
#pragma unroll
    for (int w = 0; w < THREADS / 32; w++) {
        if (w < wid) {
            first += t.wsum[w];
            pos += t.wkeep[w];
        }
        nch += t.wsum[w];
        nr += t.wkeep[w];
    }
    if (k) {
        t.begin[pos] = r.x;   // keep() may have set bit 31 anew
        t.end[pos] = r.y;
        t.first[pos] = first;
    }
    __syncthreads();
    return make_int2(nr, nch);
}

// The range that holds chunk c (0 <= c < chunks of the table's nr ranges).
template <int THREADS>
__device__ __forceinline__ int range_of_chunk(const RangeTable<THREADS> &t, int nr, int c) {
    int lo = 0, hi = nr - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (t.first[mid] <= c) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}
// The same from range e on: a warp's chunks follow one another, so it is the last range or
// one of the next, where the search is a chain of five reads of shared memory ahead of a
// tile's loads.  Single-orbital kernels, Yukawa, 50k points, one orbital 1032 -> 995 us; the
// orbital groups, whose registers are full, keep the search (32 orbitals x 1M points 1001
// and 1026 ms).
template <int THREADS>
__device__ __forceinline__ int next_range(const RangeTable<THREADS> &t, int nr, int c, int e) {
    while (e + 1 < nr && t.first[e + 1] <= c) e++;
    return e;
}

// Packed FP32 pairs.  On the sm_100 family one FADD2 / FMUL2 / FFMA2
// instruction applies the same round-to-nearest IEEE operation to two lanes
// held in a register pair, so the pair arithmetic takes half the issue slots
// of its scalar form with bit-identical per-lane results.  The field kernels
// pack two SOURCES (near field) or two proxy points (far field) per
// operation; a target's own values are duplicated once into both lanes.
__device__ __forceinline__ float2 dup2(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 rsqrt2(float2 a) { return make_float2(rsqrt_mufu(a.x), rsqrt_mufu(a.y)); }
// 2^{-a} per lane
__device__ __forceinline__ float2 ex2neg2(float2 a) { return make_float2(ex2_mufu(-a.x), ex2_mufu(-a.y)); }
// 2^{a} per lane
__device__ __forceinline__ float2 ex2pos2(float2 a) { return make_float2(ex2_mufu(a.x), ex2_mufu(a.y)); }
// -log2(r) = -log2(r^2) / 2 per lane
__device__ __forceinline__ float2 nlog2r2(float2 r2) {
    return mul2(dup2(-0.5f), make_float2(lg2_mufu(r2.x), lg2_mufu(r2.y)));
}

// Two pairs (one target, two sources) from their squared scaled distances
// r2 = r'^2; q, w the two sources' charges and weights, nfi = -f_i in both
// lanes.  Per lane:
//   Yukawa   acc += 2^{-r'} / r' * (SS ? q - f_i w : q)
//   Coulomb  acc += (SS ? q - f_i 2^{-r'^2} w : q) / r'
// MASK zeroes a coincident (r = 0) pair.
template <int KERN, bool SS, bool MASK>
__device__ __forceinline__ float2 pair2(float2 r2, float2 q, float2 w, float2 nfi, float2 acc) {
    float2 rinv = rsqrt2(r2);
    if (MASK) {
        rinv.x = r2.x > 0.f ? rinv.x : 0.f;
        rinv.y = r2.y > 0.f ? rinv.y : 0.f;
    }
    if (KERN == KERNEL_YUKAWA) {
        const float2 g = mul2(ex2neg2(mul2(r2, rinv)), rinv);
        return fma2(g, SS ? fma2(nfi, w, q) : q, acc);
    } else if (SS) {
        return fma2(rinv, fma2(mul2(nfi, ex2neg2(r2)), w, q), acc);
    } else {
        return fma2(rinv, q, acc);
    }
}

// Compensated (Kahan) addition of an FP32 partial into (sum, cmp).
__device__ __forceinline__ void kahan_add(float &sum, float &cmp, float part) {
    const float y = part - cmp;
    const float t = sum + y;
    cmp = (t - sum) - y;
    sum = t;
}

__device__ __forceinline__ float4 lds4(const float *p) { return *reinterpret_cast<const float4 *>(p); }
__device__ __forceinline__ float2 lds2(const float *p) { return *reinterpret_cast<const float2 *>(p); }

// Batch-relative source coordinates from the FP32 hi/lo splits (x = h + l to
// 2^-48 |x|, the batch center c = ch + cl likewise), for two sources at once:
// the exact difference of the hi parts as a rounded sum and its error (Knuth's
// two-sum), plus the difference of the lo parts, rounded once.  The value is
// that of FP64 arithmetic rounded to FP32, except that a difference within about
// 2^-48 |x| of a rounding tie may fall on the other side.  FP64 subtraction and
// scaling cost the FP64 pipe (2 lanes per clock and SM) 1,500 clocks per
// 512-source tile, as long as the pair loops of 64 targets take for half of it.
__device__ __forceinline__ float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }
struct Split {
    float2 h, l;   // a coordinate's hi and lo part in both lanes
    __device__ __forceinline__ explicit Split(double c) : h(dup2((float)c)), l(dup2((float)(c - (double)(float)c))) {}
};
// -(x - c) as rounded difference plus error
__device__ __forceinline__ void minus_center(float2 xh, float2 xl, const Split &c, float2 &d, float2 &e) {
    d = add2(c.h, neg2(xh));
    const float2 b = add2(d, neg2(c.h));
    e = add2(add2(c.h, neg2(add2(d, neg2(b)))), neg2(add2(xh, b)));
    e = add2(e, add2(c.l, neg2(xl)));
}
__device__ __forceinline__ float2 neg_relative(float2 xh, float2 xl, const Split &c) {
    float2 d, e;
    minus_center(xh, xl, c, d, e);
    return add2(d, e);
}
// -(x - c) sc, rounded once
__device__ __forceinline__ float2 neg_relative(float2 xh, float2 xl, const Split &c, float2 sc) {
    float2 d, e;
    minus_center(xh, xl, c, d, e);
    const float2 p = mul2(d, sc);
    return add2(p, fma2(e, sc, fma2(d, sc, neg2(p))));
}
// -(x - c) sc in FP64, rounded once (WIDE kernels, for plans whose batches lie so far from the
// origin that the splits' 48 bits would show: Plan::wide)
__device__ __forceinline__ float2 neg_relative64(const double *__restrict__ x, int j0, int j1, double c, double sc) {
    return make_float2(-(float)((x[j0] - c) * sc), -(float)((x[j1] - c) * sc));
}
__device__ __forceinline__ void sts2(float *p, float2 v) { *reinterpret_cast<float2 *>(p) = v; }

// Near-field source tile in shared memory, structure of arrays, NEGATED
// coordinates so that one FADD2 forms t - s for two sources:
//   row 0..2  -x, -y, -z   (ordinary tiles: scaled batch-relative FP32;
//                           PRECISE tiles: hi parts of the absolute FP64
//                           coordinates' FP32 splits)
//   row 3, 4  charge q = f w, weight w
//   row 5..7  -lo parts of the splits (PRECISE tiles only)
// A tile of cnt sources is padded to cnt4 = a multiple of 4 with copies of
// its first source carrying q = w = 0: their terms are exactly +-0.
//
// One slot of a tile (n sources from j0, a multiple of 4) against NT targets, two
// sources per packed operation.  Its pairs are summed in FP32 per lane and the
// two lane sums are added into out, which enters the target's Kahan sum: a long
// FP32 run loses ~sqrt(n) u of its total, and singularity subtraction
// multiplies that loss by |f_i int G| / |phi_i| (often 10-100).
// PRECISE tiles (close ranges): each difference is (t_hi - s_hi) +
// (t_lo - s_lo) -- exact hi differences for nearby points -- and the
// unscaled r^2 is multiplied by sc2 = sc^2, so the shortest pairs keep FP32
// relative precision in r whatever the batch size.
constexpr int NROWS_PRECISE = 8;
template <int KERN, bool SS, bool MASK, bool PRECISE, int NT, int TILE>
__device__ __forceinline__ void near_chunk(const float (*__restrict__ s)[TILE], int j0, int n, const float2 (&tx)[NT],
                                          const float2 (&ty)[NT], const float2 (&tz)[NT], const float2 (&lx)[NT],
                                          const float2 (&ly)[NT], const float2 (&lz)[NT], float2 sc2,
                                          const float2 (&nfi)[NT], float (&out)[NT]) {
    const int j1 = j0 + n;
    float2 part[NT];
#pragma unroll
    for (int k = 0; k < NT; k++) part[k] = make_float2(0.f, 0.f);
#pragma unroll 2
    for (int j = j0; j < j1; j += 4) {
        const float4 X = lds4(s[0] + j), Y = lds4(s[1] + j), Z = lds4(s[2] + j);
        const float4 Q = lds4(s[3] + j), W = lds4(s[4] + j);
        float4 XL = make_float4(0.f, 0.f, 0.f, 0.f), YL = XL, ZL = XL;
        if constexpr (PRECISE) {
            XL = lds4(s[5] + j);
            YL = lds4(s[6] + j);
            ZL = lds4(s[7] + j);
        }
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const float2 sx = h ? make_float2(X.z, X.w) : make_float2(X.x, X.y);
            const float2 sy = h ? make_float2(Y.z, Y.w) : make_float2(Y.x, Y.y);
            const float2 sz = h ? make_float2(Z.z, Z.w) : make_float2(Z.x, Z.y);
            const float2 q = h ? make_float2(Q.z, Q.w) : make_float2(Q.x, Q.y);
            const float2 w = h ? make_float2(W.z, W.w) : make_float2(W.x, W.y);
            const float2 sxl = h ? make_float2(XL.z, XL.w) : make_float2(XL.x, XL.y);
            const float2 syl = h ? make_float2(YL.z, YL.w) : make_float2(YL.x, YL.y);
            const float2 szl = h ? make_float2(ZL.z, ZL.w) : make_float2(ZL.x, ZL.y);
#pragma unroll
            for (int k = 0; k < NT; k++) {
                float2 dx = add2(tx[k], sx), dy = add2(ty[k], sy), dz = add2(tz[k], sz);
                if (PRECISE) {
                    dx = add2(dx, add2(lx[k], sxl));
                    dy = add2(dy, add2(ly[k], syl));
                    dz = add2(dz, add2(lz[k], szl));
                }
                float2 r2 = fma2(dx, dx, fma2(dy, dy, mul2(dz, dz)));
                if (PRECISE) r2 = mul2(r2, sc2);
                part[k] = pair2<KERN, SS, MASK>(r2, q, w, nfi[k], part[k]);
            }
        }
    }
#pragma unroll
    for (int k = 0; k < NT; k++) out[k] = part[k].x + part[k].y;
}

// ---------------------------------------------------------------------------
// Near field, mixed precision.
// ---------------------------------------------------------------------------
// PASS 0 handles the ordinary near ranges, PASS 1 the close ones (double-float
// coordinates, r = 0 mask) into a second output; two passes keep each
// kernel's register footprint at one tile variant's.
// SW warps per CTA: 8 where the mesh is small and eight splits share each target's
// sources, 4 above, where more and smaller CTAs wait less at their barriers (24 warps
// per SM either way).  near + far, ms, 8 and 4 warps: Coulomb 1.5M points 94.3 -> 92.2, 1.34M
// points, degree 4, Yukawa 71.5 -> 66.7; Yukawa 50k points, whole call 1.11 and 1.31.
template <int KERN, bool SS, int NT, int PASS, int SW, bool WIDE = false>
__global__ void __launch_bounds__(32 * SW, 24 / SW) near_mixed(const __grid_constant__ Work w) {
    constexpr int NR = PASS == 1 ? NROWS_PRECISE : 5, ST = 32 * SW, TILE = SW * SLOT;   // warp w stages slot w of a tile
    __shared__ __align__(16) float s_src[NR][TILE];
    __shared__ RangeTable<ST> s_rng;
    __shared__ __align__(16) float s_part[SW * ST];   // S > 1: partials [slot][target of the CTA]
    __shared__ int s_cnt[SW];   // sources of each slot, a multiple of 4; bit 30: leave the Gaussian out
    __shared__ int s_item;
    constexpr int NOEXP = 1 << 30;
    const int tid = threadIdx.x;
    pass_begin();
    for (;;) {
        const int item = next_item(w.queue, &s_item);
        if (item >= w.nitems) break;
        const int4 it = w.items[item];
        const Fields &a = w.sys[it.y >> 16];
        const Place pl(a.split, SW);
        const int b = it.x, orb = it.y & 0xffff;
        const int bn = a.batch_node[b];
        const int te = it.w;
        const double cbx = a.tcenter[3L * bn], cby = a.tcenter[3L * bn + 1],
                     cbz = a.tcenter[3L * bn + 2];
        const float scf = a.kc32[orb];
        const double sc = (double)scf;
        const float2 sc2 = dup2((float)(sc * sc));
        const Split ccx(cbx), ccy(cby), ccz(cbz);
        const float *q = a.q32 + (long)orb * a.ns;
        const float *ft = a.ft32 + (long)orb * a.nt;
        const int r0 = a.rng_off[b], r1 = a.rng_off[b + 1];
        // consecutive targets per thread: the threads with targets form a
        // prefix of the groups, so whole warps past it skip the pair loops.  A warp with
        // at most 32 targets left takes one per lane, at half the cost of two
        const int first = NT * 32 * pl.g;   // of the warp's targets in the item
        const bool warp_busy = it.z + first < te;
        const bool single = NT == 2 && it.z + first + 32 >= te;
        const int place = first + (single ? pl.lane : NT * pl.lane), i0 = it.z + place;
        float2 tx[NT], ty[NT], tz[NT], lx[NT], ly[NT], lz[NT], nfi[NT];
        // S == 1: the Kahan sums of this thread's own targets; S > 1: sum[0], cmp[0]
        // are those of target it.z + tid
        float sum[NT], cmp[NT];
        const int T = 32 * pl.G * NT;
        int pending = 0;   // slots of the last tile whose partials are still to be added
        auto add_pending = [&]() {
            if (tid < T)
                for (int sl = 0; sl < pending; sl++) kahan_add(sum[0], cmp[0], s_part[sl * T + tid]);
        };
#pragma unroll
        for (int k = 0; k < NT; k++) {
            const int i = i0 + k;
            const bool v = i < te && !(single && k > 0);
            if (PASS == 1) {
                const float4 h = v ? a.thi[i] : make_float4(0.f, 0.f, 0.f, 0.f);
                const float4 l = v ? a.tlo[i] : make_float4(0.f, 0.f, 0.f, 0.f);
                tx[k] = dup2(h.x);
                ty[k] = dup2(h.y);
                tz[k] = dup2(h.z);
                lx[k] = dup2(l.x);
                ly[k] = dup2(l.y);
                lz[k] = dup2(l.z);
            } else {
                tx[k] = dup2(v ? (float)((a.tx[i] - cbx) * sc) : 0.f);
                ty[k] = dup2(v ? (float)((a.ty[i] - cby) * sc) : 0.f);
                tz[k] = dup2(v ? (float)((a.tz[i] - cbz) * sc) : 0.f);
                lx[k] = ly[k] = lz[k] = dup2(0.f);
            }
            nfi[k] = dup2(v ? -ft[i] : 0.f);
            sum[k] = 0.f;
            cmp[k] = 0.f;
        }
        for (int e0 = r0; e0 < r1; e0 += ST) {
            // Ranges far enough away: Yukawa terms are exactly 0 in FP32
            // (2^{-r'} with r' > 127 flushes to zero) and the range is left out;
            // the Coulomb Gaussian correction is below 2^-40 of its term and is
            // left out (bit 31 of the table's begin, free once the pass is chosen).
            const int2 n = load_ranges(a, e0, r1, s_rng, [&](int2 &r, float dmin) {
                if (range_is_close(r) != (PASS == 1)) return false;
                const float dm = dmin * scf;
                if (KERN == KERNEL_YUKAWA && dm > 127.f) return false;
                const bool noexp = KERN == KERNEL_COULOMB && SS && PASS == 0 && dm * dm > 40.f;
                r.x = range_begin(r) | (noexp ? (int)0x80000000u : 0);
                return true;
            });
            int range = 0;
            for (int c0 = 0; c0 < n.y; c0 += SW) {
                __syncthreads();   // the previous tile is no longer read, its partials are written
                if (pl.S > 1) {
                    add_pending();
                    pending = min(SW, n.y - c0);
                }
                const int c = c0 + pl.wid;
                int cnt4 = 0, flag = 0;
                if (c < n.y) {
                    const int e = range = next_range(s_rng, n.x, c, range);
                    const int rb = s_rng.begin[e];
                    const int t0 = (rb & 0x7fffffff) + (c - s_rng.first[e]) * SLOT;
                    const int cnt = min(SLOT, s_rng.end[e] - t0);
                    cnt4 = (cnt + 3) & ~3;
                    flag = rb < 0 ? NOEXP : 0;
                    const int j = 2 * pl.lane, d = pl.wid * SLOT + j;
                    if (j < cnt4) {
                        const bool real0 = j < cnt, real1 = j + 1 < cnt;
                        const int j0 = t0 + (real0 ? j : 0), j1 = t0 + (real1 ? j + 1 : 0);   // padding: the first source
                        if constexpr (WIDE) {
                            sts2(&s_src[0][d], neg_relative64(a.sx, j0, j1, cbx, sc));
                            sts2(&s_src[1][d], neg_relative64(a.sy, j0, j1, cby, sc));
                            sts2(&s_src[2][d], neg_relative64(a.sz, j0, j1, cbz, sc));
                        } else {
                            const float4 h0 = a.shi[j0], h1 = a.shi[j1], l0 = a.slo[j0], l1 = a.slo[j1];
                            const float2 hx = make_float2(h0.x, h1.x), hy = make_float2(h0.y, h1.y),
                                         hz = make_float2(h0.z, h1.z), qx = make_float2(l0.x, l1.x),
                                         qy = make_float2(l0.y, l1.y), qz = make_float2(l0.z, l1.z);
                            if constexpr (PASS == 1) {
                                sts2(&s_src[0][d], neg2(hx));
                                sts2(&s_src[1][d], neg2(hy));
                                sts2(&s_src[2][d], neg2(hz));
                                sts2(&s_src[5][d], neg2(qx));
                                sts2(&s_src[6][d], neg2(qy));
                                sts2(&s_src[7][d], neg2(qz));
                            } else {
                                sts2(&s_src[0][d], neg_relative(hx, qx, ccx, dup2(scf)));
                                sts2(&s_src[1][d], neg_relative(hy, qy, ccy, dup2(scf)));
                                sts2(&s_src[2][d], neg_relative(hz, qz, ccz, dup2(scf)));
                            }
                        }
                        sts2(&s_src[3][d], make_float2(real0 ? q[j0] : 0.f, real1 ? q[j1] : 0.f));
                        sts2(&s_src[4][d], make_float2(real0 ? a.w32[j0] : 0.f, real1 ? a.w32[j1] : 0.f));
                    }
                }
                if (pl.lane == 0) s_cnt[pl.wid] = cnt4 | flag;
                __syncthreads();
                if (!warp_busy) continue;
                for (int sl = pl.sp; sl < SW; sl += pl.S) {
                    const int m = s_cnt[sl];
                    if (m == 0) break;
                    float part[NT];
                    auto chunk = [&](auto nt) {
                        constexpr int N = decltype(nt)::value;
                        const float2(&x)[N] = reinterpret_cast<const float2(&)[N]>(tx), (&y)[N] = reinterpret_cast<const float2(&)[N]>(ty),
                                    (&z)[N] = reinterpret_cast<const float2(&)[N]>(tz), (&u)[N] = reinterpret_cast<const float2(&)[N]>(lx),
                                    (&v)[N] = reinterpret_cast<const float2(&)[N]>(ly), (&w)[N] = reinterpret_cast<const float2(&)[N]>(lz),
                                    (&f)[N] = reinterpret_cast<const float2(&)[N]>(nfi);
                        float(&o)[N] = reinterpret_cast<float(&)[N]>(part);
                        if (PASS == 1)
                            near_chunk<KERN, SS, true, true, N, TILE>(s_src, sl * SLOT, m, x, y, z, u, v, w, sc2, f, o);
                        else if (KERN == KERNEL_COULOMB && SS && (m & NOEXP))
                            near_chunk<KERN, false, false, false, N, TILE>(s_src, sl * SLOT, m & ~NOEXP, x, y, z, u, v, w,
                                                                           sc2, f, o);
                        else
                            near_chunk<KERN, SS, false, false, N, TILE>(s_src, sl * SLOT, m, x, y, z, u, v, w, sc2, f, o);
                    };
                    if (single) chunk(std::integral_constant<int, 1>());
                    else chunk(std::integral_constant<int, NT>());
#pragma unroll
                    for (int k = 0; k < NT; k++) {
                        if (single && k > 0) break;
                        if (pl.S == 1) kahan_add(sum[k], cmp[k], part[k]);
                        else s_part[sl * T + place + k] = part[k];
                    }
                }
            }
        }
        if (pl.S > 1) {
            __syncthreads();
            add_pending();
            if (tid < T && it.z + tid < te)
                a.out[(long)orb * a.nt + it.z + tid] = ((double)sum[0] - (double)cmp[0]) * sc;
            continue;
        }
#pragma unroll
        for (int k = 0; k < NT; k++)
            if (i0 + k < te && !(single && k > 0)) a.out[(long)orb * a.nt + i0 + k] = ((double)sum[k] - (double)cmp[k]) * sc;
    }
    pass_end();
}

// ---------------------------------------------------------------------------
// Far field, mixed precision.  The proxy grid is a tensor product, so r'^2
// is assembled from per-axis squares: one packed add per two proxy points.
// Two proxy points along the innermost axis share each packed operation; the
// staged charges and weights have that axis padded to an even length n1p
// (padding: charge and weight 0, the distance of the first point).  Coulomb
// subtraction: when the whole cluster lies so far that r'^2 > 40 for every
// proxy point, the Gaussian term f_i what_k 2^{-r'^2} is below 2^-40 of
// f_i what_k and is dropped (one MUFU op less per pair); Yukawa clusters
// with r' > 127 everywhere add exactly 0 in FP32 (2^{-r'} flushes to zero)
// and are skipped.  add(k1, k, v) takes target k's partial of slab k1.
// ---------------------------------------------------------------------------
template <int MAXN1>
__host__ __device__ constexpr int even_up() { return MAXN1 + (MAXN1 & 1); }
// How much of the loops over a proxy grid is known at compile time (far_loops
// chooses).  FAR_ANY: n + 1 <= MAXN1.  FAR_ROWS: n + 1 = MAXN1 - 1 or MAXN1 (even), so a
// row is MAXN1 / 2 pairs of points without tests.  FAR_FIXED: n + 1 = MAXN1.  Whole calls,
// FAR_ANY -> FAR_ROWS: ring sweep, 150k points, 10 orbitals, degree 5 22.9 -> 21.0 ms; Yukawa,
// 657k points, degree 5 67.3 -> 63.7; two-mesh, 5 Coulomb fields, degree 10 261 -> 247; 10
// orbitals, degree 8 51.6 -> 49.3; Coulomb, 144k points, degree 4 3.70 -> 3.34.
enum { FAR_ANY, FAR_ROWS, FAR_FIXED };

template <int KERN, bool SS, bool EXPTERM, int MAXN1, int NT, int LOOPS, typename Add>
__device__ __forceinline__ void far_cluster(const float *__restrict__ s_q, const float *__restrict__ s_w,
                                            const float (*s_p)[MAXN1], int n1_in, int slab0, int slab_step,
                                            const float (&tx)[NT], const float (&ty)[NT], const float (&tz)[NT],
                                            const float2 (&nfi)[NT], Add add) {
    constexpr int MH = even_up<MAXN1>() / 2;
    constexpr bool PSS = KERN == KERNEL_YUKAWA ? SS : (SS && EXPTERM);
    const int n1 = LOOPS == FAR_FIXED ? MAXN1 : n1_in;
    const int n1p = LOOPS ? even_up<MAXN1>() : n1 + (n1 & 1);
    float2 dz2[NT][MH];
#pragma unroll
    for (int k = 0; k < NT; k++)
#pragma unroll
        for (int m = 0; m < MH; m++) {
            const float d0 = tz[k] - s_p[2][2 * m < n1 ? 2 * m : 0];
            const float d1 = tz[k] - s_p[2][2 * m + 1 < n1 ? 2 * m + 1 : 0];
            dz2[k][m] = make_float2(d0 * d0, d1 * d1);
        }
    for (int k1 = slab0; k1 < n1; k1 += slab_step) {  // one (n+1)^2 slab per FP32 partial, then Kahan
        int idx = k1 * n1 * n1p;
        float2 part[NT];
        float dx2[NT];
#pragma unroll
        for (int k = 0; k < NT; k++) {
            part[k] = make_float2(0.f, 0.f);
            const float dx = tx[k] - s_p[0][k1];
            dx2[k] = dx * dx;
        }
        for (int k2 = 0; k2 < n1; k2++) {
            float2 rxy[NT];
#pragma unroll
            for (int k = 0; k < NT; k++) {
                const float dy = ty[k] - s_p[1][k2];
                rxy[k] = dup2(fmaf(dy, dy, dx2[k]));
            }
#pragma unroll
            for (int m = 0; m < MH; m++) {
                if (LOOPS || 2 * m < n1) {
                    const float2 q = lds2(s_q + idx + 2 * m), wv = lds2(s_w + idx + 2 * m);
#pragma unroll
                    for (int k = 0; k < NT; k++)
                        part[k] = pair2<KERN, PSS, false>(add2(rxy[k], dz2[k][m]), q, wv, nfi[k], part[k]);
                }
            }
            idx += n1p;
        }
#pragma unroll
        for (int k = 0; k < NT; k++) add(k1, k, part[k].x + part[k].y);
    }
}

// The slabs of cluster number cl of a tile that split sp of S takes start here
// and go on in steps of S: slabs are dealt to the splits in turn over the
// whole tile.
__device__ __forceinline__ int first_slab(int cl, int n1, const Place &pl) { return (pl.sp - cl * n1) & (pl.S - 1); }

// FAR_CL clusters are staged per pair of barriers.
template <int MAXN1>
__host__ __device__ constexpr int far_clusters() { return MAXN1 <= 4 ? 8 : (MAXN1 <= 8 ? 4 : 2); }
// Partials of a far tile where a target's slabs are split: at least one cluster's
// slabs of the CTA's targets (two warps of targets with two targets per thread).
__host__ __device__ constexpr int far_part(int warps) { return warps == 4 ? 2048 : 4096; }
static_assert(far_part(4) >= (MAX_DEGREE + 1) * 128 && far_part(8) >= (MAX_DEGREE + 1) * 256, "slabs of one cluster");

template <int KERN, bool SS, int MAXN1, int NT, int SW, int LOOPS = FAR_ANY>
__global__ void __launch_bounds__(32 * SW, 16 / SW) far_mixed(const __grid_constant__ Work w) {
    constexpr int MAXPP = MAXN1 * MAXN1 * even_up<MAXN1>();
    constexpr int FAR_CL = far_clusters<MAXN1>(), ST = 32 * SW, FAR_PART = far_part(SW);
    __shared__ __align__(16) float s_q[FAR_CL][MAXPP];
    __shared__ __align__(16) float s_w[FAR_CL][MAXPP];
    __shared__ float s_p[FAR_CL][3][MAXN1];
    __shared__ int s_slot[ST];   // the item's next clusters that count: slot << 1 | leave the Gaussian out
    __shared__ int s_kept[SW];
    __shared__ float s_part[FAR_PART];   // S > 1: partials [cluster of the tile, slab][target of the CTA]
    __shared__ int s_item;
    const int tid = threadIdx.x;
    pass_begin();
    for (;;) {
        const int item = next_item(w.queue, &s_item);
        if (item >= w.nitems) break;
        const int4 it = w.items[item];
        const Fields &a = w.sys[it.y >> 16];
        const Place pl(a.split, SW);
        const int b = it.x, orb = it.y & 0xffff;
        const int n1 = LOOPS == FAR_FIXED ? MAXN1 : a.n1, P = LOOPS == FAR_FIXED ? MAXN1 * MAXN1 * MAXN1 : a.P;
        const int n1p = LOOPS ? even_up<MAXN1>() : n1 + (n1 & 1), Pp = n1 * n1 * n1p;
        const int f0 = a.far_off[b], f1 = a.far_off[b + 1];
        const int bn = a.batch_node[b];
        const int te = it.w;
        const double cb[3] = {a.tcenter[3L * bn], a.tcenter[3L * bn + 1], a.tcenter[3L * bn + 2]};
        const double rb = a.tradius[bn];
        const float scf = a.kc32[orb];
        const double sc = (double)scf;
        const float *ft = a.ft32 + (long)orb * a.nt;
        const float *qh = a.qhat32 + (long)orb * a.nslots * P;
        const int first = NT * 32 * pl.g;   // as in near_mixed
        const bool warp_busy = it.z + first < te;
        const bool single = NT == 2 && it.z + first + 32 >= te;
        const int place = first + (single ? pl.lane : NT * pl.lane), i0 = it.z + place;
        float tx[NT], ty[NT], tz[NT];
        // S == 1: the Kahan sums of this thread's own targets; S > 1: sum[0], cmp[0]
        // are those of target it.z + tid
        float sum[NT], cmp[NT];
        const int T = 32 * pl.G * NT;
        const int tile = pl.S == 1 ? FAR_CL : min(FAR_CL, max(1, FAR_PART / (T * n1)));
        int pending = 0;   // slabs of the last tile whose partials are still to be added
        auto add_pending = [&]() {
            if (tid < T)
                for (int u = 0; u < pending; u++) kahan_add(sum[0], cmp[0], s_part[u * T + tid]);
        };
        float2 nfi[NT];
#pragma unroll
        for (int k = 0; k < NT; k++) {
            const int i = i0 + k;
            const bool v = i < te && !(single && k > 0);
            tx[k] = v ? (float)(a.tx[i] - cb[0]) * scf : 0.f;
            ty[k] = v ? (float)(a.ty[i] - cb[1]) * scf : 0.f;
            tz[k] = v ? (float)(a.tz[i] - cb[2]) * scf : 0.f;
            nfi[k] = dup2(v ? -ft[i] : 0.f);
            sum[k] = 0.f;
            cmp[k] = 0.f;
        }
        for (int e0 = f0; e0 < f1; e0 += ST) {
            int slot = 0, mode = 2;
            if (e0 + tid < f1) {
                slot = a.node_slot[a.far_list[e0 + tid]];
                const double *g = a.geom + 6L * slot;
                // smallest scaled distance from the batch to the proxy box (conservative)
                const double dx = cb[0] - g[0], dy = cb[1] - g[1], dz = cb[2] - g[2];
                const double rc = sqrt(g[3] * g[3] + g[4] * g[4] + g[5] * g[5]);
                const double dmin = (sqrt(dx * dx + dy * dy + dz * dz) - rb - rc) * sc * (1.0 - 1e-6);
                mode = 0;
                if (KERN == KERNEL_YUKAWA && dmin > 127.0) mode = 2;  // 2^{-r'} flushes to 0: adds exactly 0
                // Gaussian correction below 2^-40 of its own term everywhere: dropped
                if (KERN == KERNEL_COULOMB && SS && dmin > 0.0 && dmin * dmin > 40.0) mode = 1;
            }
            const unsigned kept = __ballot_sync(0xffffffffu, mode != 2);
            __syncthreads();   // the previous clusters' slots are no longer read
            if (pl.lane == 0) s_kept[pl.wid] = __popc(kept);
            __syncthreads();
            int pos = __popc(kept & ((1u << pl.lane) - 1u)), ne = 0;
#pragma unroll
            for (int v = 0; v < SW; v++) {
                if (v < pl.wid) pos += s_kept[v];
                ne += s_kept[v];
            }
            if (mode != 2) s_slot[pos] = (slot << 1) | mode;
            for (int c0 = 0; c0 < ne; c0 += tile) {
                const int nc = min(tile, ne - c0);
                __syncthreads();   // slots written; the previous tile is no longer read, its partials are written
                if (pl.S > 1) {
                    add_pending();
                    pending = nc * n1;
                }
                for (int k = tid; k < Pp; k += ST) {   // the same grid point of all the tile's clusters at once
                    const int row = k / n1p, k3 = k - row * n1p, src = row * n1 + k3;
                    float vq[FAR_CL], vw[FAR_CL];
#pragma unroll
                    for (int cl = 0; cl < FAR_CL; cl++) {
                        const bool real = cl < nc && k3 < n1;
                        const long at = real ? (long)(s_slot[c0 + cl] >> 1) * P + src : 0;
                        vq[cl] = real ? qh[at] : 0.f;
                        vw[cl] = real ? a.what32[at] : 0.f;
                    }
#pragma unroll
                    for (int cl = 0; cl < FAR_CL; cl++) {
                        s_q[cl][k] = vq[cl];
                        s_w[cl][k] = vw[cl];
                    }
                }
                for (int u = tid; u < 3 * n1 * nc; u += ST) {
                    const int cl = u / (3 * n1), v = u - cl * 3 * n1;
                    const int d = v / n1, m = v - d * n1;
                    const double *g = a.geom + 6L * (s_slot[c0 + cl] >> 1);
                    const double cbd = d == 0 ? cb[0] : (d == 1 ? cb[1] : cb[2]);
                    s_p[cl][d][m] = (float)((g[d] + g[3 + d] * a.tn[m]) - cbd) * scf;
                }
                __syncthreads();
                if (!warp_busy) continue;
                for (int cl = 0; cl < nc; cl++) {
                    auto add = [&](int k1, int k, float part) {
                        if (pl.S == 1) kahan_add(sum[k], cmp[k], part);
                        else s_part[(cl * n1 + k1) * T + place + k] = part;
                    };
                    const int slab = first_slab(cl, n1, pl);
                    auto cluster = [&](auto nt) {
                        constexpr int N = decltype(nt)::value;
                        const float(&x)[N] = reinterpret_cast<const float(&)[N]>(tx), (&y)[N] = reinterpret_cast<const float(&)[N]>(ty),
                                   (&z)[N] = reinterpret_cast<const float(&)[N]>(tz);
                        const float2(&f)[N] = reinterpret_cast<const float2(&)[N]>(nfi);
                        if (s_slot[c0 + cl] & 1)
                            far_cluster<KERN, SS, false, MAXN1, N, LOOPS>(s_q[cl], s_w[cl], s_p[cl], n1, slab, pl.S, x, y,
                                                                          z, f, add);
                        else
                            far_cluster<KERN, SS, true, MAXN1, N, LOOPS>(s_q[cl], s_w[cl], s_p[cl], n1, slab, pl.S, x, y,
                                                                         z, f, add);
                    };
                    if (single) cluster(std::integral_constant<int, 1>());
                    else cluster(std::integral_constant<int, NT>());
                }
            }
        }
        if (pl.S > 1) {
            __syncthreads();
            add_pending();
            if (tid < T && it.z + tid < te)
                a.out[(long)orb * a.nt + it.z + tid] = ((double)sum[0] - (double)cmp[0]) * sc;
            continue;
        }
#pragma unroll
        for (int k = 0; k < NT; k++)
            if (i0 + k < te && !(single && k > 0)) a.out[(long)orb * a.nt + i0 + k] = ((double)sum[k] - (double)cmp[k]) * sc;
    }
    pass_end();
}

// ---------------------------------------------------------------------------
// Orbital-group kernels (Yukawa, mixed precision): one item = (batch, group of
// OG orbitals).  Per two sources (or two proxy points) the differences, r^2,
// r (via rsqrt) and -log2 r (via lg2) are formed once for the group in packed
// operations; each orbital then adds 2^{-k_o log2(e) r - log2 r} * c, which is
// e^{-k_o r} / r * c with the 1/r folded into the exponent.  -k_o log2(e) is
// the orbital's FP32 constant sc (orbital_constants), and the subtraction term
// uses the k that sc represents, so one FP32 constant suffices.  Coordinates
// are translated to the batch center but not scaled (each orbital has its own
// k).  Charges are staged as float4
// {q(o, j), q(o, j+1), q(o+1, j), q(o+1, j+1)} per (pair of sources, pair of
// orbitals), so one 16-byte shared read serves four (pair, orbital) terms.
// Orbitals past the last one of the request have zero charges and are not
// written.
// ---------------------------------------------------------------------------
constexpr int GT = 128;            // threads (targets) per CTA
constexpr int GW = GT / 32;
constexpr int GTILE = GW * SLOT;   // sources per group tile, one slot per warp

__device__ __forceinline__ int q4_pos(int j, int o, int og) {   // float index of q(o, j) in the staged layout
    return (((j >> 1) * (og >> 1) + (o >> 1)) << 2) + ((o & 1) << 1) + (j & 1);
}

// Group tile rows: 0..2 negated coordinates (batch-relative, or hi parts of
// the absolute splits), 3 weight, 4..6 negated lo parts (PRECISE).
template <bool SS, bool MASK, bool PRECISE, int OG, int N2 = OG / 2>
__device__ __forceinline__ void group_chunk(const float (*__restrict__ s)[GTILE], const float4 *__restrict__ s_q4,
                                           int j0, int n, float2 tx, float2 ty, float2 tz, float2 lx, float2 ly,
                                           float2 lz, const float2 (&nfi)[OG], const float2 (&kc)[OG],
                                           float (&sum)[OG], float (&cmp)[OG]) {
    const int j1 = j0 + n;
    float2 part[2 * N2];
#pragma unroll
    for (int o = 0; o < 2 * N2; o++) part[o] = make_float2(0.f, 0.f);
#pragma unroll 1   // measured: unrolling the source loop slows the group kernels
    for (int j = j0; j < j1; j += 2) {
        float2 dx = add2(tx, lds2(s[0] + j)), dy = add2(ty, lds2(s[1] + j)), dz = add2(tz, lds2(s[2] + j));
        if constexpr (PRECISE) {
            dx = add2(dx, add2(lx, lds2(s[4] + j)));
            dy = add2(dy, add2(ly, lds2(s[5] + j)));
            dz = add2(dz, add2(lz, lds2(s[6] + j)));
        }
        const float2 wv = lds2(s[3] + j);
        const float2 r2 = fma2(dx, dx, fma2(dy, dy, mul2(dz, dz)));
        float2 rinv = rsqrt2(r2);
        float2 nl = nlog2r2(r2);
        if (MASK) {   // r = 0: r = 0 and 2^{-inf} = 0, so the pair adds exactly 0
            rinv.x = r2.x > 0.f ? rinv.x : 0.f;
            rinv.y = r2.y > 0.f ? rinv.y : 0.f;
            nl.x = r2.x > 0.f ? nl.x : -INFINITY;
            nl.y = r2.y > 0.f ? nl.y : -INFINITY;
        }
        const float2 r = mul2(r2, rinv);
#pragma unroll
        for (int o2 = 0; o2 < N2; o2++) {
            const float4 q4 = s_q4[(j >> 1) * (OG / 2) + o2];
#pragma unroll
            for (int u = 0; u < 2; u++) {
                const int o = 2 * o2 + u;
                const float2 q = u ? make_float2(q4.z, q4.w) : make_float2(q4.x, q4.y);
                // e^{-k r} / r = 2^{-k log2(e) r - log2 r}
                const float2 g = ex2pos2(fma2(kc[o], r, nl));
                part[o] = fma2(g, SS ? fma2(nfi[o], wv, q) : q, part[o]);
            }
        }
    }
#pragma unroll
    for (int o = 0; o < 2 * N2; o++) kahan_add(sum[o], cmp[o], part[o].x + part[o].y);
}

// The chunk or proxy grid for the n2 pairs of orbitals that an item holds (its
// last ones may be missing): FN<N2>(n2's value).
template <int OG, typename FN>
__device__ __forceinline__ void for_pairs(int n2, FN &&fn) {
    if constexpr (OG == 8) {
        switch (n2) {
        case 1: fn(std::integral_constant<int, 1>()); return;
        case 2: fn(std::integral_constant<int, 2>()); return;
        case 3: fn(std::integral_constant<int, 3>()); return;
        }
    } else if (n2 == 1) {
        fn(std::integral_constant<int, 1>());
        return;
    }
    fn(std::integral_constant<int, OG / 2>());
}
// Pairs of orbitals of an item of OG that starts at g0.
template <int OG>
__device__ __forceinline__ int item_pairs(int norb, int g0) { return min(OG / 2, (norb - g0 + 1) >> 1); }

template <bool SS, int OG, int PASS, bool WIDE = false>
__global__ void __launch_bounds__(GT, 4) near_group(const __grid_constant__ Work w) {
    constexpr int NR = PASS == 1 ? 7 : 4;
    __shared__ __align__(16) float s_src[NR][GTILE];
    __shared__ float4 s_q4[GTILE * OG / 4];
    __shared__ RangeTable<GT> s_rng;
    __shared__ int s_cnt[GW];
    __shared__ int s_item;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    pass_begin();
    for (;;) {
        const int item = next_item(w.queue, &s_item);
        if (item >= w.nitems) break;
        const int4 it = w.items[item];
        const Fields &a = w.sys[it.y >> 16];
        const int b = it.x, g0 = it.y & 0xffff;
        const int bn = a.batch_node[b];
        const double cbx = a.tcenter[3L * bn], cby = a.tcenter[3L * bn + 1], cbz = a.tcenter[3L * bn + 2];
        const Split ccx(cbx), ccy(cby), ccz(cbz);
        float2 kc[OG];
        float kmin = 3.4e38f;
#pragma unroll
        for (int o = 0; o < OG; o++) {
            const int orb = g0 + o;
            kc[o] = dup2(orb < a.norb ? -a.kc32[orb] : 0.f);   // -k log2(e) as one FP32 constant
            if (orb < a.norb) kmin = fminf(kmin, a.kc32[orb]);
        }
        const int n2 = item_pairs<OG>(a.norb, g0);
        const int r0 = a.rng_off[b], r1 = a.rng_off[b + 1];
        const int i = it.z + tid;
        const bool v = i < it.w;
        const bool warp_busy = it.z + (tid & ~31) < it.w;
        float2 tx, ty, tz, lx = dup2(0.f), ly = dup2(0.f), lz = dup2(0.f);
        if (PASS == 1) {  // absolute hi/lo splits (see near_chunk)
            const float4 h = v ? a.thi[i] : make_float4(0.f, 0.f, 0.f, 0.f);
            const float4 l = v ? a.tlo[i] : make_float4(0.f, 0.f, 0.f, 0.f);
            tx = dup2(h.x);
            ty = dup2(h.y);
            tz = dup2(h.z);
            lx = dup2(l.x);
            ly = dup2(l.y);
            lz = dup2(l.z);
        } else {
            tx = dup2(v ? (float)(a.tx[i] - cbx) : 0.f);
            ty = dup2(v ? (float)(a.ty[i] - cby) : 0.f);
            tz = dup2(v ? (float)(a.tz[i] - cbz) : 0.f);
        }
        float2 nfi[OG];
        float sum[OG], cmp[OG];
#pragma unroll
        for (int o = 0; o < OG; o++) {
            const int orb = g0 + o;
            nfi[o] = dup2((v && orb < a.norb) ? -a.ft32[(long)orb * a.nt + i] : 0.f);
            sum[o] = 0.f;
            cmp[o] = 0.f;
        }
        for (int e0 = r0; e0 < r1; e0 += GT) {
            const int2 n = load_ranges(a, e0, r1, s_rng, [&](int2 &r, float dmin) {
                if (range_is_close(r) != (PASS == 1)) return false;
                r.x = range_begin(r);
                return !(dmin * kmin > 127.f);   // beyond: every orbital's term is exactly 0
            });
            for (int c0 = 0; c0 < n.y; c0 += GW) {
                __syncthreads();   // the previous tile is no longer read
                const int c = c0 + wid;
                int cnt2 = 0;
                if (c < n.y) {
                    const int e = range_of_chunk(s_rng, n.x, c);
                    const int t0 = s_rng.begin[e] + (c - s_rng.first[e]) * SLOT;
                    const int cnt = min(SLOT, s_rng.end[e] - t0);
                    cnt2 = (cnt + 1) & ~1;
                    const int j = 2 * lane, d = wid * SLOT + j;
                    if (j < cnt2) {
                        const bool real0 = j < cnt, real1 = j + 1 < cnt;
                        const int j0 = t0 + (real0 ? j : 0), j1 = t0 + (real1 ? j + 1 : 0);   // padding: the first source
                        if constexpr (WIDE) {
                            sts2(&s_src[0][d], neg_relative64(a.sx, j0, j1, cbx, 1.0));
                            sts2(&s_src[1][d], neg_relative64(a.sy, j0, j1, cby, 1.0));
                            sts2(&s_src[2][d], neg_relative64(a.sz, j0, j1, cbz, 1.0));
                        } else {
                            const float4 h0 = a.shi[j0], h1 = a.shi[j1], l0 = a.slo[j0], l1 = a.slo[j1];
                            const float2 hx = make_float2(h0.x, h1.x), hy = make_float2(h0.y, h1.y),
                                         hz = make_float2(h0.z, h1.z), qx = make_float2(l0.x, l1.x),
                                         qy = make_float2(l0.y, l1.y), qz = make_float2(l0.z, l1.z);
                            if constexpr (PASS == 1) {
                                sts2(&s_src[0][d], neg2(hx));
                                sts2(&s_src[1][d], neg2(hy));
                                sts2(&s_src[2][d], neg2(hz));
                                sts2(&s_src[4][d], neg2(qx));
                                sts2(&s_src[5][d], neg2(qy));
                                sts2(&s_src[6][d], neg2(qz));
                            } else {
                                sts2(&s_src[0][d], neg_relative(hx, qx, ccx));
                                sts2(&s_src[1][d], neg_relative(hy, qy, ccy));
                                sts2(&s_src[2][d], neg_relative(hz, qz, ccz));
                            }
                        }
                        sts2(&s_src[3][d], make_float2(real0 ? a.w32[j0] : 0.f, real1 ? a.w32[j1] : 0.f));
                    }
                    // charges: lanes take the float4s of the staged layout in turn (pairs of
                    // sources x pairs of orbitals), all loads before the first store
                    constexpr int LP = 32 * 2 / OG;   // pairs of sources per turn of the warp
                    const int o2 = lane % (OG / 2), oa = g0 + 2 * o2;
                    const bool ha = oa < a.norb, hb = oa + 1 < a.norb;
                    const float *qa = a.q32 + (long)(ha ? oa : g0) * a.ns + t0, *qb = qa + (hb ? a.ns : 0);
                    float4 q[SLOT / 2 / LP];
#pragma unroll
                    for (int u = 0; u < SLOT / 2 / LP; u++) {
                        const int ja = 2 * (u * LP + lane / (OG / 2));
                        const bool r0v = ja < cnt, r1v = ja + 1 < cnt;
                        q[u] = make_float4(ha && r0v ? qa[ja] : 0.f, ha && r1v ? qa[ja + 1] : 0.f,
                                           hb && r0v ? qb[ja] : 0.f, hb && r1v ? qb[ja + 1] : 0.f);
                    }
#pragma unroll
                    for (int u = 0; u < SLOT / 2 / LP; u++) s_q4[wid * (SLOT * OG / 4) + u * 32 + lane] = q[u];
                }
                if (lane == 0) s_cnt[wid] = cnt2;
                __syncthreads();
                if (!warp_busy) continue;
                for (int sl = 0; sl < GW; sl++) {
                    const int m = s_cnt[sl];
                    if (m == 0) break;
                    for_pairs<OG>(n2, [&](auto c) {
                        group_chunk<SS, PASS == 1, PASS == 1, OG, decltype(c)::value>(
                            s_src, s_q4, sl * SLOT, m, tx, ty, tz, lx, ly, lz, nfi, kc, sum, cmp);
                    });
                }
            }
        }
        if (v) {
#pragma unroll
            for (int o = 0; o < OG; o++)
                if (g0 + o < a.norb) a.out[(long)(g0 + o) * a.nt + i] = (double)sum[o] - (double)cmp[o];
        }
    }
    pass_end();
}

// One staged proxy grid against one target for a group of orbitals (see
// far_cluster for the padded innermost axis).
template <bool SS, int MAXN1, int OG, int LOOPS = FAR_ANY, int N2 = OG / 2>
__device__ __forceinline__ void far_group_cluster(const float4 *__restrict__ s_q4, const float *__restrict__ s_w,
                                                  const float (*s_p)[MAXN1], int n1_in,
                                                  float tx, float ty, float tz, const float2 (&nfi)[OG],
                                                  const float2 (&kc)[OG], float (&sum)[OG], float (&cmp)[OG]) {
    constexpr int MH = even_up<MAXN1>() / 2;
    const int n1 = LOOPS == FAR_FIXED ? MAXN1 : n1_in;
    const int n1p = LOOPS ? even_up<MAXN1>() : n1 + (n1 & 1);
    float2 dz2[MH];
#pragma unroll
    for (int m = 0; m < MH; m++) {
        const float d0 = tz - s_p[2][2 * m < n1 ? 2 * m : 0];
        const float d1 = tz - s_p[2][2 * m + 1 < n1 ? 2 * m + 1 : 0];
        dz2[m] = make_float2(d0 * d0, d1 * d1);
    }
    int idx = 0;
    for (int k1 = 0; k1 < n1; k1++) {
        float2 part[2 * N2];
#pragma unroll
        for (int o = 0; o < 2 * N2; o++) part[o] = make_float2(0.f, 0.f);
        const float dx = tx - s_p[0][k1];
        const float dx2 = dx * dx;
        for (int k2 = 0; k2 < n1; k2++) {
            const float dy = ty - s_p[1][k2];
            const float2 rxy = dup2(fmaf(dy, dy, dx2));
#pragma unroll
            for (int m = 0; m < MH; m++) {
                if (LOOPS || 2 * m < n1) {
                    const float2 r2 = add2(rxy, dz2[m]);
                    const float2 rr = mul2(r2, rsqrt2(r2));
                    const float2 nl = nlog2r2(r2);
                    const float2 wk = lds2(s_w + idx + 2 * m);
#pragma unroll
                    for (int o2 = 0; o2 < N2; o2++) {
                        const float4 q4 = s_q4[((idx >> 1) + m) * (OG / 2) + o2];
#pragma unroll
                        for (int u = 0; u < 2; u++) {
                            const int o = 2 * o2 + u;
                            const float2 q = u ? make_float2(q4.z, q4.w) : make_float2(q4.x, q4.y);
                            const float2 g = ex2pos2(fma2(kc[o], rr, nl));
                            part[o] = fma2(g, SS ? fma2(nfi[o], wk, q) : q, part[o]);
                        }
                    }
                }
            }
            idx += n1p;
        }
#pragma unroll
        for (int o = 0; o < 2 * N2; o++) kahan_add(sum[o], cmp[o], part[o].x + part[o].y);
    }
}

// Dynamic shared memory of far_group: the staged charges (Pp * OG floats,
// Pp = n1 * n1 * n1p) then the weights (Pp floats), for the largest grid of
// the launch's systems (above 48 KB at degree 10 with 8 orbitals).
__host__ __device__ constexpr size_t far_group_smem(int n1, int og) {
    return sizeof(float) * (size_t)n1 * n1 * (n1 + (n1 & 1)) * (og + 1);
}

template <bool SS, int MAXN1, int OG, int LOOPS = FAR_ANY>
__global__ void __launch_bounds__(GT, 4) far_group(const __grid_constant__ Work w) {
    extern __shared__ __align__(16) float s_dyn[];
    __shared__ float s_p[3][MAXN1];
    __shared__ int s_item;
    float4 *s_q4 = reinterpret_cast<float4 *>(s_dyn);
    const int tid = threadIdx.x;
    pass_begin();
    for (;;) {
        const int item = next_item(w.queue, &s_item);
        if (item >= w.nitems) break;
        const int4 it = w.items[item];
        const Fields &a = w.sys[it.y >> 16];
        const int b = it.x, g0 = it.y & 0xffff;
        const int n1 = LOOPS == FAR_FIXED ? MAXN1 : a.n1, P = LOOPS == FAR_FIXED ? MAXN1 * MAXN1 * MAXN1 : a.P;
        const int n1p = LOOPS ? even_up<MAXN1>() : n1 + (n1 & 1), Pp = n1 * n1 * n1p;
        const float *s_w = s_dyn + (size_t)Pp * OG;   // Pp * OG is a multiple of 4: float4 aligned
        const int f0 = a.far_off[b], f1 = a.far_off[b + 1];
        const int bn = a.batch_node[b];
        const double cb[3] = {a.tcenter[3L * bn], a.tcenter[3L * bn + 1], a.tcenter[3L * bn + 2]};
        float2 kc[OG];
#pragma unroll
        for (int o = 0; o < OG; o++) kc[o] = dup2((g0 + o) < a.norb ? -a.kc32[g0 + o] : 0.f);
        const int i = it.z + tid;
        const bool v = i < it.w;
        const bool warp_busy = it.z + (tid & ~31) < it.w;
        const float tx = v ? (float)(a.tx[i] - cb[0]) : 0.f;
        const float ty = v ? (float)(a.ty[i] - cb[1]) : 0.f;
        const float tz = v ? (float)(a.tz[i] - cb[2]) : 0.f;
        float2 nfi[OG];
        float sum[OG], cmp[OG];
#pragma unroll
        for (int o = 0; o < OG; o++) {
            const int orb = g0 + o;
            nfi[o] = dup2((v && orb < a.norb) ? -a.ft32[(long)orb * a.nt + i] : 0.f);
            sum[o] = 0.f;
            cmp[o] = 0.f;
        }
        for (int e = f0; e < f1; e++) {
            const int slot = a.node_slot[a.far_list[e]];
            const double *gm = a.geom + 6L * slot;
            __syncthreads();
            for (int kk = tid; kk < Pp; kk += GT) {   // a point's charges of all orbitals at once
                const int row = kk / n1p, k3 = kk - row * n1p;
                const float *q0 = a.qhat32 + ((long)g0 * a.nslots + slot) * P + row * n1 + k3;
                float q[OG];
#pragma unroll
                for (int o = 0; o < OG; o++)
                    q[o] = (k3 < n1 && g0 + o < a.norb) ? q0[(long)o * a.nslots * P] : 0.f;
#pragma unroll
                for (int o = 0; o < OG; o++) reinterpret_cast<float *>(s_q4)[q4_pos(kk, o, OG)] = q[o];
            }
            for (int k = tid; k < Pp; k += GT) {
                const int row = k / n1p, k3 = k - row * n1p;
                s_dyn[(size_t)Pp * OG + k] = k3 < n1 ? a.what32[(long)slot * P + row * n1 + k3] : 0.f;
            }
            if (tid < 3 * n1) {
                const int d = tid / n1, m = tid - d * n1;
                const double cbd = d == 0 ? cb[0] : (d == 1 ? cb[1] : cb[2]);
                s_p[d][m] = (float)((gm[d] + gm[3 + d] * a.tn[m]) - cbd);
            }
            __syncthreads();
            if (!warp_busy) continue;
            for_pairs<OG>(item_pairs<OG>(a.norb, g0), [&](auto c) {
                far_group_cluster<SS, MAXN1, OG, LOOPS, decltype(c)::value>(s_q4, s_w, s_p, n1, tx, ty, tz, nfi, kc,
                                                                            sum, cmp);
            });
        }
        if (v) {
#pragma unroll
            for (int o = 0; o < OG; o++)
                if (g0 + o < a.norb) a.out[(long)(g0 + o) * a.nt + i] = (double)sum[o] - (double)cmp[o];
        }
    }
    pass_end();
}

// ---------------------------------------------------------------------------
// far_group at degree 7 with the next cluster's charges in flight: cp.async
// copies global -> shared without registers, so the charges and weight
// charges of far cluster e+1 load while cluster e is computed, and one
// barrier per cluster separates the two buffers.  Charges are copied 8 bytes
// at a time ({q(o, j), q(o, j+1)} is contiguous both in global memory and in
// the staged layout); orbitals past the request's last get zero-filled copies.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void cp_async8(void *smem, const void *gmem, bool valid) {
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    const int n = valid ? 8 : 0;   // source bytes; the rest of the 8 are zero-filled
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(sa), "l"(gmem), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async16(void *smem, const void *gmem) {
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

constexpr int DB_N1 = 8, DB_P = DB_N1 * DB_N1 * DB_N1;   // degree 7
__host__ __device__ constexpr size_t far_group_db_smem(int og) { return sizeof(float) * 2 * (size_t)DB_P * (og + 1); }

template <bool SS, int OG>
__global__ void __launch_bounds__(GT, 4) far_group_db(const __grid_constant__ Work w) {
    constexpr int BUF = DB_P * OG + DB_P;   // floats per buffer: charges, then weight charges
    extern __shared__ __align__(16) float s_dyn[];
    __shared__ float s_p[2][3][DB_N1];
    __shared__ int s_item;
    const int tid = threadIdx.x;
    pass_begin();
    for (;;) {
        const int item = next_item(w.queue, &s_item);
        if (item >= w.nitems) break;
        const int4 it = w.items[item];
        const Fields &a = w.sys[it.y >> 16];
        const int b = it.x, g0 = it.y & 0xffff;
        const int f0 = a.far_off[b], f1 = a.far_off[b + 1];
        const int bn = a.batch_node[b];
        const double cb[3] = {a.tcenter[3L * bn], a.tcenter[3L * bn + 1], a.tcenter[3L * bn + 2]};
        float2 kc[OG];
#pragma unroll
        for (int o = 0; o < OG; o++) kc[o] = dup2((g0 + o) < a.norb ? -a.kc32[g0 + o] : 0.f);
        if (f0 == f1) continue;
        // issue the copies of far cluster e into buffer buf (completes at the next wait + barrier)
        auto stage = [&](int e, int buf) {
            const int slot = a.node_slot[a.far_list[e]];
            float *q = s_dyn + (size_t)buf * BUF;
            for (int k = tid; k < DB_P * OG / 2; k += GT) {
                const int o = k / (DB_P / 2), kk = 2 * (k - o * (DB_P / 2));
                const int orb = g0 + o;
                const bool valid = orb < a.norb;
                const float *src = a.qhat32 + ((long)(valid ? orb : g0) * a.nslots + slot) * DB_P + kk;
                cp_async8(q + q4_pos(kk, o, OG), src, valid);
            }
            for (int k = tid; k < DB_P / 4; k += GT) cp_async16(q + DB_P * OG + 4 * k, a.what32 + (long)slot * DB_P + 4 * k);
            cp_async_commit();
            if (tid < 3 * DB_N1) {
                const double *gm = a.geom + 6L * slot;
                const int d = tid / DB_N1, m = tid - d * DB_N1;
                const double cbd = d == 0 ? cb[0] : (d == 1 ? cb[1] : cb[2]);
                s_p[buf][d][m] = (float)((gm[d] + gm[3 + d] * a.tn[m]) - cbd);
            }
        };
        const int i = it.z + tid;
        const bool v = i < it.w;
        const bool warp_busy = it.z + (tid & ~31) < it.w;
        const float tx = v ? (float)(a.tx[i] - cb[0]) : 0.f;
        const float ty = v ? (float)(a.ty[i] - cb[1]) : 0.f;
        const float tz = v ? (float)(a.tz[i] - cb[2]) : 0.f;
        float2 nfi[OG];
        float sum[OG], cmp[OG];
#pragma unroll
        for (int o = 0; o < OG; o++) {
            const int orb = g0 + o;
            nfi[o] = dup2((v && orb < a.norb) ? -a.ft32[(long)orb * a.nt + i] : 0.f);
            sum[o] = 0.f;
            cmp[o] = 0.f;
        }
        __syncthreads();   // every thread is done with both buffers of the previous target chunk
        stage(f0, 0);
        for (int e = f0; e < f1; e++) {
            const int cur = (e - f0) & 1;
            cp_async_wait_all();   // this thread's copies of cluster e
            __syncthreads();       // everyone's copies visible; everyone done reading the other buffer
            if (e + 1 < f1) stage(e + 1, cur ^ 1);
            if (!warp_busy) continue;
            const float *q = s_dyn + (size_t)cur * BUF;
            for_pairs<OG>(item_pairs<OG>(a.norb, g0), [&](auto c) {
                far_group_cluster<SS, DB_N1, OG, FAR_FIXED, decltype(c)::value>(reinterpret_cast<const float4 *>(q),
                                                                           q + DB_P * OG, s_p[cur], DB_N1, tx, ty, tz,
                                                                           nfi, kc, sum, cmp);
            });
        }
        if (v) {
#pragma unroll
            for (int o = 0; o < OG; o++)
                if (g0 + o < a.norb) a.out[(long)(g0 + o) * a.nt + i] = (double)sum[o] - (double)cmp[o];
        }
    }
    pass_end();
}

// ---------------------------------------------------------------------------
// Orbital-group kernels with 16 orbitals per item, packed by ORBITAL: the two
// lanes of every packed operation are orbitals (2p, 2p+1) of one source (or
// proxy point).  The per-orbital constants -k log2(e) and -f_i are then
// natural float2 pairs -- 8 pairs of registers each for 16 orbitals, where
// the source-packed layout needs 16 duplicated pairs -- and only the
// source's r, -log2 r and weight are duplicated, once per source for all 16
// orbitals.  The geometry (differences, r^2, rsqrt, lg2) of two sources is
// still formed in packed operations and is shared by 16 orbitals: MUFU work
// per pair-orbital is 1 ex2 + (rsqrt + lg2)/16.
// Charges are staged orbital-fastest, QS16 floats per source (16 used + 4 of
// padding, which spreads the staging writes over all banks); a thread reads
// one source's 16 charges as four float4.  Each lane sums KCHUNK16 sources of
// one orbital before the Kahan step, the same run length per lane as the
// source-packed kernels.
// ---------------------------------------------------------------------------
constexpr int QS16 = 20;
constexpr int KCHUNK16 = 32;

// The slots of a tile for 16 orbitals (cnt: sources of each slot, a
// multiple of 4; the slots with sources come first).  A full slot runs on into
// the next one, so the pipeline drains only where a range ends.  Four sources
// per iteration (two packed pairs), software pipelined: the next four
// sources' geometry (loads, rsqrt, lg2) is issued before this iteration's
// 64 orbital-pair updates, which hides its latency.  The per-orbital Kahan
// sums live in shared memory (s_k[o][GT] sums, s_k[16 + o][GT]
// compensations, touched once per KCHUNK16 sources), which leaves the
// registers for the pipelined geometry.  NP: orbital pairs of the item that
// hold orbitals (the last group of a request may be partly filled); the
// pairs past NP are not computed.
template <bool SS, bool MASK, bool PRECISE, int NP = 8>
__device__ __forceinline__ void group16_tile(const float (*__restrict__ s)[GTILE], const float *__restrict__ s_q,
                                             const int *__restrict__ cnt, float2 tx, float2 ty,
                                             float2 tz, float2 lx, float2 ly, float2 lz, const float2 (&nfi)[8],
                                             const float2 (&kc)[8], float *__restrict__ s_k) {
    // r, -log2 r and w of the source pair at j (packed over the two sources)
    auto geometry = [&](int j, float2 &r, float2 &nl, float2 &wv) {
        float2 dx = add2(tx, lds2(s[0] + j)), dy = add2(ty, lds2(s[1] + j)), dz = add2(tz, lds2(s[2] + j));
        if constexpr (PRECISE) {
            dx = add2(dx, add2(lx, lds2(s[4] + j)));
            dy = add2(dy, add2(ly, lds2(s[5] + j)));
            dz = add2(dz, add2(lz, lds2(s[6] + j)));
        }
        wv = lds2(s[3] + j);
        const float2 r2 = fma2(dx, dx, fma2(dy, dy, mul2(dz, dz)));
        float2 rinv = rsqrt2(r2);
        nl = nlog2r2(r2);
        if (MASK) {   // r = 0: r = 0 and 2^{-inf} = 0, so the pair adds exactly 0
            rinv.x = r2.x > 0.f ? rinv.x : 0.f;
            rinv.y = r2.y > 0.f ? rinv.y : 0.f;
            nl.x = r2.x > 0.f ? nl.x : -INFINITY;
            nl.y = r2.y > 0.f ? nl.y : -INFINITY;
        }
        r = mul2(r2, rinv);
    };
    const int tid = threadIdx.x;
    float2 part[8];
#pragma unroll
    for (int p = 0; p < 8; p++) part[p] = make_float2(0.f, 0.f);
    float2 rc[2], nc[2], wc[2];
    for (int sl = 0; sl < GW;) {
        const int j0 = sl * SLOT;
        int n = cnt[sl++], j1 = j0 + n;
        if (n == 0) return;
        while (n == SLOT && sl < GW) {
            n = cnt[sl++];
            j1 += n;
        }
        geometry(j0, rc[0], nc[0], wc[0]);
        geometry(j0 + 2, rc[1], nc[1], wc[1]);
#pragma unroll 1
        for (int j = j0; j < j1; j += 4) {
            const int jn = j + 4 < j1 ? j + 4 : j;
            float2 rn[2], nn[2], wn[2];
            geometry(jn, rn[0], nn[0], wn[0]);
            geometry(jn + 2, rn[1], nn[1], wn[1]);
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const float ru = (u & 1) ? rc[u >> 1].y : rc[u >> 1].x;
                const float nu = (u & 1) ? nc[u >> 1].y : nc[u >> 1].x;
                const float wu = (u & 1) ? wc[u >> 1].y : wc[u >> 1].x;
                const float2 rd = dup2(ru), nd = dup2(nu), wd = dup2(wu);
                const float *qj = s_q + (j + u) * QS16;
#pragma unroll
                for (int o4 = 0; o4 < (NP + 1) / 2; o4++) {
                    const float4 q4 = lds4(qj + 4 * o4);
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const int p = 2 * o4 + h;   // orbitals 2p, 2p+1
                        if (p < NP) {
                            const float2 q = h ? make_float2(q4.z, q4.w) : make_float2(q4.x, q4.y);
                            const float2 g = ex2pos2(fma2(kc[p], rd, nd));
                            part[p] = fma2(g, SS ? fma2(nfi[p], wd, q) : q, part[p]);
                        }
                    }
                }
            }
            if ((j + 4) % KCHUNK16 == 0 || j + 4 >= j1) {   // end of a run of KCHUNK16 sources
#pragma unroll
                for (int p = 0; p < NP; p++) {
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const int o = 2 * p + h;
                        float sm = s_k[o * GT + tid], cm = s_k[(16 + o) * GT + tid];
                        kahan_add(sm, cm, h ? part[p].y : part[p].x);
                        s_k[o * GT + tid] = sm;
                        s_k[(16 + o) * GT + tid] = cm;
                    }
                    part[p] = make_float2(0.f, 0.f);
                }
            }
#pragma unroll
            for (int v = 0; v < 2; v++) {
                rc[v] = rn[v];
                nc[v] = nn[v];
                wc[v] = wn[v];
            }
        }
    }
}

// group16_tile for the item's np filled orbital pairs (1..8).
template <bool SS, bool MASK, bool PRECISE>
__device__ __forceinline__ void group16_tile_np(int np, const float (*__restrict__ s)[GTILE],
                                                const float *__restrict__ s_q, const int *__restrict__ cnt, float2 tx, float2 ty, float2 tz, float2 lx, float2 ly,
                                                float2 lz, const float2 (&nfi)[8], const float2 (&kc)[8],
                                                float *__restrict__ s_k) {
#define TAGI_G16(N) group16_tile<SS, MASK, PRECISE, N>(s, s_q, cnt, tx, ty, tz, lx, ly, lz, nfi, kc, s_k)
    switch (np) {
    case 1: TAGI_G16(1); break;
    case 2: TAGI_G16(2); break;
    case 3: TAGI_G16(3); break;
    case 4: TAGI_G16(4); break;
    case 5: TAGI_G16(5); break;
    case 6: TAGI_G16(6); break;
    case 7: TAGI_G16(7); break;
    default: TAGI_G16(8); break;
    }
#undef TAGI_G16
}

// Filled orbital pairs of a 16-orbital item starting at orbital g0.
__device__ __forceinline__ int group16_pairs(int norb, int g0) { return min(8, (norb - g0 + 1) >> 1); }

// Per-orbital constants of a 16-orbital item, as orbital pairs.
__device__ __forceinline__ void group16_constants(const Fields &a, int g0, float2 (&kc)[8], float *kmin) {
    float km = 3.4e38f;
#pragma unroll
    for (int p = 0; p < 8; p++) {
        const int o0 = g0 + 2 * p, o1 = o0 + 1;
        kc[p] = make_float2(o0 < a.norb ? -a.kc32[o0] : 0.f, o1 < a.norb ? -a.kc32[o1] : 0.f);   // -k log2(e)
        if (o0 < a.norb) km = fminf(km, a.kc32[o0]);
        if (o1 < a.norb) km = fminf(km, a.kc32[o1]);
    }
    if (kmin) *kmin = km;
}

// Dynamic shared memory of near_group16: the source rows, the charges, then
// the per-thread Kahan sums and compensations of 16 orbitals.
__host__ __device__ constexpr size_t near_group16_smem(int pass) {
    return sizeof(float) * ((size_t)GTILE * ((pass == 1 ? 7 : 4) + QS16) + 32 * GT);
}

template <bool SS, int PASS, bool WIDE = false>
__global__ void __launch_bounds__(GT, 4) near_group16(const __grid_constant__ Work w) {
    constexpr int NR = PASS == 1 ? 7 : 4;
    extern __shared__ __align__(16) float s_dyn[];
    float(*s_src)[GTILE] = reinterpret_cast<float(*)[GTILE]>(s_dyn);
    float *s_q = s_dyn + NR * GTILE;
    float *s_k = s_q + GTILE * QS16;
    __shared__ RangeTable<GT> s_rng;
    __shared__ int s_cnt[GW];
    __shared__ int s_item;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    pass_begin();
    for (;;) {
        const int item = next_item(w.queue, &s_item);
        if (item >= w.nitems) break;
        const int4 it = w.items[item];
        const Fields &a = w.sys[it.y >> 16];
        const int b = it.x, g0 = it.y & 0xffff;
        const int bn = a.batch_node[b];
        const double cbx = a.tcenter[3L * bn], cby = a.tcenter[3L * bn + 1], cbz = a.tcenter[3L * bn + 2];
        const Split ccx(cbx), ccy(cby), ccz(cbz);
        float2 kc[8];
        float kmin;
        group16_constants(a, g0, kc, &kmin);
        const int r0 = a.rng_off[b], r1 = a.rng_off[b + 1];
        const int i = it.z + tid;
        const bool v = i < it.w;
        const bool warp_busy = it.z + (tid & ~31) < it.w;
        float2 tx, ty, tz, lx = dup2(0.f), ly = dup2(0.f), lz = dup2(0.f);
        if (PASS == 1) {  // absolute hi/lo splits (see near_chunk)
            const float4 h = v ? a.thi[i] : make_float4(0.f, 0.f, 0.f, 0.f);
            const float4 l = v ? a.tlo[i] : make_float4(0.f, 0.f, 0.f, 0.f);
            tx = dup2(h.x);
            ty = dup2(h.y);
            tz = dup2(h.z);
            lx = dup2(l.x);
            ly = dup2(l.y);
            lz = dup2(l.z);
        } else {
            tx = dup2(v ? (float)(a.tx[i] - cbx) : 0.f);
            ty = dup2(v ? (float)(a.ty[i] - cby) : 0.f);
            tz = dup2(v ? (float)(a.tz[i] - cbz) : 0.f);
        }
        float2 nfi[8];
#pragma unroll
        for (int p = 0; p < 8; p++) {
            const int o0 = g0 + 2 * p, o1 = o0 + 1;
            nfi[p] = make_float2((v && o0 < a.norb) ? -a.ft32[(long)o0 * a.nt + i] : 0.f,
                                 (v && o1 < a.norb) ? -a.ft32[(long)o1 * a.nt + i] : 0.f);
        }
#pragma unroll
        for (int o = 0; o < 32; o++) s_k[o * GT + tid] = 0.f;   // this thread's own sums
        for (int e0 = r0; e0 < r1; e0 += GT) {
            const int2 n = load_ranges(a, e0, r1, s_rng, [&](int2 &r, float dmin) {
                if (range_is_close(r) != (PASS == 1)) return false;
                r.x = range_begin(r);
                return !(dmin * kmin > 127.f);   // beyond: every orbital's term is exactly 0
            });
            for (int c0 = 0; c0 < n.y; c0 += GW) {
                __syncthreads();   // the previous tile is no longer read
                const int c = c0 + wid;
                int cnt4 = 0;
                if (c < n.y) {
                    const int e = range_of_chunk(s_rng, n.x, c);
                    const int t0 = s_rng.begin[e] + (c - s_rng.first[e]) * SLOT;
                    const int cnt = min(SLOT, s_rng.end[e] - t0);
                    cnt4 = (cnt + 3) & ~3;
                    const int j = 2 * lane, d = wid * SLOT + j;
                    if (j < cnt4) {
                        const bool real0 = j < cnt, real1 = j + 1 < cnt;
                        const int j0 = t0 + (real0 ? j : 0), j1 = t0 + (real1 ? j + 1 : 0);   // padding: the first source
                        if constexpr (WIDE) {
                            sts2(&s_src[0][d], neg_relative64(a.sx, j0, j1, cbx, 1.0));
                            sts2(&s_src[1][d], neg_relative64(a.sy, j0, j1, cby, 1.0));
                            sts2(&s_src[2][d], neg_relative64(a.sz, j0, j1, cbz, 1.0));
                        } else {
                            const float4 h0 = a.shi[j0], h1 = a.shi[j1], l0 = a.slo[j0], l1 = a.slo[j1];
                            const float2 hx = make_float2(h0.x, h1.x), hy = make_float2(h0.y, h1.y),
                                         hz = make_float2(h0.z, h1.z), qx = make_float2(l0.x, l1.x),
                                         qy = make_float2(l0.y, l1.y), qz = make_float2(l0.z, l1.z);
                            if constexpr (PASS == 1) {
                                sts2(&s_src[0][d], neg2(hx));
                                sts2(&s_src[1][d], neg2(hy));
                                sts2(&s_src[2][d], neg2(hz));
                                sts2(&s_src[4][d], neg2(qx));
                                sts2(&s_src[5][d], neg2(qy));
                                sts2(&s_src[6][d], neg2(qz));
                            } else {
                                sts2(&s_src[0][d], neg_relative(hx, qx, ccx));
                                sts2(&s_src[1][d], neg_relative(hy, qy, ccy));
                                sts2(&s_src[2][d], neg_relative(hz, qz, ccz));
                            }
                        }
                        sts2(&s_src[3][d], make_float2(real0 ? a.w32[j0] : 0.f, real1 ? a.w32[j1] : 0.f));
                    }
                    // a warp stages 8 sources x 4 orbitals at a time: 32-byte global
                    // segments, conflict-free shared writes with the QS16 stride
                    // (all 32 loads of a lane are issued before the first is stored)
                    const int o4 = lane >> 3, j8 = lane & 7;
                    float q[8][4];
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        const int orb = g0 + o4 + 4 * i;
                        const float *qo = a.q32 + (long)orb * a.ns + t0;
#pragma unroll
                        for (int u = 0; u < 8; u++) q[u][i] = (j8 + 8 * u < cnt && orb < a.norb) ? qo[j8 + 8 * u] : 0.f;
                    }
#pragma unroll
                    for (int u = 0; u < 8; u++)
                        if (j8 + 8 * u < cnt4) {
#pragma unroll
                            for (int i = 0; i < 4; i++) s_q[(wid * SLOT + j8 + 8 * u) * QS16 + o4 + 4 * i] = q[u][i];
                        }
                }
                if (lane == 0) s_cnt[wid] = cnt4;
                __syncthreads();
                if (!warp_busy) continue;
                group16_tile_np<SS, PASS == 1, PASS == 1>(group16_pairs(a.norb, g0), s_src, s_q, s_cnt, tx, ty, tz, lx, ly,
                                                          lz, nfi, kc, s_k);
            }
        }
        if (v) {
#pragma unroll
            for (int o = 0; o < 16; o++)
                if (g0 + o < a.norb)
                    a.out[(long)(g0 + o) * a.nt + i] = (double)s_k[o * GT + tid] - (double)s_k[(16 + o) * GT + tid];
        }
    }
    pass_end();
}

// One staged proxy grid against one target for 16 orbitals (see far_cluster
// for the padded innermost axis; charges staged QS16 floats per proxy point).
// NP: filled orbital pairs, as in group16_tile.
template <bool SS, int MAXN1, int LOOPS, int NP = 8>
__device__ __forceinline__ void far_group16_cluster(const float *__restrict__ s_q, const float *__restrict__ s_w,
                                                    const float (*s_p)[MAXN1], int n1_in,
                                                    float tx, float ty, float tz, const float2 (&nfi)[8],
                                                    const float2 (&kc)[8], float (&sum)[16], float (&cmp)[16]) {
    constexpr int MH = even_up<MAXN1>() / 2;
    const int n1 = LOOPS == FAR_FIXED ? MAXN1 : n1_in;
    const int n1p = LOOPS ? even_up<MAXN1>() : n1 + (n1 & 1);
    float2 dz2[MH];
#pragma unroll
    for (int m = 0; m < MH; m++) {
        const float d0 = tz - s_p[2][2 * m < n1 ? 2 * m : 0];
        const float d1 = tz - s_p[2][2 * m + 1 < n1 ? 2 * m + 1 : 0];
        dz2[m] = make_float2(d0 * d0, d1 * d1);
    }
    int idx = 0;
    for (int k1 = 0; k1 < n1; k1++) {
        float2 part[8];
#pragma unroll
        for (int p = 0; p < 8; p++) part[p] = make_float2(0.f, 0.f);
        const float dx = tx - s_p[0][k1];
        const float dx2 = dx * dx;
        for (int k2 = 0; k2 < n1; k2++) {
            const float dy = ty - s_p[1][k2];
            const float2 rxy = dup2(fmaf(dy, dy, dx2));
#pragma unroll
            for (int m = 0; m < MH; m++) {
                if (LOOPS || 2 * m < n1) {
                    const float2 r2 = add2(rxy, dz2[m]);
                    const float2 rr = mul2(r2, rsqrt2(r2));
                    const float2 nl = nlog2r2(r2);
                    const float2 wk = lds2(s_w + idx + 2 * m);
#pragma unroll
                    for (int u = 0; u < 2; u++) {
                        const float2 rd = dup2(u ? rr.y : rr.x), nd = dup2(u ? nl.y : nl.x);
                        const float2 wd = dup2(u ? wk.y : wk.x);
                        const float *qk = s_q + (idx + 2 * m + u) * QS16;
#pragma unroll
                        for (int o4 = 0; o4 < (NP + 1) / 2; o4++) {
                            const float4 q4 = lds4(qk + 4 * o4);
#pragma unroll
                            for (int h = 0; h < 2; h++) {
                                const int p = 2 * o4 + h;
                                if (p < NP) {
                                    const float2 q = h ? make_float2(q4.z, q4.w) : make_float2(q4.x, q4.y);
                                    const float2 g = ex2pos2(fma2(kc[p], rd, nd));
                                    part[p] = fma2(g, SS ? fma2(nfi[p], wd, q) : q, part[p]);
                                }
                            }
                        }
                    }
                }
            }
            idx += n1p;
        }
#pragma unroll
        for (int p = 0; p < NP; p++) {
            kahan_add(sum[2 * p], cmp[2 * p], part[p].x);
            kahan_add(sum[2 * p + 1], cmp[2 * p + 1], part[p].y);
        }
    }
}

template <bool SS, int MAXN1, int LOOPS>
__device__ __forceinline__ void far_group16_cluster_np(int np, const float *__restrict__ s_q,
                                                       const float *__restrict__ s_w, const float (*s_p)[MAXN1],
                                                       int n1, float tx, float ty,
                                                       float tz, const float2 (&nfi)[8], const float2 (&kc)[8],
                                                       float (&sum)[16], float (&cmp)[16]) {
#define TAGI_F16(N) \
    far_group16_cluster<SS, MAXN1, LOOPS, N>(s_q, s_w, s_p, n1, tx, ty, tz, nfi, kc, sum, cmp)
    switch (np) {
    case 1: TAGI_F16(1); break;
    case 2: TAGI_F16(2); break;
    case 3: TAGI_F16(3); break;
    case 4: TAGI_F16(4); break;
    case 5: TAGI_F16(5); break;
    case 6: TAGI_F16(6); break;
    case 7: TAGI_F16(7); break;
    default: TAGI_F16(8); break;
    }
#undef TAGI_F16
}

// Dynamic shared memory of far_group16: charges (Pp * QS16 floats) then the
// weight charges (Pp floats), Pp = n1 * n1 * n1p.
__host__ __device__ constexpr size_t far_group16_smem(int n1) {
    return sizeof(float) * (size_t)n1 * n1 * (n1 + (n1 & 1)) * (QS16 + 1);
}

template <bool SS, int MAXN1, int LOOPS>
__global__ void __launch_bounds__(GT, 4) far_group16(const __grid_constant__ Work w) {
    extern __shared__ __align__(16) float s_dyn[];
    __shared__ float s_p[3][MAXN1];
    __shared__ int s_item;
    const int tid = threadIdx.x;
    pass_begin();
    for (;;) {
        const int item = next_item(w.queue, &s_item);
        if (item >= w.nitems) break;
        const int4 it = w.items[item];
        const Fields &a = w.sys[it.y >> 16];
        const int b = it.x, g0 = it.y & 0xffff;
        const int n1 = LOOPS == FAR_FIXED ? MAXN1 : a.n1, P = LOOPS == FAR_FIXED ? MAXN1 * MAXN1 * MAXN1 : a.P;
        const int n1p = LOOPS ? even_up<MAXN1>() : n1 + (n1 & 1), Pp = n1 * n1 * n1p;
        float *s_q = s_dyn;
        float *s_w = s_dyn + (size_t)Pp * QS16;
        const int f0 = a.far_off[b], f1 = a.far_off[b + 1];
        const int bn = a.batch_node[b];
        const double cb[3] = {a.tcenter[3L * bn], a.tcenter[3L * bn + 1], a.tcenter[3L * bn + 2]};
        float2 kc[8];
        group16_constants(a, g0, kc, nullptr);
        const int i = it.z + tid;
        const bool v = i < it.w;
        const bool warp_busy = it.z + (tid & ~31) < it.w;
        const float tx = v ? (float)(a.tx[i] - cb[0]) : 0.f;
        const float ty = v ? (float)(a.ty[i] - cb[1]) : 0.f;
        const float tz = v ? (float)(a.tz[i] - cb[2]) : 0.f;
        float2 nfi[8];
        float sum[16], cmp[16];
#pragma unroll
        for (int p = 0; p < 8; p++) {
            const int o0 = g0 + 2 * p, o1 = o0 + 1;
            nfi[p] = make_float2((v && o0 < a.norb) ? -a.ft32[(long)o0 * a.nt + i] : 0.f,
                                 (v && o1 < a.norb) ? -a.ft32[(long)o1 * a.nt + i] : 0.f);
        }
#pragma unroll
        for (int o = 0; o < 16; o++) {
            sum[o] = 0.f;
            cmp[o] = 0.f;
        }
        const int so = tid >> 3;   // the orbital whose charges this thread stages
        const bool has = g0 + so < a.norb;
        for (int e = f0; e < f1; e++) {
            const int slot = a.node_slot[a.far_list[e]];
            const double *gm = a.geom + 6L * slot;
            __syncthreads();
            // a warp stages 8 proxy points x 4 orbitals at a time (see near_group16), 16
            // loads of a thread in flight
            const float *qo = a.qhat32 + ((long)(has ? g0 + so : g0) * a.nslots + slot) * P;
            for (int k0 = tid & 7; k0 < Pp; k0 += 8 * 16) {
                float q[16];
#pragma unroll
                for (int u = 0; u < 16; u++) {
                    const int kk = k0 + 8 * u, row = kk / n1p, k3 = kk - row * n1p;
                    q[u] = (has && kk < Pp && k3 < n1) ? qo[row * n1 + k3] : 0.f;
                }
#pragma unroll
                for (int u = 0; u < 16; u++)
                    if (k0 + 8 * u < Pp) s_q[(k0 + 8 * u) * QS16 + so] = q[u];
            }
#pragma unroll 4
            for (int k = tid; k < Pp; k += GT) {
                const int row = k / n1p, k3 = k - row * n1p;
                s_w[k] = k3 < n1 ? a.what32[(long)slot * P + row * n1 + k3] : 0.f;
            }
            if (tid < 3 * n1) {
                const int d = tid / n1, m = tid - d * n1;
                const double cbd = d == 0 ? cb[0] : (d == 1 ? cb[1] : cb[2]);
                s_p[d][m] = (float)((gm[d] + gm[3 + d] * a.tn[m]) - cbd);
            }
            __syncthreads();
            if (!warp_busy) continue;
            far_group16_cluster_np<SS, MAXN1, LOOPS>(group16_pairs(a.norb, g0), s_q, s_w, s_p, n1,
                                                     tx, ty, tz,                                                      nfi, kc, sum, cmp);
        }
        if (v) {
#pragma unroll
            for (int o = 0; o < 16; o++)
                if (g0 + o < a.norb) a.out[(long)(g0 + o) * a.nt + i] = (double)sum[o] - (double)cmp[o];
        }
    }
    pass_end();
}

// ---------------------------------------------------------------------------
// FP64 near and far fields (the plain path).
//
// Bound: the FP64 pipe.  It issues 1/64 of the FP32 rate (measured 527 G DFMA/s
// against 3.9e13 FFMA/s), so one FP64 instruction costs as much as some seventy
// FP32 or integer ones.  sqrt, exp and the division of a Yukawa pair are about
// 35 FP64 instructions; here a pair is 22 in all (Coulomb with subtraction 18):
//   * 1/r from the FP32 rsqrt estimate y of r2 by one cubic Newton step:
//     z = r2 y, e = 1 - z y, 1/r = y (1 + d), r = z (1 + d), d = e/2 + 3 e^2/8;
//     e^2 < 2^-43 leaves its term to FP32;
//   * 2^{-t/EXP_N} with t = K r, K = k EXP_N / ln 2 in two doubles: n = rint(t)
//     from FP32, the remainder f = n - t by fused multiply-adds on z and z d (r
//     itself is not rounded), and a table of 2^{i/EXP_N}, i < EXP_N, times a cubic
//     in f (table lookup and short polynomial: P. T. P. Tang, ACM TOMS 15, 1989), whose upper
//     terms go to FP32.  t's FP32 error grows with it: |f| < 0.56 up to kr = 16, 0.7 at 50, 1.9
//     at 300, 3.7 at 707, where the upper terms are 2^-24 and FP32 leaves 26 units of 2^-53;
//   * conversions between FP32 and FP64 are shifts of the bit patterns.
// Against 128-bit arithmetic (estimates of 1/r up to 2 FP32 ulp off) e^{-kr}/r has an rms error of
// 0.83, 1.8, 6.9, 47, 128 units of 2^-53 for kr up to 1, 16, 50, 300, 707; sqrt, exp and a division
// have 0.62, 3.1, 14, 98, 280, and one more rounding in the sum.  A squared distance
// outside FP32's range (zero: a coincident pair; NaN) and an exponential that is a
// subnormal number (EXP_LIMIT) take the library functions.
// Near field, 50k points, split 8: 167 -> 79 ms; the whole one-shot call 177 -> 84 ms.
// ---------------------------------------------------------------------------
constexpr int EXP_BITS = 13, EXP_N = 1 << EXP_BITS;

// 2^{2^b / EXP_N} as hi + lo
__constant__ double2 c_exp_step[EXP_BITS] = {
    {0x1.00058ba01fba0p+0, -0x1.a4a4d4cad39fep-54}, {0x1.000b175effdc7p+0, 0x1.ae8e38c59c72ap-54},
    {0x1.00162f3904052p+0, -0x1.7b5d0d58ea8f4p-58}, {0x1.002c605e2e8cfp+0, -0x1.d7c96f201bb2fp-55},
    {0x1.0058c86da1c0ap+0, -0x1.5e00e62d6b30dp-56}, {0x1.00b1afa5abcbfp+0, -0x1.4f6b2a7609f71p-55},
    {0x1.0163da9fb3335p+0, 0x1.b61299ab8cdb7p-54},  {0x1.02c9a3e778061p+0, -0x1.19083535b085dp-56},
    {0x1.059b0d3158574p+0, 0x1.d73e2a475b465p-55},  {0x1.0b5586cf9890fp+0, 0x1.8a62e4adc610bp-54},
    {0x1.172b83c7d517bp+0, -0x1.19041b9d78a76p-55}, {0x1.306fe0a31b715p+0, 0x1.6f46ad23182e4p-55},
    {0x1.6a09e667f3bcdp+0, -0x1.bdd3413b26456p-54}};

// table[i] = 2^{i / EXP_N}, the product of the steps of i's bits in double-double
__global__ void exp_table(double *__restrict__ table) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    double h = 1.0, l = 0.0;
#pragma unroll 1
    for (int b = 0; b < EXP_BITS; b++) {
        if (!((i >> b) & 1)) continue;
        const double2 c = c_exp_step[b];
        const double p = __dmul_rn(h, c.x);
        const double e = __fma_rn(l, c.x, __fma_rn(h, c.y, __fma_rn(h, c.x, -p)));
        h = __dadd_rn(p, e);
        l = __dadd_rn(e, -__dadd_rn(h, -p));
    }
    table[i] = h;
}

// A positive float as a double, by its bits (zero becomes 2^-127).
__device__ __forceinline__ double bits_f2d(float x) {
    const unsigned b = __float_as_uint(x);
    return __hiloint2double((int)((b >> 3) + 0x38000000u), (int)(b << 29));
}
// A double in FP32's normal range as a float, truncated (zero becomes +-2).
__device__ __forceinline__ float bits_d2f(double x) {
    const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
    const unsigned m = __funnelshift_l(lo, hi & 0x7fffffffu, 3) + 0x40000000u;
    return __uint_as_float((m & 0x7fffffffu) | (hi & 0x80000000u));
}

// Parameters of 2^{-t / EXP_N}, t = K x: K = kh + kl.
struct ExpScale {
    double kh, kl;
    float kf;
};
// x^e with e = -a x (Yukawa: a = k) or -a^2 x (Coulomb subtraction)
__device__ __forceinline__ ExpScale exp_scale(double a, bool square) {
    constexpr double CH = 0x1.71547652b82fep+13, CL = 0x1.777d0ffda0d24p-43;   // EXP_N / ln 2
    ExpScale s;
    const double b = square ? __dmul_rn(a, a) : a, be = square ? __fma_rn(a, a, -b) : 0.0;
    s.kh = __dmul_rn(b, CH);
    s.kl = __dadd_rn(__fma_rn(b, CH, -s.kh), __fma_rn(b, CL, be * CH));
    s.kf = (float)s.kh;
    return s;
}

struct InvRoot {
    double z, y, d;   // r = z (1 + d), 1/r = y (1 + d)
    float zf;         // r in FP32
};
__device__ __forceinline__ bool in_fp32_range(double r2) {
    return (unsigned)__double2hiint(r2) - 0x38100000u < 0x0fd00000u;   // [2^-126, 2^127)
}
__device__ __forceinline__ InvRoot inv_root(double r2) {
    InvRoot q;
    const float rf = bits_d2f(r2), yf = rsqrt_mufu(rf);
    q.zf = rf * yf;
    q.y = bits_f2d(yf);
    q.z = __dmul_rn(r2, q.y);
    const double e = __fma_rn(-q.z, q.y, 1.0);
    const float ef = ((unsigned)__double2hiint(e) << 1) ? bits_d2f(e) : 0.f;
    q.d = __fma_rn(0.5, e, bits_f2d(0.375f * ef * ef));
    return q;
}

// t from which the exponential is not a normal number (pair_f64_any then), and from which it is 0
// to the last bit.
constexpr float EXP_LIMIT = 1021.f * EXP_N, EXP_NONE = 1080.f * EXP_N;
// 2^{(n - t)/EXP_N} 2^{-n/EXP_N}: tf = t in FP32; the caller forms f = n - t from nd = n.
__device__ __forceinline__ double exp_n(float tf, int &n) {
    n = __float2int_rn(tf);
    return bits_f2d((float)n);
}
__device__ __forceinline__ double exp_finish(double f, int n, const double *__restrict__ tab) {
    constexpr double C1 = 0x1.62e42fefa39efp-14;                       // ln 2 / EXP_N
    constexpr float C2 = 0x1.ebfbdff82c58fp-29, C3 = 0x1.c6b08d704a0c0p-44;   // C1^2 / 2, C1^3 / 6
    const double q = __fma_rn(f, bits_f2d(__fmaf_rn(bits_d2f(f), C3, C2)), C1);
    const double t = tab[-n & (EXP_N - 1)];
    const double ts = __hiloint2double(__double2hiint(t) + (((-n) >> EXP_BITS) << 20), __double2loint(t));
    return __fma_rn(ts, __dmul_rn(f, q), ts);
}
// e^{-k r}
__device__ __forceinline__ double exp_root(const InvRoot &q, const ExpScale &s, const double *__restrict__ tab) {
    const float tf = q.zf * s.kf;
    int n;
    double f = __fma_rn(-s.kh, q.z, exp_n(tf, n));
    f = __fma_rn(-s.kh, __dmul_rn(q.z, q.d), f);
    f = __fma_rn(-s.kl, q.z, f);
    return exp_finish(f, n, tab);
}
// e^{-a^2 x}
__device__ __forceinline__ double exp_square(double x, const ExpScale &s, const double *__restrict__ tab) {
    const float tf = bits_d2f(x) * s.kf;
    int n;
    double f = __fma_rn(-s.kh, x, exp_n(tf, n));
    f = __fma_rn(-s.kl, x, f);
    return exp_finish(f, n, tab);
}

// One pair with the library's functions: r2 outside FP32's range, or t = tf from EXP_LIMIT on.  q and w
// are the charge f w and the weight; the near field passes f and w (near: true).
template <int KERN, bool SS, bool NEAR>
__device__ __noinline__ double pair_f64_any(double r2, float tf, double q, double w, double fi, double kp) {
    if (NEAR && !(r2 > 0.0)) return 0.0;
    const bool none = tf >= EXP_NONE && in_fp32_range(r2);   // no exponential to form
    const double r = sqrt(r2);
    if (KERN == KERNEL_YUKAWA) {
        const double g = none ? 0.0 : exp(-kp * r) / r;
        return SS ? (NEAR ? w * (q - fi) : q - fi * w) * g : q * g;
    }
    if (SS) {
        const double e = none ? 0.0 : exp(-kp * kp * r2);
        return (NEAR ? w * (q - fi * e) : q - fi * w * e) / r;
    }
    return q / r;
}
template <int KERN, bool SS, bool NEAR>
__device__ __forceinline__ double pair_f64(double r2, double q, double w, double fi, double kp, const ExpScale &es,
                                           const double *__restrict__ tab, double acc) {
    const InvRoot v = inv_root(r2);
    const float tf = KERN == KERNEL_YUKAWA ? v.zf * es.kf : (SS ? bits_d2f(r2) * es.kf : 0.f);
    if (!in_fp32_range(r2) || tf >= EXP_LIMIT) return acc + pair_f64_any<KERN, SS, NEAR>(r2, tf, q, w, fi, kp);
    const double rinv = __fma_rn(v.y, v.d, v.y);
    if (KERN == KERNEL_YUKAWA) {
        const double c = SS ? (NEAR ? w * (q - fi) : __fma_rn(-fi, w, q)) : q;
        return __fma_rn(c, __dmul_rn(exp_root(v, es, tab), rinv), acc);
    }
    if (SS) {
        const double e = exp_square(r2, es, tab);
        const double c = NEAR ? w * __fma_rn(-fi, e, q) : __fma_rn(-fi * w, e, q);
        return __fma_rn(c, rinv, acc);
    }
    return __fma_rn(q, rinv, acc);
}

// Dynamic shared memory of the FP64 kernels: the exponential table, where used.
template <int KERN, bool SS>
constexpr size_t f64_smem() { return KERN == KERNEL_YUKAWA || SS ? sizeof(double) * EXP_N : 0; }
template <int KERN, bool SS>
__device__ __forceinline__ void load_exp_table(double *s_tab, const double *__restrict__ table) {
    if constexpr (KERN == KERNEL_YUKAWA || SS)
        for (int i = threadIdx.x; i < EXP_N; i += FT) s_tab[i] = table[i];   // read after the item barriers
}

template <int KERN, bool SS>
__global__ void __launch_bounds__(FT) near_f64(const __grid_constant__ Work w) {
    constexpr int T64 = 256;
    extern __shared__ double s_tab[];
    __shared__ double s_x[T64], s_y[T64], s_z[T64], s_f[T64], s_w[T64];
    __shared__ int s_item;
    const int tid = threadIdx.x;
    pass_begin();
    load_exp_table<KERN, SS>(s_tab, w.exp_table);
    for (;;) {
        const int item = next_item(w.queue, &s_item);
        if (item >= w.nitems) break;
        const int4 it = w.items[item];
        const Fields &a = w.sys[it.y >> 16];
        const Place pl(a.split, FT / 32);
        const int b = it.x, orb = it.y & 0xffff;
        const double kp = a.kp64[orb];
        const ExpScale es = exp_scale(kp, KERN == KERNEL_COULOMB);
        const double *f = a.f64 + (long)orb * a.ns;
        const double *ft = a.ft64 + (long)orb * a.nt;
        const int r0 = a.rng_off[b], r1 = a.rng_off[b + 1];
        const int first = it.z + 32 * (w.turn * pl.G + pl.g), i = first + pl.lane;
        const bool v = i < it.w;
        const bool warp_busy = first < it.w;
        const double xi = v ? a.tx[i] : 0.0, yi = v ? a.ty[i] : 0.0, zi = v ? a.tz[i] : 0.0;
        const double fi = v ? ft[i] : 0.0;
        double acc = 0.0;
        for (int e = r0; e < r1; e++) {
            const int2 r = a.rng[e];
            for (int t0 = range_begin(r); t0 < r.y; t0 += T64) {
                const int cnt = min(T64, r.y - t0);
                __syncthreads();
                if (tid < cnt) {
                    int jj = t0 + tid;
                    s_x[tid] = a.sx[jj];
                    s_y[tid] = a.sy[jj];
                    s_z[tid] = a.sz[jj];
                    s_f[tid] = SS ? f[jj] : a.w64[jj] * f[jj];
                    s_w[tid] = a.w64[jj];
                }
                __syncthreads();
                if (!warp_busy) continue;
                for (int j = pl.sp; j < cnt; j += pl.S) {
                    const double dx = xi - s_x[j], dy = yi - s_y[j], dz = zi - s_z[j];
                    acc = pair_f64<KERN, SS, true>(dx * dx + dy * dy + dz * dz, s_f[j], s_w[j], fi, kp, es, s_tab,
                                                   acc);
                }
            }
        }
        acc = add_splits(acc, pl, s_x);
        if (v && pl.sp == 0) a.out[(long)orb * a.nt + i] = acc;
    }
    pass_end();
}

template <int KERN, bool SS, int MAXN1>
__global__ void __launch_bounds__(FT) far_f64(const __grid_constant__ Work w) {
    constexpr int MAXP = MAXN1 * MAXN1 * MAXN1;
    extern __shared__ double s_tab[];
    __shared__ double s_q[MAXP], s_wh[MAXP];
    __shared__ double s_p[3][MAXN1], s_red[FT];
    __shared__ int s_item;
    const int tid = threadIdx.x;
    pass_begin();
    load_exp_table<KERN, SS>(s_tab, w.exp_table);
    for (;;) {
        const int item = next_item(w.queue, &s_item);
        if (item >= w.nitems) break;
        const int4 it = w.items[item];
        const Fields &a = w.sys[it.y >> 16];
        const Place pl(a.split, FT / 32);
        const int b = it.x, orb = it.y & 0xffff;
        const int n1 = a.n1, P = a.P;
        const int f0 = a.far_off[b], f1 = a.far_off[b + 1];
        const double kp = a.kp64[orb];
        const ExpScale es = exp_scale(kp, KERN == KERNEL_COULOMB);
        const double *ft = a.ft64 + (long)orb * a.nt;
        const double *qh = a.qhat64 + (long)orb * a.nslots * P;
        const int first = it.z + 32 * (w.turn * pl.G + pl.g), i = first + pl.lane;
        const bool v = i < it.w;
        const bool warp_busy = first < it.w;
        const double xi = v ? a.tx[i] : 0.0, yi = v ? a.ty[i] : 0.0, zi = v ? a.tz[i] : 0.0;
        const double fi = v ? ft[i] : 0.0;
        double acc = 0.0;
        for (int e = f0; e < f1; e++) {
            const int slot = a.node_slot[a.far_list[e]];
            __syncthreads();
            for (int k = tid; k < P; k += FT) {
                s_q[k] = qh[(long)slot * P + k];
                s_wh[k] = a.what64[(long)slot * P + k];
            }
            if (tid < 3 * n1) {
                int d = tid / n1, m = tid - d * n1;
                const double *g = a.geom + 6L * slot;
                s_p[d][m] = g[d] + g[3 + d] * a.tn[m];
            }
            __syncthreads();
            if (!warp_busy) continue;
            // rows (k1, k2) of the grid are dealt to the splits in turn over the clusters
            const int rows = n1 * n1;
            double dz2[MAXN1];
#pragma unroll
            for (int m = 0; m < MAXN1; m++) {
                const double dz = zi - s_p[2][m < n1 ? m : 0];
                dz2[m] = dz * dz;
            }
            for (int row = first_slab(e - f0, rows, pl); row < rows; row += pl.S) {
                const int k1 = row / n1, k2 = row - k1 * n1;
                const double dx = xi - s_p[0][k1], dy = yi - s_p[1][k2];
                const double rxy = dx * dx + dy * dy;
                const double *qr = s_q + row * n1, *wr = s_wh + row * n1;
#pragma unroll
                for (int m = 0; m < MAXN1; m++)
                    if (m < n1)
                        acc = pair_f64<KERN, SS, false>(rxy + dz2[m], qr[m], wr[m], fi, kp, es, s_tab, acc);
            }
        }
        acc = add_splits(acc, pl, s_red);
        if (v && pl.sp == 0) a.out[(long)orb * a.nt + i] = acc;
    }
    pass_end();
}

// ---------------------------------------------------------------------------
// Per-call glue: sorted charges, epilogue.
// ---------------------------------------------------------------------------
template <bool MIXED>
__global__ void prep_sources(const double *sv, const int *perm,
                             const double *w, int ns, float *q32,
                             double *q64, double *f64) {
    chain_begin();
    long j = (long)blockIdx.x * blockDim.x + threadIdx.x;
    int orb = blockIdx.y;
    if (j >= ns) return;
    long o = (long)orb * ns + j;
    double f = sv[(long)orb * ns + perm[j]];
    double q = f * w[j];
    if (MIXED) {
        q32[o] = (float)q;
    } else {
        q64[o] = q;
        f64[o] = f;
    }
}

template <bool MIXED>
__global__ void prep_targets(const double *tv, const int *perm, int nt,
                             float *f32, double *f64, double *close_out,
                             double *far_out) {
    chain_begin();
    long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    int orb = blockIdx.y;
    if (i >= nt) return;
    double f = tv[(long)orb * nt + perm[i]];
    if (MIXED) f32[(long)orb * nt + i] = (float)f;
    else f64[(long)orb * nt + i] = f;
    // the far and close-range passes write only the batches they visit
    close_out[(long)orb * nt + i] = 0.0;
    far_out[(long)orb * nt + i] = 0.0;
}

// phi_i = near + far + f_i * SS factor, scattered back to caller order.  The
// SS term uses the same f_i the pair sums used (FP32-rounded in mixed mode):
// sum_j w_j (f_j - c) G + c * int G is exact for any constant c, while mixing
// two roundings of f_i would leave delta * f_i * sum_j w_j G in the result.
template <typename TF>
__global__ void epilogue(const double *__restrict__ nearv, const double *__restrict__ near2v,
                         const double *__restrict__ farv, const TF *__restrict__ fsorted,
                         const int *__restrict__ perm, int nt, const double *__restrict__ ss,
                         double *__restrict__ out) {
    long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    int orb = blockIdx.y;
    if (i >= nt) return;
    long si = (long)orb * nt + i;
    out[(long)orb * nt + perm[i]] = (nearv[si] + near2v[si]) + farv[si] + ss[orb] * (double)fsorted[si];
}

template <typename K>
int occupancy_grid(K kern, int *grid, size_t smem = 0, int threads = FT) {
    int dev = 0, sms = 0, per = 0;
    TAGI_CUDA(cudaGetDevice(&dev));
    TAGI_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    TAGI_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, threads, smem));
    *grid = sms * (per > 0 ? per : 1);
    return TAGI_OK;
}

// Persistent launch: grid = resident CTAs (at most one per work item).  smem
// bytes of dynamic shared memory; for large requests the kernel's limit is
// raised first.  follows: whether the launch before it in the stream was another
// field pass of this call (set to true by a launch).
template <typename K>
int launch_persistent(K kern, const Work &w, cudaStream_t s, size_t smem = 0, int threads = FT,
                      bool *follows = nullptr) {
    if (w.nitems == 0) return TAGI_OK;
    if (smem > 32 * 1024)   // dynamic + static above the 48 KB default needs the opt-in
        TAGI_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int grid = 0;
    TAGI_TRY(occupancy_grid(kern, &grid, smem, threads));
    if (grid > w.nitems) grid = w.nitems;
    if (grid < 1) grid = 1;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &at;
    cfg.numAttrs = follows && *follows ? 1 : 0;
    count_launch();
    TAGI_CUDA(cudaLaunchKernelEx(&cfg, kern, w));
    if (follows) *follows = true;
    return TAGI_OK;
}

// ---------------------------------------------------------------------------
// Loop ceilings: the near/far inner loops' arithmetic with operands already
// in shared memory and registers and no global traffic, measured live on the
// same GPU.  The ratio of a field kernel's pair rate to its loop's ceiling is
// its loop efficiency (staging, scheduling and tails); the hardware roofline
// is the per-pipe rate (tagi_pipe_rates).
// ---------------------------------------------------------------------------
template <int KERN, bool SS>
__global__ void __launch_bounds__(FT) pair_peak_near(int reps, float *out) {
    __shared__ __align__(16) float s[5][NTILE];
    for (int j = threadIdx.x; j < NTILE; j += FT) {
        const float v = (float)((j * 37) % 101) * 0.01f - 0.5f;
        s[0][j] = -v;
        s[1][j] = -(0.3f * v + 0.1f);
        s[2][j] = -(0.7f - v);
        s[3][j] = 0.5f + 0.001f * j;
        s[4][j] = 0.25f;
    }
    __syncthreads();
    float2 tx[2], ty[2], tz[2], z2[2], nfi[2];
    float sum[2] = {0.f, 0.f}, cmp[2] = {0.f, 0.f};
    for (int k = 0; k < 2; k++) {
        tx[k] = dup2(0.01f * (threadIdx.x & 31) + 0.003f * k);
        ty[k] = dup2(0.02f);
        tz[k] = dup2(-0.03f * (threadIdx.x >> 5));
        z2[k] = dup2(0.f);
        nfi[k] = dup2(-0.3f);
    }
    for (int r = 0; r < reps; r++)
        for (int j0 = 0; j0 < NTILE; j0 += SLOT) {
            float part[2];
            near_chunk<KERN, SS, false, false, 2, NTILE>(s, j0, SLOT, tx, ty, tz, z2, z2, z2, dup2(1.f), nfi, part);
            for (int k = 0; k < 2; k++) kahan_add(sum[k], cmp[k], part[k]);
        }
    out[blockIdx.x * FT + threadIdx.x] = sum[0] + sum[1] - cmp[0] - cmp[1];
}

template <int KERN, bool SS>
__global__ void __launch_bounds__(FT) pair_peak_far(int reps, float *out) {
    constexpr int N1 = 8;
    __shared__ __align__(16) float s_q[N1 * N1 * N1];
    __shared__ __align__(16) float s_w[N1 * N1 * N1];
    __shared__ float s_p[3][N1];
    for (int k = threadIdx.x; k < N1 * N1 * N1; k += FT) {
        s_q[k] = 0.5f + 0.001f * k;
        s_w[k] = 0.25f;
    }
    if (threadIdx.x < 3 * N1) s_p[threadIdx.x / N1][threadIdx.x % N1] = 1.0f + 0.1f * threadIdx.x;
    __syncthreads();
    float tx[2], ty[2], tz[2], sum[2] = {0.f, 0.f}, cmp[2] = {0.f, 0.f};
    float2 nfi[2];
    for (int k = 0; k < 2; k++) {
        tx[k] = 0.01f * (threadIdx.x & 31) + 0.003f * k;
        ty[k] = 0.02f;
        tz[k] = -0.03f * (threadIdx.x >> 5);
        nfi[k] = dup2(-0.3f);
    }
    for (int r = 0; r < reps; r++)
        far_cluster<KERN, SS, true, N1, 2, FAR_FIXED>(s_q, s_w, s_p, N1, 0, 1, tx, ty, tz, nfi,
                                                 [&](int, int k, float part) { kahan_add(sum[k], cmp[k], part); });
    out[blockIdx.x * FT + threadIdx.x] = sum[0] + sum[1] - cmp[0] - cmp[1];
}

// Yukawa orbital groups, 8 orbitals per pair geometry; counted per (pair, orbital).
template <bool SS>
__global__ void __launch_bounds__(GT, 4) pair_peak_near_group(int reps, float *out) {
    constexpr int OG = 8;
    __shared__ __align__(16) float s[4][GTILE];
    __shared__ float4 s_q4[GTILE * OG / 4];
    for (int j = threadIdx.x; j < GTILE; j += GT) {
        const float v = (float)((j * 37) % 101) * 0.01f - 0.5f;
        s[0][j] = -v;
        s[1][j] = -(0.3f * v + 0.1f);
        s[2][j] = -(0.7f - v);
        s[3][j] = 0.25f;
    }
    for (int k = threadIdx.x; k < GTILE * OG; k += GT) reinterpret_cast<float *>(s_q4)[k] = 0.5f + 0.001f * k;
    __syncthreads();
    const float2 tx = dup2(0.01f * (threadIdx.x & 31)), ty = dup2(0.02f), tz = dup2(-0.03f * (threadIdx.x >> 5));
    float2 nfi[OG], kc[OG];
    float sum[OG], cmp[OG];
#pragma unroll
    for (int o = 0; o < OG; o++) {
        kc[o] = dup2((float)(-(0.5 + 0.3 * o) * LOG2E));
        nfi[o] = dup2(-0.3f);
        sum[o] = cmp[o] = 0.f;
    }
    const float2 z = dup2(0.f);
    for (int r = 0; r < reps; r++)
        for (int j0 = 0; j0 < GTILE; j0 += SLOT)
            group_chunk<SS, false, false, OG>(s, s_q4, j0, SLOT, tx, ty, tz, z, z, z, nfi, kc, sum, cmp);
    float acc = 0.f;
#pragma unroll
    for (int o = 0; o < OG; o++) acc += sum[o] - cmp[o];
    out[blockIdx.x * GT + threadIdx.x] = acc;
}

// Yukawa orbital groups in the far field: one degree-7 proxy grid, 8 orbitals.
template <bool SS>
__global__ void __launch_bounds__(GT, 4) pair_peak_far_group(int reps, float *out) {
    constexpr int OG = 8, N1 = 8, PP = N1 * N1 * N1;
    __shared__ float4 s_q4[PP * OG / 4];
    __shared__ __align__(16) float s_w[PP];
    __shared__ float s_p[3][N1];
    for (int k = threadIdx.x; k < PP * OG; k += GT) reinterpret_cast<float *>(s_q4)[k] = 0.5f + 0.001f * k;
    for (int k = threadIdx.x; k < PP; k += GT) s_w[k] = 0.25f;
    if (threadIdx.x < 3 * N1) s_p[threadIdx.x / N1][threadIdx.x % N1] = 1.0f + 0.1f * threadIdx.x;
    __syncthreads();
    const float tx = 0.01f * (threadIdx.x & 31), ty = 0.02f, tz = -0.03f * (threadIdx.x >> 5);
    float2 nfi[OG], kc[OG];
    float sum[OG], cmp[OG];
#pragma unroll
    for (int o = 0; o < OG; o++) {
        kc[o] = dup2((float)(-(0.5 + 0.3 * o) * LOG2E));
        nfi[o] = dup2(-0.3f);
        sum[o] = cmp[o] = 0.f;
    }
    for (int r = 0; r < reps; r++)
        far_group_cluster<SS, N1, OG, FAR_FIXED>(s_q4, s_w, s_p, N1, tx, ty, tz, nfi, kc, sum, cmp);
    float acc = 0.f;
#pragma unroll
    for (int o = 0; o < OG; o++) acc += sum[o] - cmp[o];
    out[blockIdx.x * GT + threadIdx.x] = acc;
}

// The same two loops with 16 orbitals packed by orbital (near: shared memory
// laid out as near_group16's, dynamic).
constexpr int PEAK16_TILE = GTILE;
template <bool SS>
__global__ void __launch_bounds__(GT, 4) pair_peak_near_group16(int reps, float *out) {
    extern __shared__ __align__(16) float s_dyn[];
    float(*s)[GTILE] = reinterpret_cast<float(*)[GTILE]>(s_dyn);
    float *s_q = s_dyn + 4 * GTILE;
    float *s_k = s_q + GTILE * QS16;
    for (int j = threadIdx.x; j < PEAK16_TILE; j += GT) {
        const float v = (float)((j * 37) % 101) * 0.01f - 0.5f;
        s[0][j] = -v;
        s[1][j] = -(0.3f * v + 0.1f);
        s[2][j] = -(0.7f - v);
        s[3][j] = 0.25f;
    }
    __shared__ int s_cnt[GW];
    if (threadIdx.x < GW) s_cnt[threadIdx.x] = SLOT;
    for (int k = threadIdx.x; k < PEAK16_TILE * QS16; k += GT) s_q[k] = 0.5f + 0.001f * k;
    __syncthreads();
    const float2 tx = dup2(0.01f * (threadIdx.x & 31)), ty = dup2(0.02f), tz = dup2(-0.03f * (threadIdx.x >> 5));
    float2 nfi[8], kc[8];
#pragma unroll
    for (int p = 0; p < 8; p++) {
        kc[p] = make_float2((float)(-(0.5 + 0.3 * (2 * p)) * LOG2E), (float)(-(0.5 + 0.3 * (2 * p + 1)) * LOG2E));
        nfi[p] = dup2(-0.3f);
    }
    for (int o = 0; o < 32; o++) s_k[o * GT + threadIdx.x] = 0.f;
    const float2 z = dup2(0.f);
    for (int r = 0; r < reps; r++)
        group16_tile<SS, false, false>(s, s_q, s_cnt, tx, ty, tz, z, z, z, nfi, kc, s_k);
    float acc = 0.f;
    for (int o = 0; o < 16; o++) acc += s_k[o * GT + threadIdx.x] - s_k[(16 + o) * GT + threadIdx.x];
    out[blockIdx.x * GT + threadIdx.x] = acc;
}

template <bool SS>
__global__ void __launch_bounds__(GT, 4) pair_peak_far_group16(int reps, float *out) {
    constexpr int N1 = 8, PP = N1 * N1 * N1;
    __shared__ __align__(16) float s_q[PP * QS16];
    __shared__ __align__(16) float s_w[PP];
    __shared__ float s_p[3][N1];
    for (int k = threadIdx.x; k < PP * QS16; k += GT) s_q[k] = 0.5f + 0.001f * k;
    for (int k = threadIdx.x; k < PP; k += GT) s_w[k] = 0.25f;
    if (threadIdx.x < 3 * N1) s_p[threadIdx.x / N1][threadIdx.x % N1] = 1.0f + 0.1f * threadIdx.x;
    __syncthreads();
    const float tx = 0.01f * (threadIdx.x & 31), ty = 0.02f, tz = -0.03f * (threadIdx.x >> 5);
    float2 nfi[8], kc[8];
    float sum[16], cmp[16];
#pragma unroll
    for (int p = 0; p < 8; p++) {
        kc[p] = make_float2((float)(-(0.5 + 0.3 * (2 * p)) * LOG2E), (float)(-(0.5 + 0.3 * (2 * p + 1)) * LOG2E));
        nfi[p] = dup2(-0.3f);
    }
#pragma unroll
    for (int o = 0; o < 16; o++) sum[o] = cmp[o] = 0.f;
    for (int r = 0; r < reps; r++)
        far_group16_cluster<SS, N1, FAR_FIXED>(s_q, s_w, s_p, N1, tx, ty, tz, nfi, kc, sum, cmp);
    float acc = 0.f;
#pragma unroll
    for (int o = 0; o < 16; o++) acc += sum[o] - cmp[o];
    out[blockIdx.x * GT + threadIdx.x] = acc;
}

template <int KERN, bool SS>
int launch_pair_peak(int variant, int grid, int reps, float *out, cudaStream_t s) {
    if (variant == 0) launch(pair_peak_near<KERN, SS>, grid, FT, 0, s, reps, out);
    else if (variant == 1) launch(pair_peak_far<KERN, SS>, grid, FT, 0, s, reps, out);
    else if (variant == 2) launch(pair_peak_near_group<SS>, grid, GT, 0, s, reps, out);
    else if (variant == 3) launch(pair_peak_far_group<SS>, grid, GT, 0, s, reps, out);
    else if (variant == 4) launch(pair_peak_near_group16<SS>, grid, GT, near_group16_smem(0), s, reps, out);
    else launch(pair_peak_far_group16<SS>, grid, GT, 0, s, reps, out);
    TAGI_LAUNCH_CHECK();
    return TAGI_OK;
}

template <int KERN, bool SS>
int run_pair_peak(int variant, double *pairs_per_s, cudaStream_t s) {
    if (variant < 0 || variant > 5)
        return set_error(TAGI_ERR_ARG,
                         "pair peak variant %d (0 near, 1 far, 2 near group, 3 far group, 4 near group of 16, "
                         "5 far group of 16)", variant);
    if (variant >= 2 && KERN != KERNEL_YUKAWA)
        return set_error(TAGI_ERR_UNSUPPORTED, "orbital-group kernels are Yukawa only");
    int grid = 0;
    if (variant == 0) TAGI_TRY(occupancy_grid(pair_peak_near<KERN, SS>, &grid));
    else if (variant == 1) TAGI_TRY(occupancy_grid(pair_peak_far<KERN, SS>, &grid));
    else if (variant == 2) TAGI_TRY(occupancy_grid(pair_peak_near_group<SS>, &grid, 0, GT));
    else if (variant == 3) TAGI_TRY(occupancy_grid(pair_peak_far_group<SS>, &grid, 0, GT));
    else if (variant == 4) {
        TAGI_CUDA(cudaFuncSetAttribute(pair_peak_near_group16<SS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)near_group16_smem(0)));
        TAGI_TRY(occupancy_grid(pair_peak_near_group16<SS>, &grid, near_group16_smem(0), GT));
    }
    else TAGI_TRY(occupancy_grid(pair_peak_far_group16<SS>, &grid, 0, GT));
    Arena tmp;
    tmp.stream = s;
    float *out = nullptr;
    TAGI_TRY(tmp.alloc(&out, (size_t)grid * FT));
    cudaEvent_t a, b;
    cudaEventCreate(&a);
    cudaEventCreate(&b);
    // pairs per repetition per thread: two targets x a tile, or one target x a tile x 8 (16) orbitals
    const int per_rep_of[6] = {2 * NTILE, 2 * 512, GTILE * 8, 512 * 8, PEAK16_TILE * 16, 512 * 16};
    const int per_rep = per_rep_of[variant];
    int reps = 16;
    float ms = 0.f;
    int rc = TAGI_OK;
    for (int attempt = 0; attempt < 6; attempt++) {  // grow until the timed launch lasts >= 20 ms
        if ((rc = launch_pair_peak<KERN, SS>(variant, grid, reps, out, s))) break;
        cudaEventRecord(a, s);
        if ((rc = launch_pair_peak<KERN, SS>(variant, grid, reps, out, s))) break;
        cudaEventRecord(b, s);
        if (cudaEventSynchronize(b) != cudaSuccess) { rc = set_error(TAGI_ERR_CUDA, "pair peak launch failed"); break; }
        cudaEventElapsedTime(&ms, a, b);
        if (ms >= 20.f) break;
        reps *= 4;
    }
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    tmp.release();
    if (rc) return rc;
    *pairs_per_s = (double)grid * (variant < 2 ? FT : GT) * per_rep * reps / (ms * 1e-3);
    return TAGI_OK;
}

// Kernel shape shared by every system of one field launch.
struct LaunchShape {
    int og = 1;     // orbitals per item (orbital-group kernels) or 1
    int nt = 1;     // targets per thread and
    int warps = 4;  // warps per CTA (single-orbital mixed kernels)
    int maxn1 = 1;        // largest proxy-grid edge n + 1
    int minn1 = 1 << 20;  // smallest proxy-grid edge n + 1
    bool wide = false;    // some plan's sources are staged from FP64 coordinates (Plan::wide)
};

// fn(WIDE) for the ordinary near pass.
template <typename FN>
int near_call(const LaunchShape &sh, FN &&fn) {
    return sh.wide ? fn(std::integral_constant<bool, true>()) : fn(std::integral_constant<bool, false>());
}

// fn(MAXN1, loops) for the far kernel of a launch: rows of a known length where all its
// systems have one, everything known at degree 7, the usual one.
template <int N, int LOOPS, typename FN>
int far_call(FN &&fn) { return fn(std::integral_constant<int, N>(), std::integral_constant<int, LOOPS>()); }
template <typename FN>
int far_loops(const LaunchShape &sh, FN &&fn) {
    const int row = sh.maxn1 + (sh.maxn1 & 1);
    if (sh.maxn1 <= 4) return far_call<4, FAR_ANY>(fn);
    if (sh.minn1 == 8 && sh.maxn1 == 8) return far_call<8, FAR_FIXED>(fn);
    if (sh.minn1 >= row - 1) {
        if (row == 6) return far_call<6, FAR_ROWS>(fn);
        if (row == 8) return far_call<8, FAR_ROWS>(fn);
        if (row == 10) return far_call<10, FAR_ROWS>(fn);
        return far_call<12, FAR_ROWS>(fn);
    }
    if (sh.maxn1 <= 8) return far_call<8, FAR_ANY>(fn);
    return far_call<MAX_DEGREE + 1, FAR_ANY>(fn);
}
static_assert(MAX_DEGREE == 10, "far_loops lists the row lengths");

template <int KERN, bool SS, int SW>
int launch_mixed(const Work &wn, const Work &wc, const Work &wf, const LaunchShape &sh, cudaStream_t s, bool *pdl) {
    constexpr int ST = 32 * SW;
    const bool one = sh.nt == 1;
    TAGI_TRY(near_call(sh, [&](auto wide) {
        // two targets per thread hold an item cut for one as well
        if constexpr (!wide())
            if (one) return launch_persistent(near_mixed<KERN, SS, 1, 0, SW>, wn, s, 0, ST, pdl);
        return launch_persistent(near_mixed<KERN, SS, 2, 0, SW, wide()>, wn, s, 0, ST, pdl);
    }));
    phase_mark(PH_NEAR, false, s);
    phase_mark(PH_NEAR_CLOSE, true, s);
    if (one) TAGI_TRY(launch_persistent(near_mixed<KERN, SS, 1, 1, SW>, wc, s, 0, ST, pdl));
    else TAGI_TRY(launch_persistent(near_mixed<KERN, SS, 2, 1, SW>, wc, s, 0, ST, pdl));
    phase_mark(PH_NEAR_CLOSE, false, s);
    phase_mark(PH_FAR, true, s);
    TAGI_TRY(far_loops(sh, [&](auto maxn1, auto loops) {
        if (one) return launch_persistent(far_mixed<KERN, SS, maxn1(), 1, SW, loops()>, wf, s, 0, ST, pdl);
        return launch_persistent(far_mixed<KERN, SS, maxn1(), 2, SW, loops()>, wf, s, 0, ST, pdl);
    }));
    phase_mark(PH_FAR, false, s);
    return TAGI_OK;
}

template <int KERN, bool SS>
int launch_fields(const SysCall *calls, const Fields *f, int nsys, const Schedule &sc, const LaunchShape &sh,
                  int precision, int *queue, cudaStream_t s) {
    Work wn{};
    wn.queue = queue;
    if (precision != PREC_MIXED && f64_smem<KERN, SS>()) {
        launch(exp_table, EXP_N / 64, 64, 0, s, calls[0].p->exp_table);
        wn.exp_table = calls[0].p->exp_table;
    }
    for (int i = 0; i < nsys; i++) wn.sys[i] = f[i];
    Work wc = wn, wf = wn;
    for (int i = 0; i < nsys; i++) {
        wn.sys[i].out = calls[i].p->near_out;
        wc.sys[i].out = calls[i].p->near2_out;
        wf.sys[i].out = calls[i].p->far_out;
    }
    wn.items = sc.items + sc.off[0];
    wn.nitems = sc.count[0];
    wc.items = sc.items + sc.off[1];
    wc.nitems = sc.count[1];
    wc.queue = queue + 2;
    wf.items = sc.items + sc.off[2];
    wf.nitems = sc.count[2];
    wf.queue = queue + 1;
    phase_mark(PH_NEAR, true, s);
    bool pdl = false;   // no field pass of this call launched yet
    if (precision == PREC_MIXED && KERN == KERNEL_YUKAWA && sh.og == 16) {
        TAGI_TRY(near_call(sh, [&](auto wide) {
            return launch_persistent(near_group16<SS, 0, wide()>, wn, s, near_group16_smem(0), GT, &pdl);
        }));
        phase_mark(PH_NEAR, false, s);
        phase_mark(PH_NEAR_CLOSE, true, s);
        TAGI_TRY(launch_persistent(near_group16<SS, 1>, wc, s, near_group16_smem(1), GT, &pdl));
        phase_mark(PH_NEAR_CLOSE, false, s);
        phase_mark(PH_FAR, true, s);
        TAGI_TRY(far_loops(sh, [&](auto maxn1, auto loops) {
            return launch_persistent(far_group16<SS, maxn1(), loops()>, wf, s, far_group16_smem(sh.maxn1), GT, &pdl);
        }));
        phase_mark(PH_FAR, false, s);
        return TAGI_OK;
    }
    if (precision == PREC_MIXED && KERN == KERNEL_YUKAWA && sh.og > 1) {
        // orbital groups share the geometry of each pair across og orbitals
        const bool g8 = sh.og == 8;
        TAGI_TRY(near_call(sh, [&](auto wide) {
            if (g8) return launch_persistent(near_group<SS, 8, 0, wide()>, wn, s, 0, GT, &pdl);
            return launch_persistent(near_group<SS, 4, 0, wide()>, wn, s, 0, GT, &pdl);
        }));
        phase_mark(PH_NEAR, false, s);
        phase_mark(PH_NEAR_CLOSE, true, s);
        if (g8) TAGI_TRY(launch_persistent(near_group<SS, 8, 1>, wc, s, 0, GT, &pdl));
        else TAGI_TRY(launch_persistent(near_group<SS, 4, 1>, wc, s, 0, GT, &pdl));
        phase_mark(PH_NEAR_CLOSE, false, s);
        phase_mark(PH_FAR, true, s);
        TAGI_TRY(far_loops(sh, [&](auto maxn1, auto loops) {
            if constexpr (loops() == FAR_FIXED) {   // pipelined staging
                if (g8) return launch_persistent(far_group_db<SS, 8>, wf, s, far_group_db_smem(8), GT, &pdl);
                return launch_persistent(far_group_db<SS, 4>, wf, s, far_group_db_smem(4), GT, &pdl);
            } else {
                const size_t fsm = far_group_smem(sh.maxn1, sh.og);
                if (g8) return launch_persistent(far_group<SS, maxn1(), 8, loops()>, wf, s, fsm, GT, &pdl);
                return launch_persistent(far_group<SS, maxn1(), 4, loops()>, wf, s, fsm, GT, &pdl);
            }
        }));
        phase_mark(PH_FAR, false, s);
        return TAGI_OK;
    }
    if (precision == PREC_MIXED && sh.warps == 8) TAGI_TRY((launch_mixed<KERN, SS, 8>(wn, wc, wf, sh, s, &pdl)));
    else if (precision == PREC_MIXED) TAGI_TRY((launch_mixed<KERN, SS, 4>(wn, wc, wf, sh, s, &pdl)));
    if (precision != PREC_MIXED) {
        // one FP64 pass over all near ranges, close ones included.  A list made for mixed precision
        // (schedule_for_capture) may hold more targets per item than a CTA: the passes are then
        // repeated for the next ones
        const int cta = FT / f[0].split, turns = sc.precision == PREC_FP64 ? 1 : (sc.most + cta - 1) / cta;
        for (int turn = 0; turn < turns; turn++) {
            if (turn) {
                TAGI_CUDA(cudaMemsetAsync(queue, 0, 3 * sizeof(int), s));
                pdl = false;
            }
            wn.turn = wf.turn = turn;
            if (turn) phase_mark(PH_NEAR, true, s);
            TAGI_TRY(launch_persistent(near_f64<KERN, SS>, wn, s, f64_smem<KERN, SS>(), FT, &pdl));
            phase_mark(PH_NEAR, false, s);
            phase_mark(PH_FAR, true, s);
            if (sh.maxn1 <= 4) TAGI_TRY(launch_persistent(far_f64<KERN, SS, 4>, wf, s, f64_smem<KERN, SS>(), FT, &pdl));
            else if (sh.maxn1 <= 8) TAGI_TRY(launch_persistent(far_f64<KERN, SS, 8>, wf, s, f64_smem<KERN, SS>(), FT, &pdl));
            else TAGI_TRY(launch_persistent(far_f64<KERN, SS, MAX_DEGREE + 1>, wf, s, f64_smem<KERN, SS>(), FT, &pdl));
            phase_mark(PH_FAR, false, s);
        }
    }
    return TAGI_OK;
}

// Per-orbital constants from kernel parameter kp[o * nkp] (host-copied or
// caller's device array): d_kp = k (or a), d_kc = coordinate scale sc,
// d_ss = subtraction factor 4 pi/k^2 (Yukawa) or 2 pi/a^2 (Coulomb), 0
// without subtraction.  A parameter the kernel cannot use sets bit 0 of err
// and makes the orbital's subtraction factor NaN, so all its outputs are NaN.
// Mixed precision: the field kernels see k only through the FP32 constant sc
// (k log2(e), or a sqrt(log2(e))), so the subtraction factor uses the k that
// sc represents exactly, k' = sc / log2(e) (a' = sc / sqrt(log2(e))): sums and
// subtraction term then belong to one kernel parameter, k' = k (1 + O(2^-24)),
// and the rounding of k moves the result by about twice that, smoothly,
// instead of entering the cancellation of the subtraction.
// Kernel parameters given on the host ride along as arguments (a copy of eight bytes from
// pageable memory takes 15 us), up to HOST_KP orbitals of them.
constexpr int HOST_KP = 64;
struct HostParams {
    double k[HOST_KP];
};
__global__ void orbital_constants(const double *kp, int nkp, const __grid_constant__ HostParams h, int norb,
                                  int kernel, int sing, int mixed, double *kpo, float *kc,
                                  double *ss, int *err, int *queue) {
    chain_begin();
    const int o = blockIdx.x * blockDim.x + threadIdx.x;
    if (queue && o < 3) queue[o] = 0;   // the field passes' work counters
    if (o >= norb) return;
    const double k = kp ? kp[(long)o * nkp] : h.k[o];
    const bool used = kernel == KERNEL_YUKAWA || sing == SING_SUBTRACTION;
    const bool bad = !isfinite(k) || (used && !(k > 0.0));
    if (bad) atomicOr(err, 1);
    kpo[o] = k;
    float c = 1.0f;
    if (kernel == KERNEL_YUKAWA) c = (float)(k * LOG2E);
    else if (sing == SING_SUBTRACTION) c = (float)(k * sqrt(LOG2E));
    kc[o] = c;
    double f = 0.0;
    double ke = k;
    if (mixed && kernel == KERNEL_YUKAWA) ke = (double)c / LOG2E;
    else if (mixed && sing == SING_SUBTRACTION) ke = (double)c / sqrt(LOG2E);
    if (sing == SING_SUBTRACTION) f = (kernel == KERNEL_YUKAWA ? 4.0 : 2.0) * M_PI / (ke * ke);
    ss[o] = bad ? __longlong_as_double(0x7ff8000000000000LL) : f;  // NaN marks every output of the orbital
}

Fields make_fields(const Plan &p, int norb) {
    Fields a{};
    a.tx = p.tgt.x;
    a.ty = p.tgt.y;
    a.tz = p.tgt.z;
    a.tcenter = p.tgt.center;
    a.tradius = p.tgt.radius;
    a.batch_node = p.batch_node;
    a.nt = p.tgt.n;
    a.norb = norb;
    a.rng_off = p.rng_off;
    a.rng = p.rng;
    a.rng_dmin = p.rng_dmin;
    a.sx = p.src.x;
    a.sy = p.src.y;
    a.sz = p.src.z;
    a.shi = p.src_hi;
    a.slo = p.src_lo;
    a.thi = p.tgt_hi;
    a.tlo = p.tgt_lo;
    a.ns = p.src.n;
    a.q32 = p.q32;
    a.w32 = p.sw32;
    a.f64 = p.f64s;
    a.w64 = p.sw64;
    a.far_off = p.far_off;
    a.far_list = p.far_list;
    a.node_slot = p.node_slot;
    a.geom = p.slot_geom;
    a.qhat32 = p.qhat32;
    a.what32 = p.what32;
    a.qhat64 = p.qhat64;
    a.what64 = p.what64;
    a.nslots = p.nslots;
    a.n1 = p.n1;
    a.P = p.P;
    for (int m = 0; m <= MAX_DEGREE; m++) a.tn[m] = m <= p.degree ? p.cheb[m] : 0.0;
    a.ft32 = p.ft32;
    a.ft64 = p.ft64;
    a.kc32 = p.d_kc;
    a.kp64 = p.d_kp;
    return a;
}

}  // namespace

bool stream_capturing(cudaStream_t s) {
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &st) != cudaSuccess) return false;
    return st == cudaStreamCaptureStatusActive;
}

// Per-call scratch for norb orbitals, one block.  Growing it is rare (a larger
// orbital count than any earlier call) and synchronizes the device first: the
// old block may still be in use by calls on any stream.  Plain cudaMalloc keeps
// the new one valid on every stream.  A one-shot plan's scratch serves one call
// of one precision on the plan's stream and comes from its arena.
int ensure_scratch(Plan &p, int norb, int precision) {
    if ((size_t)norb <= p.scratch_orbitals) return TAGI_OK;
    const size_t ns = p.src.n, nt = p.tgt.n, no = norb;
    const bool mixed = !p.one_shot || precision == PREC_MIXED, fp64 = !p.one_shot || precision == PREC_FP64;
    auto carve = [&](char *base) {   // the block's size; sets the pointers if base is given
        size_t at = 0;
        auto take = [&](auto **ptr, size_t count, bool wanted = true) {
            if (!wanted) return;
            if (base) *ptr = reinterpret_cast<std::remove_reference_t<decltype(*ptr)>>(base + at);
            at += ((count ? count : 1) * sizeof(**ptr) + 255) / 256 * 256;
        };
        take(&p.q32, no * ns, mixed);
        take(&p.ft32, no * nt, mixed);
        take(&p.q64, no * ns, fp64);
        take(&p.f64s, no * ns, fp64);
        take(&p.ft64, no * nt, fp64);
        take(&p.part, (no + (p.one_shot ? 1 : 0)) * p.nitems * p.P);
        take(&p.qhat32, no * p.nslots * p.P, mixed);
        take(&p.qhat64, no * p.nslots * p.P, fp64);
        take(&p.exp_table, EXP_N, fp64);
        take(&p.near_out, no * nt);
        take(&p.near2_out, no * nt);
        take(&p.far_out, no * nt);
        take(&p.d_kc, no);
        take(&p.d_kp, no);
        take(&p.d_ss, no);
        return at;
    };
    const size_t bytes = carve(nullptr);
    char *block = nullptr;
    if (p.one_shot) {
        TAGI_TRY(p.arena.alloc(&block, bytes));
    } else {
        TAGI_CUDA(cudaDeviceSynchronize());
        for (void *v : p.scratch) cudaFree(v);
        p.scratch.clear();
        p.scratch_orbitals = 0;
        const cudaError_t e = device_malloc(reinterpret_cast<void **>(&block), bytes);
        if (e != cudaSuccess)
            return set_error(TAGI_ERR_CUDA, "device allocation of %zu bytes failed: %s", bytes, cudaGetErrorString(e));
        p.scratch.push_back(block);
    }
    carve(block);
    p.scratch_orbitals = no;
    return TAGI_OK;
}

// Orbitals per work item: Yukawa in mixed precision shares each pair's
// geometry across a group of 4, 8 or 16 orbitals; everything else (and fewer
// than 4 orbitals) runs one orbital per item.  The choice minimises a cost
// model measured on GB300 (1M-point mesh, degree 7): a pass over all batches
// costs 1.0 per group of 8 (padded slots cost as much as filled ones), 0.59
// per group of 4, and 0.345 + 0.18 np per group of 16 with np filled orbital
// pairs (its kernels skip empty pairs); systems weigh by their point counts.
// Groups of 16 only up to degree 7: above it a 16-orbital proxy grid no
// longer fits two CTAs per SM.  requested > 0 (1, 4, 8 or 16) overrides the
// choice where the kernel supports it.
double group_cost(int og, int norb) {
    if (og == 16) {
        const int full = norb / 16, rem = norb % 16;
        return full * (0.345 + 0.18 * 8) + (rem ? 0.345 + 0.18 * ((rem + 1) / 2) : 0.0);
    }
    if (og == 8) return 1.0 * ((norb + 7) / 8);
    return 0.59 * ((norb + 3) / 4);
}

int orbitals_per_item(int kernel, int precision, const int *norb, const double *weight, int nsys, int requested,
                      int max_n1) {
    if (kernel != KERNEL_YUKAWA || precision != PREC_MIXED) return 1;
    if (requested == 1 || requested == 4 || requested == 8 || requested == 16) return requested;
    int maxo = 0;
    for (int i = 0; i < nsys; i++) maxo = norb[i] > maxo ? norb[i] : maxo;
    if (maxo < 4) return 1;
    int best = 0;
    double best_cost = 0.0;
    for (int og : {4, 8, 16}) {
        if (og == 16 && max_n1 > 8) continue;
        double c = 0.0;
        for (int i = 0; i < nsys; i++) c += (weight ? weight[i] : 1.0) * group_cost(og, norb[i]);
        if (!best || c < best_cost) {
            best = og;
            best_cost = c;
        }
    }
    return best;
}

bool schedule_matches(const Schedule &sc, const int *norb, int nsys, int og, int nt, int precision) {
    if (sc.og != og || sc.nt != nt || sc.precision != precision || (int)sc.norb.size() != nsys) return false;
    for (int i = 0; i < nsys; i++)
        if (sc.norb[i] != norb[i]) return false;
    return true;
}

// Of a plan's work lists the one for this call under stream capture, where none can be made: the
// call's own, or one that another targets-per-thread setting or precision made for these orbitals
// and this group size.  Mixed results do not depend on how a list cuts the batches; FP64 passes
// run once more for the targets that a CTA does not hold; an FP64 item's targets fit one thread
// each of a mixed kernel's CTA (cta_targets: 32 and 32 up to 131,072 targets, 64 and 64 or 128 above).
const Schedule *schedule_for_capture(const std::vector<Schedule> &scheds, int norb, int og, int nt, int precision) {
    const Schedule *best = nullptr;
    for (const Schedule &c : scheds) {
        if (!schedule_matches(c, &norb, 1, og, c.nt, c.precision)) continue;
        if (c.nt == nt && c.precision == precision) return &c;
        if (!best || c.precision == precision) best = &c;
    }
    return best;
}

// Warps that share a target's sources in the single-orbital kernels, by the
// plan's targets: a CTA then holds (warps / split) x 32 threads' targets, and a
// small mesh still has items for every SM, while a large one stages each tile for
// as many targets as fit.  An FP64 split follows from the plan alone, so the sums'
// last bits are the same however calls are batched (mixed sums do not depend on
// the split).  Measured, ms per call.  8 warps, split 1, 2, 4, 8 (targets and
// sources in one piece before: first figure): Yukawa, 50k points, plan kept
// 4.1 -> 4.2, 3.1, 2.0, 1.5; FP64, 50k points, one shot 636 -> 333, 325, 204, 180.
// 4 warps, split 1, 2, 4, one shot: Coulomb, 913k points, degree 6 42.1, 38.9,
// 38.6; 1.13M, degree 5 49.8, 48.1, 48.6; Yukawa, 1.34M, degree 4 73.0, 74.3, 76.7;
// Coulomb, 1.5M, degree 7 104.1, 106.6, 106.9.
int field_split(int nt, int warps, int precision) {
    if (precision == PREC_FP64) return nt <= 131072 ? 8 : 4;
    if (nt <= 131072) return warps;   // one warp of targets per CTA
    return nt <= 1200000 ? 2 : 1;
}

// Warps per CTA of the single-orbital kernels: 8 if all systems are small.
int field_warps(Plan *const *plans, int nsys, int precision) {
    if (precision == PREC_FP64) return FT / 32;
    for (int i = 0; i < nsys; i++)
        if (plans[i]->tgt.n > 131072) return 4;
    return 8;
}

// Targets that a CTA of the field kernels holds.
int cta_targets(int nt, int og, int nt_per_thread, int warps, int precision) {
    return og > 1 ? GT : 32 * warps / field_split(nt, warps, precision) * nt_per_thread;
}

// Targets per thread (single-orbital mixed kernels only): the caller's request, else 2
// where that leaves some 380 items of 64 targets.  Meshes whose CTAs hold one warp of targets
// (field_split): two targets per thread read each staged source once for both, but halve
// the items, and the chip holds 456 of these CTAs.  One against two, us, Yukawa, one orbital,
// leaves of 500: 9k targets 108, 140; 15k 186, 215; 21k 289, 294; 26k 382, 358; 40k 766, 643;
// 50k 1158, 963 (leaves of 300 and 1000 and Coulomb change sides at the same size).  Larger
// meshes: 2 where a batch fills a CTA, which holds the targets of up to eight warps.
int targets_per_thread(Plan *const *plans, const int *norb, int nsys, int precision, int og, int requested) {
    if (precision != PREC_MIXED || og != 1) return 1;
    if (requested == 1 || requested == 2) return requested;
    if (field_warps(plans, nsys, precision) == 8) {
        long targets = 0;
        for (int i = 0; i < nsys; i++) targets += (long)plans[i]->tgt.n * norb[i];
        return targets > 24000 ? 2 : 1;
    }
    for (int i = 0; i < nsys; i++)
        if (plans[i]->max_batch > FT) return 2;
    return 1;
}

// Work lists for one launch over nsys systems: one item per (system, batch,
// chunk of its targets, group of og orbitals), ordered by pair count, heaviest
// first (ties in system, batch, chunk, group order).  A batch's targets are cut
// evenly, in whole warps, into chunks of at most what a CTA holds (nt per thread).
// Passes that have nothing to do for a batch (no close ranges, no far entries)
// get no item: their outputs are cleared before the launch.
int build_schedule(Plan *const *plans, const int *norb, int nsys, int og, int nt, int precision, Schedule &sc,
                   cudaStream_t s) {
    if (nsys < 1 || nsys > MAX_SYSTEMS) return set_error(TAGI_ERR_ARG, "%d systems (1..%d per launch)", nsys, MAX_SYSTEMS);
    const int warps = field_warps(plans, nsys, precision);
    sc.most = 0;
    struct Batch {
        long long cost;   // pairs of one chunk
        int sys, b, begin, end, chunk;
    };
    std::vector<Batch> lists[3];
    for (int i = 0; i < nsys; i++) {
        const Plan &p = *plans[i];
        if (norb[i] < 1 || norb[i] > 0xffff) return set_error(TAGI_ERR_ARG, "system %d: %d orbitals", i, norb[i]);
        if ((int)p.cost_near.size() != p.nbatch) return set_error(TAGI_ERR_STATE, "plan without batch costs");
        const int warp = 32 * nt, most = cta_targets(p.tgt.n, og, nt, warps, precision);
        sc.most = std::max(sc.most, most);
        for (int b = 0, at = 0; b < p.nbatch; at += p.batch_size[b++]) {
            const int n = p.batch_size[b], chunks = (n + most - 1) / most;
            const int chunk = ((n + chunks - 1) / chunks + warp - 1) / warp * warp;
            const long long *cost[3] = {&p.cost_near[b], &p.cost_close[b], &p.cost_far[b]};
            for (int k = 0; k < 3; k++)
                if (k == 0 || *cost[k] > 0) lists[k].push_back({*cost[k] / n * std::min(n, chunk), i, b, at, at + n, chunk});
        }
    }
    std::vector<int4> all;
    for (int k = 0; k < 3; k++) {
        std::stable_sort(lists[k].begin(), lists[k].end(),
                         [](const Batch &a, const Batch &b) { return a.cost > b.cost; });
        sc.off[k] = (long)all.size();
        for (const Batch &v : lists[k])
            for (int t = v.begin; t < v.end; t += v.chunk)
                for (int g0 = 0; g0 < norb[v.sys]; g0 += og)
                    all.push_back(make_int4(v.b, (v.sys << 16) | g0, t, std::min(t + v.chunk, v.end)));
        sc.count[k] = (int)((long)all.size() - sc.off[k]);
    }
    if (all.empty()) all.push_back(make_int4(0, 0, 0, 0));
    if (nsys == 1 && plans[0]->one_shot) {
        TAGI_TRY(plans[0]->arena.alloc(&sc.items, all.size()));
        sc.borrowed = true;
    } else {
        // the old list may be in use on any stream: wait, then replace it
        TAGI_CUDA(cudaDeviceSynchronize());
        sc.release();
        void *v = nullptr;
        TAGI_CUDA(device_malloc(&v, sizeof(int4) * all.size()));
        sc.items = static_cast<int4 *>(v);
    }
    // pageable source: the copy has read it when the call returns
    TAGI_CUDA(cudaMemcpyAsync(sc.items, all.data(), sizeof(int4) * all.size(), cudaMemcpyHostToDevice, s));
    sc.og = og;
    sc.nt = nt;
    sc.precision = precision;
    sc.norb.assign(norb, norb + nsys);
    return TAGI_OK;
}

// Per-orbital constants of one system into p.d_kp / d_kc / d_ss.
static int orbital_setup(Plan &p, const SysCall &c, int kernel, int singularity, int mixed, int *queue, cudaStream_t s) {
    const double *src = c.kp;
    int stride = c.nkp;
    HostParams h{};
    if (!c.kp_device && c.norb <= HOST_KP) {
        for (int o = 0; o < c.norb; o++) h.k[o] = c.kp[(long)o * c.nkp];
        src = nullptr;
    } else if (!c.kp_device) {
        p.h_kp.resize(c.norb);
        for (int o = 0; o < c.norb; o++) p.h_kp[o] = c.kp[(long)o * c.nkp];
        TAGI_CUDA(cudaMemcpyAsync(p.d_kp, p.h_kp.data(), sizeof(double) * c.norb, cudaMemcpyHostToDevice, s));
        src = p.d_kp;
        stride = 1;
    }
    TAGI_CUDA(launch_chained(orbital_constants, (c.norb + 127) / 128, 128, 0, s, src, stride, h, c.norb, kernel,
                             singularity, mixed, p.d_kp, p.d_kc, p.d_ss, p.err_flag + 1, queue));
    return TAGI_OK;
}

// One convolution call over nsys systems (1..MAX_SYSTEMS) sharing kernel,
// singularity handling and precision: per-system glue and upward pass, then
// ONE persistent launch per field pass across all systems, then per-system
// epilogues.  Under stream capture nothing may allocate or copy from host
// memory: scratch, schedule and FP64 weight charges must exist already, and
// kernel parameters must be on the device.
// later: makes the schedule while the set-up kernels and the upward pass run, where the
// caller has none yet.
static int convolve_with(SysCall *calls, int nsys, int kernel, int singularity, int precision, const Schedule *ready,
                         const std::function<int(const Schedule **)> &later, int *queue, cudaStream_t s) {
    if (nsys < 1 || nsys > MAX_SYSTEMS) return set_error(TAGI_ERR_ARG, "%d systems (1..%d per launch)", nsys, MAX_SYSTEMS);
    const bool mixed = precision == PREC_MIXED;
    const bool ss = singularity == SING_SUBTRACTION;
    const bool capturing = stream_capturing(s);
    Fields f[MAX_SYSTEMS];
    Plan *plans[MAX_SYSTEMS];
    LaunchShape sh;
    for (int i = 0; i < nsys; i++) {
        SysCall &c = calls[i];
        Plan &p = *c.p;
        if (capturing) {
            if ((size_t)c.norb > p.scratch_orbitals || (!mixed && p.nslots && !p.what64_ready) || !c.kp_device)
                return set_error(TAGI_ERR_STATE,
                                 "graph capture needs a prior uncaptured call with the same orbital counts and "
                                 "precision, and kernel parameters on the device");
        }
        TAGI_TRY(ensure_scratch(p, c.norb, precision));
        TAGI_TRY(orbital_setup(p, c, kernel, singularity, mixed ? 1 : 0, i == 0 ? queue : nullptr, s));
        const int ns = p.src.n, nt = p.tgt.n;
        dim3 gs((ns + 255) / 256, c.norb), gt((nt + 255) / 256, c.norb);
        phase_mark(PH_GLUE, true, s);
        TAGI_CUDA(launch_chained(mixed ? prep_sources<true> : prep_sources<false>, gs, 256, 0, s, c.sv, p.src.perm,
                                 p.sw64, ns, p.q32, p.q64, p.f64s));
        TAGI_CUDA(launch_chained(mixed ? prep_targets<true> : prep_targets<false>, gt, 256, 0, s, c.tv, p.tgt.perm, nt,
                                 p.ft32, p.ft64, p.near2_out, p.far_out));
        phase_mark(PH_GLUE, false, s);
        phase_mark(PH_UPWARD, true, s);
        TAGI_TRY(modified_charges(p, mixed ? PREC_MIXED : PREC_FP64, c.norb, s));
        if (!mixed && !p.one_shot) TAGI_TRY(ensure_weight_charges64(p, s));  // before what64 is read below
        phase_mark(PH_UPWARD, false, s);
        if (!mixed && p.nslots && !p.what64) return set_error(TAGI_ERR_DEVICE, "FP64 weight charges missing");
        f[i] = make_fields(p, c.norb);
        plans[i] = c.p;
        sh.wide = sh.wide || p.wide;
        if (p.n1 > sh.maxn1) sh.maxn1 = p.n1;
        if (p.n1 < sh.minn1) sh.minn1 = p.n1;
    }
    if (!ready) TAGI_TRY(later(&ready));
    const Schedule &sc = *ready;
    sh.og = sc.og;
    sh.nt = sc.nt;
    sh.warps = field_warps(plans, nsys, precision);
    for (int i = 0; i < nsys; i++) f[i].split = field_split(plans[i]->tgt.n, sh.warps, precision);
    if (kernel == KERNEL_YUKAWA) {
        if (ss) TAGI_TRY((launch_fields<KERNEL_YUKAWA, true>(calls, f, nsys, sc, sh, precision, queue, s)));
        else TAGI_TRY((launch_fields<KERNEL_YUKAWA, false>(calls, f, nsys, sc, sh, precision, queue, s)));
    } else {
        if (ss) TAGI_TRY((launch_fields<KERNEL_COULOMB, true>(calls, f, nsys, sc, sh, precision, queue, s)));
        else TAGI_TRY((launch_fields<KERNEL_COULOMB, false>(calls, f, nsys, sc, sh, precision, queue, s)));
    }
    phase_mark(PH_GLUE, true, s);
    for (int i = 0; i < nsys; i++) {
        const SysCall &c = calls[i];
        const Plan &p = *c.p;
        const int nt = p.tgt.n;
        dim3 gt((nt + 255) / 256, c.norb);
        if (mixed)
            launch(epilogue<float>, gt, 256, 0, s, p.near_out, p.near2_out, p.far_out, p.ft32, p.tgt.perm, nt,
                   p.d_ss, c.out);
        else
            launch(epilogue<double>, gt, 256, 0, s, p.near_out, p.near2_out, p.far_out, p.ft64, p.tgt.perm, nt,
                   p.d_ss, c.out);
    }
    phase_mark(PH_GLUE, false, s);
    TAGI_LAUNCH_CHECK();
    return TAGI_OK;
}

int convolve_systems(SysCall *calls, int nsys, int kernel, int singularity, int precision, const Schedule &sc, int *queue,
                     cudaStream_t s) {
    return convolve_with(calls, nsys, kernel, singularity, precision, &sc, nullptr, queue, s);
}

// Single-plan call (norb orbitals over one mesh) with the plan's cached
// work list.
int convolve(Plan &p, const double *tv, const double *sv, double *out, int norb, int kernel,
             const double *kparams, int nkp, int singularity, int precision, cudaStream_t s, bool kp_device,
             int og_request, int nt_request) {
    const int og = orbitals_per_item(kernel, precision, &norb, nullptr, 1, og_request, p.n1);
    Plan *pp = &p;
    const int nt = targets_per_thread(&pp, &norb, 1, precision, og, nt_request);
    const Schedule *sc = nullptr;
    if (stream_capturing(s)) {
        sc = schedule_for_capture(p.scheds, norb, og, nt, precision);
        if (!sc)
            return set_error(TAGI_ERR_STATE, "graph capture needs a prior uncaptured call with the same orbital count");
    } else {
        for (const Schedule &c : p.scheds)
            if (schedule_matches(c, &norb, 1, og, nt, precision)) sc = &c;
    }
    if (norb < 1 || norb > 0xffff) return set_error(TAGI_ERR_ARG, "system 0: %d orbitals", norb);
    auto make_schedule = [&](const Schedule **out) -> int {
        // Lists of KEEP orbital counts and group sizes are kept (e.g. Hartree + orbital batch), each
        // in up to three forms (precision, targets per thread): a captured graph reads its list from
        // here, and calls on the same orbitals in another form must not take it away.
        constexpr int KEEP = 4;
        auto same_orbitals = [](const Schedule &a, const Schedule &b) { return a.og == b.og && a.norb == b.norb; };
        int kinds = 0;
        bool known = false;
        for (size_t i = 0; i < p.scheds.size(); i++) {
            bool first = true;
            for (size_t j = 0; j < i; j++) first = first && !same_orbitals(p.scheds[i], p.scheds[j]);
            kinds += first;
            known = known || schedule_matches(p.scheds[i], &norb, 1, og, p.scheds[i].nt, p.scheds[i].precision);
        }
        if (!known && kinds >= KEEP) {   // the oldest orbital count's lists go
            TAGI_CUDA(cudaDeviceSynchronize());
            const Schedule oldest = p.scheds.front();
            for (size_t i = 0; i < p.scheds.size();) {
                if (same_orbitals(p.scheds[i], oldest)) {
                    p.scheds[i].release();
                    p.scheds.erase(p.scheds.begin() + i);
                } else {
                    i++;
                }
            }
        }
        p.scheds.emplace_back();
        const int rc = build_schedule(&pp, &norb, 1, og, nt, precision, p.scheds.back(), s);
        if (rc) {
            p.scheds.back().release();
            p.scheds.pop_back();
            return rc;
        }
        *out = &p.scheds.back();
        return TAGI_OK;
    };
    SysCall c;
    c.p = &p;
    c.tv = tv;
    c.sv = sv;
    c.out = out;
    c.norb = norb;
    c.kp = kparams;
    c.nkp = nkp;
    c.kp_device = kp_device;
    return convolve_with(&c, 1, kernel, singularity, precision, sc, make_schedule, p.queue, s);
}

int pair_peak(int kernel, int singularity, int variant, double kp, double *pairs_per_s, cudaStream_t s) {
    (void)kp;
    const bool ss = singularity == SING_SUBTRACTION;
    if (kernel == KERNEL_YUKAWA)
        return ss ? run_pair_peak<KERNEL_YUKAWA, true>(variant, pairs_per_s, s)
                  : run_pair_peak<KERNEL_YUKAWA, false>(variant, pairs_per_s, s);
    return ss ? run_pair_peak<KERNEL_COULOMB, true>(variant, pairs_per_s, s)
              : run_pair_peak<KERNEL_COULOMB, false>(variant, pairs_per_s, s);
}

}  // namespace tagi
