// Learned extrapolation of Green iteration: a small MLP on per-cell patches,
// trained on the device by this file's kernels.  No counterpart in the
// reference (its closest relative is the Anderson mixing of orbitals,
// scfFixedPoint.py:491-597); the plain Green-iteration residual checks every
// proposal, so the plain method stays the fallback.
//
// Rows are (orbital, cell) patches of P = (order+1)^3 mesh points (the mesh
// stores each cell's points contiguously).  Features of a row, in BF16:
//   [ psi / s_psi (P), d / s_d (P), eps, 0 padding ]   d = psi_t - psi_{t-1}
// with s_psi, s_d the patch RMS values (s_d floored by a fraction of the
// orbital's RMS update).  The network predicts the next update of the patch
// in units of s_d:  d_next / s_d ~ alpha * d / s_d + MLP(features).
// MLP: Linear(Din -> H) ReLU Linear(H -> H) ReLU Linear(H -> P), weights BF16
// (FP32 master copies for Adam), every product accumulated in FP32.
//
// GEMMs run on the tensor cores, BF16 in, FP32 accumulate: C[M x N] =
// A[M x K] B[K x N] with strides, so the transposes of the backward pass need
// no copies.  Operands that TMA can read (one unit stride, the other a multiple
// of 16 bytes, base 16-byte aligned) are copied by TMA; others, such as rows of 125
// or 343 patch points, by warps.  Both feed the same tcgen05 kernel (gemm_tc,
// accumulators in TMEM).  Weight gradients split K across
// blocks into partial sums that a second kernel adds in a fixed order: results
// do not depend on scheduling.
#include "tagi_internal.h"

#include <cuda.h>
#include <cuda_bf16.h>

#include <algorithm>

namespace tagi {

namespace {

enum { EPI_F32 = 0, EPI_BIAS_RELU_BF16 = 1, EPI_MASK_BF16 = 2, EPI_BIAS_F32 = 3 };

struct GemmArgs {
    const __nv_bfloat16 *A, *B;
    long sAm, sAk, sBk, sBn;
    int M, N, K;
    int k_per_split;     // K range of one blockIdx.z
    float *C32;          // f32 output (or partials [split][M][N])
    __nv_bfloat16 *C16;  // bf16 output
    long sCm;            // output row stride (elements)
    const float *bias;   // [N]
    const __nv_bfloat16 *mask;  // [M][sCm]: multiply by (mask > 0)
    int epi;
};

__device__ __forceinline__ unsigned pack2(__nv_bfloat16 lo, __nv_bfloat16 hi) {
    return (unsigned)__bfloat16_as_ushort(lo) | ((unsigned)__bfloat16_as_ushort(hi) << 16);
}

// ---------------------------------------------------------------------------
// gemm_tc: one 128 x 128 tile of C per CTA on the 5th-generation tensor cores.
// Bound: at the extrapolator's sizes (10,752 rows, 256 wide) reading the
// activations; a K step of 64 moves 32 KB into shared memory for 128 clocks of
// tcgen05.mma.  So: 128-byte-swizzled TMA tiles in a three-stage ring (96 KB, two
// CTAs per SM: one's epilogue runs beside the other's loads), one thread issuing
// the copies, one the MMAs, the accumulator in 128 TMEM columns, and an epilogue
// through shared memory so that rows of C are written in whole sectors.  A tile
// of either operand may lie K-major (rows of 64 k) or MN-major (rows of 64 m or n:
// the weight gradients' transposes); TMA fills elements outside the matrix with 0.
// SA, SB: that operand's tiles come from eight more warps, which load 2 bytes per
// element (a row may start at any of them) into registers while the previous stage is
// read, and store them in the layout that TMA would have written.
// Five GEMMs and a column sum, hidden width 256, before with mma.sync and element-wise
// staging: 10,752 rows of 512-point patches 872 -> 78 us, 6,090 rows of 125 points
// 480 -> 114 us (219 with mma.sync in the two products that TMA cannot read).
// ---------------------------------------------------------------------------
constexpr int TC_M = 128, TC_N = 128, TC_K = 64, TC_THREADS = 128, TC_LOADERS = 256;
// Stages of the ring: 3 (two CTAs per SM), or 6 where the grid leaves an SM to each CTA and
// TMA feeds both operands: a K loop runs at the stages in flight over a load's latency.  Six
// calls at 10,752 rows, 78.5 -> 75.8 us; tiles that warps load gained nothing (343 points).
constexpr int TC_TILE = 128 * TC_K * 2;                 // bytes of one operand's tile
constexpr int TC_PITCH = TC_N + 4;                      // floats per staged row of C
__host__ __device__ constexpr size_t tc_smem(int stages) { return 1024 + (size_t)stages * 2 * TC_TILE; }
static_assert(tc_smem(3) * 5 > 228 * 1024, "at most four blocks of 128 TMEM columns each may share an SM");
static_assert((size_t)TC_M * TC_PITCH * 4 <= (size_t)3 * 2 * TC_TILE, "C tile in the ring's memory");
static_assert(tc_smem(6) <= 227 * 1024, "one block's shared memory");
// Tries of a barrier wait before it gives up, 3.8 us each where nothing comes: one second; a sixteenth for
// each stage's copies after a wait gave up.
constexpr int TC_SPINS = 1 << 18, TC_DRAIN = TC_SPINS / 16;

__device__ __forceinline__ unsigned smem_u32(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t *b, unsigned n) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(b)), "r"(n) : "memory");
}
__device__ __forceinline__ void mbar_expect(uint64_t *b, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(b)), "r"(bytes) : "memory");
}
// false if the phase did not complete within `tries` tries
__device__ __forceinline__ bool mbar_wait(uint64_t *b, unsigned parity, int tries = TC_SPINS) {
    for (int i = 0; i < tries; i++) {
        unsigned ok;
        asm volatile(
            "{\n.reg .pred p;\n"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
            "selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(ok)
            : "r"(smem_u32(b)), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    return false;
}
__device__ __forceinline__ void tma_load(void *dst, const CUtensorMap *map, int x, int y, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            smem_u32(dst)),
        "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar))
        : "memory");
}
// Shared-memory matrix descriptor, 128-byte swizzle.  K-major: rows of 64 k,
// groups of 8 rows 1024 bytes apart.  MN-major: 64 m (or n) per row of one k, 8 k
// per 1024 bytes, the next 64 m 8192 bytes on.
__device__ __forceinline__ uint64_t smem_desc(unsigned addr, bool k_major) {
    const uint64_t lbo = k_major ? 1 : 8192 >> 4, sbo = 1024 >> 4;
    return (uint64_t)((addr >> 4) & 0x3fff) | lbo << 16 | sbo << 32 | 1ULL << 46 | 2ULL << 61;
}

struct TcArgs {
    GemmArgs g;
    int a_kmajor, b_kmajor;
};

__device__ int g_tc_timeout;   // set by a CTA whose barrier wait gave up (its tile of C is NaN); tagi_mlp_check

__global__ void take_timeout(int *out) { *out = atomicExch(&g_tc_timeout, 0); }

// A wait that nothing ends, as in gemm_tc.
__global__ void wait_probe(int tries) {
    __shared__ __align__(8) uint64_t bar;
    mbar_init(&bar, 1);
    if (!mbar_wait(&bar, 0, tries)) g_tc_timeout = 1;
}

// Rows of 64 consecutive k (K-major) or of 64 m of one k (MN-major) starting at row
// `first` of a tile, `step` rows apart: the pair of elements at 2 lane, packed.
template <int ROWS>
__device__ __forceinline__ void load_rows(unsigned (&v)[ROWS], const __nv_bfloat16 *base, long smn, long sk, bool k_major,
                                          int i0, int mn, int k0, int K, int first, int step, int lane) {
    const unsigned short *p = reinterpret_cast<const unsigned short *>(base);
#pragma unroll
    for (int r = 0; r < ROWS; r++) {
        const int row = first + r * step, c = 2 * lane;
        const int i = k_major ? i0 + row : i0 + (row & 64) + c, k = k_major ? k0 + c : k0 + (row & 63);
        const long o = i * smn + k * sk;
        const bool in0 = i < mn && k < K, in1 = k_major ? i < mn && k + 1 < K : i + 1 < mn && k < K;
        const unsigned lo = in0 ? p[o] : 0, hi = in1 ? p[o + (k_major ? sk : smn)] : 0;
        v[r] = lo | hi << 16;
    }
}
template <int ROWS>
__device__ __forceinline__ void store_rows(const unsigned (&v)[ROWS], char *tile, int first, int step, int lane) {
#pragma unroll
    for (int r = 0; r < ROWS; r++) {
        const int row = first + r * step;   // 128-byte swizzle: 16-byte piece c of row r lies at c ^ (r mod 8)
        *reinterpret_cast<unsigned *>(tile + row * 128 + (((lane >> 2) ^ (row & 7)) << 4) + ((lane & 3) << 2)) = v[r];
    }
}

template <bool SA, bool SB, int STAGES>
__global__ void __launch_bounds__(TC_THREADS + (SA || SB ? TC_LOADERS : 0), STAGES == 3 ? 2 : 1) gemm_tc(
    const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB, const __grid_constant__ TcArgs t) {
    constexpr int WARPS = (TC_THREADS + (SA || SB ? TC_LOADERS : 0)) / 32, LW = TC_LOADERS / 32, ROWS = 128 / LW;
    extern __shared__ char s_raw[];
    __shared__ __align__(8) uint64_t s_full[STAGES], s_empty[STAGES], s_done;
    __shared__ unsigned s_tmem;
    __shared__ int s_fail;
    // Early: this grid is resident as a whole by then, and the next kernel's blocks wait
    // only for it.  A next gemm_tc takes its 128 TMEM columns before this one ends; shared
    // memory allows at most two of these blocks on an SM, so all of them find columns.
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const GemmArgs &g = t.g;
    char *ring = s_raw + (1024 - (smem_u32(s_raw) & 1023)) % 1024;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = blockIdx.y * TC_M, n0 = blockIdx.x * TC_N;
    const int kb = blockIdx.z * g.k_per_split, ke = min(g.K, kb + g.k_per_split);
    const int steps = (ke - kb + TC_K - 1) / TC_K;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 128;" ::"r"(smem_u32(&s_tmem))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0) {
        for (int i = 0; i < STAGES; i++) {
            mbar_init(&s_full[i], (SA && SB ? 0 : 1) + (SA || SB ? LW : 0));
            mbar_init(&s_empty[i], 1);
        }
        mbar_init(&s_done, 1);
        s_fail = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const unsigned tmem = s_tmem;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if ((!SA || !SB) && tid == 0) {   // copies
        for (int i = 0; i < steps; i++) {
            const int st = i % STAGES;
            char *a = ring + st * 2 * TC_TILE, *b = a + TC_TILE;
            if (i >= STAGES && !mbar_wait(&s_empty[st], (i / STAGES - 1) & 1)) {
                s_fail = 1;
                break;
            }
            const int k = kb + i * TC_K;
            mbar_expect(&s_full[st], (SA || SB ? 1 : 2) * TC_TILE);
            if (SA) {
            } else if (t.a_kmajor) {
                tma_load(a, &mapA, k, m0, &s_full[st]);
            } else {
                tma_load(a, &mapA, m0, k, &s_full[st]);
                tma_load(a + TC_TILE / 2, &mapA, m0 + 64, k, &s_full[st]);
            }
            if (SB) {
            } else if (t.b_kmajor) {
                tma_load(b, &mapB, k, n0, &s_full[st]);
            } else {
                tma_load(b, &mapB, n0, k, &s_full[st]);
                tma_load(b + TC_TILE / 2, &mapB, n0 + 64, k, &s_full[st]);
            }
        }
    } else if (tid == 32) {   // MMAs
        // f32 accumulator, bf16 operands, their majors, N / 8, M / 16
        const unsigned idesc = 1u << 4 | 1u << 7 | 1u << 10 | (t.a_kmajor ? 0u : 1u << 15) |
                               (t.b_kmajor ? 0u : 1u << 16) | (unsigned)(TC_N / 8) << 17 | (unsigned)(TC_M / 16) << 24;
        const unsigned stepA = t.a_kmajor ? 32 >> 4 : 2048 >> 4, stepB = t.b_kmajor ? 32 >> 4 : 2048 >> 4;
        for (int i = 0; i < steps; i++) {
            const int st = i % STAGES;
            if (!mbar_wait(&s_full[st], (i / STAGES) & 1)) {
                s_fail = 1;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const unsigned a = smem_u32(ring + st * 2 * TC_TILE);
            uint64_t da = smem_desc(a, t.a_kmajor), db = smem_desc(a + TC_TILE, t.b_kmajor);
#pragma unroll
            for (int kk = 0; kk < TC_K / 16; kk++) {
                const unsigned acc = i > 0 || kk > 0;
                asm volatile(
                    "{\n.reg .pred p;\nsetp.ne.u32 p, %4, 0;\n"
                    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem),
                    "l"(da), "l"(db), "r"(idesc), "r"(acc)
                    : "memory");
                da += stepA;
                db += stepB;
            }
            asm volatile(
                "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(&s_empty[st]))
                : "memory");
        }
        asm volatile(
            "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(&s_done))
            : "memory");
    } else if ((SA || SB) && warp >= TC_THREADS / 32) {   // loads by warps
        const int w = warp - TC_THREADS / 32;
        for (int i = 0; i < steps; i++) {
            const int st = i % STAGES, k = kb + i * TC_K;
            char *a = ring + st * 2 * TC_TILE;
            unsigned va[SA ? ROWS : 1], vb[SB ? ROWS : 1];
            if (SA) load_rows(va, g.A, g.sAm, g.sAk, t.a_kmajor, m0, g.M, k, g.K, w, LW, lane);
            if (SB) load_rows(vb, g.B, g.sBn, g.sBk, t.b_kmajor, n0, g.N, k, g.K, w, LW, lane);
            const bool ready = i < STAGES || mbar_wait(&s_empty[st], (i / STAGES - 1) & 1);
            if (!__all_sync(0xffffffffu, ready)) {
                s_fail = 1;
                break;
            }
            if (SA) store_rows(va, a, w, LW, lane);
            if (SB) store_rows(vb, a + TC_TILE, w, LW, lane);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the MMA reads through the async proxy
            __syncwarp();
            if (lane == 0)
                asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&s_full[st])) : "memory");
        }
    }
    __syncwarp();
    bool ok = mbar_wait(&s_done, 0, TC_SPINS + steps);   // the whole K loop
    __syncthreads();
    ok = ok && !s_fail;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (!ok) {   // give the copies in flight time to land before the memory is reused or left
        if (tid == 0) {
            g_tc_timeout = 1;
            for (int st = 0; st < STAGES; st++) mbar_wait(&s_full[st], 0, TC_DRAIN), mbar_wait(&s_full[st], 1, TC_DRAIN);
        }
        __syncthreads();
    }
    // accumulator: lane 32 warp + lane of TMEM is row m0 + 32 warp + lane
    float *crow = reinterpret_cast<float *>(ring) + (32 * warp + lane) * TC_PITCH;
#pragma unroll
    for (int c = 0; c < TC_N && warp < TC_THREADS / 32; c += 32) {
        unsigned v[32];
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
            "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,"
            "%29,%30,%31}, [%32];"
            : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
              "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
              "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
              "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
            : "r"(tmem + ((unsigned)(32 * warp) << 16) + c));
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int q = 0; q < 32; q += 4)
            *reinterpret_cast<float4 *>(crow + c + q) = make_float4(__uint_as_float(v[q]), __uint_as_float(v[q + 1]),
                                                                    __uint_as_float(v[q + 2]), __uint_as_float(v[q + 3]));
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 128;" ::"r"(tmem));
    const float bad = ok ? 0.f : __int_as_float(0x7fffffff);
    const float *ct = reinterpret_cast<const float *>(ring);
    const int rows = min(TC_M, g.M - m0), cols = min(TC_N, g.N - n0);
    // Four columns per lane, a row per warp and turn: bias values stay in registers, and
    // EPI_ROWS rows' mask values are on their way at once (element by element each row waited
    // for its own: 22.8 us for the masked product at 10,752 rows, 10 us for its K loop).
    constexpr int EPI_ROWS = 8;
    const int c0 = 4 * lane;
    const bool mine = c0 < cols;   // some of this lane's columns are inside
    const bool f32 = g.epi == EPI_F32 || g.epi == EPI_BIAS_F32, masked = g.epi == EPI_MASK_BF16;
    float4 bias = make_float4(0.f, 0.f, 0.f, 0.f);
    if (g.epi == EPI_BIAS_F32 || g.epi == EPI_BIAS_RELU_BF16) {
        const float *bp = g.bias + n0 + c0;
        if (mine) bias.x = bp[0];
        if (c0 + 1 < cols) bias.y = bp[1];
        if (c0 + 2 < cols) bias.z = bp[2];
        if (c0 + 3 < cols) bias.w = bp[3];
    }
    const bool whole = c0 + 3 < cols;
    if (f32) {
        float *C = g.C32 + (long)blockIdx.z * g.M * g.sCm + (long)m0 * g.sCm + n0;
        const bool vec = whole && !(g.sCm & 3) && !(reinterpret_cast<uintptr_t>(C) & 15);
        const bool add = g.epi == EPI_BIAS_F32;
#pragma unroll 4
        for (int r = warp; r < rows; r += WARPS) {
            if (!mine) break;
            const float4 t4 = *reinterpret_cast<const float4 *>(ct + r * TC_PITCH + c0);
            float4 v = make_float4(t4.x + bad, t4.y + bad, t4.z + bad, t4.w + bad);
            if (add) v = make_float4(t4.x + (bias.x + bad), t4.y + (bias.y + bad), t4.z + (bias.z + bad), t4.w + (bias.w + bad));
            float *o = C + (long)r * g.sCm + c0;
            if (vec) {
                *reinterpret_cast<float4 *>(o) = v;
            } else {
                o[0] = v.x;
                if (c0 + 1 < cols) o[1] = v.y;
                if (c0 + 2 < cols) o[2] = v.z;
                if (c0 + 3 < cols) o[3] = v.w;
            }
        }
        return;
    }
    __nv_bfloat16 *C = g.C16 + (long)m0 * g.sCm + n0;
    const __nv_bfloat16 *mask = masked ? g.mask + (long)m0 * g.sCm + n0 : nullptr;
    const bool vec = whole && !(g.sCm & 3) && !(reinterpret_cast<uintptr_t>(C) & 7);
    const bool mvec = whole && !(g.sCm & 3) && !(reinterpret_cast<uintptr_t>(mask) & 7);
    auto bits = [](__nv_bfloat16 v) { return (unsigned)__bfloat16_as_ushort(v); };
    auto relu = [&](float v, float b) {
        v = v + bad + b;
        return __float2bfloat16_rn(v > 0.f ? v : (v != v ? v : 0.f));
    };
    auto gate = [&](float v, unsigned m) {
        return __float2bfloat16_rn((v + bad) * (__bfloat162float(__ushort_as_bfloat16((unsigned short)m)) > 0.f ? 1.f : 0.f));
    };
    for (int r0 = warp; r0 < rows && mine; r0 += EPI_ROWS * WARPS) {
        uint2 mk[EPI_ROWS];
#pragma unroll
        for (int u = 0; u < EPI_ROWS; u++) {
            const int r = r0 + u * WARPS;
            mk[u] = make_uint2(0, 0);
            if (!masked || r >= rows) continue;
            const __nv_bfloat16 *mp = mask + (long)r * g.sCm + c0;
            if (mvec) {
                mk[u] = *reinterpret_cast<const uint2 *>(mp);
            } else {
                mk[u].x = bits(mp[0]);
                if (c0 + 1 < cols) mk[u].x |= bits(mp[1]) << 16;
                if (c0 + 2 < cols) mk[u].y = bits(mp[2]);
                if (c0 + 3 < cols) mk[u].y |= bits(mp[3]) << 16;
            }
        }
#pragma unroll
        for (int u = 0; u < EPI_ROWS; u++) {
            const int r = r0 + u * WARPS;
            if (r >= rows) break;
            const float4 t4 = *reinterpret_cast<const float4 *>(ct + r * TC_PITCH + c0);
            __nv_bfloat16 v[4];
            if (masked) {
                v[0] = gate(t4.x, mk[u].x & 0xffffu);
                v[1] = gate(t4.y, mk[u].x >> 16);
                v[2] = gate(t4.z, mk[u].y & 0xffffu);
                v[3] = gate(t4.w, mk[u].y >> 16);
            } else {
                v[0] = relu(t4.x, bias.x);
                v[1] = relu(t4.y, bias.y);
                v[2] = relu(t4.z, bias.z);
                v[3] = relu(t4.w, bias.w);
            }
            __nv_bfloat16 *o = C + (long)r * g.sCm + c0;
            if (vec) {
                *reinterpret_cast<uint2 *>(o) = make_uint2(pack2(v[0], v[1]), pack2(v[2], v[3]));
            } else {
                o[0] = v[0];
                if (c0 + 1 < cols) o[1] = v[1];
                if (c0 + 2 < cols) o[2] = v[2];
                if (c0 + 3 < cols) o[3] = v[3];
            }
        }
    }
}

typedef CUresult (*EncodeTiled)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiled encode_tiled() {
    static const EncodeTiled fn = [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) != cudaSuccess) {
            cudaGetLastError();
            return static_cast<EncodeTiled>(nullptr);
        }
        return reinterpret_cast<EncodeTiled>(p);
    }();
    return fn;
}

// Map of an operand with mn rows (or columns) and K: element (i, k) at
// base[i smn + k sk].  false if TMA cannot read it; *k_major says in which of the
// two orders its tiles are read in either case.
bool tc_map(CUtensorMap *map, const void *base, long smn, long sk, int mn, int K, int *k_major) {
    const bool km = sk == 1 && (smn > 1 || mn == 1), mm = !km && smn == 1;
    *k_major = !mm;
    if (!km && !mm) return false;
    const long ld = km ? smn : sk;
    const int inner = km ? K : mn, outer = km ? mn : K;
    if (ld < inner || (ld * 2) % 16 || reinterpret_cast<uintptr_t>(base) % 16 || !encode_tiled()) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)inner, (cuuint64_t)outer}, strides[1] = {(cuuint64_t)ld * 2};
    const cuuint32_t box[2] = {64, (cuuint32_t)(km ? 128 : 64)}, one[2] = {1, 1};
    return encode_tiled()(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(base), dims, strides, box, one,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// One GEMM over `splits` ranges of K (g.k_per_split is set here).
int run_gemm(GemmArgs g, int splits, int *used, cudaStream_t s) {
    CUtensorMap ma{}, mb{};
    TcArgs t;
    const bool sa = !tc_map(&ma, g.A, g.sAm, g.sAk, g.M, g.K, &t.a_kmajor),
               sb = !tc_map(&mb, g.B, g.sBn, g.sBk, g.N, g.K, &t.b_kmajor);
    const int kps = ((g.K + splits - 1) / splits + TC_K - 1) / TC_K * TC_K;
    g.k_per_split = kps;
    *used = (g.K + kps - 1) / kps;
    t.g = g;
    const dim3 grid((g.N + TC_N - 1) / TC_N, (g.M + TC_M - 1) / TC_M, *used);
    int dev = 0, sms = 0;
    TAGI_CUDA(cudaGetDevice(&dev));
    TAGI_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const bool deep = !sa && !sb && (long)grid.x * grid.y * grid.z <= sms && std::min(kps, g.K) > 3 * TC_K;
    const auto kern = sa ? (sb ? gemm_tc<true, true, 3> : gemm_tc<true, false, 3>)
                         : (sb ? gemm_tc<false, true, 3> : deep ? gemm_tc<false, false, 6> : gemm_tc<false, false, 3>);
    const size_t smem = tc_smem(deep ? 6 : 3);
    TAGI_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    TAGI_CUDA(launch_chained(kern, grid, TC_THREADS + (sa || sb ? TC_LOADERS : 0), smem, s, ma, mb, t));
    TAGI_LAUNCH_CHECK();
    return TAGI_OK;
}

// out[m][n] = sum over splits of part[s][m][n] (fixed order)
__global__ void splitk_reduce(const float *part, int splits, long mn, float *out) {
    chain_begin();
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= mn) return;
    float s = 0.f;
    for (int k = 0; k < splits; k++) s += part[(long)k * mn + i];
    out[i] = s;
}

// ---------------------------------------------------------------------------
// Patch features.  One block per row (orbital m, cell c).
// ---------------------------------------------------------------------------
constexpr int PT = 128;

__device__ __forceinline__ float block_sum_f(float v, float *sh) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) sh[wid] = v;
    __syncthreads();
    float s = 0.f;
    for (int w = 0; w < PT / 32; w++) s += sh[w];
    return s;  // every thread
}

// X[row] = [psi/s_psi, d/s_d, eps, 0...]; scale[row] = s_d; dn[row] = d/s_d (f32, for the skip term)
__global__ void __launch_bounds__(PT) patch_features(const double *__restrict__ psi, const double *__restrict__ d,
                                                     const double *__restrict__ eps, const double *__restrict__ dfloor,
                                                     int ncell, int P, long n, int ldx,
                                                     __nv_bfloat16 *__restrict__ X, float *__restrict__ scale,
                                                     float *__restrict__ dn) {
    __shared__ float sh[PT / 32];
    const int row = blockIdx.x;
    const int m = row / ncell, c = row - m * ncell;
    const double *pp = psi + (long)m * n + (long)c * P;
    const double *dd = d + (long)m * n + (long)c * P;
    float sp = 0.f, sd = 0.f;
    for (int i = threadIdx.x; i < P; i += PT) {
        const float a = (float)pp[i], b = (float)dd[i];
        sp += a * a;
        sd += b * b;
    }
    sp = block_sum_f(sp, sh);
    sd = block_sum_f(sd, sh);
    const float rp = sqrtf(sp / P) + 1e-30f;
    const float rd = fmaxf(sqrtf(sd / P), (float)dfloor[m]) + 1e-30f;
    __nv_bfloat16 *x = X + (long)row * ldx;
    for (int i = threadIdx.x; i < P; i += PT) {
        const float b = (float)dd[i] / rd;
        x[i] = __float2bfloat16_rn((float)pp[i] / rp);
        x[P + i] = __float2bfloat16_rn(b);
        dn[(long)row * P + i] = b;
    }
    for (int i = 2 * P + threadIdx.x; i < ldx; i += PT) x[i] = __float2bfloat16_rn(i == 2 * P ? (float)eps[m] : 0.f);
    if (threadIdx.x == 0) scale[row] = rd;
}

// target T = d_next / s_d (per row, from the same scale as the inputs)
__global__ void patch_target(const double *__restrict__ dnext, const float *__restrict__ scale, int ncell, int P,
                             long n, float *__restrict__ T) {
    const int row = blockIdx.x;
    const int m = row / ncell, c = row - m * ncell;
    const double *dd = dnext + (long)m * n + (long)c * P;
    const float s = scale[row];
    for (int i = threadIdx.x; i < P; i += blockDim.x) T[(long)row * P + i] = (float)dd[i] / s;
}

// Residual of the prediction and its gradient:
//   r = alpha dn + Y - T;  loss partial = sum r^2;  dY = 2 r / (rows P);  dalpha partial = sum dY dn
__global__ void __launch_bounds__(PT) mse_grad(const float *__restrict__ Y, const float *__restrict__ dn,
                                               const float *__restrict__ T, const float *__restrict__ alpha, int P,
                                               float inv_count, float *__restrict__ dY, __nv_bfloat16 *__restrict__ dY16,
                                               float *__restrict__ part) {
    __shared__ float sh[PT / 32];
    const int row = blockIdx.x;
    const float a = *alpha;
    float l = 0.f, ga = 0.f;
    for (int i = threadIdx.x; i < P; i += PT) {
        const long o = (long)row * P + i;
        const float r = a * dn[o] + Y[o] - T[o];
        const float g = 2.f * r * inv_count;
        dY[o] = g;
        dY16[o] = __float2bfloat16_rn(g);
        l += r * r;
        ga += g * dn[o];
    }
    l = block_sum_f(l, sh);
    ga = block_sum_f(ga, sh);
    if (threadIdx.x == 0) {
        part[2L * row] = l;
        part[2L * row + 1] = ga;
    }
}

// Column sums of a [rows x N] matrix (bias gradients; f32, or bf16 for the
// hidden layers' gradients): chunk b of COL_ROWS rows -> part[b][N], then the
// chunks are added in order.  A block holds 32 columns and COL_GROUPS row
// groups, whose sums are added in order: one thread per column and 1024 rows was
// a chain of loads 62 us long at 10,752 rows, 256 columns; the six calls of a step went from 157 to 124 us.
constexpr int COL_ROWS = 256, COL_GROUPS = 8;

template <typename T>
__device__ __forceinline__ float to_f(T v);
template <>
__device__ __forceinline__ float to_f<float>(float v) { return v; }
template <>
__device__ __forceinline__ float to_f<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

// Sums rows r0 + g, r0 + g + COL_GROUPS, ... of column j for this thread's group g,
// then the groups; valid in group 0.
template <typename T>
__device__ __forceinline__ float column_sum(const T *G, long r0, long r1, int N, int j) {
    __shared__ float sh[COL_GROUPS][33];
    chain_begin();
    float s = 0.f;
    if (j < N) {
#pragma unroll 8
        for (long r = r0 + threadIdx.y; r < r1; r += COL_GROUPS) s += to_f(G[r * N + j]);
    }
    sh[threadIdx.y][threadIdx.x] = s;
    __syncthreads();
    if (threadIdx.y == 0)
        for (int g = 1; g < COL_GROUPS; g++) s += sh[g][threadIdx.x];
    return s;
}

template <typename T>
__global__ void __launch_bounds__(32 * COL_GROUPS) colsum_partial(const T *G, long rows, int N,
                                                                  float *part) {
    const int j = blockIdx.y * 32 + threadIdx.x;
    const long r0 = (long)blockIdx.x * COL_ROWS;
    const float s = column_sum(G, r0, min(rows, r0 + COL_ROWS), N, j);
    if (threadIdx.y == 0 && j < N) part[(long)blockIdx.x * N + j] = s;
}

__global__ void __launch_bounds__(32 * COL_GROUPS) colsum_final(const float *part, int chunks, int N,
                                                                float *out) {
    const int j = blockIdx.x * 32 + threadIdx.x;
    const float s = column_sum(part, 0, chunks, N, j);
    if (threadIdx.y == 0 && j < N) out[j] = s;
}

// loss and dalpha from the per-row partials: thread t adds rows t, t + 256,
// ..., then a fixed tree over the threads
__global__ void __launch_bounds__(256) rows_reduce2(const float *__restrict__ part, int rows,
                                                   float *__restrict__ out) {
    __shared__ float sa[256], sb[256];
    float a = 0.f, b = 0.f;
    for (int r = threadIdx.x; r < rows; r += 256) {
        a += part[2L * r];
        b += part[2L * r + 1];
    }
    sa[threadIdx.x] = a;
    sb[threadIdx.x] = b;
    __syncthreads();
    for (int h = 128; h > 0; h >>= 1) {
        if (threadIdx.x < h) {
            sa[threadIdx.x] += sa[threadIdx.x + h];
            sb[threadIdx.x] += sb[threadIdx.x + h];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        out[0] = sa[0];
        out[1] = sb[0];
    }
}

// Adam on FP32 master weights; the BF16 copy the GEMMs read is refreshed.
__global__ void adam(float *__restrict__ w, const float *__restrict__ g, float *__restrict__ m1,
                     float *__restrict__ m2, long n, float lr, float b1, float b2, float eps, float c1, float c2,
                     __nv_bfloat16 *__restrict__ w16) {
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i];
    const float a = b1 * m1[i] + (1.f - b1) * gi;
    const float b = b2 * m2[i] + (1.f - b2) * gi * gi;
    m1[i] = a;
    m2[i] = b;
    const float v = w[i] - lr * (a / c1) / (sqrtf(b / c2) + eps);
    w[i] = v;
    if (w16) w16[i] = __float2bfloat16_rn(v);
}

// psi_next = psi + s_d (alpha dn + Y) per patch; d_next = the same increment
__global__ void patch_apply(const double *__restrict__ psi, const float *__restrict__ Y,
                            const float *__restrict__ dn, const float *__restrict__ scale,
                            const float *__restrict__ alpha, int ncell, int P, long n, double *__restrict__ psi_out,
                            double *__restrict__ d_out) {
    const int row = blockIdx.x;
    const int m = row / ncell, c = row - m * ncell;
    const long base = (long)m * n + (long)c * P;
    const float s = scale[row], a = *alpha;
    for (int i = threadIdx.x; i < P; i += blockDim.x) {
        const long o = (long)row * P + i;
        const double inc = (double)s * (double)(a * dn[o] + Y[o]);
        psi_out[base + i] = psi[base + i] + inc;
        d_out[base + i] = inc;
    }
}

__global__ void f32_to_bf16(const float *__restrict__ a, long n, __nv_bfloat16 *__restrict__ b) {
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) b[i] = __float2bfloat16_rn(a[i]);
}

}  // namespace

}  // namespace tagi

using namespace tagi;

extern "C" {

// C[M x N] = A[M x K] B[K x N] (+ epilogue), BF16 operands, FP32 accumulation;
// element (m, k) of A at A[m sAm + k sAk], (k, n) of B at B[k sBk + n sBn].
// epilogue 0: f32 C; 1: bf16 relu(C + bias); 2: bf16 C * (mask > 0);
// 3: f32 C + bias.
int tagi_mlp_gemm(const void *A, long long sAm, long long sAk, const void *B, long long sBk, long long sBn, int M,
                  int N, int K, int epilogue, float *C32, void *C16, long long ldc, const float *bias,
                  const void *mask, void *stream) {
    if (!A || !B || M <= 0 || N <= 0 || K <= 0) return set_error(TAGI_ERR_ARG, "bad GEMM arguments");
    if (epilogue < 0 || epilogue > 3) return set_error(TAGI_ERR_ARG, "epilogue %d", epilogue);
    if ((epilogue == 0 || epilogue == 3) && !C32) return set_error(TAGI_ERR_ARG, "null f32 output");
    if ((epilogue == 1 || epilogue == 2) && !C16) return set_error(TAGI_ERR_ARG, "null bf16 output");
    if ((epilogue == 1 || epilogue == 3) && !bias) return set_error(TAGI_ERR_ARG, "null bias");
    if (epilogue == 2 && !mask) return set_error(TAGI_ERR_ARG, "null mask");
    if (ldc < N) return set_error(TAGI_ERR_ARG, "ldc < N");
    GemmArgs g;
    g.A = static_cast<const __nv_bfloat16 *>(A);
    g.B = static_cast<const __nv_bfloat16 *>(B);
    g.sAm = sAm;
    g.sAk = sAk;
    g.sBk = sBk;
    g.sBn = sBn;
    g.M = M;
    g.N = N;
    g.K = K;
    g.C32 = C32;
    g.C16 = static_cast<__nv_bfloat16 *>(C16);
    g.sCm = ldc;
    g.bias = bias;
    g.mask = static_cast<const __nv_bfloat16 *>(mask);
    g.epi = epilogue;
    int used = 1;
    return run_gemm(g, 1, &used, (cudaStream_t)stream);
}

// f32 C = A B with K split over `splits` blocks; `partial` holds
// splits * M * N floats; C = sum of the partials in split order.
int tagi_mlp_gemm_splitk(const void *A, long long sAm, long long sAk, const void *B, long long sBk, long long sBn,
                         int M, int N, int K, int splits, float *partial, float *C, void *stream) {
    if (!A || !B || !partial || !C || M <= 0 || N <= 0 || K <= 0 || splits < 1)
        return set_error(TAGI_ERR_ARG, "bad split-K GEMM arguments");
    GemmArgs g;
    g.A = static_cast<const __nv_bfloat16 *>(A);
    g.B = static_cast<const __nv_bfloat16 *>(B);
    g.sAm = sAm;
    g.sAk = sAk;
    g.sBk = sBk;
    g.sBn = sBn;
    g.M = M;
    g.N = N;
    g.K = K;
    g.C32 = partial;
    g.C16 = nullptr;
    g.sCm = N;
    g.bias = nullptr;
    g.mask = nullptr;
    g.epi = EPI_F32;
    cudaStream_t s = (cudaStream_t)stream;
    TAGI_TRY(run_gemm(g, splits, &splits, s));
    const long mn = (long)M * N;
    TAGI_CUDA(launch_chained(splitk_reduce, (unsigned)((mn + 255) / 256), 256, 0, s, partial, splits, mn, C));
    TAGI_LAUNCH_CHECK();
    return TAGI_OK;
}

int tagi_mlp_check(void *stream) {
    cudaStream_t s = (cudaStream_t)stream;
    Arena tmp;
    tmp.stream = s;
    int *flag = nullptr, h = 0;
    TAGI_TRY(tmp.alloc(&flag, 1));
    launch(take_timeout, 1, 1, 0, s, flag);
    const cudaError_t e = cudaMemcpyAsync(&h, flag, sizeof(int), cudaMemcpyDeviceToHost, s);
    tmp.release();
    if (e != cudaSuccess || cudaStreamSynchronize(s) != cudaSuccess)
        return set_error(TAGI_ERR_CUDA, "GEMM status: %s", cudaGetErrorString(cudaGetLastError()));
    if (h) return set_error(TAGI_ERR_DEVICE, "a GEMM's barrier wait ran out: its tile of the result is NaN");
    return TAGI_OK;
}

int tagi_mlp_wait_probe(int tries, void *stream) {
    if (tries < 0 || tries > TC_SPINS) return set_error(TAGI_ERR_ARG, "%d tries outside [0, %d]", tries, TC_SPINS);
    launch(wait_probe, 1, 1, 0, (cudaStream_t)stream, tries);
    TAGI_LAUNCH_CHECK();
    return TAGI_OK;
}

int tagi_mlp_patch_features(const double *psi, const double *d, const double *eps, const double *dfloor,
                            int numOrbitals, int numCells, int P, long long numPoints, int ldx, void *X,
                            float *scale, float *dn, void *stream) {
    if (!psi || !d || !eps || !dfloor || !X || !scale || !dn) return set_error(TAGI_ERR_ARG, "null pointer");
    if ((long long)numCells * P != numPoints) return set_error(TAGI_ERR_ARG, "cells x P != points");
    if (ldx < 2 * P + 1) return set_error(TAGI_ERR_ARG, "ldx < 2P + 1");
    launch(patch_features, numOrbitals * numCells, PT, 0, (cudaStream_t)stream, psi, d, eps, dfloor, numCells, P,
           (long)numPoints, ldx, static_cast<__nv_bfloat16 *>(X), scale, dn);
    TAGI_LAUNCH_CHECK();
    return TAGI_OK;
}

int tagi_mlp_patch_target(const double *dnext, const float *scale, int numOrbitals, int numCells, int P,
                          long long numPoints, float *T, void *stream) {
    if (!dnext || !scale || !T) return set_error(TAGI_ERR_ARG, "null pointer");
    launch(patch_target, numOrbitals * numCells, PT, 0, (cudaStream_t)stream, dnext, scale, numCells, P,
           (long)numPoints, T);
    TAGI_LAUNCH_CHECK();
    return TAGI_OK;
}

int tagi_mlp_mse_grad(const float *Y, const float *dn, const float *T, const float *alpha, int rows, int P,
                      float *dY, void *dY16, float *part, float *lossAndDalpha, void *stream) {
    if (!Y || !dn || !T || !alpha || !dY || !dY16 || !part || !lossAndDalpha)
        return set_error(TAGI_ERR_ARG, "null pointer");
    cudaStream_t s = (cudaStream_t)stream;
    launch(mse_grad, rows, PT, 0, s, Y, dn, T, alpha, P, 1.f / ((float)rows * (float)P), dY,
           static_cast<__nv_bfloat16 *>(dY16), part);
    launch(rows_reduce2, 1, 256, 0, s, part, rows, lossAndDalpha);
    TAGI_LAUNCH_CHECK();
    return TAGI_OK;
}

long long tagi_mlp_colsum_workspace(long long rows, int N) {
    return ((rows + COL_ROWS - 1) / COL_ROWS) * (long long)N;
}

int tagi_mlp_colsum(const void *G, int isBf16, long long rows, int N, float *out, float *work, long long workFloats,
                    void *stream) {
    if (!G || !out || !work || rows <= 0 || N <= 0) return set_error(TAGI_ERR_ARG, "bad column-sum arguments");
    if (workFloats < tagi_mlp_colsum_workspace(rows, N)) return set_error(TAGI_ERR_ARG, "workspace too small");
    cudaStream_t s = (cudaStream_t)stream;
    const int chunks = (int)((rows + COL_ROWS - 1) / COL_ROWS);
    const dim3 g(chunks, (N + 31) / 32), t(32, COL_GROUPS);
    if (isBf16)
        TAGI_CUDA(launch_chained(colsum_partial<__nv_bfloat16>, g, t, 0, s, static_cast<const __nv_bfloat16 *>(G),
                                 (long)rows, N, work));
    else
        TAGI_CUDA(launch_chained(colsum_partial<float>, g, t, 0, s, static_cast<const float *>(G), (long)rows, N, work));
    TAGI_CUDA(launch_chained(colsum_final, (N + 31) / 32, t, 0, s, work, chunks, N, out));
    TAGI_LAUNCH_CHECK();
    return TAGI_OK;
}

int tagi_mlp_adam(float *w, const float *g, float *m1, float *m2, long long n, float lr, float beta1, float beta2,
                  float epsilon, int step, void *w16, void *stream) {
    if (!w || !g || !m1 || !m2 || n <= 0 || step < 1) return set_error(TAGI_ERR_ARG, "bad Adam arguments");
    const float c1 = 1.f - powf(beta1, (float)step), c2 = 1.f - powf(beta2, (float)step);
    launch(adam, (unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream, w, g, m1, m2, (long)n, lr, beta1, beta2,
           epsilon, c1, c2, static_cast<__nv_bfloat16 *>(w16));
    TAGI_LAUNCH_CHECK();
    return TAGI_OK;
}

int tagi_mlp_patch_apply(const double *psi, const float *Y, const float *dn, const float *scale, const float *alpha,
                         int numOrbitals, int numCells, int P, long long numPoints, double *psiOut, double *dOut,
                         void *stream) {
    if (!psi || !Y || !dn || !scale || !alpha || !psiOut || !dOut) return set_error(TAGI_ERR_ARG, "null pointer");
    launch(patch_apply, numOrbitals * numCells, PT, 0, (cudaStream_t)stream, psi, Y, dn, scale, alpha, numCells, P,
           (long)numPoints, psiOut, dOut);
    TAGI_LAUNCH_CHECK();
    return TAGI_OK;
}

int tagi_mlp_to_bf16(const float *a, long long n, void *b, void *stream) {
    if (!a || !b || n <= 0) return set_error(TAGI_ERR_ARG, "bad arguments");
    launch(f32_to_bf16, (unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream, a, (long)n,
           static_cast<__nv_bfloat16 *>(b));
    TAGI_LAUNCH_CHECK();
    return TAGI_OK;
}

}  // extern "C"
