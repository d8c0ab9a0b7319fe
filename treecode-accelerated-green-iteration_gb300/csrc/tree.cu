// Subsystem (a): source tree, target batches and interaction lists, on device.
//
// Rules (project-defined; BaryTree's own rules are not part of the reference,
// see 3D-GreenIteration/src/utilities/BaryTreeInterface.py:52-83):
//  * 63-bit Morton codes on the cubic box of the points' bounding box,
//    21 bits per axis, x above y above z in each 3-bit digit; stable sort.
//  * compressed octree: a node with more than `leaf` points splits at the
//    highest Morton digit in which its first and last codes differ; children
//    are the non-empty runs of that digit (2..8), numbered breadth first.
//  * tight FP64 bounding box per node; radius = half the box diagonal.
//  * batches = target-tree leaves in Morton order.
//  * per batch, pre-order DFS of the source tree:
//      (rB + rC) < theta * |cB - cC|  and  count > sizeCheck * (n+1)^3 -> far
//      (rB + rC) < theta * |cB - cC|  otherwise                       -> near
//      leaf                                                            -> near
//      else children in digit order.
// Every FP64 operation that feeds a decision uses an explicitly rounded
// intrinsic, so the lists equal the CPU oracle's integer for integer.
#include "tagi_internal.h"

#include <algorithm>
#include <numeric>

namespace tagi {

namespace {

__device__ __forceinline__ double dmax(double a, double b) { return a > b ? a : b; }
// FP64 comparisons go through the FP64 pipe (1/64 of the integer rate): smallest
// and largest coordinates are taken on the bit patterns, mapped to integers of the
// same order (-0 below +0).
__device__ __forceinline__ long long ordered(double x) {
    const long long v = __double_as_longlong(x);
    return v ^ ((v >> 63) & 0x7fffffffffffffffLL);
}
__device__ __forceinline__ double from_ordered(long long v) {
    return __longlong_as_double(v ^ ((v >> 63) & 0x7fffffffffffffffLL));
}
__device__ __forceinline__ void warp_minmax(long long (&l)[3], long long (&h)[3]) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int d = 0; d < 3; d++) {
            l[d] = min(l[d], __shfl_xor_sync(0xffffffffu, l[d], o));
            h[d] = max(h[d], __shfl_xor_sync(0xffffffffu, h[d], o));
        }
}

__global__ void bbox_partial(const double *__restrict__ x, const double *__restrict__ y,
                             const double *__restrict__ z, int n, long long *__restrict__ part) {
    long long l[3], h[3];
    l[0] = h[0] = ordered(x[0]);
    l[1] = h[1] = ordered(y[0]);
    l[2] = h[2] = ordered(z[0]);
    for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (long)gridDim.x * blockDim.x) {
        const long long p[3] = {ordered(x[i]), ordered(y[i]), ordered(z[i])};
#pragma unroll
        for (int d = 0; d < 3; d++) {
            l[d] = min(l[d], p[d]);
            h[d] = max(h[d], p[d]);
        }
    }
    warp_minmax(l, h);
    __shared__ long long sl[32][6];
    int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0)
        for (int d = 0; d < 3; d++) {
            sl[wid][d] = l[d];
            sl[wid][3 + d] = h[d];
        }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < (int)(blockDim.x >> 5); w++)
            for (int d = 0; d < 3; d++) {
                sl[0][d] = min(sl[0][d], sl[w][d]);
                sl[0][3 + d] = max(sl[0][3 + d], sl[w][3 + d]);
            }
        for (int d = 0; d < 6; d++) part[blockIdx.x * 6 + d] = sl[0][d];
    }
}

// params[0..2] = lower corner, params[3] = 2^21 / cube edge.  One block
// reduces the per-block partials (min/max are exact in any order).
__global__ void __launch_bounds__(256) bbox_final(const long long *part, int nb,
                                                  double *params) {
    chain_begin();
    long long ol[3] = {part[0], part[1], part[2]}, oh[3] = {part[3], part[4], part[5]};
    for (int b = threadIdx.x; b < nb; b += blockDim.x)
        for (int d = 0; d < 3; d++) {
            ol[d] = min(ol[d], part[b * 6 + d]);
            oh[d] = max(oh[d], part[b * 6 + 3 + d]);
        }
    warp_minmax(ol, oh);
    __shared__ long long sl[8][6];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0)
        for (int d = 0; d < 3; d++) {
            sl[wid][d] = ol[d];
            sl[wid][3 + d] = oh[d];
        }
    __syncthreads();
    if (threadIdx.x != 0) return;
    double l[3], h[3];
    for (int d = 0; d < 3; d++) {
        for (int w = 1; w < (int)(blockDim.x >> 5); w++) {
            ol[d] = min(ol[d], sl[w][d]);
            oh[d] = max(oh[d], sl[w][3 + d]);
        }
        l[d] = from_ordered(ol[d]);
        h[d] = from_ordered(oh[d]);
    }
    double ext = __dsub_rn(h[0], l[0]);
    if (__dsub_rn(h[1], l[1]) > ext) ext = __dsub_rn(h[1], l[1]);
    if (__dsub_rn(h[2], l[2]) > ext) ext = __dsub_rn(h[2], l[2]);
    if (!(ext > 0.0)) ext = 1.0;
    params[0] = l[0];
    params[1] = l[1];
    params[2] = l[2];
    params[3] = __ddiv_rn(2097152.0, ext);
}

__device__ __forceinline__ uint64_t spread21(uint32_t v) {
    uint64_t r = 0;
#pragma unroll
    for (int b = 0; b < 21; b++) r |= (uint64_t)((v >> b) & 1u) << (3 * b);
    return r;
}

__device__ __forceinline__ uint32_t quantize(double p, double lo, double scale) {
    double s = __dmul_rn(__dsub_rn(p, lo), scale);
    uint32_t v = __double2uint_rz(s);
    return v > 2097151u ? 2097151u : v;
}

__global__ void morton_codes(const double *x, const double *y,
                             const double *z, int n,
                             const double *params, uint64_t *codes,
                             int *idx) {
    chain_begin();
    long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double sc = params[3];
    uint32_t qx = quantize(x[i], params[0], sc);
    uint32_t qy = quantize(y[i], params[1], sc);
    uint32_t qz = quantize(z[i], params[2], sc);
    codes[i] = (spread21(qx) << 2) | (spread21(qy) << 1) | spread21(qz);
    idx[i] = (int)i;
}

__global__ void gather3(const double *x, const double *y,
                        const double *z, const int *perm, int n,
                        double *xs, double *ys,
                        double *zs) {
    chain_begin();
    long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int o = perm[i];
    xs[i] = x[o];
    ys[i] = y[o];
    zs[i] = z[o];
}

// First index in [lo, hi) whose code >> sh exceeds key (codes are sorted).
__device__ __forceinline__ int run_end(const uint64_t *__restrict__ codes, int lo, int hi,
                                       uint64_t key, int sh) {
    while (lo < hi) {
        int mid = lo + ((hi - lo) >> 1);
        if ((codes[mid] >> sh) > key) hi = mid;
        else lo = mid + 1;
    }
    return lo;
}

__device__ __forceinline__ int split_shift(const uint64_t *codes, int b, int e) {
    uint64_t x = codes[b] ^ codes[e - 1];
    if (x == 0) return -1;
    int hb = 63 - __clzll((long long)x);
    return 3 * (hb / 3);
}

__global__ void count_children(const uint64_t *__restrict__ codes, const int *__restrict__ begin,
                               const int *__restrict__ end, int ls, int le, int leaf,
                               int *__restrict__ cc) {
    int v = ls + blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= le) return;
    int b = begin[v], e = end[v];
    int c = 0;
    if (e - b > leaf) {
        int sh = split_shift(codes, b, e);
        if (sh >= 0) {
            int pos = b;
            while (pos < e) {
                pos = run_end(codes, pos, e, codes[pos] >> sh, sh);
                c++;
            }
        }
    }
    cc[v - ls] = c;
}

__global__ void fill_children(const uint64_t *__restrict__ codes, int *__restrict__ begin,
                              int *__restrict__ end, int *__restrict__ parent,
                              int *__restrict__ first_child, int *__restrict__ nchild, int ls,
                              int le, const int *__restrict__ cc, const int *__restrict__ off) {
    int v = ls + blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= le) return;
    int c = cc[v - ls];
    nchild[v] = c;
    if (c == 0) {
        first_child[v] = -1;
        return;
    }
    int first = le + off[v - ls];
    first_child[v] = first;
    int b = begin[v], e = end[v];
    int sh = split_shift(codes, b, e);
    int pos = b, k = 0;
    while (pos < e) {
        int nx = run_end(codes, pos, e, codes[pos] >> sh, sh);
        begin[first + k] = pos;
        end[first + k] = nx;
        parent[first + k] = v;
        pos = nx;
        k++;
    }
}

// Node header on the device: [0] nodes, [1] levels, [2 + l] first node of level l
// (and, after the last level, the node count).
constexpr int MAX_LEVELS = 23;   // 21 digits split at most
constexpr int HDR = MAX_LEVELS + 3;

// The whole octree by one block, a level at a time: a group of threads per node finds
// the starts of its eight digits, so a round of nodes is one search deep, and
// nothing waits for the host between levels.  A level of up to 32 nodes gives four
// threads to a digit, which cut its range in five at a time (a chain of 7 loads
// instead of 16 at 44,000 points), a wider one a thread: binary search, 128 nodes a
// round.  44,000 points, leaves of 1834: 33 -> 25 us.  Meshes have a few
// thousand nodes: 1.5M points, leaves of 2000: 8 levels, count + fill + scan
// launches and a synchronisation each, 1.35 -> 0.78 ms for the tree and its sort.  Above
// SMALL_TREE leaves' worth of points one launch per level is quicker.
constexpr int SMALL_TREE = 4096;
constexpr int BUILD_THREADS = 1024;
__global__ void __launch_bounds__(BUILD_THREADS) build_nodes(const uint64_t *codes, int n, int leaf,
                                                             int *begin, int *end,
                                                             int *parent, int *first_child,
                                                             int *nchild, int *hdr) {
    __shared__ int s_cnt[BUILD_THREADS / 32];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    chain_begin();
    if (tid == 0) {
        begin[0] = 0;
        end[0] = n;
        parent[0] = -1;
    }
    __syncthreads();
    int ls = 0, le = 1, level = 0;
    for (;; level++) {
        if (tid == 0) hdr[2 + level] = ls;
        int next = le;
        const int gb = le - ls <= BUILD_THREADS / 32 ? 2 : 0, probes = 1 << gb;   // threads per digit
        const int digit = (tid >> gb) & 7, q = tid & (probes - 1);
        for (int base = ls; base < le; base += BUILD_THREADS >> (3 + gb)) {
            const int v = base + (tid >> (3 + gb));
            int b = 0, e = 0, sh = -1, lo = 0;
            if (v < le) {
                b = begin[v];
                e = end[v];
                if (e - b > leaf) sh = split_shift(codes, b, e);
            }
            if (sh >= 0) {   // first index in [b, e) whose digit is >= this thread's
                const uint64_t key = ((codes[b] >> (sh + 3)) << 3) | (uint64_t)digit;
                int hi = e;
                lo = b;
                if (gb == 0) {
                    while (lo < hi) {
                        const int mid = lo + ((hi - lo) >> 1);
                        if ((codes[mid] >> sh) >= key) hi = mid;
                        else lo = mid + 1;
                    }
                } else {
                    const unsigned group = 0xfu << (lane & 28);
                    while (lo < hi) {
                        const int w = hi - lo, mid = lo + (int)((long)w * (q + 1) / 5);
                        const unsigned below = __ballot_sync(group, (codes[mid] >> sh) < key) & group;
                        const int c = __popc(below);   // the first c probes lie before the digit
                        const int left = __shfl_sync(group, mid, (lane & 28) + max(c - 1, 0));
                        const int right = __shfl_sync(group, mid, (lane & 28) + min(c, 3));
                        if (c > 0) lo = left + 1;
                        if (c < 4) hi = right;
                    }
                }
            }
            int to = __shfl_down_sync(0xffffffffu, lo, probes, 8 << gb);
            if (digit == 7) to = e;
            const bool child = sh >= 0 && to > lo && q == 0;
            const unsigned m = __ballot_sync(0xffffffffu, child);
            __syncthreads();   // s_cnt of the previous round is no longer read
            if (lane == 0) s_cnt[wid] = __popc(m);
            __syncthreads();
            int before = 0, all = 0;
            for (int w = 0; w < BUILD_THREADS / 32; w++) {
                if (w < wid) before += s_cnt[w];
                all += s_cnt[w];
            }
            const int at = next + before + __popc(m & ((1u << lane) - 1u));
            if (child) {
                begin[at] = lo;
                end[at] = to;
                parent[at] = v;
            }
            if (digit == 0 && q == 0 && v < le) {
                const int c = __popc((m >> lane) & (gb ? 0xffffffffu : 0xffu));
                nchild[v] = c;
                first_child[v] = c ? at : -1;
            }
            next += all;
        }
        __syncthreads();   // the new level's begin, end are written
        if (next == le) break;
        ls = le;
        le = next;
    }
    if (tid == 0) {
        hdr[3 + level] = le;
        hdr[0] = le;
        hdr[1] = level + 1;
    }
}

__global__ void write_header(int *hdr, int nnodes) { hdr[0] = nnodes; }

// Boxes of all nodes in one launch, with the nodes and leaves of each subtree: a
// block does a leaf, and the first warp of the one that finishes a node's last child
// goes on with the node.  The chain of the climb holds only what the parent needs;
// centers and radii (FP64) follow in preorder.  44,000 points, leaves of 1834, a warp
// per leaf and all of a node's values in the climb before: 48 -> 15 us.  1M points in 214,094
// leaves of 16: 1.2 of the plan's 27.6 ms.
constexpr int BOX_THREADS = 128;
__global__ void __launch_bounds__(BOX_THREADS) node_boxes(const int *hdr, const int *begin,
                                                          const int *end, const int *parent,
                                                          const int *first_child,
                                                          const int *nchild, const double *x,
                                                          const double *y, const double *z,
                                                          long long *box, int *size, int *leaves, int *done) {
    __shared__ long long s_box[BOX_THREADS / 32][6];
    chain_begin();
    const int nn = hdr[0], tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const long long top = ordered(INFINITY), bottom = ordered(-INFINITY);
    for (int w = blockIdx.x; w < nn; w += gridDim.x) {
        if (nchild[w]) continue;
        long long l[3] = {top, top, top}, h[3] = {bottom, bottom, bottom};
        const int e = end[w];
#pragma unroll 4
        for (int i = begin[w] + tid; i < e; i += BOX_THREADS) {
            const long long p[3] = {ordered(x[i]), ordered(y[i]), ordered(z[i])};
#pragma unroll
            for (int d = 0; d < 3; d++) {
                l[d] = min(l[d], p[d]);
                h[d] = max(h[d], p[d]);
            }
        }
        warp_minmax(l, h);
        __syncthreads();   // the previous leaf's corners are no longer read
        if (lane == 0)
#pragma unroll
            for (int d = 0; d < 3; d++) {
                s_box[wid][d] = l[d];
                s_box[wid][3 + d] = h[d];
            }
        __syncthreads();
        if (wid) continue;
        const bool part = lane < BOX_THREADS / 32;
#pragma unroll
        for (int d = 0; d < 3; d++) {
            l[d] = part ? s_box[lane][d] : top;
            h[d] = part ? s_box[lane][3 + d] : bottom;
        }
        int sz = 0, lv = 0;   // of the children
        for (int v = w;;) {
            const int pv = parent[v];
            warp_minmax(l, h);
            sz = __reduce_add_sync(0xffffffffu, sz);
            lv = __reduce_add_sync(0xffffffffu, lv);
            int last = 0;
            if (lane == 0) {
#pragma unroll
                for (int d = 0; d < 3; d++) {
                    __stcg(box + 6L * v + d, l[d]);
                    __stcg(box + 6L * v + 3 + d, h[d]);
                }
                __stcg(size + v, sz + 1);
                __stcg(leaves + v, v == w ? 1 : lv);
                if (pv >= 0) {
                    __threadfence();
                    last = atomicAdd(done + pv, 1) == nchild[pv] - 1;
                    __threadfence();
                }
            }
            if (!__shfl_sync(0xffffffffu, last, 0)) break;
            __syncwarp();   // the other lanes' reads come after lane 0's fence
            v = pv;
            const int c = first_child[v] + lane;
            const bool has = lane < nchild[v];
#pragma unroll
            for (int d = 0; d < 3; d++) {
                l[d] = has ? __ldcg(box + 6L * c + d) : top;
                h[d] = has ? __ldcg(box + 6L * c + 3 + d) : bottom;
            }
            sz = has ? __ldcg(size + c) : 0;
            lv = has ? __ldcg(leaves + c) : 0;
        }
    }
}

// Each node's center, half edges and radius; its place in pre-order (children in digit
// order) and each leaf's among the leaves, from the subtrees passed on the way to the
// root.
__global__ void preorder(const int *hdr, const int *begin, const int *end,
                         const int *parent, const int *first_child,
                         const int *nchild, const long long *box,
                         double *center, double *half, double *radius,
                         const int *size,
                         const int *leaves, PreNode *pre, int *leaf_node,
                         int *nleaves) {
    chain_begin();
    const int nn = hdr[0];
    for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < nn; v += gridDim.x * blockDim.x) {
        double cc[3], hh[3];
#pragma unroll
        for (int d = 0; d < 3; d++) {
            const double lo = from_ordered(box[6L * v + d]), hi = from_ordered(box[6L * v + 3 + d]);
            center[3L * v + d] = cc[d] = __dmul_rn(__dadd_rn(lo, hi), 0.5);
            half[3L * v + d] = hh[d] = __dmul_rn(__dsub_rn(hi, lo), 0.5);
        }
        double s = __dmul_rn(hh[0], hh[0]);
        s = __dadd_rn(s, __dmul_rn(hh[1], hh[1]));
        s = __dadd_rn(s, __dmul_rn(hh[2], hh[2]));
        radius[v] = s = __dsqrt_rn(s);
        int pos = 0, rank = 0;
        for (int c = v; c != 0;) {
            const int p = parent[c];
            pos++;
            for (int k = first_child[p]; k < c; k++) {
                pos += size[k];
                rank += leaves[k];
            }
            c = p;
        }
        PreNode q;
        q.x = cc[0];
        q.y = cc[1];
        q.z = cc[2];
        q.r = s;
        q.node = v;
        q.stop = pos + size[v];
        q.count = end[v] - begin[v];
        q.leaf = nchild[v] == 0;
        pre[pos] = q;
        if (q.leaf) leaf_node[rank] = v;
        if (v == 0) *nleaves = leaves[0];
    }
}

__global__ void init_root(int *begin, int *end, int *parent, int n) {
    begin[0] = 0;
    end[0] = n;
    parent[0] = -1;
}

}  // namespace

int build_tree(TreeBuild &w, Tree &t, const double *x, const double *y, const double *z, int n, int leaf, Arena &ar,
               cudaStream_t s) {
    t.n = n;
    Arena &tmp = w.tmp;
    tmp.stream = s;
    int rc = TAGI_OK;
    do {
        const int nbb = std::min(1024, (n + 255) / 256);
        long long *part = nullptr;
        double *params = nullptr;
        if ((rc = tmp.alloc(&part, 6L * nbb))) break;
        if ((rc = tmp.alloc(&params, 4))) break;
        launch(bbox_partial, nbb, 256, 0, s, x, y, z, n, part);
        if (launch_chained(bbox_final, 1, 256, 0, s, part, nbb, params) != cudaSuccess) {
            rc = set_error(TAGI_ERR_CUDA, "bounding box launch");
            break;
        }
        if ((rc = ar.alloc(&t.codes, n))) break;
        if ((rc = ar.alloc(&t.perm, n))) break;
        uint64_t *codes = nullptr;   // in the caller's order
        int *idx = nullptr;
        if ((rc = tmp.alloc(&codes, n)) || (rc = tmp.alloc(&idx, n))) break;
        if (launch_chained(morton_codes, (n + 255) / 256, 256, 0, s, x, y, z, n, params, codes, idx) != cudaSuccess) { rc = set_error(TAGI_ERR_CUDA, "morton launch"); break; }
        if ((rc = radix_sort_u64(codes, idx, t.codes, t.perm, n, 63, tmp, s))) break;
        if ((rc = ar.alloc(&t.x, n)) || (rc = ar.alloc(&t.y, n)) || (rc = ar.alloc(&t.z, n))) break;
        if (launch_chained(gather3, (n + 255) / 256, 256, 0, s, x, y, z, t.perm, n, t.x, t.y, t.z) != cudaSuccess) {
            rc = set_error(TAGI_ERR_CUDA, "gather launch");
            break;
        }

        // internal nodes hold more than leaf points, n / leaf of them per level at most
        const bool small = w.small = n / leaf <= SMALL_TREE;
        const long cap = std::min(2L * n + 1, small ? 8L * 21 * (n / leaf) + 9 : 2L * n + 1);
        if ((rc = ar.alloc(&t.begin, cap)) || (rc = ar.alloc(&t.end, cap)) ||
            (rc = ar.alloc(&t.parent, cap)) || (rc = ar.alloc(&t.first_child, cap)) ||
            (rc = ar.alloc(&t.nchild, cap)))
            break;
        int *hdr = nullptr, *nleaves = nullptr;
        if ((rc = tmp.alloc(&hdr, HDR + 1))) break;
        w.hdr = hdr;
        nleaves = hdr + HDR;
        t.level_start.assign(1, 0);
        if (small) {
            if (launch_chained(build_nodes, 1, BUILD_THREADS, 0, s, t.codes, n, leaf, t.begin, t.end, t.parent,
                               t.first_child, t.nchild, hdr) != cudaSuccess) {
                rc = set_error(TAGI_ERR_CUDA, "tree launch");
                break;
            }
        } else {
            int *cc = nullptr, *off = nullptr, *total = nullptr;
            if ((rc = tmp.alloc(&cc, cap)) || (rc = tmp.alloc(&off, cap)) || (rc = tmp.alloc(&total, 1)))
                break;
            launch(init_root, 1, 1, 0, s, t.begin, t.end, t.parent, n);
            int ls = 0, le = 1;
            while (ls < le) {
                int m = le - ls;
                launch(count_children, (m + 127) / 128, 128, 0, s, t.codes, t.begin, t.end, ls, le, leaf, cc);
                if ((rc = exclusive_scan(cc, off, m, total, tmp, s))) break;
                launch(fill_children, (m + 127) / 128, 128, 0, s, t.codes, t.begin, t.end, t.parent, t.first_child,
                       t.nchild, ls, le, cc, off);
                int h_total = 0;
                if (cudaMemcpyAsync(&h_total, total, sizeof(int), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
                    cudaStreamSynchronize(s) != cudaSuccess) {
                    rc = set_error(TAGI_ERR_CUDA, "tree level build: %s", cudaGetErrorString(cudaGetLastError()));
                    break;
                }
                if (le + (long)h_total > cap) { rc = set_error(TAGI_ERR_DEVICE, "tree node capacity exceeded"); break; }
                ls = le;
                le += h_total;
                t.level_start.push_back(ls);
            }
            if (rc) break;
            t.nnodes = le;
            launch(write_header, 1, 1, 0, s, hdr, t.nnodes);
        }
        const long nodes = small ? cap : t.nnodes;
        long long *box = nullptr;   // lower and upper corners, ordered()
        int *work = nullptr;
        if ((rc = tmp.alloc(&box, 6 * nodes)) || (rc = tmp.alloc(&work, 3 * nodes)) ||
            (rc = ar.alloc(&t.center, 3 * nodes)) || (rc = ar.alloc(&t.half, 3 * nodes)) ||
            (rc = ar.alloc(&t.radius, nodes)) || (rc = ar.alloc(&t.pre, nodes)) || (rc = ar.alloc(&t.leaf_node, nodes)))
            break;
        int *size = work, *leaves = work + nodes, *done = work + 2 * nodes;
        if (cudaMemsetAsync(done, 0, sizeof(int) * nodes, s) != cudaSuccess) {
            rc = set_error(TAGI_ERR_CUDA, "tree memset failed");
            break;
        }
        const unsigned bw = (unsigned)std::min(GPU_SMS * 16, nodes), bt = (unsigned)std::min(GPU_SMS * 8, (nodes + 127) / 128);
        if (launch_chained(node_boxes, bw, BOX_THREADS, 0, s, hdr, t.begin, t.end, t.parent, t.first_child, t.nchild, t.x,
                           t.y, t.z, box, size, leaves, done) != cudaSuccess ||
            launch_chained(preorder, bt, 128, 0, s, hdr, t.begin, t.end, t.parent, t.first_child, t.nchild, box, t.center,
                           t.half, t.radius, size, leaves, t.pre, t.leaf_node, nleaves) != cudaSuccess) {
            rc = set_error(TAGI_ERR_CUDA, "node box launch");
            break;
        }
        if (cudaGetLastError() != cudaSuccess) { rc = set_error(TAGI_ERR_CUDA, "node box launch"); break; }
    } while (0);
    return rc;
}

int finish_trees(TreeBuild *const *w, Tree *const *t, int count, cudaStream_t s) {
    int h[2][HDR + 1] = {};
    int rc = TAGI_OK;
    for (int k = 0; k < count && !rc; k++)
        if (cudaMemcpyAsync(h[k], w[k]->hdr, sizeof(h[k]), cudaMemcpyDeviceToHost, s) != cudaSuccess)
            rc = set_error(TAGI_ERR_CUDA, "tree build: %s", cudaGetErrorString(cudaGetLastError()));
    if (!rc && cudaStreamSynchronize(s) != cudaSuccess)
        rc = set_error(TAGI_ERR_CUDA, "tree build: %s", cudaGetErrorString(cudaGetLastError()));
    for (int k = 0; k < count; k++) {
        w[k]->tmp.release();
        if (rc) continue;
        Tree &q = *t[k];
        q.nleaves = h[k][HDR];
        if (w[k]->small) {
            q.nnodes = h[k][0];
            q.level_start.assign(h[k] + 2, h[k] + 3 + h[k][1]);
        }
        q.nlevels = (int)q.level_start.size() - 1;
    }
    return rc;
}

// ---------------------------------------------------------------------------
// Batches, lists, slots, upward-pass items.
// ---------------------------------------------------------------------------
namespace {

struct TravArgs {
    int nbatch, nn;
    const int *batch_node;
    const double *tc, *tr;                 // target centers / radii
    const PreNode *pre;                    // source nodes in pre-order
    double theta, thresh;
    int *near_cnt, *far_cnt;
    const int *near_off, *far_off;
    int *near_list, *far_list;
    int *node_flag;
};

__device__ __forceinline__ bool meets_criterion(const TravArgs &a, double cbx, double cby, double cbz, double rb,
                                                const PreNode &q) {
    const double dx = __dsub_rn(cbx, q.x), dy = __dsub_rn(cby, q.y), dz = __dsub_rn(cbz, q.z);
    double d2 = __dmul_rn(dx, dx);
    d2 = __dadd_rn(d2, __dmul_rn(dy, dy));
    d2 = __dadd_rn(d2, __dmul_rn(dz, dz));
    const double dist = __dsqrt_rn(d2);
    return __dadd_rn(rb, q.r) < __dmul_rn(a.theta, dist);
}

// The depth-first walk of one batch by one warp, 32 nodes of the pre-order at a
// time: a node that meets the criterion covers its subtree (the indices up to its
// stop), and a node is visited if no node before it covers it.  One thread per
// batch with a stack took 1 ms for 2,900 batches, a chain of dependent loads.
template <bool FILL>
__global__ void __launch_bounds__(256) traverse(TravArgs a) {
    const int b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (b >= a.nbatch) return;
    const int bn = a.batch_node[b];
    const double cbx = a.tc[3L * bn], cby = a.tc[3L * bn + 1], cbz = a.tc[3L * bn + 2];
    const double rb = a.tr[bn];
    int cn = 0, cf = 0;
    int *nl = FILL ? a.near_list + a.near_off[b] : nullptr;
    int *fl = FILL ? a.far_list + a.far_off[b] : nullptr;
    int skip = 0;   // nodes below this index are covered
    for (int base = 0; base < a.nn; base = max(base + 32, skip)) {
        const int i = base + lane;
        bool mac = false, leaf = false, big = false;
        int stop = 0, node = 0;
        if (i < a.nn) {
            const PreNode q = a.pre[i];
            mac = meets_criterion(a, cbx, cby, cbz, rb, q);
            leaf = q.leaf;
            big = (double)q.count > a.thresh;
            stop = mac ? q.stop : 0;
            node = q.node;
        }
        int reach = stop;   // the furthest stop among this lane and those before it
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, reach, o);
            if (lane >= o) reach = max(reach, v);
        }
        int before = __shfl_up_sync(0xffffffffu, reach, 1);
        if (lane == 0) before = 0;
        const bool emit = i < a.nn && max(before, skip) <= i && (mac || leaf);
        const bool far = emit && mac && big;
        const unsigned mf = __ballot_sync(0xffffffffu, far), mn = __ballot_sync(0xffffffffu, emit && !far);
        if (FILL) {
            const unsigned lt = (1u << lane) - 1u;
            if (far) {
                fl[cf + __popc(mf & lt)] = node;
                a.node_flag[node] = 1;
            } else if (emit) {
                nl[cn + __popc(mn & lt)] = node;
            }
        }
        cf += __popc(mf);
        cn += __popc(mn);
        skip = max(skip, __shfl_sync(0xffffffffu, reach, 31));
    }
    if (!FILL && lane == 0) {
        a.near_cnt[b] = cn;
        a.far_cnt[b] = cf;
    }
}

// The same walk by one thread per batch, a node at a time.  Where most subtrees are small most of
// a warp's 32 nodes are covered, and many batches hide the chain of loads: 1M points, leaves of
// 16 (214,094 batches), whole plan 133.8 ms by warps, 27.6 by threads.
template <bool FILL>
__global__ void __launch_bounds__(128) traverse_many(TravArgs a) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= a.nbatch) return;
    const int bn = a.batch_node[b];
    const double cbx = a.tc[3L * bn], cby = a.tc[3L * bn + 1], cbz = a.tc[3L * bn + 2];
    const double rb = a.tr[bn];
    int cn = 0, cf = 0;
    int *nl = FILL ? a.near_list + a.near_off[b] : nullptr;
    int *fl = FILL ? a.far_list + a.far_off[b] : nullptr;
    for (int i = 0; i < a.nn;) {
        const PreNode q = a.pre[i];
        const bool mac = meets_criterion(a, cbx, cby, cbz, rb, q);
        if (mac && (double)q.count > a.thresh) {
            if (FILL) {
                fl[cf] = q.node;
                a.node_flag[q.node] = 1;
            }
            cf++;
        } else if (mac || q.leaf) {
            if (FILL) nl[cn] = q.node;
            cn++;
        }
        i = mac ? q.stop : i + 1;
    }
    if (!FILL) {
        a.near_cnt[b] = cn;
        a.far_cnt[b] = cf;
    }
}

// Batches from which on a thread walks for each.  Whole plans by warps and by threads, us: 1,474
// batches 715, 1564; 3,724 1644, 2388; 5,599 2424, 2369; 7,272 3031, 3375; 8,870 4037, 2809;
// 10,228 4809, 4990; 16,163 8014, 6250; 37,164 19227, 8590.
constexpr int MANY_BATCHES = 8192;

// Gap between the batch box (center cb, half widths hb) and a node box: the
// Euclidean distance between the closed boxes, reduced by a relative margin so
// that touching boxes give 0.
__device__ __forceinline__ double box_gap(const double *cb, const double *hb, const double *cc,
                                          const double *hc) {
    double g2 = 0.0;
#pragma unroll
    for (int d = 0; d < 3; d++) {
        double gap = fabs(cb[d] - cc[d]) - (hb[d] + hc[d]);
        gap -= 1e-12 * (fabs(cb[d]) + fabs(cc[d]) + hb[d] + hc[d]) + 1e-300;
        if (gap > 0.0) g2 += gap * gap;
    }
    return sqrt(g2);
}

// Merge consecutive near entries whose source ranges touch and whose nodes
// are of the same class: a node is CLOSE when its box lies within
// CLOSE_RANGE_FRACTION batch radii of the batch's box (touching included).
// Close ranges are stored with bit 31 of their begin set (range_is_close).
// rng_dmin = smallest node gap of the range, rounded down: a lower bound of
// every pair distance in it.  One warp per batch, 32 entries at a time; the fill
// also writes the batch's pair counts: near, close, far (clusters), and its size with bit 32 set if an
// ordinary range is too near for its distance from the origin (Plan::wide).
template <bool FILL>
__global__ void __launch_bounds__(256) merge_ranges(int nbatch, const int *__restrict__ near_off,
                                                    const int *__restrict__ near_list, const int *__restrict__ sbegin,
                                                    const int *__restrict__ send, const double *__restrict__ scenter,
                                                    const double *__restrict__ shalf,
                                                    const int *__restrict__ batch_node,
                                                    const double *__restrict__ tcenter,
                                                    const double *__restrict__ thalf,
                                                    const double *__restrict__ tradius, int *__restrict__ cnt,
                                                    const int *__restrict__ rng_off, int2 *rng, float *rng_dmin,
                                                    const int *__restrict__ tbegin, const int *__restrict__ tend,
                                                    const int *__restrict__ far_off, long long *__restrict__ costs) {
    const int b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (b >= nbatch) return;
    const int bn = batch_node[b];
    const double cb[3] = {tcenter[3L * bn], tcenter[3L * bn + 1], tcenter[3L * bn + 2]};
    const double hb[3] = {thalf[3L * bn], thalf[3L * bn + 1], thalf[3L * bn + 2]};
    const double close_gap = CLOSE_RANGE_FRACTION * tradius[bn];
    const double wide_gap = WIDE_GAP * dmax(dmax(fabs(cb[0]), fabs(cb[1])), fabs(cb[2]));
    bool wide = false;
    const int e0 = near_off[b], e1 = near_off[b + 1];
    int k = 0, prev_end = -1, prev_close = 0;   // ranges begun; the last entry's end and class
    double carry = INFINITY;                    // smallest gap of the range in progress
    long long all = 0, close_all = 0;
    for (int base = e0; base < e1; base += 32) {
        const int e = base + lane;
        const bool valid = e < e1;
        int nb = 0, ne = 0, nclose = 0;
        double gap = INFINITY;
        if (valid) {
            const int c = near_list[e];
            nb = sbegin[c];
            ne = send[c];
            const double cc[3] = {scenter[3L * c], scenter[3L * c + 1], scenter[3L * c + 2]};
            const double hc[3] = {shalf[3L * c], shalf[3L * c + 1], shalf[3L * c + 2]};
            gap = box_gap(cb, hb, cc, hc);
            nclose = gap <= close_gap;
            all += ne - nb;
            if (nclose) close_all += ne - nb;
            else wide = wide || !(gap >= wide_gap);
        }
        int pe = __shfl_up_sync(0xffffffffu, ne, 1), pc = __shfl_up_sync(0xffffffffu, nclose, 1);
        if (lane == 0) {
            pe = prev_end;
            pc = prev_close;
        }
        const bool start = valid && (e == e0 || nb != pe || nclose != pc);
        const unsigned m = __ballot_sync(0xffffffffu, start), mv = __ballot_sync(0xffffffffu, valid);
        const unsigned le = 0xffffffffu >> (31 - lane);
        if (FILL) {
            const int first = (m & le) ? 31 - __clz(m & le) : 0;   // this entry's range begins here (or earlier)
            double v = gap;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const double u = __shfl_up_sync(0xffffffffu, v, o);
                if (lane - o >= first) v = fmin(v, u);
            }
            if (!(m & le)) v = fmin(v, carry);
            const int r = rng_off[b] + k + __popc(m & le) - 1;
            if (start) rng[r].x = nb | (nclose ? (int)0x80000000u : 0);
            const unsigned after = lane == 31 ? 0u : (mv & ~m) >> (lane + 1) & 1u;   // the next entry goes on with the range
            if (valid && !after) {   // a later round writes these again if the range goes on there
                rng[r].y = ne;
                rng_dmin[r] = (float)(v * (1.0 - 1e-6));
            }
            carry = __shfl_sync(0xffffffffu, v, 31 - __clz(mv));
            __syncwarp();
        }
        prev_end = __shfl_sync(0xffffffffu, ne, 31 - __clz(mv));
        prev_close = __shfl_sync(0xffffffffu, nclose, 31 - __clz(mv));
        k += __popc(m);
    }
    if constexpr (FILL) {
        const bool any_wide = __any_sync(0xffffffffu, wide);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            all += __shfl_xor_sync(0xffffffffu, all, o);
            close_all += __shfl_xor_sync(0xffffffffu, close_all, o);
        }
        if (lane == 0) {
            const long long nt = tend[bn] - tbegin[bn];
            costs[4L * b] = nt * all;
            costs[4L * b + 1] = nt * close_all;
            costs[4L * b + 2] = nt * (long long)(far_off[b + 1] - far_off[b]);
            costs[4L * b + 3] = nt | (long long)any_wide << 32;
        }
    } else if (lane == 0) {
        cnt[b] = k;
    }
}

// Slots (far nodes in ascending node order), their proxy boxes and the upward
// pass's work items, by one block: node_slot, slot_node, geometry (node center and
// half widths; a zero width gets a small one, 1e-3 of the largest or 1, so the
// barycentric map stays finite), slot_item_off and the items of at most `chunk`
// sources.  total[0], total[1]: slots, items.
constexpr int SLOT_THREADS = 1024;
__global__ void __launch_bounds__(SLOT_THREADS) build_slots(int nn, const int *__restrict__ flag,
                                                            const int *__restrict__ sbegin, const int *__restrict__ send,
                                                            const double *__restrict__ center,
                                                            const double *__restrict__ half, int chunk,
                                                            int *__restrict__ node_slot, int *__restrict__ slot_node,
                                                            double *__restrict__ geom, int *__restrict__ slot_item_off,
                                                            int *__restrict__ item_slot, int *__restrict__ item_begin,
                                                            int *__restrict__ item_end, int *__restrict__ total) {
    __shared__ long long s_sum[SLOT_THREADS / 32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    long long carry = 0;   // slots << 32 | items
    for (int base = 0; base < nn; base += SLOT_THREADS) {
        const int v = base + threadIdx.x;
        const bool is = v < nn && flag[v];
        int b = 0, e = 0;
        if (is) {
            b = sbegin[v];
            e = send[v];
        }
        const long long mine = is ? (1LL << 32) + (e - b + chunk - 1) / chunk : 0;
        long long incl = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const long long u = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += u;
        }
        __syncthreads();   // the previous round's sums are no longer read
        if (lane == 31) s_sum[wid] = incl;
        __syncthreads();
        long long at = carry + incl - mine;
        for (int w = 0; w < SLOT_THREADS / 32; w++) {
            if (w < wid) at += s_sum[w];
            carry += s_sum[w];
        }
        if (v < nn) node_slot[v] = is ? (int)(at >> 32) : -1;
        if (is) {
            const int sl = (int)(at >> 32);
            int k = (int)(at & 0xffffffffLL);
            slot_node[sl] = v;
            slot_item_off[sl] = k;
            const double h[3] = {half[3L * v], half[3L * v + 1], half[3L * v + 2]};
            const double hm = dmax(dmax(h[0], h[1]), h[2]);
#pragma unroll
            for (int d = 0; d < 3; d++) {
                geom[6L * sl + d] = center[3L * v + d];
                double u = h[d];
                if (!(u > 0.0)) u = hm > 0.0 ? hm * 1.0e-3 : 1.0;
                geom[6L * sl + 3 + d] = u;
            }
            for (int p = b; p < e; p += chunk, k++) {
                item_slot[k] = sl;
                item_begin[k] = p;
                item_end[k] = min(p + chunk, e);
            }
        }
    }
    if (threadIdx.x == 0) {
        total[0] = (int)(carry >> 32);
        total[1] = (int)(carry & 0xffffffffLL);
        slot_item_off[carry >> 32] = total[1];
    }
}

// Sources per upward-pass item: small meshes need items for every SM, large ones few partial
// sums (an item has (n+1)^3 of them per charge vector).  Upward pass, us, degree 7, 256, 512, 1024,
// 2048 sources per item: one charge vector 10k points 24, 35, 55, 82; 30k 30, 40, 58, 101; 60k 53,
// 49, 64, 103; 130k 107, 95, 97, 117; 260k 206, 169, 163, 171; 1M 929, 708, 621, 599; FP64 30k 198,
// 317, 324, 635; eight vectors 30k 128, 116, 114, 168; 130k 652, 521, 458, 438; 1M 6374, 4952,
// 4254, 3942.
int p2m_chunk(int n) { return n <= 65536 ? 256 : (n <= 262144 ? 512 : 2048); }

}  // namespace

int build_lists(Plan &p, cudaStream_t s) {
    Arena tmp;
    tmp.stream = s;
    Arena &ar = p.arena;
    int rc = TAGI_OK;
    do {
        const int nns = p.src.nnodes;
        p.nbatch = p.tgt.nleaves;
        p.batch_node = p.tgt.leaf_node;
        const int nb = p.nbatch;
        int *ncnt = nullptr, *fcnt = nullptr;
        if ((rc = tmp.alloc(&ncnt, nb)) || (rc = tmp.alloc(&fcnt, nb))) break;
        if ((rc = ar.alloc(&p.near_off, 2 * (nb + 1)))) break;   // both offsets: one copy brings both totals back
        p.far_off = p.near_off + nb + 1;
        int *node_flag = nullptr;
        if ((rc = tmp.alloc(&node_flag, nns))) break;
        cudaMemsetAsync(node_flag, 0, sizeof(int) * nns, s);
        TravArgs ta;
        ta.nbatch = nb;
        ta.nn = nns;
        ta.batch_node = p.batch_node;
        ta.tc = p.tgt.center;
        ta.tr = p.tgt.radius;
        ta.pre = p.src.pre;
        ta.theta = p.theta;
        ta.thresh = p.size_check * (double)p.P;
        ta.near_cnt = ncnt;
        ta.far_cnt = fcnt;
        ta.near_off = p.near_off;
        ta.far_off = p.far_off;
        ta.near_list = nullptr;
        ta.far_list = nullptr;
        ta.node_flag = node_flag;
        const unsigned bw = (unsigned)((nb + 7) / 8);   // a warp per batch
        const bool many = nb >= MANY_BATCHES;
        const unsigned bt = (unsigned)((nb + 127) / 128);
        if (many) launch(traverse_many<false>, bt, 128, 0, s, ta);
        else launch(traverse<false>, bw, 256, 0, s, ta);
        if ((rc = exclusive_scan(ncnt, p.near_off, nb, p.near_off + nb, tmp, s))) break;
        if ((rc = exclusive_scan(fcnt, p.far_off, nb, p.far_off + nb, tmp, s))) break;
        // Room that does not depend on the counts is taken while the walk runs: at most nns slots;
        // items: a slot's last chunk is partial
        const long most = nns + (long)p.src.nlevels * (p.src.n / p2m_chunk(p.src.n) + 1);
        long long *costs = nullptr;   // 4 per batch, then the range, slot and item counts
        if ((rc = ar.alloc(&p.rng_off, nb + 1)) || (rc = ar.alloc(&p.node_slot, nns)) || (rc = ar.alloc(&p.slot_node, nns)) ||
            (rc = ar.alloc(&p.slot_geom, 6L * nns)) || (rc = ar.alloc(&p.slot_item_off, nns + 1)) ||
            (rc = ar.alloc(&p.item_slot, most)) || (rc = ar.alloc(&p.item_begin, most)) ||
            (rc = ar.alloc(&p.item_end, most)) || (rc = tmp.alloc(&costs, 4L * nb + 2)))
            break;
        int totals[2] = {0, 0};
        if (cudaMemcpy2DAsync(totals, sizeof(int), p.near_off + nb, sizeof(int) * (nb + 1), sizeof(int), 2,
                              cudaMemcpyDeviceToHost, s) != cudaSuccess ||
            cudaStreamSynchronize(s) != cudaSuccess) {
            rc = set_error(TAGI_ERR_CUDA, "list build: %s", cudaGetErrorString(cudaGetLastError()));
            break;
        }
        p.near_total = totals[0];
        p.far_total = totals[1];
        // at most near_total ranges
        if ((rc = ar.alloc(&p.near_list, p.near_total)) || (rc = ar.alloc(&p.far_list, p.far_total)) ||
            (rc = ar.alloc(&p.rng, p.near_total)) || (rc = ar.alloc(&p.rng_dmin, p.near_total)))
            break;
        int *counts = reinterpret_cast<int *>(costs + 4L * nb);
        ta.near_list = p.near_list;
        ta.far_list = p.far_list;
        if (many) launch(traverse_many<true>, bt, 128, 0, s, ta);
        else launch(traverse<true>, bw, 256, 0, s, ta);
        launch(build_slots, 1, SLOT_THREADS, 0, s, nns, node_flag, p.src.begin, p.src.end, p.src.center, p.src.half,
               p2m_chunk(p.src.n), p.node_slot, p.slot_node, p.slot_geom, p.slot_item_off, p.item_slot, p.item_begin, p.item_end,
               counts + 1);
        launch(merge_ranges<false>, bw, 256, 0, s, nb, p.near_off, p.near_list, p.src.begin, p.src.end, p.src.center,
               p.src.half, p.batch_node, p.tgt.center, p.tgt.half, p.tgt.radius, ncnt, nullptr, nullptr, nullptr,
               p.tgt.begin, p.tgt.end, p.far_off, nullptr);
        if ((rc = exclusive_scan(ncnt, p.rng_off, nb, p.rng_off + nb, tmp, s))) break;
        launch(merge_ranges<true>, bw, 256, 0, s, nb, p.near_off, p.near_list, p.src.begin, p.src.end, p.src.center,
               p.src.half, p.batch_node, p.tgt.center, p.tgt.half, p.tgt.radius, nullptr, p.rng_off, p.rng,
               p.rng_dmin, p.tgt.begin, p.tgt.end, p.far_off, costs);
        // Pair counts of each batch: the field kernels' work lists go heaviest first.
        std::vector<long long> h(4L * nb + 2);
        if (cudaMemcpyAsync(counts, p.rng_off + nb, sizeof(int), cudaMemcpyDeviceToDevice, s) != cudaSuccess ||
            cudaMemcpyAsync(h.data(), costs, sizeof(long long) * h.size(), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
            cudaStreamSynchronize(s) != cudaSuccess) {
            rc = set_error(TAGI_ERR_CUDA, "list build: %s", cudaGetErrorString(cudaGetLastError()));
            break;
        }
        const int *hc = reinterpret_cast<const int *>(h.data() + 4L * nb);
        p.rng_total = hc[0];
        p.nslots = hc[1];
        p.nitems = hc[2];
        p.near_pairs = 0;
        p.near_close_pairs = 0;
        p.far_pairs = 0;
        p.max_batch = 0;
        p.cost_near.resize(nb);
        p.cost_close.resize(nb);
        p.cost_far.resize(nb);
        p.batch_size.resize(nb);
        for (int b = 0; b < nb; b++) {
            const long long *c = &h[4L * b];
            p.near_pairs += (double)c[0];
            p.near_close_pairs += (double)c[1];
            p.far_pairs += (double)c[2] * p.P;
            p.batch_size[b] = (int)(c[3] & 0xffffffffLL);
            p.wide = p.wide || c[3] >> 32;
            p.max_batch = std::max(p.max_batch, p.batch_size[b]);
            p.cost_near[b] = c[0] - c[1];
            p.cost_close[b] = c[1];
            p.cost_far[b] = c[2] * (long long)p.P;
        }
        if (cudaGetLastError() != cudaSuccess) { rc = set_error(TAGI_ERR_CUDA, "list kernels failed"); break; }
    } while (0);
    tmp.release();
    return rc;
}

}  // namespace tagi
