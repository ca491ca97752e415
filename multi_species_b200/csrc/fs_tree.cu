// Barycentric Lagrange treecode on the device (E_MQ_Treecode,
// src/FieldStructure.cpp:230-1020).
//
// Same tree, lists and moments as the reference, rebuilt every call like the
// reference does, but on the GPU:
//   k_tree_keys/sort   particles_x = fmod(x, L) (:235-247), sorted by fixed-point
//                      keys (CUB radix); k_tree_gather and k_tree_runs put points
//                      of equal keys right
//   k_build_tree       one CTA, level-synchronous midpoint bisection over the
//                      root interval [min - 0.1234, max + 0.001] (:506-632,
//                      :1032-1050): a node with n >= max_source points splits at
//                      0.5 (x0 + x1), points with x <= mid go left, children only
//                      when non-empty.  Member ranges are contiguous in sorted
//                      order, so a split is one binary search; k_heap_splits
//                      makes those of the first levels at once.
//   k_lists            a warp per leaf: the reference's tests from the root
//                      down (build_interaction_list :663-702) -- any leaf reached
//                      is near, a node is far when (r_b + r_p) / R < theta with the
//                      periodic R = min(|dxc|, L - |dxc|), else recurse -- in the
//                      same IEEE arithmetic, so far/near decisions are identical.
//   k_moments          Chebyshev-Lobatto t_k = x0 + (cos(k pi/P) + 1)/2 (x1 - x0) and
//                      M_{c,k} = sum_j lambda_j a_k(x_j) / sum_k a_k(x_j) for every
//                      node but the root (alloc_set_cluster_list :775-866): the
//                      leaves' from their points, the others' from their
//                      children's, in a fixed order.  cos(k pi/P) comes from the
//                      host C library.
//   k_far_near64       per target: far list then near list (Call_BL :904-961,
//                      Call_Ds :963-1020) in FP64.
//   k_far32 + k_near32 FP32-compensated form: far field in FP64 with a
//                      reciprocal-square-root kernel evaluation, near field as
//                      FP32 tiles of the near leaves' sources with Kahan sums.
// With many points per epsilon near and far sums go through cells instead of the
// last three kernels (csrc/fs_treecells.cu).
// The kernel of the reference treecode is sqrt(L^2+4 eps^2)/L times the direct
// sum's (:949, :1008 vs :150); both forms keep that normalisation.
#include <cub/cub.cuh>

#include <cfloat>
#include <climits>
#include <cmath>
#include <type_traits>
#include <vector>

#include "fs_tree.cuh"

namespace fsb {

namespace {


// Per-instance constants (device array of 2 x (kMaxDegree+1) doubles):
//   cheb[k] = cos(k pi / P) from the host C library, w[k] = (-1)^k (1/2 at the ends).

// signed double -> order-preserving unsigned key
__device__ __forceinline__ uint64_t order_key(double v) {
    const uint64_t b = (uint64_t)__double_as_longlong(v);
    return (b & 0x8000000000000000ull) ? ~b : (b | 0x8000000000000000ull);
}

// The points' order along x in three steps: a radix sort by fixed-point positions
// of 24 or 32 bits (half the passes of the 64-bit keys, two thirds of the bytes),
// k_tree_gather, which puts the few points of equal keys right as it fetches
// positions and charges, and k_tree_runs for long runs of equal keys that are not
// in order already.  Position and charge travel as one 16-byte record: the fetch is
// bound by its scattered sectors (121 us, two arrays 170).  The order is the one of (order_key, index).  6.3 million
// points: 455 us with the keys, 270 us less than by 64-bit keys and a fetch of charges.
constexpr int kRunMax = 32;  // longest run of equal keys that its points rank themselves in

// 24 bits up to 2^18 points (at most 1/32 of a point per key at uniform density).
inline int tree_key_bits(int n) { return n <= (1 << 18) ? 24 : 32; }

__global__ void k_tree_keys(const double* __restrict__ x, const double* __restrict__ q, int n, double L,
                            double scale, uint32_t top, uint32_t* __restrict__ keys, int* __restrict__ idx, double2* __restrict__ vq,
                            int* __restrict__ nruns) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double v = fmod(x[i], L);  // in (-L, L)
    const uint32_t k = min(__double2uint_rd((v + L) * scale), top);
    keys[i] = v != v ? (order_key(v) >> 63 ? top : 0u) : k;  // NaN last (or, by its sign, first)
    idx[i] = i;
    vq[i] = make_double2(v, q[i]);
    if (i == 0) *nruns = 0;
}

// Position and charge of every sorted point, in the order within its run.  Longer
// runs keep the radix sort's order (by index); those with points out of order are
// listed, once each (`seen`: a bit per first point, zero on entry).
__global__ void k_tree_gather(const uint32_t* __restrict__ skeys, const int* __restrict__ ord,
                              const double2* __restrict__ vq, int n, double* __restrict__ sx, double* __restrict__ lam, int* __restrict__ sidx,
                              uint32_t* __restrict__ seen, int* __restrict__ runs, int* __restrict__ nruns) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    const uint32_t k = skeys[j];
    const int id = ord[j];
    const double2 e = vq[id];
    const double v = e.x;
    int a = j, b = j + 1;
    while (a > 0 && j - a < kRunMax && skeys[a - 1] == k) --a;
    while (b < n && b - j <= kRunMax && skeys[b] == k) ++b;
    int dst = j;
    if (b - a > 1) {
        const uint64_t o = order_key(v);
        if (b - a <= kRunMax) {
            dst = a;
            for (int i = a; i < b; ++i) {
                if (i == j) continue;
                const uint64_t oi = order_key(vq[ord[i]].x);
                dst += oi < o || (oi == o && i < j);
            }
        } else if (a < j && order_key(vq[ord[j - 1]].x) > o) {
            int lo = 0, hi = j;  // the run's first point
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (skeys[mid] < k) lo = mid + 1;
                else hi = mid;
            }
            const uint32_t bit = 1u << (lo & 31);
            if (!(atomicOr(&seen[lo >> 5], bit) & bit)) runs[atomicAdd(nruns, 1)] = lo;
        }
    }
    sx[dst] = v;
    lam[dst] = e.y;
    sidx[dst] = id;
}

// Listed runs, a CTA each at a time: merge passes from runs of one, every point
// finding its place in the other half by binary search.  (Any number of points
// may share a key; the time grows as their number times its logarithm.)
__global__ void __launch_bounds__(1024) k_tree_runs(const uint32_t* __restrict__ skeys, const int* __restrict__ runs,
                                                    const int* __restrict__ nruns, const double* __restrict__ q,
                                                    int n, double* __restrict__ sx, double* __restrict__ lam,
                                                    int* __restrict__ sidx, double* __restrict__ x2,
                                                    int* __restrict__ id2) {
    const int m = *nruns;
    for (int r = blockIdx.x; r < m; r += gridDim.x) {
        const int a = runs[r];
        int e = a, hi = n;  // its end
        const uint32_t k = skeys[a];
        while (e < hi) {
            const int mid = e + ((hi - e) >> 1);
            if (skeys[mid] <= k) e = mid + 1;
            else hi = mid;
        }
        double *xs = sx, *xd = x2;
        int *is = sidx, *id = id2;
        for (long long w = 1; w < e - a; w *= 2) {
            for (int j = a + threadIdx.x; j < e; j += blockDim.x) {
                const double v = xs[j];
                const uint64_t o = order_key(v);
                const int p = is[j];
                const long long blk = (j - a) / (2 * w), mine = (j - a) / w;
                const int lo0 = (int)min(a + (mine ^ 1) * w, (long long)e);
                const int hi0 = (int)min(a + ((mine ^ 1) + 1) * w, (long long)e);
                int lo = lo0, up = hi0;
                while (lo < up) {
                    const int mid = lo + ((up - lo) >> 1);
                    const uint64_t om = order_key(xs[mid]);
                    if (om < o || (om == o && is[mid] < p)) lo = mid + 1;
                    else up = mid;
                }
                const int dst = (int)(a + blk * 2 * w) + (int)((j - a) - mine * w) + (lo - lo0);
                xd[dst] = v;
                id[dst] = p;
            }
            __syncthreads();
            double* tx = xs;
            xs = xd;
            xd = tx;
            int* ti = is;
            is = id;
            id = ti;
        }
        for (int j = a + threadIdx.x; j < e; j += blockDim.x) {
            const int p = is[j];
            const double v = xs[j];
            sx[j] = v;
            sidx[j] = p;
            lam[j] = q[p];
        }
        __syncthreads();
    }
}

__device__ __forceinline__ int upper_bound(const double* __restrict__ a, int lo, int hi, double v) {
    while (lo < hi) {
        const int mid = lo + ((hi - lo) >> 1);
        if (a[mid] <= v) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// upper_bound by kG neighbouring lanes together: each step cuts the range at kG
// places, so the chain of loads is log of the range to base kG + 1.
template <int kG>
__device__ __forceinline__ int upper_bound_group(const double* __restrict__ a, int lo, int hi, double v, int lane,
                                                 unsigned mask) {
    while (lo < hi) {
        const int len = hi - lo;
        const int at = lo + (int)(((long long)len * (lane + 1)) / (kG + 1));  // strictly below hi, rising with the lane
        const unsigned le = __ballot_sync(mask, a[at] <= v) >> ((threadIdx.x & 31) / kG * kG);
        const int n = __popc(kG == 32 ? le : le & ((1u << (kG % 32)) - 1));  // cuts at or below v (a is sorted)
        const int nlo = n == 0 ? lo : lo + (int)(((long long)len * n) / (kG + 1)) + 1;
        const int nhi = n == kG ? hi : lo + (int)(((long long)len * (n + 1)) / (kG + 1));
        lo = nlo;
        hi = max(nlo, nhi);
    }
    return lo;
}

// The splits of one level's nodes [begin, end): kG lanes per node, for kG = 1
// four nodes per thread side by side.
template <int kG>
__device__ __forceinline__ void level_splits(const TNode* __restrict__ nodes, const double* __restrict__ sx, int N0,
                                             int begin, int end, int* __restrict__ split) {
    const int t = threadIdx.x;
    if (kG > 1) {
        const int i = begin + t / kG;
        const bool on = i < end && nodes[min(i, end - 1)].m1 - nodes[min(i, end - 1)].m0 + 1 >= N0;
        const unsigned mask = __ballot_sync(0xffffffffu, on);
        if (on) {
            const TNode nd = nodes[i];
            const int k = upper_bound_group<kG>(sx, nd.m0, nd.m1 + 1, 0.5 * (nd.x0 + nd.x1), t % kG,
                                                mask & (kG == 32 ? 0xffffffffu : (((1u << (kG % 32)) - 1)
                                                                                  << ((t & 31) / kG * kG))));
            if (t % kG == 0) split[i] = k;
        }
        return;
    }
    constexpr int kILP = 4;
    for (int base = begin; base < end; base += kILP * 1024) {
        int lo[kILP], hi[kILP];
        double mid[kILP];
        bool go = false;
#pragma unroll
        for (int u = 0; u < kILP; ++u) {
            const int i = base + u * 1024 + t;
            lo[u] = hi[u] = 0;
            mid[u] = 0.0;
            if (i < end) {
                const TNode nd = nodes[i];
                mid[u] = 0.5 * (nd.x0 + nd.x1);
                lo[u] = nd.m0;
                hi[u] = nd.m1 - nd.m0 + 1 >= N0 ? nd.m1 + 1 : nd.m0;
            }
            go |= lo[u] < hi[u];
        }
        while (go) {
            go = false;
            double v[kILP];
#pragma unroll
            for (int u = 0; u < kILP; ++u) v[u] = lo[u] < hi[u] ? sx[lo[u] + ((hi[u] - lo[u]) >> 1)] : 0.0;
#pragma unroll
            for (int u = 0; u < kILP; ++u) {
                if (lo[u] < hi[u]) {
                    const int m = lo[u] + ((hi[u] - lo[u]) >> 1);
                    if (v[u] <= mid[u]) lo[u] = m + 1;
                    else hi[u] = m;
                    go |= lo[u] < hi[u];
                }
            }
        }
#pragma unroll
        for (int u = 0; u < kILP; ++u) {
            const int i = base + u * 1024 + t;
            if (i < end) split[i] = lo[u];
        }
    }
}

// The splits of the first levels, by a node's place in the full binary tree (the
// root 1, node h's children 2 h and 2 h + 1): the bisection does not depend on the
// points, so every place of these levels finds its split at once, a thread each,
// in place of a search per level one after another.
constexpr int kHeapLevels = 14;
inline int heap_levels(int n, int N0) {
    int d = 1;
    while (d < kHeapLevels && ((long long)N0 << (d - 2 > 0 ? d - 2 : 0)) < n) ++d;
    return d;
}
__global__ void k_heap_splits(const double* __restrict__ sx, int n, int levels, int* __restrict__ heap) {
    const int h = blockIdx.x * blockDim.x + threadIdx.x;
    if (h < 1 || h >= 1 << levels) return;
    double x0 = sx[0] - 0.1234, x1 = sx[n - 1] + 0.001;
    for (int b = 30 - __clz(h); b >= 0; --b) {
        const double mid = 0.5 * (x0 + x1);
        if (h >> b & 1) x0 = mid;
        else x1 = mid;
    }
    heap[h] = upper_bound(sx, 0, n, 0.5 * (x0 + x1));
}

// One CTA, level by level: a level's splits (from the heap's levels, below them
// all of a level's searches first, chains of dependent loads with as many lanes
// per node as there are to spare), then its children.  Until a node of the heap's
// levels is split, split[] holds its place there.
// meta: [0] nodes, [1] leaves, [2] error code, [3] depth.  arrived[] is cleared
// for the upward pass.  6.3 million points (13 levels): 62 us and 14 for
// k_heap_splits, against 147 with every level's searches by lane groups and 204 by
// a thread each; 395,523 (9 levels): 19 and 12, against 49 and 88.
__global__ void __launch_bounds__(1024) k_build_tree(const double* __restrict__ sx, int n, int N0, int cap_nodes,
                                                     int cap_leaves, TNode* __restrict__ nodes,
                                                     int* __restrict__ leaves, int* __restrict__ split,
                                                     int* __restrict__ arrived, const int* __restrict__ heap,
                                                     int levels, int* __restrict__ meta) {
    __shared__ int s_begin, s_end, s_next, s_nleaf, s_err;
    __shared__ int s_child[32], s_leaf[32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        TNode r;
        r.x0 = sx[0] - 0.1234;
        r.x1 = sx[n - 1] + 0.001;
        r.xc = 0.5 * (r.x0 + r.x1);
        r.m0 = 0;
        r.m1 = n - 1;
        r.child0 = r.child1 = -1;
        r.parent = -1;
        r.level = 0;
        nodes[0] = r;
        split[0] = 1;
        s_begin = 0;
        s_end = 1;
        s_next = 1;
        s_nleaf = 0;
        s_err = 0;
    }
    __syncthreads();
    int level = 0;
    while (s_begin < s_end) {
        if (level > kMaxDepth) {
            if (tid == 0) s_err = FS_ERR_TREE;
            break;
        }
        const int begin = s_begin, end = s_end, count = end - begin;
        const bool known = level < levels;
        if (!known) {
            if (count <= 32) level_splits<32>(nodes, sx, N0, begin, end, split);
            else if (count <= 128) level_splits<8>(nodes, sx, N0, begin, end, split);
            else level_splits<1>(nodes, sx, N0, begin, end, split);
            __syncthreads();
        }
        for (int base = begin; base < end; base += 1024) {
            const int i = base + tid;
            int nchild = 0, isleaf = 0, k = 0, place = 0;
            TNode nd;
            if (i < end) {
                nd = nodes[i];
                const int cnt = nd.m1 - nd.m0 + 1;
                if (cnt >= N0) {
                    k = split[i];
                    if (known) {
                        place = k;
                        k = min(max(heap[place], nd.m0), nd.m1 + 1);
                    }
                    nchild = (k > nd.m0) + (k <= nd.m1);
                } else {
                    isleaf = 1;
                }
            }
            int a = nchild, b = isleaf;  // inclusive scans over the CTA
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int u = __shfl_up_sync(0xffffffffu, a, o), v = __shfl_up_sync(0xffffffffu, b, o);
                if (lane >= o) {
                    a += u;
                    b += v;
                }
            }
            if (lane == 31) {
                s_child[warp] = a;
                s_leaf[warp] = b;
            }
            __syncthreads();
            if (warp == 0) {
                int u = s_child[lane], v = s_leaf[lane];
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int x = __shfl_up_sync(0xffffffffu, u, o), y = __shfl_up_sync(0xffffffffu, v, o);
                    if (lane >= o) {
                        u += x;
                        v += y;
                    }
                }
                s_child[lane] = u;
                s_leaf[lane] = v;
            }
            __syncthreads();
            const int cfirst = s_next + (warp ? s_child[warp - 1] : 0) + a - nchild;
            const int lslot = s_nleaf + (warp ? s_leaf[warp - 1] : 0) + b - isleaf;
            if (i < end) {
                if (isleaf) {
                    if (lslot < cap_leaves) leaves[lslot] = i;
                } else if (nchild) {
                    const double mid = 0.5 * (nd.x0 + nd.x1);
                    int c = cfirst;
                    int c0 = -1, c1 = -1;
                    if (k > nd.m0 && c < cap_nodes) {
                        TNode ch;
                        ch.x0 = nd.x0;
                        ch.x1 = mid;
                        ch.xc = 0.5 * (ch.x0 + ch.x1);
                        ch.m0 = nd.m0;
                        ch.m1 = k - 1;
                        ch.child0 = ch.child1 = -1;
                        ch.parent = i;
                        ch.level = level + 1;
                        nodes[c] = ch;
                        arrived[c] = 0;
                        split[c] = 2 * place;
                        c0 = c++;
                    }
                    if (k <= nd.m1 && c < cap_nodes) {
                        TNode ch;
                        ch.x0 = mid;
                        ch.x1 = nd.x1;
                        ch.xc = 0.5 * (ch.x0 + ch.x1);
                        ch.m0 = k;
                        ch.m1 = nd.m1;
                        ch.child0 = ch.child1 = -1;
                        ch.parent = i;
                        ch.level = level + 1;
                        nodes[c] = ch;
                        arrived[c] = 0;
                        split[c] = 2 * place + 1;
                        if (c0 < 0) c0 = c;
                        else c1 = c;
                        ++c;
                    }
                    nodes[i].child0 = c0;
                    nodes[i].child1 = c1;
                }
            }
            __syncthreads();
            if (tid == 0) {
                s_next += s_child[31];
                s_nleaf += s_leaf[31];
                if (s_next > cap_nodes || s_nleaf > cap_leaves) s_err = FS_ERR_TREE;
            }
            __syncthreads();
            if (s_err) break;
        }
        if (s_err) break;
        if (tid == 0) {
            s_begin = end;
            s_end = s_next;
        }
        ++level;
        __syncthreads();
    }
    if (tid == 0) {
        meta[0] = min(s_next, cap_nodes);
        meta[1] = min(s_nleaf, cap_leaves);
        meta[2] = s_err;
        meta[3] = level;
    }
}

__global__ void k_mark_leaves(const TNode* __restrict__ nodes, const int* __restrict__ leaves,
                              const int* __restrict__ meta, int* __restrict__ leaf_of) {
    const int l = blockIdx.x;
    if (l >= meta[1] || meta[2]) return;
    const TNode nd = nodes[leaves[l]];
    for (int j = nd.m0 + threadIdx.x; j <= nd.m1; j += blockDim.x) leaf_of[j] = l;
}

// build_interaction_list (src/FieldStructure.cpp:663-702) for one leaf, a warp
// each: the nodes still to be tested, starting with the root, are taken up to 32
// at a time, one per lane, and the children of those that are neither far nor
// leaves join the end of the queue.  The lists hold the reference's nodes, level
// by level instead of depth first; a thread per leaf spent 66 us on its chain of
// node reads at 6.3 million points, a warp 20 us.
// Every queued node leaves at least one entry in a list, so lists within their
// caps never overflow this.
constexpr int kListQueue = 512;
static_assert(kListQueue >= kFarCap + kNearCap + 64, "queue holds what the lists can");
__global__ void __launch_bounds__(128) k_lists(const TNode* __restrict__ nodes, const int* __restrict__ leaves,
                                               const int* __restrict__ meta, double L, double sqrt_sq_theta,
                                               int* __restrict__ far_list, int* __restrict__ far_n,
                                               int* __restrict__ near_list, int* __restrict__ near_n,
                                               int* __restrict__ err) {
    __shared__ int queue[4][kListQueue];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int l = blockIdx.x * 4 + warp;
    if (l >= meta[1] || meta[2]) return;
    int* q = queue[warp];
    const TNode b = nodes[leaves[l]];
    const double dfbx = b.x1 - b.xc, sq_rb = dfbx * dfbx;
    int head = 0, tail = 1;  // queued: [head, tail), places taken modulo kListQueue
    if (lane == 0) q[0] = 0;
    int nf = 0, nn = 0;
    const unsigned below = (1u << lane) - 1;
    __syncwarp();
    while (head < tail) {
        const int take = min(32, tail - head);
        bool near = false, far = false, open = false;
        int pi = 0, c0 = -1, c1 = -1;
        if (lane < take) {
            pi = q[(head + lane) % kListQueue];
            const TNode p = nodes[pi];
            const double r_dist = fabs(b.xc - p.xc);
            const double dfbpx = fmin(r_dist, L - r_dist);
            const double dfpx = p.x1 - p.xc;
            const double sq_R = dfbpx * dfbpx, sq_rp = dfpx * dfpx;
            c0 = p.child0;
            c1 = p.child1;
            near = c0 < 0 && c1 < 0;
            far = !near && (__dsqrt_rn(sq_rb) + __dsqrt_rn(sq_rp)) / __dsqrt_rn(sq_R) < sqrt_sq_theta;
            open = !near && !far;
        }
        head += take;
        const unsigned mn = __ballot_sync(0xffffffffu, near), mf = __ballot_sync(0xffffffffu, far);
        const unsigned m0 = __ballot_sync(0xffffffffu, open && c0 >= 0), m1 = __ballot_sync(0xffffffffu, open && c1 >= 0);
        if (near) {
            const int at = nn + __popc(mn & below);
            if (at < kNearCap) near_list[(size_t)l * kNearCap + at] = pi;
        }
        if (far) {
            const int at = nf + __popc(mf & below);
            if (at < kFarCap) far_list[(size_t)l * kFarCap + at] = pi;
        }
        nn += __popc(mn);
        nf += __popc(mf);
        const int add = __popc(m0) + __popc(m1);
        if (tail - head + add > kListQueue) {  // more open nodes than a list could end up with
            if (lane == 0) {
                atomicCAS(err, 0, (int)FS_ERR_TREE);
                far_n[l] = near_n[l] = 0;
            }
            return;
        }
        if (open) {
            int at = tail + __popc(m0 & below) + __popc(m1 & below);
            if (c0 >= 0) q[at++ % kListQueue] = c0;
            if (c1 >= 0) q[at % kListQueue] = c1;
        }
        tail += add;
        __syncwarp();
    }
    if (lane == 0) {
        if (nf > kFarCap || nn > kNearCap) atomicCAS(err, 0, (int)FS_ERR_TREE);
        far_n[l] = min(nf, kFarCap);
        near_n[l] = min(nn, kNearCap);
    }
}

// 1/x in FP64 for the FP32c treecode's moments: the hardware approximation
// and two Newton-Raphson steps (relative error ~1e-16 for normal x).
__device__ __forceinline__ double rcp_nr64(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    double e = fma(-x, y, 1.0);
    y = fma(y, e, y);
    e = fma(-x, y, 1.0);
    return fma(y, e, y);
}

// FP32c treecode moments with rcp_nr64 products instead of IEEE divisions:
// measured 0.9% faster per full-size treecode step.
#ifndef FS_FAST_MOMENTS
#define FS_FAST_MOMENTS 1
#endif
constexpr bool kFastMoments = FS_FAST_MOMENTS;
// Moments of every node but the root.  A CTA per leaf forms the leaf's from its
// points, with the reference's arithmetic per point (alloc_set_cluster_list
// :826-860), one rounding per operation; kPP fixes the number of Chebyshev nodes
// (degree + 1) at compile time, so that the per-point arrays live in registers.
// kFast (the FP32c treecode): divisions as products with rcp_nr64 instead of
// IEEE divisions.  Then the CTA climbs: whoever completes a node's children
// forms its moments from theirs.  A parent's Lagrange polynomials are of the
// children's degree, so l_k(x) = sum_l l_k(t_l) l_l(x) exactly, with the t_l a
// child's nodes: a fixed matrix for a left half and one for a right half
// (`halves`).  So each point is visited once instead of once per level.
// 6.3 million points: 1.55 ms (points at 12 levels, 1.44, and the chunks' sums)
// -> 0.13 ms.
constexpr int kLeafThreads = 128;
template <int kPP, bool kFast>
__global__ void __launch_bounds__(kLeafThreads) k_moments(const TNode* __restrict__ nodes, const int* __restrict__ meta,
                                                          const int* __restrict__ leaves,
                                                          const double* __restrict__ consts,
                                                          const double* __restrict__ halves,
                                                          const double* __restrict__ sx, const double* __restrict__ lam,
                                                          int* __restrict__ arrived, double* __restrict__ mom) {
    const int leaf = blockIdx.x;
    if (meta[2] || leaf >= meta[1]) return;
    const double* cheb = consts;
    const double* wk = consts + (kMaxDegree + 1);
    constexpr int PP = kPP;
    __shared__ double red[kLeafThreads / 32][kPP];
    int node = leaves[leaf];
    if (leaf == 0 && threadIdx.x <= kMaxDegree) mom[threadIdx.x] = 0.0;  // the root's are never formed
    if (node == 0) return;
    {
        const TNode nd = nodes[node];
        const int a = nd.m0, e = nd.m1;
        double t[kPP], acc[kPP];
#pragma unroll
        for (int k = 0; k < PP; ++k) {
            t[k] = dadd(nd.x0, dmul(dmul(dadd(cheb[k], 1.0), 0.5), dsub(nd.x1, nd.x0)));
            acc[k] = 0.0;
        }
        for (int j = a + threadIdx.x; j <= e; j += kLeafThreads) {
            const double x = sx[j];
            double ak[kPP];
            int exact = -1;
            double sum = 0.0;
            // w_k / dx_k, two nodes per division where both differences are
            // clear of zero: 1/dx_a = dx_b / (dx_a dx_b) (a few ulps; |dx| lies
            // between the spacing of doubles near x and the node width, so the
            // product neither underflows nor overflows)
            int k = 0;
#pragma unroll
            for (; k + 1 < PP; k += 2) {
                const double da = dsub(x, t[k]), db = dsub(x, t[k + 1]);
                if (fabs(da) <= DBL_MIN || fabs(db) <= DBL_MIN) {
                    if (fabs(da) <= DBL_MIN) {
                        exact = k;
                        ak[k] = 0.0;
                    } else {
                        ak[k] = (kFast ? wk[k] * rcp_nr64(da) : ddiv(wk[k], da));
                        sum = dadd(sum, ak[k]);
                    }
                    if (fabs(db) <= DBL_MIN) {
                        exact = k + 1;
                        ak[k + 1] = 0.0;
                    } else {
                        ak[k + 1] = (kFast ? wk[k + 1] * rcp_nr64(db) : ddiv(wk[k + 1], db));
                        sum = dadd(sum, ak[k + 1]);
                    }
                } else {
                    const double r = (kFast ? rcp_nr64(dmul(da, db)) : ddiv(1.0, dmul(da, db)));
                    ak[k] = dmul(wk[k], dmul(db, r));
                    ak[k + 1] = dmul(wk[k + 1], dmul(da, r));
                    sum = dadd(dadd(sum, ak[k]), ak[k + 1]);
                }
            }
            if (k < PP) {
                const double dx = dsub(x, t[k]);
                if (fabs(dx) <= DBL_MIN) {
                    exact = k;
                    ak[k] = 0.0;
                } else {
                    ak[k] = (kFast ? wk[k] * rcp_nr64(dx) : ddiv(wk[k], dx));
                    sum = dadd(sum, ak[k]);
                }
            }
            if (exact > -1) {
                sum = 1.0;
#pragma unroll
                for (int k = 0; k < PP; ++k) ak[k] = (k == exact) ? 1.0 : 0.0;
            }
            const double D = (kFast ? rcp_nr64(sum) : ddiv(1.0, sum));
            const double l = lam[j];
#pragma unroll
            for (int k = 0; k < PP; ++k) acc[k] = dadd(acc[k], dmul(dmul(ak[k], D), l));
        }
        // block reduction in a fixed order: a shuffle tree within each warp, then
        // the warps' sums in warp order
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
        for (int k = 0; k < PP; ++k) {
            double v = acc[k];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v = dadd(v, __shfl_down_sync(0xffffffffu, v, o));
            if (lane == 0) red[warp][k] = v;
        }
        __syncthreads();
        if (threadIdx.x < PP) {
            double sum = red[0][threadIdx.x];
            for (int w = 1; w < kLeafThreads / 32; ++w) sum = dadd(sum, red[w][threadIdx.x]);
            mom[(size_t)node * (kMaxDegree + 1) + threadIdx.x] = sum;
        }
    }
    // upward: the last child to arrive makes the parent
    if (threadIdx.x >= 32) return;
    for (;;) {
        const int up = nodes[node].parent;
        if (up == 0) return;
        const TNode p = nodes[up];
        __threadfence();  // this node's moments before the arrival
        __syncwarp();
        int go = 0;
        if (threadIdx.x == 0) go = atomicAdd(&arrived[up], 1) + 1 == (p.child0 >= 0) + (p.child1 >= 0);
        if (!__shfl_sync(0xffffffffu, go, 0)) return;
        __threadfence();  // the other child's moments after its arrival
        if (threadIdx.x < PP) {
            double s = 0.0;
            for (int c = 0; c < 2; ++c) {
                const int ch = c ? p.child1 : p.child0;
                if (ch < 0) continue;
                const double* H = halves + (nodes[ch].x0 == p.x0 ? 0 : PP * PP) + threadIdx.x * PP;
                const volatile double* m = mom + (size_t)ch * (kMaxDegree + 1);
                for (int l = 0; l < PP; ++l) s = fma(H[l], m[l], s);
            }
            mom[(size_t)up * (kMaxDegree + 1) + threadIdx.x] = s;
        }
        node = up;
    }
}

// One term of the reference sum over norm = sqrt(L^2 + 4 eps^2) / L,
// `w * -1.0 * s * (1 - sqrt(deno / (4*s*s*L*L + 4*eps*eps)))`
// (src/FieldStructure.cpp:940-950, :1000-1010), as w d (1 / (2 sqrt(d^2 + eps^2)) - c):
// the reciprocal root by the hardware approximation (2^-20) and one step of third
// order.  The pairs the reference skips (s = 0, +-1/2) are zeros of this form.
__device__ __forceinline__ double tree_term(double w, double d, double L, double invL, double e2, double c,
                                            double acc) {
    d -= L * rint(d * invL);
    const double r = fma(d, d, e2);
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(r));
    const double e = fma(-r * y, y, 1.0);
    y = fma(y * e, fma(e, 0.375, 0.5), y);
    return fma(w, d * fma(0.5, y, -c), acc);
}

// FP64 per target: far field (Call_BL) and near field (Call_Ds); result through the
// stage epilogue at the original index.  kG lanes share a target's terms and add
// their sums in a tree: a term is a chain of a dozen FP64 operations, and the trees
// that come here (below 16 points per epsilon) have too few targets to hide it
// behind one another.  Of the bump-on-tail box, against a thread per target and the
// reference's two divisions and root per term (the same lists): 2,000 points 624 ->
// 85 us per field, 10,000 2900 -> 227, 49,000 2740 -> 458; with eight lanes at any
// size 109, 274 and 460, and in the reference's operations 178, 600 and 1261.
// Points below which a target has a whole warp: 20,000 take 281 us so and 309 by
// eight lanes, 25,000 take 340 by eight lanes.
constexpr int kFarNearWide = 24000;
constexpr double kCellBox = 640.0;  // L / epsilon from which FP64 sums go through cells (Treecode::cells_take)
template <int kG>
__global__ void __launch_bounds__(128) k_far_near64(const TNode* __restrict__ nodes, const int* __restrict__ meta,
                                                    const int* __restrict__ leaf_of, const int* __restrict__ far_list,
                                                    const int* __restrict__ far_n, const int* __restrict__ near_list,
                                                    const int* __restrict__ near_n, const double* __restrict__ mom,
                                                    const double* __restrict__ consts, const double* __restrict__ sx,
                                                    const double* __restrict__ lam, const int* __restrict__ sidx, int n,
                                                    int P, double L, double eps, double norm, double cbg, Stage S) {
    if (meta[2]) return;
    const int j0 = (int)(((long long)blockIdx.x * blockDim.x + threadIdx.x) / kG), g = threadIdx.x % kG;
    const int j = min(j0, n - 1);  // lanes beyond the last target stay for the shuffles
    const int PP = P + 1;
    const double invL = 1.0 / L, e2 = fmax(eps * eps, DBL_MIN);  // a normal root at d = 0, however small eps
    const int l = leaf_of[j];
    const double x = sx[j];
    double far = 0.0;
    const int terms = far_n[l] * PP;
    for (int z = g; z < terms; z += kG) {
        const int f = z / PP, k = z - f * PP;
        const int fi = far_list[(size_t)l * kFarCap + f];
        const double x0 = nodes[fi].x0, x1 = nodes[fi].x1;
        const double t = dadd(x0, dmul(dmul(dadd(consts[k], 1.0), 0.5), dsub(x1, x0)));
        far = tree_term(mom[(size_t)fi * (kMaxDegree + 1) + k], x - t, L, invL, e2, cbg, far);
    }
    double near = 0.0;
    for (int q = 0; q < near_n[l]; ++q) {
        const TNode nd = nodes[near_list[(size_t)l * kNearCap + q]];
#pragma unroll 4
        for (int i = nd.m0 + g; i <= nd.m1; i += kG) near = tree_term(lam[i], x - sx[i], L, invL, e2, cbg, near);
    }
    double e = far + near;
#pragma unroll
    for (int o = kG / 2; o > 0; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
    if (g == 0 && j0 < n) apply_stage(S, sidx[j], norm * e);
}

// FP32-compensated form, far part: FP64 with the kernel written through one
// reciprocal square root, K_tc(d) = norm * (d / (2 sqrt(d^2+eps^2)) - c d).
// k_far32's per-node arithmetic: the nearest image by a product with 1/L and
// 1/sqrt by the hardware approximation and one Newton step (1), or by an IEEE
// division and the library's FP64 rsqrt (0).  (1) measured 4% faster per step
// of the three-species treecode workload, with E changed by about 2e-14.
#ifndef FS_FAR32_FAST
#define FS_FAR32_FAST 1
#endif
constexpr bool kFar32Fast = FS_FAR32_FAST;

__global__ void k_far32(const TNode* __restrict__ nodes, const int* __restrict__ meta, const int* __restrict__ leaf_of,
                        const int* __restrict__ far_list, const int* __restrict__ far_n,
                        const double* __restrict__ mom, const double* __restrict__ consts,
                        const double* __restrict__ sx, int n, int P, double L, double eps, double norm, double cbg,
                        double* __restrict__ efar) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n || meta[2]) return;
    const double* cheb = consts;
    const int PP = P + 1;
    const int l = leaf_of[j];
    const double x = sx[j];
    const double e2 = eps * eps;
    const double invL = 1.0 / L;
    double far = 0.0;
    for (int f = 0; f < far_n[l]; ++f) {
        const int fi = far_list[(size_t)l * kFarCap + f];
        const TNode nd = nodes[fi];
        const double* m = mom + (size_t)fi * (kMaxDegree + 1);
        for (int k = 0; k < PP; ++k) {
            const double t = nd.x0 + (cheb[k] + 1.0) * 0.5 * (nd.x1 - nd.x0);
            double d = x - t;
            if (kFar32Fast) {
                // nearest image by a product with 1/L, 1/sqrt from the hardware
                // approximation and one Newton step (relative error ~1e-14)
                d -= L * rint(d * invL);
                const double r = d * d + e2;
                double y;
                asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(r));
                y = y * fma(-0.5 * r, y * y, 1.5);
                far += m[k] * (d * (0.5 * y - cbg));
            } else {
                d -= L * rint(d / L);
                far += m[k] * (d * (0.5 * rsqrt(d * d + e2) - cbg));
            }
        }
    }
    efar[j] = norm * far;
}

// FP32-compensated form, near part: a CTA per (leaf, block of kNearThreads x
// kNearR targets), or two with two targets per thread each, the near list
// shared by several, where the targets are few.
//   K_tc(d) / norm = d/(2 sqrt(d^2+eps^2)) - c d,  d = xt - x_j  (xt = image of x_i)
// The linear term c d is summed exactly in FP64 from prefix sums of lambda and
// lambda x.  For each near leaf, when every target of the block sees the whole
// leaf in one periodic image and within the band |d| <= band (leaves narrower
// than the band), the pairs are lambda/2 d y, y = rsqrt(d^2+eps^2), accumulated
// in packed FP32x2 over two targets with Kahan compensation per tile and reduced
// in FP64 across tiles.  Otherwise the block takes the general path for that
// leaf: the leaf's sources are cut where their image changes (at most three
// images), and beyond the band the sign part sign(d) lambda/2 is summed exactly
// in FP64 while the kernel accumulates -+ lambda/2 c(v) (c = v/2 + v^2/8, v =
// eps^2 y^2).  Sources are staged through shared memory as FP32 offsets from an
// FP64 tile base; each image's target offset is formed in FP64 before rounding.
//
// What bounds it: one MUFU.RSQ per pair (16/clk/SM), and for wide leaves the
// latency of the Kahan chain, which wants warps: 99,000 points (leaves of 50
// epsilon) 2.27 ms with four targets per thread walked one by one, 0.99 ms in
// packed pairs, 0.45 ms with the near lists shared by eight CTAs, the results
// equal (the shared lists' FP64 additions to 1e-16).
#ifndef FS_NEAR_THREADS
#define FS_NEAR_THREADS 128
#endif
#ifndef FS_NEAR_R
#define FS_NEAR_R 4
#endif
constexpr int kNearThreads = FS_NEAR_THREADS;
constexpr int kNearR = FS_NEAR_R;
constexpr int kNearBlock = kNearThreads * kNearR;
static_assert(kNearR == 4, "two pairs of targets per thread");
constexpr int kNearTile = 256;
constexpr double kNearBand = 24.0;
constexpr int kNearSplit = 16;  // below this many target blocks per SM a thread takes two targets
// CTAs per SM that sharing near lists aims at, and parts of a list at most (12:
// 12 to 29% slower at 100,000 to 400,000 points; 16 parts no faster)
constexpr int kNearCtas = 24, kNearParts = 8;
// The images of a near leaf's sources as one target sees them, at most three:
// image k holds sources [start[k], start[k + 1]) at target coordinate xt[k],
// with the band |d| <= band at [U1[k], U2[k]).
struct NearImages {
    double xt[3];
    int start[4], U1[3], U2[3];
};

__device__ __forceinline__ int lower_bound_d(const double* __restrict__ a, int lo, int hi, double v) {
    while (lo < hi) {
        const int mid = lo + ((hi - lo) >> 1);
        if (a[mid] < v) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}
__device__ __forceinline__ int upper_bound_d(const double* __restrict__ a, int lo, int hi, double v) {
    while (lo < hi) {
        const int mid = lo + ((hi - lo) >> 1);
        if (a[mid] <= v) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}
__device__ __forceinline__ double range_sum(const double* __restrict__ incl, int a, int e) {
    // sum over [a, e) of the series whose inclusive prefix is incl
    if (e <= a) return 0.0;
    return incl[e - 1] - (a > 0 ? incl[a - 1] : 0.0);
}

// Cuts the leaf's sources where their image changes, finds each image's band
// and adds the exact terms: the linear term and, beyond the band, the sign part.
__device__ __forceinline__ void near_images(const TNode& nd, double x, const double* __restrict__ sx,
                                            const double* __restrict__ pl, const double* __restrict__ plx, double L,
                                            double band, double cbg, NearImages& im, double& exact,
                                            int* __restrict__ err) {
    int a = nd.m0, nim = 0;
    const double xlast = sx[nd.m1];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        im.start[k] = INT_MAX;
        im.U1[k] = im.U2[k] = 0;
        im.xt[k] = k ? im.xt[k - 1] : 0.0;
        if (a <= nd.m1) {
            // image of source j: m_j = round((x - x_j) / L), the reference's
            // choice (z - round(z)); m_j is non-increasing in j
            const double m = round((x - sx[a]) / L);
            const double xt = x - m * L;
            int e = nd.m1 + 1;  // first source of the next image
            if (round((x - xlast) / L) < m) {
                int lo = a + 1, hi = nd.m1 + 1;
                while (lo < hi) {
                    const int mid = lo + ((hi - lo) >> 1);
                    if (round((x - sx[mid]) / L) < m) hi = mid;
                    else lo = mid + 1;
                }
                e = lo;
            }
            // most leaves lie wholly inside the band or wholly to one side
            const double first = sx[a], last = sx[e - 1];
            const int U1 = first >= xt - band ? a : (last < xt - band ? e : lower_bound_d(sx, a, e, xt - band));
            const int U2 = last <= xt + band ? e : (U1 < e && sx[U1] <= xt + band ? upper_bound_d(sx, U1, e, xt + band)
                                                                                   : U1);  // first x_j > xt + band
            exact += 0.5 * (range_sum(pl, a, U1) - range_sum(pl, U2, e)) -
                     cbg * (xt * range_sum(pl, a, e) - range_sum(plx, a, e));
            im.xt[k] = xt;
            im.start[k] = a;
            im.U1[k] = U1;
            im.U2[k] = U2;
            ++nim;
            a = e;
        }
    }
    im.start[3] = INT_MAX;
    if (a <= nd.m1) atomicCAS(err, 0, (int)FS_ERR_TREE);
}

// Sources [t0, t0 + cnt) as one target sees them: its offset when they share an
// image, and 1 (beyond the band on the left), 2 (right), 3 (in the band) when
// they also share a side; 0 otherwise.
__device__ __forceinline__ int near_side(const NearImages& im, int t0, int cnt, double base, float& tau) {
    int side = 0;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        if (t0 >= im.start[k] && (im.start[k + 1] == INT_MAX || t0 + cnt <= im.start[k + 1])) {
            tau = (float)(im.xt[k] - base);
            side = t0 + cnt <= im.U1[k] ? 1 : (t0 >= im.U2[k] ? 2 : (t0 >= im.U1[k] && t0 + cnt <= im.U2[k] ? 3 : 0));
        }
    }
    return side;
}

// One tile for one target, image and side per source.
__device__ void near_mixed(const NearImages& im, int t0, int cnt, double base, const float4* sh, float eps2,
                           float& acc, float& ncmp) {
    const float tau0 = (float)(im.xt[0] - base), tau1 = (float)(im.xt[1] - base), tau2 = (float)(im.xt[2] - base);
    for (int k = 0; k < cnt; ++k) {
        const int jj = t0 + k;
        const bool g1 = jj >= im.start[1], g2 = jj >= im.start[2];
        const float tr = g2 ? tau2 : (g1 ? tau1 : tau0);
        const int U1 = g2 ? im.U1[2] : (g1 ? im.U1[1] : im.U1[0]);
        const int U2 = g2 ? im.U2[2] : (g1 ? im.U2[1] : im.U2[0]);
        const float4 e = sh[k];
        const float d = tr - e.x;
        const float y = rsqrt_approx(fmaf(d, d, eps2));
        const float z = __fmul_rn(y, y);
        const float c = __fmul_rn(z, fmaf(z, e.w, e.z));
        const float v = (jj < U1) ? -c : ((jj >= U2) ? c : __fmul_rn(e.y, __fmul_rn(d, y)));
        const float w = __fadd_rn(v, ncmp);
        const float t = __fadd_rn(acc, w);
        ncmp = __fsub_rn(w, __fsub_rn(t, acc));
        acc = t;
    }
}

// General path for a pair of targets and one near leaf (all threads of the CTA
// call it together: it stages tiles through `sh` with barriers).  Most tiles are
// of one side for all of a warp's targets, and these run in packed FP32x2; the
// others go pair by pair.  The Kahan compensation is kept negated.
__device__ void near_general2(const TNode& nd, const double (&x)[2], const double* __restrict__ sx,
                              const double* __restrict__ lam, const double* __restrict__ pl,
                              const double* __restrict__ plx, double L, double band, double cbg, float eps2, float a1,
                              float a2, float4 (*sh)[kNearTile], double* exact, double* fp, int* __restrict__ err) {
    NearImages im[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) near_images(nd, x[h], sx, pl, plx, L, band, cbg, im[h], exact[h], err);
    constexpr int kPer = kNearTile / kNearThreads;
    double nx[kPer], nl[kPer];
    double nbase = 0.0;
    auto fetch = [&](int t0) {
#pragma unroll
        for (int i = 0; i < kPer; ++i) {
            const int j = t0 + threadIdx.x + i * kNearThreads;
            nx[i] = (j <= nd.m1) ? sx[j] : 0.0;
            nl[i] = (j <= nd.m1) ? lam[j] : 0.0;
        }
        nbase = sx[t0];
    };
    fetch(nd.m0);
    int buf = 0;
    for (int t0 = nd.m0; t0 <= nd.m1; t0 += kNearTile, buf ^= 1) {
        const int cnt = min(kNearTile, nd.m1 - t0 + 1);
        const double base = nbase;
#pragma unroll
        for (int i = 0; i < kPer; ++i) {
            const float lh = (float)(0.5 * nl[i]);
            sh[buf][threadIdx.x + i * kNearThreads] =
                make_float4((float)(nx[i] - base), lh, __fmul_rn(lh, a1), __fmul_rn(lh, a2));
        }
        __syncthreads();
        if (t0 + kNearTile <= nd.m1) fetch(t0 + kNearTile);
        float tau[2] = {0.f, 0.f};
        const int s0 = near_side(im[0], t0, cnt, base, tau[0]), s1 = near_side(im[1], t0, cnt, base, tau[1]);
        const bool far = __all_sync(0xffffffffu, (s0 == 1 || s0 == 2) && (s1 == 1 || s1 == 2));
        const bool near = __all_sync(0xffffffffu, s0 == 3 && s1 == 3);
        const float2 e2v = make_float2(eps2, eps2), m1 = make_float2(-1.f, -1.f);
        const float2 tau2 = make_float2(tau[0], tau[1]);
        float2 acc = make_float2(0.f, 0.f), nc = make_float2(0.f, 0.f);
        const float4* tile = sh[buf];
        if (far) {
            const float2 sgn = make_float2(s0 == 1 ? -1.f : 1.f, s1 == 1 ? -1.f : 1.f);
#pragma unroll 4
            for (int k = 0; k < cnt; ++k) {
                const float4 e = tile[k];
                const float2 d = __ffma2_rn(make_float2(e.x, e.x), m1, tau2);
                const float2 r2 = __ffma2_rn(d, d, e2v);
                const float2 y = make_float2(rsqrt_approx(r2.x), rsqrt_approx(r2.y));
                const float2 z = __fmul2_rn(y, y);
                const float2 c = __fmul2_rn(z, __ffma2_rn(z, make_float2(e.w, e.w), make_float2(e.z, e.z)));
                const float2 w = __ffma2_rn(c, sgn, nc);  // +-c, exactly, less the compensation
                const float2 t = __fadd2_rn(acc, w);
                nc = __ffma2_rn(__ffma2_rn(acc, m1, t), m1, w);
                acc = t;
            }
        } else if (near) {
            // 1, in a form that keeps v's own rounding before it meets the compensation
            const float2 one = make_float2(s0 == 3 ? 1.f : -1.f, s1 == 3 ? 1.f : -1.f);
#pragma unroll 4
            for (int k = 0; k < cnt; ++k) {
                const float4 e = tile[k];
                const float2 d = __ffma2_rn(make_float2(e.x, e.x), m1, tau2);
                const float2 r2 = __ffma2_rn(d, d, e2v);
                const float2 y = make_float2(rsqrt_approx(r2.x), rsqrt_approx(r2.y));
                const float2 v = __fmul2_rn(make_float2(e.y, e.y), __fmul2_rn(d, y));
                const float2 w = __ffma2_rn(v, one, nc);
                const float2 t = __fadd2_rn(acc, w);
                nc = __ffma2_rn(__ffma2_rn(acc, m1, t), m1, w);
                acc = t;
            }
        } else {
            near_mixed(im[0], t0, cnt, base, tile, eps2, acc.x, nc.x);
            near_mixed(im[1], t0, cnt, base, tile, eps2, acc.y, nc.y);
        }
        fp[0] += (double)acc.x + (double)nc.x;
        fp[1] += (double)acc.y + (double)nc.y;
    }
    __syncthreads();  // the next leaf reuses shared memory
}

struct NearArgs {
    const TNode* nodes;
    const int* meta;
    const int* leaves;
    const int* near_list;
    const int* near_n;
    const double* sx;
    const double* lam;
    const double* pl;
    const double* plx;
    const double* efar;
    const int* sidx;
    double L, eps, cbg, norm;
    Stage S;
    int* err;
    // shared near lists: `parts` CTAs take a part each and leave their sums in
    // part[p * n + j] for k_near_add
    int parts, n;
    double* part;
};

// Near field of target block yb of leaf l from part `part` of its near list,
// pairs of targets h0 .. h0 + kPairs - 1 of each thread's kNearR (all threads of
// the CTA together).
template <int kPairs>
__device__ void near_item(const NearArgs& A, int l, int yb, int h0, int part, float4 (*shg)[kNearTile],
                          float2 (*shb)[kNearTile]) {
    const TNode* __restrict__ nodes = A.nodes;
    const int* __restrict__ near_list = A.near_list;
    const double* __restrict__ sx = A.sx;
    const double* __restrict__ lam = A.lam;
    const double* __restrict__ pl = A.pl;
    const double* __restrict__ plx = A.plx;
    const double L = A.L, eps = A.eps, cbg = A.cbg;
    int* __restrict__ err = A.err;
    if (l >= A.meta[1] || A.meta[2]) return;
    const TNode leaf = nodes[A.leaves[l]];
    const int tb0 = leaf.m0 + yb * kNearBlock;
    if (tb0 > leaf.m1) return;  // whole CTA beyond the leaf
    const double band = kNearBand * eps;
    const double e2d = eps * eps;
    const float eps2 = (float)e2d, a1 = (float)(e2d / 2), a2 = (float)(e2d * e2d / 8);
    if (tb0 + 2 * h0 * kNearThreads > leaf.m1) return;  // none of these targets is real
    double x[kNearR], exact[2 * kPairs], fp[2 * kPairs];
#pragma unroll
    for (int r = 0; r < kNearR; ++r) {
        const int j = tb0 + threadIdx.x + r * kNearThreads;
        x[r] = (j <= leaf.m1) ? sx[j] : sx[leaf.m0];  // padded targets repeat a real one
    }
#pragma unroll
    for (int r = 0; r < 2 * kPairs; ++r) exact[r] = fp[r] = 0.0;
    double xp[kPairs][2];  // this CTA's targets
#pragma unroll
    for (int h = 0; h < kPairs; ++h) {
        xp[h][0] = kPairs == kNearR / 2 ? x[2 * h] : (h0 ? x[2] : x[0]);
        xp[h][1] = kPairs == kNearR / 2 ? x[2 * h + 1] : (h0 ? x[3] : x[1]);
    }
    const int nn = A.near_n[l], q0 = nn * part / A.parts, q1 = nn * (part + 1) / A.parts;
    for (int q = q0; q < q1; ++q) {
        const TNode nd = nodes[near_list[(size_t)l * kNearCap + q]];
        const double xlo = sx[nd.m0], xhi = sx[nd.m1];
        // decided for all targets of the block, whichever of them this CTA takes
        double xtr[kNearR];
        bool simple = true;
#pragma unroll
        for (int r = 0; r < kNearR; ++r) {
            const double m = round((x[r] - xlo) / L);
            xtr[r] = x[r] - m * L;
            simple = simple && (round((x[r] - xhi) / L) == m) && (xlo >= xtr[r] - band) && (xhi <= xtr[r] + band);
        }
        if (__syncthreads_and(simple)) {
            double xt[2 * kPairs];
#pragma unroll
            for (int h = 0; h < kPairs; ++h) {
                xt[2 * h] = kPairs == kNearR / 2 ? xtr[2 * h] : (h0 ? xtr[2] : xtr[0]);
                xt[2 * h + 1] = kPairs == kNearR / 2 ? xtr[2 * h + 1] : (h0 ? xtr[3] : xtr[1]);
            }
            const double sl = range_sum(pl, nd.m0, nd.m1 + 1), slx = range_sum(plx, nd.m0, nd.m1 + 1);
#pragma unroll
            for (int r = 0; r < 2 * kPairs; ++r) exact[r] -= cbg * (xt[r] * sl - slx);
            const float2 e2v = make_float2(eps2, eps2), m1 = make_float2(-1.f, -1.f);
            // software pipeline: each thread holds two sources of the next tile
            // in registers while the current tile is computed; one barrier per tile
            constexpr int kPer = kNearTile / kNearThreads;
            double nx[kPer], nl[kPer];
            double nbase = sx[nd.m0];
            auto fetch = [&](int t0) {
#pragma unroll
                for (int i = 0; i < kPer; ++i) {
                    const int j = t0 + threadIdx.x + i * kNearThreads;
                    nx[i] = (j <= nd.m1) ? sx[j] : 0.0;
                    nl[i] = (j <= nd.m1) ? lam[j] : 0.0;
                }
                nbase = sx[t0];
            };
            fetch(nd.m0);
            int buf = 0;
            for (int t0 = nd.m0; t0 <= nd.m1; t0 += kNearTile, buf ^= 1) {
                const int cnt = min(kNearTile, nd.m1 - t0 + 1);
                const double base = nbase;
#pragma unroll
                for (int i = 0; i < kPer; ++i) {
                    const int k = threadIdx.x + i * kNearThreads;
                    // padding sources (q = 0, s = 0) complete the last pair
                    shb[buf][k] = (k < cnt) ? make_float2((float)(nx[i] - base), (float)(0.5 * nl[i]))
                                            : make_float2(0.f, 0.f);
                }
                __syncthreads();
                if (t0 + kNearTile <= nd.m1) fetch(t0 + kNearTile);
                float2 tau2[kPairs], acc2[kPairs], ncmp2[kPairs];
#pragma unroll
                for (int h = 0; h < kPairs; ++h) {
                    tau2[h] = make_float2((float)(xt[2 * h] - base), (float)(xt[2 * h + 1] - base));
                    acc2[h] = make_float2(0.f, 0.f);
                    ncmp2[h] = make_float2(0.f, 0.f);
                }
                const float4* pairs = reinterpret_cast<const float4*>(shb[buf]);
                const int npair = (cnt + 1) >> 1;
#pragma unroll 2
                for (int k = 0; k < npair; ++k) {
                    const float4 e4 = pairs[k];  // two sources per shared-memory load
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        const float2 sx2 = u ? make_float2(e4.z, e4.z) : make_float2(e4.x, e4.x);
                        const float2 qh = u ? make_float2(e4.w, e4.w) : make_float2(e4.y, e4.y);
#pragma unroll
                        for (int h = 0; h < kPairs; ++h) {
                            // differences as FMAs with -1 (exact products): no sign
                            // flips; Kahan with the negated compensation nc = -c
                            const float2 d = __ffma2_rn(sx2, m1, tau2[h]);
                            const float2 r2 = __ffma2_rn(d, d, e2v);
                            const float2 y = make_float2(rsqrt_approx(r2.x), rsqrt_approx(r2.y));
                            const float2 g = __fmul2_rn(d, y);
                            const float2 v = __ffma2_rn(qh, g, ncmp2[h]);
                            const float2 sum = __fadd2_rn(acc2[h], v);
                            const float2 t = __ffma2_rn(acc2[h], m1, sum);
                            ncmp2[h] = __ffma2_rn(t, m1, v);
                            acc2[h] = sum;
                        }
                    }
                }
#pragma unroll
                for (int h = 0; h < kPairs; ++h) {
                    fp[2 * h] += (double)acc2[h].x + (double)ncmp2[h].x;
                    fp[2 * h + 1] += (double)acc2[h].y + (double)ncmp2[h].y;
                }
            }
            __syncthreads();  // the general path and the next leaf reuse shared memory
        } else {
#pragma unroll 1
            for (int h = 0; h < kPairs; ++h)
                near_general2(nd, xp[h], sx, lam, pl, plx, L, band, cbg, eps2, a1, a2, shg, exact + 2 * h, fp + 2 * h,
                              err);
        }
    }
#pragma unroll
    for (int r = 0; r < 2 * kPairs; ++r) {
        const int j = tb0 + threadIdx.x + (2 * h0 + r) * kNearThreads;
        if (j > leaf.m1) continue;
        if (A.parts > 1) A.part[(size_t)part * A.n + j] = exact[r] + fp[r];
        else apply_stage(A.S, A.sidx[j], A.efar[j] + A.norm * (exact[r] + fp[r]));
    }
}

// The parts of shared near lists, in part order, and the stage epilogue.
__global__ void k_near_add(NearArgs A) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= A.n || A.meta[2]) return;
    double s = A.part[j];
    for (int p = 1; p < A.parts; ++p) s += A.part[(size_t)p * A.n + j];
    apply_stage(A.S, A.sidx[j], A.efar[j] + A.norm * s);
}

// One CTA per (leaf, target block, group of kPairs pairs of targets and part of
// the near list).
template <int kPairs>
__global__ void __launch_bounds__(kNearThreads) k_near32(NearArgs A) {
    __shared__ float4 shg[2][kNearTile];       // general path: {s, lambda/2, lambda/2 a1, lambda/2 a2}
    __shared__ __align__(16) float2 shb[2][kNearTile];  // band path: {s, lambda/2}, double-buffered
    constexpr int kGroups = kNearR / 2 / kPairs;
    near_item<kPairs>(A, blockIdx.x, blockIdx.y, blockIdx.z % kGroups * kPairs, blockIdx.z / kGroups, shg, shb);
}

__global__ void k_mul(const double* __restrict__ a, const double* __restrict__ b, int n, double* __restrict__ c) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) c[i] = a[i] * b[i];
}

// near pairs + far cluster terms of this call
__global__ void k_count_work(const TNode* __restrict__ nodes, const int* __restrict__ meta,
                             const int* __restrict__ leaves, const int* __restrict__ far_n,
                             const int* __restrict__ near_list, const int* __restrict__ near_n, int P,
                             double* __restrict__ work) {
    const int l = blockIdx.x * blockDim.x + threadIdx.x;
    if (l >= meta[1] || meta[2]) return;
    const TNode lf = nodes[leaves[l]];
    const double nt = lf.m1 - lf.m0 + 1;
    double ns = 0.0;
    for (int q = 0; q < near_n[l]; ++q) {
        const TNode nd = nodes[near_list[(size_t)l * kNearCap + q]];
        ns += nd.m1 - nd.m0 + 1;
    }
    atomicAdd(&work[0], nt * ns);
    atomicAdd(&work[1], nt * far_n[l] * (double)(P + 1));
}

__global__ void k_copy_meta_error(const int* __restrict__ meta, int* __restrict__ err) {
    if (meta[2]) atomicCAS(err, 0, meta[2]);
}

// k_moments for PP = degree + 1 Chebyshev nodes (2 .. kMaxDegree + 1).
template <bool kFast>
void launch_moments(int PP, int cap_leaves, cudaStream_t st, const TNode* nodes, const int* meta, const int* leaves,
                    const double* consts, const double* halves, const double* sx, const double* lam, int* arrived,
                    double* mom) {
#define FS_MOMENT_CASE(n)                                                                                          \
    case n:                                                                                                       \
        k_moments<n, kFast><<<cap_leaves, kLeafThreads, 0, st>>>(nodes, meta, leaves, consts, halves, sx, lam,    \
                                                                 arrived, mom);                                   \
        break;
    switch (PP) {
        FS_MOMENT_CASE(2) FS_MOMENT_CASE(3) FS_MOMENT_CASE(4) FS_MOMENT_CASE(5) FS_MOMENT_CASE(6)
        FS_MOMENT_CASE(7) FS_MOMENT_CASE(8) FS_MOMENT_CASE(9) FS_MOMENT_CASE(10) FS_MOMENT_CASE(11)
        FS_MOMENT_CASE(12) FS_MOMENT_CASE(13) FS_MOMENT_CASE(14) FS_MOMENT_CASE(15) FS_MOMENT_CASE(16)
        FS_MOMENT_CASE(17)
        default: fail(FS_ERR_ARG, "treecode degree must be 1..16");
    }
#undef FS_MOMENT_CASE
}

class Treecode final : public FieldEngine {
   public:
    Treecode(double L, double eps, double mac, int degree, int max_source, bool fp32_near)
        : L_(L), eps_(eps), mac_(mac), P_(degree), N0_(max_source), fp32_(fp32_near) {
        if (degree < 1 || degree > kMaxDegree) fail(FS_ERR_ARG, "treecode degree must be 1..16");
        if (max_source < 2) fail(FS_ERR_ARG, "treecode max_source must be >= 2");
        // Chebyshev points and barycentric weights exactly as the reference
        // forms them (pi constant and expressions of :790-806), on the host.
        const double pi = 3.14159265358979323846;
        const double h = pi / P_;
        const int PP = P_ + 1;
        std::vector<double> c(2 * (kMaxDegree + 1) + 2 * PP * PP, 0.0);
        for (int i = 0; i <= P_; ++i) c[i] = std::cos(i * h);
        for (int j = 0; j <= P_; ++j) {
            const double dj = (j == 0 || j == P_) ? 0.5 : 1.0;
            c[kMaxDegree + 1 + j] = ((j % 2 == 0) ? 1 : -1) * dj;
        }
        // H[half][k][l]: the parent's Lagrange polynomial k at node l of a half,
        // in barycentric form (the nodes in [-1, 1], a half's at (t - 1) / 2 and
        // (t + 1) / 2)
        for (int half = 0; half < 2; ++half)
            for (int l = 0; l < PP; ++l) {
                const double y = 0.5 * (c[l] + (half ? 1.0 : -1.0));
                double* H = &c[2 * (kMaxDegree + 1) + half * PP * PP];
                int hit = -1;
                double sum = 0.0;
                for (int k = 0; k < PP; ++k) {
                    if (y == c[k]) hit = k;
                    else sum += c[kMaxDegree + 1 + k] / (y - c[k]);
                }
                for (int k = 0; k < PP; ++k)
                    H[k * PP + l] = hit >= 0 ? (k == hit ? 1.0 : 0.0) : c[kMaxDegree + 1 + k] / (y - c[k]) / sum;
            }
        consts_.ensure(c.size());
        FS_CUDA(cudaMemcpy(consts_.p, c.data(), sizeof(double) * c.size(), cudaMemcpyHostToDevice));
        FS_CUDA(cudaStreamSynchronize(nullptr));  // the copy lands before the engine's non-blocking streams read it
        norm_ = std::sqrt(L * L + 4 * eps * eps) / L;
        cbg_ = 1 / std::sqrt(L * L + 4 * eps * eps);
        cells_.init(L, eps);
    }

    int* error_flag() override { return err_.p; }

    double actual_work(cudaStream_t st) override {
        if (last_pairs <= 0) return 0.0;
        FS_CUDA(cudaMemsetAsync(work_.p, 0, 2 * sizeof(double), st));
        k_count_work<<<(cap_leaves_ + 127) / 128, 128, 0, st>>>(nodes_.p, meta_.p, leaves_.p, far_n_.p, near_.p,
                                                                near_n_.p, P_, work_.p);
        FS_LAUNCHED(1);
        double h[2] = {0, 0};
        FS_CUDA(cudaMemcpyAsync(h, work_.p, sizeof(h), cudaMemcpyDeviceToHost, st));
        FS_CUDA(cudaStreamSynchronize(st));
        prof_add_work("treecode_near_pairs", h[0]);
        prof_add_work("treecode_far_terms", h[1]);
        return h[0] + h[1];
    }

    void eval(const double* d_t, int nt, const double* d_s, const double* d_q, int ns, const Stage& stage,
              cudaStream_t st, PairForm) override {
        (void)d_t;
        if (nt != ns) fail(FS_ERR_ARG, "treecode evaluates at the sources: nt must equal ns");
        last_pairs = (double)ns * (double)ns;
        if (ns <= 0) return;
        const int n = ns;
        const int cap_leaves = 2 * (n / N0_ + 1) + 16;
        const int cap_nodes = 2 * kMaxDepth * (n / N0_ + 1) + 64;
        reserve(n, cap_nodes, cap_leaves);
        cap_leaves_ = cap_leaves;
        const int T = 256;
        const int bits = tree_key_bits(n);
        uint32_t *kin = keys_.p, *kout = kin + n, *seen = kout + n;
        FS_CUDA(cudaMemsetAsync(seen, 0, sizeof(uint32_t) * ((n + 31) / 32), st));
        k_tree_keys<<<(n + T - 1) / T, T, 0, st>>>(d_s, d_q, n, L_, std::ldexp(1.0, bits - 1) / L_,
                                                   0xffffffffu >> (32 - bits), kin, iin_.p, vq_.p, nruns_.p);
        size_t tb = cub_.bytes();
        FS_CUDA(cub::DeviceRadixSort::SortPairs(cub_.p, tb, kin, kout, iin_.p, iout_.p, n, 0, bits, st));
        k_tree_gather<<<(n + T - 1) / T, T, 0, st>>>(kout, iout_.p, vq_.p, n, sx_.p, lam_.p, iin_.p, seen,
                                                     runs_.p, nruns_.p);
        k_tree_runs<<<sm_count(), 1024, 0, st>>>(kout, runs_.p, nruns_.p, d_q, n, sx_.p, lam_.p, iin_.p, efar_.p,
                                                 iout_.p);
        const int* sidx = iin_.p;
        FS_LAUNCHED(2);
        const int levels = heap_levels(n, N0_);
        k_heap_splits<<<((1 << levels) + 63) / 64, 64, 0, st>>>(sx_.p, n, levels, heap_.p);
        k_build_tree<<<1, 1024, 0, st>>>(sx_.p, n, N0_, cap_nodes, cap_leaves, nodes_.p, leaves_.p, split_.p,
                                         arrived_.p, heap_.p, levels, meta_.p);
        k_mark_leaves<<<cap_leaves, 256, 0, st>>>(nodes_.p, leaves_.p, meta_.p, leaf_of_.p);
        k_lists<<<(cap_leaves + 3) / 4, 128, 0, st>>>(nodes_.p, leaves_.p, meta_.p, L_, std::sqrt(mac_ * mac_),
                                                          far_.p, far_n_.p, near_.p, near_n_.p, err_.p);
        if (fp32_ && kFastMoments)
            launch_moments<true>(P_ + 1, cap_leaves, st, nodes_.p, meta_.p, leaves_.p, consts_.p, halves(), sx_.p,
                                 lam_.p, arrived_.p, mom_.p);
        else
            launch_moments<false>(P_ + 1, cap_leaves, st, nodes_.p, meta_.p, leaves_.p, consts_.p, halves(), sx_.p,
                                  lam_.p, arrived_.p, mom_.p);
        k_copy_meta_error<<<1, 1, 0, st>>>(meta_.p, err_.p);
        if (cells_take(n)) {
            const TreeView T{nodes_.p, leaves_.p, meta_.p, leaf_of_.p, far_.p, far_n_.p, near_.p, near_n_.p,
                             mom_.p, consts_.p, sx_.p, lam_.p, sidx, n, P_, cap_leaves};
            ProfScope prof("k_tree_cells", st, last_pairs);
            cells_.eval(T, N0_, norm_, stage, st);
            FS_LAUNCHED(7);
        } else if (!fp32_) {
            ProfScope prof("k_far_near64", st, last_pairs);
            auto go = [&](auto lanes) {
                constexpr int kG = decltype(lanes)::value;
                k_far_near64<kG><<<(int)(((long long)n * kG + 127) / 128), 128, 0, st>>>(
                    nodes_.p, meta_.p, leaf_of_.p, far_.p, far_n_.p, near_.p, near_n_.p, mom_.p, consts_.p, sx_.p,
                    lam_.p, sidx, n, P_, L_, eps_, norm_, cbg_, stage);
            };
            if (n < kFarNearWide) go(std::integral_constant<int, 32>{});
            else go(std::integral_constant<int, 8>{});
            FS_LAUNCHED(8);
        } else {
            {
                ProfScope prof("k_far32", st);
                k_far32<<<(n + 127) / 128, 128, 0, st>>>(nodes_.p, meta_.p, leaf_of_.p, far_.p, far_n_.p, mom_.p,
                                                        consts_.p, sx_.p, n, P_, L_, eps_, norm_, cbg_, efar_.p);
            }
            // leaves hold < max_source points: at most ceil(max_source/kNearBlock) target blocks each
            const int nyb = (N0_ + kNearBlock - 1) / kNearBlock;
            scan_f64_inclusive(lam_.p, pl_.p, n, scan_.p, st);
            k_mul<<<(n + T - 1) / T, T, 0, st>>>(lam_.p, sx_.p, n, lx_.p);
            scan_f64_inclusive(lx_.p, plx_.p, n, scan_.p, st);
            // CTAs of two targets per thread, near lists shared by `parts` of
            // them, where CTAs of four would leave SMs idle
            const bool split = n < kNearSplit * kNearBlock * sm_count();
            const int parts = split ? std::max(1, std::min(kNearParts, kNearCtas * sm_count() * (kNearBlock / 2) / n)) : 1;
            if (parts > 1) npart_.ensure((size_t)parts * n);
            const NearArgs A{nodes_.p, meta_.p, leaves_.p, near_.p, near_n_.p, sx_.p, lam_.p, pl_.p, plx_.p, efar_.p,
                             sidx, L_, eps_, cbg_, norm_, stage, err_.p, parts, n, npart_.p};
            ProfScope prof("k_near32", st, last_pairs);
            if (split) k_near32<1><<<dim3(cap_leaves, nyb, 2 * parts), kNearThreads, 0, st>>>(A);
            else k_near32<2><<<dim3(cap_leaves, nyb), kNearThreads, 0, st>>>(A);
            if (parts > 1) {
                k_near_add<<<(n + T - 1) / T, T, 0, st>>>(A);
                FS_LAUNCHED(1);
            }
            FS_LAUNCHED(10);
        }
    }

   private:
    const double* halves() const { return consts_.p + 2 * (kMaxDegree + 1); }
    // Sums through cells (csrc/fs_treecells.cu) where leaves hold many points
    // per cell.  The FP32c form changes over where its FP32 near sums are
    // themselves within 6e-10 of the FP64 treecode (1.7e-9 at 32 points per
    // epsilon, 5e-10 at 126, 4e-11 at 2000), so that E does not step there.
    // The FP64 form sums short boxes pair by pair: a cell that the half period
    // cuts sees the kernel's jump there (48 eps^2 / L^4 in the second derivative),
    // which leaves up to 4.7e-3 (eps / L)^4 of the charge half a period away.
    // Error of E, relative L2 against sums in long double, pair by pair and
    // through cells: 3e-14 and 1.1e-12 at L = 251 epsilon, 3e-14 and 9e-14 at
    // 400, 1e-13 and 5e-14 at 640, 1.5e-13 and 5e-14 at 1571.
    bool cells_take(int n) const {
        if (!cells_.ready()) return false;
        const double per_eps = n * eps_ / L_;  // points per epsilon at uniform density
        return fp32_ ? per_eps >= 128 : per_eps >= 16 && L_ >= kCellBox * eps_;
    }

    void reserve(int n, int cap_nodes, int cap_leaves) {
        keys_.ensure(2 * (size_t)n + (n + 31) / 32);
        runs_.ensure(n / kRunMax + 1);
        nruns_.ensure(1);
        vq_.ensure(n);
        iin_.ensure(n);
        iout_.ensure(n);
        sx_.ensure(n);
        lam_.ensure(n);
        leaf_of_.ensure(n);
        efar_.ensure(n);
        if (fp32_) {
            pl_.ensure(n);
            plx_.ensure(n);
            lx_.ensure(n);
            scan_.ensure(scan_f64_scratch(n));
        }
        nodes_.ensure(cap_nodes);
        leaves_.ensure(cap_leaves);
        meta_.ensure(4);
        work_.ensure(2);
        far_.ensure((size_t)cap_leaves * kFarCap);
        far_n_.ensure(cap_leaves);
        near_.ensure((size_t)cap_leaves * kNearCap);
        near_n_.ensure(cap_leaves);
        split_.ensure(cap_nodes);
        heap_.ensure((size_t)1 << kHeapLevels);
        arrived_.ensure(cap_nodes);
        mom_.ensure((size_t)cap_nodes * (kMaxDegree + 1));
        if (!err_.p) {
            err_.ensure(1);
            FS_CUDA(cudaMemset(err_.p, 0, sizeof(int)));
        }
        size_t need = 0, b = 0;
        FS_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, b, (uint32_t*)nullptr, (uint32_t*)nullptr, (int*)nullptr,
                                                (int*)nullptr, n, 0, tree_key_bits(n)));
        need = std::max(need, b);
        cub_.ensure(need);
    }

    double L_, eps_, mac_;
    int P_, N0_;
    bool fp32_;
    double norm_ = 1, cbg_ = 0;
    DevBuf<uint32_t> keys_;
    DevBuf<double2> vq_;
    DevBuf<int> runs_, nruns_, iin_, iout_, leaf_of_, leaves_, meta_, far_, far_n_, near_, near_n_, split_, heap_, arrived_, err_;
    DevBuf<double> npart_, sx_, lam_, efar_, mom_, consts_, pl_, plx_, lx_, work_, scan_;
    int cap_leaves_ = 0;
    DevBuf<TNode> nodes_;
    TreeCells cells_;
    DevBuf<unsigned char> cub_;
};

}  // namespace

FieldEngine* make_treecode(double L, double eps, double mac, int degree, int max_source, bool fp32_near) {
    return new Treecode(L, eps, mac, degree, max_source, fp32_near);
}

}  // namespace fsb
