// The treecode's sums through cells in FP64 (sm_100a).
//
// The treecode sums its near leaves' sources pair by pair (Call_Ds,
// src/FieldStructure.cpp:963-1020): with leaves of up to 2000 points some ten
// thousand pairs per target, 73% to 95% of an evaluation.  Its kernel is smooth
// on the scale of epsilon, so on cells no wider than epsilon / 1.6 both sides of
// a pair enter through 16 Chebyshev terms to FP64 rounding (csrc/fs_cells.cu).
// The grid of cells is the period's, fixed with its tables for (L, eps); a
// leaf's points take the cells the leaf covers, each (leaf, cell) having a
// slot of its own, so leaf boundaries need not be cell boundaries:
//   k_leaf_slots    cells and slots of every leaf, chunks of kW target cells
//   k_slot_moments  M_s[k] = sum of lambda_j T_k(place in cell), a warp per slot
//   k_chunk_sums    per chunk: sum over the leaf's near leaves' slots of
//                   T^{(I-J)} M, plus the far clusters' terms (Call_BL :904-961,
//                   the same clusters and moments) at the cell's 16 nodes,
//                   transformed to coefficients
//   k_slot_eval     E_j = norm * sum_l A_s[l] T_l(place), stage epilogue
// Near lists, far lists and cluster moments are the treecode's own; only how
// their sums are formed differs (E of long boxes changes by 2e-15 against pair by pair
// in FP64; of boxes below 640 epsilon more: Treecode::cells_take, csrc/fs_tree.cu).
//
// Measured per evaluation, near and far pair by pair against this: 395,523 points
// in FP64 9.8 ms (of 9.97) and 0.12; 6,300,675 points in FP32c 13.4 ms and 0.34
// (slot moments 109, chunk sums 121, evaluation 89 and slots 20 us).
#include <climits>
#include <cmath>

#include "fs_cells.cuh"
#include "fs_tree.cuh"

namespace fsb {

namespace {

constexpr int kP = kCellTerms;
constexpr int kPP = kP * kP;
constexpr int kSlotT = 1024;

// A position of (-L, L) wrapped into [0, L], from the left of 0 into (0, L]: where
// x / L underflows to -0, cell_wrap would give 0, a period away from x's neighbours.
__device__ __forceinline__ double open_wrap(double x, const CellPlan& P) {
    const double w = cell_wrap(x, P.L);
    return x < 0.0 && w == 0.0 ? P.L : w;
}
// Its cell counted without the period: negative left of 0, rising with x.
__device__ __forceinline__ int open_cell(double x, const CellPlan& P) {
    const int c = cell_of(open_wrap(x, P), P);
    return x < 0.0 ? c - P.M : c;
}

// One CTA: leaf l's first cell and slot, the slots' leaves, and the chunks of up
// to `width` cells (a leaf's chunks hold equally many, its last perhaps fewer).
// count: [0] slots, [1] chunks, [2] extra parts of chunks, [3] set by a NaN position
// (sorted to an end of its leaf, it reaches every sum).
__global__ void __launch_bounds__(kSlotT) k_leaf_slots(CellPlan P, TreeView T, int width, int* __restrict__ leaf_c0,
                                                       int* __restrict__ leaf_slot, int* __restrict__ leaf_chunk,
                                                       int* __restrict__ chunk_leaf, int* __restrict__ chunk_c,
                                                       int* __restrict__ chunk_arrived,
                                                       int* __restrict__ count) {
    __shared__ int ws[32], wc[32];
    __shared__ int s_slot, s_chunk, s_nan;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    if (t == 0) s_slot = s_chunk = s_nan = 0;
    const int nl = T.meta[2] ? 0 : T.meta[1];
    __syncthreads();
    for (int base = 0; base < nl; base += kSlotT) {
        const int l = base + t;
        int c0 = 0, nc = 0, nk = 0;
        if (l < nl) {
            const TNode nd = T.nodes[T.leaves[l]];
            const double a = T.sx[nd.m0], e = T.sx[nd.m1];
            c0 = open_cell(a, P);
            nc = max(open_cell(e, P) - c0 + 1, 1);  // (a NaN counts to cell 0)
            if (a != a || e != e) s_nan = 1;
            nk = (nc + width - 1) / width;
        }
        const int even = nk ? (nc + nk - 1) / nk : 0;
        int a = nc, b = nk;  // inclusive scans over the CTA
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, a, o), v = __shfl_up_sync(0xffffffffu, b, o);
            if (lane >= o) {
                a += u;
                b += v;
            }
        }
        if (lane == 31) {
            ws[warp] = a;
            wc[warp] = b;
        }
        __syncthreads();
        if (warp == 0) {
            int u = ws[lane], v = wc[lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int x = __shfl_up_sync(0xffffffffu, u, o), y = __shfl_up_sync(0xffffffffu, v, o);
                if (lane >= o) {
                    u += x;
                    v += y;
                }
            }
            ws[lane] = u;
            wc[lane] = v;
        }
        __syncthreads();
        const int slot = s_slot + (warp ? ws[warp - 1] : 0) + a - nc;
        const int chunk = s_chunk + (warp ? wc[warp - 1] : 0) + b - nk;
        if (l < nl) {
            leaf_c0[l] = c0;
            leaf_slot[l] = slot;
            leaf_chunk[l] = chunk;
            for (int k = 0; k < nk; ++k) {
                chunk_leaf[chunk + k] = l;
                chunk_c[chunk + k] = k * even;
                chunk_arrived[chunk + k] = 0;
            }
        }
        __syncthreads();
        if (t == 0) {
            s_slot += ws[31];
            s_chunk += wc[31];
        }
        __syncthreads();
    }
    if (t == 0) {
        leaf_slot[nl] = s_slot;
        count[0] = s_slot;
        count[1] = s_chunk;
        count[2] = 0;
        count[3] = s_nan;
        leaf_chunk[nl] = s_chunk;
    }
}

// One warp per slot: its points (between two binary searches in the leaf's
// sorted range) over the lanes, 16 moments each, then a shuffle tree.
__global__ void __launch_bounds__(256) k_slot_moments(CellPlan P, TreeView T, const int* __restrict__ leaf_c0,
                                                      const int* __restrict__ leaf_slot, const int* __restrict__ count,
                                                      double* __restrict__ mom) {
    const int lane = threadIdx.x & 31;
    const int s = (blockIdx.x * 256 + threadIdx.x) >> 5;
    if (s >= count[0]) return;
    int lo = 0, hi = T.meta[1] - 1;  // last leaf whose first slot is at most s
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (leaf_slot[mid] <= s) lo = mid;
        else hi = mid - 1;
    }
    const TNode nd = T.nodes[T.leaves[lo]];
    const int oc = leaf_c0[lo] + (s - leaf_slot[lo]);
    auto first = [&](int c) {  // first point of the leaf in cell c or later
        int a = nd.m0, e = nd.m1 + 1;
        while (a < e) {
            const int mid = (a + e) >> 1;
            if (open_cell(T.sx[mid], P) < c) a = mid + 1;
            else e = mid;
        }
        return a;
    };
    const int j0 = first(oc), j1 = first(oc + 1);
    const int c = oc < 0 ? oc + P.M : oc;
    double acc[kP];
#pragma unroll
    for (int k = 0; k < kP; ++k) acc[k] = 0.0;
    for (int j = j0 + lane; j < j1; j += 32) {
        const double xi = fma(open_wrap(T.sx[j], P), P.two_inv_h, -(double)(2 * c + 1));
        double a = T.lam[j], b = a * xi;
        const double x2 = xi + xi;
        acc[0] += a;
        acc[1] += b;
#pragma unroll
        for (int k = 2; k < kP; ++k) {
            const double v = fma(x2, b, -a);
            acc[k] += v;
            a = b;
            b = v;
        }
    }
    double out = 0.0;
#pragma unroll
    for (int k = 0; k < kP; ++k) {
        double v = acc[k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == k) out = v;
    }
    if (lane < kP) mom[(size_t)s * kP + lane] = out;
}

// Cells a chunk of nc of them is summed as.
__host__ __device__ inline int chunk_width(int nc) { return nc <= 4 ? 4 : (nc <= 8 ? 8 : (nc <= 12 ? 12 : 16)); }

__device__ __forceinline__ NearSlots near_leaf(const TreeView& T, int node, const int* __restrict__ leaf_c0,
                                               const int* __restrict__ leaf_slot) {
    const int l = T.leaf_of[T.nodes[node].m0], s0 = leaf_slot[l];
    return NearSlots{s0, leaf_slot[l + 1] - s0, leaf_c0[l]};
}

// One warp per leaf: its near leaves' slots, and in how many parts its chunks' near
// sums are formed.  A step is one pass of chunk_width offsets over the cells;
// kSteps of them are a part, kPartsMax parts at most: leaves in thinly filled
// places cover ten times the cells of others, and the launch would end on their
// chunks (71 steps where the median has 12).  Parts but the first join a list.
constexpr int kSteps = 16, kPartsMax = 4;
__global__ void __launch_bounds__(128) k_near_slots(TreeView T, const int* __restrict__ leaf_c0,
                                                    const int* __restrict__ leaf_slot,
                                                    const int* __restrict__ leaf_chunk, NearSlots* __restrict__ near,
                                                    int2* __restrict__ leaf_steps, int2* __restrict__ extra,
                                                    int* __restrict__ count) {
    const int l = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (T.meta[2] || l >= T.meta[1]) return;
    const int cells = leaf_slot[l + 1] - leaf_slot[l], nk = leaf_chunk[l + 1] - leaf_chunk[l], nn = T.near_n[l];
    const int W = chunk_width((cells + nk - 1) / nk);
    int steps = 0;
    for (int q = lane; q < nn; q += 32) {
        const NearSlots Q = near_leaf(T, T.near_list[(size_t)l * kNearCap + q], leaf_c0, leaf_slot);
        near[(size_t)l * kNearCap + q] = Q;
        steps += (Q.n + W - 1 + W - 1) / W;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) steps += __shfl_xor_sync(0xffffffffu, steps, o);
    const int parts = min(kPartsMax, max(1, (steps + kSteps - 1) / kSteps));
    if (lane) return;
    leaf_steps[l] = make_int2(steps, parts);
    if (parts > 1) {
        int at = atomicAdd(&count[2], nk * (parts - 1));
        for (int k = 0; k < nk; ++k)
            for (int p = 1; p < parts; ++p) extra[at++] = make_int2(leaf_chunk[l] + k, p);
    }
}

// Steps [g0, g1) of what a chunk takes from its near leaves' slots, kW cells at a
// time: thread (k, l) holds moment k's share of local coefficient l; along a near
// leaf's slots one table entry serves all cells.  near's c0: the cell distance of a
// near leaf's last slot from the chunk's first cell.
template <int kW>
__device__ __forceinline__ void near_slots(const NearSlots* near, int nn, int g0, int g1, int M,
                                           const double* __restrict__ tab, const double* __restrict__ mom,
                                           double (*red)[kP]) {
    const int t = threadIdx.x, l = t & 15, k = t >> 4;
    double acc[kW];
#pragma unroll
    for (int i = 0; i < kW; ++i) acc[i] = 0.0;
    int g = 0;  // first step of near leaf q
    for (int q = 0; q < nn && g < g1; ++q) {
        const NearSlots Q = near[q];
        const int S = Q.n, all = (S + kW - 1 + kW - 1) / kW;  // offsets 0 .. S + kW - 2
        const int a = max(g0 - g, 0) * kW, e = min(g1 - g, all) * kW;
        g += all;
        if (a >= e) continue;
        const double* W = mom + (size_t)Q.slot * kP + k;
        const int m = Q.c0;
        double w[kW];  // W(e) in place e mod kW, as in slide (csrc/fs_cells.cu)
#pragma unroll
        for (int i = 0; i < kW; ++i) w[i] = 0.0;
        if (a > 0) {
#pragma unroll
            for (int i = 1; i < kW; ++i) {
                const int j = S - 1 - a + i;
                w[i] = j >= 0 && j < S ? W[(size_t)j * kP] : 0.0;
            }
        }
        for (int o = a; o < e; o += kW) {
            double tv[kW], nv[kW];
#pragma unroll
            for (int u = 0; u < kW; ++u) {
                int at = m + o + u;  // below 4 M
                at -= at >= 2 * M ? 2 * M : 0;
                at -= at >= M ? M : 0;
                tv[u] = tab[(size_t)at * kPP + t];
                const int j = S - 1 - o - u;
                nv[u] = j >= 0 ? W[(size_t)j * kP] : 0.0;
            }
#pragma unroll
            for (int u = 0; u < kW; ++u) {
                w[(kW - u) % kW] = nv[u];
#pragma unroll
                for (int i = 0; i < kW; ++i) acc[i] = fma(tv[u], w[(i - u + kW) % kW], acc[i]);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < kW; ++i) red[k * kW + i][l] = acc[i];
}

// A chunk of up to kMax cells of a leaf, or one part of its near sums, per turn of
// a CTA (parts but the first before all chunks: they are the longest chunks').  Far (part 0): the chunk's cells have 16 nodes each, and the threads
// share the far clusters' terms at a node among as many as there are threads per
// node; clusters come through shared memory, kFarTile at a time.  Near:
// near_slots, as many cells wide as the chunk needs.  The last part to be done adds
// them up in their order.  What bounds it: the latency of a step's table and moment
// reads (1.5 us; the FP64 pipe needs 18 us of the 76 below).  395,523 points
// (20 cells a leaf, up to 160): 121 -> 76 us and 7 for k_near_slots, against chunks
// of fixed width with each list entry's own chain of reads, all of a chunk's steps
// in one CTA.  Chunks of four cells (leaves of three, 6.3 million points) stay
// whole: 136 -> 121 us; in parts of 12 steps 131, of 40 steps 126.
constexpr int kFarTile = 32;
struct ChunkWork {
    const int *leaf_c0, *leaf_slot, *chunk_leaf, *chunk_c;
    const NearSlots* near;
    const int2 *leaf_steps, *extra;
    int *arrived, *count;
    double* part;  // kPartsMax * kMax * kP per chunk
};
template <int kMax>
__global__ void __launch_bounds__(kPP, kMax > 4 ? 2 : 5) k_chunk_sums(CellPlan P, TreeView T, ChunkWork X,
                                                                      const double* __restrict__ tab,
                                                                      const double* __restrict__ mom,
                                                                      double* __restrict__ loc) {
    __shared__ double red[kP * kMax][kP];
    __shared__ double far[kPP];
    __shared__ double cx[kFarTile * (kMaxDegree + 1)], cm[kFarTile * (kMaxDegree + 1)];
    __shared__ NearSlots near[kNearCap];
    __shared__ int s_before;
    const int t = threadIdx.x, l = t & 15, i = t >> 4;
    const double* C = tab + (size_t)P.M * kPP;  // node a's share of coefficient l at [a][l], then the nodes
    constexpr bool kSplit = kMax > 4;
    const int nextra = kSplit ? X.count[2] : 0, nitems = nextra + X.count[1], M = P.M, PP = T.P + 1;
    for (int item = blockIdx.x; item < nitems; item += gridDim.x) {
        if (kSplit) __syncthreads();  // the last turn's shared sums have been read
        const int2 it = item < nextra ? X.extra[item] : make_int2(item - nextra, 0);
        const int chunk = it.x, part = it.y;
        const int leaf = X.chunk_leaf[chunk], cc = X.chunk_c[chunk];
        const int oc0 = X.leaf_c0[leaf] + cc;
        const int first = X.leaf_slot[leaf], cells = X.leaf_slot[leaf + 1] - first;
        const int nk = (cells + kMax - 1) / kMax, even = (cells + nk - 1) / nk, nc = min(even, cells - cc);
        const int nn = T.near_n[leaf], W = chunk_width(even);
        const int2 steps = kSplit ? X.leaf_steps[leaf] : make_int2(INT_MAX, 1);
        if (t < nn) {
            NearSlots Q = kSplit ? X.near[(size_t)leaf * kNearCap + t]
                                 : near_leaf(T, T.near_list[(size_t)leaf * kNearCap + t], X.leaf_c0, X.leaf_slot);
            Q.c0 = (oc0 - Q.c0 - (Q.n - 1)) % M;  // cell distance of its last slot
            Q.c0 += Q.c0 < 0 ? M : 0;
            near[t] = Q;
        }
        int cp = 1;  // cells of the far terms' thread map: a power of two
        while (cp < nc) cp *= 2;
        const int nodes = cp * kP;
        if (part == 0) {
            const int nf = T.far_n[leaf];
            const int sh = kPP / nodes, node = t % nodes, ps = t / nodes;
            const double x = (oc0 + node / kP + 0.5 + 0.5 * C[kPP + node % kP]) * P.h;
            const double e2 = P.eps * P.eps, invL = 1.0 / P.L;
            double s = 0.0;
            for (int base = 0; base < nf; base += kFarTile) {
                const int terms = min(kFarTile, nf - base) * PP;
                __syncthreads();
                for (int z = t; z < terms; z += kPP) {
                    const int f = z / PP, j = z - f * PP;
                    const int fi = T.far_list[(size_t)leaf * kFarCap + base + f];
                    const double x0 = T.nodes[fi].x0, w = 0.5 * (T.nodes[fi].x1 - x0);
                    cx[z] = fma(T.consts[j] + 1.0, w, x0);
                    cm[z] = T.mom[(size_t)fi * (kMaxDegree + 1) + j];
                }
                __syncthreads();
                if (node < nc * kP) {
#pragma unroll 4
                    for (int z = ps; z < terms; z += sh) {
                        double d = x - cx[z];
                        d -= P.L * rint(d * invL);
                        const double r = fma(d, d, e2);
                        double y;
                        asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(r));
                        const double e = fma(-r * y, y, 1.0);
                        y = fma(y * e, fma(e, 0.375, 0.5), y);
                        s = fma(cm[z], d * fma(0.5, y, -P.cbg), s);
                    }
                }
            }
            far[t] = s;
        }
        __syncthreads();
        int g0 = 0, g1 = INT_MAX;
        if (kSplit) {
            g0 = (int)((long long)steps.x * part / steps.y);
            g1 = (int)((long long)steps.x * (part + 1) / steps.y);
        }
        if (kMax == 4 || W == 4) near_slots<4>(near, nn, g0, g1, M, tab, mom, red);
        if (kMax > 4) {
            if (W == 8) near_slots<8>(near, nn, g0, g1, M, tab, mom, red);
            if (W == 12) near_slots<12>(near, nn, g0, g1, M, tab, mom, red);
            if (W == 16) near_slots<16>(near, nn, g0, g1, M, tab, mom, red);
        }
        __syncthreads();
        double s = 0.0;
        if (i < nc) {
#pragma unroll
            for (int kk = 0; kk < kP; ++kk) s += red[kk * W + i][l];
            if (part == 0) {
#pragma unroll
                for (int a = 0; a < kP; ++a) {
                    double f = far[i * kP + a];
                    for (int p = nodes; p < kPP; p += nodes) f += far[p + i * kP + a];
                    s = fma(C[a * kP + l], f, s);
                }
            }
        }
        if (kSplit && steps.y > 1) {
            double* out = X.part + (size_t)chunk * kPartsMax * kMax * kP + t;
            if (i < nc) out[part * kMax * kP] = s;
            __threadfence();
            __syncthreads();
            if (t == 0) s_before = atomicAdd(&X.arrived[chunk], 1);
            __syncthreads();
            if (s_before != steps.y - 1) continue;
            __threadfence();
            if (i < nc) {
                s = 0.0;
                for (int p = 0; p < steps.y; ++p) s += __ldcg(&out[p * kMax * kP]);
            }
        }
        if (i < nc) loc[(size_t)(first + cc + i) * kP + l] = s;
        if (!kSplit) return;  // as many CTAs as chunks
    }
}

// Node a's share of coefficient l, [a][l], then the nodes themselves.
__global__ void __launch_bounds__(kPP) k_node_table(double* __restrict__ out) {
    const int t = threadIdx.x, a = t >> 4, l = t & 15;
    out[t] = cospi((a + 0.5) * l / kP) * (l ? 2.0 : 1.0) / kP;
    if (t < kP) out[kPP + t] = cospi((t + 0.5) / kP);
}

__global__ void __launch_bounds__(256) k_slot_eval(CellPlan P, TreeView T, const int* __restrict__ leaf_c0,
                                                   const int* __restrict__ leaf_slot, const int* __restrict__ count,
                                                   const double* __restrict__ loc, double norm, Stage S) {
    const int j = blockIdx.x * 256 + threadIdx.x;
    if (j >= T.n || T.meta[2]) return;
    const double x = T.sx[j];
    const int l = T.leaf_of[j];
    const int oc = open_cell(x, P);
    const int slot = leaf_slot[l] + min(max(oc - leaf_c0[l], 0), leaf_slot[l + 1] - leaf_slot[l] - 1);
    const int c = oc < 0 ? oc + P.M : oc;
    const double xi = fma(open_wrap(x, P), P.two_inv_h, -(double)(2 * c + 1));
    const double E = norm * cheb_sum(loc + (size_t)slot * kP, xi);
    apply_stage(S, T.sidx[j], count[3] ? nan("") : E);
}

// The stage epilogue of fields formed in another order: a point's stage arrays are
// six to eight scattered sectors from k_slot_eval, which at 6.3 million points (twice
// the L2) takes 314 us on average over a step's stages (482 the last); E alone
// scattered 75 and this 62 to 88.  Without a tree there is no E, and the state stays.
__global__ void __launch_bounds__(256) k_apply_stage(TreeView T, const double* __restrict__ E, Stage S) {
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i < T.n && !T.meta[2]) apply_stage(S, i, E[i]);
}
constexpr int kApart = 1 << 20;  // points from which the stage arrays leave the L2

}  // namespace

bool TreeCells::init(double L, double eps) {
    if (!cell_plan(L, eps, &plan_)) {
        plan_.M = 0;
        return false;
    }
    return true;
}

void TreeCells::eval(const TreeView& T, int max_source, double norm, const Stage& S, cudaStream_t st) {
    // positions span (-L, L): a leaf boundary adds at most one slot
    const int cap_slots = 2 * plan_.M + T.cap_leaves;
    // target cells per chunk: a leaf of the mean width has M max_source / n
    // cells or fewer; four cells waste least where leaves have two or three
    // (6.3 million points), sixteen reuse a table entry most where they have
    // twenty and more (400,000)
    const bool wide = (double)plan_.M * max_source > 8.0 * T.n;
    const int width = wide ? 16 : 4;
    const int cap_chunks = cap_slots / width + T.cap_leaves;
    leaf_c0_.ensure(T.cap_leaves + 1);
    leaf_chunk_.ensure(T.cap_leaves + 1);
    arrived_.ensure(cap_chunks);
    if (wide) {
        near_.ensure((size_t)T.cap_leaves * kNearCap);
        leaf_steps_.ensure(T.cap_leaves);
        extra_.ensure((size_t)cap_chunks * (kPartsMax - 1));
        part_.ensure((size_t)cap_chunks * kPartsMax * width * kP);
    }
    leaf_slot_.ensure(T.cap_leaves + 1);
    chunk_leaf_.ensure(cap_chunks);
    chunk_c_.ensure(cap_chunks);
    count_.ensure(4);
    mom_.ensure((size_t)cap_slots * kP);
    loc_.ensure((size_t)cap_slots * kP);
    if (!tab_.p) {
        // once: it depends on L and epsilon alone.  On this stream, without a wait:
        // evaluations of an engine share its buffers and come one after another,
        // whatever their streams
        tab_.ensure((size_t)plan_.M * kPP + kPP + kP);
        cell_offset_table(plan_, tab_.p, st);
        k_node_table<<<1, kPP, 0, st>>>(tab_.p + (size_t)plan_.M * kPP);
        FS_LAUNCHED(1);
    }
    k_leaf_slots<<<1, kSlotT, 0, st>>>(plan_, T, width, leaf_c0_.p, leaf_slot_.p, leaf_chunk_.p, chunk_leaf_.p,
                                       chunk_c_.p, arrived_.p, count_.p);
    if (wide) k_near_slots<<<(T.cap_leaves + 3) / 4, 128, 0, st>>>(T, leaf_c0_.p, leaf_slot_.p, leaf_chunk_.p, near_.p,
                                                         leaf_steps_.p, extra_.p, count_.p);
    k_slot_moments<<<(cap_slots + 7) / 8, 256, 0, st>>>(plan_, T, leaf_c0_.p, leaf_slot_.p, count_.p, mom_.p);
    const ChunkWork X{leaf_c0_.p, leaf_slot_.p, chunk_leaf_.p, chunk_c_.p, near_.p, leaf_steps_.p, extra_.p,
                      arrived_.p, count_.p, part_.p};
    if (wide) k_chunk_sums<16><<<cap_chunks, kPP, 0, st>>>(plan_, T, X, tab_.p, mom_.p, loc_.p);
    else k_chunk_sums<4><<<cap_chunks, kPP, 0, st>>>(plan_, T, X, tab_.p, mom_.p, loc_.p);
    const bool apart = S.kind != STAGE_STORE && T.n >= kApart;
    Stage field;
    if (apart) {
        e_.ensure(T.n);
        field.out = e_.p;
    }
    k_slot_eval<<<(T.n + 255) / 256, 256, 0, st>>>(plan_, T, leaf_c0_.p, leaf_slot_.p, count_.p, loc_.p, norm,
                                                   apart ? field : S);
    if (apart) {
        k_apply_stage<<<(T.n + 255) / 256, 256, 0, st>>>(T, e_.p, S);
        FS_LAUNCHED(1);
    }
    FS_LAUNCHED(wide ? 5 : 4);
}

}  // namespace fsb
