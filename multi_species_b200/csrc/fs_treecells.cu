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
// their sums are formed differs (E changes by 2e-15 against pair by pair in FP64).
//
// Measured per evaluation: 395,523 points in FP64 9.97 -> 0.29 ms (near and far
// pair by pair 9.8 ms of it); 6,300,675 points in FP32c 18.6 -> 2.4 ms (near 12.3
// and far 1.1 ms became 0.36 ms: slot moments 107, chunk sums 135, evaluation 89
// and slots 22 us).
#include <cmath>

#include "fs_cells.cuh"
#include "fs_tree.cuh"

namespace fsb {

namespace {

constexpr int kP = kCellTerms;
constexpr int kPP = kP * kP;
constexpr int kSlotT = 1024;

// Cell of a position of (-L, L) counted without the period: negative left of 0.
__device__ __forceinline__ int open_cell(double x, const CellPlan& P) {
    const int c = cell_of(cell_wrap(x, P.L), P);
    return x < 0.0 ? c - P.M : c;
}

// One CTA: leaf l's first cell and slot, the slots' leaves, and the chunks of
// `width` cells.  count: [0] slots, [1] chunks.
__global__ void __launch_bounds__(kSlotT) k_leaf_slots(CellPlan P, TreeView T, int width, int* __restrict__ leaf_c0,
                                                       int* __restrict__ leaf_slot, int* __restrict__ chunk_leaf,
                                                       int* __restrict__ chunk_c, int* __restrict__ count) {
    __shared__ int ws[32], wc[32];
    __shared__ int s_slot, s_chunk;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    if (t == 0) s_slot = s_chunk = 0;
    const int nl = T.meta[2] ? 0 : T.meta[1];
    __syncthreads();
    for (int base = 0; base < nl; base += kSlotT) {
        const int l = base + t;
        int c0 = 0, nc = 0, nk = 0;
        if (l < nl) {
            const TNode nd = T.nodes[T.leaves[l]];
            c0 = open_cell(T.sx[nd.m0], P);
            nc = open_cell(T.sx[nd.m1], P) - c0 + 1;
            nk = (nc + width - 1) / width;
        }
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
            for (int k = 0; k < nk; ++k) {
                chunk_leaf[chunk + k] = l;
                chunk_c[chunk + k] = k * width;
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
        const double xi = fma(cell_wrap(T.sx[j], P.L), P.two_inv_h, -(double)(2 * c + 1));
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

// One CTA per chunk of kW cells of a leaf.  Near: thread (k, l) holds moment
// k's share of local coefficient l for the kW cells; along a near leaf's slots
// one table entry serves all of them.  Far: thread
// (part, node) sums a quarter (kW = 4) or half (8) of the far clusters at one
// of the chunk's 16 kW nodes.
template <int kW>
__global__ void __launch_bounds__(kPP) k_chunk_sums(CellPlan P, TreeView T, const double* __restrict__ tab,
                                                    const int* __restrict__ leaf_c0, const int* __restrict__ leaf_slot,
                                                    const int* __restrict__ chunk_leaf,
                                                    const int* __restrict__ chunk_c, const int* __restrict__ count,
                                                    const double* __restrict__ mom, double* __restrict__ loc) {
    constexpr int kParts = kPP / (kW * kP);
    __shared__ double red[kP][kW][kP];
    __shared__ double far[kParts][kW * kP];
    __shared__ double C[kP][kP];
    if ((int)blockIdx.x >= count[1]) return;
    const int t = threadIdx.x, l = t & 15, k = t >> 4;
    C[k][l] = cospi((k + 0.5) * l / kP) * (l ? 2.0 : 1.0) / kP;  // node k's share of coefficient l
    const int leaf = chunk_leaf[blockIdx.x], cc = chunk_c[blockIdx.x];
    const int oc0 = leaf_c0[leaf] + cc;
    const int slot0 = leaf_slot[leaf] + cc, nc = min(kW, leaf_slot[leaf + 1] - slot0);
    // far
    {
        const int node = t % (kW * kP), part = t / (kW * kP);
        const double x = (oc0 + node / kP + 0.5 + 0.5 * cospi((node % kP + 0.5) / kP)) * P.h;
        const double e2 = P.eps * P.eps, invL = 1.0 / P.L;
        double s = 0.0;
        const int nf = T.far_n[leaf];
        for (int f = part; f < nf; f += kParts) {
            const int fi = T.far_list[(size_t)leaf * kFarCap + f];
            const double x0 = T.nodes[fi].x0, w = 0.5 * (T.nodes[fi].x1 - x0);
            const double* m = T.mom + (size_t)fi * (kMaxDegree + 1);
            for (int j = 0; j <= T.P; ++j) {
                double d = x - fma(T.consts[j] + 1.0, w, x0);
                d -= P.L * rint(d * invL);
                const double r = fma(d, d, e2);
                double y;
                asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(r));
                const double e = fma(-r * y, y, 1.0);
                y = fma(y * e, fma(e, 0.375, 0.5), y);
                s = fma(m[j], d * fma(0.5, y, -P.cbg), s);
            }
        }
        far[part][node] = s;
    }
    // near
    double acc[kW];
#pragma unroll
    for (int i = 0; i < kW; ++i) acc[i] = 0.0;
    const int nn = T.near_n[leaf], M = P.M;
    for (int q = 0; q < nn; ++q) {
        const int ql = T.leaf_of[T.nodes[T.near_list[(size_t)leaf * kNearCap + q]].m0];
        const int s0 = leaf_slot[ql], S = leaf_slot[ql + 1] - s0;
        // offsets o = 0 .. S + kW - 2: cell distance oc0 - c0 - (S - 1) + o
        int m = (oc0 - leaf_c0[ql] - (S - 1)) % P.M;
        m += m < 0 ? P.M : 0;
        const double* W = mom + (size_t)s0 * kP + k;
        const int n = (S + kW - 1 + kW - 1) / kW * kW;
        double w[kW];  // W(e) in place e mod kW, as in slide (csrc/fs_cells.cu)
#pragma unroll
        for (int i = 0; i < kW; ++i) w[i] = 0.0;
        for (int o = 0; o < n; o += kW) {
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
    for (int i = 0; i < kW; ++i) red[k][i][l] = acc[i];
    __syncthreads();
    if (t < kW * kP) {
        const int i = t / kP;
        double s = 0.0;
#pragma unroll
        for (int kk = 0; kk < kP; ++kk) s += red[kk][i][l];
#pragma unroll
        for (int a = 0; a < kP; ++a) {
            double f = far[0][i * kP + a];
#pragma unroll
            for (int p = 1; p < kParts; ++p) f += far[p][i * kP + a];
            s = fma(C[a][l], f, s);
        }
        if (i < nc) loc[(size_t)(slot0 + i) * kP + l] = s;
    }
}

__global__ void __launch_bounds__(256) k_slot_eval(CellPlan P, TreeView T, const int* __restrict__ leaf_c0,
                                                   const int* __restrict__ leaf_slot, const double* __restrict__ loc,
                                                   double norm, Stage S) {
    const int j = blockIdx.x * 256 + threadIdx.x;
    if (j >= T.n || T.meta[2]) return;
    const double x = T.sx[j];
    const int l = T.leaf_of[j];
    const int oc = open_cell(x, P);
    const int slot = leaf_slot[l] + min(max(oc - leaf_c0[l], 0), leaf_slot[l + 1] - leaf_slot[l] - 1);
    const int c = oc < 0 ? oc + P.M : oc;
    const double xi = fma(cell_wrap(x, P.L), P.two_inv_h, -(double)(2 * c + 1));
    apply_stage(S, T.sidx[j], norm * cheb_sum(loc + (size_t)slot * kP, xi));
}

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
    leaf_slot_.ensure(T.cap_leaves + 1);
    chunk_leaf_.ensure(cap_chunks);
    chunk_c_.ensure(cap_chunks);
    count_.ensure(2);
    mom_.ensure((size_t)cap_slots * kP);
    loc_.ensure((size_t)cap_slots * kP);
    if (!tab_.p) {
        // once, before any (non-blocking) stream reads it: it depends on L and
        // epsilon alone
        tab_.ensure((size_t)plan_.M * kPP);
        cell_offset_table(plan_, tab_.p, nullptr);
        FS_CUDA(cudaStreamSynchronize(nullptr));
    }
    k_leaf_slots<<<1, kSlotT, 0, st>>>(plan_, T, width, leaf_c0_.p, leaf_slot_.p, chunk_leaf_.p, chunk_c_.p, count_.p);
    k_slot_moments<<<(cap_slots + 7) / 8, 256, 0, st>>>(plan_, T, leaf_c0_.p, leaf_slot_.p, count_.p, mom_.p);
    if (wide)
        k_chunk_sums<16><<<cap_chunks, kPP, 0, st>>>(plan_, T, tab_.p, leaf_c0_.p, leaf_slot_.p, chunk_leaf_.p,
                                                     chunk_c_.p, count_.p, mom_.p, loc_.p);
    else
        k_chunk_sums<4><<<cap_chunks, kPP, 0, st>>>(plan_, T, tab_.p, leaf_c0_.p, leaf_slot_.p, chunk_leaf_.p,
                                                    chunk_c_.p, count_.p, mom_.p, loc_.p);
    k_slot_eval<<<(T.n + 255) / 256, 256, 0, st>>>(plan_, T, leaf_c0_.p, leaf_slot_.p, loc_.p, norm, S);
    FS_LAUNCHED(4);
}

}  // namespace fsb
