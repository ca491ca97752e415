// Periodic direct sum through cell expansions in FP64 (sm_100a).
//
// Same field as E_MQ_DirectSum (src/FieldStructure.cpp:106-156),
//   E_i = sum_j q_j G(x_i - x_j),  G(d) = d / (2 sqrt(d^2 + eps^2)) - c d,
//   c = 1 / sqrt(L^2 + 4 eps^2),  d wrapped to [-L/2, L/2].
// G is smooth on the scale of eps (its nearest singularities are d = +-i eps),
// so on cells no wider than eps / 1.6 its dependence on the source's and on
// the target's place in their cells is a polynomial to FP64 rounding: with
// half-width a the Chebyshev series converges like rho^-n, rho = eps/a +
// sqrt((eps/a)^2 + 1) = 6.5: 16 terms leave 6.5^-16 = 1e-13 of a pair's charge at
// most, 3e-14 as formed (within a cell; 4e-15 from the second neighbour on).  The
// sum over all pairs becomes
//   k_cell_moments / k_cell_gather  M_J[k] = sum_{j in J} q_j T_k(xi_j)
//   k_cell_pairs                    A_I[l] = sum_J sum_k T^{(I-J)}[k][l] M_J[k]
//   k_cell_eval                     E_i = sum_l A_I[l] T_l(xi_i)
// O(N) work for the points and (cells x 16)-sized pair sums between them,
// where the pairwise sum is O(N^2): at 525,825 points of the two-stream box
// (2,528 cells) one evaluation takes 4e7 FP64 pair terms in place of 2.8e11,
// 84 us in place of 42.1 ms by the pairwise kernel.  Its error there is 1e-15 of
// E, the pairwise kernel's 1e-11.
//
// The pair sums run on two levels.  16 cells form a group; the near groups
// (-1, 0, +1) and the group half a period away, whose pairs change their
// periodic image, interact cell by cell, the rest group by group.  Of those the
// nearest are a group's width apart, 10 eps: three half-widths from a group's
// middle to the other's points, rho = 5.8, and 5.8^-16 = 6e-13 of what of a term is
// not a polynomial (eps^2 / d^2 of it), 5.4e-14 of the charge as formed.  G and G'
// are continuous at d = +-L/2 and G'' jumps by 48 eps^2 / L^4 there; only the one
// cell pair per target cell that straddles it sees the jump, which leaves of that
// cell's charge up to 1.3e-10 at L = 33 eps, where the pairwise FP32 terms round by
// as much, 8e-13 at 251 and 2e-14 at 640.  Measured relative L2 in E: 1e-14 to 4e-13.
//
// T^{(m)} depends on L and eps alone: it is formed once per (L, eps).  Every
// sum has a fixed association, so results are a function of the inputs.
#include <cub/cub.cuh>

#include <cmath>

#include "fs_bulk.cuh"
#include "fs_cells.cuh"

namespace fsb {

namespace {

constexpr int kP = kCellTerms;    // Chebyshev terms of a cell
constexpr int kC = kCellGroup;    // cells of a group
constexpr int kPP = kP * kP;
constexpr int kNearOff = 64;      // fine offsets -32 .. 31 (-32 unused: zero)
constexpr int kSeamOff = 32;      // fine offsets M/2 - 16 .. M/2 + 15 (M/2 - 16 unused: zero)
constexpr int kSub = 16;          // sorted points of one partial moment
constexpr int kFarGroups = 4;     // target groups of one far item
constexpr int kPairT = 512;       // threads of k_cell_pairs
static_assert(kP == 16 && kC == 16, "thread maps below");

// Bound of the waits on the moment copies (fs_debug_set_wait_limits).
__device__ long long g_cell_polls = kMbarPolls;

__global__ void k_cell_keys(CellPlan P, const double* __restrict__ x, int n, uint32_t* __restrict__ key,
                            int* __restrict__ idx) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    key[i] = (uint32_t)cell_of(cell_wrap(x[i], P.L), P);
    idx[i] = i;
}

// Partial moments of 256 points in cell order per CTA: each thread forms q T_k
// of its point in shared memory, then thread (k, s) sums the 16 points of
// sub-chunk s in order, one partial per cell met.  Sub-chunk index and cell
// both only grow along the sorted points, so (sub-chunk + cell) numbers the
// partials without a scan.  Balanced whatever the points' distribution: a
// thread's work does not depend on how many points a cell holds.  Also writes
// each cell's first sorted point.  kSorted: x (wrapped) and q are in order
// themselves, skey and sidx are not read; a NaN at the end counts to cell 0.
template <bool kSorted>
__global__ void __launch_bounds__(256) k_cell_moments(CellPlan P, const uint32_t* __restrict__ skey,
                                                      const int* __restrict__ sidx, const double* __restrict__ x,
                                                      const double* __restrict__ q, int n, int* __restrict__ start,
                                                      double* __restrict__ part) {
    __shared__ double val[kP][257];
    __shared__ int sk[256];
    const int t = threadIdx.x, i = blockIdx.x * 256 + t;
    int key = P.M;  // beyond the last point
    if (i < n) {
        key = kSorted ? cell_of(x[i], P) : (int)skey[i];
        const int prev = i > 0 ? (kSorted ? cell_of(x[i - 1], P) : (int)skey[i - 1]) : -1;
        for (int c = prev + 1; c <= key; ++c) start[c] = i;
        if (i == n - 1)
            for (int c = key + 1; c <= P.M; ++c) start[c] = n;
        const int id = kSorted ? i : sidx[i];
        const double w = kSorted ? x[id] : cell_wrap(x[id], P.L), qi = q[id];
        const double xi = fma(w, P.two_inv_h, -(double)(2 * key + 1));
        double a = qi, b = qi * xi;
        const double x2 = xi + xi;
        val[0][t] = a;
        val[1][t] = b;
#pragma unroll
        for (int k = 2; k < kP; ++k) {
            const double c = fma(x2, b, -a);
            val[k][t] = c;
            a = b;
            b = c;
        }
    }
    sk[t] = key;
    __syncthreads();
    const int k = t & (kP - 1), s = t / kP;
    const int g = blockIdx.x * (256 / kSub) + s;
    double acc = 0.0;
    int cur = sk[s * kSub];
#pragma unroll
    for (int j = 0; j < kSub; ++j) {
        const int c = sk[s * kSub + j];
        if (c != cur) {
            if (cur < P.M) part[(size_t)(g + cur) * kP + k] = acc;
            acc = 0.0;
            cur = c;
        }
        if (c < P.M) acc += val[k][s * kSub + j];
    }
    if (cur < P.M) part[(size_t)(g + cur) * kP + k] = acc;
}

// One CTA per group: its cells' moments from their partials (four interleaved
// slices per moment, added in slice order), then the group's moments through
// T_k(child's place in the group) = sum_l B[child][k][l] T_l(place in child).
__global__ void __launch_bounds__(1024) k_cell_gather(CellPlan P, const int* __restrict__ start,
                                                      const double* __restrict__ part,
                                                      const double* __restrict__ child, double* __restrict__ mom,
                                                      double* __restrict__ momc) {
    __shared__ double sh[4][kC][kP];
    __shared__ double m[kC][kP];
    const int t = threadIdx.x, k = t & 15, c = (t >> 4) & 15, slice = t >> 8;
    const int J = blockIdx.x * kC + c;
    const int a = start[J], e = start[J + 1];
    double s = 0.0;
    if (e > a) {
        const int g1 = (e - 1) / kSub;
#pragma unroll 4
        for (int g = a / kSub + slice; g <= g1; g += 4) s += part[(size_t)(g + J) * kP + k];
    }
    sh[slice][c][k] = s;
    __syncthreads();
    if (slice == 0) {
        const double v = (sh[0][c][k] + sh[1][c][k]) + (sh[2][c][k] + sh[3][c][k]);
        m[c][k] = v;
        mom[(size_t)J * kP + k] = v;
    }
    __syncthreads();
    // thread (k, c, slice): child c's part of group moment k over four terms
    double v = 0.0;
    const double* B = child + ((size_t)c * kP + k) * kP + slice * 4;
#pragma unroll
    for (int l = 0; l < 4; ++l) v = fma(B[l], m[c][slice * 4 + l], v);
    sh[slice][c][k] = v;
    __syncthreads();
    if (t < kP) {
        double u = 0.0;
#pragma unroll
        for (int cc = 0; cc < kC; ++cc) u += (sh[0][cc][t] + sh[1][cc][t]) + (sh[2][cc][t] + sh[3][cc][t]);
        momc[(size_t)blockIdx.x * kP + t] = u;
    }
}

// acc[i] += T[o] W(i - o) over the offsets o = 0 .. n - 1 (n a multiple of kW).
// Each offset needs one new source value; the others slide: W(e) sits in
// slot e mod kW, and slot -o mod kW is free when offset o is reached.
template <int kW, class Load>
__device__ __forceinline__ void slide(const double* __restrict__ T, int n, Load load, double (&acc)[kW]) {
    double w[kW];
#pragma unroll
    for (int i = 1; i < kW; ++i) w[i] = load(i);
    w[0] = 0.0;
    for (int o = 0; o < n; o += kW) {
        double tv[kW], nv[kW];
#pragma unroll
        for (int u = 0; u < kW; ++u) {
            tv[u] = T[(size_t)(o + u) * kPP];
            nv[u] = load(-(o + u));
        }
#pragma unroll
        for (int u = 0; u < kW; ++u) {
            w[(kW - u) % kW] = nv[u];
#pragma unroll
            for (int i = 0; i < kW; ++i) acc[i] = fma(tv[u], w[(i - u + kW) % kW], acc[i]);
        }
    }
}

// Pair sums between cells.  Thread (half, k, l) of an item holds moment k's
// share of local coefficient l; the shares are added over k (and halves) in
// shared memory in a fixed order.
//  near item g: the 16 cells of group g from groups g-1, g, g+1 and the group
//    half a period away, whose moments arrive by bulk copies on one mbarrier;
//    per offset one table entry from L2 serves eight target cells (two halves).
//  far item: groups 4f .. 4f+3 from all other groups, group moments from L2;
//    the halves split the offsets.
// What bounds it: the FP64 pipe for the 16 x 96 x 256 multiply-adds of a near
// item (3 us on one SM) and the L2 reads of the tables (192 KB per near item).
struct CellSmem {
    union {
        struct {
            double near_m[80][kP];   // cells -31 .. 48 about group g (zero outside -16 .. 31)
            double seam_m[48][kP];   // cells -15 .. 32 about the seam group (zero outside 0 .. 15)
        };
        double red[16][kC / 2][2][kP];  // k, target, half, l (after the sums)
    };
    uint64_t bar;
};

struct CellSums {
    const double *mom, *momc, *tab;
    double *loc, *locc;
    int Mc;
};

// kNear: with the near groups (else the one half a period away alone).
template <bool kNear>
__device__ __forceinline__ void cell_near(const CellSums& J, int g, CellSmem& S, int* __restrict__ err) {
    const int t = threadIdx.x, l = t & 15, k = (t >> 4) & 15, half = t >> 8;
    const int Mc = J.Mc;
    for (int z = t; z < 15 * kP; z += kPairT) {
        (&S.near_m[0][0])[z] = 0.0;
        (&S.seam_m[0][0])[z] = 0.0;
    }
    for (int z = t; z < 17 * kP; z += kPairT) {
        (&S.near_m[63][0])[z] = 0.0;
        (&S.seam_m[31][0])[z] = 0.0;
    }
    constexpr uint32_t kBytes = kC * kP * sizeof(double);
    if (t == 0) {
        mbar_init(&S.bar, 1);
        fence_mbar_init();
        fence_proxy_async();
        mbar_expect_tx(&S.bar, 4 * kBytes);
        const int gm = g == 0 ? Mc - 1 : g - 1, gp = g == Mc - 1 ? 0 : g + 1;
        const int gs = g >= Mc / 2 ? g - Mc / 2 : g + Mc / 2;
        bulk_load(&S.near_m[15], J.mom + (size_t)gm * kC * kP, kBytes, &S.bar);
        bulk_load(&S.near_m[31], J.mom + (size_t)g * kC * kP, kBytes, &S.bar);
        bulk_load(&S.near_m[47], J.mom + (size_t)gp * kC * kP, kBytes, &S.bar);
        bulk_load(&S.seam_m[15], J.mom + (size_t)gs * kC * kP, kBytes, &S.bar);
    }
    __syncthreads();
    const bool ok = mbar_wait_bounded(&S.bar, 0, g_cell_polls);
    if (!__syncthreads_and(ok)) {
        if (t == 0) {
            atomicExch(err, (int)FS_ERR_TIMEOUT);
            (void)mbar_wait_bounded(&S.bar, 0, kMbarPolls);  // the copies land before the CTA exits
        }
        return;
    }
    double acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    const int i0 = half * 8;
    const double* T = J.tab + k * kP + l;
    // near offsets m = o - 32: source cell i - m, stored at i - m + 31
    if (kNear) slide<8>(T, kNearOff, [&](int d) { return S.near_m[i0 + d + 63][k]; }, acc);
    // seam offsets m = o - 16: stored at i - m + 15
    slide<8>(T + (size_t)kNearOff * kPP, kSeamOff, [&](int d) { return S.seam_m[i0 + d + 31][k]; }, acc);
    __syncthreads();  // the shares take the moments' place
#pragma unroll
    for (int i = 0; i < 8; ++i) S.red[k][i][half][l] = acc[i];
    __syncthreads();
    if (t < kC * kP) {
        const int i = t >> 4;
        double s = 0.0;
#pragma unroll
        for (int kk = 0; kk < 16; ++kk) s += S.red[kk][i & 7][i >> 3][l];
        J.loc[(size_t)(g * kC + i) * kP + l] = s;
    }
}

__device__ __forceinline__ void cell_far(const CellSums& J, const double* __restrict__ far_tab,
                                         double* __restrict__ locc, int f, CellSmem& S) {
    const int t = threadIdx.x, l = t & 15, k = (t >> 4) & 15, half = t >> 8;
    const int Mc = J.Mc, g0 = f * kFarGroups;
    // offsets in two halves of a multiple of 4 (the table is zero from Mc on)
    const int n = (Mc + 7) / 8 * 4;
    const int o0 = half * n;
    const double* __restrict__ W = J.momc + k;
    double acc[kFarGroups] = {0, 0, 0, 0};
    slide<kFarGroups>(far_tab + (size_t)o0 * kPP + k * kP + l, n,
                      [&](int d) {
                          int s = g0 - o0 + d;  // above -2 Mc - 8
                          s += s < 0 ? Mc : 0;
                          s += s < 0 ? Mc : 0;
                          s -= s >= Mc ? Mc : 0;
                          return W[(size_t)s * kP];
                      },
                      acc);
#pragma unroll
    for (int i = 0; i < kFarGroups; ++i) S.red[k][i][half][l] = acc[i];
    __syncthreads();
    if (t < kFarGroups * kP && g0 + (t >> 4) < Mc) {
        const int i = t >> 4;
        double s = 0.0;
#pragma unroll
        for (int kk = 0; kk < 16; ++kk) s += S.red[kk][i][0][l] + S.red[kk][i][1][l];
        locc[(size_t)(g0 + i) * kP + l] = s;
    }
}

inline int cell_far_items(int Mc) { return (Mc + kFarGroups - 1) / kFarGroups; }

__global__ void __launch_bounds__(kPairT) k_cell_pairs(CellSums J, int* __restrict__ err) {
    __shared__ __align__(128) CellSmem S;
    const int nf = (J.Mc + kFarGroups - 1) / kFarGroups;
    const int b = blockIdx.x;  // far items first: theirs is the longer chain of L2 reads
    if (b < nf) cell_far(J, J.tab + (size_t)(kNearOff + kSeamOff) * kPP, J.locc, b, S);
    else cell_near<true>(J, b - nf, S, err);
}

// What a windowed sum leaves to the cells: for every group the other groups'
// share without those of a window about itself, and again about the group before
// it (targets of a block that runs over into the next group), and for every cell
// the group half a period away.  15 us at 158 groups, beside 8.1 ms of pairs.
__global__ void __launch_bounds__(kPairT) k_cell_rest(CellSums J, const double* __restrict__ rest_tab,
                                                      int* __restrict__ err) {
    __shared__ __align__(128) CellSmem S;
    const int nf = (J.Mc + kFarGroups - 1) / kFarGroups, noff = (J.Mc + 7) / 8 * 8;
    const int b = blockIdx.x;
    if (b < 2 * nf) {
        const int v = b >= nf;
        cell_far(J, rest_tab + (size_t)v * noff * kPP, J.locc + (size_t)v * J.Mc * kP, b - v * nf, S);
    } else {
        cell_near<false>(J, b - 2 * nf, S, err);
    }
}

// Group offsets with the window's left out: |m| <= kWinGroups, and then shifted by one.
__global__ void __launch_bounds__(kPP) k_rest_table(CellPlan P, const double* __restrict__ tab,
                                                    double* __restrict__ rest) {
    const int noff = (P.Mc + 7) / 8 * 8, v = blockIdx.x / noff, m = blockIdx.x % noff;
    int c = m - v;  // offset from the window's middle, about 0
    if (c > P.Mc / 2) c -= P.Mc;
    const bool out = c >= -kWinGroups && c <= kWinGroups;
    const double t = tab[(size_t)(kNearOff + kSeamOff + m) * kPP + threadIdx.x];
    rest[(size_t)blockIdx.x * kPP + threadIdx.x] = out ? 0.0 : t;
}

// E at the targets (in the caller's order: coalesced stage arrays; a cell's
// coefficients are one 128-byte line) through the stage epilogue.
__global__ void __launch_bounds__(256) k_cell_eval(CellPlan P, const double* __restrict__ x, int n,
                                                   const double* __restrict__ loc, const double* __restrict__ locc,
                                                   Stage S) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double w = cell_wrap(x[i], P.L);
    const int c = cell_of(w, P), g = c / kC;
    const double xi = fma(w, P.two_inv_h, -(double)(2 * c + 1));
    const double xg = fma(w, P.two_inv_h, -(double)((2 * g + 1) * kC)) * (1.0 / kC);
    const double E = cheb_sum(loc + (size_t)c * kP, xi) + cheb_sum(locc + (size_t)g * kP, xg);
    apply_stage(S, i, E);
}

// G on the 16 x 16 Chebyshev nodes of two cells of width hh whose centres are d0
// apart, both sides to coefficients, as T[k][l] (a CTA of kPP threads).
__device__ void offset_table(const CellPlan& P, double d0, double hh, bool zero, double* __restrict__ out) {
    __shared__ double A[kP][kP + 1], C[kP][kP + 1], X[kP][kP + 1];
    const int t = threadIdx.x, a = t >> 4, b = t & 15;
    C[a][b] = cospi((a + 0.5) * b / kP) * (b ? 2.0 : 1.0) / kP;  // node a's share of coefficient b
    const double na = cospi((a + 0.5) / kP), nb = cospi((b + 0.5) / kP);
    double d = d0 + (na - nb) * (0.5 * hh);
    d -= P.L * rint(d / P.L);
    A[a][b] = zero ? 0.0 : d / (2.0 * sqrt(d * d + P.eps * P.eps)) - P.cbg * d;
    __syncthreads();
    double s = 0.0;  // X[l][b] = sum_a C[a][l] A[a][b], thread (l = a, b)
    for (int n = 0; n < kP; ++n) s = fma(C[n][a], A[n][b], s);
    X[a][b] = s;
    __syncthreads();
    s = 0.0;  // T[k][l], thread (k = a, l = b)
    for (int n = 0; n < kP; ++n) s = fma(C[n][a], X[b][n], s);
    out[t] = s;
}

// One CTA per offset of the two levels; the last kC CTAs form the child matrices.
__global__ void __launch_bounds__(kPP) k_cell_table(CellPlan P, double* __restrict__ tab,
                                                    double* __restrict__ child) {
    const int o = blockIdx.x;
    const int noff = cell_table_offsets(P.Mc);
    if (o >= noff) {
        __shared__ double A[kP][kP + 1];
        const int t = threadIdx.x, a = t >> 4, b = t & 15;
        // T_k of child node a's place in the group, k = b: then its coefficients
        const int c = o - noff;
        const double y = (cospi((a + 0.5) / kP) + (double)(2 * c + 1 - kC)) * (1.0 / kC);
        double u = 1.0, v = y;
        for (int k = 0; k < b; ++k) {
            const double z = fma(2.0 * y, v, -u);
            u = v;
            v = z;
        }
        A[a][b] = u;
        __syncthreads();
        double s = 0.0;  // thread (k = a, l = b)
        for (int n = 0; n < kP; ++n)
            s = fma(cospi((n + 0.5) * b / kP) * (b ? 2.0 : 1.0) / kP, A[n][a], s);
        child[((size_t)c * kP + a) * kP + b] = s;
        return;
    }
    double d0, hh = P.h;
    bool zero;
    if (o < kNearOff) {
        d0 = (o - 32) * P.h;
        zero = o == 0;
    } else if (o < kNearOff + kSeamOff) {
        d0 = (P.M / 2 + (o - kNearOff) - 16) * P.h;
        zero = o == kNearOff;
    } else {
        const int m = o - kNearOff - kSeamOff;
        hh = P.h * kC;
        d0 = m * hh;
        zero = m <= 1 || m >= P.Mc - 1 || m == P.Mc / 2;
    }
    offset_table(P, d0, hh, zero, tab + (size_t)o * kPP);
}

// One CTA per cell offset 0 .. M - 1.
__global__ void __launch_bounds__(kPP) k_offset_table(CellPlan P, double* __restrict__ tab) {
    offset_table(P, blockIdx.x * P.h, P.h, false, tab + (size_t)blockIdx.x * kPP);
}

int key_bits(int M) {
    int b = 1;
    while ((1 << b) < M) ++b;
    return b;
}

}  // namespace

bool cell_plan(double L, double eps, CellPlan* P) {
    // L > 32 eps: the far field exists at all (see the seam's error above);
    // cells up to kCellMax bound the tables and the group-by-group sums.
    if (!(L > 32 * eps) || !(L <= kCellMax / 1.6 * eps)) return false;
    const int step = 2 * kC;
    const int M = std::max(256, (int)std::ceil(1.6 * L / eps / step) * step);
    if (M > kCellMax) return false;
    P->L = L;
    P->eps = eps;
    P->cbg = 1 / std::sqrt(L * L + 4 * eps * eps);
    P->h = L / M;
    P->inv_h = M / L;
    P->two_inv_h = 2 * (M / L);
    P->M = M;
    P->Mc = M / kC;
    return true;
}

size_t cell_sort_bytes(int n, int M) {
    size_t b = 0;
    FS_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, b, (const uint32_t*)nullptr, (uint32_t*)nullptr,
                                            (const int*)nullptr, (int*)nullptr, n, 0, key_bits(M)));
    return std::max<size_t>(b, 1);
}

void cell_table(const CellPlan& P, double* tab, double* child, cudaStream_t st) {
    k_cell_table<<<cell_table_offsets(P.Mc) + kC, kPP, 0, st>>>(P, tab, child);
    FS_LAUNCHED(1);
}

void cell_offset_table(const CellPlan& P, double* tab, cudaStream_t st) {
    k_offset_table<<<P.M, kPP, 0, st>>>(P, tab);
    FS_LAUNCHED(1);
}

void cell_field(const CellPlan& P, const CellBuffers& B, const double* d_t, int nt, const double* d_s,
                const double* d_q, int ns, const Stage& S, int* err, cudaStream_t st) {
    const int T = 256, nb = (ns + T - 1) / T;
    k_cell_keys<<<nb, T, 0, st>>>(P, d_s, ns, B.kin, B.iin);
    size_t tb = B.sort_bytes;
    FS_CUDA(cub::DeviceRadixSort::SortPairs(B.sort_tmp, tb, B.kin, B.kout, B.iin, B.iout, ns, 0, key_bits(P.M), st));
    k_cell_moments<false><<<nb, T, 0, st>>>(P, B.kout, B.iout, d_s, d_q, ns, B.start, B.part);
    k_cell_gather<<<P.Mc, 1024, 0, st>>>(P, B.start, B.part, B.child, B.mom, B.momc);
    {
        ProfScope prof("k_cell_pairs", st, (double)nt * (double)ns);
        k_cell_pairs<<<cell_far_items(P.Mc) + P.Mc, kPairT, 0, st>>>(
            CellSums{B.mom, B.momc, B.tab, B.loc, B.locc, P.Mc}, err);
    }
    k_cell_eval<<<(nt + T - 1) / T, T, 0, st>>>(P, d_t, nt, B.loc, B.locc, S);
    FS_LAUNCHED(5);
}

size_t cell_rest_table_size(const CellPlan& P) { return 2 * (size_t)((P.Mc + 7) / 8 * 8) * kPP; }

void cell_rest_table(const CellPlan& P, const double* tab, double* rest_tab, cudaStream_t st) {
    k_rest_table<<<2 * ((P.Mc + 7) / 8 * 8), kPP, 0, st>>>(P, tab, rest_tab);
    FS_LAUNCHED(1);
}

void cell_rest(const CellPlan& P, const CellBuffers& B, const double* rest_tab, const double* d_x, const double* d_q,
               int ns, double* locc2, int* err, cudaStream_t st) {
    const int T = 256, nb = (ns + T - 1) / T;
    k_cell_moments<true><<<nb, T, 0, st>>>(P, nullptr, nullptr, d_x, d_q, ns, B.start, B.part);
    k_cell_gather<<<P.Mc, 1024, 0, st>>>(P, B.start, B.part, B.child, B.mom, B.momc);
    k_cell_rest<<<2 * cell_far_items(P.Mc) + P.Mc, kPairT, 0, st>>>(
        CellSums{B.mom, B.momc, B.tab, B.loc, locc2, P.Mc}, rest_tab, err);
    FS_LAUNCHED(3);
}

void set_cell_polls(long long polls) {
    const long long v = polls < 0 ? kMbarPolls : polls;
    FS_CUDA(cudaMemcpyToSymbol(g_cell_polls, &v, sizeof(v)));
}

}  // namespace fsb
