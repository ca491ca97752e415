// Plain FP64 periodic direct sum: the reference's arithmetic on the GPU.
//
// E_MQ_DirectSum::operator() (src/FieldStructure.cpp:106-156) with every
// target's sum formed in the reference's order and with its roundings (no
// contraction): the result is bit-identical to E_MQ_DirectSum.
//
// Only the additions into a target's sum are sequential; the terms are not.  A
// CTA takes 32 targets, one per lane.  kWarps warps form the terms of
// consecutive sources into a double buffer in shared memory while one more
// warp adds the previous round's terms in the reference's order: one addition
// per pair, 8 clocks each behind one another, where forming 32 targets' terms
// for a source takes an SM's FP64 pipe 12.  So even the few targets of a small
// run (a 32-target CTA) keep an SM busy.
//
// What bounds it is the FP64 pipe (64 lanes/clk/SM).  In IEEE operations a
// pair costs 40 FP64 instructions, most of them in the two divisions and the
// square root.  pair_terms_fast forms the same correctly rounded values in 23:
//  * the division by L (the same for all pairs) as a product with 1/L in two
//    parts, Brisebarre, Muller and Raina, "Accelerating correctly rounded
//    floating-point division when the divisor is known in advance", IEEE
//    Trans. Comput. 53 (2004): correct for all dividends unless one of a few
//    near-midpoint ones, which the host enumerates for its L
//    (division_is_product);
//  * square root and the reciprocal of its rounded value from one approximate
//    1/sqrt, refined by a third-order step, each finished by Markstein's
//    residual step (Markstein, "Computation of elementary functions on the
//    IBM RISC System/6000 processor", IBM J. Res. Dev. 34 (1990)).  The
//    residual is exact, so the result is the correctly rounded one unless the
//    true value lies within 2^-102 of a rounding boundary; the mantissas where
//    it does (the roots of x^2 = t mod 2^54 and 2^55 for small t, the divisors
//    of 2^106 + t) were enumerated and tried: the roots come out right, the
//    reciprocals of two mantissas (all ones, Markstein's exception, and one
//    more) do not, and their pairs take the IEEE operations;
//  * factors of 4 carried exactly (sqrt(4 R) = 2 sqrt(R));
//  * no tests for the pairs the reference skips: with z = 0 or |z| = 1/2 the
//    term is a zero (1/sqrt(r2) is then the reference's own constant), which
//    leaves a running sum that started at +0 unchanged.
// Tiles with values for which that does not hold (charges not below 2^800,
// positions that are tiny but not 0) take the IEEE operations, as do all pairs
// when L or epsilon is out of range.
//
// Measured on 16,770 points alone: 639 us in place of 5.09 ms (one thread per
// target, IEEE operations), with 72% of the FP64 pipe's cycles used; 65,537
// sources at 33,333 targets 4.6 in place of 20.4 ms; 1,025 points 19 in place of
// 322 us.  Eight term warps of eight terms were the fastest of 2 to 16 by 4 to 16.
#include <cfloat>
#include <cmath>

#include "fs_device.cuh"

namespace fsb {

namespace {

constexpr int kThreads64 = 128;  // k_direct64_open
constexpr int kTile64 = 1024;    // k_direct64_open
constexpr int kTerms = 8;          // terms of a warp per round
constexpr int kSrcTile = 512;      // sources staged at a time

struct Pair64 {
    double L, four_eps2, norm;  // reference constants
    double zh, zl, eps2;        // 1/L in two parts, four_eps2 / 4
};

// One term in IEEE operations, 0 where the reference skips the pair (adding
// +0 leaves a running sum that started at +0 unchanged).
__device__ __forceinline__ double pair_term_ieee(const Pair64& K, double xi, double xj, double nq) {
    double z = ddiv(dsub(xi, xj), K.L);
    z = dsub(z, round(z));
    if (fabs(dsub(z, 0.5)) < DBL_MIN || fabs(dadd(z, 0.5)) < DBL_MIN || fabs(z) < DBL_MIN) return 0.0;
    const double r2 = dadd(dmul(dmul(dmul(dmul(4.0, z), z), K.L), K.L), K.four_eps2);
    const double inv = ddiv(1.0, __dsqrt_rn(r2));
    return dmul(dmul(dmul(nq, z), K.L), dsub(K.norm, inv));
}

__device__ __noinline__ void pair_terms_ieee(const Pair64& K, double xi, const double2* p, double (*row)[32],
                                             int lane) {
    for (int u = 0; u < kTerms; ++u) row[u][lane] = pair_term_ieee(K, xi, p[u].x, p[u].y);
}

// The same values for kTerms sources {x, -q} at once, step by step so that the
// chains interleave; true when one of them needs the IEEE operations.  rint and the reference's round differ at
// ties only, where |z| = 1/2.
__device__ __forceinline__ bool pair_terms_fast(const Pair64& K, double xi, const double2* p, double (&t)[kTerms]) {
    double z[kTerms], R[kTerms], y[kTerms], a[kTerms], q[kTerms];
#define FS_EACH _Pragma("unroll") for (int u = 0; u < kTerms; ++u)
    FS_EACH {
        const double2 e = p[u];
        z[u] = dsub(xi, e.x);
        q[u] = e.y;
    }
    FS_EACH a[u] = dmul(z[u], K.zl);
    FS_EACH z[u] = fma(z[u], K.zh, a[u]);
    FS_EACH z[u] = dsub(z[u], rint(z[u]));
    FS_EACH R[u] = dmul(z[u], z[u]);
    FS_EACH R[u] = dmul(R[u], K.L);
    FS_EACH R[u] = dmul(R[u], K.L);
    FS_EACH R[u] = dadd(R[u], K.eps2);
    FS_EACH asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y[u]) : "d"(R[u]));
    FS_EACH q[u] = dmul(q[u], z[u]);
    FS_EACH a[u] = dmul(R[u], y[u]);
    FS_EACH a[u] = fma(-a[u], y[u], 1.0);
    FS_EACH z[u] = dmul(y[u], a[u]);
    FS_EACH a[u] = fma(a[u], 0.375, 0.5);
    FS_EACH y[u] = fma(z[u], a[u], y[u]);
    FS_EACH a[u] = dmul(R[u], y[u]);
    FS_EACH z[u] = __hiloint2double(__double2hiint(y[u]) - 0x100000, __double2loint(y[u]));  // y / 2
    FS_EACH R[u] = fma(-a[u], a[u], R[u]);
    FS_EACH R[u] = fma(R[u], z[u], a[u]);  // s = sqrt(R)
    FS_EACH a[u] = fma(-R[u], y[u], 1.0);
    FS_EACH a[u] = fma(a[u], y[u], y[u]);  // 1 / s
    // the two mantissas of s whose reciprocal comes out one ulp low (2^53 - 1
    // and 2^52 + 0x0699d36aec84e), known here by their low words
    bool rare = false;
    FS_EACH {
        const unsigned lo = (unsigned)__double2loint(R[u]);
        rare |= lo == 0xffffffffu || lo == 0x36aec84eu;
    }
    FS_EACH q[u] = dmul(q[u], K.L);
    FS_EACH a[u] = fma(-0.5, a[u], K.norm);
    FS_EACH t[u] = dmul(q[u], a[u]);
#undef FS_EACH
    return rare;
}

// Whether a nonzero |x| is so small that differences may be (with |x| from
// 2^-800 up, two positions are equal or 2^-853 apart at least).
__device__ __forceinline__ bool tiny(double x) { return x != 0.0 && fabs(x) < 0x1p-800; }

template <int kWarps>
struct Direct64Smem {
    double2 tile[2][kSrcTile];               // {x, -q}
    double term[2][kWarps * kTerms][32];
};

template <int kWarps, bool kFast>
__global__ void __launch_bounds__((kWarps + 1) * 32)
k_direct64(const double* __restrict__ tx, int nt, const double* __restrict__ sx, const double* __restrict__ sq, int ns,
           Pair64 K, Stage S) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Direct64Smem<kWarps>& sh = *reinterpret_cast<Direct64Smem<kWarps>*>(smem_raw);
    constexpr int kRound = kWarps * kTerms, kProd = kWarps * 32, kPer = kSrcTile / kProd;
    static_assert(kSrcTile % kRound == 0 && kSrcTile % kProd == 0, "whole rounds and loads per tile");
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool adder = warp == kWarps;
    const int i = blockIdx.x * 32 + lane;
    const double xi = (i < nt) ? tx[i] : 0.0;
    const bool tiny_i = __any_sync(0xffffffffu, tiny(xi));
    double2 next[kPer];
    auto fetch = [&](int base) {
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            const int j = base + threadIdx.x + k * kProd;
            // times -1.0, exactly; the last tile is filled up with charges 0
            next[k] = j < ns ? make_double2(sx[j], -sq[j]) : make_double2(0.0, 0.0);
        }
    };
    auto store = [&](double2* tile) {
        bool odd = false;
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            tile[threadIdx.x + k * kProd] = next[k];
            odd |= !(fabs(next[k].y) < 0x1p800) || tiny(next[k].x);
        }
        return odd;
    };
    bool odd = false;
    if (!adder) {
        fetch(0);
        odd = store(sh.tile[0]);
    }
    bool ieee = (bool)__syncthreads_or(odd) || tiny_i || !kFast;
    double ei = 0.0;
    int par = 0, pending = 0;  // term buffer of this round, rows of the previous one
    auto add_rows = [&](const double (*row)[32], int n) {
        int j = 0;
        for (; j + 16 <= n; j += 16) {
            double v[16];
#pragma unroll
            for (int u = 0; u < 16; ++u) v[u] = row[j + u][lane];
#pragma unroll
            for (int u = 0; u < 16; ++u) ei = dadd(ei, v[u]);
        }
        for (; j < n; ++j) ei = dadd(ei, row[j][lane]);
    };
    for (int base = 0, b = 0; base < ns; base += kSrcTile, b ^= 1) {
        const int cnt = min(kSrcTile, ns - base);
        const bool more = base + kSrcTile < ns;
        if (!adder && more) fetch(base + kSrcTile);
        bool next_ieee = false;
        for (int r = 0; r * kRound < cnt; ++r) {
            if (adder) {
                add_rows(sh.term[par ^ 1], pending);
                pending = min(kRound, cnt - r * kRound);
            } else {
                const double2* p = sh.tile[b] + r * kRound + warp * kTerms;
                double(*row)[32] = sh.term[par] + warp * kTerms;
                bool rest = true;
                if (kFast && !ieee) {
                    double t[kTerms];
                    rest = pair_terms_fast(K, xi, p, t);
#pragma unroll
                    for (int u = 0; u < kTerms; ++u) row[u][lane] = t[u];
                }
                if (rest) pair_terms_ieee(K, xi, p, row, lane);
            }
            if (more && (r + 1) * kRound >= cnt) {
                odd = adder ? false : store(sh.tile[b ^ 1]);
                next_ieee = __syncthreads_or(odd);
            } else {
                __syncthreads();
            }
            par ^= 1;
        }
        ieee = next_ieee || tiny_i || !kFast;
    }
    if (adder) {
        add_rows(sh.term[par ^ 1], pending);
        if (i < nt) apply_stage(S, i, ei);
    }
}

// Open boundaries, E_MQ_DirectSum_openbcs::operator() (src/FieldStructure.cpp:170-192):
// es_i = sum_j ((q_j * 0.5) * z) / sqrt(z*z + eps^2) - x_i, z = x_i - x_j, in the
// reference's order and roundings (bit-identical).
__global__ void __launch_bounds__(kThreads64)
k_direct64_open(const double* __restrict__ tx, int nt, const double* __restrict__ sx, const double* __restrict__ sq,
                int ns, double eps, Stage S) {
    __shared__ double sh_x[kTile64];
    __shared__ double sh_q[kTile64];
    const int i = blockIdx.x * kThreads64 + threadIdx.x;
    const double xi = (i < nt) ? tx[i] : 0.0;
    const double eps_sq = dmul(eps, eps);
    double ei = 0.0;
    for (int base = 0; base < ns; base += kTile64) {
        const int cnt = min(kTile64, ns - base);
        for (int k = threadIdx.x; k < cnt; k += kThreads64) {
            sh_x[k] = sx[base + k];
            sh_q[k] = sq[base + k];
        }
        __syncthreads();
        for (int j = 0; j < cnt; ++j) {
            const double z = dsub(xi, sh_x[j]);
            ei = dadd(ei, ddiv(dmul(dmul(sh_q[j], 0.5), z), __dsqrt_rn(dadd(dmul(z, z), eps_sq))));
        }
        __syncthreads();
    }
    if (i < nt) apply_stage(S, i, dsub(ei, xi));
}

class Direct64Open final : public FieldEngine {
   public:
    explicit Direct64Open(double eps) : eps_(eps) {}
    void eval(const double* d_t, int nt, const double* d_s, const double* d_q, int ns, const Stage& stage,
              cudaStream_t st, PairForm) override {
        last_pairs = (double)nt * (double)ns;
        if (nt <= 0) return;
        const int blocks = (nt + kThreads64 - 1) / kThreads64;
        ProfScope prof("k_direct64_open", st, last_pairs);
        k_direct64_open<<<blocks, kThreads64, 0, st>>>(d_t, nt, d_s, d_q, ns, eps_, stage);
        FS_LAUNCHED(1);
    }

   private:
    double eps_;
};

// q = fma(a, zh, a zl) with zh = RN(1/L), zl = RN(1/L - zh) is RN(a/L) for
// every a (within the exponent range checked by the kernel) unless a/L comes
// within the product's error, below 2^-104 of it, of the midpoint of two
// doubles.  With a = A 2^f, L = B 2^e, A and B 53-bit integers, and a midpoint
// M (odd, 54 bits), that needs |A 2^s - M B| <= 16 with s = 53 (A >= B) or 54:
// M is fixed modulo a power of two by B and the small difference, so the few
// candidates are solved for and tried.
bool division_is_product(double L, double zh, double zl) {
    int e = 0;
    const double m = std::frexp(L, &e);
    const uint64_t B = (uint64_t)std::ldexp(m, 53);
    int t = 0;
    uint64_t odd = B;
    while (!(odd & 1)) {
        odd >>= 1;
        ++t;
    }
    uint64_t inv = odd;  // inverse of the odd part modulo 2^64 (Newton)
    for (int k = 0; k < 6; ++k) inv *= 2 - odd * inv;
    for (int s = 53; s <= 54; ++s)
        for (int delta = -16; delta <= 16; ++delta) {
            if (delta % (1 << std::min(t, 20)) || t > 4) continue;  // 2^t must divide the difference
            const int bits = s - t;
            const uint64_t mask = (1ull << bits) - 1;
            const uint64_t M0 = ((uint64_t)(-(int64_t)(delta >> t)) * inv) & mask;
            for (uint64_t M = M0; M < (1ull << 54); M += 1ull << bits) {
                if (M < (1ull << 53) || !(M & 1)) continue;
                const unsigned __int128 num = (unsigned __int128)M * B + (unsigned __int128)(__int128)delta;
                if (num & (((unsigned __int128)1 << s) - 1)) continue;
                const uint64_t A = (uint64_t)(num >> s);
                if (A < (1ull << 52) || A >= (1ull << 53)) continue;
                const double a = (double)A;
                if (std::fma(a, zh, a * zl) != a / L) return false;
            }
        }
    return true;
}

class Direct64 final : public FieldEngine {
   public:
    Direct64(double L, double eps) {
        // same expressions as the reference
        K_.L = L;
        K_.norm = 1 / std::sqrt(L * L + 4 * eps * eps);
        K_.four_eps2 = 4.0 * eps * eps;
        K_.zh = 1 / L;
        K_.zl = std::fma(-K_.zh, L, 1.0) / L;
        K_.eps2 = K_.four_eps2 / 4;
        auto mid = [](double v) { return v > 0x1p-200 && v < 0x1p200; };
        fast_ = mid(L) && mid(eps) && division_is_product(L, K_.zh, K_.zl);
    }
    void eval(const double* d_t, int nt, const double* d_s, const double* d_q, int ns,
              const Stage& stage, cudaStream_t st, PairForm) override {
        last_pairs = (double)nt * (double)ns;
        if (nt <= 0) return;
        ProfScope prof("k_direct64", st, last_pairs);
        // more warps per CTA where the targets do not give each SM two CTAs
        // (4,290 points: 55 us; lanes sharing a target 124 us and more)
        const bool few = nt <= 2 * 32 * sm_count();
        if (fast_ && few) launch<16, true>(d_t, nt, d_s, d_q, ns, stage, st);
        else if (fast_) launch<8, true>(d_t, nt, d_s, d_q, ns, stage, st);
        else launch<8, false>(d_t, nt, d_s, d_q, ns, stage, st);
        FS_LAUNCHED(1);
    }

   private:
    template <int kWarps, bool kFast>
    void launch(const double* d_t, int nt, const double* d_s, const double* d_q, int ns, const Stage& S,
                cudaStream_t st) const {
        constexpr size_t smem = sizeof(Direct64Smem<kWarps>);
        FS_CUDA(cudaFuncSetAttribute(k_direct64<kWarps, kFast>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        k_direct64<kWarps, kFast><<<(nt + 31) / 32, (kWarps + 1) * 32, smem, st>>>(d_t, nt, d_s, d_q, ns, K_, S);
    }

    Pair64 K_;
    bool fast_ = false;
};

}  // namespace

FieldEngine* make_direct64(double L, double eps) { return new Direct64(L, eps); }
FieldEngine* make_direct64_open(double eps) { return new Direct64Open(eps); }

}  // namespace fsb
