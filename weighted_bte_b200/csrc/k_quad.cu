// Kernels over quads (quad.cuh) for calls bound by the length of a scalar
// multiple's chain: the Horner tail of an MSM, transform stages of few arrays,
// MSMs of a few terms, single multiples and Schnorr checks.  One warp per
// block; every lane runs to the end of its kernel.
#include <algorithm>
#include <type_traits>

#include "launch.h"
#include "quad.cuh"

namespace wbte {

namespace {
constexpr int WARP = 32;
inline unsigned blocks_for(int64_t n, int64_t per) { return (unsigned)((n + per - 1) / per); }

template <class Q> struct SizeOf {
    static constexpr size_t AFF = 2 * Q::Field::FIELD, XYZZ = 4 * Q::Field::FIELD;
    static constexpr int PER_WARP = WARP / Q::WIDTH;
};
using G1Quad = Quad<OnLane>;
using G2Quad = Quad<OnPair>;
// this lane's point among all the launch's
template <class Q> __device__ __forceinline__ int64_t point_index() {
    return (int64_t)blockIdx.x * SizeOf<Q>::PER_WARP + (threadIdx.x & 31) / Q::WIDTH;
}
// a doubling of a Horner chain of points on the curve
__device__ __forceinline__ Fp horner_dbl(Oct, const Fp& p) { return Oct::dbl(p); }
__device__ __forceinline__ Fp horner_dbl(Quad<OnPair, 8>, const Fp& p) { return Quad<OnPair, 8>::dbl_on_curve(p); }

// Whether `count` XYZZ records are of points on the curve (or infinity), a lane
// (G1) or a pair (G2) to each: Y^2 = X^3 + b ZZZ^2.
template <class P> __device__ __forceinline__ bool records_on_curve(const uint8_t* rec, int64_t count) {
    using Pt = Point<P>;
    bool on = true;
    for (int64_t i0 = 0; i0 < count; i0 += WARP / P::LANES) {
        const int64_t i = i0 + (threadIdx.x & 31) / P::LANES;
        const uint8_t* r = rec + 4 * P::FIELD * (i < count ? i : count - 1);
        const Fp X = load_vec(Pt::at(r, 0)), Y = load_vec(Pt::at(r, 1)), Z = load_vec(Pt::at(r, 3));
        const Fp rhs = fp_add(P::mul(P::mul(X, X), X), P::times_b(P::mul(Z, Z)));
        const bool curve = P::zero(fp_sub(P::mul(Y, Y), rhs)), inf = P::zero(load_vec(Pt::at(r, 2)));
        on = on && (curve || inf);
    }
    return __all_sync(FULL, on);
}

template <class Q, bool ON_CURVE>
__device__ __forceinline__ void combine(uint8_t* out, const uint8_t* wins, int64_t k, int windows, int c) {
    const int64_t j = (int64_t)blockIdx.x * (WARP / Q::WIDTH) + (threadIdx.x & 31) / Q::WIDTH;
    const bool active = j < k;
    const uint8_t* W = wins + SizeOf<Q>::XYZZ * (active ? j : k - 1) * windows;
    Fp acc = Q::load(W + SizeOf<Q>::XYZZ * (windows - 1));
    for (int w = windows - 2; w >= 0; w--) {
        for (int i = 0; i < c; i++) {
            if constexpr (ON_CURVE)
                acc = horner_dbl(Q(), acc);
            else
                acc = Q::dbl(acc);
        }
        acc = Q::add(acc, Q::load(W + SizeOf<Q>::XYZZ * w), true);
    }
    acc = Q::affine(acc);
    if (active) Q::store_affine(out + SizeOf<Q>::AFF * j, acc);
}

// out[j] = sum_w 2^(c w) wins[j windows + w], the sums of each window.  About 250
// doublings in a row bound it, whatever the MSM's size; they use the curve's
// equation where the warp's window sums satisfy it.  Looking at them is one to four
// records a lane, a chain of some ten products beside the tail's thousand: MSMs of
// 65,536 points in G1 2.432 -> 2.426 ms, of 20,011 in G2 3.161 -> 3.177 ms (runs
// differ by 0.2 %).
template <class Q>
__global__ void __launch_bounds__(WARP) k_combine(uint8_t* out, const uint8_t* wins, int64_t k, int windows, int c) {
    using P = typename Q::Field;
    constexpr int PER = WARP / Q::WIDTH;
    const int64_t first = (int64_t)blockIdx.x * PER, here = k - first < PER ? k - first : PER;
    if (records_on_curve<P>(wins + SizeOf<Q>::XYZZ * first * windows, here * windows))
        combine<Q, true>(out, wins, k, windows, c);
    else
        combine<Quad<P, 8>, false>(out, wins, k, windows, c);
}

// A radix-2^kappa step of a decimation-in-time transform merges the radix-2
// stages of half sizes h, 2h, .., 2^(kappa-1) h: in a block of rho h values
// (rho = 2^kappa) and for each offset j < h, with x_k the value at j + q h, q the
// bit reversal of k, and s = n / (rho h),
//   out[j + m h] = sum_k w^(k s (j + m h)) x_k.
// For k = 2^e odd the multiples repeat up to sign after V_k = rho / 2^(e+1)
// values of m, so a block and offset need sum_k V_k = (4^kappa - 1) / 3 of them,
// all independent: 5 instead of 4 for two stages, 21 instead of 12 for three.
// A scalar multiple is a chain of about 550 rounds and a sum one of four, so
// where schedulers idle a step of three stages takes about a third of their time.
//
// Multiple r of a block and offset: those of k = 1, 2, .., rho - 1 in order.
struct RadixTerm { int k, m; };
__device__ __forceinline__ int radix_variants(int k, int rho) { return rho / (2 * (k & -k)); }
__device__ __forceinline__ RadixTerm radix_term(int r, int rho) {
    int k = 1;
    for (; r >= radix_variants(k, rho); k++) r -= radix_variants(k, rho);
    return {k, r};
}
__device__ __forceinline__ int radix_slot(int k, int m, int rho) {
    int r = m;
    for (int i = 1; i < k; i++) r += radix_variants(i, rho);
    return r;
}

// multiples[(t per + r)] for the blocks and offsets t (array-major, then block,
// then offset) and the per = (4^kappa - 1) / 3 multiples r, DIGITS points each
template <class Q>
__global__ void __launch_bounds__(WARP) k_ntt_multiples(uint8_t* multiples, const uint8_t* work, const uint8_t* tw, int64_t n,
                                                        int64_t h, int kappa, int64_t total, int per) {
    constexpr int D = QuadDigits<Q>::DIGITS;
    const int rho = 1 << kappa;
    const int64_t p = point_index<Q>();
    const int dig = (int)(p % D);
    const bool active = p / D < total;
    const int64_t g = active ? p / D : total - 1;
    const int64_t t = g / per, j = t % h, blk = t / h;
    const RadixTerm term = radix_term((int)(g % per), rho);
    const int q = (int)(__brev((uint32_t)term.k) >> (32 - kappa));
    const Fp v = Q::load(work + SizeOf<Q>::XYZZ * (blk * rho * h + j + q * h));
    int64_t idx = (int64_t)term.k * (n / (rho * h)) * (j + term.m * h) % n;
    const bool minus = idx >= n / 2;  // w^(i + n/2) = -w^i
    if (minus) idx -= n / 2;
    uint64_t d[4] = {1, 0, 0, 0};
    if (idx) {
        uint32_t s[8];
        load_scalar(s, tw + FR_SZ * idx);
        decompose_base_x(d, s);
    }
    Fp r = v;
    // w^0 alone in the whole warp needs no digits
    if (__any_sync(FULL, idx != 0)) {
        uint64_t lo[1], hi[1];
        quad_digit<typename Q::Field>(lo[0], hi[0], d, dig);
        const Fp base[1] = {quad_image<Q>(v, dig)};
        r = quad_sum<Q>(quad_straus<Q>(base, lo, hi, 1), D);
    }
    if (minus) r = Q::neg(r);
    if (active && dig == 0) Q::store(multiples + SizeOf<Q>::XYZZ * g, r);
}

// the sums of a step, L points (a power of two that a warp holds) per output
template <class Q>
__global__ void __launch_bounds__(WARP) k_ntt_sums(uint8_t* out, const uint8_t* work, const uint8_t* multiples, int64_t h,
                                                   int kappa, int64_t total, int per, int L) {
    const int rho = 1 << kappa;
    const int64_t p = point_index<Q>();
    const int sub = (int)(p % L);
    const bool active = p / L < total;
    const int64_t o = active ? p / L : total - 1;
    const int64_t t = o / rho, j = t % h, blk = t / h;
    const int m = (int)(o % rho);
    Fp acc = Q::infinity();
    for (int k = sub; k < rho; k += L) {
        const int V = k ? radix_variants(k, rho) : 1;
        Fp x = Q::load(k ? multiples + SizeOf<Q>::XYZZ * (t * per + radix_slot(k, m % V, rho))
                         : work + SizeOf<Q>::XYZZ * (blk * rho * h + j));
        if (k && (m / V) & 1) x = Q::neg(x);
        acc = k == sub ? x : Q::add(acc, x, true);
    }
    acc = quad_sum<Q>(acc, L);
    if (active && sub == 0) Q::store(out + SizeOf<Q>::XYZZ * (blk * rho * h + j + m * h), acc);
}

// out[o] = sum_t scalars[vsel[o] n + t] points[pbase[o] + idx[t]] for n <=
// SMALL_MSM_MAX: the (term, digit) pairs of an output are dealt to L points
// (a power of two that a warp holds), the sums meet in a tree
template <class Q>
__device__ __forceinline__ void small_msm(uint8_t* out, const uint8_t* points, const int64_t* pbase, const int32_t* idx,
                                          const uint8_t* scalars, const int32_t* vsel, int64_t k, int64_t n, int L) {
    constexpr int D = QuadDigits<Q>::DIGITS, MOST = SMALL_MSM_MAX * D;
    const int64_t p = point_index<Q>();
    const int sub = (int)(p % L);
    const bool active = p / L < k;
    const int64_t o = active ? p / L : k - 1;
    const int64_t v = vsel ? (int64_t)vsel[o] : 0;
    const int pairs = (int)n * D, mine = (pairs + L - 1) / L;
    Fp base[MOST];
    uint64_t lo[MOST], hi[MOST];
    for (int r = 0; r < mine; r++) {
        const int x = sub + r * L, t = x < pairs ? x / D : 0, c = x % D;
        base[r] = quad_image<Q>(Q::load_affine(points + SizeOf<Q>::AFF * (pbase[o] + (idx ? (int64_t)idx[t] : t))), c);
        uint32_t s[8];
        load_scalar(s, scalars + FR_SZ * (v * n + t));
        uint64_t d[4];
        decompose_base_x(d, s);
        quad_digit<typename Q::Field>(lo[r], hi[r], d, c);
        if (x >= pairs) lo[r] = hi[r] = 0;
    }
    const Fp r = Q::affine(quad_sum<Q>(quad_straus<Q>(base, lo, hi, mine), L));
    if (active && sub == 0) Q::store_affine(out + SizeOf<Q>::AFF * o, r);
}
template <class Q>
__global__ void __launch_bounds__(WARP) k_small_msm(uint8_t* out, const uint8_t* points, const int64_t* pbase,
                                                    const int32_t* idx, const uint8_t* scalars, const int32_t* vsel,
                                                    int64_t k, int64_t n, int L) {
    if constexpr (std::is_same<Q, Oct>::value) {
        using G = Oct::General;
        const int64_t p = point_index<Q>(), o = p / L < k ? p / L : k - 1;
        bool on = true;
        for (int64_t t = 0; t < n; t++) {
            const bool here = G::on_curve(G::load_affine(points + G1_AFF * (pbase[o] + (idx ? (int64_t)idx[t] : t))));
            on = on && here;
        }
        if (!__all_sync(FULL, on)) {
            small_msm<G>(out, points, pbase, idx, scalars, vsel, k, n, L);
            return;
        }
    }
    small_msm<Q>(out, points, pbase, idx, scalars, vsel, k, n, L);
}

// out[i] = scalars[i] points[i stride] for any points (no endomorphism, and of the
// curve's equation only its form): 4-bit windows of the 256-bit scalar
template <class Q>
__device__ __forceinline__ void mul_batch(uint8_t* out, const uint8_t* pts, int64_t stride, const uint8_t* scalars,
                                          int64_t n) {
    int64_t i = point_index<Q>();
    const bool active = i < n;
    if (!active) i = n - 1;
    uint32_t s[8];
    load_scalar(s, scalars + FR_SZ * i);
    Fp tab[16];
    tab[0] = Q::infinity();
    tab[1] = Q::load_affine(pts + SizeOf<Q>::AFF * stride * i);
    tab[2] = Q::dbl(tab[1]);
    for (int d = 3; d < 16; d++) tab[d] = Q::add(tab[d - 1], tab[1], true);
    Fp acc = Q::infinity();
    bool started = false;
    for (int w = 63; w >= 0; w--) {
        if (started)
            for (int r = 0; r < 4; r++) acc = Q::dbl(acc);
        const uint32_t d = (s[w >> 3] >> (4 * (w & 7))) & 15u;
        if (!__any_sync(FULL, d != 0)) continue;
        started = true;
        acc = Q::add(acc, tab[d], d != 0);
    }
    const Fp r = Q::affine(acc);
    if (active) Q::store_affine(out + SizeOf<Q>::AFF * i, r);
}
template <class Q>
__global__ void __launch_bounds__(WARP) k_mul_batch(uint8_t* out, const uint8_t* pts, int64_t stride,
                                                    const uint8_t* scalars, int64_t n) {
    if constexpr (std::is_same<Q, Oct>::value) {
        using G = Oct::General;
        const int64_t p = point_index<Q>(), i = p < n ? p : n - 1;
        if (!__all_sync(FULL, G::on_curve(G::load_affine(pts + G1_AFF * stride * i)))) {
            mul_batch<G>(out, pts, stride, scalars, n);
            return;
        }
    }
    mul_batch<Q>(out, pts, stride, scalars, n);
}

// valid[i] = ([s_i] G == R_i + [c_i] X_i), four points per check: two take the
// digits of [c]X, two the even and odd bytes of [s]G from the generator table
template <class Q>
__device__ __forceinline__ void schnorr_verify(uint8_t* valid, const uint8_t* X, const uint8_t* R, const uint8_t* sresp,
                                               const uint8_t* c, int64_t n, const uint8_t* gen_table) {
    const int64_t p = point_index<Q>();
    const int sub = (int)(p & 3);
    const bool active = p / 4 < n;
    const int64_t i = active ? p / 4 : n - 1;
    uint32_t s[8];
    load_scalar(s, c + FR_SZ * i);
    uint64_t d[4], lo[1], hi[1];
    decompose_base_x(d, s);
    quad_digit<OnLane>(lo[0], hi[0], d, sub & 1);
    if (sub >= 2) lo[0] = hi[0] = 0;
    const Fp base[1] = {quad_image<Q>(Q::load_affine(X + G1_AFF * i), sub & 1)};
    Fp acc = quad_straus<Q>(base, lo, hi, 1);
    // R joins the first point's sum; -[s]G gathers on the third and fourth
    const uint8_t* sb = sresp + FR_SZ * i;
    for (int w = 0; w < 16; w++) {
        const uint32_t by = sub >= 2 ? sb[2 * w + (sub & 1)] : 0u;
        const uint8_t* src = sub >= 2 ? gen_table + G1_AFF * (256 * (2 * w + (sub & 1)) + by) : R + G1_AFF * i;
        Fp m = Q::load_affine(src);
        if (sub >= 2) m = Q::neg(m);
        acc = Q::add(acc, m, sub >= 2 ? by != 0 : (sub == 0 && w == 0));
    }
    acc = quad_sum<Q>(acc, 4);
    const bool inf = Q::is_inf(acc);
    if (active && sub == 0 && Q::place() == 0) valid[i] = inf ? 1 : 0;
}
template <class Q>
__global__ void __launch_bounds__(WARP) k_schnorr_verify(uint8_t* valid, const uint8_t* X, const uint8_t* R,
                                                         const uint8_t* sresp, const uint8_t* c, int64_t n,
                                                         const uint8_t* gen_table) {
    if constexpr (std::is_same<Q, Oct>::value) {
        using G = Oct::General;
        const int64_t p = point_index<Q>(), i = p / 4 < n ? p / 4 : n - 1;
        if (!__all_sync(FULL, G::on_curve(G::load_affine((p & 1 ? R : X) + G1_AFF * i)))) {
            schnorr_verify<G>(valid, X, R, sresp, c, n, gen_table);
            return;
        }
    }
    schnorr_verify<Q>(valid, X, R, sresp, c, n, gen_table);
}

// ------------------------------------------- fixed-base G2 MSMs of few terms
// For G2 points that stay fixed across many calls (a committee's verification
// keys), table[p][w][m - 1] = [m 64^w] P_p (w < FB_WINDOWS, 1 <= m <= 32,
// affine).  A term [s]P then costs one mixed addition per nonzero signed
// radix-64 digit of each base-|x| digit of s (digit c acting through
// (-1)^c psi^c, applied to the table entry), and no doublings.

// signed radix-64 digit k of d (d < 2^64): digits in [-31, 32], the carry
// into digit k set when the low k digits of d exceed 0x20..20 (32 in each)
WBTE_INL int r64_digit(uint64_t d, int k) {
    auto carry = [&](int j) -> int {
        if (j == 0 || 6 * j > 64) return 0;  // above bit 64 the bound exceeds any d < 2^64
        const uint64_t m = (1ull << (6 * j)) - 1;
        const uint64_t e = 0x820820820820820ull & m;  // 32 * 64^i summed over i < j
        return (d & m) > e;
    };
    const int nib = 6 * k < 64 ? (int)((d >> (6 * k)) & 63u) : 0;
    return nib + carry(k) - 64 * carry(k + 1);
}

// out[o] = sum_t scalars[vsel[o] n + t] * P(tbase[o] + tidx[t]), L pairs of lanes
// per output.  One pair takes the four digits in turn, applying |x| to its sum
// between them; of four or sixteen pairs each takes one digit (and of sixteen
// a quarter of its windows) and applies |x| to its own sum at the end.  Applied
// to sums instead of table entries, psi is 3 actions an output instead of 66 a
// term.  Measured on B200: 32,768 outputs of three terms 8.3 -> 6.1 ms; the
// six classes of 24 uneven weighted_pfe batches 36 -> 3.0 ms.
__global__ void __launch_bounds__(WARP) k_fixed_msm_g2(uint8_t* out, const uint8_t* tables, const int64_t* tbase,
                                                      const int32_t* tidx, const uint8_t* scalars, const int32_t* vsel,
                                                      int64_t k, int64_t n, int L) {
    using Pt = Point<OnPair>;
    const int64_t p = ((int64_t)blockIdx.x * WARP + threadIdx.x) / 2;
    const int sub = (int)(p % L), parts = L > 4 ? L / 4 : 1;
    const bool active = p / L < k;
    const int64_t o = active ? p / L : k - 1;
    const int64_t v = vsel ? (int64_t)vsel[o] : 0;
    Pt acc = Pt::infinity();
    const int digits = L == 1 ? 4 : 1;
    for (int i = 0; i < digits; i++) {
        const int c = L == 1 ? 3 - i : sub & 3;
        if (i) acc = Pt::image(acc);
        for (int64_t t = 0; t < n; t++) {
            const uint8_t* T = tables + FIXED_TABLE_BYTES * (tbase[o] + (tidx ? (int64_t)tidx[t] : t));
            uint32_t sc[8];
            load_scalar(sc, scalars + FR_SZ * (v * n + t));
            uint64_t d[4];
            decompose_base_x(d, sc);
            const uint64_t dc = c < 2 ? (c == 0 ? d[0] : d[1]) : (c == 2 ? d[2] : d[3]);
            for (int w0 = 0; w0 < FB_WINDOWS; w0 += parts) {
                const int w = w0 + sub / 4 % parts;
                const int dd = w < FB_WINDOWS ? r64_digit(dc, w) : 0;
                if (!__any_sync(FULL, dd != 0)) continue;
                const int a = dd < 0 ? -dd : dd;
                const uint8_t* e = T + G2_AFF * ((w < FB_WINDOWS ? w : 0) * FB_ENTRIES + (a ? a - 1 : 0));
                const Fp x = load_vec(Pt::at(e, 0)), y = load_vec(Pt::at(e, 1));
                acc = Pt::madd(acc, x, dd < 0 ? fp_neg(y) : y, dd != 0);
            }
        }
    }
    if (L > 1) {
        for (int i = 0; i < 3; i++) acc = Pt::select((sub & 3) > i, Pt::image(acc), acc);
        for (int w = 1; w < L; w *= 2) acc = Pt::add(acc, Pt::above(acc, 2 * w), true);
    }
    Fp x, y;
    acc.affine(x, y);
    if (active && sub == 0) {
        store_vec(const_cast<Fp*>(Pt::at(out + G2_AFF * o, 0)), x);
        store_vec(const_cast<Fp*>(Pt::at(out + G2_AFF * o, 1)), y);
    }
}

// out[i] = [scalars[i]] generator from its table [d 256^w]G at 256 w + d, L lanes (G1)
// or pairs (G2) per output: each adds every L-th byte's entry, the sums meet in a
// tree.  Measured on B200 against 32 additions by one thread: 512 outputs 0.36 ->
// 0.13 ms in G1 and 1.12 -> 0.19 ms in G2, 16,384 outputs 0.37 -> 0.31 and 1.13 ->
// 0.76 ms.
template <class P>
__global__ void __launch_bounds__(WARP) k_mul_generator(uint8_t* out, const uint8_t* table, const uint8_t* scalars,
                                                       int64_t n, int L) {
    using Pt = Point<P>;
    const int64_t p = ((int64_t)blockIdx.x * WARP + threadIdx.x) / P::LANES;
    const int sub = (int)(p % L);
    const bool active = p / L < n;
    const int64_t i = active ? p / L : n - 1;
    Pt acc = Pt::infinity();
    for (int w = sub; w < 32; w += L) {
        const uint32_t d = scalars[FR_SZ * i + w];
        if (!__any_sync(FULL, d != 0)) continue;
        const uint8_t* e = table + 2 * P::FIELD * (256 * w + d);
        acc = Pt::madd(acc, load_vec(Pt::at(e, 0)), load_vec(Pt::at(e, 1)), d != 0);
    }
    for (int w = 1; w < L; w *= 2) {
        const Pt up = Pt::above(acc, P::LANES * w);
        const bool live = !up.is_inf() && sub % (2 * w) == 0;
        if (__any_sync(FULL, live)) acc = Pt::add(acc, up, live);
    }
    Fp x, y;
    acc.affine(x, y);
    if (active && sub == 0) {
        store_vec(const_cast<Fp*>(Pt::at(out + 2 * P::FIELD * i, 0)), x);
        store_vec(const_cast<Fp*>(Pt::at(out + 2 * P::FIELD * i, 1)), y);
    }
}

}  // namespace

bool launch_quad_mul_generator(Group g, uint8_t* out, const uint8_t* table, const uint8_t* scalars, int64_t n, cudaStream_t s) {
    const bool g1 = g == GROUP_G1;
    const int lanes = g1 ? OnLane::LANES : OnPair::LANES;
    int L = 1;
    double best = 0;
    for (int l = 1; l <= 8; l *= 2) {  // products of a lane: 10 an entry, 14 a level of the tree, 60 the inversion
        const double levels = l == 8 ? 3 : l / 2;
        const double t = launch_time(320.0 / l + 14 * levels + 60, (double)n * l * lanes / WARP);
        if (l == 1 || t < best) best = t, L = l;
    }
    if (g1 && L == 1) return false;
    note_launch();
    const unsigned blocks = blocks_for(n * L * lanes, WARP);
    if (g1)
        k_mul_generator<OnLane><<<blocks, WARP, 0, s>>>(out, table, scalars, n, L);
    else
        k_mul_generator<OnPair><<<blocks, WARP, 0, s>>>(out, table, scalars, n, L);
    return true;
}

void launch_msm_combine(Group g, uint8_t* out, const uint8_t* wins, int64_t k, int windows, int c, cudaStream_t s) {
    note_launch();
    if (g == GROUP_G1)
        k_combine<Oct><<<blocks_for(k, SizeOf<Oct>::PER_WARP), WARP, 0, s>>>(out, wins, k, windows, c);
    else
        k_combine<Quad<OnPair, 8>><<<blocks_for(k, SizeOf<Quad<OnPair, 8>>::PER_WARP), WARP, 0, s>>>(out, wins, k, windows, c);
}

// doublings and additions of a multiple of one digit: 128 and 41 in G1, 64 and 24
// in G2
static ChainTime multiples_time(bool g1, double points, double alone) {
    return g1 ? chain_time(true, 128, 41, points, alone) : chain_time(false, 64, 24, points, alone);
}

// Steps of a transform of `bits` stages over `count` arrays: steps[i] stages each,
// the cheapest composition by the cost model; returns its time.
double quad_ntt_plan(Group g, int bits, int64_t count, int* steps, int* nsteps) {
    const bool g1 = g == GROUP_G1;
    const double points = (double)((int64_t)1 << bits) * (double)count;
    const int digits = g1 ? 2 : 4;
    // a pair's products keep two chains in flight: one warp fills a scheduler
    // (1,024 points in G2: 0.52 ms a stage at 0.9 warps, 1.05 ms at 2.2)
    const double alone = g1 ? 1.6 : 1.0;
    double best[64];
    int last[64];
    best[0] = 0;
    for (int done = 1; done <= bits; done++) {
        best[done] = -1;
        for (int kappa = 1; kappa <= 4 && kappa <= done; kappa++) {
            // a first step multiplies by powers of its own root only: one of a k's V_k is one
            const double multiples = ((double)((1 << (2 * kappa)) - 1) / 3.0) / (double)(1 << kappa) * points * digits;
            const double chain = done == kappa && kappa == 1 ? 0.0 : multiples_time(g1, multiples, alone).time;
            const double t = best[done - kappa] + chain +
                             launch_time(4.0 * kappa * (g1 ? 360.0 : 530.0), points / (g1 ? 8 : 4), alone);
            if (best[done] < 0 || t < best[done]) best[done] = t, last[done] = kappa;
        }
    }
    *nsteps = 0;
    for (int done = bits; done > 0; done -= last[done]) steps[(*nsteps)++] = last[done];
    std::reverse(steps, steps + *nsteps);
    return best[bits];
}

uint8_t* launch_quad_ntt(Group g, uint8_t* work, uint8_t* other, const uint8_t* tw, int64_t n, int64_t count, cudaStream_t s) {
    int bits = 0;
    while ((int64_t(1) << bits) < n) bits++;
    int steps[64], nsteps = 0;
    quad_ntt_plan(g, bits, count, steps, &nsteps);
    const bool g1 = g == GROUP_G1;
    const size_t rec = g1 ? G1_XYZZ : G2_XYZZ;
    const int per_warp = g1 ? SizeOf<G1Quad>::PER_WARP : SizeOf<G2Quad>::PER_WARP, digits = g1 ? 2 : 4;
    int64_t most = 0;
    for (int i = 0; i < nsteps; i++) most = std::max<int64_t>(most, ((1 << (2 * steps[i])) - 1) / 3 * (n >> steps[i]) * count);
    uint8_t* multiples = nullptr;
    if (cudaMallocAsync(&multiples, rec * (size_t)std::max<int64_t>(most, 1), s) != cudaSuccess) return nullptr;
    int64_t h = 1;
    for (int i = 0; i < nsteps; i++) {
        const int kappa = steps[i], per = ((1 << (2 * kappa)) - 1) / 3;
        const int64_t total = (n >> kappa) * count * per, outs = n * count;
        // sums: as many points per output as leave no scheduler waiting
        int L = 1;
        while (2 * L <= per_warp && 2 * L <= (1 << kappa) && (double)(outs * 2 * L) / per_warp <= 1.6 * schedulers()) L *= 2;
        note_launch(2);
        if (g1) {
            if (multiples_time(true, (double)(total * digits), 1.6).eight)
                k_ntt_multiples<Oct><<<blocks_for(total * digits, SizeOf<Oct>::PER_WARP), WARP, 0, s>>>(
                    multiples, work, tw, n, h, kappa, total, per);
            else
                k_ntt_multiples<G1Quad><<<blocks_for(total * digits, per_warp), WARP, 0, s>>>(multiples, work, tw, n, h, kappa,
                                                                                           total, per);
            k_ntt_sums<G1Quad><<<blocks_for(outs * L, per_warp), WARP, 0, s>>>(other, work, multiples, h, kappa, outs, per, L);
        } else {
            k_ntt_multiples<G2Quad><<<blocks_for(total * digits, per_warp), WARP, 0, s>>>(multiples, work, tw, n, h, kappa,
                                                                                       total, per);
            k_ntt_sums<G2Quad><<<blocks_for(outs * L, per_warp), WARP, 0, s>>>(other, work, multiples, h, kappa, outs, per, L);
        }
        std::swap(work, other);
        h <<= kappa;
    }
    cudaFreeAsync(multiples, s);
    return work;
}

void launch_quad_small_msm(Group g, uint8_t* out, const uint8_t* points, const int64_t* pbase, const int32_t* idx,
                           const uint8_t* scalars, const int32_t* vsel, int64_t k, int64_t n, int L, bool eight, cudaStream_t s) {
    note_launch();
    if (g == GROUP_G2)
        k_small_msm<G2Quad><<<blocks_for(L * k, SizeOf<G2Quad>::PER_WARP), WARP, 0, s>>>(out, points, pbase, idx, scalars,
                                                                                      vsel, k, n, L);
    else if (eight)
        k_small_msm<Oct><<<blocks_for(L * k, SizeOf<Oct>::PER_WARP), WARP, 0, s>>>(out, points, pbase, idx, scalars, vsel,
                                                                                k, n, L);
    else
        k_small_msm<G1Quad><<<blocks_for(L * k, SizeOf<G1Quad>::PER_WARP), WARP, 0, s>>>(out, points, pbase, idx, scalars,
                                                                                      vsel, k, n, L);
}

void launch_quad_mul_batch(Group g, uint8_t* out, const uint8_t* pts, int64_t stride, const uint8_t* scalars, int64_t n,
                           bool eight, cudaStream_t s) {
    note_launch();
    if (g == GROUP_G2)
        k_mul_batch<G2Quad><<<blocks_for(n, SizeOf<G2Quad>::PER_WARP), WARP, 0, s>>>(out, pts, stride, scalars, n);
    else if (eight)
        k_mul_batch<Oct><<<blocks_for(n, SizeOf<Oct>::PER_WARP), WARP, 0, s>>>(out, pts, stride, scalars, n);
    else
        k_mul_batch<G1Quad><<<blocks_for(n, SizeOf<G1Quad>::PER_WARP), WARP, 0, s>>>(out, pts, stride, scalars, n);
}

void launch_quad_schnorr_verify(uint8_t* valid, const uint8_t* X, const uint8_t* R, const uint8_t* sresp, const uint8_t* c,
                                int64_t n, const uint8_t* gen_table, bool eight, cudaStream_t s) {
    note_launch();
    if (eight)
        k_schnorr_verify<Oct><<<blocks_for(4 * n, SizeOf<Oct>::PER_WARP), WARP, 0, s>>>(valid, X, R, sresp, c, n, gen_table);
    else
        k_schnorr_verify<G1Quad><<<blocks_for(4 * n, SizeOf<G1Quad>::PER_WARP), WARP, 0, s>>>(valid, X, R, sresp, c, n,
                                                                                           gen_table);
}

void launch_fixed_msm_g2(uint8_t* out, const uint8_t* tables, const int64_t* tbase, const int32_t* tidx,
                         const uint8_t* scalars, const int32_t* vsel, int64_t k, int64_t n, cudaStream_t s) {
    ProfScope prof_("fixed_msm_g2", s);
    if (k <= 0) return;
    // mixed additions of one pair: 44 a term, or 11 or 3 and the tree's
    int L = 1;
    double best = launch_time(44.0 * n, (double)k / 16, 1.25);
    for (int pairs : {4, 16}) {
        const double t = launch_time((pairs == 4 ? 11.0 : 3.0) * n + 1.5 * (pairs == 4 ? 2 : 4), (double)k * pairs / 16, 1.25);
        if (t < best) best = t, L = pairs;
    }
    note_launch();
    k_fixed_msm_g2<<<blocks_for(2 * L * k, WARP), WARP, 0, s>>>(out, tables, tbase, tidx, scalars, vsel, k, n, L);
}

}  // namespace wbte
