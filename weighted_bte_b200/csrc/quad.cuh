// Curve arithmetic with one point spread over a quad: four places holding X, Y,
// ZZ and ZZZ of its XYZZ form.  A place is one lane in G1 and a pair of lanes in
// G2, the lanes of a pair holding the two Fp components of every Fp2 value.
//
// What bounds it: the length of the chain.  The kernels that use quads run one
// scalar multiple, Horner sum or butterfly per point in calls that leave most
// schedulers with less than one warp, where a dependent Fp product takes about
// 1 us whatever else runs.  A doubling is nine products in three rounds of up to
// four independent ones, an addition fourteen in four rounds, so a quad takes a
// third of one thread's time; it spends 12 and 16 product slots on them, so
// calls that fill the chip stay with one thread per point.  A pair takes an Fp2
// product as two sums of two products with one reduction each (444 wide
// multiply-adds per lane against 900 for three products on one lane).
//
// Measured on B200 against one thread per point (or per digit of it): the tail
// of a G1 MSM 4.0 -> 1.25 ms and of a G2 MSM 9.1 -> 1.8 ms, transforms of 1,024
// points 16.5 -> 2.9 ms in G1 and 26.0 -> 4.7 ms in G2, 512 Schnorr checks
// 2.9 -> 0.8 ms, 128 multiples in G1 3.3 -> 1.05 ms; G1 calls of fewer points take
// eight lanes (Oct).
//
// All lanes of a warp run every step (shuffles name the whole warp); special
// cases are selected afterwards.
#pragma once
#include "pairing.cuh"

namespace wbte {

constexpr uint32_t FULL = 0xffffffffu;

WBTE_INL Fp fp_shfl(const Fp& a, int src) {
    Fp r;
    _Pragma("unroll") for (int i = 0; i < 12; i++) r.v[i] = __shfl_sync(FULL, a.v[i], src);
    return r;
}
WBTE_INL Fp fp_shfl_xor(const Fp& a, int m) {
    Fp r;
    _Pragma("unroll") for (int i = 0; i < 12; i++) r.v[i] = __shfl_xor_sync(FULL, a.v[i], m);
    return r;
}
// ------------------------------------------------------------------ fields
// The field over the lanes of one place: every lane holds one Fp.  LANES lanes
// per value; product, square and the constants of the curve.
struct OnLane {  // Fp
    static constexpr int LANES = 1;
    static constexpr size_t FIELD = 48;  // bytes of a value in memory
    static constexpr bool G1 = true;
    static WBTE_INL Fp mul(const Fp& a, const Fp& b) { return fp_mul(a, b); }
    static WBTE_INL bool zero(const Fp& a) { return fp_is_zero(a); }
    // a value that several products use
    struct Shared { Fp own; };
    static WBTE_INL Shared share(const Fp& a) { return Shared{a}; }
    static WBTE_INL Fp mul(const Shared& a, const Shared& b) { return fp_mul(a.own, b.own); }
    static WBTE_INL Fp sqr(const Shared& a) { return fp_sqr(a.own); }
    // a b - c d
    static WBTE_INL Fp mul_sub(const Shared& a, const Shared& b, const Shared& c, const Shared& d) {
        return fp_mul2(a.own, b.own, fp_minus(c.own), d.own);
    }
    static WBTE_INL uint32_t all_lanes(uint32_t ballot) { return ballot; }
    static WBTE_INL Fp one() { return fp_one(); }
    static WBTE_INL Fp inv(const Fp& a) { return fp_inv(a); }
    // the curve's constant times a
    static WBTE_INL Fp times_b(const Fp& a) { return fp_dbl(fp_dbl(a)); }
};
struct OnPair {  // Fp2, component = lane parity
    static constexpr int LANES = 2;
    static constexpr size_t FIELD = 96;
    static constexpr bool G1 = false;
    static WBTE_INL bool odd() { return threadIdx.x & 1; }
    // even: a0 b0 + (-a1) b1, odd: a0 b1 + a1 b0; a < p, b < 4p
    static WBTE_INL Fp mul(const Fp& a, const Fp& b) {
        const Fp pa = fp_shfl_xor(a, 1), pb = fp_shfl_xor(b, 1);
        const Fp n = fp_minus(pa);
        return fp_mul2(fp_select(odd(), pa, a), b, fp_select(odd(), a, n), pb);
    }
    // a value that several products use, with the partner's component
    struct Shared { Fp own, other; };
    static WBTE_INL Shared share(const Fp& a) { return Shared{a, fp_shfl_xor(a, 1)}; }
    static WBTE_INL Fp mul(const Shared& a, const Shared& b) {
        return fp_mul2(fp_select(odd(), a.other, a.own), b.own, fp_select(odd(), a.own, fp_minus(a.other)), b.other);
    }
    // even: (a0 + a1)(a0 - a1), odd: a0 2a1
    static WBTE_INL Fp sqr(const Shared& a) {
        return fp_mul(fp_select(odd(), a.other, fp_add_lazy(a.own, a.other)),
                      fp_select(odd(), fp_add_lazy(a.own, a.own), fp_sub(a.own, a.other)));
    }
    static WBTE_INL Fp mul_sub(const Shared& a, const Shared& b, const Shared& c, const Shared& d) {
        return fp_sub(mul(a, b), mul(c, d));
    }
    // bits of the lanes whose pair agrees on a set bit
    static WBTE_INL uint32_t all_lanes(uint32_t ballot) {
        const uint32_t both = ballot & (ballot >> 1) & 0x55555555u;
        return both | (both << 1);
    }
    static WBTE_INL bool zero(const Fp& a) {
        const bool z = fp_is_zero(a);
        const bool o = __shfl_xor_sync(FULL, (int)z, 1);
        return z && o;
    }
    static WBTE_INL Fp one() { return fp_select(odd(), fp_zero(), fp_one()); }
    static WBTE_INL Fp inv(const Fp& a) {
        const Fp s = fp_sqr(a);
        const Fp n = fp_inv(fp_add(s, fp_shfl_xor(s, 1)));
        const Fp r = fp_mul(a, n);
        return fp_select(odd(), fp_neg(r), r);
    }
    // (1 + u) a
    static WBTE_INL Fp times_b4(const Fp& a) {
        const Fp o = fp_shfl_xor(a, 1);
        return fp_select(odd(), fp_add(a, o), fp_sub(a, o));
    }
    static WBTE_INL Fp times_b(const Fp& a) { return fp_dbl(fp_dbl(times_b4(a))); }
};

// ------------------------------------------------------------------- points
// With PLACES = 8 the places past the coordinates make room for the fifth
// product of a doubling in two rounds (dbl_on_curve).
template <class P, int PLACES = 4> struct Quad {
    using Field = P;
    static constexpr int L = P::LANES, WIDTH = PLACES * L;  // lanes per point
    static WBTE_INL int lane() { return threadIdx.x & 31; }
    static WBTE_INL int place() { return (lane() / L) & (PLACES - 1); }  // 0 X, 1 Y, 2 ZZ, 3 ZZZ
    // the value at place s of this point
    static WBTE_INL Fp from(const Fp& a, int s) { return fp_shfl(a, (lane() & ~(WIDTH - 1)) + s * L + (lane() & (L - 1))); }
    // whether `a` is zero at place s of this point
    static WBTE_INL bool zero_at(const Fp& a, int s) {
        const uint32_t z = __ballot_sync(FULL, P::zero(a));
        return (z >> ((lane() & ~(WIDTH - 1)) + s * L)) & 1;
    }
    static WBTE_INL Fp infinity() { return place() == 1 ? P::one() : fp_zero(); }
    static WBTE_INL bool is_inf(const Fp& p) { return zero_at(p, 2); }
    static WBTE_INL Fp neg(const Fp& p) { return place() == 1 ? fp_neg(p) : p; }
    // whether p is infinity or on the curve, Y^2 = X^3 + b ZZZ^2
    static WBTE_INL bool on_curve(const Fp& p) {
        const Fp s = P::mul(p, p), x3 = P::mul(s, p);
        const Fp d = fp_sub(fp_sub(from(s, 1), from(x3, 0)), P::times_b(from(s, 3)));
        const bool zero = zero_at(d, 0), inf = is_inf(p);
        return zero || inf;
    }

    // 2p (infinity stays infinity: ZZ = 0 is kept)
    static __device__ __noinline__ Fp dbl(Fp p) {
        const int c = place();
        const Fp u = c == 1 ? fp_dbl(p) : p;
        const Fp s1 = P::mul(u, u);  // X^2, V = U^2
        const Fp t = from(s1, c == 3 ? 0 : 1);
        const Fp x2 = c == 3 ? t : s1;
        const Fp M = fp_add(fp_dbl(x2), x2);  // at 0 and 3
        const bool mm = c == 3;
        const Fp s2 = P::mul(fp_select(mm, M, u), fp_select(mm, M, t));  // S, W, V ZZ, M^2
        const Fp g = from(s2, c == 0 ? 3 : 1);                            // M^2 at 0, W at 3
        const Fp X3 = fp_sub(fp_sub(g, s2), s2);                          // at 0
        // M (S - X3), W Y, -, W ZZZ
        const Fp s3 = P::mul(c == 0 ? M : (c == 1 ? s2 : g), c == 0 ? fp_sub(s2, X3) : p);
        const Fp y = fp_sub(from(s3, 0), s3);  // at 1
        return c == 0 ? X3 : (c == 1 ? y : (c == 2 ? s2 : s3));
    }

    // a for a < 4p
    static WBTE_INL Fp reduce4(Fp a) {
        fp_csub_2p(a.v, a.v);
        fp_csub_p(a.v, a.v);
        return a;
    }
    // 2p for p on the curve y^2 = x^3 + b, in two rounds of products instead of
    // three.  With B = Y^2 and c = b ZZZ^2 the curve's equation is X^3 = B - c,
    // and the doubled coordinates become
    //   X' = X (B - 9c)  Y' = (B + 9c)^2 - 108 c^2  ZZ' = 4B ZZ  ZZZ' = 8 Y B ZZZ,
    // the same values that dbl gives.  Sums enter products without reduction
    // (second factors stay below 4p).  G2 tails use it (2.1 -> 1.8 ms); G1 tails
    // run on eight lanes (Oct).
    static __device__ __noinline__ Fp dbl_on_curve(Fp p) {
        static_assert(PLACES == 8, "five products in the second round");
        const int c = place();
        const Fp s = from(p, c == 3 ? 1 : 3);  // Y at 3, ZZZ at 4
        const Fp z = c == 3 ? p : s;           // ZZZ at 3 and 4
        const Fp z2 = fp_add_lazy(z, z), z4 = fp_add_lazy(z2, z2);
        // B = Y Y, 4 Y ZZZ, 4 ZZZ^2
        const Fp r1 = P::mul(c == 1 ? p : s, c == 1 ? p : z4);
        Fp cc = P::times_b4(r1);  // at 4: b ZZZ^2
        const Fp e = from(reduce4(fp_add_lazy(fp_add_lazy(cc, cc), cc)), 4);  // 3c
        const Fp B = from(r1, 1);
        const Fp e3 = fp_add_lazy(fp_add_lazy(e, e), e);
        Fp m3;  // 3p - 3e
        fp_3p_minus(m3.v, e3.v);
        const Fp plus = reduce4(fp_add_lazy(B, e3)), B2 = fp_add_lazy(B, B), e2 = fp_add_lazy(e, e);
        // X (B - 9c), (B + 9c)^2, ZZ 4B, 4 Y ZZZ 2B, e 4e
        const Fp a = c == 1 ? plus : (c == 3 ? r1 : (c == 4 ? e : p));
        const Fp b = c == 0 ? fp_add_lazy(B, m3)
                            : (c == 1 ? plus : (c == 2 ? fp_add_lazy(B2, B2) : (c == 3 ? B2 : fp_add_lazy(e2, e2))));
        const Fp r2 = P::mul(a, b);
        const Fp t = from(r2, 4);  // 4 e^2, a third of 108 c^2
        Fp n3;
        fp_3p_minus(n3.v, fp_add_lazy(fp_add_lazy(t, t), t).v);
        return c == 1 ? reduce4(fp_add_lazy(r2, n3)) : r2;
    }

    // p + q; lanes of a point agree on `live` (false: p)
    static __device__ __noinline__ Fp add(Fp p, Fp q, bool live) {
        const int c = place();
        const Fp r1 = P::mul(p, from(q, c ^ 2));  // U1, S1, U2, S2
        const Fp o1 = from(r1, c ^ 2);
        const Fp d = c < 2 ? fp_sub(o1, r1) : fp_sub(r1, o1);  // P, R, P, R
        const Fp r2 = P::mul(c < 2 ? d : p, c < 2 ? d : q);    // PP, RR, ZZ1 ZZ2, ZZZ1 ZZZ2
        const Fp pp = from(r2, 0), dp = from(d, 0);
        // Q = U1 PP, PPP = P PP, ZZ3
        const Fp r3 = P::mul(c == 0 ? r1 : (c == 1 ? dp : r2), pp);
        const Fp t = from(fp_sub(r2, r3), 1);               // RR - PPP
        const Fp X3 = fp_sub(fp_sub(t, r3), r3);            // at 0
        const Fp g = from(c == 3 ? d : r3, c == 0 ? 3 : 1);  // R at 0, PPP at 3
        // R (Q - X3), S1 PPP, -, ZZZ1 ZZZ2 PPP
        const Fp r4 = P::mul(c == 0 ? g : (c == 1 ? r1 : r2), c == 0 ? fp_sub(r3, X3) : (c == 1 ? r3 : g));
        const Fp y = fp_sub(from(r4, 0), r4);
        Fp r = c == 0 ? X3 : (c == 1 ? y : (c == 2 ? r3 : r4));
        const bool pinf = is_inf(p), qinf = is_inf(q) || !live;
        const bool same_x = zero_at(d, 0) && !pinf && !qinf, same_y = zero_at(d, 1);
        if (__any_sync(FULL, same_x)) {
            const Fp two = dbl(p);
            if (same_x) r = same_y ? two : infinity();
        }
        if (pinf) r = q;
        if (qinf) r = p;
        return r;
    }

    // from and to memory: affine points in blst's layout, XYZZ records
    static WBTE_INL Fp load_affine(const uint8_t* pt) {
        const int c = place();
        const Fp v = load_vec(reinterpret_cast<const Fp*>(pt + (c & 1) * P::FIELD + 48 * (lane() & (L - 1))));
        const bool z = P::zero(v);
        const uint32_t b = __ballot_sync(FULL, z);
        const uint32_t both = b >> (lane() & ~(WIDTH - 1));
        const bool inf = (both & 1) && ((both >> L) & 1);
        const Fp hi = inf ? fp_zero() : P::one();
        return c < 2 ? (inf ? infinity() : v) : hi;
    }
    static WBTE_INL Fp load(const uint8_t* xyzz) {
        return load_vec(reinterpret_cast<const Fp*>(xyzz + (place() & 3) * P::FIELD + 48 * (lane() & (L - 1))));
    }
    static WBTE_INL void store(uint8_t* xyzz, const Fp& p) {
        if (place() < 4) store_vec(reinterpret_cast<Fp*>(xyzz + place() * P::FIELD + 48 * (lane() & (L - 1))), p);
    }
    // the affine x at place 0 and y at place 1 (zero for infinity)
    static WBTE_INL Fp affine(const Fp& p) {
        const Fp zz = from(p, 2), zzz = from(p, 3);
        const Fp t = P::inv(P::mul(zz, zzz));
        const Fp r = P::mul(p, P::mul(t, place() == 0 ? zzz : zz));
        return is_inf(p) ? fp_zero() : r;
    }
    static WBTE_INL void store_affine(uint8_t* pt, const Fp& a) {
        if (place() < 2) store_vec(reinterpret_cast<Fp*>(pt + place() * P::FIELD + 48 * (lane() & (L - 1))), a);
    }
    // the value of the point `points` further on in the warp
    static WBTE_INL Fp above(const Fp& p, int points) { return fp_shfl(p, (lane() + points * WIDTH) & 31); }
};

// G1 points for the calls with the fewest: homogeneous X, Y, Z at the first three
// of eight lanes, the others carry anything between operations.  Both operations
// are two rounds of products: the complete addition for odd order and a = 0 of
// Renes, Costello and Batina (six products in each round, no special cases to
// select) and the doubling that goes with it, on the isomorphic curve
// y^2 = x^3 + 2/3, where their 3b is 2: (x, y) -> (u^2 x, u^3 y), u^6 = 1/6.  That
// small constant and factors that are sums without reduction (their product
// below 9 p^2) leave the second round's factors a few carry chains away from the
// first's results, and one reduction at the end.
// Measured on B200 against quads: 512 Schnorr checks 0.81 -> 0.51 ms, 128
// multiples 1.05 -> 0.68 ms, transforms of 32 points 1.5 -> 1.05 ms, the tail of an
// MSM 1.11 -> 0.95 ms.  Eight lanes cost as many product slots as a quad for an
// addition and a third more for a doubling, so calls with more points than
// schedulers take quads (chain_time).
// These formulas use the curve's constant: of a point elsewhere they make another
// value than the XYZZ ones, or (0, 0, 0), which swallows every sum it enters and
// reads as infinity.  Kernels that multiply or add a caller's points look at them
// first and run General, an XYZZ point on the same lanes, where a warp holds one off
// the curve: two products of a chain of five hundred.  (Transforms do not look: outside
// the subgroup of order r their roots of unity are none.)
struct Oct {
    using Field = OnLane;
    using General = Quad<OnLane, 8>;
    static constexpr int WIDTH = 8;
    static WBTE_INL int lane() { return threadIdx.x & 31; }
    static WBTE_INL int place() { return lane() & 7; }
    static WBTE_INL Fp from(const Fp& a, int s) { return fp_shfl(a, (lane() & ~7) + s); }
    static WBTE_INL Fp above(const Fp& p, int points) { return fp_shfl(p, (lane() + points * WIDTH) & 31); }
    static WBTE_INL Fp infinity() { return place() == 1 ? fp_one() : fp_zero(); }
    static WBTE_INL bool is_inf(const Fp& p) { return (__ballot_sync(FULL, fp_is_zero(p)) >> ((lane() & ~7) + 2)) & 1; }
    static WBTE_INL Fp neg(const Fp& p) { return place() == 1 ? fp_neg(p) : p; }
    static WBTE_INL Fp reduce4(Fp a) {
        fp_csub_2p(a.v, a.v);
        fp_csub_p(a.v, a.v);
        return a;
    }

    // in line: the two operations together are four products (0.54 -> 0.51 ms for
    // Schnorr checks against calls)
    static WBTE_INL Fp mul(const Fp& a, const Fp& b) {
        Fp r;
        fp_mont_mul(r.v, a.v, b.v);
        return r;
    }

    // with B = Y^2 and z = Z^2: 2 XY (B - 6z), B^2 + 12 z (B - z), 8 YZ B
    static __device__ __noinline__ Fp dbl(Fp p) {
        const int c = place();
        const Fp s = from(p, c == 3 ? 2 : 1);
        const Fp r1 = mul(c == 3 ? s : p, s);  // XY, YY, ZY, ZZ
        const Fp B = from(r1, 1), z = from(r1, 3), n = fp_minus(z);
        const Fp n2 = fp_add_lazy(n, n), n6 = fp_add_lazy(fp_add_lazy(n2, n2), n2);
        const Fp z2 = fp_add_lazy(z, z), B2 = fp_add_lazy(B, B), B4 = fp_add_lazy(B2, B2);
        // XY (B - 6z), B B, YZ 8B, 4z (B - z)
        const Fp b = c == 1 ? B : fp_add_lazy(c == 2 ? B4 : B, c == 0 ? n6 : (c == 2 ? B4 : n));
        const Fp r2 = mul(c == 3 ? fp_add_lazy(z2, z2) : r1, b);
        const Fp t = from(r2, 3);
        const Fp more = c == 0 ? r2 : (c == 1 ? fp_add_lazy(fp_add_lazy(t, t), t) : fp_zero());
        return reduce4(fp_add_lazy(r2, more));
    }

    // with t0, t1, t2 = X1X2, Y1Y2, Z1Z2 and the mixed sums t3 = X1Y2 + X2Y1, t4 of
    // Y and Z, t5 of X and Z: X = t3 (t1 - 2 t2) - 2 t4 t5, Y = (t1 + 2 t2)(t1 - 2 t2)
    // + 6 t0 t5, Z = t4 (t1 + 2 t2) + 3 t0 t3.  Lanes of a point agree on `live`
    // (false: p).
    static __device__ __noinline__ Fp add(Fp p, Fp q, bool live) {
        const int c = place();
        const int i = (int)((0x00010210u >> (4 * c)) & 15u), j = (int)((0x00221000u >> (4 * c)) & 15u);
        const bool mixed = c >= 3;
        const Fp pj = from(p, j), qj = from(q, j), none = fp_zero();
        const Fp r1 = mul(fp_add_lazy(from(p, i), fp_select(mixed, pj, none)),
                             fp_add_lazy(from(q, i), fp_select(mixed, qj, none)));
        const Fp g = fp_minus(from(r1, i)), h = fp_minus(from(r1, j));
        const Fp t = fp_add_lazy(r1, fp_select(mixed, fp_add_lazy(g, h), none));  // below 3p
        // t3, t1 - 2 t2, t4 | t4, t5, t3 times t1 - 2 t2, t1 + 2 t2, t1 + 2 t2 | t5, 3 t0, 3 t0
        const Fp f = from(t, (int)((0x00354413u >> (4 * c)) & 15u)), e = from(t, (int)((0x00005111u >> (4 * c)) & 15u));
        const Fp t2 = from(t, 2), n = fp_minus(t2), n2 = fp_add_lazy(n, n);
        const Fp x = c == 3 ? none : (c > 3 ? e : (c == 0 ? n : t2));
        const Fp r2 = mul(fp_add_lazy(f, fp_select(c == 1, n2, none)), fp_add_lazy(e, fp_add_lazy(x, x)));
        const Fp o = from(r2, c < 3 ? c + 3 : c);
        const Fp y = c == 0 ? fp_minus(o) : o;
        const Fp r = reduce4(fp_add_lazy(fp_add_lazy(r2, y), c == 2 ? none : y));
        return live ? r : p;
    }

    // from and to memory: affine points in blst's layout, XYZZ records
    static WBTE_INL Fp load_affine(const uint8_t* pt) {
        const Fp v = load_vec(reinterpret_cast<const Fp*>(pt + 48 * (place() & 1)));
        const uint32_t zeros = __ballot_sync(FULL, fp_is_zero(v)) >> (lane() & ~7);
        const Fp k = fp_mul(v, fp_from_const(C_ISO_IN[place() & 1]));
        return (zeros & 3) == 3 ? infinity() : (place() < 2 ? k : (place() == 2 ? fp_one() : fp_zero()));
    }
    // x / zz and y / zzz over the common denominator zz zzz
    static WBTE_INL Fp load(const uint8_t* xyzz) {
        const Fp v = load_vec(reinterpret_cast<const Fp*>(xyzz + 48 * (place() & 3)));
        const Fp w = fp_mul(v, from(v, place() == 1 ? 2 : 3));
        const Fp r = fp_mul(w, place() < 2 ? fp_from_const(C_ISO_IN[place() & 1]) : fp_one());
        return is_inf(v) ? infinity() : r;
    }
    static WBTE_INL void store(uint8_t* xyzz, const Fp& p) {
        const int c = place();
        const Fp z = from(p, 2);
        const Fp z2 = fp_mul(z, z);
        // X z, Y z^2, z^2, z^3
        const Fp a = fp_mul(c < 2 ? p : z2, c == 1 ? z2 : z);
        const Fp r = fp_mul(c == 2 ? z2 : a, c < 2 ? fp_from_const(C_ISO_OUT[c & 1]) : fp_one());
        const Fp s = is_inf(p) ? infinity() : r;
        if (c < 4) store_vec(reinterpret_cast<Fp*>(xyzz + 48 * c), s);
    }
    static WBTE_INL Fp affine(const Fp& p) {
        const Fp r = fp_mul(fp_mul(p, fp_inv(from(p, 2))), fp_from_const(C_ISO_OUT[place() & 1]));
        return is_inf(p) ? fp_zero() : r;
    }
    static WBTE_INL void store_affine(uint8_t* pt, const Fp& a) {
        if (place() < 2) store_vec(reinterpret_cast<Fp*>(pt + 48 * place()), a);
    }
};

// ----------------------------------------------------- sums and multiples
// Q: a point's spread, Quad or Oct.
// sum over groups of n neighbouring points, valid in the first of each
template <class Q> WBTE_INL Fp quad_sum(Fp p, int n) {
    for (int w = 1; w < n; w *= 2) p = Q::add(p, Q::above(p, w), true);
    return p;
}

// The acting of |x|^j: on G2 (-1)^j psi^j, psi acting as [x].  G1 splits scalars
// in two 128-bit digits, the second acting as |x|^2 on phi(p) + p.
template <class Q> struct QuadDigits {
    static constexpr int DIGITS = Q::Field::G1 ? 2 : 4, TOP = Q::Field::G1 ? 32 : 16;
};
template <class Q> WBTE_INL Fp quad_image(Fp p, int j) {
    const int c = Q::place();
    if constexpr (Q::Field::G1) {
        const Fp f = c == 0 ? fp_mul(p, fp_from_const(C_GLV_BETA)) : p;
        const Fp s = Q::add(f, p, true);
        return j ? s : p;
    } else {
        for (int i = 0; i < 3; i++) {
            // conjugate every coordinate, scale x and y
            const Fp k = OnPair::odd() ? (c == 0 ? fp_from_const(C_PSI_CX[1]) : fp_from_const(C_PSI_CY[1]))
                                       : (c == 0 ? fp_from_const(C_PSI_CX[0]) : fp_from_const(C_PSI_CY[0]));
            const Fp cj = OnPair::odd() ? fp_neg(p) : p;
            const Fp m = Q::Field::mul(cj, k);
            const Fp n = Q::neg(c < 2 ? m : cj);
            if (i < j) p = n;
        }
        return p;
    }
}

// sum over r < n of [w_r] p_r for w_r = hi_r 2^64 + lo_r < 16^TOP, signed
// radix-16 digits over one run of doublings; terms past this point's own
// count have zero scalars
template <class Q, int N>
WBTE_INL Fp quad_straus(const Fp (&p)[N], const uint64_t (&lo)[N], const uint64_t (&hi)[N], int n) {
    constexpr int TOP = QuadDigits<Q>::TOP;
    Fp tab[N][8];
    for (int r = 0; r < n; r++) {
        tab[r][0] = p[r];
        tab[r][1] = Q::dbl(p[r]);
        for (int k = 2; k < 8; k++) tab[r][k] = Q::add(tab[r][k - 1], p[r], true);
    }
    Fp acc = Q::infinity();
    bool started = false;
    for (int k = TOP; k >= 0; k--) {
        if (started)
            for (int i = 0; i < 4; i++) acc = Q::dbl(acc);
        for (int r = 0; r < n; r++) {
            const int d = r16_digit(lo[r], hi[r], k, TOP);
            if (!__any_sync(FULL, d != 0)) continue;
            started = true;
            const int a = d < 0 ? -d : d;
            Fp m = tab[r][a ? a - 1 : 0];
            if (d < 0) m = Q::neg(m);
            acc = Q::add(acc, m, d != 0);
        }
    }
    return acc;
}

// the digits of a canonical scalar that act through quad_image
template <class P> WBTE_INL void quad_digit(uint64_t& lo, uint64_t& hi, const uint64_t d[4], int j) {
    if constexpr (P::G1) {
        const uint64_t plo = d[2 * j + 1] * X_ABS, phi = __umul64hi(d[2 * j + 1], X_ABS);
        lo = plo + d[2 * j];
        hi = phi + (lo < plo ? 1 : 0);
    } else {
        lo = d[j];
        hi = 0;
    }
}

// ------------------------------------------------- a point on one lane or pair
// For kernels that fill the chip: a lane (G1) or a pair (G2) holds all four
// coordinates.  In G2 that halves the registers of a point against one thread
// per point, which spilled its way through 255 of them, and takes an Fp2 product
// as 888 wide multiply-adds over the pair, none of its factors in local memory.
// Every lane of the warp runs every step, `live` says whose result counts.
template <class P> struct Point {
    Fp X, Y, ZZ, ZZZ;

    static WBTE_INL bool flag(bool mine) {
        return (P::all_lanes(__ballot_sync(FULL, mine)) >> (threadIdx.x & 31)) & 1;
    }
    static WBTE_INL Point infinity() { return Point{fp_zero(), P::one(), fp_zero(), fp_zero()}; }
    static WBTE_INL Point select(bool c, const Point& a, const Point& b) {
        return Point{fp_select(c, a.X, b.X), fp_select(c, a.Y, b.Y), fp_select(c, a.ZZ, b.ZZ), fp_select(c, a.ZZZ, b.ZZZ)};
    }
    WBTE_INL bool is_inf() const { return flag(fp_is_zero(ZZ)); }

    static __device__ __noinline__ Point dbl(Point p) {
        const typename P::Shared U = P::share(fp_dbl(p.Y)), X = P::share(p.X);
        const typename P::Shared V = P::share(P::sqr(U)), W = P::share(P::mul(U, V));
        const Fp S = P::mul(X, V), x2 = P::sqr(X);
        const typename P::Shared M = P::share(fp_add(fp_dbl(x2), x2));
        Point r;
        r.X = fp_sub(fp_sub(P::sqr(M), S), S);
        r.Y = P::mul_sub(M, P::share(fp_sub(S, r.X)), W, P::share(p.Y));
        r.ZZ = P::mul(V, P::share(p.ZZ));
        r.ZZZ = P::mul(W, P::share(p.ZZZ));
        return r;
    }
    // p + (x, y), zero for infinity
    static __device__ __noinline__ Point madd(Point p, Fp x, Fp y, bool live) {
        const typename P::Shared ZZ = P::share(p.ZZ), ZZZ = P::share(p.ZZZ);
        const Fp d = fp_sub(P::mul(P::share(x), ZZ), p.X), e = fp_sub(P::mul(P::share(y), ZZZ), p.Y);
        Point r = chord(p.X, p.Y, P::share(d), P::share(e), ZZ, ZZZ);
        const bool qinf = flag(fp_is_zero(x) && fp_is_zero(y)) || !live, pinf = p.is_inf();
        const bool same = flag(fp_is_zero(d)) && !pinf && !qinf, twice = flag(fp_is_zero(e));
        if (__any_sync(FULL, same)) {
            const Point two = dbl(p);
            r = select(same, select(twice, two, infinity()), r);
        }
        r = select(pinf, Point{x, y, P::one(), P::one()}, r);
        return select(qinf, p, r);
    }
    static __device__ __noinline__ Point add(Point p, Point q, bool live) {
        const typename P::Shared ZZ1 = P::share(p.ZZ), ZZZ1 = P::share(p.ZZZ);
        const typename P::Shared ZZ2 = P::share(q.ZZ), ZZZ2 = P::share(q.ZZZ);
        const Fp u = P::mul(P::share(p.X), ZZ2), s = P::mul(P::share(p.Y), ZZZ2);
        const Fp d = fp_sub(P::mul(P::share(q.X), ZZ1), u), e = fp_sub(P::mul(P::share(q.Y), ZZZ1), s);
        Point r = chord(u, s, P::share(d), P::share(e), P::share(P::mul(ZZ1, ZZ2)), P::share(P::mul(ZZZ1, ZZZ2)));
        const bool pinf = p.is_inf(), qinf = q.is_inf() || !live;
        const bool same = flag(fp_is_zero(d)) && !pinf && !qinf, twice = flag(fp_is_zero(e));
        if (__any_sync(FULL, same)) {
            const Point two = dbl(p);
            r = select(same, select(twice, two, infinity()), r);
        }
        r = select(pinf, q, r);
        return select(qinf, p, r);
    }
    // (u, s) and (u + d, s + e) over the common denominators
    static WBTE_INL Point chord(const Fp& u, const Fp& s, const typename P::Shared& d, const typename P::Shared& e,
                                const typename P::Shared& ZZ, const typename P::Shared& ZZZ) {
        const typename P::Shared PP = P::share(P::sqr(d)), PPP = P::share(P::mul(d, PP));
        const Fp Q = P::mul(P::share(u), PP);
        Point r;
        r.X = fp_sub(fp_sub(fp_sub(P::sqr(e), PPP.own), Q), Q);
        r.Y = P::mul_sub(e, P::share(fp_sub(Q, r.X)), P::share(s), PPP);
        r.ZZ = P::mul(ZZ, PP);
        r.ZZZ = P::mul(ZZZ, PPP);
        return r;
    }
    // [g]p, the lanes running the longest of their multiples' bits
    static WBTE_INL Point multiple(const Point& p, uint32_t g) {
        Point r = infinity();
        for (int b = 31 - __clz(__reduce_or_sync(FULL, g) | 1); b >= 0; b--) {
            r = dbl(r);
            if (__any_sync(FULL, (g >> b) & 1)) r = add(r, p, (g >> b) & 1);
        }
        return r;
    }

    // the action of |x| on G2: -psi
    static WBTE_INL Point image(const Point& p) {
        const auto conj = [](const Fp& a) { return OnPair::odd() ? fp_neg(a) : a; };
        const Fp kx = fp_select(OnPair::odd(), fp_from_const(C_PSI_CX[1]), fp_from_const(C_PSI_CX[0]));
        const Fp ky = fp_select(OnPair::odd(), fp_from_const(C_PSI_CY[1]), fp_from_const(C_PSI_CY[0]));
        return Point{P::mul(conj(p.X), kx), fp_neg(P::mul(conj(p.Y), ky)), conj(p.ZZ), conj(p.ZZZ)};
    }
    // the point `by` lanes further on
    static WBTE_INL Point above(const Point& p, int by) {
        const int l = ((threadIdx.x & 31) + by) & 31;
        return Point{fp_shfl(p.X, l), fp_shfl(p.Y, l), fp_shfl(p.ZZ, l), fp_shfl(p.ZZZ, l)};
    }
    // X and Y of the affine point (zero for infinity)
    WBTE_INL void affine(Fp& x, Fp& y) const {
        const Fp t = P::inv(P::mul(ZZ, ZZZ));
        const bool inf = is_inf();
        const Fp ax = P::mul(X, P::mul(t, ZZZ)), ay = P::mul(Y, P::mul(t, ZZ));
        x = fp_select(inf, fp_zero(), ax);
        y = fp_select(inf, fp_zero(), ay);
    }

    // this lane's component of coordinate i of a record in memory
    static WBTE_INL const Fp* at(const uint8_t* rec, int i) {
        return reinterpret_cast<const Fp*>(rec + i * P::FIELD + 48 * (threadIdx.x & (P::LANES - 1)));
    }
    WBTE_INL void store(uint8_t* rec) const {
        store_vec(const_cast<Fp*>(at(rec, 0)), X);
        store_vec(const_cast<Fp*>(at(rec, 1)), Y);
        store_vec(const_cast<Fp*>(at(rec, 2)), ZZ);
        store_vec(const_cast<Fp*>(at(rec, 3)), ZZZ);
    }
};

}  // namespace wbte
