// Fp12 arithmetic with one element spread over a team of six lanes: lane k
// holds the Fp2 coefficient of w^k (w^6 = xi = 1 + u), five teams per warp.  Calls
// of few values take teams of twelve (below).
//
// What bounds it: the wide multiply-add pipe (a 32 x 32 + 64-bit multiply-add
// every four cycles per scheduler).  One thread per element needs 288 words
// for two operands and streams them through local memory; a lane of a team
// holds 24 words per operand, so nothing spills, a chain of products is six
// times shorter for calls that do not fill the chip, and products can stay
// double width until the six coefficients are put together: an Fp12 product
// is 18 Fp2 products of three 12 x 12-word products each (nine per lane) and
// one Montgomery reduction per output component (two per lane), 1,608 wide
// multiply-adds per lane and 9,648 in all against 16,200 for 54 reduced Fp
// products.
//
// Measured on B200 against one thread per element (one batch of B = 512, then
// 64 of them): truncated GT transform 48 -> 2.8 ms and 82 -> 44 ms, hard parts
// 10.7 -> 1.4 ms and 15.0 -> 12.3 ms, prepared Miller loops 7.2 -> 0.9 ms and
// 21.4 -> 15.0 ms, opening multi-Miller loops of three pairs 20.4 -> 15.7 ms
// (64 batches).  At 64 batches the multiply-add pipe is 55-62 % busy: the
// rest is the latency of carry chains between products, with two warps per
// scheduler, and instruction fetch.
//
// Lanes meet in shared memory: rows of 32 16-byte vectors, a value of a lane
// being one column ("slot") of consecutive rows, so that the lanes of a warp
// touch distinct bank groups.  Slot 31 of every row is zero (the absent second
// term of a Karatsuba sum).  Lanes 30 and 31 shadow lanes 24 and 25: they
// compute and store the same values to the same places.
//
// Double-width values are kept modulo 2^768 in two's complement; the sums that
// are reduced are bounded integers (bounds at each use), shifted to be
// non-negative by a multiple of p 2^384 before the reduction.
#pragma once
#include "quad.cuh"

namespace wbte {

constexpr int TEAMS = 5;  // of six lanes per warp
// Resident one-warp blocks per SM that the team kernels are compiled for: the
// registers of eight warps, two per scheduler.  Ten and twelve (168 registers)
// measured 45.9 -> 56 and 57 ms for the GT transform of 64 batches of 512 and
// changed the hard parts by 1 %: what more warps hide they lose to
// instruction fetch (the loop's 45 KB) and to the tables' share of L1.
constexpr int T6_BLOCKS = 8;
constexpr int T6_ZERO = 31;
// rows: three double-width exchange areas (12 each), the first also holding the
// operands A and B
constexpr int T6_A = 0, T6_B = 6, T6_X = 0, T6_Y = 12, T6_Z = 24, T6_ROWS = 36;
constexpr int T6_BYTES = T6_ROWS * 32 * 16;

struct Wide { uint32_t v[24]; };
struct Wide2 { Wide c0, c1; };

struct Team {
    uint4* sh;  // this warp's rows
    int k;      // this lane's power of w
    int h;      // this lane's component of the coefficient (teams of twelve)
    int base;   // slot of the team's coefficient 0
};

WBTE_INL int nib(uint32_t packed, int k) { return (int)((packed >> (4 * k)) & 15u); }

// `per` teams per warp of `lanes` lanes (a multiple of six: one lane or two
// neighbours per coefficient); lanes past them shadow the last team's
WBTE_INL Team team_init(uint4* sh, int lanes, int per) {
    const int lane = threadIdx.x & 31;
    const int used = lanes * per, each = lanes / 6;
    const int l = lane < used ? lane : used - lanes + (lane - used) % lanes;
    Team t;
    t.sh = sh;
    t.k = l % lanes / each;
    t.h = l % each;
    t.base = 6 * (l / lanes);
    for (int r = lane; r < T6_ROWS; r += 32) sh[r * 32 + T6_ZERO] = make_uint4(0, 0, 0, 0);
    __syncwarp();
    return t;
}

template <class T> WBTE_INL T team_ld(const Team& t, int row, int slot) {
    T r;
    uint4* d = reinterpret_cast<uint4*>(&r);
    const uint4* s = t.sh + row * 32 + slot;
    _Pragma("unroll") for (int i = 0; i < (int)(sizeof(T) / 16); i++) d[i] = s[i * 32];
    return r;
}
template <class T> WBTE_INL void team_st(const Team& t, int row, int slot, const T& v) {
    const uint4* s = reinterpret_cast<const uint4*>(&v);
    uint4* d = t.sh + row * 32 + slot;
    _Pragma("unroll") for (int i = 0; i < (int)(sizeof(T) / 16); i++) d[i * 32] = s[i];
}

// ------------------------------------------------------------ double width
WBTE_INL Wide fp_wide_inl(const Fp& a, const Fp& b) { Wide r; fp_mul_wide(r.v, a.v, b.v); return r; }
static __device__ __noinline__ Wide fp_wide(Fp a, Fp b) { return fp_wide_inl(a, b); }
// t / 2^384 mod p for 0 <= t < 3 p 2^384
static __device__ __noinline__ Fp wide_reduce(Wide t) {
    Fp r;
    fp_redc(r.v, t.v);
    fp_csub_2p(r.v, r.v);
    fp_csub_p(r.v, r.v);
    return r;
}
WBTE_INL Wide w_add(const Wide& a, const Wide& b) { Wide r; wide_add(r.v, a.v, b.v); return r; }
WBTE_INL Wide w_sub(const Wide& a, const Wide& b) { Wide r; wide_sub(r.v, a.v, b.v); return r; }
WBTE_INL Wide2 w2_add(const Wide2& a, const Wide2& b) { return Wide2{w_add(a.c0, b.c0), w_add(a.c1, b.c1)}; }
WBTE_INL Wide2 w2_sub(const Wide2& a, const Wide2& b) { return Wide2{w_sub(a.c0, b.c0), w_sub(a.c1, b.c1)}; }
WBTE_INL Fp2 fp2_add_lazy(const Fp2& a, const Fp2& b) { return Fp2{fp_add_lazy(a.c0, b.c0), fp_add_lazy(a.c1, b.c1)}; }

// a b for components whose sums stay below 2^384 (8 p)
WBTE_INL Wide2 fp2_wide(const Fp2& a, const Fp2& b) {
    const Wide x = fp_wide(a.c0, b.c0), y = fp_wide(a.c1, b.c1);
    const Wide z = fp_wide(fp_add_lazy(a.c0, a.c1), fp_add_lazy(b.c0, b.c1));
    return Wide2{w_sub(x, y), w_sub(w_sub(z, x), y)};
}
// the same in line: faster where a kernel's loop holds few of them (Miller loops
// of one pair each 1.02 -> 0.89 ms), slower in t6_mul (GT transforms of 64
// batches 44 -> 57 ms, instruction fetch)
WBTE_INL Wide2 fp2_wide_inl(const Fp2& a, const Fp2& b) {
    const Wide x = fp_wide_inl(a.c0, b.c0), y = fp_wide_inl(a.c1, b.c1);
    const Wide z = fp_wide_inl(fp_add_lazy(a.c0, a.c1), fp_add_lazy(b.c0, b.c1));
    return Wide2{w_sub(x, y), w_sub(w_sub(z, x), y)};
}
// reductions of sums in (-19.6 p^2, 9.8 p^2) and (-9.8 p^2, 19.6 p^2)
WBTE_INL Fp2 w2_reduce_21(Wide2 t) {
    fp_add_2p(t.c0.v + 12, t.c0.v + 12);
    fp_add_p(t.c1.v + 12, t.c1.v + 12);
    return Fp2{wide_reduce(t.c0), wide_reduce(t.c1)};
}
// both in (-9.8 p^2, 19.6 p^2)
WBTE_INL Fp2 w2_reduce_11(Wide2 t) {
    fp_add_p(t.c0.v + 12, t.c0.v + 12);
    fp_add_p(t.c1.v + 12, t.c1.v + 12);
    return Fp2{wide_reduce(t.c0), wide_reduce(t.c1)};
}
// one lane's Fp2 product, components below 4 p: two reductions instead of three
static __device__ __noinline__ Fp2 t6_fp2_mul(Fp2 a, Fp2 b) { return w2_reduce_11(fp2_wide_inl(a, b)); }

// --------------------------------------------------------- Fp12 products
// The Karatsuba products of an Fp6 product, one per lane: x0y0, x1y1, x2y2,
// (x1+x2)(y1+y2), (x0+x1)(y0+y1), (x0+x2)(y0+y2).  Slots of a lane's two terms
// in the even half (c0); the odd half is one slot up.
WBTE_INL int t6_term0(const Team& t) { return t.base + 2 * nib(0x001210u, t.k); }
WBTE_INL int t6_term1(const Team& t) {
    const int j = nib(0x212fffu, t.k);
    return j == 15 ? T6_ZERO : t.base + 2 * j;
}
WBTE_INL int t6_odd(int slot) { return slot == T6_ZERO ? slot : slot + 1; }
WBTE_INL Fp2 t6_pair(const Team& t, int row, int s0, int s1) {
    return fp2_add_lazy(team_ld<Fp2>(t, row, s0), team_ld<Fp2>(t, row, s1));
}

// Where coefficient i of an Fp6 product takes its Karatsuba products from:
//   i = 0: X0 + xi (X3 - X1 - X2)   i = 1: X4 - X0 - X1 + xi X2
//   i = 2: X5 - X0 - X2 + X1
// as G + H + (xi - 1) M with G = X[g0] - X[g1] - X[g2], H = X[h] and M = G or
// X[m]; (xi - 1) M = (-M1, M0).
struct T6Comb { int row, g0, g1, g2, h, m; bool gm; };
WBTE_INL T6Comb t6_comb_of(const Team& t, int row) {
    const int i = t.k >> 1;
    T6Comb c;
    c.row = row;
    c.g0 = t.base + 3 + i;
    c.g1 = t.base + (i == 0 ? 1 : 0);
    c.g2 = t.base + (i == 1 ? 1 : 2);
    c.h = t.base + (i == 0 ? 0 : (i == 1 ? 2 : 1));
    c.m = i == 1 ? c.h : T6_ZERO;
    c.gm = i == 0;
    return c;
}
WBTE_INL Wide2 t6_comb(const Team& t, const T6Comb& c) {
    Wide2 G = w2_sub(w2_sub(team_ld<Wide2>(t, c.row, c.g0), team_ld<Wide2>(t, c.row, c.g1)),
                     team_ld<Wide2>(t, c.row, c.g2));
    Wide2 M = team_ld<Wide2>(t, c.row, c.m);
    _Pragma("unroll") for (int i = 0; i < 24; i++) {
        M.c0.v[i] = c.gm ? G.c0.v[i] : M.c0.v[i];
        M.c1.v[i] = c.gm ? G.c1.v[i] : M.c1.v[i];
    }
    G = w2_add(G, team_ld<Wide2>(t, c.row, c.h));
    return Wide2{w_sub(G.c0, M.c1), w_add(G.c1, M.c0)};
}
// the slot of the odd lane whose v-multiple joins this (even) lane's output:
// v (e0 + e1 v + e2 v^2) = xi e2 + e0 v + e1 v^2
WBTE_INL int t6_vslot(const Team& t) {
    const int i = t.k >> 1;
    return t.base + 2 * (i == 0 ? 2 : i - 1) + 1;
}
// a b.  With a = a0 + a1 w, b = b0 + b1 w: c0 = a0 b0 + v a1 b1 and
// c1 = (a0 + a1)(b0 + b1) - a0 b0 - a1 b1, every Fp6 product by its Karatsuba
// products.  As integers the outputs are sums of one product and five
// xi-multiples at most: components in (-16 p^2, 6 p^2) and (-5 p^2, 17 p^2).
static __device__ __noinline__ Fp2 t6_mul(Team t, Fp2 a, Fp2 b) {
    const int own = t.base + t.k;
    const bool odd = t.k & 1;
    __syncwarp();
    team_st(t, T6_A, own, a);
    team_st(t, T6_B, own, b);
    __syncwarp();
    const int s0 = t6_term0(t), s1 = t6_term1(t);
    Fp2 u = t6_pair(t, T6_A, s0, s1), v = t6_pair(t, T6_B, s0, s1);
    const Fp2 u1 = t6_pair(t, T6_A, t6_odd(s0), t6_odd(s1)), v1 = t6_pair(t, T6_B, t6_odd(s0), t6_odd(s1));
    __syncwarp();
    Wide2 x = fp2_wide(u, v);
    team_st(t, T6_X, own, x);
    {
        const Wide2 y = fp2_wide(u1, v1);
        team_st(t, T6_Y, own, y);
        x = w2_add(x, y);
        u = fp2_add_lazy(u, u1);
        v = fp2_add_lazy(v, v1);
    }
    team_st(t, T6_Z, own, w2_sub(fp2_wide(u, v), x));
    __syncwarp();
    // first the coefficients of a0 b0 (even lanes) and a1 b1 (odd lanes), then
    // the odd lanes' own and, on the even ones, v a1 b1 joining their a0 b0
    T6Comb c = t6_comb_of(t, odd ? T6_Y : T6_X);
    const Wide2 e = t6_comb(t, c);
    __syncwarp();
    team_st(t, T6_X, own, e);
    __syncwarp();
    if (odd) {
        c.row = T6_Z;
    } else {
        c.row = T6_X;
        c.g0 = t6_vslot(t);
        c.g1 = c.g2 = c.m = T6_ZERO;
        c.h = own;
    }
    return w2_reduce_21(t6_comb(t, c));
}

// a^2 by complex squaring: c1 = 2 a0 a1, c0 = (a0 + a1)(a0 + v a1) - a0 a1 -
// v a0 a1.  v a1 is taken with its coefficient xi a12 reduced, which adds
// a0i ((xi a12 mod p) - xi a12), components in [0, 2 p^2) and (-p^2, p^2), to
// the integer value: (-14 p^2, 8 p^2) and (-5 p^2, 17 p^2).
static __device__ __noinline__ Fp2 t6_sqr(Team t, Fp2 a) {
    const int own = t.base + t.k;
    const bool odd = t.k & 1;
    __syncwarp();
    team_st(t, T6_A, own, a);
    if (odd) team_st(t, T6_B, t.base + 2 * (t.k == 5 ? 0 : (t.k >> 1) + 1) + 1, t.k == 5 ? fp2_mul_xi(a) : a);
    __syncwarp();
    const int s0 = t6_term0(t), s1 = t6_term1(t);
    const Fp2 u0 = t6_pair(t, T6_A, s0, s1), u1 = t6_pair(t, T6_A, t6_odd(s0), t6_odd(s1));
    const Fp2 v1 = t6_pair(t, T6_B, t6_odd(s0), t6_odd(s1));
    __syncwarp();
    const Wide2 x = fp2_wide_inl(u0, u1);
    team_st(t, T6_X, own, x);
    team_st(t, T6_Y, own, w2_sub(fp2_wide_inl(fp2_add_lazy(u0, u1), fp2_add_lazy(u0, v1)), x));
    __syncwarp();
    T6Comb c = t6_comb_of(t, odd ? T6_X : T6_Y);
    team_st(t, T6_Z, own, t6_comb(t, c));
    __syncwarp();
    // odd lanes double, even lanes subtract v a0 a1
    c.row = T6_Z;
    c.g0 = odd ? own : T6_ZERO;
    c.g1 = odd ? T6_ZERO : t6_vslot(t);
    c.g2 = c.m = T6_ZERO;
    c.h = own;
    c.gm = c.gm && !odd;
    return w2_reduce_21(t6_comb(t, c));
}

// Granger-Scott squaring in the cyclotomic subgroup: even lanes hold
// a^2 + xi b^2, odd lanes 2ab of the pairs (w^0, w^3), (w^1, w^4), (w^2, w^5),
// and z' = 3t -+ 2z.  Lane 1 takes xi 2ab of the pair (w^2, w^5), lane 4 its
// a^2 + xi b^2.  Four 12 x 12-word products on each lane:
//   even: A = (a0+a1)(a0-a1)  B = 2a0 a1  C = (b0+b1)(b0-b1)  D = 2b0 b1
//   odd:  A = 2a0 b0          B = 2a0 b1  C = 2a1 b0          D = 2a1 b1
//   c0 = A + [even] C - D,  c1 = B + C + [even] D
// Which value a factor starts from differs between the lanes, so they read it
// from the place it has in shared memory instead of selecting it: c0, c1, p -
// c1 and (for lane 1) xi z without reduction.  Most lanes' time besides the
// products goes into carry chains, and this is two thirds of the chains of a
// form with selections and a branch per parity; the four products stand in
// line, which lets their chains overlap (hard parts of 32,768 values 15.2 ->
// 13.7 ms against calls).  Components: (-4 p^2, 8 p^2) and [0, 12 p^2) at lane 1,
// inside that elsewhere.
static __device__ __noinline__ Fp2 t6_cyc_sqr(Team t, Fp2 z) {
    constexpr int C0 = 0, C1 = 3, NEG = 6, XI0 = 9, XI1 = 12;
    const bool even = !(t.k & 1);
    const int own = t.base + t.k;
    Fp n, m;
    fp_p_minus(n.v, z.c1.v);
    __syncwarp();
    team_st(t, C0, own, z.c0);
    team_st(t, C1, own, z.c1);
    team_st(t, NEG, own, n);
    team_st(t, XI0, own, fp_add_lazy(z.c0, n));
    team_st(t, XI1, own, fp_add_lazy(z.c0, z.c1));
    __syncwarp();
    const int pa = t.base + nib(0x120120u, t.k), pb = pa + 3;
    const int a0r = t.k == 1 ? XI0 : C0, a1r = t.k == 1 ? XI1 : C1;
    const Fp a0 = team_ld<Fp>(t, a0r, pa), b0 = team_ld<Fp>(t, C0, pb), b1 = team_ld<Fp>(t, C1, pb);
    const Fp d = team_ld<Fp>(t, even ? C0 : a1r, even ? pb : pa);  // b0 or a1
    const Wide A = fp_wide_inl(fp_add_lazy(a0, team_ld<Fp>(t, even ? C1 : a0r, pa)),
                               fp_add_lazy(team_ld<Fp>(t, C0, even ? pa : pb), team_ld<Fp>(t, NEG, even ? pa : T6_ZERO)));
    const Wide B = fp_wide_inl(fp_add_lazy(a0, a0), team_ld<Fp>(t, C1, even ? pa : pb));
    const Wide C = fp_wide_inl(fp_add_lazy(d, team_ld<Fp>(t, even ? C1 : a1r, even ? pb : pa)),
                               fp_add_lazy(b0, team_ld<Fp>(t, NEG, even ? pb : T6_ZERO)));
    const Wide D = fp_wide_inl(fp_add_lazy(d, d), b1);
    const uint32_t mask = even ? 0xffffffffu : 0u;
    Wide c, e;
    _Pragma("unroll") for (int i = 0; i < 24; i++) {
        c.v[i] = C.v[i] & mask;
        e.v[i] = D.v[i] & mask;
    }
    c = w_sub(w_add(A, c), D);
    fp_add_p(c.v + 12, c.v + 12);
    e = w_add(w_add(B, C), e);
    Fp2 q;
    fp_redc(q.c0.v, c.v);
    fp_redc(q.c1.v, e.v);
    fp_csub_2p(q.c0.v, q.c0.v);
    fp_csub_2p(q.c1.v, q.c1.v);
    // 3q -+ 2z = 2 (q + (p - z or z)) + q, below 8p
    fp_p_minus(m.v, z.c0.v);
    m = fp_select(even, m, z.c0);
    q.c0 = fp_add_lazy(fp_add_lazy(q.c0, q.c0), fp_add_lazy(q.c0, fp_add_lazy(m, m)));
    n = fp_select(even, n, z.c1);
    q.c1 = fp_add_lazy(fp_add_lazy(q.c1, q.c1), fp_add_lazy(q.c1, fp_add_lazy(n, n)));
    fp_csub_4p(q.c0.v, q.c0.v);
    fp_csub_4p(q.c1.v, q.c1.v);
    fp_csub_2p(q.c0.v, q.c0.v);
    fp_csub_2p(q.c1.v, q.c1.v);
    fp_csub_p(q.c0.v, q.c0.v);
    fp_csub_p(q.c1.v, q.c1.v);
    return q;
}

// f (l0 + l1 w^2 + l2 w^3) with the line's six Fp components in rows T6_Y.. of
// the team's slots (component c of the record at slot base + c): three Fp2
// products per lane, no exchange after them.  Components in (-3 p^2, 3 p^2)
// and [0, 6 p^2).
WBTE_INL Fp2 team_ld_line(const Team& t, int row, int c) {
    return Fp2{team_ld<Fp>(t, row, t.base + 2 * c), team_ld<Fp>(t, row, t.base + 2 * c + 1)};
}
static __device__ __noinline__ Fp2 t6_mul_line(Team t, Fp2 f, Fp line_component) {
    const int own = t.base + t.k;
    __syncwarp();
    team_st(t, T6_A, own, f);
    team_st(t, T6_B, own, fp2_mul_xi(f));
    team_st(t, T6_Y, own, line_component);
    __syncwarp();
    Wide2 acc = fp2_wide_inl(f, team_ld_line(t, T6_Y, 0));
    const int k2 = t.k < 2 ? t.k + 4 : t.k - 2, k3 = t.k < 3 ? t.k + 3 : t.k - 3;
    acc = w2_add(acc, fp2_wide_inl(team_ld<Fp2>(t, t.k < 2 ? T6_B : T6_A, t.base + k2), team_ld_line(t, T6_Y, 1)));
    acc = w2_add(acc, fp2_wide_inl(team_ld<Fp2>(t, t.k < 3 ? T6_B : T6_A, t.base + k3), team_ld_line(t, T6_Y, 2)));
    return w2_reduce_11(acc);
}

// ------------------------------------------------------------- teams of twelve
// Two lanes per coefficient, one Fp component each: for calls of so few values
// that a team's own chain is all that counts.  An Fp2 product is two 12 x
// 12-word products on each lane, without Karatsuba (c0 = a0 b0 - a1 b1, c1 = a0
// b1 + a1 b0): 1,020 wide multiply-adds per lane and Fp12 product against 1,608,
// 444 per cyclotomic squaring against 888, at two teams per warp instead of
// five: slower once every scheduler has its warps.  Measured on B200, 100 values
// (six lanes, twelve): final exponentiations 1.49 and 0.92 ms, Miller loops of
// computed lines 1.76 and 1.04 ms, of prepared ones 0.89 and 0.63 ms; 500
// products of three pairings 3.6 and 2.65 ms with the call.
WBTE_INL Wide w_add_signed(const Wide& a, const Wide& b, bool minus) {
    const uint32_t m[1] = {minus ? 0xffffffffu : 0u};
    Wide r;
    wide_add_signed(r.v, a.v, b.v, m);
    return r;
}
WBTE_INL Wide w_partner(const Wide& a) {
    Wide r;
    _Pragma("unroll") for (int i = 0; i < 24; i++) r.v[i] = __shfl_xor_sync(FULL, a.v[i], 1);
    return r;
}
// this lane's component of u v
WBTE_INL Wide t12_wide(const Team& t, const Fp2& u, const Fp2& v) {
    const Wide x = fp_wide_inl(u.c0, fp_select(t.h, v.c1, v.c0)), y = fp_wide_inl(u.c1, fp_select(t.h, v.c0, v.c1));
    return w_add_signed(x, y, !t.h);
}
WBTE_INL Fp t12_reduce(const Team& t, Wide s, bool two) {
    fp_add_p(s.v + 12, s.v + 12);
    if (two) {  // the first component's sums reach -16 p^2
        Fp hi, more;
        _Pragma("unroll") for (int i = 0; i < 12; i++) hi.v[i] = s.v[12 + i];
        fp_add_p(more.v, hi.v);
        _Pragma("unroll") for (int i = 0; i < 12; i++) s.v[12 + i] = t.h ? hi.v[i] : more.v[i];
    }
    return wide_reduce(s);
}
WBTE_INL Wide t12_comb(const Team& t, const T6Comb& c) {
    const int row = c.row + 6 * t.h;
    Wide G = w_sub(w_sub(team_ld<Wide>(t, row, c.g0), team_ld<Wide>(t, row, c.g1)), team_ld<Wide>(t, row, c.g2));
    Wide M = team_ld<Wide>(t, row, c.m);
    _Pragma("unroll") for (int i = 0; i < 24; i++) M.v[i] = c.gm ? G.v[i] : M.v[i];
    G = w_add(G, team_ld<Wide>(t, row, c.h));
    return w_add_signed(G, w_partner(M), !t.h);
}
static __device__ __noinline__ Fp t12_mul(Team t, Fp a, Fp b) {
    const int own = t.base + t.k;
    const bool odd = t.k & 1;
    __syncwarp();
    team_st(t, T6_A + 3 * t.h, own, a);
    team_st(t, T6_B + 3 * t.h, own, b);
    __syncwarp();
    const int s0 = t6_term0(t), s1 = t6_term1(t);
    const Fp2 u = t6_pair(t, T6_A, s0, s1), v = t6_pair(t, T6_B, s0, s1);
    const Fp2 u1 = t6_pair(t, T6_A, t6_odd(s0), t6_odd(s1)), v1 = t6_pair(t, T6_B, t6_odd(s0), t6_odd(s1));
    __syncwarp();
    const Wide x = t12_wide(t, u, v);
    team_st(t, T6_X + 6 * t.h, own, x);
    const Wide y = t12_wide(t, u1, v1);
    team_st(t, T6_Y + 6 * t.h, own, y);
    const Wide z = t12_wide(t, fp2_add_lazy(u, u1), fp2_add_lazy(v, v1));
    team_st(t, T6_Z + 6 * t.h, own, w_sub(w_sub(z, x), y));
    __syncwarp();
    T6Comb c = t6_comb_of(t, odd ? T6_Y : T6_X);
    const Wide e = t12_comb(t, c);
    __syncwarp();
    team_st(t, T6_X + 6 * t.h, own, e);
    __syncwarp();
    if (odd) {
        c.row = T6_Z;
    } else {
        c.row = T6_X;
        c.g0 = t6_vslot(t);
        c.g1 = c.g2 = c.m = T6_ZERO;
        c.h = own;
    }
    return t12_reduce(t, t12_comb(t, c), true);
}
WBTE_INL Fp t12_xi(const Team& t, const Fp& a) {
    const Fp o = fp_shfl_xor(a, 1);
    return fp_select(t.h, fp_add(a, o), fp_sub(a, o));
}
static __device__ __noinline__ Fp t12_sqr(Team t, Fp a) {
    const int own = t.base + t.k;
    const bool odd = t.k & 1;
    const Fp xa = t12_xi(t, a);
    __syncwarp();
    team_st(t, T6_A + 3 * t.h, own, a);
    if (odd) team_st(t, T6_B + 3 * t.h, t.base + 2 * (t.k == 5 ? 0 : (t.k >> 1) + 1) + 1, t.k == 5 ? xa : a);
    __syncwarp();
    const int s0 = t6_term0(t), s1 = t6_term1(t);
    const Fp2 u0 = t6_pair(t, T6_A, s0, s1), u1 = t6_pair(t, T6_A, t6_odd(s0), t6_odd(s1));
    const Fp2 v1 = t6_pair(t, T6_B, t6_odd(s0), t6_odd(s1));
    __syncwarp();
    const Wide x = t12_wide(t, u0, u1);
    team_st(t, T6_X + 6 * t.h, own, x);
    team_st(t, T6_Y + 6 * t.h, own, w_sub(t12_wide(t, fp2_add_lazy(u0, u1), fp2_add_lazy(u0, v1)), x));
    __syncwarp();
    T6Comb c = t6_comb_of(t, odd ? T6_X : T6_Y);
    team_st(t, T6_Z + 6 * t.h, own, t12_comb(t, c));
    __syncwarp();
    c.row = T6_Z;
    c.g0 = odd ? own : T6_ZERO;
    c.g1 = odd ? T6_ZERO : t6_vslot(t);
    c.g2 = c.m = T6_ZERO;
    c.h = own;
    c.gm = c.gm && !odd;
    return t12_reduce(t, t12_comb(t, c), true);
}
// the four products of t6_cyc_sqr, A and D on the first lane, B and C on the
// second; even coefficients exchange C and D
static __device__ __noinline__ Fp t12_cyc_sqr(Team t, Fp z) {
    constexpr int C0 = 0, C1 = 3, NEG = 6, XI0 = 9, XI1 = 12, UNUSED = 15;
    const bool even = !(t.k & 1), h = t.h;
    const int own = t.base + t.k;
    const Fp o = fp_shfl_xor(z, 1);
    const Fp n = fp_minus(h ? z : o);  // p - c1
    __syncwarp();
    team_st(t, h ? C1 : C0, own, z);
    team_st(t, h ? NEG : XI0, own, h ? n : fp_add_lazy(z, n));
    team_st(t, h ? XI1 : UNUSED, own, fp_add_lazy(z, o));
    __syncwarp();
    const int pa = t.base + nib(0x120120u, t.k), pb = pa + 3;
    const int a0r = t.k == 1 ? XI0 : C0, a1r = t.k == 1 ? XI1 : C1;
    const Fp a0 = team_ld<Fp>(t, a0r, pa);
    const Fp d = team_ld<Fp>(t, even ? C0 : a1r, even ? pb : pa);  // b0 or a1
    // A = (a0 + a1 or a0)(a0 or b0, less a1 or not) and B = 2a0 (a1 or b1)
    const Wide x = fp_wide_inl(fp_add_lazy(a0, team_ld<Fp>(t, even && !h ? C1 : a0r, pa)),
                               fp_add_lazy(team_ld<Fp>(t, h ? C1 : C0, even ? pa : pb),
                                           team_ld<Fp>(t, NEG, even && !h ? pa : T6_ZERO)));
    // D = 2d b1 and C = (d + b1 or a1)(b0, less b1 or not)
    const Wide y = fp_wide_inl(fp_add_lazy(d, team_ld<Fp>(t, even ? (h ? C1 : C0) : a1r, even ? pb : pa)),
                               fp_add_lazy(team_ld<Fp>(t, h ? C0 : C1, pb),
                                           team_ld<Fp>(t, NEG, even && h ? pb : T6_ZERO)));
    Wide w = w_partner(y);
    const uint32_t mask = even ? 0xffffffffu : 0u;
    _Pragma("unroll") for (int i = 0; i < 24; i++) w.v[i] &= mask;
    w = w_add_signed(w_add(x, w), y, !h);
    fp_add_p(w.v + 12, w.v + 12);
    Fp q;
    fp_redc(q.v, w.v);
    fp_csub_2p(q.v, q.v);
    const Fp m = fp_select(even, fp_minus(z), z);
    q = fp_add_lazy(fp_add_lazy(q, q), fp_add_lazy(q, fp_add_lazy(m, m)));
    fp_csub_4p(q.v, q.v);
    fp_csub_2p(q.v, q.v);
    fp_csub_p(q.v, q.v);
    return q;
}
static __device__ __noinline__ Fp t12_mul_line(Team t, Fp f, int component, Fp line_component) {
    const int own = t.base + t.k;
    const Fp xf = t12_xi(t, f);
    __syncwarp();
    team_st(t, T6_A + 3 * t.h, own, f);
    team_st(t, T6_B + 3 * t.h, own, xf);
    team_st(t, T6_Y, t.base + component, line_component);
    __syncwarp();
    const int k2 = t.k < 2 ? t.k + 4 : t.k - 2, k3 = t.k < 3 ? t.k + 3 : t.k - 3;
    Wide acc = t12_wide(t, team_ld<Fp2>(t, T6_A, own), team_ld_line(t, T6_Y, 0));
    acc = w_add(acc, t12_wide(t, team_ld<Fp2>(t, t.k < 2 ? T6_B : T6_A, t.base + k2), team_ld_line(t, T6_Y, 1)));
    acc = w_add(acc, t12_wide(t, team_ld<Fp2>(t, t.k < 3 ? T6_B : T6_A, t.base + k3), team_ld_line(t, T6_Y, 2)));
    return t12_reduce(t, acc, false);
}

// the canonical value as 48 big-endian bytes
WBTE_INL void fp_store_be48(uint8_t* out, const Fp& m) {
    Fp c = fp_from_mont(m);
    for (int i = 0; i < 48; i++) out[47 - i] = (uint8_t)(c.v[i >> 2] >> (8 * (i & 3)));
}

// --------------------------------------------------- what both kinds of team do
// E: what a lane holds of an Fp12 value's coefficient, and so of any Fp2 value
// that the team computes with.
struct Six {
    using E = Fp2;
    static constexpr int LANES = 6, PER = TEAMS, WARPS = 1;
    static WBTE_INL void step() {}
    static WBTE_INL E mul(const Team& t, const E& a, const E& b) { return t6_mul(t, a, b); }
    static WBTE_INL E sqr(const Team& t, const E& a) { return t6_sqr(t, a); }
    static WBTE_INL E cyc_sqr(const Team& t, const E& a) { return t6_cyc_sqr(t, a); }
    static WBTE_INL E mul_line(const Team& t, const E& f, const Fp& c) { return t6_mul_line(t, f, c); }
    // the record component that this lane brings of a line
    static WBTE_INL int line_index(const Team& t) { return t.k; }
    static WBTE_INL Fp component(const E& a, int c) { return c ? a.c1 : a.c0; }
    static WBTE_INL E of(const Team&, const Fp2& a) { return a; }
    static WBTE_INL E load(const Team&, const uint8_t* v) { return load_vec(reinterpret_cast<const Fp2*>(v)); }
    static WBTE_INL void store(const Team&, uint8_t* v, const E& a) { store_vec(reinterpret_cast<Fp2*>(v), a); }
    static WBTE_INL void store_be(const Team&, uint8_t* v, const E& a) {
        fp_store_be48(v, a.c0);
        fp_store_be48(v + 48, a.c1);
    }
    static WBTE_INL bool same(const E& a, const E& b) { return fp_eq(a.c0, b.c0) && fp_eq(a.c1, b.c1); }
    static WBTE_INL E ld(const Team& t, int row, int slot) { return team_ld<Fp2>(t, row, slot); }
    static WBTE_INL void st(const Team& t, int row, int slot, const E& a) { team_st(t, row, slot, a); }
    static WBTE_INL E f_add(const E& a, const E& b) { return fp2_add(a, b); }
    static WBTE_INL E f_sub(const E& a, const E& b) { return fp2_sub(a, b); }
    static WBTE_INL E f_neg(const E& a) { return fp2_neg(a); }
    static WBTE_INL E f_xi(const Team&, const E& a) { return fp2_mul_xi(a); }
    static WBTE_INL E f_conj(const Team&, const E& a) { return fp2_conj(a); }
    static WBTE_INL E f_mul(const E& a, const E& b) { return t6_fp2_mul(a, b); }
};
struct Twelve {
    using E = Fp;
    static constexpr int LANES = 12, PER = 2, WARPS = 1;
    static WBTE_INL void step() {}
    static WBTE_INL E mul(const Team& t, const E& a, const E& b) { return t12_mul(t, a, b); }
    static WBTE_INL E sqr(const Team& t, const E& a) { return t12_sqr(t, a); }
    static WBTE_INL E cyc_sqr(const Team& t, const E& a) { return t12_cyc_sqr(t, a); }
    static WBTE_INL E mul_line(const Team& t, const E& f, const Fp& c) { return t12_mul_line(t, f, line_index(t), c); }
    static WBTE_INL int line_index(const Team& t) { return 2 * (t.k % 3) + t.h; }
    static WBTE_INL Fp component(const E& a, int) { return a; }
    static WBTE_INL E of(const Team& t, const Fp2& a) { return fp_select(t.h, a.c1, a.c0); }
    static WBTE_INL E load(const Team& t, const uint8_t* v) { return load_vec(reinterpret_cast<const Fp*>(v) + t.h); }
    static WBTE_INL void store(const Team& t, uint8_t* v, const E& a) { store_vec(reinterpret_cast<Fp*>(v) + t.h, a); }
    static WBTE_INL void store_be(const Team& t, uint8_t* v, const E& a) { fp_store_be48(v + 48 * t.h, a); }
    static WBTE_INL bool same(const E& a, const E& b) { return fp_eq(a, b); }
    static WBTE_INL E ld(const Team& t, int row, int slot) { return team_ld<Fp>(t, row + 3 * t.h, slot); }
    static WBTE_INL void st(const Team& t, int row, int slot, const E& a) { team_st(t, row + 3 * t.h, slot, a); }
    static WBTE_INL E f_add(const E& a, const E& b) { return fp_add(a, b); }
    static WBTE_INL E f_sub(const E& a, const E& b) { return fp_sub(a, b); }
    static WBTE_INL E f_neg(const E& a) { return fp_neg(a); }
    static WBTE_INL E f_xi(const Team& t, const E& a) { return t12_xi(t, a); }
    static WBTE_INL E f_conj(const Team& t, const E& a) { return fp_select(t.h, fp_neg(a), a); }
    static WBTE_INL E f_mul(const E& a, const E& b) { return OnPair::mul(a, b); }
};
// Six, in blocks of four warps that meet before each step of a loop: warps that
// drift apart fetch 45 KB of loop body each for itself, warps in step share the
// fetches.  Measured on B200 for 64 batches of 512: GT transform 44.5 -> 39.9
// ms (of its stalls the missing instructions fall from 20 to 8 %), Miller loops
// of six computed pairs 14.5 -> 11.4, of prepared lines 15.0 -> 14.2 and, three
// pairs at a time, 15.6 -> 15.3.  Two warps: 42.9, 13.4, 14.7 and 15.2; eight
// (one block per SM) 44.1, 11.1, 16.3 and 16.4.  Hard parts, whose loop is one
// squaring, 12.2 -> 12.4, so they stay apart.
struct SixBlock : Six {
    static constexpr int WARPS = 4;
    static WBTE_INL void step() { __syncthreads(); }
};
template <class T> using ElemOf = typename T::E;
template <class T> WBTE_INL ElemOf<T> team_dbl(const ElemOf<T>& a) { return T::f_add(a, a); }
template <class T> WBTE_INL ElemOf<T> team_mul3(const ElemOf<T>& a) { return T::f_add(T::f_add(a, a), a); }
template <class T> WBTE_INL ElemOf<T> team_mul4(const ElemOf<T>& a) { return team_dbl<T>(team_dbl<T>(a)); }

template <class T> WBTE_INL Team team_of(uint4* sh, int per = T::PER) {
    return team_init(sh + (T::WARPS > 1 ? (threadIdx.x >> 5) * (T6_ROWS * 32) : 0), T::LANES, per);
}
// this lane's team in the launch (shadow lanes belong to the warp's last one);
// kernels have teams past the end take the last value again without storing it,
// which is their own warp's, so that a call may work in place
template <class T> __device__ __forceinline__ int64_t team_index(int per = T::PER) {
    const int tm = (int)(threadIdx.x & 31) / T::LANES;
    const int64_t warp = T::WARPS > 1 ? (int64_t)blockIdx.x * T::WARPS + (threadIdx.x >> 5) : (int64_t)blockIdx.x;
    return warp * per + (tm < per ? tm : per - 1);
}

template <class T> WBTE_INL ElemOf<T> team_one(const Team& t) {
    Fp2 r = fp2_zero();
    if (t.k == 0) r.c0 = fp_one();
    return T::of(t, r);
}
template <class T> WBTE_INL ElemOf<T> team_conj(const Team& t, const ElemOf<T>& a) {
    const ElemOf<T> n = T::f_neg(a);
    return (t.k & 1) ? n : a;
}
// x^(p^pw), pw in 1..3
template <class T> static __device__ __noinline__ ElemOf<T> team_frobenius(Team t, ElemOf<T> a, int pw) {
    const ElemOf<T> c = T::f_conj(t, a);
    a = (pw & 1) ? c : a;
    return T::f_mul(a, T::of(t, fp2_from_const(C_FROB[pw - 1][t.k])));
}

// coefficient k in blst's Fp12 layout (c0.c0, c0.c1, c0.c2, c1.c0, ..)
WBTE_INL size_t team_offset(const Team& t) { return 96 * (size_t)((t.k & 1) * 3 + (t.k >> 1)); }
template <class T> WBTE_INL ElemOf<T> team_load(const Team& t, const uint8_t* gt) { return T::load(t, gt + team_offset(t)); }
template <class T> WBTE_INL void team_store(const Team& t, uint8_t* gt, const ElemOf<T>& a) {
    T::store(t, gt + team_offset(t), a);
}

// ------------------------------------------------------ final exponentiation
// 1/d for the Fp2 value d that is coefficient 0
template <class T> WBTE_INL ElemOf<T> team_inverse_of_first(const Team& t, const ElemOf<T>& a) {
    __syncwarp();
    T::st(t, T6_A, t.base + t.k, a);
    __syncwarp();
    return T::of(t, fp2_inv(team_ld<Fp2>(t, T6_A, t.base)));
}
// f^((p^6 - 1)(p^2 + 1)) = (conj(f)^2 / (f conj(f)))^(p^2 + 1).  N = f conj(f)
// lies in Fp6, and 1/N = N^(p^2) N^(p^4) / (N N^(p^2) N^(p^4)), whose
// denominator lies in Fp2.  f = 0 gives 0.
template <class T> static __device__ __noinline__ ElemOf<T> team_final_exp_easy(Team t, ElemOf<T> f) {
    const ElemOf<T> g = team_conj<T>(t, f);
    const ElemOf<T> n = T::mul(t, f, g);
    const ElemOf<T> n2 = team_frobenius<T>(t, n, 2);
    const ElemOf<T> m = T::mul(t, n2, team_frobenius<T>(t, n2, 2));
    const ElemOf<T> d = team_inverse_of_first<T>(t, T::mul(t, n, m));
    const ElemOf<T> r = T::mul(t, T::mul(t, g, g), T::f_mul(m, d));
    return T::mul(t, r, team_frobenius<T>(t, r, 2));
}
// x^(|z|/2) conjugated: squaring runs between the set bits of |z|
template <class T> static __device__ __noinline__ ElemOf<T> team_raise_to_z_div_by_2(Team t, ElemOf<T> x) {
    ElemOf<T> acc = T::cyc_sqr(t, x);
    const uint64_t runs = 2ull | (3ull << 8) | (9ull << 16) | (32ull << 24) | (15ull << 32);
    for (int r = 0; r < 5; r++) {
        acc = T::mul(t, acc, x);
        for (int i = (int)((runs >> (8 * r)) & 255u); i > 0; i--) acc = T::cyc_sqr(t, acc);
    }
    return team_conj<T>(t, acc);
}
template <class T> WBTE_INL ElemOf<T> team_raise_to_z(const Team& t, const ElemOf<T>& x) {
    return T::cyc_sqr(t, team_raise_to_z_div_by_2<T>(t, x));
}
// the addition chain of btx/src/final_exponentiation.rs:255-283 (raise_to_z at
// :399-413), which computes f^(3 (p^4 - p^2 + 1) / r)
template <class T> static __device__ __noinline__ ElemOf<T> team_final_exp_hard(Team t, ElemOf<T> in) {
    const ElemOf<T> y0 = T::cyc_sqr(t, in);
    ElemOf<T> y1 = team_raise_to_z<T>(t, y0);
    ElemOf<T> y2 = team_raise_to_z_div_by_2<T>(t, y1);
    y1 = team_conj<T>(t, T::mul(t, y1, team_conj<T>(t, in)));
    y1 = T::mul(t, y1, y2);
    y2 = team_raise_to_z<T>(t, y1);
    ElemOf<T> y3 = team_raise_to_z<T>(t, y2);
    y1 = team_conj<T>(t, y1);
    y3 = T::mul(t, y3, y1);
    y1 = team_frobenius<T>(t, team_conj<T>(t, y1), 3);
    y1 = T::mul(t, y1, team_frobenius<T>(t, y2, 2));
    y2 = T::mul(t, team_raise_to_z<T>(t, y3), y0);
    y1 = T::mul(t, y1, T::mul(t, y2, in));
    return T::mul(t, y1, team_frobenius<T>(t, y3, 1));
}

// The launch of a kernel over `items` values, `per` of them to a warp
template <class T, class K, class... A> void team_launch(K* kernel, int64_t items, int per, cudaStream_t s, A... args) {
    constexpr int bytes = T::WARPS * T6_BYTES;
    if (bytes > 48 * 1024) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    const int64_t each = (int64_t)per * T::WARPS;
    kernel<<<(unsigned)((items + each - 1) / each), 32 * T::WARPS, bytes, s>>>(args...);
}

// -------------------------------------------------------------- Miller loops
// Lines (pairing.cuh) enter as their six Fp components, already scaled by (1, 1,
// xP, xP, yP, yP).
WBTE_INL bool miller_bit(int i) { return (X_ABS >> i) & 1; }

// this lane's scale for lines through P; identities get the line 1
struct TeamPoint { Fp scale; bool inf; };
template <class T> WBTE_INL TeamPoint team_point(const Team& t, const G1A& P) {
    const int c = T::line_index(t);
    TeamPoint r;
    r.inf = is_inf(P);
    r.scale = c < 2 ? fp_one() : (c < 4 ? P.x : P.y);
    return r;
}
template <class T> WBTE_INL Fp team_line_value(const Team& t, const Fp& component, const TeamPoint& P) {
    const Fp v = fp_mul(component, P.scale);
    const Fp id = T::line_index(t) == 0 ? fp_one() : fp_zero();
    return P.inf ? id : v;
}

// G2 point of a running loop in homogeneous coordinates: X, Y, Z at
// coefficients 0, 1, 2 (the others carry anything).  The products of a step go
// one to a coefficient; every lane forms the sums it needs from shared memory.
constexpr int T6_P = T6_Y, T6_Q = T6_Y + 6, T6_R = T6_Z, T6_S = T6_Z + 6;
template <class T> WBTE_INL void team_exchange(const Team& t, int row, const ElemOf<T>& v) {
    T::st(t, row, t.base + t.k, v);
    __syncwarp();
}
// S <- 2S; returns this lane's component of the tangent line
template <class T> static __device__ __noinline__ Fp team_line_double(Team t, ElemOf<T>& S) {
    using E = ElemOf<T>;
    __syncwarp();
    team_exchange<T>(t, T6_P, S);
    // Y Y, Z Z, X X, Y Z, X Y
    team_exchange<T>(t, T6_Q, T::f_mul(T::ld(t, T6_P, t.base + nib(0x001021u, t.k)),
                                       T::ld(t, T6_P, t.base + nib(0x112021u, t.k))));
    const E t0 = T::ld(t, T6_Q, t.base);
    const E t2 = team_mul4<T>(team_mul3<T>(T::f_xi(t, T::ld(t, T6_Q, t.base + 1))));  // 3 b' Z^2
    const E t23 = team_mul3<T>(t2);
    const E YZ = T::ld(t, T6_Q, t.base + 3);
    // XY (t0 - t23), (t0 + t23)^2, t2^2, t0 YZ
    E a = t0, b = YZ;
    if (t.k == 0) {
        a = T::ld(t, T6_Q, t.base + 4);
        b = T::f_sub(t0, t23);
    } else if (t.k == 1) {
        a = b = T::f_add(t0, t23);
    } else if (t.k == 2) {
        a = b = t2;
    }
    __syncwarp();
    team_exchange<T>(t, T6_R, T::f_mul(a, b));
    if (t.k == 0) {
        S = team_dbl<T>(T::ld(t, T6_R, t.base));
    } else if (t.k == 1) {
        S = T::f_sub(T::ld(t, T6_R, t.base + 1), team_mul4<T>(team_mul3<T>(T::ld(t, T6_R, t.base + 2))));
    } else {
        S = team_mul4<T>(team_dbl<T>(T::ld(t, T6_R, t.base + 3)));
    }
    const int c = T::line_index(t);
    E l;
    if (c < 2) {
        l = T::f_sub(t2, t0);
    } else if (c < 4) {
        l = team_mul3<T>(T::ld(t, T6_Q, t.base + 2));
    } else {
        l = T::f_neg(team_dbl<T>(YZ));
    }
    return T::component(l, c & 1);
}
// S <- S + Q; returns this lane's component of the chord
template <class T> static __device__ __noinline__ Fp team_line_add(Team t, ElemOf<T>& S, const G2A& Q) {
    using E = ElemOf<T>;
    __syncwarp();
    team_exchange<T>(t, T6_P, S);
    const E X = T::ld(t, T6_P, t.base), Y = T::ld(t, T6_P, t.base + 1), Z = T::ld(t, T6_P, t.base + 2);
    const E qx = T::of(t, Q.x), qy = T::of(t, Q.y);
    team_exchange<T>(t, T6_Q, T::f_mul(t.k == 0 ? qy : qx, Z));
    const E u = T::f_sub(T::ld(t, T6_Q, t.base), Y), v = T::f_sub(T::ld(t, T6_Q, t.base + 1), X);
    // u u, v v, u xQ, v yQ
    team_exchange<T>(t, T6_R, T::f_mul((t.k == 0 || t.k == 2) ? u : v, t.k == 0 ? u : (t.k == 1 ? v : (t.k == 2 ? qx : qy))));
    const E v2 = T::ld(t, T6_R, t.base + 1);
    // v2 v, v2 X, u2 Z
    team_exchange<T>(t, T6_S, T::f_mul(t.k < 2 ? v2 : T::ld(t, T6_R, t.base), t.k == 0 ? v : (t.k == 1 ? X : Z)));
    const E v3 = T::ld(t, T6_S, t.base), v2X = T::ld(t, T6_S, t.base + 1);
    const E A = T::f_sub(T::f_sub(T::ld(t, T6_S, t.base + 2), v3), team_dbl<T>(v2X));
    // v A, u (v2X - A), v3 Y, v3 Z
    const E w = T::f_sub(v2X, A);
    const E r = T::f_mul(t.k == 0 ? v : (t.k == 1 ? u : v3), t.k == 0 ? A : (t.k == 1 ? w : (t.k == 2 ? Y : Z)));
    team_exchange<T>(t, T6_Q, r);
    S = T::ld(t, T6_Q, t.base + (t.k < 2 ? t.k : 3));
    const E y = T::f_sub(S, T::ld(t, T6_Q, t.base + 2));
    if (t.k == 1) S = y;
    const int c = T::line_index(t);
    E l;
    if (c < 2) {
        l = T::f_sub(T::ld(t, T6_R, t.base + 2), T::ld(t, T6_R, t.base + 3));
    } else {
        l = c < 4 ? T::f_neg(u) : v;
    }
    return T::component(l, c & 1);
}

}  // namespace wbte
