// Fp12 arithmetic with one element spread over a team of six lanes: lane k
// holds the Fp2 coefficient of w^k (w^6 = xi = 1 + u), five teams per warp.
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
#include "pairing.cuh"

namespace wbte {

constexpr int TEAM_LANES = 6;
constexpr int TEAMS = 5;  // per warp
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

struct Wide { uint32_t v[24]; };
struct Wide2 { Wide c0, c1; };

struct Team {
    uint4* sh;  // this warp's rows
    int k;      // this lane's power of w
    int base;   // slot of the team's lane 0
};

WBTE_INL int nib(uint32_t packed, int k) { return (int)((packed >> (4 * k)) & 15u); }

// `per` teams per warp (4 or 5); lanes past them shadow the last team's
WBTE_INL Team team_init(uint4* sh, int per = TEAMS) {
    const int lane = threadIdx.x & 31;
    const int used = TEAM_LANES * per;
    const int l = lane < used ? lane : used - TEAM_LANES + (lane - used) % TEAM_LANES;
    Team t;
    t.sh = sh;
    t.k = l % TEAM_LANES;
    t.base = l - t.k;
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

WBTE_INL Fp2 t6_one(const Team& t) {
    Fp2 r = fp2_zero();
    if (t.k == 0) r.c0 = fp_one();
    return r;
}
WBTE_INL Fp2 t6_conj(const Team& t, const Fp2& a) {
    const Fp2 n = fp2_neg(a);
    return (t.k & 1) ? n : a;
}
// x^(p^pw), pw in 1..3
static __device__ __noinline__ Fp2 t6_frobenius(Team t, Fp2 a, int pw) {
    if (pw & 1) a.c1 = fp_neg(a.c1);
    const Fp2 c = fp2_from_const(C_FROB[pw - 1][t.k]);
    return t6_fp2_mul(a, c);
}

// lane k's coefficient in blst's Fp12 layout (c0.c0, c0.c1, c0.c2, c1.c0, ..)
WBTE_INL size_t t6_offset(const Team& t) { return 96 * (size_t)((t.k & 1) * 3 + (t.k >> 1)); }
WBTE_INL Fp2 t6_load(const Team& t, const uint8_t* gt) {
    return load_vec(reinterpret_cast<const Fp2*>(gt + t6_offset(t)));
}
WBTE_INL void t6_store(const Team& t, uint8_t* gt, const Fp2& a) {
    store_vec(reinterpret_cast<Fp2*>(gt + t6_offset(t)), a);
}

// ------------------------------------------------------ final exponentiation
// 1/d for the Fp2 value that lane 0 of the team holds, on every lane
WBTE_INL Fp2 t6_inverse_of_lane0(const Team& t, const Fp2& a) {
    __syncwarp();
    team_st(t, T6_A, t.base + t.k, a);
    __syncwarp();
    return fp2_inv(team_ld<Fp2>(t, T6_A, t.base));
}
// f^((p^6 - 1)(p^2 + 1)) = (conj(f)^2 / (f conj(f)))^(p^2 + 1).  N = f conj(f)
// lies in Fp6, and 1/N = N^(p^2) N^(p^4) / (N N^(p^2) N^(p^4)), whose
// denominator lies in Fp2 (lane 0).  f = 0 gives 0.
static __device__ __noinline__ Fp2 t6_final_exp_easy(Team t, Fp2 f) {
    const Fp2 g = t6_conj(t, f);
    const Fp2 n = t6_mul(t, f, g);
    const Fp2 n2 = t6_frobenius(t, n, 2);
    const Fp2 m = t6_mul(t, n2, t6_frobenius(t, n2, 2));
    const Fp2 d = t6_inverse_of_lane0(t, t6_mul(t, n, m));
    Fp2 r = t6_mul(t, t6_mul(t, g, g), t6_fp2_mul(m, d));
    return t6_mul(t, r, t6_frobenius(t, r, 2));
}
// x^(|z|/2) conjugated: squaring runs between the set bits of |z|
static __device__ __noinline__ Fp2 t6_raise_to_z_div_by_2(Team t, Fp2 x) {
    Fp2 acc = t6_cyc_sqr(t, x);
    const uint64_t runs = 2ull | (3ull << 8) | (9ull << 16) | (32ull << 24) | (15ull << 32);
    for (int r = 0; r < 5; r++) {
        acc = t6_mul(t, acc, x);
        for (int i = (int)((runs >> (8 * r)) & 255u); i > 0; i--) acc = t6_cyc_sqr(t, acc);
    }
    return t6_conj(t, acc);
}
WBTE_INL Fp2 t6_raise_to_z(const Team& t, const Fp2& x) { return t6_cyc_sqr(t, t6_raise_to_z_div_by_2(t, x)); }
// the chain of final_exp_hard
static __device__ __noinline__ Fp2 t6_final_exp_hard(Team t, Fp2 in) {
    const Fp2 y0 = t6_cyc_sqr(t, in);
    Fp2 y1 = t6_raise_to_z(t, y0);
    Fp2 y2 = t6_raise_to_z_div_by_2(t, y1);
    y1 = t6_conj(t, t6_mul(t, y1, t6_conj(t, in)));
    y1 = t6_mul(t, y1, y2);
    y2 = t6_raise_to_z(t, y1);
    Fp2 y3 = t6_raise_to_z(t, y2);
    y1 = t6_conj(t, y1);
    y3 = t6_mul(t, y3, y1);
    y1 = t6_frobenius(t, t6_conj(t, y1), 3);
    y1 = t6_mul(t, y1, t6_frobenius(t, y2, 2));
    y2 = t6_mul(t, t6_raise_to_z(t, y3), y0);
    y1 = t6_mul(t, y1, t6_mul(t, y2, in));
    return t6_mul(t, y1, t6_frobenius(t, y3, 1));
}

// -------------------------------------------------------------- Miller loops
// Lines (pairing.cuh) enter as their six Fp components, component k on lane
// k, already scaled by (1, 1, xP, xP, yP, yP).
WBTE_INL bool t6_bit(int i) { return (X_ABS >> i) & 1; }

// this lane's scale for lines through P; identities get the line 1
struct T6Point { Fp scale; bool inf; };
WBTE_INL T6Point t6_point(const Team& t, const G1A& P) {
    T6Point r;
    r.inf = is_inf(P);
    r.scale = t.k < 2 ? fp_one() : (t.k < 4 ? P.x : P.y);
    return r;
}
WBTE_INL Fp t6_line_value(const Team& t, const Fp& component, const T6Point& P) {
    const Fp v = fp_mul(component, P.scale);
    const Fp id = t.k == 0 ? fp_one() : fp_zero();
    return P.inf ? id : v;
}

// G2 point of a running loop in homogeneous coordinates: X, Y, Z on lanes 0, 1,
// 2 (the others carry anything).  The products of a step go one to a lane;
// every lane forms the sums it needs from shared memory.
constexpr int T6_P = T6_Y, T6_Q = T6_Y + 6, T6_R = T6_Z, T6_S = T6_Z + 6;
WBTE_INL Fp2 t6_exchange(const Team& t, int row, const Fp2& v) {
    team_st(t, row, t.base + t.k, v);
    __syncwarp();
    return v;
}
// T <- 2T; returns this lane's component of the tangent line (line_double)
static __device__ __noinline__ Fp t6_line_double(Team t, Fp2& T) {
    __syncwarp();
    t6_exchange(t, T6_P, T);
    // Y Y, Z Z, X X, Y Z, X Y
    t6_exchange(t, T6_Q, t6_fp2_mul(team_ld<Fp2>(t, T6_P, t.base + nib(0x001021u, t.k)),
                                    team_ld<Fp2>(t, T6_P, t.base + nib(0x112021u, t.k))));
    const Fp2 t0 = team_ld<Fp2>(t, T6_Q, t.base);
    const Fp2 t2 = fp2_mul4(fp2_mul3(fp2_mul_xi(team_ld<Fp2>(t, T6_Q, t.base + 1))));  // 3 b' Z^2
    const Fp2 t23 = fp2_mul3(t2);
    const Fp2 YZ = team_ld<Fp2>(t, T6_Q, t.base + 3);
    // XY (t0 - t23), (t0 + t23)^2, t2^2, t0 YZ
    Fp2 a = t0, b = YZ;
    if (t.k == 0) {
        a = team_ld<Fp2>(t, T6_Q, t.base + 4);
        b = fp2_sub(t0, t23);
    } else if (t.k == 1) {
        a = b = fp2_add(t0, t23);
    } else if (t.k == 2) {
        a = b = t2;
    }
    t6_exchange(t, T6_R, t6_fp2_mul(a, b));
    if (t.k == 0) {
        T = fp2_dbl(team_ld<Fp2>(t, T6_R, t.base));
    } else if (t.k == 1) {
        T = fp2_sub(team_ld<Fp2>(t, T6_R, t.base + 1), fp2_mul4(fp2_mul3(team_ld<Fp2>(t, T6_R, t.base + 2))));
    } else {
        T = fp2_mul4(fp2_dbl(team_ld<Fp2>(t, T6_R, t.base + 3)));
    }
    Fp2 l;
    if (t.k < 2) {
        l = fp2_sub(t2, t0);
    } else if (t.k < 4) {
        l = fp2_mul3(team_ld<Fp2>(t, T6_Q, t.base + 2));
    } else {
        l = fp2_neg(fp2_dbl(YZ));
    }
    return (t.k & 1) ? l.c1 : l.c0;
}
// T <- T + Q; returns this lane's component of the chord (line_add)
static __device__ __noinline__ Fp t6_line_add(Team t, Fp2& T, const G2A& Q) {
    __syncwarp();
    t6_exchange(t, T6_P, T);
    const Fp2 X = team_ld<Fp2>(t, T6_P, t.base), Y = team_ld<Fp2>(t, T6_P, t.base + 1);
    const Fp2 Z = team_ld<Fp2>(t, T6_P, t.base + 2);
    const Fp2 qx = Q.x, qy = Q.y;
    t6_exchange(t, T6_Q, t6_fp2_mul(t.k == 0 ? qy : qx, Z));
    const Fp2 u = fp2_sub(team_ld<Fp2>(t, T6_Q, t.base), Y);
    const Fp2 v = fp2_sub(team_ld<Fp2>(t, T6_Q, t.base + 1), X);
    // u u, v v, u xQ, v yQ
    t6_exchange(t, T6_R, t6_fp2_mul((t.k == 0 || t.k == 2) ? u : v,
                                    t.k == 0 ? u : (t.k == 1 ? v : (t.k == 2 ? qx : qy))));
    const Fp2 v2 = team_ld<Fp2>(t, T6_R, t.base + 1);
    // v2 v, v2 X, u2 Z
    t6_exchange(t, T6_S, t6_fp2_mul(t.k < 2 ? v2 : team_ld<Fp2>(t, T6_R, t.base), t.k == 0 ? v : (t.k == 1 ? X : Z)));
    const Fp2 v3 = team_ld<Fp2>(t, T6_S, t.base), v2X = team_ld<Fp2>(t, T6_S, t.base + 1);
    const Fp2 A = fp2_sub(fp2_sub(team_ld<Fp2>(t, T6_S, t.base + 2), v3), fp2_dbl(v2X));
    // v A, u (v2X - A), v3 Y, v3 Z
    const Fp2 r = t6_fp2_mul(t.k == 0 ? v : (t.k == 1 ? u : v3), t.k == 0 ? A : (t.k == 1 ? fp2_sub(v2X, A) : (t.k == 2 ? Y : Z)));
    t6_exchange(t, T6_Q, r);
    T = team_ld<Fp2>(t, T6_Q, t.base + (t.k < 2 ? t.k : 3));
    if (t.k == 1) T = fp2_sub(T, team_ld<Fp2>(t, T6_Q, t.base + 2));
    Fp2 l;
    if (t.k < 2) {
        l = fp2_sub(team_ld<Fp2>(t, T6_R, t.base + 2), team_ld<Fp2>(t, T6_R, t.base + 3));
    } else {
        l = t.k < 4 ? fp2_neg(u) : v;
    }
    return (t.k & 1) ? l.c1 : l.c0;
}

}  // namespace wbte
