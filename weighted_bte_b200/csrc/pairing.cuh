// What the pairing and the decomposed exponentiations rest on: the lines of the
// optimal-ate Miller loop over the M-type twist E'(Fp2): y^2 = x^3 + 4(1+u), which
// team.cuh computes, and the recodings of scalars in base |x|.
//
// Lines.  For T on E' and P = (xP, yP) in G1 the line through the untwisted
// points, scaled by w^3 and by an Fp2 factor (both killed by the easy part
// of the final exponentiation), is  c0 + (c1 xP) v + (c2 yP) v w  with
//   doubling (T = (X:Y:Z) homogeneous):  c0 = 3b'Z^2 - Y^2, c1 = 3X^2, c2 = -2YZ
//   addition (T + Q, Q affine):          c0 = u xQ - v yQ,  c1 = -u,   c2 = v
// where u = yQ Z - Y, v = xQ Z - X.  Only final-exponentiated values are
// canonical, so this scaling is free to differ from any other implementation.
#pragma once
#include "curves.cuh"

namespace wbte {

// pairs of one run of a Miller loop that computes its lines
constexpr int MULTI_MILLER_MAX = 8;

// ------------------------------------------ decomposed GT exponentiation
// A canonical scalar s < r is written s = d0 + d1|x| + d2|x|^2 + d3|x|^3
// with 0 <= di < |x|; on GT, Frobenius^i followed by conjugation for odd i
// acts as exponentiation by |x|^i.  Each digit is recoded in width-4 NAF
// and the four recodings share one run of at most 65 cyclotomic squarings.
// On cyclotomic elements outside GT the result agrees with x^s after the
// hard part of the final exponentiation.
struct CycPlan {
    int8_t naf[4][65];
};

// |x| = 2^16 * X_ODD with X_ODD < 2^48
constexpr uint64_t X_ODD = X_ABS >> 16;

WBTE_INL void make_cyc_plan(CycPlan& pl, const uint32_t s_in[8]) {
    uint32_t s[8];
    _Pragma("unroll") for (int i = 0; i < 8; i++) s[i] = s_in[i];
    for (int c = 0; c < 4; c++) {
        // s = q |x| + rem:  q = (s >> 16) div X_ODD, rem = ((s >> 16) mod X_ODD) 2^16 + (s & 0xffff)
        uint32_t lo16 = s[0] & 0xffffu;
        uint16_t chunks[15];
        for (int j = 0; j < 15; j++) {
            int bit = 16 + 16 * j;
            chunks[j] = (uint16_t)(s[bit >> 5] >> (bit & 31));
        }
        uint64_t rem = 0;
        uint16_t q[15];
        for (int j = 14; j >= 0; j--) {
            uint64_t cur = (rem << 16) | chunks[j];
            q[j] = (uint16_t)(cur / X_ODD);
            rem = cur % X_ODD;
        }
        uint64_t comp = (rem << 16) | lo16;
        for (int i = 0; i < 8; i++) s[i] = 0;
        for (int j = 0; j < 15; j++) s[j >> 1] |= (uint32_t)q[j] << (16 * (j & 1));
        // width-4 NAF of comp; a negative digit may carry into bit 64
        uint64_t v = comp;
        uint32_t carry_bit = 0;  // bit 64 of the running value
        int pos = 0;
        for (int i = 0; i < 65; i++) pl.naf[c][i] = 0;
        while (v != 0 || carry_bit) {
            if (v & 1) {
                int d = (int)(v & 15);
                if (d >= 8) d -= 16;
                pl.naf[c][pos] = (int8_t)d;
                if (d > 0) {
                    v -= (uint64_t)d;
                } else {
                    uint64_t nv = v + (uint64_t)(-d);
                    if (nv < v) carry_bit = 1;
                    v = nv;
                }
            }
            v = (v >> 1) | ((uint64_t)carry_bit << 63);
            carry_bit = 0;
            pos++;
        }
    }
}

// ------------------------------------------------ fixed-schedule recodings
// s = d0 + d1|x| + d2|x|^2 + d3|x|^3 with 0 <= dc < |x| (s < r < |x|^4)
WBTE_INL void decompose_base_x(uint64_t d[4], const uint32_t s_in[8]) {
    uint32_t s[8];
    _Pragma("unroll") for (int i = 0; i < 8; i++) s[i] = s_in[i];
    for (int c = 0; c < 4; c++) {
        uint32_t lo16 = s[0] & 0xffffu;
        uint16_t chunks[15];
        for (int j = 0; j < 15; j++) {
            int bit = 16 + 16 * j;
            chunks[j] = (uint16_t)(s[bit >> 5] >> (bit & 31));
        }
        uint64_t rem = 0;
        uint16_t q[15];
        for (int j = 14; j >= 0; j--) {
            uint64_t cur = (rem << 16) | chunks[j];
            q[j] = (uint16_t)(cur / X_ODD);
            rem = cur % X_ODD;
        }
        d[c] = (rem << 16) | lo16;
        for (int i = 0; i < 8; i++) s[i] = 0;
        for (int j = 0; j < 15; j++) s[j >> 1] |= (uint32_t)q[j] << (16 * (j & 1));
    }
}

// Signed radix-16 recoding of v = hi 2^64 + lo with `top` nibbles (16 or 32):
// v = sum_{k=0..top} digit_k 16^k with digits in [-7, 8].  Rounding a nibble
// above 8 down by 16 carries one into the next digit, and the carry into
// digit k is set exactly when the low k nibbles of v exceed 0x88...8 (k
// eights), so each digit is computed on its own, without a digit array.
WBTE_INL int r16_carry(uint64_t lo, uint64_t hi, int k) {
    constexpr uint64_t E = 0x8888888888888888ull;
    if (k <= 16) {
        uint64_t m = k == 16 ? ~0ull : ((1ull << (4 * k)) - 1);
        return (lo & m) > (E & m);
    }
    int kh = k - 16;
    uint64_t m = kh == 16 ? ~0ull : ((1ull << (4 * kh)) - 1);
    uint64_t h = hi & m, e = E & m;
    return h > e || (h == e && lo > E);
}
WBTE_INL int r16_digit(uint64_t lo, uint64_t hi, int k, int top) {
    int nib = 0;
    if (k < top) nib = (int)(((k < 16) ? (lo >> (4 * k)) : (hi >> (4 * (k - 16)))) & 15u);
    int cout = k < top ? r16_carry(lo, hi, k + 1) : 0;
    return nib + r16_carry(lo, hi, k) - 16 * cout;
}

// psi (untwist-Frobenius-twist) on G2 in XYZZ coordinates; acts as [x]
WBTE_INL G2X g2_psi(const G2X& p) {
    G2X r;
    r.X = fp2_mul(fp2_conj(p.X), fp2_from_const(C_PSI_CX));
    r.Y = fp2_mul(fp2_conj(p.Y), fp2_from_const(C_PSI_CY));
    r.ZZ = fp2_conj(p.ZZ);
    r.ZZZ = fp2_conj(p.ZZZ);
    return r;
}
// phi (x, y) -> (beta x, y) on G1 in XYZZ coordinates; acts as [x^2 - 1]
WBTE_INL G1X g1_phi(const G1X& p) {
    G1X r = p;
    r.X = fp_mul(p.X, fp_from_const(C_GLV_BETA));
    return r;
}

}  // namespace wbte
