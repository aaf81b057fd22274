// Out-of-line tower arithmetic.  Included once by fields.cuh; every function
// has internal linkage, so each translation unit carries its own copy.
#pragma once

namespace wbte {

// a^(p-2) with a 4-bit fixed window over the constant exponent.
WBTE_NOINL Fp fp_inv(Fp a) {
    Fp tab[16];
    tab[0] = fp_one();
    tab[1] = a;
    for (int i = 2; i < 16; i++) tab[i] = fp_mul(tab[i - 1], a);
    Fp r = fp_one();
    bool started = false;
    for (int w = 95; w >= 0; w--) {
        if (started) {
            r = fp_sqr(r);
            r = fp_sqr(r);
            r = fp_sqr(r);
            r = fp_sqr(r);
        }
        uint32_t d = (C_P_MINUS_2[w / 8] >> (4 * (w % 8))) & 15u;
        if (d) {
            r = started ? fp_mul(r, tab[d]) : tab[d];
            started = true;
        }
    }
    return r;
}

WBTE_NOINL Fr fr_inv(Fr a) {
    Fr tab[16];
    tab[0] = fr_one();
    tab[1] = a;
    for (int i = 2; i < 16; i++) tab[i] = fr_mul(tab[i - 1], a);
    Fr r = fr_one();
    bool started = false;
    for (int w = 63; w >= 0; w--) {
        if (started) {
            r = fr_mul(r, r);
            r = fr_mul(r, r);
            r = fr_mul(r, r);
            r = fr_mul(r, r);
        }
        uint32_t d = (C_R_MINUS_2[w / 8] >> (4 * (w % 8))) & 15u;
        if (d) {
            r = started ? fr_mul(r, tab[d]) : tab[d];
            started = true;
        }
    }
    return r;
}

WBTE_NOINL Fp2 fp2_inv(Fp2 a) {
    Fp n = fp_add(fp_sqr(a.c0), fp_sqr(a.c1));
    n = fp_inv(n);
    return Fp2{fp_mul(a.c0, n), fp_neg(fp_mul(a.c1, n))};
}

// Karatsuba over Fp2: 6 Fp2 products.
WBTE_NOINL void fp6_mul(Fp6& r, const Fp6& a, const Fp6& b) {
    Fp2 t0 = fp2_mul(a.c0, b.c0);
    Fp2 t1 = fp2_mul(a.c1, b.c1);
    Fp2 t2 = fp2_mul(a.c2, b.c2);
    Fp2 s12 = fp2_mul(fp2_add(a.c1, a.c2), fp2_add(b.c1, b.c2));
    Fp2 s01 = fp2_mul(fp2_add(a.c0, a.c1), fp2_add(b.c0, b.c1));
    Fp2 s02 = fp2_mul(fp2_add(a.c0, a.c2), fp2_add(b.c0, b.c2));
    Fp2 c0 = fp2_add(t0, fp2_mul_xi(fp2_sub(fp2_sub(s12, t1), t2)));
    Fp2 c1 = fp2_add(fp2_sub(fp2_sub(s01, t0), t1), fp2_mul_xi(t2));
    Fp2 c2 = fp2_add(fp2_sub(fp2_sub(s02, t0), t2), t1);
    r.c0 = c0;
    r.c1 = c1;
    r.c2 = c2;
}

WBTE_NOINL void fp6_inv(Fp6& r, const Fp6& a) {
    Fp2 A = fp2_sub(fp2_sqr(a.c0), fp2_mul_xi(fp2_mul(a.c1, a.c2)));
    Fp2 B = fp2_sub(fp2_mul_xi(fp2_sqr(a.c2)), fp2_mul(a.c0, a.c1));
    Fp2 C = fp2_sub(fp2_sqr(a.c1), fp2_mul(a.c0, a.c2));
    Fp2 F = fp2_add(fp2_mul_xi(fp2_add(fp2_mul(a.c2, B), fp2_mul(a.c1, C))), fp2_mul(a.c0, A));
    F = fp2_inv(F);
    r.c0 = fp2_mul(A, F);
    r.c1 = fp2_mul(B, F);
    r.c2 = fp2_mul(C, F);
}

}  // namespace wbte
