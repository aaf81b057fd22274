// Out-of-line tower arithmetic.  Included once by fields.cuh; every function
// has internal linkage, so each translation unit carries its own copy.
#pragma once

namespace wbte {

// Modular inversion by division steps (Bernstein and Yang, "Fast constant-time
// gcd computation and modular inversion", 2019), in the variant that starts
// from delta = 1/2, with its bound on the number of steps (Wuille and Maxwell,
// "Bounds on divsteps iterations in safegcd", 2021).  A chain of about 480 dependent Fp products (a^(p-2))
// bounds every kernel with one inversion per value from below: about 490 us on
// one warp.  The division steps work on the low word of f and g, 30 at a
// time, in about 23 one-word instructions each; their 2 x 2 matrix is then
// applied to f, g and to the cofactors d, e modulo the modulus, as signed
// 30-bit limbs.  The loop is fixed, so lanes do not diverge: 879 steps suffice for
// 381 bits and 589 for 255 ((45907 n + 26313) / 19929), 30 and 20 batches.
// The multiple of the modulus that makes d, e divisible by 2^30 is centred, so
// |d| grows by half the modulus per batch at most and stays below 16 of it.
// Zero gives zero.  Measured on B200: the easy parts of 65,536 values 14.2 -> 3.0
// ms and of one value 0.58 -> 0.12 ms, GT encodings of 512 values 0.60 -> 0.14 ms.
template <int N> struct Limbs30 { int32_t v[N]; };

template <int N>
WBTE_INL void divsteps_apply(Limbs30<N>& a, Limbs30<N>& b, const int32_t t[4], const int32_t* m, uint32_t neg_inv) {
    // (a, b) <- ((t0 a + t1 b) + k m, (t2 a + t3 b) + l m) / 2^30; m null: exact already
    constexpr int32_t MASK = (1 << 30) - 1;
    int64_t ca = (int64_t)t[0] * a.v[0] + (int64_t)t[1] * b.v[0];
    int64_t cb = (int64_t)t[2] * a.v[0] + (int64_t)t[3] * b.v[0];
    int32_t k = 0, l = 0;
    if (m) {
        k = (int32_t)(((uint32_t)ca * neg_inv) << 2) >> 2;
        l = (int32_t)(((uint32_t)cb * neg_inv) << 2) >> 2;
        ca += (int64_t)k * m[0];
        cb += (int64_t)l * m[0];
    }
    ca >>= 30;
    cb >>= 30;
    _Pragma("unroll") for (int i = 1; i < N; i++) {
        ca += (int64_t)t[0] * a.v[i] + (int64_t)t[1] * b.v[i];
        cb += (int64_t)t[2] * a.v[i] + (int64_t)t[3] * b.v[i];
        if (m) {
            ca += (int64_t)k * m[i];
            cb += (int64_t)l * m[i];
        }
        a.v[i - 1] = (int32_t)ca & MASK;
        b.v[i - 1] = (int32_t)cb & MASK;
        ca >>= 30;
        cb >>= 30;
    }
    a.v[N - 1] = (int32_t)ca;
    b.v[N - 1] = (int32_t)cb;
}

// x <- 1/x mod m, x < m in 30-bit limbs; mk[j] = 2^j m
template <int N> WBTE_INL void divsteps_inverse(Limbs30<N>& x, const int32_t (&mk)[5][N], uint32_t neg_inv, int batches) {
    constexpr int32_t MASK = (1 << 30) - 1;
    Limbs30<N> f, g = x, d, e;
    _Pragma("unroll") for (int i = 0; i < N; i++) {
        f.v[i] = mk[0][i];
        d.v[i] = 0;
        e.v[i] = i == 0;
    }
    int32_t delta = 1;  // delta + 1/2
    for (int n = 0; n < batches; n++) {
        uint32_t fl = (uint32_t)f.v[0] | ((uint32_t)f.v[1] << 30), gl = (uint32_t)g.v[0] | ((uint32_t)g.v[1] << 30);
        int32_t t[4] = {1, 0, 0, 1};
        _Pragma("unroll 6") for (int i = 0; i < 30; i++) {
            const bool odd = gl & 1, swap = odd && delta > 0;
            const uint32_t af = odd ? (swap ? 0u - fl : fl) : 0u;
            const int32_t au = odd ? (swap ? -t[0] : t[0]) : 0, av = odd ? (swap ? -t[1] : t[1]) : 0;
            const int32_t nu = swap ? t[2] : t[0], nv = swap ? t[3] : t[1];
            fl = swap ? gl : fl;
            gl = (gl + af) >> 1;
            t[2] += au;
            t[3] += av;
            t[0] = 2 * nu;
            t[1] = 2 * nv;
            delta = swap ? 2 - delta : delta + 1;
        }
        divsteps_apply<N>(f, g, t, nullptr, 0);
        divsteps_apply<N>(d, e, t, mk[0], neg_inv);
    }
    // f = +-1 (or the modulus, for x = 0): x = f d, brought from (-16 m, 16 m) to [0, m)
    const bool negative = f.v[N - 1] < 0;
    int32_t c = 0;
    _Pragma("unroll") for (int i = 0; i < N; i++) {
        c += (negative ? -d.v[i] : d.v[i]) + mk[4][i];
        x.v[i] = i < N - 1 ? (c & MASK) : c;
        c >>= 30;
    }
    for (int j = 4; j >= 0; j--) {
        Limbs30<N> y;
        c = 0;
        _Pragma("unroll") for (int i = 0; i < N; i++) {
            c += x.v[i] - mk[j][i];
            y.v[i] = i < N - 1 ? (c & MASK) : c;
            c >>= 30;
        }
        const bool less = y.v[N - 1] < 0;
        _Pragma("unroll") for (int i = 0; i < N; i++) x.v[i] = less ? x.v[i] : y.v[i];
    }
}

// 32-bit words to 30-bit limbs and back
template <int N, int W> WBTE_INL Limbs30<N> to_limbs30(const uint32_t (&a)[W]) {
    Limbs30<N> r;
    _Pragma("unroll") for (int i = 0; i < N; i++) {
        const int bit = 30 * i, w = bit >> 5, o = bit & 31;
        uint32_t x = w < W ? a[w] >> o : 0u;
        if (o > 2 && w + 1 < W) x |= a[w + 1] << (32 - o);
        r.v[i] = (int32_t)(x & 0x3fffffffu);
    }
    return r;
}
template <int N, int W> WBTE_INL void from_limbs30(uint32_t (&a)[W], const Limbs30<N>& r) {
    _Pragma("unroll") for (int w = 0; w < W; w++) {
        const int bit = 32 * w, i = bit / 30, o = bit % 30;
        uint32_t x = (uint32_t)r.v[i] >> o;
        if (i + 1 < N) x |= (uint32_t)r.v[i + 1] << (30 - o);
        if (30 - o + 30 < 32 && i + 2 < N) x |= (uint32_t)r.v[i + 2] << (60 - o);
        a[w] = x;
    }
}

// Montgomery form in and out: the inverse of a R is taken as an integer and
// multiplied by R^3 / R
WBTE_NOINL Fp fp_inv(Fp a) {
    Limbs30<13> x = to_limbs30<13>(a.v);
    divsteps_inverse<13>(x, C_P30, P30_NEG_INV, 30);
    from_limbs30<13>(a.v, x);
    return fp_mul(a, fp_from_const(C_FP_R3));
}

WBTE_NOINL Fr fr_inv(Fr a) {
    Limbs30<9> x = to_limbs30<9>(a.v);
    divsteps_inverse<9>(x, C_R30, R30_NEG_INV, 20);
    from_limbs30<9>(a.v, x);
    Fr r3;
    _Pragma("unroll") for (int i = 0; i < 8; i++) r3.v[i] = C_FR_R3[i];
    return fr_mul(a, r3);
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
