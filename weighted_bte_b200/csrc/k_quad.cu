// Kernels over quads (quad.cuh) for calls bound by the length of a scalar
// multiple's chain: the Horner tail of an MSM, transform stages of few arrays,
// MSMs of a few terms, single multiples and Schnorr checks.  One warp per
// block; every lane runs to the end of its kernel.
#include <algorithm>

#include "launch.h"
#include "quad.cuh"

namespace wbte {

namespace {
constexpr int WARP = 32;
inline unsigned blocks_for(int64_t n, int64_t per) { return (unsigned)((n + per - 1) / per); }

template <class P> struct SizeOf {
    static constexpr size_t AFF = 2 * P::FIELD, XYZZ = 4 * P::FIELD;
    static constexpr int PER_WARP = WARP / Quad<P>::WIDTH;
};
// this lane's point among all the launch's
template <class P> __device__ __forceinline__ int64_t point_index() {
    return (int64_t)blockIdx.x * SizeOf<P>::PER_WARP + (threadIdx.x & 31) / Quad<P>::WIDTH;
}

// out[j] = sum_w 2^(c w) wins[j windows + w], the sums of each window
template <class P>
__global__ void __launch_bounds__(WARP) k_combine(uint8_t* out, const uint8_t* wins, int64_t k, int windows, int c) {
    using Q = Quad<P>;
    const int64_t j = point_index<P>();
    const bool active = j < k;
    const uint8_t* W = wins + SizeOf<P>::XYZZ * (active ? j : k - 1) * windows;
    Fp acc = Q::load(W + SizeOf<P>::XYZZ * (windows - 1));
    for (int w = windows - 2; w >= 0; w--) {
        for (int i = 0; i < c; i++) acc = Q::dbl(acc);
        acc = Q::add(acc, Q::load(W + SizeOf<P>::XYZZ * w), true);
    }
    acc = Q::affine(acc);
    if (active) Q::store_affine(out + SizeOf<P>::AFF * j, acc);
}

// One radix-2 butterfly per DIGITS points: point j takes digit j of the
// twiddle (Quad::image), the parts are summed, and the first two points write
// u + t and u - t.
template <class P>
__global__ void __launch_bounds__(WARP) k_ntt_stage(uint8_t* work, const uint8_t* tw, int64_t n, int64_t half,
                                                    int64_t count) {
    using Q = Quad<P>;
    constexpr int D = Q::DIGITS;
    const int64_t p = point_index<P>(), total = (n / 2) * count;
    const int dig = (int)(p % D);
    const bool active = p / D < total;
    const int64_t t = active ? p / D : total - 1;
    const int64_t q = t / (n / 2), tt = t % (n / 2), chunk = tt / half, j = tt % half;
    const int64_t a = q * n + chunk * 2 * half + j, b = a + half;
    Fp v = Q::load(work + SizeOf<P>::XYZZ * b);
    const Fp u = Q::load(work + SizeOf<P>::XYZZ * a);
    if (half > 1) {
        uint64_t d[4] = {1, 0, 0, 0};
        if (j) {
            uint32_t s[8];
            load_scalar(s, tw + FR_SZ * (j * (n / (2 * half))));
            decompose_base_x(d, s);
        }
        uint64_t lo[1], hi[1];
        quad_digit<P>(lo[0], hi[0], d, dig);
        const Fp base[1] = {Q::image(v, dig)};
        v = Q::group_sum(Q::straus(base, lo, hi, 1), D);
    }
    // the sum is valid in the butterfly's first point
    const int lane = threadIdx.x & 31;
    const Fp first = fp_shfl(v, (lane & ~(D * Q::WIDTH - 1)) + (lane & (Q::WIDTH - 1)));
    const Fp r = Q::add(u, dig == 1 ? Q::neg(first) : first, true);
    if (active && dig < 2) Q::store(work + SizeOf<P>::XYZZ * (dig == 0 ? a : b), r);
}

// out[o] = sum_t scalars[vsel[o] n + t] points[pbase[o] + idx[t]] for n <=
// SMALL_MSM_MAX: the (term, digit) pairs of an output are dealt to L points
// (a power of two that a warp holds), the sums meet in a tree
template <class P>
__global__ void __launch_bounds__(WARP) k_small_msm(uint8_t* out, const uint8_t* points, const int64_t* pbase,
                                                    const int32_t* idx, const uint8_t* scalars, const int32_t* vsel,
                                                    int64_t k, int64_t n, int L) {
    using Q = Quad<P>;
    constexpr int D = Q::DIGITS, MOST = SMALL_MSM_MAX * D;
    const int64_t p = point_index<P>();
    const int sub = (int)(p % L);
    const bool active = p / L < k;
    const int64_t o = active ? p / L : k - 1;
    const int64_t v = vsel ? (int64_t)vsel[o] : 0;
    const int pairs = (int)n * D, mine = (pairs + L - 1) / L;
    Fp base[MOST];
    uint64_t lo[MOST], hi[MOST];
    for (int r = 0; r < mine; r++) {
        const int x = sub + r * L, t = x < pairs ? x / D : 0, c = x % D;
        base[r] = Q::image(Q::load_affine(points + SizeOf<P>::AFF * (pbase[o] + (idx ? (int64_t)idx[t] : t))), c);
        uint32_t s[8];
        load_scalar(s, scalars + FR_SZ * (v * n + t));
        uint64_t d[4];
        decompose_base_x(d, s);
        quad_digit<P>(lo[r], hi[r], d, c);
        if (x >= pairs) lo[r] = hi[r] = 0;
    }
    const Fp r = Q::affine(Q::group_sum(Q::straus(base, lo, hi, mine), L));
    if (active && sub == 0) Q::store_affine(out + SizeOf<P>::AFF * o, r);
}

// out[i] = scalars[i] points[i stride] for any points of the curve (no
// endomorphism): 4-bit windows of the 256-bit scalar
template <class P>
__global__ void __launch_bounds__(WARP) k_mul_batch(uint8_t* out, const uint8_t* pts, int64_t stride,
                                                    const uint8_t* scalars, int64_t n) {
    using Q = Quad<P>;
    int64_t i = point_index<P>();
    const bool active = i < n;
    if (!active) i = n - 1;
    uint32_t s[8];
    load_scalar(s, scalars + FR_SZ * i);
    Fp tab[16];
    tab[0] = Q::infinity();
    tab[1] = Q::load_affine(pts + SizeOf<P>::AFF * stride * i);
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
    if (active) Q::store_affine(out + SizeOf<P>::AFF * i, r);
}

// valid[i] = ([s_i] G == R_i + [c_i] X_i), four points per check: two take the
// digits of [c]X, two the even and odd bytes of [s]G from the generator table
__global__ void __launch_bounds__(WARP) k_schnorr_verify(uint8_t* valid, const uint8_t* X, const uint8_t* R,
                                                         const uint8_t* sresp, const uint8_t* c, int64_t n,
                                                         const uint8_t* gen_table) {
    using Q = Quad<OnLane>;
    const int64_t p = point_index<OnLane>();
    const int sub = (int)(p & 3);
    const bool active = p / 4 < n;
    const int64_t i = active ? p / 4 : n - 1;
    uint32_t s[8];
    load_scalar(s, c + FR_SZ * i);
    uint64_t d[4], lo[1], hi[1];
    decompose_base_x(d, s);
    quad_digit<OnLane>(lo[0], hi[0], d, sub & 1);
    if (sub >= 2) lo[0] = hi[0] = 0;
    const Fp base[1] = {Q::image(Q::load_affine(X + G1_AFF * i), sub & 1)};
    Fp acc = Q::straus(base, lo, hi, 1);
    // R joins the first point's sum; -[s]G gathers on the third and fourth
    const uint8_t* sb = sresp + FR_SZ * i;
    for (int w = 0; w < 16; w++) {
        const uint32_t by = sub >= 2 ? sb[2 * w + (sub & 1)] : 0u;
        const uint8_t* src = sub >= 2 ? gen_table + G1_AFF * (256 * (2 * w + (sub & 1)) + by) : R + G1_AFF * i;
        Fp m = Q::load_affine(src);
        if (sub >= 2) m = Q::neg(m);
        acc = Q::add(acc, m, sub >= 2 ? by != 0 : (sub == 0 && w == 0));
    }
    acc = Q::group_sum(acc, 4);
    const bool inf = Q::is_inf(acc);
    if (active && sub == 0 && Q::place() == 0) valid[i] = inf ? 1 : 0;
}

}  // namespace

void launch_msm_combine(Group g, uint8_t* out, const uint8_t* wins, int64_t k, int windows, int c, cudaStream_t s) {
    note_launch();
    if (g == GROUP_G1)
        k_combine<OnLane><<<blocks_for(k, SizeOf<OnLane>::PER_WARP), WARP, 0, s>>>(out, wins, k, windows, c);
    else
        k_combine<OnPair><<<blocks_for(k, SizeOf<OnPair>::PER_WARP), WARP, 0, s>>>(out, wins, k, windows, c);
}

void launch_quad_ntt_stage(Group g, uint8_t* work, const uint8_t* tw, int64_t n, int64_t half, int64_t count,
                           cudaStream_t s) {
    const int64_t butterflies = (n / 2) * count;
    note_launch();
    if (g == GROUP_G1)
        k_ntt_stage<OnLane><<<blocks_for(2 * butterflies, SizeOf<OnLane>::PER_WARP), WARP, 0, s>>>(work, tw, n, half, count);
    else
        k_ntt_stage<OnPair><<<blocks_for(4 * butterflies, SizeOf<OnPair>::PER_WARP), WARP, 0, s>>>(work, tw, n, half, count);
}

void launch_quad_small_msm(Group g, uint8_t* out, const uint8_t* points, const int64_t* pbase, const int32_t* idx,
                           const uint8_t* scalars, const int32_t* vsel, int64_t k, int64_t n, int L, cudaStream_t s) {
    note_launch();
    if (g == GROUP_G1)
        k_small_msm<OnLane><<<blocks_for(L * k, SizeOf<OnLane>::PER_WARP), WARP, 0, s>>>(out, points, pbase, idx, scalars,
                                                                                      vsel, k, n, L);
    else
        k_small_msm<OnPair><<<blocks_for(L * k, SizeOf<OnPair>::PER_WARP), WARP, 0, s>>>(out, points, pbase, idx, scalars,
                                                                                      vsel, k, n, L);
}

void launch_quad_mul_batch(Group g, uint8_t* out, const uint8_t* pts, int64_t stride, const uint8_t* scalars, int64_t n,
                           cudaStream_t s) {
    note_launch();
    if (g == GROUP_G1)
        k_mul_batch<OnLane><<<blocks_for(n, SizeOf<OnLane>::PER_WARP), WARP, 0, s>>>(out, pts, stride, scalars, n);
    else
        k_mul_batch<OnPair><<<blocks_for(n, SizeOf<OnPair>::PER_WARP), WARP, 0, s>>>(out, pts, stride, scalars, n);
}

void launch_quad_schnorr_verify(uint8_t* valid, const uint8_t* X, const uint8_t* R, const uint8_t* sresp, const uint8_t* c,
                                int64_t n, const uint8_t* gen_table, cudaStream_t s) {
    note_launch();
    k_schnorr_verify<<<blocks_for(4 * n, SizeOf<OnLane>::PER_WARP), WARP, 0, s>>>(valid, X, R, sresp, c, n, gen_table);
}

}  // namespace wbte
