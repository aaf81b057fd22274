// GT transforms and GT exponentiation over teams of lanes (team.cuh): the
// radix-4 stages of the (truncated) cyclotomic transforms and batched GT
// powers.
//
// An exponentiation v^s splits s into its four base-|x| digits, each acting
// through conj o Frobenius, over one run of cyclotomic squarings.  What bounds
// it depends on how many there are.  A transform of 64 arrays is bound by the
// wide multiply-add pipe; there five neighbouring teams take the same twiddle
// of five blocks or arrays, so its recoding is uniform in the warp and a
// width-4 NAF skips zero digits without divergence.  A transform of one array
// leaves schedulers idle and is bound by the length of the chain, so the
// digits are spread over teams that meet in a product.
#include <algorithm>
#include <cstdlib>

#include "launch.h"
#include "team.cuh"

namespace wbte {

namespace {
constexpr int WARP = 32;
inline unsigned blocks_for(int64_t n, int64_t per) { return (unsigned)((n + per - 1) / per); }

__device__ __forceinline__ int64_t bitrev64(int64_t i, int bits) {
    return bits ? (int64_t)(__brevll((unsigned long long)i) >> (64 - bits)) : 0;
}

// one 16-byte piece of an element per thread
__global__ void k_gt_bitrev(uint8_t* dst, const uint8_t* src, int64_t n, int bits, int64_t count) {
    const int64_t x = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    constexpr int64_t PIECES = GT_SZ / 16;
    const int64_t i = x / PIECES, p = x % PIECES;
    if (i >= n * count) return;
    const int64_t q = i / n, j = i % n;
    reinterpret_cast<uint4*>(dst)[(q * n + bitrev64(j, bits)) * PIECES + p] = reinterpret_cast<const uint4*>(src)[x];
}

// ------------------------------------------------------------- recodings
// The base-|x| digits of one scalar, recoded: REC_DIGITS signed digits for each
// of the four, width-4 NAF (digit i at bit i) or radix 16 in [-7, 8] (digit i
// at bit 4i).
constexpr int REC_DIGITS = 68;
constexpr int NAF_DIGITS = 65, R16_DIGITS = 17;
constexpr size_t REC_SZ = 4 * REC_DIGITS;

__global__ void k_gt_recode(int8_t* rec, const uint8_t* scalars, int64_t n, int naf) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint32_t s[8];
    load_scalar(s, scalars + FR_SZ * i);
    int8_t* out = rec + REC_SZ * i;
    if (naf) {
        CycPlan pl;
        make_cyc_plan(pl, s);
        for (int c = 0; c < 4; c++)
            for (int p = 0; p < NAF_DIGITS; p++) out[c * REC_DIGITS + p] = pl.naf[c][p];
    } else {
        uint64_t d[4];
        decompose_base_x(d, s);
        for (int c = 0; c < 4; c++)
            for (int k = 0; k < R16_DIGITS; k++) out[c * REC_DIGITS + k] = (int8_t)r16_digit(d[c], 0, k, 16);
    }
}

// out = v^s for the recoded s: the digits c0, c0 + L, .. of each team.  R16
// tables hold the powers 1..8 of phi^c0(v), phi = conj o Frobenius (which acts
// as |x|), NAF tables 1, 3, 5, 7; the other digits' tables are their images.
// Digits may differ between the teams of a warp: a product is skipped only
// where every team's digit is zero, and is by one where a team's is.
template <class T, int L, bool NAF>
__device__ __forceinline__ ElemOf<T> team_pow(const Team& t, ElemOf<T> x, const int8_t* rec, int c0) {
    constexpr int R = 4 / L, ND = NAF ? 4 : 8, TOP = NAF ? NAF_DIGITS : R16_DIGITS, RUN = NAF ? 1 : 4;
    if (L > 1) {
        const ElemOf<T> y = team_frobenius<T>(t, x, c0 ? c0 : 1);
        const ElemOf<T> z = (c0 & 1) ? team_conj<T>(t, y) : y;
        x = c0 ? z : x;
    }
    ElemOf<T> tab[R][ND];
    const ElemOf<T> two = T::cyc_sqr(t, x);
    tab[0][0] = x;
    if (NAF) {
        for (int i = 1; i < ND; i++) tab[0][i] = T::mul(t, tab[0][i - 1], two);
    } else {
        tab[0][1] = two;
        for (int i = 2; i < ND; i++) tab[0][i] = T::mul(t, tab[0][i - 1], x);
    }
    for (int r = 1; r < R; r++)
        for (int i = 0; i < ND; i++) {
            const ElemOf<T> y = team_frobenius<T>(t, tab[0][i], r * L);
            tab[r][i] = ((r * L) & 1) ? team_conj<T>(t, y) : y;
        }
    ElemOf<T> acc = team_one<T>(t);
    bool started = false;  // the same in all lanes
    for (int pos = TOP - 1; pos >= 0; pos--) {
        T::step();
        if (started)
            for (int i = 0; i < RUN; i++) acc = T::cyc_sqr(t, acc);
        for (int r = 0; r < R; r++) {
            const int d = rec[(c0 + r * L) * REC_DIGITS + pos];
            if (!__any_sync(0xffffffffu, d != 0)) continue;
            const int ad = d < 0 ? -d : d;
            ElemOf<T> m = team_one<T>(t);
            if (d) m = tab[r][NAF ? (ad >> 1) : (ad - 1)];
            if (d < 0) m = team_conj<T>(t, m);
            acc = started ? T::mul(t, acc, m) : m;
            started = true;
        }
    }
    return acc;
}

// the product over a group of L neighbouring teams, valid in the first
template <class T, int L> __device__ __forceinline__ ElemOf<T> team_group_product(const Team& t, ElemOf<T> x, int sub) {
    for (int w = 1; w < L; w *= 2) {
        __syncwarp();
        T::st(t, T6_A, t.base + t.k, x);
        __syncwarp();
        const ElemOf<T> y = T::ld(t, T6_A, t.base + t.k + (sub % (2 * w) == 0 ? 6 * w : 0));
        x = T::mul(t, x, y);
    }
    return x;
}

// teams per warp where L of them share a power
template <class T, int L> struct PerWarp { static constexpr int N = T::PER / L * L; };

// The twiddle powers of a radix-4 stage (k_gt_radix4_outputs): power e of
// butterfly j of block b, for j < J.  Teams take the blocks of all arrays
// fastest over nbp >= nb = blocks * count slots, so that with nbp a multiple of
// five a warp has one twiddle.
template <class T, int L, bool NAF>
__global__ void __launch_bounds__(32 * T::WARPS, T6_BLOCKS / T::WARPS) k_gt_radix4_pows(uint8_t* ex, const uint8_t* io, const int8_t* rec, int64_t n,
                                                         int64_t h, int64_t J, int64_t nb, int64_t nbp) {
    extern __shared__ uint4 sh[];
    constexpr int PER = PerWarp<T, L>::N;
    const Team t = team_of<T>(sh, PER);
    const int64_t g = team_index<T>(PER) / L;
    const int sub = (int)(team_index<T>(PER) % L);
    int64_t je = g / nbp, b = g % nbp;
    const bool active = je < 3 * J && b < nb;
    if (!active) je = 0, b = 0;
    const int64_t j = je / 3, nblk = n / (4 * h), q = b / nblk, blk = b % nblk;
    const int e = (int)(je % 3);
    int64_t idx = (e == 0 ? 2 * j : (e == 1 ? j : 3 * j)) * (n / (4 * h));
    const bool neg = idx >= n / 2;  // w^(k + n/2) = -w^k: the inverse
    if (neg) idx -= n / 2;
    const ElemOf<T> x = team_load<T>(t, io + GT_SZ * (q * n + blk * 4 * h + j + (int64_t)(e + 1) * h));
    ElemOf<T> r = team_pow<T, L, NAF>(t, x, rec + REC_SZ * idx, sub);
    if (L > 1) r = team_group_product<T, L>(t, r, sub);
    if (neg) r = team_conj<T>(t, r);
    if (active && sub == 0) team_store<T>(t, ex + GT_SZ * (3 * (q * (n / 4) + blk * h + j) + e), r);
}

// x^(omega_4) under the decomposed action.  The forward domain's primitive
// 4th root of unity is omega_4 = |x|^3 (its base-|x| digits are 0, 0, 0, 1),
// which acts as conj(Frobenius^3(x)); the inverse domain's omega_4^-1 acts as
// its inverse, Frobenius^3(x).  (Agrees with the plain power after the hard
// part, like every decomposed action.)
//
// One radix-4 DIT stage merging the radix-2 stages of half sizes h and 2h:
// per block of 4h and offset j < h, with a, b, c, d at j, j+h, j+2h, j+3h and
// w1 = w^(2j s), w2 = w^(j s), w3 = w1 w2 (s = n / 4h):
//   t1 = b^w1, u = c^w2, v = d^w3, cw = u v, dw = (u / v)^omega_4
//   j: a t1 cw   j+h: a/t1 dw   j+2h: a t1 / cw   j+3h: a/t1 / dw
// Three exponentiations per four outputs instead of the radix-2 pair's four.
// A team makes the two outputs that share a t1^(+-1) and cw or dw, from src
// and the powers ex (null: all twiddles are one, the powers are src's own
// values), into dst.  prefix: only outputs below `keep` of each array are
// wanted, of butterflies j < J.
template <class T>
__global__ void __launch_bounds__(32 * T::WARPS, T6_BLOCKS / T::WARPS) k_gt_radix4_outputs(uint8_t* dst, const uint8_t* src, const uint8_t* ex,
                                                            int64_t n, int64_t h, int64_t J, int64_t nb, int inverse,
                                                            int64_t keep) {
    extern __shared__ uint4 sh[];
    const Team t = team_of<T>(sh);
    int64_t g = team_index<T>();
    const bool active = g < 2 * J * nb;
    if (!active) g = 2 * J * nb - 1;
    const int par = (int)(g & 1);
    const int64_t j = (g >> 1) % J, b = (g >> 1) / J, nblk = n / (4 * h), q = b / nblk, blk = b % nblk;
    const int64_t at = q * n + blk * 4 * h + j;
    const uint8_t* powers = ex ? ex + GT_SZ * 3 * (q * (n / 4) + blk * h + j) : src + GT_SZ * (at + h);
    const size_t step = ex ? GT_SZ : GT_SZ * h;
    const ElemOf<T> a = team_load<T>(t, src + GT_SZ * at);
    ElemOf<T> t1 = team_load<T>(t, powers), e2 = team_load<T>(t, powers + 2 * step);
    if (par) {
        t1 = team_conj<T>(t, t1);
        e2 = team_conj<T>(t, e2);
    }
    ElemOf<T> m = T::mul(t, team_load<T>(t, powers + step), e2);
    const ElemOf<T> w = team_frobenius<T>(t, m, 3);
    if (par) m = inverse ? w : team_conj<T>(t, w);
    const ElemOf<T> at1 = T::mul(t, a, t1);
    const int64_t o0 = blk * 4 * h + j + par * h, o1 = o0 + 2 * h;
    const ElemOf<T> r0 = T::mul(t, at1, m);
    if (active && o0 < keep) team_store<T>(t, dst + GT_SZ * (q * n + o0), r0);
    if (!__any_sync(0xffffffffu, active && o1 < keep)) return;
    const ElemOf<T> r1 = T::mul(t, at1, team_conj<T>(t, m));
    if (active && o1 < keep) team_store<T>(t, dst + GT_SZ * (q * n + o1), r1);
}

// the first radix-2 stage (all twiddles one): u v and u / v of neighbours
template <class T>
__global__ void __launch_bounds__(32 * T::WARPS, T6_BLOCKS / T::WARPS) k_gt_radix2_first(uint8_t* dst, const uint8_t* src, int64_t total) {
    extern __shared__ uint4 sh[];
    const Team t = team_of<T>(sh);
    int64_t g = team_index<T>();
    const bool active = g < total;
    if (!active) g = total - 1;
    const uint8_t* pair = src + GT_SZ * (g & ~(int64_t)1);
    ElemOf<T> v = team_load<T>(t, pair + GT_SZ);
    if (g & 1) v = team_conj<T>(t, v);
    const ElemOf<T> r = T::mul(t, team_load<T>(t, pair), v);
    if (active) team_store<T>(t, dst + GT_SZ * g, r);
}

// out[q B + i] = base[(q B + i) stride]^(scalar i) for K arrays of B values
// sharing the B exponents: teams take the arrays fastest over Kp >= K slots
template <class T, int L, bool NAF>
__global__ void __launch_bounds__(32 * T::WARPS, T6_BLOCKS / T::WARPS) k_gt_pow(uint8_t* out, const uint8_t* base, int64_t stride, const int8_t* rec,
                                                 int64_t B, int64_t K, int64_t Kp) {
    extern __shared__ uint4 sh[];
    constexpr int PER = PerWarp<T, L>::N;
    const Team t = team_of<T>(sh, PER);
    const int64_t g = team_index<T>(PER) / L;
    const int sub = (int)(team_index<T>(PER) % L);
    int64_t i = g / Kp, q = g % Kp;
    const bool active = i < B && q < K;
    if (!active) i = 0, q = 0;
    const ElemOf<T> x = team_load<T>(t, base + GT_SZ * stride * (q * B + i));
    ElemOf<T> r = team_pow<T, L, NAF>(t, x, rec + REC_SZ * i, sub);
    if (L > 1) r = team_group_product<T, L>(t, r, sub);
    if (active && sub == 0) team_store<T>(t, out + GT_SZ * (q * B + i), r);
}

// out[i] = base[i stride]^c_i for small signed c_i on cyclotomic values:
// square-and-multiply over the bits of |c_i| with cyclotomic squarings, then
// the inverse (conjugation) for negative c_i -- mul_cyclotomic_signed_small of
// weighted_pfe/src/fft.rs:671-699.  c_i = 0 gives one.
template <class T>
__global__ void __launch_bounds__(32 * T::WARPS, T6_BLOCKS / T::WARPS) k_gt_pow_small(uint8_t* out, const uint8_t* base, int64_t stride,
                                                       const int32_t* coeffs, int64_t n) {
    extern __shared__ uint4 sh[];
    const Team t = team_of<T>(sh);
    int64_t i = team_index<T>();
    const bool active = i < n;
    if (!active) i = n - 1;
    const int32_t c = coeffs[i];
    const uint32_t mag = c < 0 ? (uint32_t)(-(int64_t)c) : (uint32_t)c;
    const ElemOf<T> x = team_load<T>(t, base + GT_SZ * stride * i);
    const uint32_t all = __reduce_or_sync(0xffffffffu, mag);
    ElemOf<T> acc = team_one<T>(t);
    for (int b = 31 - __clz(all | 1); b >= 0; b--) {
        acc = T::cyc_sqr(t, acc);
        if (!__any_sync(0xffffffffu, (mag >> b) & 1)) continue;
        acc = T::mul(t, acc, ((mag >> b) & 1) ? x : team_one<T>(t));
    }
    if (c < 0) acc = team_conj<T>(t, acc);
    if (active) team_store<T>(t, out + GT_SZ * i, acc);
}

// How the powers of a launch of E are spread: over teams of six or twelve lanes,
// L teams each.
struct PowSpread { bool twelve; int L; };
// From a cost model: the wide multiply-adds of one lane, in thousands.  Teams
// of six: 64 squarings of 888; products of 1,608, 52 and three for the table with
// the warp-uniform NAF, 17 a digit and seven for the table in radix 16; table
// images of 744.  Teams of twelve: 444, 1,020 and 444, one team a power with a tenth
// more for its share of other instructions.  Measured on B200, powers of as many
// exponents: 300 0.41 ms, 900 0.67, 2,400 1.10, 4,800 1.51, 6,000 2.54; counted by warps per
// scheduler instead of turns 2,400 1.72.  WBTE_GT_LANES = 1, 2 or 4
// forces that many teams of six, and so does the calling context's tuning knob.
PowSpread gt_pow_spread(int64_t E, bool uniform) {
    if (const char* env = getenv("WBTE_GT_LANES")) {
        const int v = atoi(env);
        if (v == 1 || v == 2 || v == 4) return {false, v};
    }
    if (g_tune.gt_lanes == 1 || g_tune.gt_lanes == 2 || g_tune.gt_lanes == 4) return {false, g_tune.gt_lanes};
    struct Way { PowSpread spread; double work, per; };
    const Way ways[] = {{{false, 1}, uniform ? 156.0 : 195.0, 5.0}, {{false, 2}, 130.0, 2.0}, {{false, 4}, 98.0, 1.0},
                        {{true, 1}, 125.0, 2.0},                    {{true, 2}, 74.0, 1.0}};
    const Way* best = ways;
    double best_t = 0;
    for (const Way& w : ways) {
        const double t = run_time(w.work, (double)E / w.per);
        if (&w == ways || t < best_t) best = &w, best_t = t;
    }
    return best->spread;
}

int64_t pad5(int64_t x) { return (x + TEAMS - 1) / TEAMS * TEAMS; }
// One exponent for every five neighbouring teams: worth idle teams up to the
// difference between the recodings (156 against 195 of gt_pow_spread).
bool uniform_pays(int64_t same) { return same >= TEAMS && 5 * same >= 4 * pad5(same); }

// rec <- the recodings of n scalars; null if there is no memory
int8_t* recode(const uint8_t* scalars, int64_t n, bool naf, cudaStream_t s) {
    int8_t* rec = nullptr;
    if (cudaMallocAsync(&rec, REC_SZ * (size_t)n, s) != cudaSuccess) return nullptr;
    note_launch();
    k_gt_recode<<<blocks_for(n, 64), 64, 0, s>>>(rec, scalars, n, naf ? 1 : 0);
    return rec;
}

void gt_pow_run(uint8_t* out, const uint8_t* base, int64_t stride, const uint8_t* scalars, int64_t B, int64_t K,
                cudaStream_t s) {
    const bool uniform = uniform_pays(K);
    const PowSpread how = gt_pow_spread(B * K, uniform);
    const bool naf = !how.twelve && how.L == 1 && uniform;
    int8_t* rec = recode(scalars, B, naf, s);
    if (!rec) return;
    const int64_t Kp = naf ? pad5(K) : K, items = B * Kp;
    note_launch();
    if (naf)
        team_launch<SixBlock>(k_gt_pow<SixBlock, 1, true>, items, 5, s, out, base, stride, rec, B, K, Kp);
    else if (how.twelve && how.L == 1)
        team_launch<Twelve>(k_gt_pow<Twelve, 1, false>, items, 2, s, out, base, stride, rec, B, K, Kp);
    else if (how.twelve)
        team_launch<Twelve>(k_gt_pow<Twelve, 2, false>, items, 1, s, out, base, stride, rec, B, K, Kp);
    else if (how.L == 1)
        team_launch<SixBlock>(k_gt_pow<SixBlock, 1, false>, items, 5, s, out, base, stride, rec, B, K, Kp);
    else if (how.L == 2)
        team_launch<Six>(k_gt_pow<Six, 2, false>, items, 2, s, out, base, stride, rec, B, K, Kp);
    else
        team_launch<Six>(k_gt_pow<Six, 4, false>, items, 1, s, out, base, stride, rec, B, K, Kp);
    cudaFreeAsync(rec, s);
}

}  // namespace

void launch_gt_pow(uint8_t* out, const uint8_t* base, int64_t stride, const uint8_t* scalars, int64_t n, cudaStream_t s) {
    ProfScope prof_("gt_pow", s);
    if (n <= 0) return;
    gt_pow_run(out, base, stride, scalars, n, 1, s);
}

void launch_gt_pow_shared(uint8_t* out, const uint8_t* base, const uint8_t* scalars, int64_t B, int64_t K,
                          cudaStream_t s) {
    ProfScope prof_("gt_pow", s);
    if (B <= 0 || K <= 0) return;
    gt_pow_run(out, base, 1, scalars, B, K, s);
}

void launch_gt_pow_small(uint8_t* out, const uint8_t* base, int64_t stride, const int32_t* coeffs, int64_t n,
                         cudaStream_t s) {
    ProfScope prof_("gt_pow_small", s);
    if (n <= 0) return;
    note_launch();
    if (few_values(n))
        team_launch<Twelve>(k_gt_pow_small<Twelve>, n, Twelve::PER, s, out, base, stride, coeffs, n);
    else
        team_launch<Six>(k_gt_pow_small<Six>, n, Six::PER, s, out, base, stride, coeffs, n);
}

// The unscaled transform of `count` arrays of n values, keeping the first
// `keep` outputs of each (the rest of io is then undefined).
static void gt_transform(uint8_t* io, const uint8_t* tw, int64_t n, int64_t keep, cudaStream_t s, int64_t count,
                         bool inverse) {
    if (n <= 1 || count <= 0 || keep <= 0) return;
    ProfScope prof_("gt_ifft", s);
    int bits = 0;
    while ((int64_t(1) << bits) < n) bits++;
    const size_t bytes = GT_SZ * (size_t)(n * count);
    // stages go from one buffer to the other
    uint8_t *cur = nullptr, *other = nullptr, *ex = nullptr;
    int8_t *naf = nullptr, *r16 = nullptr;
    bool ok = cudaMallocAsync(&cur, bytes, s) == cudaSuccess && cudaMallocAsync(&other, bytes, s) == cudaSuccess;
    if (ok) {
        note_launch();
        k_gt_bitrev<<<blocks_for(n * count * (int64_t)(GT_SZ / 16), 256), 256, 0, s>>>(cur, io, n, bits, count);
    }
    int64_t half = 1;
    if (ok && (bits & 1)) {
        // an odd number of stages starts with one radix-2 stage, the rest pair up
        note_launch();
        if (few_values(n * count))
            team_launch<Twelve>(k_gt_radix2_first<Twelve>, n * count, Twelve::PER, s, other, cur, n * count);
        else
            team_launch<Six>(k_gt_radix2_first<Six>, n * count, Six::PER, s, other, cur, n * count);
        std::swap(cur, other);
        half = 2;
    }
    for (; ok && half < n; half *= 4) {
        const int64_t nb = n / (4 * half) * count;
        const bool last = 4 * half == n;
        // butterflies with an output below keep (their second output is at j + h)
        const int64_t J = last ? std::min(half, keep) : half;
        if (half > 1) {
            const bool uniform = uniform_pays(nb);
            const PowSpread how = gt_pow_spread(3 * J * nb, uniform);
            const bool use_naf = !how.twelve && how.L == 1 && uniform;
            int8_t*& rec = use_naf ? naf : r16;
            if (!rec) rec = recode(tw, n / 2, use_naf, s);
            if (!rec || (!ex && cudaMallocAsync(&ex, GT_SZ * 3 * (size_t)(n / 4 * count), s) != cudaSuccess)) {
                ok = false;
                break;
            }
            const int64_t nbp = use_naf ? pad5(nb) : nb, items = 3 * J * nbp;
            note_launch();
            if (use_naf)
                team_launch<SixBlock>(k_gt_radix4_pows<SixBlock, 1, true>, items, 5, s, ex, cur, rec, n, half, J, nb, nbp);
            else if (how.twelve && how.L == 1)
                team_launch<Twelve>(k_gt_radix4_pows<Twelve, 1, false>, items, 2, s, ex, cur, rec, n, half, J, nb, nbp);
            else if (how.twelve)
                team_launch<Twelve>(k_gt_radix4_pows<Twelve, 2, false>, items, 1, s, ex, cur, rec, n, half, J, nb, nbp);
            else if (how.L == 1)
                team_launch<SixBlock>(k_gt_radix4_pows<SixBlock, 1, false>, items, 5, s, ex, cur, rec, n, half, J, nb, nbp);
            else if (how.L == 2)
                team_launch<Six>(k_gt_radix4_pows<Six, 2, false>, items, 2, s, ex, cur, rec, n, half, J, nb, nbp);
            else
                team_launch<Six>(k_gt_radix4_pows<Six, 4, false>, items, 1, s, ex, cur, rec, n, half, J, nb, nbp);
        }
        note_launch();
        const uint8_t* powers = half > 1 ? ex : nullptr;
        if (few_values(2 * J * nb))
            team_launch<Twelve>(k_gt_radix4_outputs<Twelve>, 2 * J * nb, Twelve::PER, s, other, cur, powers, n, half, J, nb, inverse ? 1 : 0, last ? keep : n);
        else
            team_launch<Six>(k_gt_radix4_outputs<Six>, 2 * J * nb, Six::PER, s, other, cur, powers, n, half, J, nb,
                                                                                  inverse ? 1 : 0, last ? keep : n);
        std::swap(cur, other);
    }
    if (ok) {
        if (keep == n)
            cudaMemcpyAsync(io, cur, bytes, cudaMemcpyDeviceToDevice, s);
        else
            cudaMemcpy2DAsync(io, GT_SZ * n, cur, GT_SZ * n, GT_SZ * keep, count, cudaMemcpyDeviceToDevice, s);
    }
    for (void* p : {(void*)cur, (void*)other, (void*)ex, (void*)naf, (void*)r16})
        if (p) cudaFreeAsync(p, s);
}
void launch_cyclotomic_prefix_ifft(uint8_t* io, const uint8_t* tw_inv, int64_t n, int64_t out_count, cudaStream_t s,
                                   int64_t count) {
    gt_transform(io, tw_inv, n, std::min(out_count, n), s, count, true);
}
void launch_gt_ntt(uint8_t* io, const uint8_t* tw, int64_t n, cudaStream_t s, int64_t count, bool inverse) {
    gt_transform(io, tw, n, n, s, count, inverse);
}

}  // namespace wbte
