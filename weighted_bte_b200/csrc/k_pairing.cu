// Pairing-side kernels: G2 line tables, Miller loops, split final
// exponentiation and the GT element kernels (products, masks, encodings).
// The GT transforms live in k_gt.cu.
#include <algorithm>
#include <atomic>
#include <cstdlib>

#include "launch.h"
#include "team.cuh"

namespace wbte {

namespace {
constexpr int TPB = 64, WARP = 32;
inline unsigned blocks_for(int64_t n, int tpb = TPB) { return (unsigned)((n + tpb - 1) / tpb); }

WBTE_INL Fp12* as_gt(uint8_t* p) { return reinterpret_cast<Fp12*>(p); }
WBTE_INL const Fp12* as_gt(const uint8_t* p) { return reinterpret_cast<const Fp12*>(p); }

// the line table of one point per team: lane k writes component k of each record
template <class T>
__global__ void __launch_bounds__(32 * T::WARPS, T6_BLOCKS / T::WARPS) k_prepare_lines(uint8_t* lines, const uint8_t* q, int64_t n) {
    extern __shared__ uint4 sh[];
    const Team t = team_of<T>(sh);
    int64_t i = team_index<T>();
    const bool active = i < n;
    if (!active) i = n - 1;
    const G2A Q = load_affine(reinterpret_cast<const G2A*>(q + G2_AFF * i));
    // identity lines: every line value is 1, so the loop returns 1
    const bool inf = is_inf(Q);
    const int component = T::line_index(t);
    const Fp one = component == 0 ? fp_one() : fp_zero();
    Fp* L = reinterpret_cast<Fp*>(lines + LINE_SZ * i) + component;
    ElemOf<T> S = T::of(t, t.k == 0 ? Q.x : (t.k == 1 ? Q.y : fp2_one()));
    for (int b = 62; b >= 0; b--)
        for (int step = 0; step <= (miller_bit(b) ? 1 : 0); step++) {
            const Fp c = step ? team_line_add<T>(t, S, Q) : team_line_double<T>(t, S);
            if (active) store_vec(L, fp_select(inf, one, c));
            L += n * (int64_t)(LINE_SZ / sizeof(Fp));
        }
}

// out[o chunks + ch] = prod over run ch (at most C of t < pairs) of
// Miller(P[(o / p_per) pairs + t], lines of table (o % per) pairs + t), one team
// per run: the opening of K batches against one committee's prepared opening keys
// (tables line-major with stride per * pairs), each batch with its own shares
// (p_per = per: weighted_btx) or each slot with its own points (p_per = 1:
// weighted_pfe, and single pairs).  The pairs of a run share the 62
// squarings.
template <class T>
__global__ void __launch_bounds__(32 * T::WARPS, T6_BLOCKS / T::WARPS) k_miller_lines_multi(uint8_t* out, const uint8_t* lines, const uint8_t* p,
                                                             int64_t n, int64_t per, int64_t p_per, int64_t pairs, int64_t C,
                                                             int64_t chunks) {
    extern __shared__ uint4 sh[];
    const Team t = team_of<T>(sh);
    int64_t g = team_index<T>();
    const bool active = g < n * chunks;
    if (!active) g = n * chunks - 1;
    const int64_t o = g / chunks, lo = (g % chunks) * C;
    const int64_t cnt = pairs - lo < C ? pairs - lo : C;
    const Fp* L = reinterpret_cast<const Fp*>(lines + LINE_SZ * ((o % per) * pairs + lo)) + T::line_index(t);
    const int64_t stride = per * pairs * (int64_t)(LINE_SZ / sizeof(Fp));
    const G1A* P = reinterpret_cast<const G1A*>(p) + (o / p_per) * pairs + lo;
    ElemOf<T> f = team_one<T>(t);
    for (int i = 62; i >= 0; i--) {
        if (i != 62) f = T::sqr(t, f);
        for (int step = 0; step <= (miller_bit(i) ? 1 : 0); step++) {
            // runs of one launch differ in length only at the end; the
            // shorter ones take lines of value one
            for (int64_t r = 0; r < C; r++) {
                T::step();
                const int64_t x = r < cnt ? r : 0;
                TeamPoint pt = team_point<T>(t, load_affine(P + x));
                pt.inf |= r >= cnt;
                f = T::mul_line(t, f, team_line_value<T>(t, load_vec(L + x * (int64_t)(LINE_SZ / sizeof(Fp))), pt));
            }
            L += stride;
        }
    }
    f = team_conj<T>(t, f);
    if (active) team_store<T>(t, out + GT_SZ * g, f);
}

// Segment s of `per` consecutive pairs is split into `chunks` runs of at most
// C pairs; the team of (s, ch) writes the product of its run's Miller loops,
// lines computed on the fly, one multi-Miller loop sharing the squarings.
// Pair i is (P[p_mod ? i % p_mod : i], Q[q_mod ? i % q_mod : i]).
template <class T>
__global__ void __launch_bounds__(32 * T::WARPS, T6_BLOCKS / T::WARPS) k_miller_chunks(uint8_t* out, const uint8_t* p, const uint8_t* q, int64_t per,
                                                        int64_t K, int C, int64_t chunks, int64_t p_mod, int64_t q_mod) {
    extern __shared__ uint4 sh[];
    const Team t = team_of<T>(sh);
    int64_t g = team_index<T>();
    const bool active = g < K * chunks;
    if (!active) g = K * chunks - 1;
    const int64_t s = g / chunks, lo = (g % chunks) * C;
    const int cnt = (int)(per - lo < C ? per - lo : C);
    ElemOf<T> S[MULTI_MILLER_MAX];
    auto P_of = [&](int r) {
        const int64_t i = s * per + lo + (r < cnt ? r : 0);
        return load_affine(reinterpret_cast<const G1A*>(p) + (p_mod ? i % p_mod : i));
    };
    auto Q_of = [&](int r) {
        const int64_t i = s * per + lo + (r < cnt ? r : 0);
        return load_affine(reinterpret_cast<const G2A*>(q) + (q_mod ? i % q_mod : i));
    };
    uint32_t dead = 0;  // pairs past the run or with an identity: lines of value one
    for (int r = 0; r < C; r++) {
        const G2A Q = Q_of(r);
        S[r] = T::of(t, t.k == 0 ? Q.x : (t.k == 1 ? Q.y : fp2_one()));
        if (r >= cnt || is_inf(Q)) dead |= 1u << r;
    }
    ElemOf<T> f = team_one<T>(t);
    for (int i = 62; i >= 0; i--) {
        if (i != 62) f = T::sqr(t, f);
        for (int step = 0; step <= (miller_bit(i) ? 1 : 0); step++)
            for (int r = 0; r < C; r++) {
                T::step();
                const Fp c = step ? team_line_add<T>(t, S[r], Q_of(r)) : team_line_double<T>(t, S[r]);
                TeamPoint pt = team_point<T>(t, P_of(r));
                pt.inf |= (dead >> r) & 1;
                f = T::mul_line(t, f, team_line_value<T>(t, c, pt));
            }
    }
    f = team_conj<T>(t, f);
    if (active) team_store<T>(t, out + GT_SZ * g, f);
}

template <class T>
__global__ void __launch_bounds__(32 * T::WARPS, T6_BLOCKS / T::WARPS) k_fp12_segment_product(uint8_t* out, const uint8_t* in, const int64_t* offsets,
                                                               int64_t k) {
    extern __shared__ uint4 sh[];
    const Team t = team_of<T>(sh);
    int64_t j = team_index<T>();
    const bool active = j < k;
    if (!active) j = k - 1;
    const int64_t lo = offsets[j], len = active ? offsets[j + 1] - lo : 0;
    const int64_t longest = __reduce_max_sync(0xffffffffu, (unsigned)len);
    ElemOf<T> acc = team_one<T>(t);
    for (int64_t i = 0; i < longest; i++) {
        const ElemOf<T> x = i < len ? team_load<T>(t, in + GT_SZ * (lo + i)) : team_one<T>(t);
        acc = i ? T::mul(t, acc, x) : x;
    }
    if (active) team_store<T>(t, out + GT_SZ * j, acc);
}

template <class T>
__global__ void __launch_bounds__(32 * T::WARPS, T6_BLOCKS / T::WARPS) k_final_exp(uint8_t* out, const uint8_t* in, int64_t n, int mode) {
    extern __shared__ uint4 sh[];
    const Team t = team_of<T>(sh);
    int64_t i = team_index<T>();
    const bool active = i < n;
    if (!active) i = n - 1;
    ElemOf<T> f = team_load<T>(t, in + GT_SZ * i);
    if (mode != FE_HARD) f = team_final_exp_easy<T>(t, f);
    if (mode != FE_EASY) f = team_final_exp_hard<T>(t, f);
    if (active) team_store<T>(t, out + GT_SZ * i, f);
}

template <class T>
__global__ void __launch_bounds__(32 * T::WARPS, T6_BLOCKS / T::WARPS) k_fp12_mul(uint8_t* out, const uint8_t* a, int64_t sa, const uint8_t* b,
                                                   int64_t sb, bool conj_b, int64_t n) {
    extern __shared__ uint4 sh[];
    const Team t = team_of<T>(sh);
    int64_t i = team_index<T>();
    const bool active = i < n;
    if (!active) i = n - 1;
    ElemOf<T> y = team_load<T>(t, b + GT_SZ * sb * i);
    if (conj_b) y = team_conj<T>(t, y);
    const ElemOf<T> r = T::mul(t, team_load<T>(t, a + GT_SZ * sa * i), y);
    if (active) team_store<T>(t, out + GT_SZ * i, r);
}

template <class T>
__global__ void __launch_bounds__(32 * T::WARPS, T6_BLOCKS / T::WARPS) k_unmask(uint8_t* out, const uint8_t* second, const uint8_t* alpha,
                                                 const uint8_t* beta, const uint8_t* valid, int64_t n) {
    extern __shared__ uint4 sh[];
    const Team t = team_of<T>(sh);
    int64_t i = team_index<T>();
    const bool active = i < n;
    if (!active) i = n - 1;
    ElemOf<T> r = T::mul(t, team_load<T>(t, second + GT_SZ * i), team_conj<T>(t, team_load<T>(t, alpha + GT_SZ * i)));
    r = T::mul(t, r, team_load<T>(t, beta + GT_SZ * i));
    if (!valid[i]) r = team_one<T>(t);
    if (active) team_store<T>(t, out + GT_SZ * i, r);
}

// off[i] = i step
__global__ void k_offsets(int64_t* off, int64_t n, int64_t step) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n) off[i] = i * step;
}

// Tagged torus compression of GT: identity -> 0; otherwise 1 followed by the
// six Fp2 coefficients of (c0 + 1) / c1, each Fp as 48 big-endian bytes.
__global__ void k_gt_compress(uint8_t* out, const uint8_t* in, int64_t n) {
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    Fp12 f = load_vec(as_gt(in) + i);
    uint8_t* o = out + 289 * i;
    if (fp12_is_one(f)) {
        for (int b = 0; b < 289; b++) o[b] = 0;
        return;
    }
    Fp6 c0 = f.c0, inv, b;
    c0.c0 = fp2_add(c0.c0, fp2_one());
    fp6_inv(inv, f.c1);
    fp6_mul(b, c0, inv);
    o[0] = 1;
    const Fp2* cs[3] = {&b.c0, &b.c1, &b.c2};
    for (int k = 0; k < 3; k++) {
        fp_store_be48(o + 1 + 96 * k, cs[k]->c0);
        fp_store_be48(o + 1 + 96 * k + 48, cs[k]->c1);
    }
}

// The same by teams, for few values: 1 / c1 = N^(p^2) N^(p^4) / (N N^(p^2) N^(p^4))
// for N = c1 in Fp6.  Measured on B200: 512 values 0.14 -> 0.07 ms; one thread per value
// once a team's copies of the inversion no longer run on idle schedulers.
template <class T>
__global__ void __launch_bounds__(32 * T::WARPS, T6_BLOCKS / T::WARPS) k_gt_compress_team(uint8_t* out, const uint8_t* in, int64_t n) {
    extern __shared__ uint4 sh[];
    const Team t = team_of<T>(sh);
    int64_t i = team_index<T>();
    const bool active = i < n;
    if (!active) i = n - 1;
    const ElemOf<T> f = team_load<T>(t, in + GT_SZ * i), one = team_one<T>(t), zero = T::f_sub(one, one);
    const uint32_t differ = __ballot_sync(FULL, !T::same(f, one));
    const bool odd = t.k & 1, is_one = !((differ >> (t.base / 6 * T::LANES)) & ((1u << T::LANES) - 1u));
    __syncwarp();
    T::st(t, T6_A, t.base + t.k, f);
    __syncwarp();
    const ElemOf<T> above = T::ld(t, T6_A, t.base + (t.k | 1));
    const ElemOf<T> c1 = odd ? zero : above, sum = T::f_add(f, one), c0 = odd ? zero : sum;
    const ElemOf<T> c2 = team_frobenius<T>(t, c1, 2);
    const ElemOf<T> m = T::mul(t, c2, team_frobenius<T>(t, c2, 2));
    const ElemOf<T> d = team_inverse_of_first<T>(t, T::mul(t, c1, m));
    const ElemOf<T> r = T::mul(t, c0, T::f_mul(m, d));
    if (!active || odd) return;
    uint8_t* o = out + 289 * i;
    if (t.k == 0 && t.h == 0) o[0] = is_one ? 0 : 1;
    T::store_be(t, o + 1 + 48 * t.k, is_one ? zero : r);
}

__global__ void k_fp12_conj(uint8_t* out, const uint8_t* in, int64_t n) {
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    Fp12 x = load_vec(as_gt(in) + i);
    fp12_conj(x, x);
    store_vec(as_gt(out) + i, x);
}

__global__ void k_fp12_mask(uint8_t* io, const uint8_t* valid, int64_t n) {
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (!valid[i]) store_vec(as_gt(io) + i, fp12_one());
}

__global__ void k_fp12_is_one(uint8_t* flags, const uint8_t* in, int64_t n) {
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    flags[i] = fp12_is_one(load_vec(as_gt(in) + i)) ? 1 : 0;
}
}  // namespace

// ============================================================ launchers
// How a launch of `outputs` products of `pairs` Miller loops each is spread: over
// teams of six or twelve lanes, C pairs to a team.  Sharing the 62 squarings
// saves 73 thousand of a lane's wide multiply-adds (45 in a team of twelve) for
// each further pair of a run; `line` is one pair's 68 lines (LINE_PREPARED,
// LINE_COMPUTED; the second figure for teams of twelve).  Whole turns count (65,664
// pairs, runs of six instead of eight 28.8 -> 23.0 ms; 49,248, of three 27.5 -> 18.0).
struct MillerSpread { bool twelve; int64_t C; };
struct LineWork { double six, twelve; };
static constexpr LineWork LINE_PREPARED = {130.0, 90.0}, LINE_COMPUTED = {245.0, 160.0};
static MillerSpread miller_spread(int64_t outputs, int64_t pairs, LineWork line, int64_t most) {
    MillerSpread best = {false, 1};
    double best_t = 0;
    for (int64_t C = 1; C <= std::min(pairs, most); C++) {
        const double runs = (double)outputs * (double)((pairs + C - 1) / C);
        const double six = run_time(73.0 + line.six * C, runs / Six::PER);
        const double twelve = run_time(45.0 + line.twelve * C, runs / Twelve::PER);
        if (C == 1 || six < best_t) best = {false, C}, best_t = six;
        if (twelve < best_t) best = {true, C}, best_t = twelve;
    }
    return best;
}

void launch_prepare_lines(uint8_t* lines, const uint8_t* q, int64_t n, cudaStream_t s) {
    ProfScope prof_("prepare_lines", s);
    if (n <= 0) return;
    note_launch();
    if (run_time(95.0, (double)n / Twelve::PER) < run_time(150.0, (double)n / Six::PER))
        team_launch<Twelve>(k_prepare_lines<Twelve>, n, Twelve::PER, s, lines, q, n);
    else
        team_launch<Six>(k_prepare_lines<Six>, n, Six::PER, s, lines, q, n);
}

static void segment_product(uint8_t* out, const uint8_t* in, const int64_t* offsets, int64_t k, cudaStream_t s) {
    note_launch();
    if (few_values(k))
        team_launch<Twelve>(k_fp12_segment_product<Twelve>, k, Twelve::PER, s, out, in, offsets, k);
    else
        team_launch<Six>(k_fp12_segment_product<Six>, k, Six::PER, s, out, in, offsets, k);
}

// false (nothing launched, the runtime's error pending) if there is no memory for
// the runs' products
static bool miller_lines(uint8_t* out, const uint8_t* lines, const uint8_t* p, int64_t n, int64_t per, int64_t p_per,
                         int64_t pairs, cudaStream_t s) {
    const MillerSpread how = miller_spread(n, pairs, LINE_PREPARED, pairs);
    const int64_t chunks = (pairs + how.C - 1) / how.C;
    uint8_t* runs = out;
    int64_t* offs = nullptr;
    if (chunks > 1) {
        if (cudaMallocAsync(&runs, GT_SZ * (size_t)(n * chunks), s) != cudaSuccess) return false;
        if (cudaMallocAsync(&offs, sizeof(int64_t) * (size_t)(n + 1), s) != cudaSuccess) {
            cudaFreeAsync(runs, s);
            return false;
        }
    }
    note_launch();
    if (how.twelve)
        team_launch<Twelve>(k_miller_lines_multi<Twelve>, n * chunks, Twelve::PER, s, runs, lines, p, n, per, p_per, pairs,
                                                                                      how.C, chunks);
    else
        team_launch<SixBlock>(k_miller_lines_multi<SixBlock>, n * chunks, Six::PER, s, runs, lines, p, n, per, p_per, pairs,
                                                                                how.C, chunks);
    if (chunks > 1) {
        note_launch();
        k_offsets<<<blocks_for(n + 1), TPB, 0, s>>>(offs, n + 1, chunks);
        segment_product(out, runs, offs, n, s);
        cudaFreeAsync(runs, s);
        cudaFreeAsync(offs, s);
    }
    return true;
}
void launch_miller_lines(uint8_t* out, const uint8_t* lines, const uint8_t* p, int64_t n, cudaStream_t s,
                         int64_t lines_n) {
    ProfScope prof_("miller_lines", s);
    if (n <= 0) return;
    miller_lines(out, lines, p, n, lines_n > 0 ? lines_n : n, 1, 1, s);  // one run a value: no scratch
}
bool launch_miller_lines_multi(uint8_t* out, const uint8_t* lines, const uint8_t* p, int64_t n, int64_t per, int T,
                               cudaStream_t s, int64_t p_per) {
    ProfScope prof_("miller_lines_multi", s);
    if (T < 1 || per < 1) return false;
    if (n <= 0) return true;
    return miller_lines(out, lines, p, n, per, p_per > 0 ? p_per : per, T, s);
}
static void miller_chunks(uint8_t* out, const uint8_t* p, const uint8_t* q, int64_t per, int64_t K, int C, int64_t p_mod,
                          int64_t q_mod, cudaStream_t s) {
    const int64_t chunks = (per + C - 1) / C, runs = K * chunks;
    note_launch();
    if (run_time(45.0 + LINE_COMPUTED.twelve * C, (double)runs / Twelve::PER) <
        run_time(73.0 + LINE_COMPUTED.six * C, (double)runs / Six::PER))
        team_launch<Twelve>(k_miller_chunks<Twelve>, runs, Twelve::PER, s, out, p, q, per, K, C, chunks, p_mod, q_mod);
    else
        team_launch<SixBlock>(k_miller_chunks<SixBlock>, runs, Six::PER, s, out, p, q, per, K, C, chunks, p_mod, q_mod);
}
void launch_miller(uint8_t* out, const uint8_t* p, const uint8_t* q, int64_t n, cudaStream_t s, int64_t p_mod,
                   int64_t q_mod) {
    ProfScope prof_("miller", s);
    if (n <= 0) return;
    miller_chunks(out, p, q, 1, n, 1, p_mod, q_mod, s);
}
int miller_chunk(int64_t pairs) {
    if (g_tune.miller_chunk > 0) return g_tune.miller_chunk;
    return (int)miller_spread(1, pairs, LINE_COMPUTED, MULTI_MILLER_MAX).C;
}
int64_t launch_miller_chunks(uint8_t* out, const uint8_t* p, const uint8_t* q, int64_t per, int64_t K, int C,
                             cudaStream_t s) {
    if (per <= 0 || K <= 0) return 0;
    if (C < 1) C = 1;
    if (C > MULTI_MILLER_MAX) C = MULTI_MILLER_MAX;
    // the profile tag names the run length, which fixes the product count
    static const char* const tags[MULTI_MILLER_MAX + 1] = {"", "miller_c1", "miller_c2", "miller_c3", "miller_c4",
                                                          "miller_c5", "miller_c6", "miller_c7", "miller_c8"};
    ProfScope prof_(tags[C], s);
    miller_chunks(out, p, q, per, K, C, 0, 0, s);
    return (per + C - 1) / C;
}
void launch_fp12_mask(uint8_t* io, const uint8_t* valid, int64_t n, cudaStream_t s) {
    if (n <= 0) return;
    note_launch();
    k_fp12_mask<<<blocks_for(n), TPB, 0, s>>>(io, valid, n);
}
void launch_fp12_segment_product(uint8_t* out, const uint8_t* in, const int64_t* offsets, int64_t k, cudaStream_t s) {
    ProfScope prof_("fp12_product", s);
    if (k <= 0) return;
    segment_product(out, in, offsets, k, s);
}
void launch_final_exp(uint8_t* out, const uint8_t* in, int64_t n, FinalExpMode mode, cudaStream_t s) {
    ProfScope prof_(mode == FE_EASY ? "final_exp_easy" : (mode == FE_HARD ? "final_exp_hard" : "final_exp"), s);
    if (n <= 0) return;
    note_launch();
    // 315 cyclotomic squarings and 35 products of the hard part, an eighth more for
    // a team of twelve's share of other instructions (2,400 hard parts 1.42 ms, 6,000
    // 3.28; counted by warps per scheduler instead of turns 2.01 and 3.29)
    if (run_time(198.0, (double)n / Twelve::PER) < run_time(336.0, (double)n / Six::PER))
        team_launch<Twelve>(k_final_exp<Twelve>, n, Twelve::PER, s, out, in, n, (int)mode);
    else
        team_launch<Six>(k_final_exp<Six>, n, Six::PER, s, out, in, n, (int)mode);
}

void launch_fp12_mul(uint8_t* out, const uint8_t* a, int64_t sa, const uint8_t* b, int64_t sb, bool conj_b, int64_t n, cudaStream_t s) {
    if (n <= 0) return;
    note_launch();
    if (few_values(n))
        team_launch<Twelve>(k_fp12_mul<Twelve>, n, Twelve::PER, s, out, a, sa, b, sb, conj_b, n);
    else
        team_launch<Six>(k_fp12_mul<Six>, n, Six::PER, s, out, a, sa, b, sb, conj_b, n);
}
void launch_unmask(uint8_t* out, const uint8_t* second, const uint8_t* alpha, const uint8_t* beta, const uint8_t* valid,
                   int64_t n, cudaStream_t s) {
    ProfScope prof_("unmask", s);
    if (n <= 0) return;
    note_launch();
    if (few_values(n))
        team_launch<Twelve>(k_unmask<Twelve>, n, Twelve::PER, s, out, second, alpha, beta, valid, n);
    else
        team_launch<Six>(k_unmask<Six>, n, Six::PER, s, out, second, alpha, beta, valid, n);
}
void launch_gt_compress(uint8_t* out, const uint8_t* in, int64_t n, cudaStream_t s) {
    ProfScope prof_("gt_compress", s);
    if (n <= 0) return;
    note_launch();
    if (few_values(n))
        team_launch<Twelve>(k_gt_compress_team<Twelve>, n, Twelve::PER, s, out, in, n);
    else
        k_gt_compress<<<blocks_for(n), TPB, 0, s>>>(out, in, n);
}
void launch_fp12_conj(uint8_t* out, const uint8_t* in, int64_t n, cudaStream_t s) {
    if (n <= 0) return;
    note_launch();
    k_fp12_conj<<<blocks_for(n), TPB, 0, s>>>(out, in, n);
}
void launch_fp12_is_one(uint8_t* flags, const uint8_t* in, int64_t n, cudaStream_t s) {
    if (n <= 0) return;
    note_launch();
    k_fp12_is_one<<<blocks_for(n), TPB, 0, s>>>(flags, in, n);
}

}  // namespace wbte
