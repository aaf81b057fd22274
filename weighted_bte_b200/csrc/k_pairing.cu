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

// this lane's team in the launch (shadow lanes belong to the warp's last one);
// teams past the end take the last value again without storing it, which is
// their own warp's, so that a call may work in place
__device__ __forceinline__ int64_t team_index() {
    const int tm = (int)(threadIdx.x & 31) / TEAM_LANES;
    return (int64_t)blockIdx.x * TEAMS + (tm < TEAMS ? tm : TEAMS - 1);
}

// the line table of one point per team: lane k writes component k of each record
__global__ void __launch_bounds__(WARP, T6_BLOCKS) k_prepare_lines(uint8_t* lines, const uint8_t* q, int64_t n) {
    __shared__ uint4 sh[T6_ROWS * 32];
    const Team t = team_init(sh);
    int64_t i = team_index();
    const bool active = i < n;
    if (!active) i = n - 1;
    const G2A Q = load_affine(reinterpret_cast<const G2A*>(q + G2_AFF * i));
    // identity lines: every line value is 1, so the loop returns 1
    const bool inf = is_inf(Q);
    const Fp one = t.k == 0 ? fp_one() : fp_zero();
    Fp* L = reinterpret_cast<Fp*>(lines + LINE_SZ * i) + t.k;
    Fp2 T = t.k == 0 ? Q.x : (t.k == 1 ? Q.y : fp2_one());
    for (int b = 62; b >= 0; b--)
        for (int step = 0; step <= (t6_bit(b) ? 1 : 0); step++) {
            const Fp c = step ? t6_line_add(t, T, Q) : t6_line_double(t, T);
            if (active) store_vec(L, fp_select(inf, one, c));
            L += n * (int64_t)(LINE_SZ / sizeof(Fp));
        }
}

// out[o chunks + ch] = prod over run ch (at most C of t < T) of
// Miller(P[(o / p_per) T + t], lines of table (o % per) T + t), one team per
// run: the opening of K batches against one committee's prepared opening keys
// (tables line-major with stride per T), each batch with its own T shares
// (p_per = per: weighted_btx) or each slot with its own T points (p_per = 1:
// weighted_pfe, and single pairs with T = 1).  The pairs of a run share the 62
// squarings.
__global__ void __launch_bounds__(WARP, T6_BLOCKS) k_miller_lines_multi(uint8_t* out, const uint8_t* lines, const uint8_t* p,
                                                             int64_t n, int64_t per, int64_t p_per, int64_t T, int64_t C,
                                                             int64_t chunks) {
    __shared__ uint4 sh[T6_ROWS * 32];
    const Team t = team_init(sh);
    int64_t g = team_index();
    const bool active = g < n * chunks;
    if (!active) g = n * chunks - 1;
    const int64_t o = g / chunks, lo = (g % chunks) * C;
    const int64_t cnt = T - lo < C ? T - lo : C;
    const Fp* L = reinterpret_cast<const Fp*>(lines + LINE_SZ * ((o % per) * T + lo)) + t.k;
    const int64_t stride = per * T * (int64_t)(LINE_SZ / sizeof(Fp));
    const G1A* P = reinterpret_cast<const G1A*>(p) + (o / p_per) * T + lo;
    Fp2 f = t6_one(t);
    for (int i = 62; i >= 0; i--) {
        if (i != 62) f = t6_sqr(t, f);
        for (int step = 0; step <= (t6_bit(i) ? 1 : 0); step++) {
            // runs of one launch differ in length only at the end of T; the
            // shorter ones take lines of value one
            for (int64_t r = 0; r < C; r++) {
                const int64_t x = r < cnt ? r : 0;
                T6Point pt = t6_point(t, load_affine(P + x));
                pt.inf |= r >= cnt;
                f = t6_mul_line(t, f, t6_line_value(t, load_vec(L + x * (int64_t)(LINE_SZ / sizeof(Fp))), pt));
            }
            L += stride;
        }
    }
    f = t6_conj(t, f);
    if (active) t6_store(t, out + GT_SZ * g, f);
}

// Segment s of `per` consecutive pairs is split into `chunks` runs of at most
// C pairs; the team of (s, ch) writes the product of its run's Miller loops,
// lines computed on the fly, one multi-Miller loop sharing the squarings.
// Pair i is (P[p_mod ? i % p_mod : i], Q[q_mod ? i % q_mod : i]).
__global__ void __launch_bounds__(WARP, T6_BLOCKS) k_miller_chunks(uint8_t* out, const uint8_t* p, const uint8_t* q, int64_t per,
                                                        int64_t K, int C, int64_t chunks, int64_t p_mod, int64_t q_mod) {
    __shared__ uint4 sh[T6_ROWS * 32];
    const Team t = team_init(sh);
    int64_t g = team_index();
    const bool active = g < K * chunks;
    if (!active) g = K * chunks - 1;
    const int64_t s = g / chunks, lo = (g % chunks) * C;
    const int cnt = (int)(per - lo < C ? per - lo : C);
    Fp2 T[MULTI_MILLER_MAX];
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
        T[r] = t.k == 0 ? Q.x : (t.k == 1 ? Q.y : fp2_one());
        if (r >= cnt || is_inf(Q)) dead |= 1u << r;
    }
    Fp2 f = t6_one(t);
    for (int i = 62; i >= 0; i--) {
        if (i != 62) f = t6_sqr(t, f);
        for (int step = 0; step <= (t6_bit(i) ? 1 : 0); step++)
            for (int r = 0; r < C; r++) {
                const Fp c = step ? t6_line_add(t, T[r], Q_of(r)) : t6_line_double(t, T[r]);
                T6Point pt = t6_point(t, P_of(r));
                pt.inf |= (dead >> r) & 1;
                f = t6_mul_line(t, f, t6_line_value(t, c, pt));
            }
    }
    f = t6_conj(t, f);
    if (active) t6_store(t, out + GT_SZ * g, f);
}

__global__ void __launch_bounds__(WARP, T6_BLOCKS) k_fp12_segment_product(uint8_t* out, const uint8_t* in, const int64_t* offsets,
                                                               int64_t k) {
    __shared__ uint4 sh[T6_ROWS * 32];
    const Team t = team_init(sh);
    int64_t j = team_index();
    const bool active = j < k;
    if (!active) j = k - 1;
    const int64_t lo = offsets[j], len = active ? offsets[j + 1] - lo : 0;
    const int64_t longest = __reduce_max_sync(0xffffffffu, (unsigned)len);
    Fp2 acc = t6_one(t);
    for (int64_t i = 0; i < longest; i++) {
        const Fp2 x = i < len ? t6_load(t, in + GT_SZ * (lo + i)) : t6_one(t);
        acc = i ? t6_mul(t, acc, x) : x;
    }
    if (active) t6_store(t, out + GT_SZ * j, acc);
}

__global__ void __launch_bounds__(WARP, T6_BLOCKS) k_final_exp(uint8_t* out, const uint8_t* in, int64_t n, int mode) {
    __shared__ uint4 sh[T6_ROWS * 32];
    const Team t = team_init(sh);
    int64_t i = team_index();
    const bool active = i < n;
    if (!active) i = n - 1;
    Fp2 f = t6_load(t, in + GT_SZ * i);
    if (mode != FE_HARD) f = t6_final_exp_easy(t, f);
    if (mode != FE_EASY) f = t6_final_exp_hard(t, f);
    if (active) t6_store(t, out + GT_SZ * i, f);
}

__global__ void __launch_bounds__(WARP, T6_BLOCKS) k_fp12_mul(uint8_t* out, const uint8_t* a, int64_t sa, const uint8_t* b,
                                                   int64_t sb, bool conj_b, int64_t n) {
    __shared__ uint4 sh[T6_ROWS * 32];
    const Team t = team_init(sh);
    int64_t i = team_index();
    const bool active = i < n;
    if (!active) i = n - 1;
    Fp2 y = t6_load(t, b + GT_SZ * sb * i);
    if (conj_b) y = t6_conj(t, y);
    const Fp2 r = t6_mul(t, t6_load(t, a + GT_SZ * sa * i), y);
    if (active) t6_store(t, out + GT_SZ * i, r);
}

__global__ void __launch_bounds__(WARP, T6_BLOCKS) k_unmask(uint8_t* out, const uint8_t* second, const uint8_t* alpha,
                                                 const uint8_t* beta, const uint8_t* valid, int64_t n) {
    __shared__ uint4 sh[T6_ROWS * 32];
    const Team t = team_init(sh);
    int64_t i = team_index();
    const bool active = i < n;
    if (!active) i = n - 1;
    Fp2 r = t6_mul(t, t6_load(t, second + GT_SZ * i), t6_conj(t, t6_load(t, alpha + GT_SZ * i)));
    r = t6_mul(t, r, t6_load(t, beta + GT_SZ * i));
    if (!valid[i]) r = t6_one(t);
    if (active) t6_store(t, out + GT_SZ * i, r);
}

// off[i] = i step
__global__ void k_offsets(int64_t* off, int64_t n, int64_t step) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n) off[i] = i * step;
}

WBTE_INL void fp_store_be48(uint8_t* out, const Fp& m) {
    Fp c = fp_from_mont(m);
    for (int i = 0; i < 48; i++) out[47 - i] = (uint8_t)(c.v[i >> 2] >> (8 * (i & 3)));
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
void launch_prepare_lines(uint8_t* lines, const uint8_t* q, int64_t n, cudaStream_t s) {
    ProfScope prof_("prepare_lines", s);
    if (n <= 0) return;
    note_launch();
    k_prepare_lines<<<blocks_for(n, TEAMS), WARP, 0, s>>>(lines, q, n);
}
// Pairs per team of a launch of `outputs` products of T Miller loops each.
// Sharing the 62 squarings saves 73 of a first pair's wide multiply-adds (in
// thousands per lane: 62 squarings of 1,176; `line` for one pair's 68 lines),
// so runs are cut only while the launch leaves schedulers idle.
static int64_t miller_run(int64_t outputs, int64_t T, double line, int64_t most) {
    int64_t best = 1;
    double best_t = 0;
    for (int64_t C = 1; C <= std::min(T, most); C++) {
        const int64_t chunks = (T + C - 1) / C;
        const double time = launch_time(73.0 + line * C, (double)(outputs * chunks) / TEAMS);
        if (C == 1 || time < best_t) best = C, best_t = time;
    }
    return best;
}
static constexpr double LINE_PREPARED = 130.0, LINE_COMPUTED = 245.0;

static bool miller_lines(uint8_t* out, const uint8_t* lines, const uint8_t* p, int64_t n, int64_t per, int64_t p_per,
                         int64_t T, cudaStream_t s) {
    const int64_t C = miller_run(n, T, LINE_PREPARED, T), chunks = (T + C - 1) / C;
    uint8_t* runs = out;
    int64_t* offs = nullptr;
    if (chunks > 1 && (cudaMallocAsync(&runs, GT_SZ * (size_t)(n * chunks), s) != cudaSuccess ||
                       cudaMallocAsync(&offs, sizeof(int64_t) * (size_t)(n + 1), s) != cudaSuccess))
        return false;
    note_launch();
    k_miller_lines_multi<<<blocks_for(n * chunks, TEAMS), WARP, 0, s>>>(runs, lines, p, n, per, p_per, T, C, chunks);
    if (chunks > 1) {
        note_launch(2);
        k_offsets<<<blocks_for(n + 1), TPB, 0, s>>>(offs, n + 1, chunks);
        k_fp12_segment_product<<<blocks_for(n, TEAMS), WARP, 0, s>>>(out, runs, offs, n);
        cudaFreeAsync(runs, s);
        cudaFreeAsync(offs, s);
    }
    return true;
}
void launch_miller_lines(uint8_t* out, const uint8_t* lines, const uint8_t* p, int64_t n, cudaStream_t s,
                         int64_t lines_n) {
    ProfScope prof_("miller_lines", s);
    if (n <= 0) return;
    miller_lines(out, lines, p, n, lines_n > 0 ? lines_n : n, 1, 1, s);
}
bool launch_miller_lines_multi(uint8_t* out, const uint8_t* lines, const uint8_t* p, int64_t n, int64_t per, int T,
                               cudaStream_t s, int64_t p_per) {
    ProfScope prof_("miller_lines_multi", s);
    if (T < 1 || per < 1) return false;
    if (n <= 0) return true;
    miller_lines(out, lines, p, n, per, p_per > 0 ? p_per : per, T, s);
    return true;
}
void launch_miller(uint8_t* out, const uint8_t* p, const uint8_t* q, int64_t n, cudaStream_t s, int64_t p_mod,
                   int64_t q_mod) {
    ProfScope prof_("miller", s);
    if (n <= 0) return;
    note_launch();
    k_miller_chunks<<<blocks_for(n, TEAMS), WARP, 0, s>>>(out, p, q, 1, n, 1, 1, p_mod, q_mod);
}
int miller_chunk(int64_t pairs) {
    if (g_tune.miller_chunk > 0) return g_tune.miller_chunk;
    return (int)miller_run(1, pairs, LINE_COMPUTED, MULTI_MILLER_MAX);
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
    const int64_t chunks = (per + C - 1) / C;
    note_launch();
    k_miller_chunks<<<blocks_for(K * chunks, TEAMS), WARP, 0, s>>>(out, p, q, per, K, C, chunks, 0, 0);
    return chunks;
}
void launch_fp12_mask(uint8_t* io, const uint8_t* valid, int64_t n, cudaStream_t s) {
    if (n <= 0) return;
    note_launch();
    k_fp12_mask<<<blocks_for(n), TPB, 0, s>>>(io, valid, n);
}
void launch_fp12_segment_product(uint8_t* out, const uint8_t* in, const int64_t* offsets, int64_t k, cudaStream_t s) {
    ProfScope prof_("fp12_product", s);
    if (k <= 0) return;
    note_launch();
    k_fp12_segment_product<<<blocks_for(k, TEAMS), WARP, 0, s>>>(out, in, offsets, k);
}
void launch_final_exp(uint8_t* out, const uint8_t* in, int64_t n, FinalExpMode mode, cudaStream_t s) {
    ProfScope prof_(mode == FE_EASY ? "final_exp_easy" : (mode == FE_HARD ? "final_exp_hard" : "final_exp"), s);
    if (n <= 0) return;
    note_launch();
    k_final_exp<<<blocks_for(n, TEAMS), WARP, 0, s>>>(out, in, n, (int)mode);
}

void launch_fp12_mul(uint8_t* out, const uint8_t* a, int64_t sa, const uint8_t* b, int64_t sb, bool conj_b, int64_t n, cudaStream_t s) {
    if (n <= 0) return;
    note_launch();
    k_fp12_mul<<<blocks_for(n, TEAMS), WARP, 0, s>>>(out, a, sa, b, sb, conj_b, n);
}
void launch_unmask(uint8_t* out, const uint8_t* second, const uint8_t* alpha, const uint8_t* beta, const uint8_t* valid,
                   int64_t n, cudaStream_t s) {
    ProfScope prof_("unmask", s);
    if (n <= 0) return;
    note_launch();
    k_unmask<<<blocks_for(n, TEAMS), WARP, 0, s>>>(out, second, alpha, beta, valid, n);
}
void launch_gt_compress(uint8_t* out, const uint8_t* in, int64_t n, cudaStream_t s) {
    ProfScope prof_("gt_compress", s);
    if (n <= 0) return;
    note_launch();
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
