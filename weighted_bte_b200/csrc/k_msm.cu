// Pippenger multi-scalar multiplication for families of equal-length MSMs.
//
//   out[j] = sum_t scalars[v_j][t] * points[pbase[j] + idx[t]]
//
// This covers blst's contiguous `p{1,2}s_mult_pippenger` blocks (one MSM,
// idx = identity), the reference's sparse indexed G2 MSMs
// (weighted_btx/src/blst_utils.rs:106-125: idx = accepted virtual indices,
// one base block per kernel offset) and the per-slot party blocks of
// weighted_btx/src/decryption.rs:463-481 (one family per party).  Scalars are
// shared by every MSM using the same vector, so the signed-digit recoding and
// the per-window bucket sort are done once per (vector, window).
//
// Pipeline:
//  1. digits:  signed c-bit windows, digit in (-2^(c-1), 2^(c-1)], the highest
//              as it is
//  2. sort:    one CTA per (vector, window) counting-sorts term indices by
//              |digit| in descending order (zero digits dropped)
//  3. segments: one thread per (MSM, window, segment of S sorted terms)
//              evaluates sum_e |d_e| * (+-P_e) over its segment with a running
//              sum (Abel summation) -- no bucket array is materialised
//  4. reduce:  tree sums over the segments of each (MSM, window)
//  5. combine: Horner over windows, then conversion to affine.
// Group addition is exact and commutative, so the result does not depend on
// the order that atomics give terms inside a bucket.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <mutex>
#include <type_traits>

#include "launch.h"
#include "quad.cuh"

namespace wbte {

namespace {
constexpr int TPB = 128;
constexpr int SEG_TPB = 64;  // threads per block of k_segments
inline unsigned blocks_for(int64_t n, int tpb = TPB) { return (unsigned)((n + tpb - 1) / tpb); }

template <class F> struct Aff;
template <> struct Aff<Fp> { static constexpr size_t SZ = G1_AFF; };
template <> struct Aff<Fp2> { static constexpr size_t SZ = G2_AFF; };

// entry packing: term index (32 bits) | bucket (16 bits) << 32 | sign << 63
WBTE_INL uint64_t pack_entry(uint32_t t, uint32_t b, bool negative) {
    return (uint64_t)t | ((uint64_t)b << 32) | ((uint64_t)(negative ? 1 : 0) << 63);
}

__global__ void k_digits(int16_t* digits, const uint8_t* scalars, int64_t total, int64_t n, int c, int windows) {
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;  // i = v * n + t
    if (i >= total) return;
    uint32_t k[8];
    load_scalar(k, scalars + FR_SZ * i);
    int64_t v = i / n, t = i % n;
    int carry = 0;
    const int full = 1 << c, half = 1 << (c - 1);
    for (int w = 0; w < windows; w++) {
        int bit = w * c;
        uint32_t val = 0;
        if (bit < 256) {
            int word = bit >> 5, off = bit & 31;
            uint64_t two = (uint64_t)k[word] | ((word + 1 < 8) ? ((uint64_t)k[word + 1] << 32) : 0ull);
            val = (uint32_t)(two >> off) & (uint32_t)(full - 1);
        }
        int d = (int)val + carry;
        // the highest digit has no window to carry into
        if (d > half && w + 1 < windows) {
            d -= full;
            carry = 1;
        } else {
            carry = 0;
        }
        digits[(v * windows + w) * n + t] = (int16_t)d;
    }
}

// One CTA per (vector, window).  counts lives in dynamic shared memory.  `top`:
// the highest window's buckets.  They are the others' unless the windows end at bit
// 256 (c = 4 and 8), where its digits, recoded no further, go up to 2^c: those of
// scalars from 2^255 on, which are no residues but multiply all the same.
__global__ void k_sort(uint64_t* entries, int32_t* nnz, const int16_t* digits, int64_t n, int buckets, int top,
                       int windows) {
    extern __shared__ int32_t sh[];
    if (blockIdx.x % windows == windows - 1) buckets = top;
    int32_t* cnt = sh;                // buckets + 1
    int32_t* cur = sh + buckets + 1;  // buckets + 1
    int64_t vw = blockIdx.x;
    const int16_t* d = digits + vw * n;
    for (int b = threadIdx.x; b <= buckets; b += blockDim.x) cnt[b] = 0;
    __syncthreads();
    for (int64_t t = threadIdx.x; t < n; t += blockDim.x) {
        int x = d[t];
        atomicAdd(&cnt[x < 0 ? -x : x], 1);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        // descending bucket order; bucket 0 is dropped
        int32_t run = 0;
        for (int b = buckets; b >= 1; b--) {
            cur[b] = run;
            run += cnt[b];
        }
        nnz[vw] = run;
    }
    __syncthreads();
    uint64_t* out = entries + vw * n;
    for (int64_t t = threadIdx.x; t < n; t += blockDim.x) {
        int x = d[t];
        int b = x < 0 ? -x : x;
        if (b == 0) continue;
        int32_t pos = atomicAdd(&cur[b], 1);
        out[pos] = pack_entry((uint32_t)t, (uint32_t)b, x < 0);
    }
}

// One lane (G1) or pair of lanes (G2) per segment of S sorted terms of one
// (MSM, window): the running sum `run` of the terms seen so far, and at each
// bucket transition (bucket cur_b to b < cur_b) acc += (cur_b - b) * run; at the
// end acc += cur_b * run (Abel summation: acc = sum over the segment of
// |d| * (+-P)).
// Adding at the transition itself would have a warp run the addition whenever
// any of its segments does, so every segment would pay an XYZZ addition per term
// besides its mixed addition.  Instead a lane stores a snapshot of run (and the
// gap) in a small queue in shared memory, and all segments of the warp add
// their oldest entry together: when each segment that still has terms holds
// one, or when one's queue is full.  An entry with a gap above one stays for its
// next turn unless the warp's largest gap makes double-and-add cheaper.  The sum
// is the same: the group is commutative and every snapshot is added as often
// as its gap says.
// The multiply-add pipe bounds it.  Measured on B200: see Point for why G2 takes
// pairs; the families of a committee preparation at B = 512 (512 MSMs for each
// of three parties, 1,382 terms together, and 1,023 of 1,382) 171 -> 84 ms,
// one MSM of 20,011 points 2.5 -> 1.3 ms; G1 as one thread per segment was,
// 1.3 ms at 65,536 points.
// The MSMs of a family run fastest over the lanes: those that share a scalar
// vector have the same transitions, so a warp's segments queue and add
// together (84 -> 81 ms), and the block's warps meet before each term, which
// lets them share instruction fetches (81 -> 79 ms; blocks of 128 threads 79.5,
// of 256 84 ms).
constexpr int SEG_QUEUE = 4;
constexpr size_t SEG_SMEM = (sizeof(Point<OnLane>) + sizeof(uint32_t)) * SEG_QUEUE * SEG_TPB;

template <class P>
__global__ void __launch_bounds__(SEG_TPB) k_segments(uint8_t* seg_out, const uint8_t* points, const int64_t* pbase,
                                                        const int32_t* idx, const uint64_t* entries,
                                                        const int32_t* nnz, const int32_t* vsel, int64_t k, int64_t n,
                                                        int windows, int64_t S, int64_t nseg) {
    using Pt = Point<P>;
    extern __shared__ __align__(16) uint8_t seg_sh[];
    Pt* qv = reinterpret_cast<Pt*>(seg_sh) + threadIdx.x;
    uint32_t* qg = reinterpret_cast<uint32_t*>(seg_sh + sizeof(Pt) * SEG_QUEUE * SEG_TPB) + threadIdx.x;
    const int64_t gid = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / P::LANES;
    // lanes past the grid's work run along with an empty segment
    const bool real = gid < k * windows * nseg;
    int64_t lo = 0, hi = 0, out = 0;
    const uint64_t* e = entries;
    const uint8_t* base = points;
    if (real) {
        const int64_t j = gid % k;
        const int64_t seg = (gid / k) % nseg;
        const int64_t w = gid / (k * nseg);
        out = (j * windows + w) * nseg + seg;
        const int64_t vw = (vsel ? (int64_t)vsel[j] : 0) * windows + w;
        lo = seg * S;
        hi = lo + S;
        const int64_t cnt = nnz[vw];
        if (hi > cnt) hi = cnt;
        if (lo > hi) lo = hi;
        e = entries + vw * n;
        base = points + 2 * P::FIELD * pbase[j];
    }
    Pt run = Pt::infinity(), acc = Pt::infinity();
    uint32_t cur_b = lo < hi ? ((uint32_t)(e[lo] >> 32) & 0x7fffu) : 0u;
    int qh = 0, qn = 0;
    // every segment with an entry adds its oldest
    auto turn = [&]() {
        const bool has = qn > 0;
        const int at = qh * SEG_TPB;
        const uint32_t g = has ? qg[at] : 0u;
        Pt m = has ? qv[at] : Pt::infinity();
        uint32_t left = 0;
        if (__reduce_max_sync(FULL, g) > 2)
            m = Pt::multiple(m, g);
        else
            left = g == 2;
        acc = Pt::add(acc, m, has);
        if (left) {
            qg[at] = left;
        } else if (has) {
            qh = (qh + 1) % SEG_QUEUE;
            qn--;
        }
    };
    for (int64_t i = 0; i < S; i++) {
        __syncthreads();
        const int64_t x = lo + i;
        const bool live = x < hi;
        const uint64_t en = live ? e[x] : 0;
        const uint32_t b = (uint32_t)(en >> 32) & 0x7fffu;
        const bool step = live && b != cur_b;
        while (__any_sync(FULL, step && qn == SEG_QUEUE)) turn();
        if (step) {
            const int at = (qh + qn) % SEG_QUEUE * SEG_TPB;
            qv[at] = run;
            qg[at] = cur_b - b;
            qn++;
            cur_b = b;
        }
        Fp px = fp_zero(), py = fp_zero();
        if (live) {
            const uint32_t t = (uint32_t)en;
            const uint8_t* pt = base + 2 * P::FIELD * (idx ? (int64_t)idx[t] : (int64_t)t);
            px = load_affine(Pt::at(pt, 0));
            py = load_affine(Pt::at(pt, 1));
            if (en >> 63) py = fp_neg(py);
        }
        run = Pt::madd(run, px, py, live);
        // segments without terms left never hold the warp back
        if (__all_sync(FULL, qn > 0 || x + 1 >= hi) && __any_sync(FULL, qn > 0)) turn();
    }
    acc = Pt::add(acc, Pt::multiple(run, cur_b), lo < hi);
    while (__any_sync(FULL, qn > 0)) turn();
    if (real) acc.store(seg_out + 4 * P::FIELD * out);
}

// out[row * out_len + i] = sum of in[row * len + G i .. G i + G - 1], G = 2, 4,
// .., 32: G lanes per output, a shuffle tree of log2 G additions (lanes past len
// hold the identity); every lane runs each level, so the warp never diverges
// around the shuffles.
template <class F>
__global__ void k_reduce(uint8_t* out, const uint8_t* in, int64_t rows, int64_t len, int64_t out_len, int G) {
    const int64_t gid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31, sub = lane & (G - 1);
    const int64_t o = gid / G, row = o / out_len, x = o % out_len * G + sub;
    Xyzz<F> acc;
    if (row < rows && x < len) {
        acc = load_vec(reinterpret_cast<const Xyzz<F>*>(in) + row * len + x);
    } else {
        set_inf(acc);
    }
    constexpr int WORDS = sizeof(Xyzz<F>) / 4;
    for (int off = G / 2; off > 0; off >>= 1) {
        Xyzz<F> other;
        uint32_t* dst = reinterpret_cast<uint32_t*>(&other);
        const uint32_t* src = reinterpret_cast<const uint32_t*>(&acc);
#pragma unroll
        for (int w = 0; w < WORDS; w++) dst[w] = __shfl_down_sync(0xffffffffu, src[w], off);
        if (sub + off >= G) set_inf(other);
        acc = xyzz_add(acc, other);
    }
    if (row < rows && sub == 0) store_vec(reinterpret_cast<Xyzz<F>*>(out) + o, acc);
}

struct ScratchLayout {
    size_t digits, entries, nnz, seg, red, total;
};
ScratchLayout layout_for(size_t xyzz, int32_t V, int64_t k, int64_t n, const MsmPlan& p) {
    auto align = [](size_t x) { return (x + 255) & ~size_t(255); };
    ScratchLayout L;
    size_t off = 0;
    L.digits = off;
    off += align(sizeof(int16_t) * (size_t)V * p.windows * n);
    L.entries = off;
    off += align(sizeof(uint64_t) * (size_t)V * p.windows * n);
    L.nnz = off;
    off += align(sizeof(int32_t) * (size_t)V * p.windows);
    L.seg = off;
    off += align(xyzz * (size_t)k * p.windows * p.segments);
    L.red = off;
    size_t red_len = (size_t)((p.segments + 7) / 8);
    off += align(xyzz * (size_t)k * p.windows * (red_len > 1 ? red_len : 1));
    L.total = off;
    return L;
}

template <class F>
void run_family(uint8_t* out, const uint8_t* points, const int64_t* pbase, const int32_t* idx, const uint8_t* scalars,
                const int32_t* vsel, int32_t V, int64_t k, int64_t n, const MsmPlan& p, uint8_t* scratch, cudaStream_t s) {
    const size_t XZ = sizeof(Xyzz<F>);
    ScratchLayout L = layout_for(XZ, V, k, n, p);
    int16_t* digits = reinterpret_cast<int16_t*>(scratch + L.digits);
    uint64_t* entries = reinterpret_cast<uint64_t*>(scratch + L.entries);
    int32_t* nnz = reinterpret_cast<int32_t*>(scratch + L.nnz);
    uint8_t* seg = scratch + L.seg;
    uint8_t* red = scratch + L.red;
    int64_t total = (int64_t)V * n;
    const bool g1 = sizeof(F) == sizeof(Fp);
    void* tok = nullptr;
    prof_begin(g1 ? "msm_sort_g1" : "msm_sort_g2", s, &tok);
    note_launch();
    k_digits<<<blocks_for(total), TPB, 0, s>>>(digits, scalars, total, n, p.c, p.windows);
    const int top = p.windows * p.c == 256 ? 2 * p.buckets : p.buckets;
    size_t shmem = sizeof(int32_t) * 2 * (top + 1);
    note_launch();
    k_sort<<<(unsigned)((int64_t)V * p.windows), 256, shmem, s>>>(entries, nnz, digits, n, p.buckets, top, p.windows);
    prof_end(tok, s);
    prof_begin(g1 ? "msm_segments_g1" : "msm_segments_g2", s, &tok);
    int64_t segthreads = k * p.windows * p.segments;
    note_launch();
    // the queues take about 49 KB of shared memory per block, past the 48 KB
    // default, so the kernel opts in once
    using P = typename std::conditional<sizeof(F) == sizeof(Fp), OnLane, OnPair>::type;
    static const bool smem_ok =
        cudaFuncSetAttribute(k_segments<P>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SEG_SMEM) == cudaSuccess;
    (void)smem_ok;
    k_segments<P><<<blocks_for(segthreads * P::LANES, SEG_TPB), SEG_TPB, SEG_SMEM, s>>>(
        seg, points, pbase, idx, entries, nnz, vsel, k, n, p.windows, p.segment, p.segments);
    prof_end(tok, s);
    prof_begin(g1 ? "msm_reduce_g1" : "msm_reduce_g2", s, &tok);
    // tree-reduce segments per (MSM, window)
    int64_t rows = k * p.windows, len = p.segments;
    uint8_t* src = seg;
    uint8_t* bufs[2] = {red, seg};
    int flip = 0;
    while (len > 1) {
        int G = 2;
        while (G < 32 && G < len) G *= 2;
        const int64_t out_len = (len + G - 1) / G;
        uint8_t* dst = bufs[flip];
        note_launch();
        k_reduce<F><<<blocks_for(rows * out_len * G, 64), 64, 0, s>>>(dst, src, rows, len, out_len, G);
        src = dst;
        flip ^= 1;
        len = out_len;
    }
    launch_msm_combine(g1 ? GROUP_G1 : GROUP_G2, out, src, k, p.windows, p.c, s);
    prof_end(tok, s);
}
}  // namespace

// Segments of k_segments resident on the whole device (one wave), from the
// occupancy of the compiled kernel; cached per device and group.
template <class P> static int64_t segment_wave() {
    static std::atomic<int64_t> cache[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148 * 256 / P::LANES;
    int64_t v = cache[dev].load();
    if (v > 0) return v;
    int sms = 0, blocks = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaFuncSetAttribute(k_segments<P>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SEG_SMEM);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, k_segments<P>, SEG_TPB, SEG_SMEM);
    v = (int64_t)(sms > 0 ? sms : 148) * (blocks > 0 ? blocks : 4) * SEG_TPB / P::LANES;
    cache[dev].store(v);
    return v;
}

// Window width and segments per (MSM, window) from a cost model in mixed
// additions.  Every segment's lanes walk S sorted terms, so the launch takes
// ceil(segments / wave) waves of S terms, an addition (1.43) per bucket that a
// segment of terms spread evenly over the buckets meets, and, where a row has
// several segments, the last bucket's multiple (a doubling and an addition per
// bit) and a tree of additions; the sort's count of buckets takes one thread, the
// tail adds the windows' sums in one chain (0.53 each; the doublings do not
// depend on c).  Narrow windows make few
// buckets and short multiples, wide ones few rows.  Measured on B200, one G1
// MSM of 65,536 points: c = 8 2.58 ms, 10 2.60, 13 (the former log2(n) - 2,
// capped) 2.79; of 32 points c = 8 1.30, 4 1.40.
// `limit`: plans whose scratch is larger are left out; none left, c = 0.
MsmPlan msm_plan(Group g, int64_t n, int64_t k, size_t limit) {
    const double wave = (double)(g == GROUP_G1 ? segment_wave<OnLane>() : segment_wave<OnPair>());
    int c0 = 4, c1 = 13;
    if (g_tune.msm_window >= c0 && g_tune.msm_window <= c1) c0 = c1 = g_tune.msm_window;
    const int64_t forced = g_tune.msm_segments > 0 ? std::min<int64_t>(std::min<int64_t>(g_tune.msm_segments, 1024), n) : 0;
    const int64_t most = std::min<int64_t>(1024, n);
    MsmPlan best;
    double best_cost = 0;
    for (int c = c0; c <= c1; c++) {
        const int windows = (256 + c - 1) / c;
        const double buckets = (double)(1 << (c - 1)), rows = (double)(k * windows);
        const double terms = (double)n * (1.0 - 1.0 / (2.0 * buckets));
        auto consider = [&](int64_t s) {
            s = forced ? forced : std::max<int64_t>(1, std::min(s, most));
            const double S = std::ceil(terms / (double)s);
            // buckets without terms leave gaps of several between those with
            const double gap = 2.3 * std::max(0.0, std::log2(buckets / (double)n));
            const double met = std::min(std::min(S, buckets), S * buckets / (double)n + 1.0);
            double each = S + met * (1.43 + gap) + (s > 1 ? 2.3 * (c - 1) : 0.0), tree = buckets / 900;
            if (s > 1) {
                for (double len = (double)s; len > 1; len = std::ceil(len / 32)) tree += 1.43 * std::min(5.0, std::ceil(std::log2(len)));
            }
            const double cost = std::ceil(rows * (double)s / wave) * each + tree + 0.53 * windows;
            if (best.c != 0 && cost >= best_cost) return;
            MsmPlan p;
            p.c = c;
            p.windows = windows;
            p.buckets = 1 << (c - 1);
            p.segment = (n + s - 1) / s;
            p.segments = std::max<int64_t>(1, (n + p.segment - 1) / p.segment);
            if (limit != SIZE_MAX && msm_family_scratch_bytes(g, 1, k, n, p) > limit) return;
            best_cost = cost;
            best = p;
        };
        // counts an eighth apart, and those that just fill whole waves
        for (int64_t s = 1; s <= most; s += 1 + s / 8) consider(s);
        for (int w = 1; w <= 4; w++) consider((int64_t)(wave * w / rows));
    }
    return best;
}

size_t msm_family_scratch_bytes(Group g, int32_t V, int64_t k, int64_t n, const MsmPlan& plan) {
    return layout_for(g == GROUP_G1 ? G1_XYZZ : G2_XYZZ, V, k, n, plan).total;
}

void launch_msm_family_scratch(Group g, uint8_t* out, const uint8_t* points, const int64_t* pbase, const int32_t* idx,
                               const uint8_t* scalars, const int32_t* vsel, int32_t V, int64_t k, int64_t n,
                               const MsmPlan& plan, void* scratch, cudaStream_t s) {
    if (k <= 0) return;
    if (g == GROUP_G1)
        run_family<Fp>(out, points, pbase, idx, scalars, vsel, V, k, n, plan, (uint8_t*)scratch, s);
    else
        run_family<Fp2>(out, points, pbase, idx, scalars, vsel, V, k, n, plan, (uint8_t*)scratch, s);
}

void launch_msm_family(Group g, uint8_t* out, const uint8_t* points, const int64_t* pbase, const int32_t* idx,
                       const uint8_t* scalars, const int32_t* vsel, int32_t V, int64_t k, int64_t n, cudaStream_t s,
                       const MsmPlan* forced) {
    if (k <= 0) return;
    if (n <= 0) {
        cudaMemsetAsync(out, 0, (g == GROUP_G1 ? G1_AFF : G2_AFF) * (size_t)k, s);
        return;
    }
    if (!forced && n <= SMALL_MSM_MAX) {
        launch_small_msm(g, out, points, pbase, idx, scalars, vsel, k, n, s);
        return;
    }
    MsmPlan p = forced ? *forced : msm_plan(g, n, k);
    size_t bytes = msm_family_scratch_bytes(g, V, k, n, p);
    void* scratch = nullptr;
    if (cudaMallocAsync(&scratch, bytes, s) != cudaSuccess) return;
    launch_msm_family_scratch(g, out, points, pbase, idx, scalars, vsel, V, k, n, p, scratch, s);
    cudaFreeAsync(scratch, s);
}

}  // namespace wbte

// ===================================================================
// Allocation-free G1 MSM.
//
// Some callers must not allocate device memory while they serve a request:
// a service that has reserved HBM up front for its resident key material
// and its request buffers cannot let the library take more, because an
// allocation can fail under memory pressure in the middle of a request,
// can stall on device-wide synchronisation, and fragments a carefully
// partitioned device.  For them, wbte_g1_msm_static runs the same Pippenger
// kernels as wbte_g1_msm but takes its working memory from one fixed array
// that is part of the library's device image (every GPU that loads the
// library holds it until the process exits).
namespace {
constexpr size_t STATIC_MSM_BYTES = size_t(8) << 20;        // 8 MiB of scratch
constexpr size_t STATIC_MSM_TAIL = 256;                     // holds the point-base entry
constexpr uint64_t STATIC_MSM_MAX_POINTS = 16384;
static __device__ __align__(256) uint8_t g_static_msm_scratch[STATIC_MSM_BYTES];

std::mutex g_static_mu;
uint8_t* g_static_addr[128] = {};

// Plain device memory of device `dev` only: host, managed and other GPUs'
// memory are rejected (a peer pointer would be read over the interconnect).
bool static_is_device(const void* p, int dev) {
    cudaPointerAttributes a;
    if (!p || cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeDevice && a.device == dev;
}

// The best plan whose scratch fits the array.  One exists for every n <=
// STATIC_MSM_MAX_POINTS: the widest windows take 10 bytes a point and window for
// digits and sorted entries (3.3 MB for 16,384 points), and one segment a window is
// 0.4 KB with its place in the tree.  Measured on B200 against the general plan with
// its segments cut until they fit: 16,384 points 1.69 -> 1.58 ms, 12,000 1.61 -> 1.58,
// 4,096 1.40 -> 1.42, fewer the same plan.
constexpr size_t STATIC_MSM_LEAST = (sizeof(int16_t) + sizeof(uint64_t)) * 20 * STATIC_MSM_MAX_POINTS + (size_t(1) << 16);
static_assert(STATIC_MSM_LEAST <= STATIC_MSM_BYTES - STATIC_MSM_TAIL, "windows of 13 bits fit");
bool static_plan(wbte::MsmPlan& p, int64_t n, size_t avail) {
    using namespace wbte;
    const Tuning saved = g_tune;
    g_tune = Tuning();
    p = msm_plan(GROUP_G1, n, 1, avail);
    g_tune = saved;
    return p.c != 0;
}
}  // namespace

extern "C" int32_t wbte_g1_msm_static(void* out, const void* points, const void* scalars, uint64_t n, void* stream) {
    using namespace wbte;
    if (n > STATIC_MSM_MAX_POINTS) return -2;  // WBTE_ERR_SIZE
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 128) return -5;  // WBTE_ERR_CUDA
    if (!static_is_device(out, dev) || (n > 0 && (!static_is_device(points, dev) || !static_is_device(scalars, dev))))
        return -1;  // WBTE_ERR_INVALID_ARG: device pointers of the current device only
    cudaStream_t s = (cudaStream_t)stream;
    // an error left pending by earlier, unrelated runtime calls on this
    // thread must not be reported as this call's failure
    cudaGetLastError();
    uint8_t* base = nullptr;
    {
        // one-time set-up per device, with that device current
        std::lock_guard<std::mutex> lock(g_static_mu);
        if (!g_static_addr[dev]) {
            void* ptr = nullptr;
            if (cudaGetSymbolAddress(&ptr, g_static_msm_scratch) != cudaSuccess) {
                cudaGetLastError();
                return -5;
            }
            g_static_addr[dev] = static_cast<uint8_t*>(ptr);
        }
        base = g_static_addr[dev];
    }
    if (n == 0) return cudaMemsetAsync(out, 0, G1_AFF, s) == cudaSuccess ? 0 : -5;
    MsmPlan p;
    if (!static_plan(p, (int64_t)n, STATIC_MSM_BYTES - STATIC_MSM_TAIL)) return -2;
    // point base of the single MSM: zero (the tail of the array is reused by
    // every call, so it is cleared here; nothing else must start at zero)
    int64_t* pbase = reinterpret_cast<int64_t*>(base + STATIC_MSM_BYTES - STATIC_MSM_TAIL);
    if (cudaMemsetAsync(pbase, 0, sizeof(int64_t), s) != cudaSuccess) return -5;
    // the opt-in per-kernel profiler would create CUDA events; keep it out of this call
    g_prof_suppress = true;
    launch_msm_family_scratch(GROUP_G1, static_cast<uint8_t*>(out), static_cast<const uint8_t*>(points), pbase,
                              nullptr, static_cast<const uint8_t*>(scalars), nullptr, 1, 1, (int64_t)n, p, base, s);
    g_prof_suppress = false;
    return cudaGetLastError() == cudaSuccess ? 0 : -5;
}
