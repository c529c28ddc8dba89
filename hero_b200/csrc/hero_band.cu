// hero_band.cu -- kernels of the window DP (hero_band.cuh): which segments take
// it, their order, the fill and traceback.  What it cannot certify goes to the
// whole-matrix kernels of hero_kernels.cu.
#include <cuda_runtime.h>

#include <algorithm>

#include "hero_band.cuh"
#include "hero_internal.cuh"

namespace hero {

namespace {

__device__ __forceinline__ uint32_t lane_id() { return threadIdx.x & 31u; }

// segment as the window reads it; R and C of the longer and shorter side
__device__ __forceinline__ BandSeg band_seg(const DpLaunch &a, const DpSeg &g, bool &reversed) {
    const uint32_t orient = (g.flags >> kSegOrientShift) & 1u, qrc = (g.flags >> kSegQrcShift) & 1u;
    const int64_t so = int64_t(a.soff[g.subj]), qo = int64_t(a.qoff[g.query]);
    PackSeq s{a.spack, orient ? so + int64_t(a.slen[g.subj]) - 1 - g.s0 : so + g.s0, orient ? -1 : 1};
    PackSeq q{a.qpack, qo + g.q0, 1};
    if (qrc) q = PackSeq{a.qpack, int64_t(a.qoff[g.query + 1]) - 1 - g.q0, -1};
    const int32_t ls = g.s1 - g.s0, lq = g.q1 - g.q0;
    reversed = lq > ls;
    BandSeg b;
    b.row = reversed ? q : s;
    b.col = reversed ? s : q;
    b.R = reversed ? lq : ls;
    b.C = reversed ? ls : lq;
    b.base = 0;
    b.m = g.band > b.R - b.C ? g.band : b.R - b.C;  // the aligner widens its band (BandAligner.cpp:59-62)
    return b;
}

__device__ __forceinline__ int band_type(const DpSeg &g) {
    return (g.flags & DPF_RIGHT) ? BT_RIGHT : ((g.flags & DPF_LEFT) ? BT_LEFT : BT_NONE);
}

// Window classes, widest first: 0..3 whole-band segments, 4..5 segments whose
// band cuts the matrix.  A segment's mismatches on the main diagonal, e, bound
// its deficit by 5 e, so few mismatches need only a narrow window: the limits
// of 11, 19, 26 and 40 diagonals are 10, 16, 20 and 30 for the affine aligner, of
// 8 and 16 diagonals 19 and 35 for the global one.  From five on the cause is
// mostly a gap, whose own deficit is small: the widest certifies 83 % of them.
// (Windows of 8, 16, 24 and 40 took 31 ms where these take 28.6.)
constexpr int kBandMostMismatches = 5;
template <bool AFFINE, int CLS>
__host__ __device__ constexpr int band_width() {
    return AFFINE ? (CLS == 0 ? 40 : CLS == 1 ? 26 : CLS == 2 ? 19 : CLS == 3 ? 11 : CLS == 4 ? 24 : 16)
                  : (CLS == 0 || CLS == 4 || CLS == 5 ? 16 : 8);
}
__device__ __forceinline__ int band_class(bool affine, bool masked, int32_t e) {
    if (masked) return affine && e > 2 ? 4 : 5;
    if (affine) return e > 4 ? 0 : (e == 4 ? 1 : (e == 3 ? 2 : 3));
    return e > 3 ? 0 : 3;
}

// appends the lanes with `on` to the whole-matrix list and counts their shape
__device__ __forceinline__ void rest_append(const DpLaunch &a, bool on, uint32_t si, const DpSeg &g) {
    const uint32_t m = __ballot_sync(0xffffffffu, on);
    if (!m) return;
    const uint32_t lane = lane_id(), leader = uint32_t(__ffs(int(m))) - 1u;
    unsigned long long at = 0;
    if (lane == leader) at = atomicAdd(a.n_rest, (unsigned long long)__popc(m));
    at = __shfl_sync(0xffffffffu, at, int(leader));
    const uint32_t key = on ? shape_key(g) : 0xffffffffu;
    const uint32_t same = __match_any_sync(0xffffffffu, key);
    if (on) {
        a.rest[at + __popc(m & ((1u << lane) - 1u))] = si;
        if (lane == uint32_t(__ffs(int(same))) - 1u) atomicAdd(&a.bins[key], uint32_t(__popc(same)));
    }
}

// One thread a segment: its reference cells; segments without a mismatch on
// their main diagonal (deficit 0: nothing can equal it), and nearly all of those
// with one, are done here, the others are counted by window class, type and
// columns, or listed for the whole-matrix kernels.  Bound by the scattered reads
// of the packed bases and the op words written; it replaces the whole matrix for
// 61 % (150 bp, affine) to 85 % (100 bp) of the segments.
__global__ void __launch_bounds__(256) k_band_screen(DpLaunch a, BandWork w) {
    const uint32_t lane = lane_id();
    for (uint64_t b0 = (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) & ~uint64_t(31); b0 < a.nd;
         b0 += uint64_t(gridDim.x) * blockDim.x) {
        const uint64_t i = b0 + lane;
        const bool has = i < a.nd;
        DpSeg g{};
        uint32_t key = kBandNoKey;
        bool rest = false, done = false, reversed = false;
        int type = BT_NONE;
        int32_t f = 0, e = kBandMostMismatches, R = 0, C = 0;
        if (has) {
            g = a.segs[i];
            const BandSeg s = band_seg(a, g, reversed);
            R = s.R;
            C = s.C;
            if (a.cells) {
                const uint64_t cl = band_cells(R, C, s.m);
                a.cells[i] = uint32_t(cl > 0xffffffffull ? 0xffffffffull : cl);
            }
            type = band_type(g);
            const int32_t d = R - C;
            const bool masked = s.m < R, affine = a.affine != 0;
            // both ends anchored on different diagonals: the widest window must hold both
            const int32_t most_d = affine ? (masked ? 12 : 24) : 8;
            rest = !w.on || (g.flags & 3u) == 3u || C > kBandMaxC || (type == BT_NONE && d > most_d);
            if (!rest) {
                if (type != BT_NONE || d == 0)
                    e = main_mismatches(s.row, s.col, main_row(type, R, C), C, kBandMostMismatches, f);
                done = e == 0 || (e == 1 && (affine ? one_mismatch_straight<true>(s.row, s.col, type, R, C, f)
                                                    : one_mismatch_straight<false>(s.row, s.col, type, R, C, f)));
                if (!done) key = (uint32_t(band_class(affine, masked, e) * 3 + type) << kBandColBits) | uint32_t(kBandMaxC - C);
            }
        }
        // the segment's place among those of its key: counted now, placed by k_band_scatter
        const uint32_t same = __match_any_sync(0xffffffffu, key);
        const uint32_t leader = uint32_t(__ffs(int(same))) - 1u;
        uint32_t rank = 0;
        if (key != kBandNoKey && lane == leader) rank = atomicAdd(&w.count[key], uint32_t(__popc(same)));
        if (done) {
            DpSum sum;
            plain_ops(type, R, C, e, f, reversed ? uint32_t(OP_I) : uint32_t(OP_D), a.ops + i * a.stride, a.stride, sum);
            a.sums[i] = sum;
        }
        rank = __shfl_sync(0xffffffffu, rank, int(leader)) + __popc(same & ((1u << lane) - 1u));
        if (has && w.on) w.key[i] = make_uint2(key, rank);
        rest_append(a, rest, uint32_t(i), g);
    }
}

// One block: first position and first task (64 segments) of every non-empty
// bin, in key order -- the widest windows and longest segments first.
constexpr int kTaskSegs = 64;
__global__ void __launch_bounds__(1024) k_band_tasks(BandWork w) {
    __shared__ uint32_t tot[32][3];
    constexpr int per = (kBandBins + 1023) / 1024;
    const uint32_t lane = lane_id(), wid = threadIdx.x >> 5;
    uint32_t n = 0, t = 0, b = 0;  // segments, tasks, bins of this thread's keys
    for (int k = 0; k < per; k++) {
        const uint32_t key = threadIdx.x * per + k;
        const uint32_t c = key < kBandBins ? w.count[key] : 0u;
        n += c;
        t += (c + kTaskSegs - 1) / kTaskSegs;
        b += c != 0u;
    }
    uint32_t v[3] = {n, t, b}, ex[3];
#pragma unroll
    for (int q = 0; q < 3; q++) {
        uint32_t x = v[q];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (int(lane) >= o) x += y;
        }
        ex[q] = x - v[q];
        if (lane == 31) tot[wid][q] = x;
    }
    __syncthreads();
    uint32_t all[3] = {0, 0, 0};
    for (int k = 0; k < 32; k++)
#pragma unroll
        for (int q = 0; q < 3; q++) {
            if (k < int(wid)) ex[q] += tot[k][q];
            all[q] += tot[k][q];
        }
    for (int k = 0; k < per; k++) {
        const uint32_t key = threadIdx.x * per + k;
        const uint32_t c = key < kBandBins ? w.count[key] : 0u;
        if (!c) continue;
        w.start[key] = ex[0];
        w.bin[ex[2]] = BandBin{key, ex[1], ex[0], c};
        ex[0] += c;
        ex[1] += (c + kTaskSegs - 1) / kTaskSegs;
        ex[2]++;
    }
    if (threadIdx.x == 0) {
        w.head[0] = all[2];  // bins
        w.head[1] = all[1];  // tasks
        w.head[2] = 0;       // next task
        w.head[3] = 0;       // segments for the wide window
        w.head[4] = 0;       // next of its tasks
    }
}

__global__ void __launch_bounds__(256) k_band_scatter(uint64_t nd, BandWork w) {
    for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < nd; i += uint64_t(gridDim.x) * blockDim.x) {
        const uint2 k = w.key[i];
        if (k.x != kBandNoKey) w.order[w.start[k.x] + k.y] = uint32_t(i);
    }
}

// a warp's traceback codes in global memory: word k of column j, 32 lanes wide
template <int WORDS>
struct WarpStore {
    uint32_t *base, *p;
    __device__ __forceinline__ void column(int32_t j) { p = base + size_t(j - 1) * (WORDS * 32); }
    __device__ __forceinline__ void put(int k, uint32_t bits) { p[k * 32] = bits; }
};
template <int WORDS>
struct WarpCodes {
    const uint32_t *base;  // + lane of the segment
    uint32_t shift;        // 16 for the high halves
    __device__ __forceinline__ uint32_t get(int32_t j, int32_t k) const {
        return (base[(size_t(j - 1) * WORDS + k) * 32] >> shift) & 0xffffu;
    }
};

// One task: up to 64 segments of one class, type and column count, two a lane
// (positions lane and lane + 32).  Registers hold the window (M and IY of every
// diagonal, the row selectors): two cells take eight ALU instructions (affine: byte
// select, add, two add-max, 3-way max, two masks, the code word's add) or seven
// (global), and the move of a selector; a column touches memory only for its code words.
template <bool AFFINE, int NB, int TYPE, bool MASK>
__device__ __noinline__ void band_task(const DpLaunch &a, const BandWork &w, const uint32_t *order, uint32_t n,
                                       int32_t C, uint32_t *codes) {
    constexpr int WORDS = (NB + 7) / 8;
    const uint32_t lane = lane_id();
    BandSeg s[2];
    uint32_t si[2];
    bool rev[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const uint32_t k = lane + 32u * h;
        si[h] = order[k < n ? k : 0u];
        s[h] = band_seg(a, a.segs[si[h]], rev[h]);
        s[h].base = band_base<AFFINE, NB, TYPE>(s[h].R - s[h].C);
    }
    int32_t jp = -s[0].base > -s[1].base ? -s[0].base : -s[1].base;
    jp = __reduce_max_sync(0xffffffffu, jp);
    WarpStore<WORDS> st{codes + lane, codes + lane};
    BandEnd e[2];
    band_fill<AFFINE, NB, TYPE, MASK>(s[0], s[1], C, jp, st, e[0], e[1]);
    uint32_t walk[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const bool has = lane + 32u * h < n;
        const bool sure = has && C - e[h].v <= band_limit<AFFINE, TYPE>(s[h], NB);
        if (sure && e[h].straight) {
            DpSum sum;
            straight_ops(s[h].row, s[h].col, TYPE, s[h].R, C, rev[h] ? uint32_t(OP_I) : uint32_t(OP_D),
                         a.ops + uint64_t(si[h]) * a.stride, a.stride, sum);
            a.sums[si[h]] = sum;
        }
        walk[h] = __ballot_sync(0xffffffffu, sure && !e[h].straight);
        const bool wide = has && !sure && !MASK;  // whole bands only
        rest_append(a, has && !sure && !wide, si[h], a.segs[si[h]]);
        const uint32_t m = __ballot_sync(0xffffffffu, wide);
        if (m) {
            uint32_t at = 0;
            if (lane == 0) at = atomicAdd(&w.head[3], uint32_t(__popc(m)));
            at = __shfl_sync(0xffffffffu, at, 0);
            if (wide) w.again[at + __popc(m & ((1u << lane) - 1u))] = si[h];
        }
    }
    __syncwarp();  // the codes of every lane are written
    // the paths with gaps, one a lane: lane l traces the l-th of them
    const uint32_t nw0 = __popc(walk[0]), nw = nw0 + __popc(walk[1]);
    for (uint32_t r = lane; r < nw; r += 32u) {
        const int h = r >= nw0;
        const uint32_t at = __fns(h ? walk[1] : walk[0], 0, int(r - (h ? nw0 : 0u)) + 1);
        const uint32_t sj = order[at + 32u * h];
        bool reversed;
        const DpSeg g = a.segs[sj];
        BandSeg t = band_seg(a, g, reversed);
        t.base = band_base<AFFINE, NB, TYPE>(t.R - t.C);
        OpsPut put{a.ops + uint64_t(sj) * a.stride, int32_t(a.stride * 16u)};
        DpSum sum;
        const int32_t np = band_walk<AFFINE, NB, TYPE>(t, WarpCodes<WORDS>{codes + at, h ? 16u : 0u},
                                                       reversed ? uint32_t(OP_I) : uint32_t(OP_D),
                                                       reversed ? uint32_t(OP_D) : uint32_t(OP_I), put);
        ops_summary(put.w, a.stride * 16u - uint32_t(np), uint32_t(np), sum);
        a.sums[sj] = sum;
    }
    __syncwarp();
}

template <bool AFFINE, int CLS>
__device__ __forceinline__ void band_dispatch(int type, const DpLaunch &a, const BandWork &w, const uint32_t *order,
                                              uint32_t n, int32_t C, uint32_t *codes) {
    constexpr int NB = band_width<AFFINE, CLS>();
    constexpr bool MASK = CLS >= 4;
    if (type == BT_RIGHT) {
        band_task<AFFINE, NB, BT_RIGHT, MASK>(a, w, order, n, C, codes);
    } else if (type == BT_LEFT) {
        band_task<AFFINE, NB, BT_LEFT, MASK>(a, w, order, n, C, codes);
    } else {
        band_task<AFFINE, NB, BT_NONE, MASK>(a, w, order, n, C, codes);
    }
}

// Persistent warps fed by a queue of tasks.  Measured, DP stage of one
// correction before (every matrix whole) and with the window: 5 Mbp affine,
// 1.67 M x 150 bp, 109 M segments, 358 -> 42 ms; 1 Mbp global, 300 k x 100 bp,
// 7.3 -> 1.0 ms; 300 kbp affine with -i 2 (bands of a few diagonals), 80 k x
// 150 bp, 34.5 -> 1.5 ms.
constexpr int kBandWarps = 4, kBandBlocks = 3;  // 12 warps an SM: 168 registers hold the widest window

template <bool AFFINE>
__global__ void __launch_bounds__(kBandWarps * 32, kBandBlocks) k_band(DpLaunch a, BandWork w) {
    const uint32_t lane = lane_id();
    uint32_t *codes = w.codes + size_t(blockIdx.x * kBandWarps + (threadIdx.x >> 5)) * w.code_words;
    const uint32_t nbin = w.head[0], ntask = w.head[1];
    for (;;) {
        uint32_t q = 0;
        if (lane == 0) q = atomicAdd(&w.head[2], 1u);
        q = __shfl_sync(0xffffffffu, q, 0);
        if (q >= ntask) break;
        uint32_t lo = 0, hi = nbin;  // the last bin whose first task is at most q
        while (hi - lo > 1u) {
            const uint32_t mid = (lo + hi) >> 1;
            if (w.bin[mid].task <= q) lo = mid; else hi = mid;
        }
        const BandBin b = w.bin[lo];
        const uint32_t first = (q - b.task) * kTaskSegs;
        const uint32_t n = b.count - first < kTaskSegs ? b.count - first : kTaskSegs;
        const uint32_t *order = w.order + b.first + first;
        const int32_t C = kBandMaxC - int32_t(b.key & ((1u << kBandColBits) - 1u));
        const uint32_t ct = b.key >> kBandColBits;
        const int type = int(ct % 3u);
        switch (ct / 3u) {
            case 0: band_dispatch<AFFINE, 0>(type, a, w, order, n, C, codes); break;
            case 1: if (AFFINE) band_dispatch<AFFINE, AFFINE ? 1 : 0>(type, a, w, order, n, C, codes); break;
            case 2: if (AFFINE) band_dispatch<AFFINE, AFFINE ? 2 : 0>(type, a, w, order, n, C, codes); break;
            case 3: band_dispatch<AFFINE, 3>(type, a, w, order, n, C, codes); break;
            case 4: if (AFFINE) band_dispatch<AFFINE, AFFINE ? 4 : 5>(type, a, w, order, n, C, codes); break;
            default: band_dispatch<AFFINE, 5>(type, a, w, order, n, C, codes); break;
        }
    }
}

// The wide window of what the register windows left: a group of 8 lanes (64
// diagonals; or 16 and 136, see wide_lanes) a pair of segments, in list order
// (theirs: class, type, columns).  Bound by the chain down the strips, nine steps a
// strip; a thread a pair, strip after strip, was six times that chain and slower
// than whole matrices for all but large batches.  What it
// replaces -- the whole matrix -- took 31 of 33 ms on 300-600 bp reads, 8 of 38 ms
// on 75-250 bp ones and 0.38 ms on 4310 such reads: now 2.1, 4.6 and 0.32
// with what it leaves to them.
struct WideCodes {
    const uint32_t *p;  // + first lane of the group
    int32_t lanes;
    uint32_t shift;
    __device__ __forceinline__ uint32_t get(int32_t k, int32_t t) const {
        return (p[size_t(kWideLag * k + t) * 32 + (k & (lanes - 1))] >> shift) & 0xffffu;
    }
};

constexpr int kWideWarps = 4;
// 64 diagonals on 8 lanes do a pair's work with half the lanes, but leave more to
// whole matrices, a second chain; 136 on 16 leave almost nothing, which counts where
// a batch only waits for its longest chains.  DP of one batch, 8 / 16 lanes, ms:
//   global  250 bp  0.1 M segments 0.29 / 0.37, 0.4 M 0.48 / 0.56, 3.4 M 1.8 / 2.7
//           75-250  0.1 M 0.27 / 0.30, 3.3 M 1.07 / 1.27; 100 and 150 bp alike
//   affine  100 bp  0.1 M 0.21 / 0.23, 1 M 0.52 / 0.54, 2.9 M 0.76 / 0.82
//           150 bp  0.2 M 0.58 / 0.39, 1.1 M 1.15 / 0.99, 3.3 M 1.56 / 1.52, batches
//                   of 8.4 M 43 / 50 (13 of them)
//           200 bp  0.2 M 0.81 / 0.57, 1.2 M 1.56 / 1.58, 3.4 M 2.6 / 3.1
//           250 bp  0.2 M 0.95 / 0.67, 0.4 M 1.35 / 1.31, 0.6 M 1.61 / 1.71, 3.4 M 3.9 / 5.3
//           75-250  0.2 M 0.81 / 0.60, 0.8 M 1.54 / 1.26, 1.7 M 1.66 / 1.62, 3.3 M 2.2 / 2.4
// So 8 for the global aligner, and for the affine one where the longest matrix has
// hardly more columns than its window diagonals (100 bp: 61) or segments x columns
// squared, the cells left, pass 3e10: 2.4 M segments of 150 bp reads, 1.2 M of 200,
// 0.7 M of 250.  Past 256 columns 16: a matrix left takes panels (k_dp_long).
inline int wide_lanes(uint64_t nd, uint64_t columns, bool affine) {
    if (columns > 256) return 16;
    return !affine || columns <= 64 || nd * columns * columns >= 30000000000ull ? 8 : 16;
}

template <bool AFFINE, int LANES>
__global__ void __launch_bounds__(kWideWarps * 32) k_band_wide(DpLaunch a, BandWork w) {
    constexpr int NB = wide_diagonals(LANES), ROWS = wide_rows(NB);
    constexpr uint32_t SEGS = 64 / LANES;  // segments a task
    const uint32_t lane = lane_id(), gl = lane % LANES, gbase = lane - gl;
    uint32_t *codes = w.codes + size_t(blockIdx.x * kWideWarps + (threadIdx.x >> 5)) * w.wide_words;
    const uint32_t count = w.head[3];
    for (;;) {
        uint32_t q = 0;
        if (lane == 0) q = atomicAdd(&w.head[4], 1u);
        q = __shfl_sync(0xffffffffu, q, 0);
        if (q >= (count + SEGS - 1) / SEGS) break;
        const uint32_t *list = w.again + size_t(q) * SEGS;
        const uint32_t n = min(count - q * SEGS, SEGS);
        BandSeg s[2];
        uint32_t si[2];
        int type[2];
        bool rev[2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const uint32_t k = 2u * (lane / LANES) + uint32_t(h);
            si[h] = list[k < n ? k : 0u];
            const DpSeg g = a.segs[si[h]];
            s[h] = band_seg(a, g, rev[h]);
            type[h] = band_type(g);
            s[h].base = wide_base(AFFINE, NB, type[h], s[h].R - s[h].C);
        }
        const int32_t strips = (max(s[0].C, s[1].C) + kWideStrip - 1) / kWideStrip;
        const int32_t most = __reduce_max_sync(0xffffffffu, strips);
        const int32_t steps = kWideLag * (most - 1) + ROWS;
        WideLane<AFFINE, LANES> x{int(gl)};
        const int src = int(gbase + (gl + LANES - 1) % LANES);
        uint32_t *out = codes + lane;
#pragma unroll 1
        for (int32_t t = 0; t < steps; t++, out += 32) {
            const uint32_t in_m = __shfl_sync(0xffffffffu, x.out_m, src);
            const uint32_t in_y = AFFINE ? __shfl_sync(0xffffffffu, x.out_y, src) : 0u;
            const int32_t u = t - kWideLag * x.k;
            const bool on = u >= 0 && u < ROWS && x.k < strips;
            if (on && u == 0) x.begin(s[0], s[1], type[0], type[1]);
            if ((t & 15) == 0 && on) x.refill(s[0], s[1]);
            const bool any_ends = __any_sync(0xffffffffu, on && x.ends);
            if (on) *out = x.row(s[0], s[1], type[0], type[1], in_m, in_y, any_ends);
            if (u == ROWS) x.k += LANES;
            x.last_m = in_m;
        }
        int32_t v[2];
        v[0] = __shfl_sync(0xffffffffu, x.va, int(gbase) + ((s[0].C - 1) / kWideStrip) % LANES);
        v[1] = __shfl_sync(0xffffffffu, x.vb, int(gbase) + ((s[1].C - 1) / kWideStrip) % LANES);
        __syncwarp();  // the codes of every lane are written
        // lanes 0 and 1 of a group trace its two segments
        const int h = int(gl & 1u);
        const BandSeg sh = h ? s[1] : s[0];
        const int th = h ? type[1] : type[0];
        const uint32_t sih = h ? si[1] : si[0];
        const bool has = gl < 2u && 2u * (lane / LANES) + uint32_t(h) < n;
        const bool sure = has && sh.C - (h ? v[1] : v[0]) <= wide_limit<AFFINE>(sh, th, NB);
        if (sure) {
            const bool reversed = h ? rev[1] : rev[0];
            OpsPut put{a.ops + uint64_t(sih) * a.stride, int32_t(a.stride * 16u)};
            DpSum sum;
            const int32_t np = wide_walk<AFFINE>(sh, th, NB, WideCodes{codes + gbase, LANES, h ? 16u : 0u},
                                                 reversed ? uint32_t(OP_I) : uint32_t(OP_D),
                                                 reversed ? uint32_t(OP_D) : uint32_t(OP_I), put);
            ops_summary(put.w, a.stride * 16u - uint32_t(np), uint32_t(np), sum);
            a.sums[sih] = sum;
        }
        rest_append(a, has && !sure, sih, a.segs[sih]);
        __syncwarp();
    }
}

template <bool AFFINE>
void wide_launch(const DpLaunch &a, const BandWork &w, cudaStream_t st) {
    const unsigned g = unsigned(w.wide_blocks);
    if (w.wide_lanes == 8) {
        k_band_wide<AFFINE, 8><<<g, kWideWarps * 32, 0, st>>>(a, w);
    } else {
        k_band_wide<AFFINE, 16><<<g, kWideWarps * 32, 0, st>>>(a, w);
    }
}

}  // namespace

// Warps of the window kernels and the code words of each -- and, in the same words,
// the wide window's blocks, whose warps need others.  A job of a few hundred
// thousand segments is over in a few tasks a warp: more warps then only spread the
// codes (135 KB a warp at 250 bp, affine) past the L2, and a new context pays 0.65
// ms for every 100 MB of them.  So a warp for every 32 segments up to 400 warps,
// then for every 500 (affine; 256 for the global aligner, whose codes take 2/5) up
// to the resident ones.  DP in ms with a warp for every 32 segments (as it was),
// 256 and 600:
//   affine  75-250 bp  0.2 M segments 0.80 0.60 0.54, 0.4 M 0.98 0.88 0.67, 1.3 M 1.60 1.60 1.64
//           250 bp     0.2 M 0.91 0.69 0.79, 0.4 M 1.31 1.33 1.03
//   global  250 bp     0.2 M 0.51 0.37 0.38, 0.4 M 0.57 0.48 0.47
//           300-600    0.4 M - 1.14 1.38
// (400 warps or more in each; on 23 k segments 200, 400 and 800 warps: 0.44 0.33
// 0.39).  On 0.2 M segments of 75-250 bp reads the codes were 300 MB and are 71
// now; a new context's first pass 4.3 -> 2.6 ms (whole matrices: 3.8).
size_t band_sizes(int device, uint64_t nd, int32_t cmax, bool affine, BandWork &w) {
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    const uint32_t c = uint32_t(cmax < kBandMaxC ? cmax : kBandMaxC);
    const uint64_t full = uint64_t(sms) * kBandBlocks, few = 400;
    w.code_words = c * 32u * (affine ? 5u : 2u);
    w.wide_lanes = wide_lanes(nd, c, affine);
    w.wide_words = uint32_t(kWideLag * ((c + kWideStrip - 1) / kWideStrip - 1) + wide_rows(wide_diagonals(w.wide_lanes))) * 32u;
    const uint64_t block = uint64_t(w.wide_words) * kWideWarps;
    const uint64_t warps = std::max(nd / (affine ? 500 : 256), std::min((nd + 31) / 32, few));
    w.warps = kBandWarps * std::min((warps + kBandWarps - 1) / kBandWarps, full);
    const uint64_t words = std::max<uint64_t>(w.warps * w.code_words, block);
    w.wide_blocks = std::min<uint64_t>(words / block, full);
    return words * 4;
}

void launch_band(const DpLaunch &a, const BandWork &w, cudaStream_t st) {
    if (!a.nd) return;
    const uint64_t g = (a.nd + 255) / 256;
    const unsigned grid = unsigned(g < 148u * 64u ? g : 148u * 64u);
    count_launch();
    k_band_screen<<<grid, 256, 0, st>>>(a, w);
    if (!w.on) return;
    count_launch();
    k_band_tasks<<<1, 1024, 0, st>>>(w);
    count_launch();
    k_band_scatter<<<grid, 256, 0, st>>>(a.nd, w);
    count_launch();
    const unsigned blocks = unsigned(w.warps / kBandWarps);
    if (a.affine) {
        k_band<true><<<blocks, kBandWarps * 32, 0, st>>>(a, w);
    } else {
        k_band<false><<<blocks, kBandWarps * 32, 0, st>>>(a, w);
    }
    count_launch();
    if (a.affine) {
        wide_launch<true>(a, w, st);
    } else {
        wide_launch<false>(a, w, st);
    }
}

}  // namespace hero
