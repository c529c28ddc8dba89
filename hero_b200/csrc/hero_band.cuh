// hero_band.cuh -- banded DP of a segment inside a window of diagonals, with a
// certificate that the window's path is the whole matrix's path.
//
// Segments join two reads at a shared k-mer, so the true path almost always
// runs a few diagonals from the main one.  The window DP computes NB adjacent
// diagonals only.  Let a path's deficit at column j be j minus its score: a
// match adds nothing, a mismatch 5, a base skipped on the columns 5 (2 in an
// extension), one skipped on the rows 4 (1 in an extension; none in column 0
// of an align-right or column C of an align-left segment).  Deficits never
// fall along a path, and never rise along the traceback (every move leads to a
// cell whose best deficit is no larger), so every cell of the traceback has at
// most the deficit D of the end cell.  A path that leaves the window pays for
// the diagonals it crosses; band_limit() gives the largest D that is below
// every such path's deficit at every cell the traceback can visit.  If the
// window's own D is within the limit, no path outside the window can equal or
// beat the values the traceback reads, so the moves -- ties included -- are the
// whole matrix's.  Segments that miss the limit are computed in full.
//
// Two segments run in the 16-bit halves of each register, as dp_pair_row does.
// Values are 4 (v + potential) + tag (tags as in dp_pair_row).  The potential
// grows with the row and the column so that a gap extension costs nothing:
// each of the two gap states is then one add-max a cell.
#pragma once
#include "hero_core.cuh"

namespace hero {

enum : int { BT_NONE = 0, BT_RIGHT = 1, BT_LEFT = 2 };  // anchored at both ends, at the end, at the start

constexpr int32_t kBandMaxC = 1023;   // columns of a window segment: 16-bit values hold 4 * 5 * C
// Start of what lies outside the matrix or the aligner's band.  Such a cell may
// match on along its diagonal, where a value rises as the potential does, so a
// path through it keeps a deficit of at least 3000 at every column: the
// certificate takes no larger one, whatever the window holds.
constexpr int32_t kBandDead = -12000;
constexpr int32_t kBandMostDeficit = -kBandDead / 4 - 1;
constexpr int kPackPad = 8;           // words (128 bases) before and after packed reads that fetches may touch

// ---------------------------------------------------------------------------
// packed reads: 2 bits a base, base g of the read array at bits 2 (g % 16) of
// word g / 16
// ---------------------------------------------------------------------------
struct PackSeq {          // a stretch of a read, oriented: base t is at + dir * t, complemented when dir < 0
    const uint32_t *w;
    int64_t at;
    int32_t dir;
};

HERO_HD uint32_t reverse_fields(uint32_t x) {  // the sixteen 2-bit fields in reverse order
#if defined(__CUDA_ARCH__)
    x = __brev(x);
    return ((x >> 1) & 0x55555555u) | ((x & 0x55555555u) << 1);
#else
    uint32_t r = 0;
    for (int i = 0; i < 16; i++) r |= ((x >> (2 * i)) & 3u) << (2 * (15 - i));
    return r;
#endif
}

// bases t .. t + 15, base t in the lowest bits
HERO_HD uint32_t pack16(const PackSeq &s, int32_t t) {
    const int64_t p = s.dir > 0 ? s.at + t : s.at - t - 15;
    const int64_t k = p >> 4;
    const uint32_t sh = uint32_t(p & 15) * 2u;
    const uint32_t lo = s.w[k], hi = s.w[k + 1];
#if defined(__CUDA_ARCH__)
    const uint32_t x = __funnelshift_r(lo, hi, sh);
#else
    const uint32_t x = uint32_t(((uint64_t(hi) << 32) | lo) >> sh);
#endif
    return s.dir > 0 ? x : reverse_fields(x) ^ 0xaaaaaaaau;
}

// pack16 at t0, t0 + 16, ... of a stretch, one word loaded a call
struct PackStream {
    const uint32_t *p;
    uint32_t cur, sh;
    int32_t step;
    HERO_HD PackStream(const PackSeq &s, int32_t t0) {
        const int64_t at = s.dir > 0 ? s.at + t0 : s.at - t0 - 15;
        const uint32_t *w = s.w + (at >> 4);
        step = s.dir;
        sh = uint32_t(at & 15) * 2u;
        cur = w[step > 0 ? 0 : 1];
        p = w + (step > 0 ? 1 : 0);
    }
    HERO_HD uint32_t next() {
        const uint32_t n = *p, lo = step > 0 ? cur : n, hi = step > 0 ? n : cur;
        p += step;
        cur = n;
#if defined(__CUDA_ARCH__)
        const uint32_t x = __funnelshift_r(lo, hi, sh);
#else
        const uint32_t x = uint32_t(((uint64_t(hi) << 32) | lo) >> sh);
#endif
        return step > 0 ? x : reverse_fields(x) ^ 0xaaaaaaaau;
    }
};

// 01 in every field where two packed words differ: OP_X there, OP_M elsewhere
HERO_HD uint32_t mismatch16(uint32_t a, uint32_t b) {
    const uint32_t x = a ^ b;
    return (x | (x >> 1)) & 0x55555555u;
}

struct BandSeg {  // a segment as the window DP reads it (rows = longer side)
    PackSeq row, col;
    int32_t R, C;
    int32_t base;   // offset (row - column) of the window's first diagonal
    int32_t m;      // the aligner's band: cells with |row - column| > m do not exist
};

// window shape: the side on which leaving costs less a diagonal is the longer
template <bool AFFINE, int NB>
struct BandWin {
    static constexpr int near = AFFINE ? (NB - 1) / 3 : (NB - 1) / 2;
    static constexpr int far = NB - 1 - near;
};
// window position of the main diagonal (the one the anchored end lies on; both
// ends of a BT_NONE segment of equal sides)
template <bool AFFINE, int NB, int TYPE>
HERO_HD constexpr int band_main() {
    return TYPE == BT_RIGHT ? BandWin<AFFINE, NB>::far : TYPE == BT_LEFT ? BandWin<AFFINE, NB>::near : (NB - 1) / 2;
}
template <bool AFFINE, int NB, int TYPE>
HERO_HD int32_t band_base(int32_t d) {
    return TYPE == BT_RIGHT ? d - BandWin<AFFINE, NB>::far
         : TYPE == BT_LEFT ? -BandWin<AFFINE, NB>::near : -((NB - 1 - d) / 2);
}

// The largest end deficit at which no path through cells outside the window
// [base, base + NB) can match the values of the traceback.  Below the window a
// path has skipped columns (and must skip rows to return), or, aligned right,
// started on an earlier row of column 0 (and must skip rows to reach the end's
// diagonal); above it the reverse.  The affine column 0 and row 0 let a gap
// turn without a second opening cost, so only one opening is counted.  An
// align-left path may also reach column C outside the window: above it the
// moves there are still up while its deficit is no smaller than D (a tie goes
// up for the affine aligner, not for the global one), below it the free climb
// would carry its score to the cells of the traceback.  The limits are the
// deficits of those paths, less one where a tie would change a move, and at most
// what cells outside the aligner's band cannot reach (kBandMostDeficit), which
// alone counts where the window holds the whole band.
template <bool AFFINE, int TYPE>
HERO_HD int32_t band_limit(const BandSeg &s, int32_t nb) {
    const int32_t d = s.R - s.C, lo = s.base, hi = s.base + nb - 1;
    const int32_t v1 = AFFINE ? 1 : 4, h1 = AFFINE ? 2 : 5, open = AFFINE ? 3 : 0;
    int32_t below = kBandMostDeficit, above = kBandMostDeficit;
    if (lo > -s.m && lo > -s.C) {
        const int32_t h = lo > 0 ? 0 : 1 - lo;  // columns skipped to get below the window
        if (TYPE == BT_RIGHT) below = open + h * h1 + (d - lo + 1) * v1 - 1;
        if (TYPE == BT_LEFT) below = open + h * h1 - 1;
        if (TYPE == BT_NONE) below = open + h * h1 + (h + d) * v1 - 1;
    }
    if (hi < s.m && hi < s.R) {
        if (TYPE == BT_RIGHT) above = open + (hi - d + 1) * h1 - 1;
        if (TYPE == BT_LEFT) above = open + (hi + 1) * v1 + (hi < d ? (AFFINE ? 0 : -1) : h1 - 1);
        if (TYPE == BT_NONE) above = open + (hi + 1) * v1 + (hi + 1 - d) * h1 - 1;
    }
    const int32_t most = below < above ? below : above;
    return most < kBandMostDeficit ? most : kBandMostDeficit;
}

// byte select with sign replication, as PRMT: nibble n of sel picks byte n & 7
// of {a, b}, or its sign byte when bit 3 is set
HERO_HD uint32_t byte_sel(uint32_t a, uint32_t b, uint32_t sel) {
#if defined(__CUDA_ARCH__)
    uint32_t r;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
    return r;
#else
    const uint64_t ab = (uint64_t(b) << 32) | a;
    uint32_t r = 0;
    for (int i = 0; i < 4; i++) {
        const uint32_t n = (sel >> (4 * i)) & 15u;
        uint32_t v = uint32_t(ab >> (8 * (n & 7u))) & 0xffu;
        if (n & 8u) v = (v & 0x80u) ? 0xffu : 0u;
        r |= v << (8 * i);
    }
    return r;
#endif
}

HERO_HD uint32_t min_2(uint32_t a, uint32_t b) {  // per half, signed
#if defined(__CUDA_ARCH__)
    return __vmins2(a, b);
#else
    const int32_t l = half_lo(a) < half_lo(b) ? half_lo(a) : half_lo(b);
    const int32_t h = half_hi(a) < half_hi(b) ? half_hi(a) : half_hi(b);
    return pack2(l, h);
#endif
}

HERO_HD constexpr uint32_t band_half2(int32_t v) { return (uint32_t(v) & 0xffffu) * 0x10001u; }

// the costs in window values
template <bool AFFINE>
struct BandCost {
    using T = PairTags<AFFINE>;
    static constexpr int32_t pot = AFFINE ? 1 : 2;  // potential a row and a column
    static constexpr int32_t match = 4 * (kHIT + 2 * pot) + T::diag, miss = 4 * (kMISS + 2 * pot) + T::diag;
    // score bytes by the column's base: `miss` everywhere, `match` at byte `code`
    static constexpr uint32_t table = (uint32_t(miss) & 0xffu) * 0x01010101u;
    static constexpr uint32_t flip = (uint32_t(miss) ^ uint32_t(match)) & 0xffu;
    static constexpr uint32_t down = band_half2(AFFINE ? 4 * (kDX + pot) + T::up - T::diag : 4 * (kDX + pot) + T::up);
    static constexpr uint32_t right = band_half2(AFFINE ? 4 * (kDY + pot) + T::left - T::diag : 4 * (kDY + pot) + T::left);
    // column C of an align-left segment: rows there cost sx = 0
    static constexpr uint32_t free_open = band_half2(AFFINE ? 4 * (kSX + pot) + T::up - T::diag : 4 * (kSX + pot) + T::up);
    static constexpr uint32_t free_more = band_half2(4 * (kSX + pot));
};

struct BandEnd {
    int32_t v;      // score at (R, C)
    bool straight;  // the path is the main diagonal (and the free run of an anchored segment)
};

// selector of a row's two bases for byte_sel on the column's two score tables:
// the low half takes segment A's score byte, sign-extended, the high half B's
HERO_HD uint32_t band_sel(uint32_t a, uint32_t b) { return a * 0x11u + b * 0x1100u + 0xc480u; }

template <bool AFFINE>
HERO_HD uint32_t band_table(uint32_t code) { return BandCost<AFFINE>::table ^ (BandCost<AFFINE>::flip << (8u * code)); }

// M of column 0 at row i, and IY of (i, 1) (affine), as plain scores
template <bool AFFINE, int TYPE>
HERO_HD int32_t band_col0(int32_t i) {
    if (i == 0 || TYPE == BT_RIGHT) return 0;
    return AFFINE ? kDX - kEX + i * kEX : i * kDX;
}
template <int TYPE>
HERO_HD int32_t band_col0_right(int32_t i) {
    return (i == 0 || TYPE == BT_RIGHT) ? kDY : kDX - kEX + (i + 1) * kEX;
}

// One column of the window.  M: clean M of the column before, then of this one
// (global: F); L (affine): IY of this column's cell one diagonal below, then of
// the next column's.  sel[c]: the selector of cell c's row.  INJECT (affine):
// z{a,b} is the window position of row 0, whose IX equals its IY.  Codes (two
// bits a cell, eight cells a word) go to st.put(word, bits); the tags of the
// main diagonal are and-ed into `straight`.
template <bool AFFINE, int NB, int TYPE, bool MASK, bool INJECT, class Store>
HERO_HD void band_column(uint32_t (&M)[NB], uint32_t (&L)[AFFINE ? NB : 1], const uint32_t (&P)[MASK ? NB : 1],
                         const uint32_t (&sel)[NB], uint32_t ta, uint32_t tb, int32_t za, int32_t zb,
                         uint32_t &straight, Store &st) {
    using K = BandCost<AFFINE>;
    constexpr int main_c = band_main<AFFINE, NB, TYPE>();
    const uint32_t dead = band_half2(kBandDead);
    uint32_t x = dead, acc = 0;  // IX of the cell (affine), M of the cell above (global)
#pragma unroll
    for (int c = 0; c < NB; c++) {
        const uint32_t f = add2(M[c], byte_sel(ta, tb, sel[c]));
        uint32_t y = c + 1 < NB ? (AFFINE ? L[c + 1 < NB && AFFINE ? c + 1 : 0] : M[c + 1 < NB ? c + 1 : 0]) : dead;
        uint32_t mt;
        if (AFFINE) {
            if (MASK) {
                y = min_2(y, P[MASK ? c : 0]);
                x = min_2(x, P[MASK ? c : 0]);
            }
            if (INJECT) {
                const uint32_t on = (za == c ? 0xffffu : 0u) | (zb == c ? 0xffff0000u : 0u);
                x = (x & ~on) | ((y + 0x00020002u) & on);
            }
            mt = max3_2(f, x, y);
            L[AFFINE ? c : 0] = add_max2(f, K::right, y);
            x = add_max2(f, K::down, x);
        } else {
            if (MASK) {
                y = min_2(y, P[MASK ? c : 0]);
                x = min_2(x, P[MASK ? c : 0]);
            }
            mt = add_max2(y, K::right, add_max2(x, K::down, f));
        }
        const uint32_t tg = mt & kTagMask2;
        M[c] = mt & ~kTagMask2;
        if (!AFFINE) x = M[c];
        if (c == main_c) straight &= tg;
        acc += tg << (2 * (c & 7));
        if ((c & 7) == 7 || c == NB - 1) {
            st.put(c >> 3, acc);
            acc = 0;
        }
    }
}

// The window of two segments of the same type and columns (C).  jp: columns in
// which any segment of the warp has row 0 in its window (affine).  Store:
// column(j) before each column's puts.
template <bool AFFINE, int NB, int TYPE, bool MASK, class Store>
HERO_HD void band_fill(const BandSeg &a, const BandSeg &b, int32_t C, int32_t jp, Store &st, BandEnd &ea,
                       BandEnd &eb) {
    using K = BandCost<AFFINE>;
    using T = PairTags<AFFINE>;
    constexpr int main_c = band_main<AFFINE, NB, TYPE>();
    uint32_t M[NB], L[AFFINE ? NB : 1], P[MASK ? NB : 1], sel[NB];
    // column 0
#pragma unroll
    for (int c = 0; c < NB; c++) {
        const int32_t ia = a.base + c, ib = b.base + c;
        const bool oka = ia >= 0 && (!MASK || ia <= a.m), okb = ib >= 0 && (!MASK || ib <= b.m);
        M[c] = pack2(oka ? 4 * (band_col0<AFFINE, TYPE>(ia) + K::pot * c) : kBandDead,
                     okb ? 4 * (band_col0<AFFINE, TYPE>(ib) + K::pot * c) : kBandDead);
        if (AFFINE)
            L[AFFINE ? c : 0] = pack2(oka ? 4 * (band_col0_right<TYPE>(ia) + c + 1) : kBandDead,
                                      okb ? 4 * (band_col0_right<TYPE>(ib) + c + 1) : kBandDead);
        if (MASK)
            P[MASK ? c : 0] = pack2(ia >= -a.m && ia <= a.m ? 0x7fff : kBandDead,
                                    ib >= -b.m && ib <= b.m ? 0x7fff : kBandDead);
    }
    // selectors of rows 1 + base .. base + NB - 1 (the last NB-th row joins with each column)
#pragma unroll
    for (int c0 = 0; c0 < NB - 1; c0 += 16) {
        const uint32_t wa = pack16(a.row, a.base + c0), wb = pack16(b.row, b.base + c0);
#pragma unroll
        for (int c = 0; c < 16; c++)
            if (c0 + c < NB - 1) sel[c0 + c] = band_sel((wa >> (2 * c)) & 3u, (wb >> (2 * c)) & 3u);
    }
    uint32_t ra = 0, rb = 0, ca = 0, cb = 0, straight = 0xffffffffu;
    const int32_t last = TYPE == BT_LEFT ? C - 1 : C;  // column C of an align-left segment follows the loop
    // One column an iteration: the loop's code then stays near the instructions a
    // scheduler caches (four columns an iteration waited for instructions: 34 ms
    // of window kernels against 31 on the 1.67 M x 150 bp workload).
#pragma unroll 1
    for (int32_t j = 1; j <= last; j++) {
        if (((j - 1) & 15) == 0) {  // sixteen more rows and columns
            ra = pack16(a.row, a.base + NB - 2 + j);
            rb = pack16(b.row, b.base + NB - 2 + j);
            ca = pack16(a.col, j - 1);
            cb = pack16(b.col, j - 1);
        }
        sel[NB - 1] = band_sel(ra & 3u, rb & 3u);
        const uint32_t ta = band_table<AFFINE>(ca & 3u), tb = band_table<AFFINE>(cb & 3u);
        ra >>= 2;
        rb >>= 2;
        ca >>= 2;
        cb >>= 2;
        st.column(j);
        if (AFFINE && j <= jp) {
            band_column<AFFINE, NB, TYPE, MASK, true>(M, L, P, sel, ta, tb, -a.base - j, -b.base - j, straight, st);
        } else {
            band_column<AFFINE, NB, TYPE, MASK, false>(M, L, P, sel, ta, tb, 0, 0, straight, st);
        }
#pragma unroll
        for (int c = 0; c < NB - 1; c++) sel[c] = sel[c + 1];
    }
    const int32_t da = a.R - a.C, db = b.R - b.C;
    if (TYPE != BT_LEFT) {
        const int32_t cea = TYPE == BT_RIGHT ? main_c : da - a.base, ceb = TYPE == BT_RIGHT ? main_c : db - b.base;
        int32_t va = 0, vb = 0;
#pragma unroll
        for (int c = 0; c < NB; c++) {
            if (c == cea) va = (half_lo(M[c]) >> 2) - K::pot * (2 * C + c);
            if (c == ceb) vb = (half_hi(M[c]) >> 2) - K::pot * (2 * C + c);
        }
        const bool eqa = TYPE == BT_RIGHT || (da == 0 && cea == main_c), eqb = TYPE == BT_RIGHT || (db == 0 && ceb == main_c);
        ea = BandEnd{va, eqa && (straight & uint32_t(T::diag)) != 0u};
        eb = BandEnd{vb, eqb && (straight & (uint32_t(T::diag) << 16)) != 0u};
        return;
    }
    // column C of align-left segments: rows cost nothing there
    st.column(C);
    const uint32_t ta = band_table<AFFINE>(pack16(a.col, C - 1) & 3u), tb = band_table<AFFINE>(pack16(b.col, C - 1) & 3u);
    const uint32_t dead = band_half2(kBandDead);
    const int32_t cea = main_c + da < NB - 1 ? main_c + da : NB - 1, ceb = main_c + db < NB - 1 ? main_c + db : NB - 1;
    uint32_t x = dead, acc = 0, wa = 0, wb = 0;
    int32_t va = 0, vb = 0;
    bool sa = (straight & uint32_t(T::diag)) != 0u, sb = (straight & (uint32_t(T::diag) << 16)) != 0u;
#pragma unroll
    for (int c = 0; c < NB; c++) {
        if ((c & 15) == 0) {
            wa = pack16(a.row, C - 1 + a.base + c);
            wb = pack16(b.row, C - 1 + b.base + c);
        }
        const uint32_t f = add2(M[c], byte_sel(ta, tb, band_sel(wa & 3u, wb & 3u)));
        wa >>= 2;
        wb >>= 2;
        uint32_t y = c + 1 < NB ? (AFFINE ? L[c + 1 < NB && AFFINE ? c + 1 : 0] : M[c + 1 < NB ? c + 1 : 0]) : dead;
        if (MASK) {
            y = min_2(y, P[MASK ? c : 0]);
            x = min_2(x, P[MASK ? c : 0]);
        }
        uint32_t mt, fx;  // fx: the states a further row's free move reads
        if (AFFINE) {
            const uint32_t on = (C + a.base + c == 0 ? 0xffffu : 0u) | (C + b.base + c == 0 ? 0xffff0000u : 0u);
            x = (x & ~on) | ((y + 0x00020002u) & on);
            mt = max3_2(f, x, y);
            fx = max3_2(f, x, x);
            x = add_max2(f, K::free_open, add2(x, K::free_more));
        } else {
            mt = add_max2(y, K::right, add_max2(x, c == 0 ? K::down : K::free_open, f));
            fx = mt;
            x = mt & ~kTagMask2;
        }
        const uint32_t tg = mt & kTagMask2;
        const int32_t p = K::pot * (2 * C + c);
        if (c == cea) va = (half_lo(c == NB - 1 && main_c + da > c ? fx : mt) >> 2) - p;
        if (c == ceb) vb = (half_hi(c == NB - 1 && main_c + db > c ? fx : mt) >> 2) - p;
        if (c == main_c) {
            sa = sa && (tg & 3u) == uint32_t(T::diag);
            sb = sb && (tg >> 16) == uint32_t(T::diag);
        } else if (c > main_c) {
            sa = sa && (c > cea || (tg & 3u) == uint32_t(T::up));
            sb = sb && (c > ceb || (tg >> 16) == uint32_t(T::up));
        }
        acc += tg << (2 * (c & 7));
        if ((c & 7) == 7 || c == NB - 1) {
            st.put(c >> 3, acc);
            acc = 0;
        }
    }
    ea = BandEnd{va, sa};
    eb = BandEnd{vb, sb};
}

// Packed ops written last to first at descending positions.
struct OpsPut {
    uint32_t *w;
    int32_t p;  // position of the op put last
    uint32_t acc = 0;

    // k <= 16 ops: the low k fields of `bits`, the lowest first in path order
    HERO_HD void fields(uint32_t bits, uint32_t k) {
        const uint32_t room = uint32_t((p - 1) & 15) + 1u;  // fields left in the current word
        if (k < room) {
            acc |= bits << (2u * (room - k));
        } else {
            w[(p - 1) >> 4] = acc | (bits >> (2u * (k - room)));
            acc = k == room ? 0u : bits << (32u - 2u * (k - room));
        }
        p -= int32_t(k);
    }
    HERO_HD void run(uint32_t op, uint32_t k) {
        for (; k > 0;) {
            const uint32_t take = k < 16u ? k : 16u;
            fields(op * ops_mask(0, take - 1u), take);
            k -= take;
        }
    }
    HERO_HD void flush() {
        if (p & 15) w[p >> 4] = acc;
    }
};

// Traceback inside the window (dp_walk's moves; codes.get(column, word) holds
// eight cells of a segment).  Diagonal runs are found eight columns at a time:
// their codes are loaded together, since the cell's place in the window stays.
// gap_up / gap_left: the op of a row / column skipped.  Returns the ops put, or
// -1 if the path leaves the window (not reached within band_limit).
template <bool AFFINE, int NB, int TYPE, class Codes>
HERO_HD int32_t band_walk(const BandSeg &s, const Codes &codes, uint32_t gap_up, uint32_t gap_left, OpsPut &out) {
    using T = PairTags<AFFINE>;
    constexpr int32_t AHEAD = 8;
    const int32_t end = out.p;
    int32_t i = s.R, j = s.C, c = i - j - s.base;
    if (TYPE == BT_LEFT) {  // column C: the rows above the window, then its climb inside
        int32_t k = c > NB - 1 ? c - (NB - 1) : 0;
        while (c - k > 0 && ((codes.get(j, (c - k) >> 3) >> (2 * ((c - k) & 7))) & 3u) == uint32_t(T::up)) k++;
        if (k > i) k = i;
        out.run(gap_up, uint32_t(k));
        i -= k;
        c -= k;
    }
    while (i > 0 && j > 0) {
        if (uint32_t(c) >= uint32_t(NB)) return -1;
        const int32_t k = c >> 3, sh = 2 * (c & 7), n = i < j ? (i < AHEAD ? i : AHEAD) : (j < AHEAD ? j : AHEAD);
        uint32_t code[AHEAD];
#pragma unroll
        for (int t = 0; t < AHEAD; t++) code[t] = t < n ? (codes.get(j - t, k) >> sh) & 3u : 3u;
        int32_t run = 0;
        uint32_t stop = 3u;  // the code that ends the run (3: none in these columns)
#pragma unroll
        for (int t = AHEAD - 1; t >= 0; t--)
            if (code[t] != uint32_t(T::diag)) {
                run = t;
                stop = code[t];
            }
        if (stop == 3u) run = n;
        if (run > 0) {
            i -= run;
            j -= run;
            out.fields(mismatch16(pack16(s.row, i), pack16(s.col, j)) & ops_mask(0, uint32_t(run - 1)), uint32_t(run));
        }
        if (stop == uint32_t(T::up)) {
            out.fields(gap_up, 1u);
            i--;
            c--;
        } else if (stop == uint32_t(T::left)) {
            out.fields(gap_left, 1u);
            j--;
            c++;
        }
    }
    out.run(gap_up, uint32_t(i));
    out.run(gap_left, uint32_t(j));
    out.flush();
    return end - out.p;
}

// ---------------------------------------------------------------------------
// The wide window: for the segments whose deficit the register windows cannot
// certify.  Strips of eight columns, one lane a strip, in turn: a strip's row t
// is row first column + base + t, so cell (t, w) lies on window diagonal t - w,
// and rows 0 .. nb + 6 hold the window and some cells beside it, whose values are
// paths' all the same.  The strip before reaches a matrix row eight rows of its
// own later and started nine steps earlier, so a group of lanes, strip k on lane
// k mod lanes starting at step 9 k, passes each row's last M and next IY on by
// one shuffle a step, and a lane is free again when its next strip starts.  The
// two segments of a pair may differ in type and columns.
// ---------------------------------------------------------------------------
constexpr int kWideStrip = 8;
constexpr int kWideLag = kWideStrip + 1;  // steps between the starts of neighbouring strips
HERO_HD constexpr int wide_rows(int nb) { return nb + kWideStrip - 1; }
HERO_HD constexpr int wide_diagonals(int lanes) { return kWideLag * lanes - kWideStrip; }  // one step of rest a strip

HERO_HD int wide_near(bool affine, int nb) { return affine ? (nb - 1) / 3 : (nb - 1) / 2; }
HERO_HD int32_t wide_base(bool affine, int nb, int type, int32_t d) {
    const int near = wide_near(affine, nb);
    return type == BT_RIGHT ? d - (nb - 1 - near) : type == BT_LEFT ? -near : -((nb - 1 - d) / 2);
}

template <bool AFFINE>
HERO_HD int32_t wide_limit(const BandSeg &s, int type, int32_t nb) {
    return type == BT_RIGHT ? band_limit<AFFINE, BT_RIGHT>(s, nb)
         : type == BT_LEFT ? band_limit<AFFINE, BT_LEFT>(s, nb) : band_limit<AFFINE, BT_NONE>(s, nb);
}

// scores of column 0 at row i: M, and IY of (i, 1)
template <bool AFFINE>
HERO_HD int32_t wide_col0(int type, int32_t i) {
    return type == BT_RIGHT ? band_col0<AFFINE, BT_RIGHT>(i) : band_col0<AFFINE, BT_LEFT>(i);
}

// one row of a strip; ENDS: column C of a segment is in the strip (free: the
// halves of align-left ones, whose rows cost nothing there)
template <bool AFFINE, bool ENDS>
HERO_HD uint32_t wide_row(uint32_t (&m)[kWideStrip], uint32_t (&xn)[kWideStrip], const uint32_t (&sel)[kWideStrip],
                          uint32_t ta, uint32_t tb, uint32_t dm, uint32_t &y, const uint32_t (&free)[kWideStrip],
                          uint32_t (&mts)[kWideStrip], uint32_t (&fxs)[kWideStrip]) {
    using K = BandCost<AFFINE>;
    uint32_t acc = 0;
#pragma unroll
    for (int w = 0; w < kWideStrip; w++) {
        const uint32_t f = add2(dm, byte_sel(ta, tb, sel[w]));
        const uint32_t x = xn[w];
        uint32_t mt;
        if (AFFINE) {
            mt = max3_2(f, x, y);
            if (ENDS) fxs[w] = max3_2(f, x, x);
            y = add_max2(f, K::right, y);
            xn[w] = add_max2(f, K::down, x);
            if (ENDS) xn[w] = (xn[w] & ~free[w]) | (add_max2(f, K::free_open, add2(x, K::free_more)) & free[w]);
        } else {  // xn: the clean score of the row above plus the row's cost
            mt = add_max2(y, K::right, max3_2(f, x, x));
            if (ENDS) fxs[w] = mt;
            y = mt & ~kTagMask2;
            xn[w] = add2(y, K::down);
            if (ENDS) xn[w] = (xn[w] & ~free[w]) | (add2(y, K::free_open) & free[w]);
        }
        const uint32_t tg = mt & kTagMask2;
        if (ENDS) mts[w] = mt;
        dm = m[w];
        m[w] = mt & ~kTagMask2;
        acc += tg << (2 * w);
    }
    return acc;
}

// A lane of the wide window: the strip it is on.
template <bool AFFINE, int LANES>
struct WideLane {
    using K = BandCost<AFFINE>;
    static constexpr int NB = wide_diagonals(LANES), ROWS = wide_rows(NB), PERIOD = kWideLag * LANES;
    uint32_t m[kWideStrip], xn[kWideStrip], sel[kWideStrip], free[kWideStrip];
    uint32_t ra = 0, rb = 0;      // the next rows' bases
    uint32_t out_m, out_y;        // last column's M and next column's IY of the row done last
    uint32_t last_m;              // the neighbour's M a step ago
    int32_t k, t = 0;             // strip, row
    int32_t va = kBandDead, vb = kBandDead;  // scores at the segments' ends, on the lanes that meet them
    bool ends = false;            // a segment's column C is in the strip

    HERO_HD explicit WideLane(int lane) : k(lane) { out_m = out_y = last_m = band_half2(kBandDead); }

    // M of column 0 at the row of strip 0's row u (u >= -1), and IY of its right neighbour
    HERO_HD static int32_t col0(int type, int32_t base, int32_t u) {
        const int32_t i = base + 1 + u;
        return i < 0 ? kBandDead : 4 * (wide_col0<AFFINE>(type, i) + K::pot * (u + 1));
    }
    HERO_HD static int32_t col0_right(int type, int32_t base, int32_t u) {
        const int32_t i = base + 1 + u;
        if (i < 0) return kBandDead;
        if (!AFFINE) return col0(type, base, u);
        return 4 * ((type == BT_RIGHT ? band_col0_right<BT_RIGHT>(i) : band_col0_right<BT_LEFT>(i)) + u + 2);
    }

    HERO_HD void begin(const BandSeg &a, const BandSeg &b, int type_a, int type_b) {
        const uint32_t dead = band_half2(kBandDead);
        const int32_t j0 = kWideStrip * k + 1;
        const int32_t ja = j0 < a.C ? j0 : a.C, jb = j0 < b.C ? j0 : b.C;  // no reads past a shorter segment's end
        uint32_t wa = pack16(a.col, ja - 1), wb = pack16(b.col, jb - 1);
        ends = (a.C >= j0 && a.C < j0 + kWideStrip) || (b.C >= j0 && b.C < j0 + kWideStrip);
#pragma unroll
        for (int w = 0; w < kWideStrip; w++) {
            m[w] = xn[w] = dead;
            sel[w] = band_sel(wa & 3u, wb & 3u);
            wa >>= 2;
            wb >>= 2;
            free[w] = (type_a == BT_LEFT && j0 + w == a.C ? 0xffffu : 0u) |
                      (type_b == BT_LEFT && j0 + w == b.C ? 0xffff0000u : 0u);
        }
        t = 0;
        refill(a, b);
    }

    // the bases of the next sixteen rows: at the strip's first row, and every
    // sixteen steps of the warp, so that its lanes load together
    HERO_HD void refill(const BandSeg &a, const BandSeg &b) {
        const int32_t j0 = kWideStrip * k + 1;
        ra = pack16(a.row, (j0 < a.C ? j0 : a.C) + a.base - 1 + t);
        rb = pack16(b.row, (j0 < b.C ? j0 : b.C) + b.base - 1 + t);
    }

    // Row t of strip k; in_m, in_y: what the neighbour passed on.  any_ends: some
    // lane of the warp has a column C in its strip.  Returns the row's codes.
    HERO_HD uint32_t row(const BandSeg &a, const BandSeg &b, int type_a, int type_b, uint32_t in_m, uint32_t in_y,
                         bool any_ends) {
        const uint32_t dead = band_half2(kBandDead);
        const int32_t j0 = kWideStrip * k + 1;
        uint32_t dm = t + kWideStrip - 1 < ROWS ? last_m : dead;  // (row above, j0 - 1)
        uint32_t y = t + kWideStrip < ROWS ? in_y : dead;
        if (k == 0) {
            dm = pack2(col0(type_a, a.base, t - 1), col0(type_b, b.base, t - 1));
            y = pack2(col0_right(type_a, a.base, t), col0_right(type_b, b.base, t));
            if (t + kWideStrip >= ROWS) y = dead;  // past the window
            if (t + kWideStrip - 1 >= ROWS) dm = dead;
        } else if (!AFFINE) {
            y = t + kWideStrip < ROWS ? in_m : dead;
        }
        const uint32_t ta = band_table<AFFINE>(ra & 3u), tb = band_table<AFFINE>(rb & 3u);
        ra >>= 2;
        rb >>= 2;
        // row 0: its IX equal its IY, which a row's gap extensions leave as they are
        const uint32_t row0 = (j0 + a.base + t == 0 ? 0xffffu : 0u) | (j0 + b.base + t == 0 ? 0xffff0000u : 0u);
        const uint32_t y0 = y + 0x00020002u;
        uint32_t mts[kWideStrip], fxs[kWideStrip], acc;
        if (any_ends) {
            acc = wide_row<AFFINE, true>(m, xn, sel, ta, tb, dm, y, free, mts, fxs);
            const int32_t da = a.R - a.C - a.base, db = b.R - b.C - b.base;  // the ends' window places
            const int32_t cea = da < NB - 1 ? da : NB - 1, ceb = db < NB - 1 ? db : NB - 1;
#pragma unroll
            for (int w = 0; w < kWideStrip; w++) {
                // above the window an align-left path climbs freely: its row, or the window's last
                const int32_t pot = K::pot * (2 * (j0 + w) + t - w);
                if (j0 + w == a.C && t - w == cea) va = (half_lo(da > cea ? fxs[w] : mts[w]) >> 2) - pot;
                if (j0 + w == b.C && t - w == ceb) vb = (half_hi(db > ceb ? fxs[w] : mts[w]) >> 2) - pot;
            }
        } else {
            acc = wide_row<AFFINE, false>(m, xn, sel, ta, tb, dm, y, free, mts, fxs);
        }
        if (AFFINE && row0) {
#pragma unroll
            for (int w = 0; w < kWideStrip; w++) xn[w] = (xn[w] & ~row0) | (add2(y0, free[w] & K::free_more) & row0);
        }
        out_m = m[kWideStrip - 1];
        out_y = y;
        t++;
        return acc;
    }
};

// band_walk over the wide window's codes: codes.get(strip, row) holds the
// strip's eight cells of a row.  Diagonal runs are found eight cells at a time.
template <bool AFFINE, class Codes>
HERO_HD int32_t wide_walk(const BandSeg &s, int type, int32_t nb, const Codes &codes, uint32_t gap_up,
                          uint32_t gap_left, OpsPut &out) {
    using T = PairTags<AFFINE>;
    constexpr int32_t AHEAD = 8;
    const int32_t end = out.p;
    int32_t i = s.R, j = s.C;
    auto code_at = [&](int32_t ci, int32_t cj) {
        const int32_t k = (cj - 1) >> 3;
        return (codes.get(k, ci - (kWideStrip * k + 1) - s.base) >> (2 * ((cj - 1) & 7))) & 3u;
    };
    if (type == BT_LEFT && i - j - s.base > nb - 1) {
        const int32_t k = i - j - s.base - (nb - 1);
        out.run(gap_up, uint32_t(k));
        i -= k;
    }
    while (i > 0 && j > 0) {
        if (uint32_t(i - j - s.base) >= uint32_t(nb)) return -1;
        const int32_t n = i < j ? (i < AHEAD ? i : AHEAD) : (j < AHEAD ? j : AHEAD);
        uint32_t code[AHEAD];
#pragma unroll
        for (int t = 0; t < AHEAD; t++) code[t] = t < n ? code_at(i - t, j - t) : 3u;
        int32_t run = 0;
        uint32_t stop = 3u;
#pragma unroll
        for (int t = AHEAD - 1; t >= 0; t--)
            if (code[t] != uint32_t(T::diag)) {
                run = t;
                stop = code[t];
            }
        if (stop == 3u) run = n;
        if (run > 0) {
            i -= run;
            j -= run;
            out.fields(mismatch16(pack16(s.row, i), pack16(s.col, j)) & ops_mask(0, uint32_t(run - 1)), uint32_t(run));
        }
        if (stop == uint32_t(T::up)) {
            out.fields(gap_up, 1u);
            i--;
        } else if (stop == uint32_t(T::left)) {
            out.fields(gap_left, 1u);
            j--;
        }
    }
    out.run(gap_up, uint32_t(i));
    out.run(gap_left, uint32_t(j));
    out.flush();
    return end - out.p;
}

// row (0-based) at which the main diagonal starts: the free run of an
// align-right segment lies before it, that of an align-left one behind it
HERO_HD int32_t main_row(int type, int32_t R, int32_t C) { return type == BT_RIGHT ? R - C : 0; }

// mismatches on the main diagonal, counted up to `most` (or a few more); first:
// the column (0-based) of the first
HERO_HD int32_t main_mismatches(const PackSeq &row, const PackSeq &col, int32_t r0, int32_t C, int32_t most,
                                int32_t &first) {
    int32_t e = 0;
    first = C;
    PackStream a(row, r0), b(col, 0);
    for (int32_t t = 0; t < C && e < most; t += 16) {
        uint32_t x = mismatch16(a.next(), b.next());
        if (C - t < 16) x &= ops_mask(0, uint32_t(C - t - 1));
        if (x && first == C) first = t + (low_bit(x) >> 1);
        e += popc32(x);
    }
    return e;
}

// a mismatch among columns [a, b) (0-based) against the rows r0 + column
HERO_HD bool any_mismatch(const PackSeq &row, const PackSeq &col, int32_t r0, int32_t a, int32_t b) {
    PackStream u(row, r0 + a), v(col, a);
    for (int32_t t = a; t < b; t += 16) {
        uint32_t x = mismatch16(u.next(), v.next());
        if (b - t < 16) x &= ops_mask(0, uint32_t(b - t - 1));
        if (x) return true;
    }
    return false;
}

// One mismatch on the main diagonal, at column f: is the straight path the
// traceback's?  Its deficit is 5, so only paths of one gap and no mismatch
// compete.  Anchored at the end (align-right): rows skipped after a start one
// row higher (deficit 4; two rows higher, 5, wins its tie for the affine
// aligner), with every column up to f matching there.  Anchored at the start:
// one row skipped before f (deficit 4) with the rest matching; or, a tie the
// affine aligner gives to the free climb, one column skipped with the rest
// matching and at least one match behind it.  Anchored on both ends a gap needs
// its opposite, and both cost at least 6.
template <bool AFFINE>
HERO_HD bool one_mismatch_straight(const PackSeq &row, const PackSeq &col, int type, int32_t R, int32_t C, int32_t f) {
    const int32_t d = R - C;
    if (type == BT_RIGHT)
        return (d < 1 || any_mismatch(row, col, d - 1, 0, f + 1)) &&
               (!AFFINE || d < 2 || any_mismatch(row, col, d - 2, 0, f + 1));
    if (type == BT_LEFT)
        return (d < 1 || any_mismatch(row, col, 1, f, C)) &&
               (!AFFINE || (C > 1 && any_mismatch(row, col, -1, f + 1 < C ? f + 1 : C - 1, C)));
    return true;
}

// Ops of the straight path, right-aligned in `stride` words: the main diagonal's
// matches and mismatches with the free run of R - C rows before (align-right)
// or after (align-left) it, and their DpSum.
HERO_HD void straight_ops(const PackSeq &row, const PackSeq &col, int type, int32_t R, int32_t C, uint32_t gap_up,
                          uint32_t *w, uint32_t stride, DpSum &sum) {
    const int32_t d = R - C, r0 = main_row(type, R, C);
    const int32_t end = int32_t(stride) * 16, first = end - R;  // R = d + C ops
    const int32_t ds = type == BT_RIGHT ? first + d : first, de = ds + C;
    const int32_t gs = type == BT_RIGHT ? first : de;           // the gap's range [gs, gs + d)
    // bases are read for the diagonal's words alone: the free run may be longer
    // than the room around a read array
    PackStream u(row, r0 + (ds & ~15) - ds), v(col, (ds & ~15) - ds);
    for (int32_t k = first >> 4; k < int32_t(stride); k++) {
        const int32_t p0 = k * 16;
        uint32_t x = 0;
        const int32_t a = ds > p0 ? ds - p0 : 0, b = de - p0 < 16 ? de - p0 : 16;  // the diagonal's fields [a, b)
        if (a < b) x = mismatch16(u.next(), v.next()) & ops_mask(uint32_t(a), uint32_t(b - 1));
        const int32_t g = gs > p0 ? gs - p0 : 0, h = gs + d - p0 < 16 ? gs + d - p0 : 16;
        if (g < h) x |= gap_up * ops_mask(uint32_t(g), uint32_t(h - 1));
        w[k] = x;
    }
    ops_summary(w, uint32_t(first), uint32_t(R), sum);
}

// straight_ops of a diagonal with no mismatch (e = 0) or one, at column f: the
// words and the summary follow without reading the bases again
HERO_HD void plain_ops(int type, int32_t R, int32_t C, int32_t e, int32_t f, uint32_t gap_up, uint32_t *w,
                       uint32_t stride, DpSum &sum) {
    const int32_t d = R - C, end = int32_t(stride) * 16, first = end - R;
    const int32_t ds = type == BT_RIGHT ? first + d : first;
    const int32_t gs = type == BT_RIGHT ? first : end - d;
    const int32_t px = e ? ds + f : -1;
    for (int32_t k = first >> 4; k < int32_t(stride); k++) {
        const int32_t p0 = k * 16;
        uint32_t x = (px >> 4) == k ? 1u << (2 * (px & 15)) : 0u;
        const int32_t g = gs > p0 ? gs - p0 : 0, h = gs + d - p0 < 16 ? gs + d - p0 : 16;
        if (g < h) x |= gap_up * ops_mask(uint32_t(g), uint32_t(h - 1));
        w[k] = x;
    }
    const bool lead = type == BT_RIGHT && d > 0, tail = type != BT_RIGHT && d > 0;
    const bool fx = e && f == 0, lx = e && f == C - 1;
    for (int i = 0; i < 4; i++) sum.tot[i] = 0;
    sum.tot[OP_M] = uint16_t(C - e);
    sum.tot[OP_X] = uint16_t(e);
    if (d > 0) sum.tot[gap_up] = uint16_t(d);
    sum.ft = uint8_t(lead ? gap_up : fx ? uint32_t(OP_X) : uint32_t(OP_M));
    sum.fc = uint16_t(lead ? d : fx ? 1 : e ? f : C);
    sum.lt = uint8_t(tail ? gap_up : lx ? uint32_t(OP_X) : uint32_t(OP_M));
    sum.lc = uint16_t(tail ? d : lx ? 1 : e ? C - 1 - f : C);
    sum.nruns = sum.fc == R ? 1 : 2;
    sum.pad = 0;
}

}  // namespace hero
