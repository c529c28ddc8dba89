// band_emu.cpp -- TEST HARNESS ONLY: the window DP of hero_band.cuh compiled for the
// host, run beside the whole-matrix DP of hero_core.cuh on the same segments.
#include <cstdint>
#include <cstring>
#include <vector>

#include "../../hero_b200/csrc/hero_band.cuh"

using namespace hero;

namespace {

struct Scratch {
    int32_t R = 0;
    std::vector<uint32_t> t;
    std::vector<int32_t> v;
    void tb_set(int32_t s, int32_t i, uint32_t bits) { t[size_t(s) * (R + 1) + i] = bits; }
    uint32_t tb_get(int32_t s, int32_t i) const { return t[size_t(s) * (R + 1) + i]; }
    int32_t &b(int32_t st, int32_t i) { return v[size_t(st) * (R + 1) + i]; }
};

std::vector<uint8_t> whole(const SegView &v, bool affine, DpSum &sum) {
    Scratch sc;
    sc.R = v.R;
    sc.t.assign(size_t((v.C + 7) / 8) * size_t(v.R + 1), 0);
    sc.v.assign(size_t(3) * size_t(v.R + 1), 0);
    if (affine) dp_fill<8, true>(v, sc); else dp_fill<8, false>(v, sc);
    std::vector<uint8_t> rev;
    auto emit = [&](uint8_t op) { rev.push_back(op); };
    dp_traceback<8>(v, sc, emit, sum);
    return std::vector<uint8_t>(rev.rbegin(), rev.rend());
}

struct Store {
    int words;
    std::vector<uint32_t> w;
    int32_t j = 0;
    void column(int32_t c) { j = c; }
    void put(int k, uint32_t bits) { w[size_t(j) * words + k] = bits; }
};
struct Codes {
    const Store &s;
    int half;
    uint32_t get(int32_t j, int32_t k) const { return (s.w[size_t(j) * s.words + k] >> (16 * half)) & 0xffffu; }
};

// a segment: codes of its two sides packed with room around them; either side
// may be stored reversed and complemented (dir -1)
struct Seg {
    std::vector<uint8_t> rowc, colc;  // oriented codes
    std::vector<uint32_t> rp, cp;
    BandSeg b;
    SegView v;
    bool rev;
};
void pack(const std::vector<uint8_t> &c, int dir, std::vector<uint32_t> &p, PackSeq &s, int shift) {
    p.assign(2 * kPackPad + (c.size() + shift) / 16 + 2, 0x9c3a5f71u);
    for (size_t t = 0; t < c.size(); t++) {
        const size_t g = shift + (dir > 0 ? t : c.size() - 1 - t);
        const uint32_t x = dir > 0 ? c[t] : c[t] ^ 2u;
        uint32_t &w = p[kPackPad + g / 16];
        w = (w & ~(3u << (2 * (g % 16)))) | (x << (2 * (g % 16)));
    }
    s = PackSeq{p.data() + kPackPad, int64_t(shift) + (dir > 0 ? 0 : int64_t(c.size()) - 1), dir};
}
void make(Seg &g, const uint8_t *s, int n, const uint8_t *q, int m, int64_t band, bool right, bool left, int salt) {
    g.rev = m > n;
    g.rowc.assign(g.rev ? q : s, g.rev ? q + m : s + n);
    g.colc.assign(g.rev ? s : q, g.rev ? s + n : q + m);
    pack(g.rowc, (salt & 1) ? -1 : 1, g.rp, g.b.row, (salt * 7) & 15);
    pack(g.colc, (salt & 2) ? -1 : 1, g.cp, g.b.col, (salt * 5) & 15);
    g.b.R = int32_t(g.rowc.size());
    g.b.C = int32_t(g.colc.size());
    const int64_t d = g.b.R - g.b.C, bb = band > d ? band : d;
    g.b.m = int32_t(bb > 65535 ? 65535 : bb);
    g.v = SegView{g.rowc.data(), g.colc.data(), 1, 1, 0, 0, g.b.R, g.b.C, bb, right, left, g.rev};
}

struct Count {
    uint64_t *c;  // segments, certified, straight, wrong ops, wrong summaries, wrong straight ops
};

// the segments the screen finishes: no mismatch, or one that one_mismatch_straight accepts
template <bool AFFINE>
void screen_run(const Seg &g, int type, Count n) {
    const int32_t d = g.b.R - g.b.C;
    if (type == BT_NONE && d > 0) return;
    int32_t f = 0;
    const int32_t e = main_mismatches(g.b.row, g.b.col, main_row(type, g.b.R, g.b.C), g.b.C, 4, f);
    n.c[0]++;
    if (e > 1 || (e == 1 && !one_mismatch_straight<AFFINE>(g.b.row, g.b.col, type, g.b.R, g.b.C, f))) return;
    n.c[1]++;
    n.c[2] += e == 0;
    DpSum want, sum;
    const std::vector<uint8_t> ops = whole(g.v, AFFINE, want);
    const uint32_t stride = uint32_t((g.b.R + g.b.C + 15) / 16);
    std::vector<uint32_t> w(stride + 1, 0xffffffffu);
    plain_ops(type, g.b.R, g.b.C, e, f, g.rev ? OP_I : OP_D, w.data(), stride, sum);
    bool same = int(ops.size()) == g.b.R;
    for (size_t k = 0; same && k < ops.size(); k++) same = ops_field(w.data(), uint32_t(stride * 16 - ops.size() + k)) == ops[k];
    n.c[3] += !same;
    n.c[4] += memcmp(&sum, &want, sizeof(sum)) != 0;
}

template <bool AFFINE, int NB, int TYPE, bool MASK>
void pair_run(Seg &a, Seg &b, Count n) {
    a.b.base = band_base<AFFINE, NB, TYPE>(a.b.R - a.b.C);
    b.b.base = band_base<AFFINE, NB, TYPE>(b.b.R - b.b.C);
    Store st;
    st.words = (NB + 7) / 8;
    st.w.assign(size_t(a.b.C + 1) * st.words, 0);
    BandEnd e[2];
    int32_t jp = -a.b.base > -b.b.base ? -a.b.base : -b.b.base;
    band_fill<AFFINE, NB, TYPE, MASK>(a.b, b.b, a.b.C, jp, st, e[0], e[1]);
    for (int h = 0; h < 2; h++) {
        const Seg &g = h ? b : a;
        n.c[0]++;
        if (g.b.C - e[h].v > band_limit<AFFINE, TYPE>(g.b, NB)) continue;
        n.c[1]++;
        DpSum want, sum;
        const std::vector<uint8_t> ops = whole(g.v, AFFINE, want);
        const uint32_t stride = uint32_t((g.b.R + g.b.C + 15) / 16);
        std::vector<uint32_t> w(stride + 1, 0xffffffffu);
        const uint32_t up = g.rev ? OP_I : OP_D, left = g.rev ? OP_D : OP_I;
        OpsPut put{w.data(), int32_t(stride * 16)};
        const int32_t np = band_walk<AFFINE, NB, TYPE>(g.b, Codes{st, h}, up, left, put);
        bool ok = np == int32_t(ops.size());
        if (ok) ops_summary(w.data(), stride * 16 - uint32_t(np), uint32_t(np), sum);
        for (size_t k = 0; ok && k < ops.size(); k++) ok = ops_field(w.data(), uint32_t(stride * 16 - ops.size() + k)) == ops[k];
        n.c[3] += !ok;
        n.c[4] += memcmp(&sum, &want, sizeof(sum)) != 0;
        if (!e[h].straight) continue;
        n.c[2]++;
        std::vector<uint32_t> w2(stride + 1, 0xffffffffu);
        straight_ops(g.b.row, g.b.col, TYPE, g.b.R, g.b.C, up, w2.data(), stride, sum);
        bool same = int(ops.size()) == g.b.R;
        for (size_t k = 0; same && k < ops.size(); k++) same = ops_field(w2.data(), uint32_t(stride * 16 - ops.size() + k)) == ops[k];
        n.c[5] += !same || memcmp(&sum, &want, sizeof(sum)) != 0;
    }
}

struct WideCodes {
    const std::vector<uint32_t> &w;
    int lanes, half;
    uint32_t get(int32_t k, int32_t t) const {
        return (w[size_t(kWideLag * k + t) * lanes + k % lanes] >> (16 * half)) & 0xffffu;
    }
};

// the wide window; b may be of another type and size
template <bool AFFINE, int LANES>
void wide_pair(int ta, int tb, Seg &a, Seg &b, Count n) {
    constexpr int nb = wide_diagonals(LANES);
    a.b.base = wide_base(AFFINE, nb, ta, a.b.R - a.b.C);
    b.b.base = wide_base(AFFINE, nb, tb, b.b.R - b.b.C);
    const int32_t cmax = a.b.C > b.b.C ? a.b.C : b.b.C, strips = (cmax + 7) / 8;
    const int32_t steps = kWideLag * (strips - 1) + wide_rows(nb);
    std::vector<uint32_t> codes(size_t(steps) * LANES, 0u);
    std::vector<WideLane<AFFINE, LANES>> lane;
    for (int l = 0; l < LANES; l++) lane.emplace_back(l);
    for (int32_t s = 0; s < steps; s++) {  // the lanes of a step read what the step before left
        std::vector<uint32_t> in_m(LANES), in_y(LANES);
        for (int l = 0; l < LANES; l++) {
            in_m[l] = lane[(l + LANES - 1) % LANES].out_m;
            in_y[l] = lane[(l + LANES - 1) % LANES].out_y;
        }
        for (int l = 0; l < LANES; l++) {
            WideLane<AFFINE, LANES> &w = lane[l];
            const int32_t u = s - kWideLag * w.k;
            if (u == 0 && w.k < strips) w.begin(a.b, b.b, ta, tb);
            if (u >= 0 && u < wide_rows(nb) && w.k < strips && (s & 15) == 0) w.refill(a.b, b.b);
            if (u >= 0 && u < wide_rows(nb) && w.k < strips)
                codes[size_t(s) * LANES + l] = w.row(a.b, b.b, ta, tb, in_m[l], in_y[l], w.ends);
            if (u == wide_rows(nb)) w.k += LANES;
            w.last_m = in_m[l];
        }
    }
    int32_t v[2];
    const int ka = ((a.b.C - 1) / 8) % LANES, kb = ((b.b.C - 1) / 8) % LANES;
    v[0] = lane[ka].va;
    v[1] = lane[kb].vb;
    for (int h = 0; h < 2; h++) {
        const Seg &g = h ? b : a;
        n.c[0]++;
        if (g.b.C - v[h] > wide_limit<AFFINE>(g.b, h ? tb : ta, nb)) continue;
        n.c[1]++;
        DpSum want, sum{};
        const std::vector<uint8_t> ops = whole(g.v, AFFINE, want);
        const uint32_t stride = uint32_t((g.b.R + g.b.C + 15) / 16);
        std::vector<uint32_t> w(stride + 1, 0xffffffffu);
        OpsPut put{w.data(), int32_t(stride * 16)};
        const int32_t np = wide_walk<AFFINE>(g.b, h ? tb : ta, nb, WideCodes{codes, LANES, h}, g.rev ? OP_I : OP_D, g.rev ? OP_D : OP_I, put);
        bool ok = np == int32_t(ops.size());
        if (ok) ops_summary(w.data(), stride * 16 - uint32_t(np), uint32_t(np), sum);
        for (size_t k = 0; ok && k < ops.size(); k++) ok = ops_field(w.data(), uint32_t(stride * 16 - ops.size() + k)) == ops[k];
        n.c[3] += !ok;
        n.c[4] += memcmp(&sum, &want, sizeof(sum)) != 0;
    }
}

template <bool AFFINE, int NB>
void pair_type(int type, bool mask, Seg &a, Seg &b, Count n) {
#define HERO_RUN(T) (mask ? pair_run<AFFINE, NB, T, true>(a, b, n) : pair_run<AFFINE, NB, T, false>(a, b, n))
    if (type == BT_RIGHT) HERO_RUN(BT_RIGHT);
    else if (type == BT_LEFT) HERO_RUN(BT_LEFT);
    else HERO_RUN(BT_NONE);
#undef HERO_RUN
}

bool takes(int nb, bool mask, const Seg &g, int type) {
    const int d = g.b.R - g.b.C;
    if (!mask && g.b.m < g.b.R) return false;
    return type != BT_NONE || d < nb - 1;
}

void pair_any(bool affine, int nb, int type, bool mask, Seg &a, Seg &b, Count n) {
    if (nb == 0) {  // the screen alone
        for (const Seg *g : {&a, &b}) affine ? screen_run<true>(*g, type, n) : screen_run<false>(*g, type, n);
        return;
    }
    if (nb < 0) {  // the wide window of -nb diagonals: a segment beside the one before it
        static Seg before;
        static int before_type = -1, before_nb = 0;
        if (before_nb != nb) before_type = -1;
        before_nb = nb;
        for (Seg *g : {&a, &b}) {
            if (g->b.m < g->b.R || (type == BT_NONE && g->b.R - g->b.C >= -nb - 1)) continue;
            if (before_type >= 0) {
                if (affine && nb == -10) wide_pair<true, 2>(before_type, type, before, *g, n);
                if (affine && nb == -64) wide_pair<true, 8>(before_type, type, before, *g, n);
                if (affine && nb == -136) wide_pair<true, 16>(before_type, type, before, *g, n);
                if (!affine && nb == -10) wide_pair<false, 2>(before_type, type, before, *g, n);
                if (!affine && nb == -64) wide_pair<false, 8>(before_type, type, before, *g, n);
                if (!affine && nb == -136) wide_pair<false, 16>(before_type, type, before, *g, n);
            }
            before = *g;
            before.b.row.w = before.rp.data() + kPackPad;
            before.b.col.w = before.cp.data() + kPackPad;
            before.v.row_base = before.rowc.data();
            before.v.col_base = before.colc.data();
            before_type = type;
        }
        return;
    }
    if (!takes(nb, mask, a, type) || !takes(nb, mask, b, type)) return;
    if (affine) {
        if (nb == 4) pair_type<true, 4>(type, mask, a, b, n);
        if (nb == 8) pair_type<true, 8>(type, mask, a, b, n);
        if (nb == 16) pair_type<true, 16>(type, mask, a, b, n);
        if (nb == 11) pair_type<true, 11>(type, mask, a, b, n);
        if (nb == 19) pair_type<true, 19>(type, mask, a, b, n);
        if (nb == 24) pair_type<true, 24>(type, mask, a, b, n);
        if (nb == 26) pair_type<true, 26>(type, mask, a, b, n);
        if (nb == 40) pair_type<true, 40>(type, mask, a, b, n);
    } else {
        if (nb == 4) pair_type<false, 4>(type, mask, a, b, n);
        if (nb == 8) pair_type<false, 8>(type, mask, a, b, n);
        if (nb == 16) pair_type<false, 16>(type, mask, a, b, n);
    }
}

uint64_t rng_next(uint64_t &x) {
    x ^= x << 13;
    x ^= x >> 7;
    x ^= x << 17;
    return x * 0x2545f4914f6cdd1dull;
}

struct CountWalk {
    uint32_t n = 0;
    void begin(int64_t, int64_t, int64_t) {}
    void position(int64_t) {}
    void run(uint8_t, int64_t) {}
    void dp(int64_t, int64_t, int64_t, int64_t, uint32_t, int64_t) { n++; }
    bool check(int64_t, int64_t) { return true; }
    void finish() {}
};

}  // namespace

extern "C" {

// keys of random windows: from packed codes against base by base, for every k
uint64_t window_keys(uint64_t seed) {
    uint64_t x = seed * 0x9e3779b97f4a7c15ull + 1, wrong = 0;
    for (int32_t k = 1; k <= 63; k++)
        for (int rep = 0; rep < 50; rep++) {
            uint32_t w[4];
            for (uint32_t &v : w) v = uint32_t(rng_next(x) >> 16);  // bits above 2k arbitrary
            Kmer f{0, 0}, r{0, 0}, gf, gr;
            for (int32_t t = 0; t < k; t++) {
                const uint32_t c = (w[t >> 4] >> (2 * (t & 15))) & 3u;
                kmer_push(f, c, k);
                kmer_push_front(r, c ^ 2u, k);
            }
            kmer_from_window(w, k, gf, gr);
            wrong += gf.lo != f.lo || gf.hi != f.hi || gr.lo != r.lo || gr.hi != r.hi;
        }
    return wrong;
}

// random chains of increasing keys, with touching, overlapping and end-aligned
// ones: chain_dp_count against the BandAligner calls of walk_chain
uint64_t chain_counts(uint64_t seed, uint64_t chains) {
    uint64_t x = seed * 0x9e3779b97f4a7c15ull + 1, wrong = 0;
    for (uint64_t c = 0; c < chains; c++) {
        Params p{int32_t(1 + rng_next(x) % 20), int32_t(rng_next(x) % 40), 1, 0, 1.0, double(rng_next(x) % 3) / 2, 0.6};
        const int32_t n = 1 + int32_t(rng_next(x) % 5);
        std::vector<uint64_t> keys;
        int32_t q = int32_t(rng_next(x) % 4) * int32_t(rng_next(x) % 9), s = int32_t(rng_next(x) % 4) * int32_t(rng_next(x) % 9);
        for (int32_t i = 0; i < n; i++) {
            keys.push_back(hit_pack(0, uint32_t(q), uint32_t(s)));
            const int32_t step = 1 + int32_t(rng_next(x) % uint64_t(2 * p.k));
            q += rng_next(x) % 4 == 0 ? p.k : step;
            s += rng_next(x) % 4 == 0 ? p.k : step + (rng_next(x) % 3 == 0 ? int32_t(rng_next(x) % 3) : 0);
        }
        const int32_t Lq = hit_posQ(keys.back()) + p.k + int32_t(rng_next(x) % 3) * int32_t(rng_next(x) % 20);
        const int32_t Ls = hit_posS(keys.back()) + p.k + int32_t(rng_next(x) % 3) * int32_t(rng_next(x) % 20);
        auto key = [&keys](int32_t i) { return keys[size_t(i)]; };
        CountWalk w;
        walk_chain(p, Lq, Ls, key, n, w);
        wrong += w.n != chain_dp_count(p, Lq, Ls, key, n);
    }
    return wrong;
}

// every pair of strings of the first `letters` bases with R rows and C columns (codes 0..3)
void band_exhaustive(int affine, int nb, int type, int mask, int letters, int R, int C, int64_t band, uint64_t *counts) {
    uint64_t total = 1;
    for (int i = 0; i < R + C; i++) total *= uint64_t(letters);
    uint8_t s[2][32], q[2][32];
    Seg g[2];
    for (uint64_t k = 0; k < total; k += 2) {
        for (int h = 0; h < 2; h++) {
            uint64_t x = (k + h) % total;
            for (int i = 0; i < R; i++, x /= letters) s[h][i] = uint8_t(x % letters);
            for (int i = 0; i < C; i++, x /= letters) q[h][i] = uint8_t(x % letters);
            make(g[h], s[h], R, q[h], C, band, type == BT_RIGHT, type == BT_LEFT, int((k + 3 * h) & 15));
        }
        pair_any(affine != 0, nb, type, mask != 0, g[0], g[1], Count{counts});
    }
}

// random segments as reads give them: one side a copy of the other with
// substitutions and short indels, or a tandem repeat of a short unit, joined to
// random bases on the free side
void band_random(int affine, int nb, int mask, uint64_t seed, uint64_t pairs, int cmax, int64_t band_max, uint64_t *counts) {
    uint64_t x = seed * 0x9e3779b97f4a7c15ull + 1;
    for (uint64_t k = 0; k < pairs; k++) {
        const int type = int(rng_next(x) % 3), C = 1 + int(rng_next(x) % cmax);
        Seg g[2];
        for (int h = 0; h < 2; h++) {
            const int period = 1 + int(rng_next(x) % 6), kind = int(rng_next(x) % 4), rate = int(rng_next(x) % 30);
            std::vector<uint8_t> col(C), row;
            for (int i = 0; i < C; i++)
                col[i] = kind == 0 && i >= period ? col[i - period] : uint8_t(rng_next(x) % (kind == 1 ? 2 : 4));
            for (int i = 0; i < C; i++) {
                const int r = int(rng_next(x) % 400);
                if (r < rate) { row.push_back(uint8_t(rng_next(x) & 3)); continue; }
                if (r < rate + 4) for (int n = 1 + int(rng_next(x) % 3); n > 0; n--) row.push_back(uint8_t(rng_next(x) & 3));
                if (r >= rate + 4 && r < rate + 8) i += int(rng_next(x) % 3);
                if (i < C) row.push_back(col[i]);
            }
            if (row.empty()) row.push_back(0);
            const int extra = type == BT_NONE ? 0 : int(rng_next(x) % (3 + (rng_next(x) & 1) * 60));
            for (int i = 0; i < extra; i++) {
                const uint8_t c = kind == 0 && C > period ? col[i % period] : uint8_t(rng_next(x) % (kind == 1 ? 2 : 4));
                row.insert(type == BT_RIGHT ? row.begin() : row.end(), c);
            }
            while (int(row.size()) < C) row.push_back(uint8_t(rng_next(x) & 3));
            if (type == BT_NONE && int(row.size()) > C + (nb > 2 ? nb - 2 : nb < -2 ? -nb - 2 : 0)) row.resize(C);
            const bool swap = (rng_next(x) & 1) && int(row.size()) > C;  // the query on the rows
            const int64_t band = band_max > 0 ? int64_t(rng_next(x) % uint64_t(band_max)) : 65535;
            const auto &s = swap ? col : row, &q = swap ? row : col;
            make(g[h], s.data(), int(s.size()), q.data(), int(q.size()), band, type == BT_RIGHT, type == BT_LEFT, int(rng_next(x) & 15));
        }
        pair_any(affine != 0, nb, type, mask != 0, g[0], g[1], Count{counts});
    }
}

// segments whose band lies inside the window and whose path is bad, while a
// diagonal beside the band matches: one side the other's bases moved by `shift`
// rows (random ones, or a repeat of `period` bases), `free_rows` rows on the free
// side of an anchored one
void band_shifted(int affine, int nb, uint64_t seed, uint64_t pairs, int C, int64_t band, int shift, int period,
                  int free_rows, uint64_t *counts) {
    uint64_t x = seed * 0x9e3779b97f4a7c15ull + 1;
    for (uint64_t k = 0; k < pairs; k++) {
        const int type = int(k % 3), extra = type == BT_NONE ? 0 : free_rows;
        Seg g[2];
        for (int h = 0; h < 2; h++) {
            std::vector<uint8_t> col(C), row;
            for (int i = 0; i < C; i++) col[i] = period && i >= period ? col[i - period] : uint8_t(rng_next(x) & 3);
            for (int i = 0; i < C; i++) {
                const int j = h ? i + shift : i - shift;
                row.push_back(j >= 0 && j < C ? col[j] : uint8_t(rng_next(x) & 3));
            }
            for (int i = 0; i < extra; i++) row.insert(type == BT_RIGHT ? row.begin() : row.end(), uint8_t(rng_next(x) & 3));
            make(g[h], row.data(), int(row.size()), col.data(), C, band, type == BT_RIGHT, type == BT_LEFT, int(rng_next(x) & 15));
        }
        pair_any(affine != 0, nb, type, true, g[0], g[1], Count{counts});
    }
}
}
