// band_bounds.cpp -- TEST HARNESS ONLY: the window DP of hero_band.cuh over reads
// packed into arrays of exactly the room the framework gives them, built with
// address checking: a segment's side is its whole read array, stored forward or
// reversed and complemented, so both its ends lie at the array's ends.
#include <cstdio>

#include "band_emu.cpp"

namespace {

// the array of one read: (n + 15) / 16 words with kPackPad words on both sides
void pack_exact(const std::vector<uint8_t> &c, int dir, std::vector<uint32_t> &p, PackSeq &s) {
    std::vector<uint32_t> w(size_t((c.size() + 15) / 16 + 2 * kPackPad), 0u);
    for (size_t t = 0; t < c.size(); t++) {
        const size_t g = dir > 0 ? t : c.size() - 1 - t;
        w[kPackPad + g / 16] |= uint32_t(dir > 0 ? c[t] : c[t] ^ 2u) << (2 * (g % 16));
    }
    w.shrink_to_fit();
    p.swap(w);
    s = PackSeq{p.data() + kPackPad, dir > 0 ? 0 : int64_t(c.size()) - 1, dir};
}

void at_the_ends(Seg &g, int salt) {
    pack_exact(g.rowc, (salt & 1) ? -1 : 1, g.rp, g.b.row);
    pack_exact(g.colc, (salt & 2) ? -1 : 1, g.cp, g.b.col);
}

// a column of C bases inside a row of R: anchored at the row's end or start,
// e mismatches beside the first column
void segment(Seg &g, int R, int C, int type, int e, int64_t band, int salt, uint64_t &x) {
    std::vector<uint8_t> row(R), col(C);
    for (uint8_t &b : row) b = uint8_t(rng_next(x) >> 20 & 3);
    const int at = type == BT_RIGHT ? R - C : 0;
    for (int i = 0; i < C; i++) col[i] = row[at + i];
    for (int i = 0; i < e; i++) col[(1 + size_t(i) * 7) % size_t(C)] ^= 1;
    make(g, row.data(), R, col.data(), C, band, type == BT_RIGHT, type == BT_LEFT, salt);
    at_the_ends(g, salt);
}

}  // namespace

int main() {
    uint64_t x = 12345, counts[6] = {0, 0, 0, 0, 0, 0};
    const int free_rows[] = {0, 1, 17, 24, 112, 113, 127, 129, 500};
    const int widths[][2] = {{1, 0}, {1, 11}, {1, 19}, {1, 26}, {1, 40}, {1, -64}, {1, -136}, {0, 0}, {0, 8}, {0, 16}, {0, -64}, {0, -136}};
    for (int C : {1, 17, 60, 255})
        for (int d : free_rows)
            for (int type = 0; type < 3; type++)
                for (int salt = 0; salt < 4; salt++)
                    for (const auto &w : widths)
                        for (int e : {0, 1, 3}) {
                            if (type == BT_NONE && d > 24) continue;
                            Seg a, b;
                            segment(a, C + d, C, type, e, 65535, salt, x);
                            segment(b, C + d, C, type, e, 65535, 3 - salt, x);
                            pair_any(w[0] != 0, w[1], type, false, a, b, Count{counts});
                            if (w[1] == 16) {  // cut bands: |row - column| <= d
                                segment(a, C + d, C, type, e, 0, salt, x);
                                segment(b, C + d, C, type, e, 0, 3 - salt, x);
                                if (a.b.m < a.b.R) pair_any(w[0] != 0, w[1], type, true, a, b, Count{counts});
                            }
                        }
    for (uint64_t c : counts) std::printf("%llu ", (unsigned long long)c);
    return counts[3] || counts[4] || counts[5];
}
