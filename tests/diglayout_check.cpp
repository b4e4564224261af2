// Host check of the places that the tensor-core contractions read
// (extreme_gb300/csrc/egx_diglayout.cuh), built with the host compiler by
// tests/test_diglayout.py. For nz = 1..48 it prints one line:
//   nz <nz> errors <n>
// errors counts, over every pair of entries of the padded matrix: an entry that is
// not the packed block's of its (row, column), written here from the packed
// layout's definition; a padded entry that is not one of the block, or that
// lies in a padded column and is not one of its row.
#include <algorithm>
#include <cstdio>
#include <set>
#include <vector>

#include "egx_diglayout.cuh"

// packed place of the staged matrix's entry, rows and columns 0 .. 3 nz - 1
static int packed(int nz, int row, int col, bool &turned) {
    const int S = nz * (nz + 1) / 2, A = nz * (nz + 1);
    const int cr = row / nz, i = row % nz, cc = col / nz, j = col % nz;
    turned = (cr == 2) != (cc == 2);
    if (turned) {
        // xz, yz: rows of the receiver's layer, nz + 1 apart
        const int c = cr == 2 ? cc : cr, rc = cr == 2 ? j : i, tr = cr == 2 ? i : j;
        return 4 * S + c * A + rc * (nz + 1) + tr;
    }
    const int k = cr == 2 ? 3 : cr + cc;  // xx, xy, yy, zz
    const int lo = std::min(i, j), hi = std::max(i, j);
    return k * S + lo + hi * (hi + 1) / 2;
}

int main() {
    for (int nz = 1; nz <= 48; nz++) {
        const int np = (nz + 1) / 2 * 2, rows = (3 * np + 15) / 16 * 16, Bs = 4 * nz * (nz + 1);
        int errors = 0;
        auto real = [&](int r) { return r / np < 3 && r % np < nz; };
        auto plain = [&](int r) { return r / np * nz + r % np; };
        std::vector<std::set<int>> of_row(rows);
        for (int r = 0; r < rows; r++)
            for (int c = 0; c < 3 * nz && real(r); c++) {
                bool t;
                of_row[r].insert(packed(nz, plain(r), c, t));
            }
        for (int r = 0; r < rows; r++)
            for (int c0 = 0; c0 < rows; c0 += 2) {
                const uint32_t w = egx::dig_word(nz, r, c0);
                const int at[2] = {(int)(w & 0x3fff), (int)(w >> 16)};
                for (int j = 0; j < 2; j++) {
                    const int c = c0 + j, p = at[j];
                    bool turned = false;
                    if (p < 0 || p >= Bs) errors++;
                    else if (real(r) && real(c)) errors += packed(nz, plain(r), plain(c), turned) != p || turned != (w >> 15 & 1);
                    else if (real(r)) errors += !of_row[r].count(p);
                }
            }
        std::printf("nz %d errors %d\n", nz, errors);
    }
    return 0;
}
