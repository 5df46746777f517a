// Sweeps the CTU search's shared-memory layout (xavs2_gb300/csrc/ctu_layout.h)
// as its kernel walks it, over every even search range and chunk height: each
// access inside its area, each word of the window formed from the samples it
// stands for.  Prints the first violation and returns 1, or 0.
#include "ctu_layout.h"

#include <cstdio>
#include <vector>

using namespace xg;

static int bad(const char *what, int R, int dyw, int a, int b)
{
    printf("%s at R = %d, %d rows per warp (%d, %d)\n", what, R, dyw, a, b);
    return 1;
}

static int check(int R, int dyw)
{
    const int pitch = ctu_pitch(R), wrows = ctu_window_rows(dyw), plane = ctu_plane(R, dyw), np = tma_pieces(R);
    const size_t keys = ctu_key_bytes(R, dyw), win = ctu_win_bytes(R, dyw);
    const int piece_end = np * kTmaPieceBytes;
    if (keys % 128 || win % 128) return bad("unaligned areas", R, dyw, (int)keys, (int)win);
    if (ctu_smem_bytes(R, dyw, true) < keys + win + piece_end + 16 || ctu_smem_bytes(R, dyw, false) < keys + win)
        return bad("shared memory too small", R, dyw, np, 0);
    if (wrows > kTmaBoxRows) return bad("more rows than a box", R, dyw, wrows, 0);
    // staging: which sample (row << 9 | column) each byte holds
    std::vector<int> stage(piece_end, -1);
    for (int r = 0; r < wrows; r++)
        for (int c = 0; c < 64 + 2 * R; c++) {
            const int at = ctu_stage_at(r, c);
            if (at < 0 || at >= piece_end || stage[at] != -1) return bad("staged sample", R, dyw, r, c);
            stage[at] = r << 9 | c;
        }
    // the window's entries: first sample of each of their two words
    std::vector<int> entry(2 * plane, -1);
    auto place = [&](int r, int k) {
        if (k >= pitch) return 0;
        const int e = ctu_entry(r, pitch) + k;
        if (e >= plane || (size_t)(8 * (e + plane + 1)) > win || entry[e] != -1) return bad("window entry", R, dyw, r, k);
        entry[e] = r << 9 | 4 * k;
        entry[e + plane] = r << 9 | (4 * k + 2);
        return 0;
    };
    const int quads = ctu_quads(pitch), items = wrows * quads, mq = (65536 + quads - 1) / quads;
    for (int e = 0; e < items + 4 * 128; e++)
        if ((e * mq) >> 16 != e / quads) return bad("item", R, dyw, e, quads);
    for (int e = 0; e < items; e++) {
        const int r = e / quads, q = e % quads;
        const int last = ctu_quad_full(q, pitch) ? 20 : 16;   // samples the item reads
        for (int k = 0; k < last; k += 4) {
            const int at = ctu_stage_at(r, 16 * q + k);
            if (at < 0 || at + 4 > piece_end || at % 4 || (k == 0 && at % 16)) return bad("staging read", R, dyw, r, 16 * q + k);
            // an entry that is part of the window is made of its own 8 samples
            const int ent = 4 * q + k / 4;
            for (int b = 0; b < 4; b++) {
                const int want = r << 9 | (16 * q + k + b);
                const bool used = (ent < pitch && k < 16) || (k > 0 && ent - 1 < pitch);
                if (used && stage[at + b] != want) return bad("sample", R, dyw, r, 16 * q + k + b);
            }
        }
        for (int k = 0; k < 4; k++)
            if (place(r, 4 * q + k)) return 1;
    }
    // the search's reads: lane (rx, ry, half), two rows and two displacements a pass
    for (int row = 0; row < kCtuWarps * dyw; row += 2)
        for (int q8 = 0; q8 < 64; q8 += 8)
            for (int r = 0; r < 9; r++)
                for (int rx = 0; rx < 4; rx++)
                    for (int j = 0; j < R; j++)
                        for (int c = 0; c < 4; c++) {
                            const int wr = q8 + row + r;
                            if (wr >= wrows) return bad("row", R, dyw, row, r);
                            const int e = ctu_entry(wr, pitch) + 4 * rx + c + (j >> 1) + (j & 1 ? plane : 0);
                            if (e >= 2 * plane || entry[e] != (wr << 9 | (16 * rx + 4 * c + 2 * j)))
                                return bad("search read", R, dyw, wr, 4 * rx + c);
                        }
    return 0;
}

int main()
{
    for (int R = 2; R <= 128; R += 2)
        for (int dyw = 2; dyw <= kDyWarpMax; dyw *= 2)
            if (check(R, dyw)) return 1;
    return 0;
}
