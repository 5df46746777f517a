// ctu_layout.h -- the CTU search's shared memory: the MV-cost keys of a chunk
// of search rows, the reference window and the staging area its samples pass
// through.  Plain index arithmetic, the kernel's and the launch's
// (fs_ctu.cuh), which a host program can check over every range.
#pragma once

#include <stddef.h>
#include <stdint.h>

#ifdef __CUDACC__
#define XG_HD __host__ __device__ __forceinline__
#else
#define XG_HD inline
#endif

namespace xg {

constexpr int kCtuWarps = 4;
constexpr int kDyWarpMax = 8;           // search rows per warp: 8, 4 or 2 (3 key bits)
constexpr int kDyChunkMax = kCtuWarps * kDyWarpMax;

// Window layout in 8-byte entries: a row is ctu_pitch(R) entries (15 + R/2:
// word 4*rx + c + (displacement >> 2) of rx, c <= 3), one entry is skipped
// after every 8 rows, and the second plane follows the first.  An 8-byte shared
// load serves 16 lanes at a time; lane bits 0-3 are half, rx bit 0, ry bit 0 and
// rx bit 1, so these read rows 8q + t of four consecutive q = 2*ry + half
// (skewed by 0..3 entries) at entries 4*rx: 16 distinct pairs of banks.
XG_HD int ctu_pitch(int R) { return 15 + (R >> 1); }
XG_HD int ctu_entry(int row, int pitch) { return row * pitch + (row >> 3); }
// rows of the window of a chunk of dyw search rows per warp
XG_HD int ctu_window_rows(int dyw) { return 64 + kCtuWarps * dyw - 1; }

// bytes of a chunk's MV-cost keys and of its window (multiples of 128), and
// the distance of the window's planes in entries
XG_HD uint32_t ctu_key_bytes(int R, int dyw) { return 4u * (uint32_t)(kCtuWarps * dyw * 2 * R); }
XG_HD uint32_t ctu_win_bytes(int R, int dyw)
{
    const int rows = ctu_window_rows(dyw);   // two planes of 8-byte entries
    return (uint32_t)(ctu_entry(rows - 1, ctu_pitch(R)) + ctu_pitch(R) + 7) / 8 * 128;
}
XG_HD int ctu_plane(int R, int dyw) { return (int)(ctu_win_bytes(R, dyw) >> 4); }

// The staging area: the window's samples as np = tma_pieces(R) pieces of 64
// columns and the most rows a window has, each piece dense, the copies'
// barrier after the last.
constexpr int kTmaBoxCols = 64;
constexpr int kTmaBoxRows = 64 + kDyChunkMax - 1;
constexpr int kTmaPieceBytes = (kTmaBoxCols * kTmaBoxRows + 127) / 128 * 128;   // 6144
XG_HD constexpr int tma_pieces(int R) { return (64 + 2 * R + 8 + kTmaBoxCols - 1) / kTmaBoxCols; }
// byte of the staging area that holds column `col` of window row `row`
XG_HD int ctu_stage_at(int row, int col)
{
    const unsigned c = (unsigned)col;
    return (int)(c / kTmaBoxCols) * kTmaPieceBytes + row * kTmaBoxCols + (int)(c % kTmaBoxCols);
}

// The window is formed four entries of a row at a time (a quad: the 16
// samples from column 16 q on and, for its last entry, the word after them).
// A row's last quad may hold fewer than four entries; its word after is then
// not part of the window, nor, where the quads fill the pieces (72 + 2R a
// multiple of 64), of the staging area.
XG_HD int ctu_quads(int pitch) { return (pitch + 3) >> 2; }
XG_HD bool ctu_quad_full(int q, int pitch) { return 4 * q + 3 < pitch; }

// a chunk's dynamic shared memory: keys, window and, with staging, the boxes
// and their barrier
inline size_t ctu_smem_bytes(int R, int dyw, bool staging)
{
    const size_t b = (size_t)ctu_key_bytes(R, dyw) + ctu_win_bytes(R, dyw);
    return staging ? b + (size_t)tma_pieces(R) * kTmaPieceBytes + 16 : b;
}

}  // namespace xg
