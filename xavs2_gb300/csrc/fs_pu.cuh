// fs_pu.cuh -- per-PU full search with exact elimination by 4x4 block means.
//
// A PU with its own search centre and predictor shares no SADs with other
// PUs, so the plain search (fs_pu_search in me.cu) pays w*h pixel differences
// at each of the (2R)^2 displacements.  Most displacements cannot win, and a
// bound far cheaper than their SAD shows it (successive elimination, Li and
// Salari, IEEE Trans. Image Processing 4(1), 1995; here on 4x4 sub-blocks):
// with S a 4x4 block's sum and q = S >> 4,
//     SAD >= sum over the PU's 4x4 blocks of |S_cur - S_ref|
//         >= 16 * D - 15 * (number of blocks),   D = sum of |q_cur - q_ref|,
// and D takes one byte difference per 16 pixels.  A displacement whose bound
// plus MV cost exceeds the best cost known is dropped; the others get their
// SAD.  Every displacement that could win or tie is evaluated, so the minimum
// (cost, visit order) key is the plain search's, bit for bit.
//
// The q of every position of a reference plane is computed once per run
// (mean_planes_kernel).  A plane row keeps its four column phases apart
// (position X at byte (X & 3) * stride / 4 + X / 4), so the blocks of a PU,
// 4 columns apart, are adjacent bytes: D over a phase is a SAD search at
// quarter resolution, four displacements 4 columns apart from one word pair
// and three byte permutes, four displacement rows (4 apart) per word read.
//
// A CTA takes one PU at a time:
//   1. columns and rows whose MV cost alone (monotone in the distance from
//      the predictor) reaches the candidate's cost are cut off;
//   2. the window's q go to shared memory, word [row][k][phase], so that the
//      32 lanes (8 k x 4 phases at R = 64) read 32 consecutive words;
//   3. each warp computes D for its displacements, evaluates the one with the
//      smallest bound (which tightens the best cost for the whole CTA) and
//      marks the 4x4 cells of displacements that may still win; the first
//      round takes every fourth window row, so its best cost is close to the
//      final one;
//   4. the marked cells get their SADs like the plain search's (a thread per
//      cell, or per cell and slice of block rows when there are few cells),
//      from shared memory when they read more than the window holds.
// Content on which the bound says nothing (flat areas) marks every cell and
// pays step 3, about a tenth, on top of the plain search's work.
//
// Integer issue bounds it.  Per PU at R = 64 on block-local motion with noise
// (SM time; plain search in brackets): 4x4 4.4 us (5.0), 8x8 5.8 (8.1), 16x16
// 11 (19), 32x32 41 (59), 64x64 202 (220); the bound excludes less where the
// reference is blocky and the best match poor.
#pragma once

#include "pu_lists.h"

#ifndef XG_PRUNE_SMALL
#define XG_PRUNE_SMALL 128
#endif
#ifndef XG_PRUNE_LARGE
#define XG_PRUNE_LARGE 256
#endif
#ifndef XG_PRUNE_SMALL_MINB
#define XG_PRUNE_SMALL_MINB 6
#endif
#ifndef XG_PRUNE_LARGE_MINB
#define XG_PRUNE_LARGE_MINB 3
#endif

namespace xg {

// Two launches: PUs of at most 16x16 (many, little work each: 128 threads
// and 25 KB of shared memory a CTA at R = 64; with 256 threads the fixed work
// per thread took 7.7 us of SM time per 4x4 PU against 4.4) and the larger
// ones.
template <int DIM> struct PruneShape {
    static constexpr int kThreads = DIM <= kSmallDim ? XG_PRUNE_SMALL : XG_PRUNE_LARGE;
    static constexpr int kWarps = kThreads / 32;
};

// groups of 16 columns / rows a window of n columns / rows needs
__host__ __device__ __forceinline__ int prune_groups(int n) { return (n + 15) >> 4; }

// shared memory of the bounded search at range R of PUs up to dim x dim:
// block, its means, MV-cost tables, their minima per item column / row, cell
// bitmap and list, control words, then the window's means and after them its
// samples
__host__ __device__ __forceinline__ int prune_fixed_smem(int R, int dim)
{
    const int nc = 4 * prune_groups(2 * R);
    return dim * dim + 256 + 2 * (2 * R) * 4 + 2 * 64 * 4 + 64 * 8 + 2 * nc * nc + 32;
}
__host__ __device__ __forceinline__ int prune_pitch(int ni, int w) { return ((ni + w + 10) >> 2) | 1; }   // words
__host__ __device__ __forceinline__ int prune_smem(int R, int dim)
{
    const int ng = prune_groups(2 * R);
    const int means = (16 * ng + dim) * 16 * (ng + (dim >> 4));
    const int samples = (2 * R + dim + 2) * 4 * prune_pitch(2 * R, dim);
    return prune_fixed_smem(R, dim) + (means > samples ? means : samples);
}

// q of every position of every reference plane of the launch's sessions that
// have a means buffer.  A thread computes 16 positions of a row (one word per
// phase) from 4 rows of 5 words with byte dot products.  Positions whose
// block leaves the padded plane get values no admissible displacement reads.
// blockIdx.y: session * max_refs + reference.
__global__ void __launch_bounds__(256) mean_planes_kernel(const SessView *__restrict__ views, int max_refs)
{
    const SessView &v = views[blockIdx.y / max_refs];
    const int r = blockIdx.y % max_refs;
    if (!v.means || r >= v.nrefs) return;
    const int stride = v.g.stride, rows = v.g.H + 2 * kPad, nx = stride >> 4;
    const uint8_t *src = v.ref0[r] - (ptrdiff_t)kPad * stride - kPad;
    uint8_t *dst = v.means + (size_t)r * v.plane_bytes;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < nx * rows; t += gridDim.x * blockDim.x) {
        const int y = t / nx, x = t - y * nx;
        uint32_t acc[4][4];   // [word][phase]
#pragma unroll
        for (int k = 0; k < 4; k++)
#pragma unroll
            for (int p = 0; p < 4; p++) acc[k][p] = 0;
#pragma unroll
        for (int dy = 0; dy < 4; dy++) {
            const uint8_t *row = src + (ptrdiff_t)min(y + dy, rows - 1) * stride + 16 * x;
            const uint4 w = __ldg(reinterpret_cast<const uint4 *>(row));
            const uint32_t w4 = x + 1 < nx ? __ldg(reinterpret_cast<const uint32_t *>(row + 16)) : 0u;
            const uint32_t ws[5] = {w.x, w.y, w.z, w.w, w4};
#pragma unroll
            for (int k = 0; k < 4; k++) {
                acc[k][0] = __dp4a(ws[k], 0x01010101u, acc[k][0]);
                acc[k][1] = __dp4a(__byte_perm(ws[k], ws[k + 1], 0x4321), 0x01010101u, acc[k][1]);
                acc[k][2] = __dp4a(__byte_perm(ws[k], ws[k + 1], 0x5432), 0x01010101u, acc[k][2]);
                acc[k][3] = __dp4a(__byte_perm(ws[k], ws[k + 1], 0x6543), 0x01010101u, acc[k][3]);
            }
        }
        uint8_t *o = dst + (ptrdiff_t)y * stride + 4 * x;
#pragma unroll
        for (int p = 0; p < 4; p++)
            *reinterpret_cast<uint32_t *>(o + p * (stride >> 2)) =
                (acc[0][p] >> 4) | (acc[1][p] >> 4) << 8 | (acc[2][p] >> 4) << 16 | (acc[3][p] >> 4) << 24;
    }
}

// one launch for all sessions of the views
static void mean_planes_run(const SessView *views, int nviews, int max_refs, cudaStream_t st)
{
    mean_planes_kernel<<<dim3(sm_count() * 2, max_refs * nviews), 256, 0, st>>>(views, max_refs);
    count_launch();
}

// SAD of the staged block (cur, w/4 = wq words a row, nw words) against the
// block at ref, by the whole warp
__device__ __forceinline__ uint32_t sad_warp(const uint32_t *cur, const uint8_t *ref, int stride, int wq, int inv,
                                             int nw, int lane)
{
    uint32_t s = 0;
    for (int k = lane; k < nw; k += 32) {
        const int y = (k * inv) >> 16, c = k - y * wq;   // k < 1024
        s = sad4_acc(cur[k], ld4_any(ref + (ptrdiff_t)y * stride + 4 * c), s);
    }
    return __reduce_add_sync(0xffffffffu, s);
}

// One window row (words lo, hi) against the block rows it meets: block row
// r - a of displacement row a, a = 0..3, for the rows FIRST (r < 3: only
// a <= r) and LAST (r >= rows: only a > r - rows) leave.
template <bool FIRST, bool LAST, int RR>
__device__ __forceinline__ void cell_row(uint32_t lo, uint32_t hi, const uint32_t (&cw)[4], uint32_t (&acc)[4][4])
{
    const uint32_t b1 = __byte_perm(lo, hi, 0x4321), b2 = __byte_perm(lo, hi, 0x5432), b3 = __byte_perm(lo, hi, 0x6543);
#pragma unroll
    for (int a = 0; a < 4; a++) {
        if (FIRST && a > RR) continue;
        if (LAST && a <= RR) continue;
        const uint32_t c = cw[(RR - a) & 3];   // cw[k]: block row = k mod 4
        acc[a][0] = sad4_acc(c, lo, acc[a][0]);
        acc[a][1] = sad4_acc(c, b1, acc[a][1]);
        acc[a][2] = sad4_acc(c, b2, acc[a][2]);
        acc[a][3] = sad4_acc(c, b3, acc[a][3]);
    }
}

// window words at a cell's row: STAGED, from shared memory (words aligned to
// the window's first column); otherwise from the plane at any alignment
template <bool STAGED>
struct CellRow {
    const uint32_t *w;
    int sh;
    __device__ __forceinline__ void get(int step, uint32_t &lo, uint32_t &hi)
    {
        if (STAGED) {
            lo = w[0];
            hi = w[1];
        } else {
            const uint32_t a = __ldg(w), b = __ldg(w + 1), c = __ldg(w + 2);
            lo = __funnelshift_r(a, b, sh);
            hi = __funnelshift_r(b, c, sh);
        }
        w += step;   // words to the next row
    }
};

// SADs of the 4x4 displacements of a cell over `rows` block rows (a multiple
// of 4): base at the cell's first word, cur the block's first row of the
// slice.  Column by column, so that a block word is read once for the four
// displacement rows it meets.
template <bool STAGED>
__device__ __forceinline__ void cell_sads(const uint32_t *base, int sh, int step, const uint32_t *cur, int wq, int rows,
                                          uint32_t (&acc)[4][4])
{
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
        for (int t = 0; t < 4; t++) acc[a][t] = 0;
    for (int c = 0; c < wq; c++) {
        CellRow<STAGED> row{base + c, sh};
        const uint32_t *cp = cur + c;
        uint32_t cw[4], lo, hi;
        row.get(step, lo, hi);
        cw[0] = cp[0];
        cell_row<true, false, 0>(lo, hi, cw, acc);
        row.get(step, lo, hi);
        cw[1] = cp[wq];
        cell_row<true, false, 1>(lo, hi, cw, acc);
        row.get(step, lo, hi);
        cw[2] = cp[2 * wq];
        cell_row<true, false, 2>(lo, hi, cw, acc);
        row.get(step, lo, hi);
        cw[3] = cp[3 * wq];
        cell_row<false, false, 3>(lo, hi, cw, acc);
        for (int r = 4; r < rows; r += 4) {
            cp += 4 * wq;
            row.get(step, lo, hi);
            cw[0] = cp[0];
            cell_row<false, false, 0>(lo, hi, cw, acc);
            row.get(step, lo, hi);
            cw[1] = cp[wq];
            cell_row<false, false, 1>(lo, hi, cw, acc);
            row.get(step, lo, hi);
            cw[2] = cp[2 * wq];
            cell_row<false, false, 2>(lo, hi, cw, acc);
            row.get(step, lo, hi);
            cw[3] = cp[3 * wq];
            cell_row<false, false, 3>(lo, hi, cw, acc);
        }
        row.get(step, lo, hi);
        cell_row<false, true, 0>(lo, hi, cw, acc);
        row.get(step, lo, hi);
        cell_row<false, true, 1>(lo, hi, cw, acc);
        row.get(step, lo, hi);
        cell_row<false, true, 2>(lo, hi, cw, acc);
    }
}

// the largest bound a displacement may have: the candidates (order 0 and 1)
// win ties, a window displacement may still be tied by an earlier one
__device__ __forceinline__ int prune_limit(const unsigned long long *key)
{
    const unsigned long long k = *reinterpret_cast<const volatile unsigned long long *>(key);
    return (int)(k >> 32) - ((uint32_t)k < 2u ? 1 : 0);
}

// Window positions lo..hi (of a 2R-wide window around `centre`) whose MV
// bits stay within `bits`: bits are 2 len(|d|) + 1 with d the distance to the
// predictor in quarter-pels, so |d| < 2^((bits - 1) / 2).
__device__ __forceinline__ void cut_range(int bits, int centre, int R, int mvp, int &lo, int &hi)
{
    const int l = bits < 1 ? -1 : min((bits - 1) >> 1, 24);
    const int d = l < 0 ? -1 : (1 << l) - 1;          // largest |4 m - mvp|
    // 4 m >= mvp - d, 4 m <= mvp + d with m = centre + k - R
    lo = max(lo, ((mvp - d + 3) >> 2) - centre + R);
    hi = d < 0 ? -1 : min(hi, ((mvp + d) >> 2) - centre + R);
}

// smallest MV bits of the window positions lo..hi
__device__ __forceinline__ int min_bits(int centre, int R, int mvp, int lo, int hi)
{
    const int at = (mvp >> 2) - centre + R;   // window position of the predictor, rounded down
    const int a = min(max(at, lo), hi), b = min(max(at + 1, lo), hi);
    return min(mvbits_hd(4 * (centre + a - R) - mvp), mvbits_hd(4 * (centre + b - R) - mvp));
}

// D of the 4x4 displacements of an item (columns 4 apart, rows 4 apart): the
// search of an hq-row, nwc-word block of means.  q: the item's first word,
// the next word of a row 4 further; cq: the block's rows.
template <bool MASKED>
__device__ __forceinline__ void item_diffs(const uint32_t *q, int pitch, const uint32_t *cq, int hq, int nwc,
                                           uint32_t mask, uint32_t (&acc)[4][4])
{
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
        for (int t = 0; t < 4; t++) acc[a][t] = 0;
    for (int c = 0; c < nwc; c++, q += 4, cq++) {
        const uint32_t *row = q, *cp = cq;
        uint32_t cw[4] = {0, 0, 0, 0};   // block rows r, r - 1, r - 2, r - 3
        const bool tail = MASKED && c == nwc - 1;
        for (int r = 0; r < hq + 3; r++, row += 4 * pitch) {
            cw[3] = cw[2];
            cw[2] = cw[1];
            cw[1] = cw[0];
            const bool in = r < hq;
            if (in) cw[0] = *cp;
            cp += nwc;
            uint32_t b[4] = {row[0], 0, 0, 0};
            const uint32_t hi = row[4];
            b[1] = __byte_perm(b[0], hi, 0x4321);
            b[2] = __byte_perm(b[0], hi, 0x5432);
            b[3] = __byte_perm(b[0], hi, 0x6543);
            if (tail) {
#pragma unroll
                for (int t = 0; t < 4; t++) b[t] &= mask;
            }
#pragma unroll
            for (int a = 0; a < 4; a++) {
                if (a == 0 ? !in : r < a || r - a >= hq) continue;
#pragma unroll
                for (int t = 0; t < 4; t++) acc[a][t] = sad4_acc(cw[a], b[t], acc[a][t]);
            }
        }
    }
}

// the same with the block's height known (one word wide: PUs up to 16x16)
template <bool MASKED, int HQ>
__device__ __forceinline__ void item_diffs_small(const uint32_t *q, int pitch, const uint32_t *cq, uint32_t mask,
                                                 uint32_t (&acc)[4][4])
{
    uint32_t cw[HQ];
#pragma unroll
    for (int r = 0; r < HQ; r++) cw[r] = cq[r];
#pragma unroll
    for (int r = 0; r < HQ + 3; r++, q += 4 * pitch) {
        uint32_t b[4] = {q[0], 0, 0, 0};
        const uint32_t hi = q[4];
        b[1] = __byte_perm(b[0], hi, 0x4321);
        b[2] = __byte_perm(b[0], hi, 0x5432);
        b[3] = __byte_perm(b[0], hi, 0x6543);
        if (MASKED) {
#pragma unroll
            for (int t = 0; t < 4; t++) b[t] &= mask;
        }
#pragma unroll
        for (int a = 0; a < 4; a++) {
            if (r - a < 0 || r - a >= HQ) continue;
#pragma unroll
            for (int t = 0; t < 4; t++) acc[a][t] = sad4_acc(cw[r - a], b[t], r == a ? 0u : acc[a][t]);
        }
    }
}

template <int DIM>
__device__ __forceinline__ void item_diffs_any(const uint32_t *q, int pitch, const uint32_t *cq, int hq, int nwc,
                                               uint32_t mask, uint32_t (&acc)[4][4])
{
    if constexpr (DIM <= kSmallDim) {
        if (mask == 0xffffffffu) {
            if (hq == 4) item_diffs_small<false, 4>(q, pitch, cq, mask, acc);
            else if (hq == 3) item_diffs_small<false, 3>(q, pitch, cq, mask, acc);
            else if (hq == 2) item_diffs_small<false, 2>(q, pitch, cq, mask, acc);
            else item_diffs_small<false, 1>(q, pitch, cq, mask, acc);
        } else {
            if (hq == 4) item_diffs_small<true, 4>(q, pitch, cq, mask, acc);
            else if (hq == 2) item_diffs_small<true, 2>(q, pitch, cq, mask, acc);
            else item_diffs_small<true, 1>(q, pitch, cq, mask, acc);
        }
    } else {
        if (mask == 0xffffffffu) item_diffs<false>(q, pitch, cq, hq, nwc, mask, acc);
        else item_diffs<true>(q, pitch, cq, hq, nwc, mask, acc);
    }
}

// The bounded search of one PU by the CTA.
template <int DIM>
__device__ __forceinline__ void fs_pu_bounded(const xavs2gpu_pu_t &p, const PuState &st, const SessView &v, int R,
                                              int lambda, uint8_t *smem, unsigned long long *__restrict__ keys, int i)
{
    constexpr int kThreads = PruneShape<DIM>::kThreads, kWarps = PruneShape<DIM>::kWarps;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    uint32_t *s_cur = reinterpret_cast<uint32_t *>(smem);              // [h][w/4]
    uint8_t *s_cq = smem + DIM * DIM;                                  // [h/4][4 * nwc] means of the block
    int *s_lx = reinterpret_cast<int *>(smem + DIM * DIM + 256);       // [2R] lambda x MV bits per column
    int *s_ly = s_lx + 2 * R;
    int *s_lxm = s_ly + 2 * R;                                         // minima per item column / item row
    int *s_lym = s_lxm + 64;
    uint32_t *s_map = reinterpret_cast<uint32_t *>(s_lym + 64);        // [cell row][2] marked cells
    unsigned long long *s_key = reinterpret_cast<unsigned long long *>(s_map + 128);   // best (cost, order)
    int *s_ncell = reinterpret_cast<int *>(s_key + 1);
    uint16_t *s_list = reinterpret_cast<uint16_t *>(s_key + 4);        // marked cells (column | row << 8)
    uint32_t *s_q = reinterpret_cast<uint32_t *>(smem + prune_fixed_smem(R, DIM));
    const Geometry g = v.g;
    const int w = c_pu_w[p.part], h = c_pu_h[p.part], wq = w >> 2, hq = h >> 2;
    const int wx0 = p.x + st.cx - R, wy0 = p.y + st.cy - R;
    const uint8_t *ref = v.ref0[p.ref];
    const unsigned long long key0 = keys[i];   // the best candidate (order 0 or 1: it wins ties)
    const int lim0 = (int)(key0 >> 32) - 1;
    // window positions inside the limits, cut to those whose MV cost alone
    // does not exceed lim0: (lambda x bits) >> 16 <= lim0
    int i0 = max(0, p.min_x - (st.cx - R)), ihi = min(2 * R - 1, p.max_x - (st.cx - R));
    int j0 = max(0, p.min_y - (st.cy - R)), jhi = min(2 * R - 1, p.max_y - (st.cy - R));
    if (lim0 < 0 || i0 > ihi || j0 > jhi) return;
    if (lambda > 0) {
        // the cost of `bits` is at most lim0 up to this many bits (the
        // quotient rounded up by one at most, which only cuts less)
        const int bits = (int)fminf(__fdividef((float)(lim0 + 1) * 65536.f, (float)lambda) + 1.f, 1000.f);
        const int bx = min_bits(st.cx, R, p.mvp_x, i0, ihi), by = min_bits(st.cy, R, p.mvp_y, j0, jhi);
        cut_range(bits - by, st.cx, R, p.mvp_x, i0, ihi);
        cut_range(bits - bx, st.cy, R, p.mvp_y, j0, jhi);
    }
    const int ni = ihi - i0 + 1, nj = jhi - j0 + 1;
    if (ni <= 0 || nj <= 0) return;   // nothing can beat the candidate
    if (tid == 0) {
        *s_key = key0;
        *s_ncell = 0;
    }
    for (int k = tid; k < 128; k += kThreads) s_map[k] = 0;
    // block words
    const uint8_t *o = v.cur + (ptrdiff_t)p.y * g.stride + p.x;
    const int inv = (65536 + wq - 1) / wq;   // k / wq = k * inv >> 16 for k < 1024
    for (int k = tid; k < h * wq; k += kThreads) {
        const int y = (k * inv) >> 16, c = k - y * wq;
        s_cur[k] = ld4_any(o + (ptrdiff_t)y * g.stride + 4 * c);
    }
    // lambda x MV bits of the columns and rows (me.c:614-641)
    for (int k = tid; k < ni; k += kThreads) s_lx[k] = lambda * mvbits_hd(4 * (st.cx + i0 + k - R) - p.mvp_x);
    for (int k = tid; k < nj; k += kThreads) s_ly[k] = lambda * mvbits_hd(4 * (st.cy + j0 + k - R) - p.mvp_y);
    const int ngx = prune_groups(ni), ngy = prune_groups(nj), ncol = 4 * ngx;
    const int nwc = (wq + 3) >> 2, pitch = 4 * (ngx + nwc);
    const uint32_t last_mask = 0xffffffffu >> (8 * (4 * nwc - wq));
    const uint8_t *base = ref + (ptrdiff_t)(wy0 + j0) * g.stride + wx0 + i0;
    // the window's means: row r is plane row wy0 + j0 + r, byte b of word
    // (k, phase) the position 16 k + 4 b + phase columns after wx0 + i0
    {
        const int X = wx0 + i0 + kPad, Y = wy0 + j0 + kPad, x = X + (lane & 3);
        const uint8_t *m0 = v.means + (size_t)p.ref * v.plane_bytes + (x & 3) * (g.stride >> 2) + (x >> 2);
        const int nrow = 16 * ngy + 4 * hq - 4, ylast = Y + nj + h - 5;
        for (int r = warp; r < nrow; r += kWarps) {
            const uint8_t *row = m0 + (ptrdiff_t)min(Y + r, ylast) * g.stride;
            for (int c = lane; c < pitch; c += 32) s_q[r * pitch + c] = ld4_any(row + (c & ~3));
        }
    }
    __syncthreads();
    auto mv_cost = [&](int ci, int cj) { return (uint32_t)((s_lx[ci] + s_ly[cj]) >> 16); };
    const unsigned order0 = 2u + (unsigned)(j0 * 2 * R + i0);
    auto order = [&](int ci, int cj) { return order0 + (unsigned)(cj * 2 * R + ci); };
    auto take = [&](uint32_t cost, unsigned ord) { atomicMin(s_key, ((unsigned long long)cost << 32) | ord); };
    const int slack = 15 * wq * hq, nw = wq * h;
    // means of the block (unused bytes 0), smallest MV cost of each item's
    // columns and rows
    for (int k = tid; k < hq * 4 * nwc; k += kThreads) {
        const int by = DIM <= kSmallDim ? k >> 2 : k / (4 * nwc), bx = k - by * 4 * nwc;
        uint32_t s = 0;
        if (bx < wq)
#pragma unroll
            for (int y = 0; y < 4; y++) s = __dp4a(s_cur[(4 * by + y) * wq + bx], 0x01010101u, s);
        s_cq[k] = (uint8_t)(s >> 4);
    }
    // item column e: columns 16 (e / 4) + 4 t + e % 4; item row e: rows
    // 16 (e / 4) + 4 t + e % 4, kept as [e % 4][e / 4]
    for (int k = tid; k < 4 * (ngx + ngy); k += kThreads) {
        const bool col = k < ncol;
        const int e = col ? k : k - ncol, first = 16 * (e >> 2) + (e & 3), n = col ? ni : nj;
        const int *l = col ? s_lx : s_ly;
        int m = 0x3fffffff;   // no such column or row
#pragma unroll
        for (int t = 0; t < 4; t++)
            if (first + 4 * t < n) m = min(m, l[first + 4 * t]);
        if (col) s_lxm[e] = m;
        else s_lym[(e & 3) * ngy + (e >> 2)] = m;
    }
    // the displacements around the centre, where a good predictor's match is:
    // a lane each (small PUs; larger ones take the smallest bounds below)
    if (DIM <= kSmallDim && warp == kWarps - 1) {
        const int ci = R - i0 + lane % 5 - 2, cj = R - j0 + lane / 5 - 2;
        uint32_t cost = 0xffffffffu, ord = 0xffffffffu;
        if (lane < 25 && ci >= 0 && ci < ni && cj >= 0 && cj < nj) {
            const uint8_t *q = base + (ptrdiff_t)cj * g.stride + ci;
            const uint32_t *cw = s_cur;
            const int sh = 8 * (int)((uintptr_t)q & 3);
            const uint8_t *row = reinterpret_cast<const uint8_t *>((uintptr_t)q & ~(uintptr_t)3);
            uint32_t s = 0;
            for (int y = 0; y < h; y++, row += g.stride) {
                const uint32_t *a = reinterpret_cast<const uint32_t *>(row);
                uint32_t lo = __ldg(a);
                for (int c = 0; c < wq; c++) {
                    const uint32_t hi = __ldg(a + c + 1);
                    s = sad4_acc(*cw++, __funnelshift_r(lo, hi, sh), s);
                    lo = hi;
                }
            }
            cost = s + mv_cost(ci, cj);
            ord = order(ci, cj);
        }
        const uint32_t cmin = __reduce_min_sync(0xffffffffu, cost);
        const uint32_t omin = __reduce_min_sync(0xffffffffu, cost == cmin ? ord : 0xffffffffu);
        if (lane == 0 && cmin != 0xffffffffu) take(cmin, omin);
    }
    __syncthreads();
    const int nrowi = 4 * ngy, nitems = ncol * nrowi;
    // k / n = k * inv >> 20 for k < 4224 and n <= 64
    const int invc = ((1 << 20) + ncol - 1) / ncol, invy = ((1 << 20) + ngy - 1) / ngy;
    for (int it0 = 0; it0 < nitems; it0 += kThreads) {
        // items row by row, the rows in the order [row % 4][row / 16]
        const int item = it0 + tid;
        const bool active = item < nitems;
        const int rowi = active ? (item * invc) >> 20 : 0, col = active ? item - rowi * ncol : 0;
        const int pj = (rowi * invy) >> 20, gy = rowi - pj * ngy, gx = col >> 2;
        const int ci0 = 16 * gx + (col & 3), cj0 = 16 * gy + pj;
        int lim = prune_limit(s_key);
        const int mvmin = (s_lxm[col] + s_lym[rowi]) >> 16;
        uint32_t acc[4][4];
        bool pass = active && mvmin <= lim;
        int low = 0x7fffffff;
        if (pass) {
            item_diffs_any<DIM>(s_q + (16 * gy + pj) * pitch + col, pitch, reinterpret_cast<const uint32_t *>(s_cq),
                                hq, nwc, last_mask, acc);
            uint32_t d = acc[0][0];
#pragma unroll
            for (int a = 0; a < 4; a++) d = min(min(d, min(acc[a][0], acc[a][1])), min(acc[a][2], acc[a][3]));
            low = 16 * (int)d + mvmin;
            pass = low - slack <= lim;
        }
        unsigned who = __ballot_sync(0xffffffffu, pass);
        if (it0 == 0 || __popc(who) >= 16) {
            // the displacement with the smallest bound, by the whole warp
            const int wlow = __reduce_min_sync(0xffffffffu, pass ? low : 0x7fffffff);
            if (wlow != 0x7fffffff) {
                const int src = __ffs(__ballot_sync(0xffffffffu, pass && low == wlow)) - 1;
                int at = 0;
                if (lane == src) {
#pragma unroll
                    for (int k = 1; k < 16; k++)
                        if (16 * (int)acc[k >> 2][k & 3] + mvmin == low) at = k;
                    at = (cj0 + 4 * (at >> 2)) << 8 | (ci0 + 4 * (at & 3));
                }
                at = __shfl_sync(0xffffffffu, at, src);
                const int ci = min(at & 0xff, ni - 1), cj = min(at >> 8, nj - 1);
                const uint32_t s = sad_warp(s_cur, base + (ptrdiff_t)cj * g.stride + ci, g.stride, wq, inv, nw, lane);
                if (lane == 0) take(s + mv_cost(ci, cj), order(ci, cj));
                __syncwarp();
            }
            if (it0 == 0) __syncthreads();   // every warp's first best is in
            lim = prune_limit(s_key);
            pass = pass && low - slack <= lim;
            who = __ballot_sync(0xffffffffu, pass);
        }
        if (!who) continue;
        if (pass) {
            // the displacements whose own bound stays within the limit: mark
            // their cells, 4 gx .. 4 gx + 3 of cell row 4 gy + a
            lim += slack;
#pragma unroll
            for (int a = 0; a < 4; a++) {
                const int cj = cj0 + 4 * a;
                if (cj >= nj) continue;
                uint32_t m = 0;
#pragma unroll
                for (int t = 0; t < 4; t++)
                    if (16 * (int)acc[a][t] + mvmin <= lim && ci0 + 4 * t < ni &&
                        16 * (int)acc[a][t] + (int)mv_cost(ci0 + 4 * t, cj) <= lim)
                        m |= 1u << t;
                if (m) atomicOr(&s_map[2 * (4 * gy + a) + (gx >> 3)], m << (4 * (gx & 7)));
            }
        }
    }
    __syncthreads();
    for (int k = tid; k < 8 * ngy; k += kThreads) {
        uint32_t m = s_map[k];
        if (m) {
            int at = atomicAdd(s_ncell, __popc(m));
            for (; m; m &= m - 1) s_list[at++] = (uint16_t)((32 * (k & 1) + __ffs(m) - 1) | (k >> 1) << 8);
        }
    }
    __syncthreads();
    const int ncell = *s_ncell;
    if (ncell) {
        unsigned long long best = kNoKey;
        const int spitch = prune_pitch(ni, w), srows = nj + h + 2;
        const bool staged = ncell * (h + 3) * (wq + 1) > srows * spitch;
        if (staged) {   // the window's samples, word-aligned to its first column, over the means
            const int sh = 8 * (int)((uintptr_t)base & 3), nw4 = (ni + w + 9) >> 2;
            for (int r = warp; r < srows; r += kWarps) {
                const int y = min(wy0 + j0 + r, g.H + kPad - 1);
                const uint8_t *q = ref + (ptrdiff_t)y * g.stride + wx0 + i0;
                const uint32_t *a = reinterpret_cast<const uint32_t *>(reinterpret_cast<uintptr_t>(q) & ~(uintptr_t)3);
                for (int c = lane; c < nw4; c += 32)
                    s_q[r * spitch + c] = __funnelshift_r(__ldg(a + c), __ldg(a + c + 1), sh);
            }
            __syncthreads();
        }
        // slices of block rows per cell, while cells alone leave threads idle
        int lsl = 0;
        while (lsl < 3 && (ncell << lsl) < kThreads && (h & ((8 << lsl) - 1)) == 0) lsl++;
        const int hs = h >> lsl, units = ncell << lsl;
        for (int u0 = warp * 32; u0 < units; u0 += kThreads) {
            const int u = u0 + lane;
            const bool on = u < units;
            const uint32_t cell = s_list[on ? u >> lsl : 0];
            const int ci0 = 4 * (int)(cell & 0xff), cj0 = 4 * (int)(cell >> 8), y0 = (u & ((1 << lsl) - 1)) * hs;
            uint32_t acc[4][4];
            if (staged) {
                cell_sads<true>(s_q + (cj0 + y0) * spitch + (ci0 >> 2), 0, spitch, s_cur + y0 * wq, wq, hs, acc);
            } else {
                const uint8_t *q = base + (ptrdiff_t)(cj0 + y0) * g.stride + ci0;
                cell_sads<false>(reinterpret_cast<const uint32_t *>(reinterpret_cast<uintptr_t>(q) & ~(uintptr_t)3),
                                 8 * (int)((uintptr_t)q & 3), g.stride >> 2, s_cur + y0 * wq, wq, hs, acc);
            }
            for (int m = 1; m < (1 << lsl); m *= 2)
#pragma unroll
                for (int a = 0; a < 4; a++)
#pragma unroll
                    for (int t = 0; t < 4; t++) acc[a][t] += __shfl_xor_sync(0xffffffffu, acc[a][t], m);
            if (!on) continue;
            uint32_t bc = 0xffffffffu, bo = 0;   // the cell's positions in visit order
#pragma unroll
            for (int a = 0; a < 4; a++) {
                const int cj = cj0 + a;
                if (cj >= nj) continue;
                const int ly = s_ly[cj];
#pragma unroll
                for (int t = 0; t < 4; t++) {
                    const uint32_t cost = acc[a][t] + (uint32_t)((s_lx[min(ci0 + t, ni - 1)] + ly) >> 16);
                    if (ci0 + t < ni && cost < bc) {
                        bc = cost;
                        bo = 2u * (unsigned)(R * a) + (unsigned)t;
                    }
                }
            }
            const unsigned long long key = ((unsigned long long)bc << 32) | (order(ci0, cj0) + bo);
            best = key < best ? key : best;
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            const unsigned long long other = __shfl_xor_sync(0xffffffffu, best, off);
            best = other < best ? other : best;
        }
        if (lane == 0 && best != kNoKey) atomicMin(s_key, best);
        __syncthreads();
    }
    if (tid == 0) {
        const unsigned long long k = *s_key;
        if (k < key0) keys[i] = k;
    }
}

// The n PUs of the list (*count of them where count is given), up to
// DIM x DIM, of sessions with a means buffer; a CTA takes one at a time.
template <int DIM>
__global__ void __launch_bounds__(PruneShape<DIM>::kThreads, DIM <= kSmallDim ? XG_PRUNE_SMALL_MINB : XG_PRUNE_LARGE_MINB)
    fs_bounded_kernel(const uint32_t *__restrict__ list, int n, const int *__restrict__ count,
                      const SessView *__restrict__ views, int R, int lambda)
{
    extern __shared__ __align__(16) uint8_t smem_pu[];
    if (count) n = *count;
    for (int li = blockIdx.x; li < n; li += gridDim.x) {
        const uint32_t e = list[li];
        const SessView &v = views[e >> kSessShift];
        const int i = (int)(e & kIdxMask);
        const PuState st = v.state[i];
        if (li != blockIdx.x) __syncthreads();   // the previous PU's readers are done
        if (st.valid) fs_pu_bounded<DIM>(v.pus[i], st, v, R, lambda, smem_pu, v.keys, i);
    }
}

// Whether PUs of range R and factor lambda take the bounded search where
// their session has a means buffer (sums of two lambda x bits must stay below
// 2^30).
static inline bool prune_ok(int lambda) { return lambda < (1 << 23); }

template <int DIM>
static int prune_launch_one(const uint32_t *list, int n, const int *count, const SessView *views, int R, int lambda,
                            cudaStream_t st)
{
    static std::atomic<int> attr_bytes[64];
    const int dev = current_device(), bytes = prune_smem(R, DIM);
    if (dev < 0 || dev >= 64) return XAVS2GPU_ERR_ARG;
    if (n == 0) return XAVS2GPU_OK;
    if (attr_bytes[dev].load(std::memory_order_relaxed) < bytes) {
        const int most = prune_smem(128, DIM);   // the largest range: set once, whatever thread comes first
        XG_CUDA(cudaFuncSetAttribute(fs_bounded_kernel<DIM>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
        attr_bytes[dev].store(most, std::memory_order_relaxed);
    }
    // lists of unknown length: a few CTAs per SM walk them
    const int grid = count ? std::min(n, sm_count() * 8) : n;
    fs_bounded_kernel<DIM><<<grid, PruneShape<DIM>::kThreads, bytes, st>>>(list, n, count, views, R, lambda);
    count_launch();
    XG_CUDA(cudaGetLastError());
    return XAVS2GPU_OK;
}

// list: n_large PUs with a side above 16, then n_small others
static int prune_launch(const uint32_t *list, int n_large, int n_small, const SessView *views, int R, int lambda,
                        cudaStream_t st)
{
    const int rc = prune_launch_one<64>(list, n_large, nullptr, views, R, lambda, st);
    return rc != XAVS2GPU_OK ? rc
                             : prune_launch_one<kSmallDim>(list + n_large, n_small, nullptr, views, R, lambda, st);
}

}  // namespace xg
