// fs_ctu.cuh -- shared-window full search over every PU of a 64x64 CTU.
//
// The PU set of a CTU is the one an AVS2 encoder's mode decision searches:
// for CU sizes 64, 32 and 16 at every quadtree position the 13 PUs of the
// partitions 2Nx2N, 2NxN, Nx2N, 2NxnU, 2NxnD, nLx2N and nRx2N, and for every
// 8x8 CU its 8x8, 8x4 and 4x8 PUs plus the four 4x4 blocks -- 849 "slots",
// covering all 25 LumaPU shapes.  For PUs that share the search centre (0,0)
// and the MV predictor, the SAD of every PU at a displacement is a sum of the
// SADs of its 4x4 blocks at that displacement, so one warp computes the 256
// block SADs of the CTU once per displacement and derives all 849 PU costs
// from them (sums in registers, warp shuffles across regions).
//
// Warp layout: a lane is (rx, ry, half): (rx, ry) is one of the 16 16x16
// regions of the CTU, half selects its top or bottom 8 rows.  A lane owns the
// 8 4x4 SADs of its half-region, the 18 PUs of its two 8x8 CUs and 6-7 PUs of
// its 16x16 CU; the 52 PUs of the 32x32 CUs and the 13 of the 64x64 CU are
// spread over the lanes (2 + 1 per lane at most).
//
// A CTA of 4 warps handles one (CTU, reference) and a chunk of 8, 16 or 32
// search rows (2, 4 or 8 per warp) over the whole horizontal range; its
// reference window lives in shared memory.  Each warp keeps, per PU, the
// minimum of a 32-bit key (cost << 11 | row-in-warp << 8 | dx+R) and merges it
// into the global 64-bit (cost, visit order) keys with atomicMin.  A warp takes
// two search rows per pass over the window.
//
// The search is bound by instruction issue and, within it, by the pipe that
// byte SADs share with permutes, selects and minima (half rate).  So the window
// holds every 4-sample word at its four byte alignments, as two planes of
// 8-byte entries (row, k): {w(4k), w(4k+1)} and {w(4k+2), w(4k+3)}, w(i) the
// samples i .. i+3.  An 8-byte load then serves two displacements of two rows,
// where a row's four words took five word loads and twelve byte permutes.  A
// pass covers two rows and two displacements: 32 accumulators and no spill at
// 168 registers, so three CTAs share an SM (16-byte entries of all four
// alignments need 64 accumulators, spill at 255 registers and wait on their
// loads).  1080p, one reference, R = 64: 1677 us with the permutes (two CTAs per
// SM), 1354 now, where 16-byte entries took 2119 and passes of four rows 1493.
//
// Search limits: a PU is valid at a displacement iff the referenced block
// lies within [-58, W+58) x [-58, H+58) -- the limits pred_inter_search_single
// derives (md_inter.c:910-926) whenever they bind inside the search window.
// CTUs near the picture edge run a variant that replaces the SAD of every
// 4x4 block whose reference falls outside that region by a large value; the
// PUs containing such a block then never win and are not merged.
#pragma once

#include "ctu_layout.h"
#include "pu_lists.h"

namespace xg {

constexpr int kCtuThreads = 32 * kCtuWarps;
constexpr uint32_t kPoisonSmall = 126976u;     // > any valid cost of a PU up to 16x16
constexpr uint32_t kPoisonLarge = 1u << 22;    // replaces a 4x4 SAD outside the limits
constexpr uint32_t kCapLarge = 2000000u;       // > any valid cost of a 64x64 PU
constexpr int kLimitMargin = 58;               // 64-pixel margin minus 6 (md_inter.c:913-926)

struct CtuJob {
    int16_t x0, y0;       // CTU origin
    uint8_t ref;
    uint8_t levels;       // CU sizes with a PU in the job: 1 8x8, 2 16x16, 4 32x32, 8 64x64
    int16_t mvp_x, mvp_y;
    uint8_t border;       // 1: limits may bind inside the window
    uint8_t sess;         // index into the session views of the launch
    int32_t slot_base;    // index of this job's row in its session's slot map
};

struct CtuPlan {
    int n_jobs = 0, cap_jobs = 0;
    int n_border = 0;             // jobs whose search limits may bind (border variant)
    CtuJob *d_jobs = nullptr;
    int32_t *d_slots = nullptr;   // [n_jobs][kSlots]: PU index or -1
    std::vector<CtuJob> h_jobs;   // host copy (sess = 0), for multi-session launches
};

// ---- device helpers ------------------------------------------------------------------

__device__ __forceinline__ uint32_t addmin(uint32_t a, uint32_t b, uint32_t c)
{
    return __viaddmin_u32(a, b, c);   // min(a + b, c)
}

// slot of small key k (0..24) of a lane
__device__ __forceinline__ int small_slot(int rx, int ry, int half, int k)
{
    if (k < 18) {
        const int side = k / 9, m = k % 9;
        const int gx = 2 * rx + side, gy = 2 * ry + half;
        return (gy * 8 + gx) * 9 + m;
    }
    // 16-CU keys 18..24 -> modes (half 0 / half 1)
    const int i = k - 18;
    const int m0[7] = {0, 1, 3, 5, 6, 9, 10};
    const int m1[7] = {4, 2, 3, 8, 7, 12, 11};
    return 576 + (ry * 4 + rx) * 13 + (half ? m1[i] : m0[i]);
}

// 32-CU key modes per (half, qx, qy) (-1: none); keys A and B.  A lane's own
// pair of regions sums to X1, its outer-half part (top 8 rows or left 8 columns
// of the pair) to X2, the CU's other pair to X3: A = a X1 + b X2, B = c X1 +
// d X2 + X3.
__constant__ int8_t c_m32[2][2][2][2] = {
    // half 0: [qx][qy] -> {A, B}
    {{{1, 0}, {2, 7}}, {{5, 6}, {8, -1}}},
    // half 1
    {{{3, 10}, {9, -1}}, {{4, 11}, {12, -1}}}};
__constant__ int8_t c_c32[2][2][2][4] = {   // a, b, c, d
    {{{1, 0, 1, 0}, {1, 0, 0, 1}}, {{0, 1, 1, -1}, {1, -1, 0, 0}}},
    {{{1, 0, 1, -1}, {0, 1, 0, 0}}, {{1, 0, 0, 1}, {1, -1, 0, 0}}}};
// 64-CU key per ry*8 + rx*2 + half: mode (-1 none) and
// coefficients over (TOT, P, RS) -- half-0 entries hold row quantities (RS =
// sum of a row of regions, P = pair of rows), half-1 entries the column ones.
__constant__ int8_t c_m64[32] = {0, 3, 1, -1, 5, 4, 6, 11, -1, 9, -1, -1, -1, -1, -1, 12,
                                 2, 10, -1, -1, -1, -1, -1, -1, 7, -1, 8, -1, -1, -1, -1, -1};
__constant__ int8_t c_c64[32][3] = {
    {1, 0, 0}, {0, 1, 0}, {0, 1, 0}, {0, 0, 0}, {0, 0, 1}, {0, 1, 0}, {1, 0, -1}, {1, 0, -1},
    {0, 0, 0}, {0, 0, 1}, {0, 0, 0}, {0, 0, 0}, {0, 0, 0}, {0, 0, 0}, {0, 0, 0}, {0, 0, 1},
    {0, 1, 0}, {1, 0, -1}, {0, 0, 0}, {0, 0, 0}, {0, 0, 0}, {0, 0, 0}, {0, 0, 0}, {0, 0, 0},
    {1, 0, -1}, {0, 0, 0}, {0, 0, 1}, {0, 0, 0}, {0, 0, 0}, {0, 0, 0}, {0, 0, 0}, {0, 0, 0}};

// Per-lane constants of the warp layout.
struct LaneRole {
    int half, rx, ry;
    int nh;                         // -half
    int pr1, pr2, pr3, pr4, pr5;    // shuffle partners (see below)
    int c32[4], c64[3];             // coefficients of the 32-CU / 64-CU keys
    int bx0, by0;                   // picture position of the half-region
};

// Folds the costs of one displacement into the lane's keys.  `raw` are the
// lane's eight 4x4 SADs; `mks` = (mvc << 11) | (row << 8) | dx+R.
// LV (a compile-time set of CU sizes, as CtuJob::levels) drops the key
// updates of the CU sizes a job has no PU of.  BORDER poisons the blocks
// outside the limits; the poisoned sums of the large PUs are formed unshifted
// and capped before they become keys (a valid cost, and the cap, plus an MV
// cost stay below 2^21).
template <bool BORDER, int LV>
__device__ __forceinline__ void fold_displacement(const LaneRole &LR, uint32_t (&raw)[2][4], uint32_t mks, int dx,
                                                  bool brow0, bool brow1, const Geometry &g, uint32_t (&ks)[25],
                                                  uint32_t (&kl)[3])
{
    const int half = LR.half;
    if (BORDER) {
#pragma unroll
        for (int c = 0; c < 4; c++) {
            const int xb = LR.bx0 + 4 * c + dx;
            const bool colok = xb >= -kLimitMargin && xb + 4 <= g.W + kLimitMargin;
            if (!(colok && brow0)) raw[0][c] = kPoisonLarge;
            if (!(colok && brow1)) raw[1][c] = kPoisonLarge;
        }
    }
    // small-key domain: SAD << 11 (poison clamped for the small PUs)
    uint32_t t[2][4];
#pragma unroll
    for (int br = 0; br < 2; br++)
#pragma unroll
        for (int c = 0; c < 4; c++) t[br][c] = (BORDER ? min(raw[br][c], kPoisonSmall) : raw[br][c]) << 11;
    // 8x8 CUs of this half: left (cols 0,1) and right (cols 2,3)
    uint32_t qv[2], at[2], ab[2], vl[2], vr[2];
#pragma unroll
    for (int sd = 0; sd < 2; sd++) {
        const int c0 = 2 * sd;
        at[sd] = t[0][c0] + t[0][c0 + 1];
        ab[sd] = t[1][c0] + t[1][c0 + 1];
        vl[sd] = t[0][c0] + t[1][c0];
        vr[sd] = t[0][c0 + 1] + t[1][c0 + 1];
        qv[sd] = at[sd] + ab[sd];
        if (!(LV & 1)) continue;
        const int kb = 9 * sd;
        ks[kb + 0] = addmin(qv[sd], mks, ks[kb + 0]);
        ks[kb + 1] = addmin(at[sd], mks, ks[kb + 1]);
        ks[kb + 2] = addmin(ab[sd], mks, ks[kb + 2]);
        ks[kb + 3] = addmin(vl[sd], mks, ks[kb + 3]);
        ks[kb + 4] = addmin(vr[sd], mks, ks[kb + 4]);
        ks[kb + 5] = addmin(t[0][c0], mks, ks[kb + 5]);
        ks[kb + 6] = addmin(t[0][c0 + 1], mks, ks[kb + 6]);
        ks[kb + 7] = addmin(t[1][c0], mks, ks[kb + 7]);
        ks[kb + 8] = addmin(t[1][c0 + 1], mks, ks[kb + 8]);
    }
    // 16x16 CU: own half (Fh, Lh, strips) + partner half
    const uint32_t Fh = qv[0] + qv[1];
    const uint32_t Lh = qv[0];
    const uint32_t rr_ = half ? ab[0] + ab[1] : at[0] + at[1];   // own outer 16x4 strip
    const uint32_t c0h = vl[0], c3h = vr[1];
    const uint32_t Fh_o = __shfl_xor_sync(0xffffffffu, Fh, 1);
    const uint32_t Lh_o = __shfl_xor_sync(0xffffffffu, Lh, 1);
    const uint32_t xs = half ? c0h : c3h;
    const uint32_t xs_o = __shfl_xor_sync(0xffffffffu, xs, 1);
    const uint32_t F = Fh + Fh_o, L = Lh + Lh_o;
    const uint32_t cc = (half ? c3h : c0h) + xs_o;          // col 3 (half 1) / col 0 (half 0)
    if (LV & 2) {
        ks[18] = addmin(F + L * (uint32_t)LR.nh, mks, ks[18]); // 16x16 | 8x16 right
        ks[19] = addmin(Fh, mks, ks[19]);                      // 16x8 top | bottom
        ks[20] = addmin(L, mks, ks[20]);                       // 8x16 left (both halves)
        ks[21] = addmin(rr_, mks, ks[21]);                     // 16x4 y0 | y12
        ks[22] = addmin(F - rr_, mks, ks[22]);                 // 16x12 y4 | y0
        ks[23] = addmin(cc, mks, ks[23]);                      // 4x16 x0 | x12
        ks[24] = addmin(F - cc, mks, ks[24]);                  // 12x16 x4 | x0
    }
    // large PUs: the region's sum and its top (half 0) or left (half 1) part
    uint32_t Fr = F, a1 = half ? L : Fh;
    if (BORDER) {
        uint32_t fh = 0, lh = 0;
#pragma unroll
        for (int br = 0; br < 2; br++)
#pragma unroll
            for (int c = 0; c < 4; c++) {
                fh += raw[br][c];
                if (c < 2) lh += raw[br][c];
            }
        const uint32_t lh_o = __shfl_xor_sync(0xffffffffu, lh, 1);
        Fr = fh + __shfl_xor_sync(0xffffffffu, fh, 1);
        a1 = half ? lh + lh_o : fh;
    }
    // 32x32 CUs
    const uint32_t F_p = __shfl_xor_sync(0xffffffffu, Fr, LR.pr1);
    const uint32_t a_p = __shfl_xor_sync(0xffffffffu, a1, LR.pr1);
    const uint32_t X1 = Fr + F_p, X2 = a1 + a_p;           // FH, TH  |  FV, LV
    const uint32_t X3 = __shfl_xor_sync(0xffffffffu, X1, LR.pr2);
    const int va = LR.c32[0] * (int)X1 + LR.c32[1] * (int)X2;
    const int vb = LR.c32[2] * (int)X1 + LR.c32[3] * (int)X2 + (int)X3;
    // 64x64 CU
    const uint32_t RS = X1 + __shfl_xor_sync(0xffffffffu, X1, LR.pr3);     // row | column sums
    const uint32_t P = RS + __shfl_xor_sync(0xffffffffu, RS, LR.pr4);      // row | column pairs
    const uint32_t TOT = P + __shfl_xor_sync(0xffffffffu, P, LR.pr5);
    const int v64 = LR.c64[0] * (int)TOT + LR.c64[1] * (int)P + LR.c64[2] * (int)RS;
    auto key = [](int v) { return BORDER ? min((uint32_t)v, kCapLarge) << 11 : (uint32_t)v; };
    if (LV & 4) {
        kl[0] = addmin(key(va), mks, kl[0]);
        kl[1] = addmin(key(vb), mks, kl[1]);
    }
    if (LV & 8) kl[2] = addmin(key(v64), mks, kl[2]);
}

// 4x4 SADs of the lane's half-region at the first displacement of an entry:
// row0 = its first window row, k the entry of its first word
__device__ __forceinline__ void sad_at(const uint2 *win, int pitch, int row0, int k, const uint32_t (&cw)[8][4],
                                       uint32_t (&raw)[2][4])
{
#pragma unroll
    for (int br = 0; br < 2; br++)
#pragma unroll
        for (int c = 0; c < 4; c++) raw[br][c] = 0;
#pragma unroll
    for (int r = 0; r < 8; r++) {
        const uint2 *wp = win + ctu_entry(row0 + r, pitch) + k;
#pragma unroll
        for (int c = 0; c < 4; c++) raw[r >> 2][c] = sad4_acc(cw[r][c], wp[c].x, raw[r >> 2][c]);
    }
}

// border jobs: the interior fold for displacements that need no limit
#ifndef XG_CTU_SAFE_SPLIT
#define XG_CTU_SAFE_SPLIT 1
#endif

// Window fill by the tensor memory accelerator: where the session has a
// tensor map over its plane pool (3-D: column, row, plane; box 64 columns x
// 95 rows) and the window lies inside the padded plane at 16-byte alignment, one thread issues
// the window as 64-column boxes into a dense staging area before the CTA
// computes its MV-cost keys, so the copy overlaps that work; a
// shared-to-shared pass then forms the window's entries.
#ifndef XG_CTU_TMA
#define XG_CTU_TMA 1
#endif
constexpr int kWaitLimit = 1 << 20;   // mbarrier polls before a CTA gives up its window

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ bool mbar_wait_bounded(uint32_t bar, uint32_t parity)
{
    for (int i = 0; i < kWaitLimit; i++) {
        uint32_t ok;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok)
                     : "r"(bar), "r"(parity)
                     : "memory");
        if (ok) return true;
    }
    return false;
}

// Thread 0 only: rows [y, y + 95) of plane z (a smaller chunk's window is the
// first of them; rows outside the plane are filled with zeros), columns x .. x + 64*np
// (x a multiple of 16), as np boxes into stage (128-byte aligned), counted
// on the barrier at bar.
__device__ __forceinline__ void tma_window_issue(const void *tmap, uint32_t stage, uint32_t bar, int x, int y, int z,
                                                 int np)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(tmap) : "memory");
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar),
                 "r"((uint32_t)(np * kTmaBoxCols * kTmaBoxRows))
                 : "memory");
    for (int p = 0; p < np; p++)
        asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
                     " [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(stage + (uint32_t)(p * kTmaPieceBytes)),
                     "l"(tmap), "r"(x + p * kTmaBoxCols), "r"(y), "r"(z), "r"(bar)
                     : "memory");
}

// resident CTAs per SM the register budget is sized for (3: 168 registers; 2
// measured 2 % slower at R = 64)
#ifndef XG_CTU_MINB
#define XG_CTU_MINB 3
#endif

// Folds the displacements d0 and d0 + 1 of one search row (SADs s[o], key
// parts mk) into the lane's keys.
template <bool BORDER, int LV>
__device__ __forceinline__ void fold_group(const LaneRole &L, uint32_t (&s)[2][2][4], uint2 mk, int d0, int R, int dy,
                                           const CtuJob &job, const Geometry &g, uint32_t (&ks)[25],
                                           uint32_t (&kl)[3])
{
    const uint32_t m[2] = {mk.x, mk.y};
    // in a border job, displacements whose every block stays inside the
    // limits take the interior fold (same keys: nothing to poison)
    if (BORDER && !(XG_CTU_SAFE_SPLIT && job.y0 + dy >= -kLimitMargin && job.y0 + 64 + dy <= g.H + kLimitMargin &&
                    job.x0 + d0 - R >= -kLimitMargin && job.x0 + 65 + d0 - R <= g.W + kLimitMargin)) {
        const int yb = L.by0 + dy;
        const bool b0 = yb >= -kLimitMargin && yb + 4 <= g.H + kLimitMargin;
        const bool b1 = yb + 4 >= -kLimitMargin && yb + 8 <= g.H + kLimitMargin;
#pragma unroll
        for (int o = 0; o < 2; o++) fold_displacement<true, LV>(L, s[o], m[o], d0 + o - R, b0, b1, g, ks, kl);
    } else {
#pragma unroll
        for (int o = 0; o < 2; o++) fold_displacement<false, LV>(L, s[o], m[o], d0 + o - R, true, true, g, ks, kl);
    }
}

template <bool BORDER, int LV>
__device__ __forceinline__ void ctu_search(const CtuJob &job, int chunk, int dyw, const SessView *__restrict__ views,
                                           int R, int lambda, uint8_t *smem)
{
    const SessView &view = views[job.sess];
    const int32_t *__restrict__ slots = view.slots;
    const uint8_t *__restrict__ cur = view.cur;
    const uint8_t *const *refs = view.ref0;
    const Geometry g = view.g;
    unsigned long long *__restrict__ keys = view.keys;
    const int rows = kCtuWarps * dyw;                 // search rows of the chunk
    const int dy0 = -R + chunk * rows;
    const int wrows = ctu_window_rows(dyw), pitch = ctu_pitch(R), nd = 2 * R;
    uint32_t *mvk = reinterpret_cast<uint32_t *>(smem);                      // [rows][nd] MV-cost keys
    uint2 *win = reinterpret_cast<uint2 *>(smem + ctu_key_bytes(R, dyw));    // the window's entries
    const int plane = ctu_plane(R, dyw);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // reference window: rows y0+dy0 .., columns x0-R .. (64 + 2R), clamped into the plane
    const uint8_t *ref = refs[job.ref];
    const int wx0 = job.x0 - R, wy0 = job.y0 + dy0;
    const bool inside = wx0 >= -kPad && wx0 + 64 + 2 * R <= g.W + kPad && wy0 >= -kPad && wy0 + wrows <= g.H + kPad &&
                        (g.stride & 15) == 0 && ((uintptr_t)(ref + (ptrdiff_t)wy0 * g.stride + wx0) & 15) == 0;
    // staging area after the window (128-byte aligned when the dynamic shared
    // memory base is), the barrier after it; the launch does not give it
    // where that would cost a CTA per SM
    uint8_t *stage = smem + ctu_key_bytes(R, dyw) + ctu_win_bytes(R, dyw);
    const int np = tma_pieces(R);
    const uint32_t stage_s = smem_u32(stage), bar_s = stage_s + (uint32_t)(np * kTmaPieceBytes);
    uint32_t dyn_smem;
    asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dyn_smem));
    const bool staged = XG_CTU_TMA && (uint32_t)(stage - smem) + (uint32_t)(np * kTmaPieceBytes) + 16u <= dyn_smem;
    bool use_tma = false;
    if (view.tmap != nullptr && staged && inside && (stage_s & 127) == 0) {
        const ptrdiff_t off = (ref + (ptrdiff_t)wy0 * g.stride + wx0) - view.pool;
        const int tz = (int)(off / (ptrdiff_t)view.plane_bytes);
        const ptrdiff_t rem = off - (ptrdiff_t)tz * view.plane_bytes;
        const int ty = (int)(rem / g.stride);
        const int tx = (int)(rem - (ptrdiff_t)ty * g.stride);
        use_tma = off >= 0 && (tx & 15) == 0;
        if (use_tma && tid == 0) tma_window_issue(view.tmap, stage_s, bar_s, tx, ty, tz, np);
    }
    __syncthreads();   // the barrier's initialisation, before any thread polls it

    // MV cost keys of this chunk's displacements (uniform over the CTU)
    for (int row = warp; row < rows; row += kCtuWarps)
        for (int dxr = lane; dxr < nd; dxr += 32) {
            const uint32_t mvc = (uint32_t)mv_cost_hd(lambda, (dxr - R) * 4, (dy0 + row) * 4, job.mvp_x, job.mvp_y);
            mvk[row * nd + dxr] = (mvc << 11) | ((uint32_t)(row & (dyw - 1)) << 8) | (uint32_t)dxr;
        }
    // the window's entries, a row per warp
    if (use_tma) {
        const bool ok = mbar_wait_bounded(bar_s, 0);
        if (__syncthreads_or(!ok)) {
            // the copy did not land: record it, give the copies in flight
            // one more bounded wait, and leave this chunk unsearched
            if (tid == 0 && view.wait_flag) atomicOr(view.wait_flag, 1u);
            mbar_wait_bounded(bar_s, 0);
            return;
        }
    } else if (staged && !inside) {
        for (int r = warp; r < wrows; r += kCtuWarps) {
            const uint8_t *row = ref + (ptrdiff_t)min(max(wy0 + r, -kPad), g.H + kPad - 1) * g.stride;
            for (int c = lane; c < 64 + 2 * R; c += 32)
                stage[ctu_stage_at(r, c)] = row[min(max(wx0 + c, -kPad), g.W + kPad - 1)];
        }
        __syncthreads();
    }
    // four entries per item, the words of several items read before any is
    // placed (one item at a time waited for memory 40 times over)
    const bool from_stage = use_tma || (staged && !inside);
    const int quads = ctu_quads(pitch), items = wrows * quads, mq = (65536 + quads - 1) / quads;
    auto place = [&](int r, int k, uint32_t lo, uint32_t hi) {
        if (k >= pitch) return;
        uint2 *d = win + ctu_entry(r, pitch) + k;
        d[0] = make_uint2(lo, __byte_perm(lo, hi, 0x4321));
        d[plane] = make_uint2(__byte_perm(lo, hi, 0x5432), __byte_perm(lo, hi, 0x6543));
    };
    if (from_stage || inside) {
        constexpr int NB = 4;
        for (int e0 = tid; e0 < items; e0 += NB * kCtuThreads) {
            uint4 v[NB];
            uint32_t nx[NB];
#pragma unroll
            for (int b = 0; b < NB; b++) {
                const int e = min(e0 + b * kCtuThreads, items - 1), r = (e * mq) >> 16, q = e - r * quads;
                const int after = ctu_quad_full(q, pitch) ? 16 : 0;   // where there is no word after, any in its place
                if (from_stage) {
                    v[b] = *reinterpret_cast<const uint4 *>(stage + ctu_stage_at(r, 16 * q));
                    nx[b] = *reinterpret_cast<const uint32_t *>(stage + ctu_stage_at(r, 16 * q + after));
                } else {
                    const uint4 *t = reinterpret_cast<const uint4 *>(ref + (ptrdiff_t)(wy0 + r) * g.stride + wx0) + q;
                    v[b] = __ldg(t);
                    nx[b] = __ldg(reinterpret_cast<const uint32_t *>(t) + after / 4);
                }
            }
#pragma unroll
            for (int b = 0; b < NB; b++) {
                const int e = e0 + b * kCtuThreads, r = (e * mq) >> 16, k = 4 * (e - r * quads);
                if (e >= items) break;
                place(r, k, v[b].x, v[b].y);
                place(r, k + 1, v[b].y, v[b].z);
                place(r, k + 2, v[b].z, v[b].w);
                place(r, k + 3, v[b].w, nx[b]);
            }
        }
    } else {
        for (int r = warp; r < wrows; r += kCtuWarps) {
            const uint8_t *row = ref + (ptrdiff_t)min(max(wy0 + r, -kPad), g.H + kPad - 1) * g.stride;
            for (int k = lane; k < pitch; k += 32) {
                uint32_t w[2] = {0, 0};
#pragma unroll
                for (int b = 0; b < 8; b++)
                    w[b >> 2] |= (uint32_t)row[min(max(wx0 + 4 * k + b, -kPad), g.W + kPad - 1)] << (8 * (b & 3));
                place(r, k, w[0], w[1]);
            }
        }
    }
    __syncthreads();

    LaneRole L;
    L.half = lane & 1;
    L.rx = ((lane >> 1) & 1) + 2 * ((lane >> 3) & 1);
    L.ry = ((lane >> 2) & 1) + 2 * (lane >> 4);
    L.nh = -L.half;
    const int half = L.half, rx = L.rx, ry = L.ry;
    const int qx = rx & 1, qy = ry & 1, id = ry * 8 + rx * 2 + half;
    // current block: 8 rows x 16 pixels of this half-region
    uint32_t cw[8][4];
    {
        const uint8_t *o = cur + (ptrdiff_t)(job.y0 + 16 * ry + 8 * half) * g.stride + job.x0 + 16 * rx;
#pragma unroll
        for (int r = 0; r < 8; r++) {
            const uint4 v = *reinterpret_cast<const uint4 *>(o + (ptrdiff_t)r * g.stride);
            cw[r][0] = v.x; cw[r][1] = v.y; cw[r][2] = v.z; cw[r][3] = v.w;
        }
    }
#pragma unroll
    for (int k = 0; k < 4; k++) L.c32[k] = c_c32[half][qx][qy][k];
#pragma unroll
    for (int k = 0; k < 3; k++) L.c64[k] = c_c64[id][k];
    // shuffle partners: region pairs along the axis this half works on (lane
    // bits: 1 rx0, 2 ry0, 3 rx1, 4 ry1)
    L.pr1 = half ? 4 : 2;     // 32-CU pair (vertical for half 1, horizontal for half 0)
    L.pr2 = half ? 2 : 4;     // the other 32-CU row/column
    L.pr3 = half ? 16 : 8;    // 64-CU row / column sums
    L.pr4 = half ? 2 : 4;     // 64-CU pairs
    L.pr5 = half ? 8 : 16;    // 64-CU total
    L.bx0 = job.x0 + 16 * rx;
    L.by0 = job.y0 + 16 * ry + 8 * half;
    const int32_t *smap = slots + (size_t)job.slot_base;
    const int cu32 = (ry >> 1) * 2 + (rx >> 1);
    const int lm[3] = {c_m32[half][qx][qy][0], c_m32[half][qx][qy][1], c_m64[id]};

    uint32_t ks[25], kl[3];
    auto clear = [&]() {
#pragma unroll
        for (int k = 0; k < 25; k++) ks[k] = 0xffffffffu;
#pragma unroll
        for (int k = 0; k < 3; k++) kl[k] = 0xffffffffu;
    };
    // the warp's minima into the global keys; order(row, dxr) is the visit
    // order.  The slots are read before any of them is needed.
    auto merge = [&](auto order) {
        int pus[25], pul[3];
#pragma unroll
        for (int k = 0; k < 25; k++)
            if ((LV & 1) || k >= 18) pus[k] = smap[small_slot(rx, ry, half, k)];
#pragma unroll
        for (int k = 0; k < 3; k++) pul[k] = lm[k] < 0 ? -1 : smap[k < 2 ? 784 + cu32 * 13 + lm[k] : 836 + lm[k]];
#pragma unroll
        for (int k = 0; k < 25; k++) {
            if (!(LV & 1) && k < 18) continue;
            const uint32_t cost = ks[k] >> 11;
            if (cost < kPoisonSmall && pus[k] >= 0)
                atomicMin(&keys[pus[k]], ((unsigned long long)cost << 32) | order((ks[k] >> 8) & 7u, ks[k] & 0xffu));
        }
#pragma unroll
        for (int k = 0; k < 3; k++) {
            const uint32_t cost = kl[k] >> 11;
            if (cost < kCapLarge && pul[k] >= 0)
                atomicMin(&keys[pul[k]], ((unsigned long long)cost << 32) | order((kl[k] >> 8) & 7u, kl[k] & 0xffu));
        }
    };
    clear();
    const int q8 = 16 * ry + 8 * half;   // the half-region's first row

    // The search candidate (0,0) is visited before the window (me.c:913-917):
    // its cost enters with visit order 0, so it wins every tie.  The CTA whose
    // rows contain dy = 0 evaluates it (warp 0).
    if (warp == 0 && dy0 <= 0 && 0 < dy0 + rows) {
        uint32_t raw[2][4];
        sad_at(win + ((R >> 1) & 1) * plane, pitch, q8 - dy0, 4 * rx + (R >> 2), cw, raw);   // R is even
        const uint32_t mvc0 = (uint32_t)mv_cost_hd(lambda, 0, 0, job.mvp_x, job.mvp_y);
        bool b0 = true, b1 = true;
        if (BORDER) {
            b0 = L.by0 >= -kLimitMargin && L.by0 + 4 <= g.H + kLimitMargin;
            b1 = L.by0 + 4 >= -kLimitMargin && L.by0 + 8 <= g.H + kLimitMargin;
        }
        fold_displacement<BORDER, LV>(L, raw, mvc0 << 11, 0, b0, b1, g, ks, kl);
        merge([](uint32_t, uint32_t) { return 0u; });
        clear();
    }

    // two displacement rows per pass: window rows q8 + row .. + 8 are read
    // once; row r serves block row r of the first displacement row and block
    // row r - 1 of the second
    const int dyw0 = dy0 + warp * dyw;
    for (int rr = 0; rr < dyw; rr += 2) {
        const int row = warp * dyw + rr;
        const int dy = dy0 + row;
        if (dy >= R) break;     // 2R and dyw are even: a pair is all in or all out
        uint32_t rp[9];   // the window rows' shared-memory addresses
#pragma unroll
        for (int r = 0; r < 9; r++) rp[r] = smem_u32(win + ctu_entry(q8 + row + r, pitch) + 4 * rx);
        const uint2 *mk = reinterpret_cast<const uint2 *>(mvk + row * nd);
#pragma unroll 1
        for (uint32_t j = 0, step = 8u * plane; j < (uint32_t)R; j++) {   // displacements 2j and 2j + 1
            uint32_t s[2][2][2][4];     // [displacement row][displacement][block row][block column]
#pragma unroll
            for (int k = 0; k < 32; k++) s[k >> 4][(k >> 3) & 1][(k >> 2) & 1][k & 3] = 0;
#pragma unroll
            for (int r = 0; r < 9; r++) {
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    uint2 v;
                    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(rp[r] + 8 * c));
#pragma unroll
                    for (int i = 0; i < 2; i++) {
                        const int b = r - i;
                        if (b < 0 || b > 7) continue;
                        s[i][0][b >> 2][c] = sad4_acc(cw[b][c], v.x, s[i][0][b >> 2][c]);
                        s[i][1][b >> 2][c] = sad4_acc(cw[b][c], v.y, s[i][1][b >> 2][c]);
                    }
                }
                rp[r] += step;
            }
            step = 8u - step;   // to the other plane and back one entry further
#pragma unroll
            for (int i = 0; i < 2; i++)
                fold_group<BORDER, LV>(L, s[i], mk[i * R + j], 2 * j, R, dy + i, job, g, ks, kl);
        }
    }
    merge([&](uint32_t row, uint32_t dxr) { return (uint32_t)(2 + (dyw0 + (int)row + R) * nd + (int)dxr); });
}

// CU sizes with separate compiled folds (serving's leaf CUs often have no
// 8x8 / 16x16 CU in a CTU): 1 on, 0 every job with the full fold
#ifndef XG_CTU_LEVELS
#define XG_CTU_LEVELS 1
#endif

template <bool BORDER>
__global__ void __launch_bounds__(kCtuThreads, XG_CTU_MINB)
    fs_ctu_kernel(const CtuJob *__restrict__ jobs, int nchunks, int dyw, const SessView *__restrict__ views, int R,
                  int lambda)
{
    extern __shared__ __align__(16) uint8_t smem[];
    const int job_idx = blockIdx.x / nchunks, chunk = blockIdx.x % nchunks;
    const CtuJob job = jobs[job_idx];
    if (BORDER != (job.border != 0)) return;
#if XG_CTU_LEVELS
    if (job.levels & 1) ctu_search<BORDER, 15>(job, chunk, dyw, views, R, lambda, smem);
    else if (job.levels & 2) ctu_search<BORDER, 14>(job, chunk, dyw, views, R, lambda, smem);
    else ctu_search<BORDER, 12>(job, chunk, dyw, views, R, lambda, smem);
#else
    ctu_search<BORDER, 15>(job, chunk, dyw, views, R, lambda, smem);
#endif
}

// ---- host planning -----------------------------------------------------------------
static inline void ctu_plan_free(CtuPlan &p)
{
    if (p.d_jobs) cudaFree(p.d_jobs);
    if (p.d_slots) cudaFree(p.d_slots);
    p = CtuPlan();
}

// Splits a PU list into CTU jobs and the rest (`generic`).  A PU joins its
// CTU's job when it sits on one of the CTU's slots, its MVP rounds to (0,0)
// (so the search centre is (0,0)), all PUs of the job share that MVP, and
// inside the (2R)^2 window its limits allow exactly the displacements the
// edge rule allows.
static inline bool same_range_in_window(int lo, int hi, int rule_lo, int rule_hi, int R)
{
    return max(lo, -R) == max(rule_lo, -R) && min(hi, R - 1) == min(rule_hi, R - 1);
}

static void ctu_plan_build(CtuPlan &p, const std::vector<xavs2gpu_pu_t> &pus, int W, int H, int nrefs, int R,
                           bool allow, std::vector<int> &generic, cudaStream_t st)
{
    const SlotTable &table = slot_table();
    const int cw = (W + 63) / 64, ch = (H + 63) / 64;
    const int ngroups = cw * ch * nrefs;
    std::vector<int> group_job(ngroups, -1);
    std::vector<CtuJob> jobs;
    std::vector<int32_t> slots;
    generic.clear();
    // the CTU kernel takes even ranges (odd R: every PU per-PU): displacements in
    // pairs from -R on, an entry each, so that displacement 0 begins one, and
    // search rows in pairs
    const bool range_ok = allow && R % 2 == 0;
    for (int i = 0; i < (int)pus.size(); i++) {
        const xavs2gpu_pu_t &u = pus[i];
        const int w = h_pu_w[u.part], h = h_pu_h[u.part];
        bool ok = range_ok && ((u.mvp_x + 2) >> 2) == 0 && ((u.mvp_y + 2) >> 2) == 0 && !(u.x & 3) && !(u.y & 3);
        // (0,0) must be inside the limits for it to be the centre
        ok = ok && u.min_x <= 0 && u.max_x >= 0 && u.min_y <= 0 && u.max_y >= 0;
        ok = ok && same_range_in_window(u.min_x, u.max_x, -kLimitMargin - u.x, W + kLimitMargin - u.x - w, R) &&
             same_range_in_window(u.min_y, u.max_y, -kLimitMargin - u.y, H + kLimitMargin - u.y - h, R);
        const int s = ok ? table.t[u.part][(u.y & 63) >> 2][(u.x & 63) >> 2] : -1;
        if (s < 0) { generic.push_back(i); continue; }
        const int gidx = ((u.y >> 6) * cw + (u.x >> 6)) * nrefs + u.ref;
        int j = group_job[gidx];
        if (j < 0) {
            j = (int)jobs.size();
            group_job[gidx] = j;
            CtuJob cj;
            cj.x0 = (int16_t)(u.x & ~63); cj.y0 = (int16_t)(u.y & ~63); cj.ref = u.ref;
            cj.levels = 0;
            cj.mvp_x = u.mvp_x; cj.mvp_y = u.mvp_y;
            // can the edge rule bind for any block of this CTU inside the window?
            cj.border = (cj.x0 - R < -kLimitMargin || cj.x0 + 64 + R > W + kLimitMargin ||
                         cj.y0 - R < -kLimitMargin || cj.y0 + 64 + R > H + kLimitMargin) ? 1 : 0;
            cj.sess = 0;
            cj.slot_base = j * kSlots;
            jobs.push_back(cj);
            slots.resize(slots.size() + kSlots, -1);
        }
        CtuJob &cj = jobs[j];
        int32_t &slot = slots[(size_t)cj.slot_base + s];
        if (cj.mvp_x != u.mvp_x || cj.mvp_y != u.mvp_y || slot >= 0) { generic.push_back(i); continue; }
        slot = i;
        cj.levels |= (uint8_t)(s < 576 ? 1 : s < 784 ? 2 : s < 836 ? 4 : 8);
    }
    if ((int)jobs.size() > p.cap_jobs) {
        if (p.d_jobs) cudaFree(p.d_jobs);
        if (p.d_slots) cudaFree(p.d_slots);
        p.cap_jobs = (int)jobs.size() + 16;
        XG_CUDA(cudaMalloc((void **)&p.d_jobs, sizeof(CtuJob) * p.cap_jobs));
        XG_CUDA(cudaMalloc((void **)&p.d_slots, sizeof(int32_t) * kSlots * p.cap_jobs));
    }
    p.n_jobs = (int)jobs.size();
    p.n_border = 0;
    for (const CtuJob &j : jobs) p.n_border += j.border ? 1 : 0;
    p.h_jobs = jobs;
    if (p.n_jobs) {
        XG_CUDA(cudaMemcpyAsync(p.d_jobs, jobs.data(), sizeof(CtuJob) * p.n_jobs, cudaMemcpyHostToDevice, st));
        XG_CUDA(cudaMemcpyAsync(p.d_slots, slots.data(), sizeof(int32_t) * slots.size(), cudaMemcpyHostToDevice, st));
        XG_CUDA(cudaStreamSynchronize(st));
    }
}

constexpr int kCtuSmemMax = 227 * 1024;

// The kernels' dynamic shared-memory limit (the largest range's need), once
// per device; launches and occupancy queries come after it.
static void ctu_attrs(int dev)
{
    static std::atomic<bool> done[64];
    if (dev < 0 || dev >= 64 || done[dev].load(std::memory_order_acquire)) return;
    const int maxb = kCtuSmemMax;
    XG_CUDA(cudaFuncSetAttribute(fs_ctu_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, maxb));
    XG_CUDA(cudaFuncSetAttribute(fs_ctu_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, maxb));
    done[dev].store(true, std::memory_order_release);
}

// What a launch at range R with dyw search rows per warp runs with: its
// dynamic shared memory (the TMA staging area included where it costs no CTA
// per SM; the CTAs fill their windows with word loads without it) and the
// CTAs an SM holds.  Kept per device and range.
struct CtuFit {
    int smem = 0, ctas = 0;
};
static CtuFit ctu_fit(int dev, int R, int dyw)
{
    static std::atomic<int> known[64][129][3];   // smem << 4 | ctas (threads agree)
    const int with = (int)ctu_smem_bytes(R, dyw, true), base = (int)ctu_smem_bytes(R, dyw, false);
    CtuFit f;
    const bool keep = dev >= 0 && dev < 64 && R >= 1 && R <= 128;
    std::atomic<int> *slot = keep ? &known[dev][R][dyw == 8 ? 2 : dyw == 4 ? 1 : 0] : nullptr;
    const int v = slot ? slot->load(std::memory_order_relaxed) : 0;
    if (v) {
        f.smem = v >> 4;
        f.ctas = v & 15;
        return f;
    }
    ctu_attrs(dev);
    auto resident = [](int bytes) {
        int a = 0, b = 0;
        if (bytes > kCtuSmemMax) return 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, fs_ctu_kernel<false>, kCtuThreads, bytes) != cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, fs_ctu_kernel<true>, kCtuThreads, bytes) != cudaSuccess) {
            cudaGetLastError();
            return 0;
        }
        return std::min(std::min(a, b), 15);
    };
    const int n0 = resident(base), n1 = XG_CTU_TMA ? resident(with) : 0;
    f.smem = n1 > 0 && n1 >= n0 ? with : base;
    f.ctas = std::max(n0, n1);
    if (slot) slot->store(f.smem << 4 | f.ctas, std::memory_order_relaxed);
    return f;
}

// Search rows per warp: 8, 4 or 2 (a CTA's chunk is four times that).  More
// rows share a window and a final merge; fewer make a smaller window, which
// lets an SM hold more CTAs (R = 64: 2 at 8 rows, 3 at 4; R = 128: 1, 2 at 2),
// and more CTAs.  So: the most rows at which an SM holds the most CTAs, halved while
// the launch is below two rounds of the GPU.  Measured, one reference, us at 8 /
// 4 / 2 rows: 1080p R = 64 1440 / 1357 / 1360, R = 32 352 / 356 / 384, R = 16
// 112 / 106 / 119; 720p R = 16 98 / 78 / 74; 416x240 R = 16 41 / 28 / 20,
// R = 64 210 / 153 / 112; 1080p R = 128 6848 / 6972 / 5617.
#ifndef XG_CTU_DYW
#define XG_CTU_DYW 0   // 0: by the rule
#endif
static int ctu_rows(int dev, int R, int n_jobs)
{
    if (XG_CTU_DYW) return XG_CTU_DYW;
    int dyw = kDyWarpMax;
    for (int d = dyw / 2; d >= 2; d /= 2)
        if (ctu_fit(dev, R, d).ctas > ctu_fit(dev, R, dyw).ctas) dyw = d;
    const long long slots = (long long)sm_count() * ctu_fit(dev, R, dyw).ctas;
    auto chunks = [&](int d) { return (2 * R + kCtuWarps * d - 1) / (kCtuWarps * d); };
    while (dyw > 2 && (long long)n_jobs * chunks(dyw) < 2 * slots) dyw /= 2;
    return dyw;
}

// Run the border variant on a side stream forked from the caller's, so its
// CTAs fill the SMs the interior launch's last wave leaves idle (and the
// reverse); joined back before the call returns.
#ifndef XG_CTU_FORK
#define XG_CTU_FORK 1
#endif

// A side stream and its fork / join events, per host thread and device
// (a thread's launches are sequenced, so they may share them; the fork and
// the join happen within one call, so stream capture sees a complete
// fork-join).
struct CtuSide {
    cudaStream_t st = nullptr;
    cudaEvent_t fork = nullptr, join = nullptr;
    ~CtuSide()   // at thread exit (a pool's threads do not keep theirs)
    {
        if (join) cudaEventDestroy(join);
        if (fork) cudaEventDestroy(fork);
        if (st) cudaStreamDestroy(st);
    }
};
// Side stream k (0 the search's own, 1 the per-PU search's, 2 the per-PU
// search's second) for launches beside `st`, or null: the launches then stay
// on st.
static CtuSide *ctu_side(int dev, cudaStream_t st, int k = 0)
{
    thread_local CtuSide side[3][64];
    if (dev < 0 || dev >= 64 || k < 0 || k > 2) return nullptr;
    CtuSide &s = side[k][dev];
    if (!s.st) {
        if (cudaStreamCreateWithFlags(&s.st, cudaStreamNonBlocking) != cudaSuccess ||
            cudaEventCreateWithFlags(&s.fork, cudaEventDisableTiming) != cudaSuccess ||
            cudaEventCreateWithFlags(&s.join, cudaEventDisableTiming) != cudaSuccess) {
            cudaGetLastError();
            return nullptr;
        }
    }
    return side_usable(st, s.st) ? &s : nullptr;
}

// Creates what a search at range R launches with on this thread -- the side
// stream and the shared-memory choices -- ahead of a stream capture.
static void ctu_prime(int R)
{
    const int dev = current_device();
    if (XG_CTU_FORK) {
        for (int k = 0; k < 3; k++) ctu_side(dev, nullptr, k);
    }
    if (R < 1 || R > 128) return;
    for (int dyw = 2; dyw <= kDyWarpMax; dyw *= 2) ctu_fit(dev, R, dyw);
}

// One launch of each variant over `n_jobs` jobs (sessions per job.sess).
// n_border of the jobs need the border variant; a variant with no job of
// its kind is not launched.
static void ctu_jobs_run(const CtuJob *d_jobs, int n_jobs, int n_border, const SessView *d_views,
                         const xavs2gpu_me_params_t &prm, cudaStream_t st)
{
    if (n_jobs == 0) return;
    const int R = prm.search_range;
    const int dev = current_device();
    ctu_attrs(dev);
    const int dyw = ctu_rows(dev, R, n_jobs), rows = kCtuWarps * dyw;
    const size_t smem = (size_t)ctu_fit(dev, R, dyw).smem;
    const int nchunks = (2 * R + rows - 1) / rows;
    const int grid = n_jobs * nchunks;
    const int lam = prm.lambda_factor;
    // the border launch on the side stream when both variants run
    CtuSide *side = XG_CTU_FORK && n_border > 0 && n_border < n_jobs ? ctu_side(dev, st) : nullptr;
    cudaStream_t bst = st;
    if (side) {
        XG_CUDA(cudaEventRecord(side->fork, st));
        XG_CUDA(cudaStreamWaitEvent(side->st, side->fork, 0));
        bst = side->st;
    }
    if (n_border < n_jobs) {
        fs_ctu_kernel<false><<<grid, kCtuThreads, smem, st>>>(d_jobs, nchunks, dyw, d_views, R, lam);
        count_launch();
    }
    if (n_border > 0) {
        fs_ctu_kernel<true><<<grid, kCtuThreads, smem, bst>>>(d_jobs, nchunks, dyw, d_views, R, lam);
        count_launch();
    }
    if (side) {
        XG_CUDA(cudaEventRecord(side->join, side->st));
        XG_CUDA(cudaStreamWaitEvent(st, side->join, 0));
    }
}

}  // namespace xg
