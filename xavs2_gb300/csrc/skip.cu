// skip.cu -- rough cost of skip / direct candidates for sm_103a
// (cu_check_skip_direct_rough2, encoder/rdo.c:2395-2480): for every
// candidate of a CU its prediction from the resident sub-pel planes of a
// motion-search session (one list or the average of two, pixel_avg,
// pixel.c:680-719), the SA8D of the luma prediction against the source
// (pixf.sa8d, pixel.c:416-530) and rdcost = distortion + lambda * rate
// (rdcost_t, double); per CU the first candidate with the strictly smallest
// rdcost.  A candidate whose motion equals an earlier candidate's of the
// same CU is not evaluated (update_skip_mv_list, rdo.c:2366-2389).
#include "xavs2gpu_common.cuh"

#include <algorithm>

namespace xg {
namespace skp {

constexpr int kPad = 80;   // plane margin of a session (XAVS2_PAD, defines.h:298)

struct Ctx {
    const uint8_t *cur;
    const uint8_t *const *planes;   // 16 r + k
    int stride, W, H, nrefs;
    const xavs2gpu_skip_cand_t *cands;
    int n;
    double lambda;
    int32_t *dist;
    double *cost;
};

// motion of two candidates equal (the n_pu PUs' references and vectors)
__device__ __forceinline__ bool same_motion(const xavs2gpu_skip_cand_t &a, const xavs2gpu_skip_cand_t &b)
{
    if (a.n_pu != b.n_pu) return false;
    for (int q = 0; q < a.n_pu; q++)
        for (int l = 0; l < 2; l++) {
            if (a.ref[q][l] != b.ref[q][l]) return false;
            if (a.ref[q][l] >= 0 && (a.mv[q][l][0] != b.mv[q][l][0] || a.mv[q][l][1] != b.mv[q][l][1])) return false;
        }
    return true;
}

// a PU's prediction stays inside the planes' margin
__device__ __forceinline__ bool pu_inside(const Ctx &c, int x, int y, int w, int h, int ref, int mvx, int mvy)
{
    if (ref < 0) return true;
    if (ref >= c.nrefs) return false;
    const int px = x + (mvx >> 2), py = y + (mvy >> 2);
    return px >= -kPad && py >= -kPad && px + w <= c.W + kPad && py + h <= c.H + kPad;
}

// Validity of a candidate (shape, inside the picture, every PU with a list,
// references inside the session and their blocks inside the planes'
// margin) and the encoder's repeated-motion check against the earlier
// candidates of the same CU.
__device__ bool cand_ok(const Ctx &c, int i, const xavs2gpu_skip_cand_t &k)
{
    const int S = 1 << k.size_log2;
    if (k.size_log2 < 3 || k.size_log2 > 6 || (k.n_pu != 1 && k.n_pu != 4) || k.x < 0 || k.y < 0 ||
        k.x + S > c.W || k.y + S > c.H)
        return false;
    const int hp = k.n_pu == 4 ? S >> 1 : S;
    for (int q = 0; q < k.n_pu; q++) {
        if (k.ref[q][0] < 0 && k.ref[q][1] < 0) return false;
        for (int l = 0; l < 2; l++)
            if (!pu_inside(c, k.x + (q & 1) * hp, k.y + (q >> 1) * hp, hp, hp, k.ref[q][l], k.mv[q][l][0],
                           k.mv[q][l][1]))
                return false;
    }
    for (int j = i - 1; j >= 0; j--) {
        const xavs2gpu_skip_cand_t &e = c.cands[j];
        if (e.cu != k.cu) break;
        if (same_motion(e, k)) return false;
    }
    return true;
}

// Prediction source of one PU: per list the address of the PU's top-left
// prediction sample in the sub-pel plane of its fractional vector.
struct PuSrc {
    const uint8_t *p[2];
    int n;
};
__device__ __forceinline__ PuSrc pu_src(const Ctx &c, const xavs2gpu_skip_cand_t &k, int q, int X, int Y)
{
    PuSrc s{{nullptr, nullptr}, 0};
    for (int l = 0; l < 2; l++) {
        const int r = k.ref[q][l];
        if (r < 0) continue;
        const int mx = k.mv[q][l][0], my = k.mv[q][l][1];
        s.p[s.n++] = c.planes[16 * r + ((my & 3) << 2) + (mx & 3)] + (long long)(Y + (my >> 2)) * c.stride + X +
                     (mx >> 2);
    }
    if (s.n == 1) s.p[1] = s.p[0];
    return s;
}

// 4 samples at any byte address, from the two aligned words holding them
// (the word after the last sample is read too: planes and pictures have an
// 80-sample margin, so it is inside the allocation)
__device__ __forceinline__ uint32_t ld4u(const uint8_t *p)
{
    const uintptr_t a = reinterpret_cast<uintptr_t>(p);
    const uint32_t *w = reinterpret_cast<const uint32_t *>(a & ~(uintptr_t)3);
    return __funnelshift_r(w[0], w[1], (unsigned)(a & 3) * 8u);
}

// bytewise (a + b + 1) >> 1 of four packed samples (pixel_avg, pixel.c:680-700)
__device__ __forceinline__ uint32_t avg4(uint32_t a, uint32_t b) { return (a | b) - (((a ^ b) >> 1) & 0x7F7F7F7Fu); }

// |H8 (src - pred) H8^T| of the 8x8 block at (X, Y), predicted by candidate
// k's PU `pu`, or (QUAD) by its four 4x4 PUs, the block's quadrants.
// Rows are read as words: the current block's aligned, the prediction's at
// any alignment.
// Samples k and k + 4 of a row share an integer (hi * 2^16 + lo, signed), so a
// plain add or subtract is one butterfly of both; the last stage, across the
// two halves, is |a + b| + |a - b| = 2 max(|a|, |b|), taken of two integers'
// halves at a time with the values (at most 8160 before it) biased to unsigned.
// Half the instructions and registers of 64 separate samples.
constexpr uint32_t kSkipBias = 0x20002000u;
__device__ __forceinline__ void byte_pairs(uint32_t lo, uint32_t hi, uint32_t (&q)[4])
{
    const uint32_t t = __byte_perm(lo, hi, 0x5140), u = __byte_perm(lo, hi, 0x7362);   // b0 b4 b1 b5 | b2 b6 b3 b7
    q[0] = __byte_perm(t, 0, 0x7170);
    q[1] = __byte_perm(t, 0, 0x7372);
    q[2] = __byte_perm(u, 0, 0x7170);
    q[3] = __byte_perm(u, 0, 0x7372);
}
__device__ __forceinline__ void butterfly(uint32_t &a, uint32_t &b)
{
    const uint32_t s = a + b;
    b = a - b;
    a = s;
}

template <bool QUAD>
__device__ int hsum8_pred(const Ctx &c, const xavs2gpu_skip_cand_t &k, int X, int Y, int pu)
{
    uint32_t m[8][4];   // [row][k]: columns k and k + 4
    PuSrc src[2];       // of the block, or of the quadrants of rows y .. y + 3
    if (!QUAD) src[0] = pu_src(c, k, pu, X, Y);
#pragma unroll
    for (int y = 0; y < 8; y++) {
        // the current picture is the session's plane: stride a multiple of
        // 64, origin 16-byte aligned, X a multiple of 8
        const uint2 cw = *reinterpret_cast<const uint2 *>(c.cur + (long long)(Y + y) * c.stride + X);
        const uint32_t c0 = cw.x, c1 = cw.y;
        uint32_t pw[2];
        if (QUAD) {
            if ((y & 3) == 0)
#pragma unroll
                for (int h = 0; h < 2; h++) src[h] = pu_src(c, k, (y >> 2) * 2 + h, X + 4 * h, Y + y);
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const PuSrc &ps = src[h];
                const long long o = (long long)(y & 3) * c.stride;
                const uint32_t a = ld4u(ps.p[0] + o);
                pw[h] = ps.n == 2 ? avg4(a, ld4u(ps.p[1] + o)) : a;   // one list: the plane's samples
            }
        } else {
            // the row's 8 prediction samples from the 3 aligned words holding them
            auto ld8u = [&](const uint8_t *q, uint32_t &lo, uint32_t &hi) {
                const uintptr_t a = reinterpret_cast<uintptr_t>(q);
                const uint32_t *w = reinterpret_cast<const uint32_t *>(a & ~(uintptr_t)3);
                const unsigned sh = (unsigned)(a & 3) * 8u;
                const uint32_t w0 = w[0], w1 = w[1], w2 = w[2];
                lo = __funnelshift_r(w0, w1, sh);
                hi = __funnelshift_r(w1, w2, sh);
            };
            const long long o = (long long)y * c.stride;
            ld8u(src[0].p[0] + o, pw[0], pw[1]);
            if (src[0].n == 2) {
                uint32_t b0, b1;
                ld8u(src[0].p[1] + o, b0, b1);
                pw[0] = avg4(pw[0], b0);
                pw[1] = avg4(pw[1], b1);
            }
        }
        uint32_t cq[4], pq[4];
        byte_pairs(c0, c1, cq);
        byte_pairs(pw[0], pw[1], pq);
#pragma unroll
        for (int x = 0; x < 4; x++) m[y][x] = cq[x] - pq[x];
        butterfly(m[y][0], m[y][1]);
        butterfly(m[y][2], m[y][3]);
        butterfly(m[y][0], m[y][2]);
        butterfly(m[y][1], m[y][3]);
    }
    uint32_t s = 0;
#pragma unroll
    for (int x = 0; x < 4; x++) {
#pragma unroll
        for (int d = 1; d < 8; d <<= 1)
#pragma unroll
            for (int y = 0; y < 8; y++)
                if (!(y & d)) butterfly(m[y][x], m[y + d][x]);
#pragma unroll
        for (int y = 0; y < 8; y += 2) {
            const uint32_t u = m[y][x] + kSkipBias, v = m[y + 1][x] + kSkipBias;
            const uint32_t a = __byte_perm(u, v, 0x5410), b = __byte_perm(u, v, 0x7632);
            s = __dp2a_lo(__vmaxu2(__vmaxu2(a, b), 2 * kSkipBias - __vminu2(a, b)), 0x0101u, s);
        }
    }
    return 2 * ((int)s - 32 * 0x2000);
}

// Candidate classes: by CU size (0..3: 8x8 .. 64x64), the 8x8 CUs with four 4x4
// PUs by themselves (4: their code reads quadrants, and a warp that held both
// kinds ran both).
constexpr int kClasses = 5;
__device__ __forceinline__ int class_of(const xavs2gpu_skip_cand_t &k)
{
    const int sl = k.size_log2;
    if (sl < 3 || sl > 6) return -1;
    return sl == 3 && k.n_pu == 4 ? 4 : sl - 3;
}
__device__ __forceinline__ int class_lanes(int cl) { return cl == 4 ? 1 : min(32, 1 << (2 * cl)); }

// 1. per-class counts (warp-aggregated); malformed candidates are reported here
__global__ void skip_count_kernel(Ctx c, int *__restrict__ counts)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    int cl = -1;
    if (i < c.n) {
        cl = class_of(c.cands[i]);
        if (cl < 0) {
            c.dist[i] = -1;
            c.cost[i] = (double)(1LL << 50);
        }
    }
    const unsigned valid = __ballot_sync(0xffffffffu, cl >= 0);
    if (cl >= 0) {
        const unsigned same = __match_any_sync(valid, cl);
        if ((threadIdx.x & 31) == __ffs(same) - 1) atomicAdd(&counts[cl], __popc(same));
    }
}

// 2. scatter into class order; a candidate that is not evaluated enters as ~i.
// (The comparison with the CU's earlier candidates is a chain of dependent
// reads: here a thread per candidate hides it, in the cost kernel it stood
// before every warp's gathers.)
__global__ void skip_scatter_kernel(Ctx c, const int *__restrict__ counts, int *__restrict__ cursor,
                                    int *__restrict__ sorted)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31;
    const int cl = i < c.n ? class_of(c.cands[i]) : -1;
    const unsigned valid = __ballot_sync(0xffffffffu, cl >= 0);
    if (cl < 0) return;
    const unsigned same = __match_any_sync(valid, cl);
    const int leader = __ffs(same) - 1;
    int base = 0;
    if (lane == leader) base = atomicAdd(&cursor[cl], __popc(same));
    const bool ok = cand_ok(c, i, c.cands[i]);
    __syncwarp(same);
    base = __shfl_sync(same, base, leader);
    int start = 0;
    for (int k = 0; k < cl; k++) start += counts[k];
    sorted[start + base + __popc(same & ((1u << lane) - 1))] = ok ? i : ~i;
}

// 3. costs: a warp takes 32 / L candidates of one class, L = min(32, number
// of 8x8 blocks) lanes each; lane s of a candidate takes 8x8 blocks s and
// s + 32 in z-order, so the four blocks of a 16x16 SA8D unit sit in four
// consecutive lanes (their sums are rounded together, pixel.c:470-500).
// The CTAs that fit walk the warps' worth of work, largest CUs first (the
// number of warps is known on the device alone: a grid for the most there
// could be, one per candidate, was 92 % empty CTAs for a 1080p picture).
// Bound by the latency of its plane gathers: XG_SKIP_MINB resident 128-thread
// CTAs (a 1080p picture's 214,500 candidates, whole call: 4 CTAs of 128
// registers 50.4 us, 6 48.8, 8 47.0; 110 before the classes, the walk, the
// repeated-motion check in the scatter and the paired transform).
#ifndef XG_SKIP_MINB
#define XG_SKIP_MINB 8
#endif
__global__ void __launch_bounds__(128, XG_SKIP_MINB) skip_cost_kernel(Ctx c, const int *__restrict__ counts,
                                                                      const int *__restrict__ sorted)
{
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    int cnt[kClasses];
#pragma unroll
    for (int k = 0; k < kClasses; k++) cnt[k] = counts[k];
    for (int item = warp;; item += gridDim.x * (blockDim.x >> 5)) {
        int cl = -1, pos = 0, end = 0;   // this warp's class, first list position, the class's end
        int first = 0;
#pragma unroll
        for (int t = 0; t < kClasses; t++) {
            const int k = t < 3 ? 3 - t : t == 3 ? 4 : 0;   // 64x64, 32x32, 16x16, 8x8 of four PUs, 8x8
            int start = 0;
#pragma unroll
            for (int j = 0; j < k; j++) start += cnt[j];
            const int L = class_lanes(k), groups = (cnt[k] * L + 31) / 32;
            if (cl < 0 && item < first + groups) {
                cl = k;
                pos = start + (item - first) * (32 / L);
                end = start + cnt[k];
            }
            first += groups;
        }
        if (cl < 0) return;
        const int L = class_lanes(cl), nsub = cl == 4 ? 1 : 1 << (2 * cl);
        const int slot = lane / L, sub = lane - slot * L;
        pos += slot;
        const bool live = pos < end;
        const int e = live ? sorted[pos] : -1, i = e < 0 ? ~e : e;
        const bool ok = e >= 0;
        // fields are read where they are used (a copy indexed by PU lives in
        // local memory); lane 0 of a warp is always live, i = 0 stands in for -1
        const xavs2gpu_skip_cand_t &k = c.cands[live ? i : 0];
        int acc = 0;
        const int hp = ok ? (1 << k.size_log2) >> (k.n_pu == 4) : 8;
        for (int s0 = 0; s0 < nsub; s0 += 32) {   // the same trip count for every lane of the warp
            const int s = s0 + sub;
            int h = 0;
            if (ok && s < nsub) {
                // z-order position of 8x8 block s
                int bx = 0, by = 0;
#pragma unroll
                for (int b = 0; b < 3; b++) {
                    bx |= ((s >> (2 * b)) & 1) << b;
                    by |= ((s >> (2 * b + 1)) & 1) << b;
                }
                const int X = k.x + 8 * bx, Y = k.y + 8 * by;
                if (cl == 4)
                    h = hsum8_pred<true>(c, k, X, Y, 0);
                else
                    h = hsum8_pred<false>(c, k, X, Y, k.n_pu == 4 ? (8 * bx >= hp) + 2 * (8 * by >= hp) : 0);
            }
            if (cl == 0 || cl == 4) {
                acc += (h + 2) >> 2;                          // one 8x8 SA8D unit
            } else {
                h += __shfl_xor_sync(0xffffffffu, h, 1);      // the 16x16 unit of 4 lanes
                h += __shfl_xor_sync(0xffffffffu, h, 2);
                if ((sub & 3) == 0) acc += (h + 2) >> 2;
            }
        }
        for (int o = L >> 1; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (live && sub == 0) {
            c.dist[i] = ok ? acc : -1;
            c.cost[i] = ok ? __dadd_rn((double)acc, __dmul_rn(c.lambda, (double)k.rate)) : (double)(1LL << 50);
        }
    }
}

// per CU: the first candidate with the strictly smallest rdcost
__global__ void skip_best_kernel(const xavs2gpu_skip_cand_t *__restrict__ cands, int n, const double *__restrict__ cost,
                                 int n_cus, int32_t *__restrict__ best)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int cu = cands[i].cu;
    if (cu < 0 || cu >= n_cus || (i > 0 && cands[i - 1].cu == cu)) return;
    int b = -1;
    double m = (double)(1LL << 50);
    for (int j = i; j < n && cands[j].cu == cu; j++)
        if (cost[j] < m) {
            m = cost[j];
            b = j;
        }
    best[cu] = b;
}

}  // namespace skp
}  // namespace xg

using namespace xg;

extern "C" int xavs2gpu_skip_costs(xavs2gpu_me_session_t *s, const xavs2gpu_skip_cand_t *cands, int n, double lambda,
                                   int n_cus, int32_t *dist, double *cost, int32_t *best, void *stream)
{
    if (!s || n < 0 || n_cus < 0 || (n > 0 && (!cands || !dist || !cost)) || (n_cus > 0 && !best)) {
        fail(XAVS2GPU_ERR_ARG, "xavs2gpu_skip_costs", "bad session, count or pointer");
        return XAVS2GPU_ERR_ARG;
    }
    int W = 0, H = 0, nrefs = 0, npus = 0;
    xavs2gpu_me_session_info(s, &W, &H, &nrefs, &npus);
    const cudaStream_t st = stream ? (cudaStream_t)stream : (cudaStream_t)xavs2gpu_me_stream(s);
    if (n_cus > 0) XG_CUDA(cudaMemsetAsync(best, 0xFF, sizeof(int32_t) * (size_t)n_cus, st));
    if (n == 0) return XAVS2GPU_OK;
    skp::Ctx c{xavs2gpu_me_plane_device(s, -1, 0), xavs2gpu_me_plane_table_device(s), xavs2gpu_me_plane_stride(s), W, H,
               nrefs, cands, n, lambda, dist, cost};
    // scratch: class counts and cursors, then the class-ordered list
    int *scratch = nullptr;
    XG_CUDA(cudaMallocAsync((void **)&scratch, sizeof(int) * (16 + (size_t)n), st));
    if (!scratch) return XAVS2GPU_ERR_CUDA;
    int *counts = scratch, *cursor = scratch + 8, *sorted = scratch + 16;
    XG_CUDA(cudaMemsetAsync(scratch, 0, sizeof(int) * 16, st));
    const int nb = (n + 255) / 256;
    skp::skip_count_kernel<<<nb, 256, 0, st>>>(c, counts);
    skp::skip_scatter_kernel<<<nb, 256, 0, st>>>(c, counts, cursor, sorted);
    // the CTAs that fit, or fewer where even a warp per candidate is fewer
    const long long most = ((long long)n * 32 + 127) / 128;
    skp::skip_cost_kernel<<<(unsigned)std::min<long long>(most, (long long)sm_count() * XG_SKIP_MINB), 128, 0, st>>>(
        c, counts, sorted);
    count_launch(3);
    XG_CUDA(cudaFreeAsync(scratch, st));
    if (n_cus > 0) {
        skp::skip_best_kernel<<<(n + 127) / 128, 128, 0, st>>>(cands, n, cost, n_cus, best);
        count_launch();
    }
    XG_CUDA(cudaGetLastError());
    return XAVS2GPU_OK;
}
