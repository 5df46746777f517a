// xavs2gpu_common.cuh -- shared definitions of the GB300 (sm_103a) hot-path
// library: PU shape tables, the error channel, per-thread call contexts and
// device helpers used by several kernels.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <stddef.h>

#include "../../include/xavs2_gb300.h"
#include "pu_shapes.h"

namespace xg {

// (one copy per translation unit: the library is built without relocatable
// device code)
static __constant__ uint8_t c_pu_w[kNumParts] = {4, 8, 16, 32, 64, 8, 4, 16, 8, 32, 16, 64, 32,
                                                 16, 12, 16, 4, 32, 24, 32, 8, 64, 48, 64, 16};
static __constant__ uint8_t c_pu_h[kNumParts] = {4, 8, 16, 32, 64, 4, 8, 8, 16, 16, 32, 32, 64,
                                                 12, 16, 4, 16, 24, 32, 8, 32, 48, 64, 16, 64};

// ---- error channel ---------------------------------------------------------
// The reference's primitive signatures have no error return.  Failures are
// recorded here (status + message); unless the caller switched it off with
// xavs2gpu_set_abort_on_error(0), a failure prints the message and aborts, so
// a wrong cost is never returned silently.
void fail(int status, const char *where, const char *msg);
void count_launch(int n = 1);   // kernel launch counter (xavs2gpu_kernel_launches)
void check_cuda(cudaError_t e, const char *where);
#define XG_CUDA(call) ::xg::check_cuda((call), #call)

// ---- per-thread call context ------------------------------------------------
// Every host thread that calls a per-call entry point gets its own stream and
// its own pinned host / device staging buffers, so the entry points are
// re-entrant from the encoder's frame and row threads.
struct CallCtx {
    int device = -1;
    cudaStream_t stream = nullptr;
    uint8_t *h_stage = nullptr;   // pinned host staging
    uint8_t *d_stage = nullptr;   // device staging
    size_t cap = 0;
};
CallCtx &call_ctx(size_t need_bytes);
// 1: per-call block costs read host blocks in place where the device allows
int percall_mode();
int current_device();
// Number of SMs of the current device (queried once per device).
int sm_count();
// A reference picture (W x H, any stride, no border needed) into its 16
// planes: the full-pel plane with `pad` replicated border and the 15
// quarter-pel planes, one kernel (mc.cu).
int reference_planes_from(const uint8_t *src, int src_stride, int width, int height, int pad, uint8_t *const planes[16],
                          int stride, cudaStream_t st);

// Whether work forked from `stream` may go to `side` now.  A stream that was
// joined to a capture belongs to it until that capture ends; from any other
// stream it must not be forked to meanwhile (the launches then stay on `stream`).
static inline bool side_usable(cudaStream_t stream, cudaStream_t side)
{
    cudaStreamCaptureStatus a = cudaStreamCaptureStatusNone, b = cudaStreamCaptureStatusNone;
    unsigned long long ia = 0, ib = 0;
    if (cudaStreamGetCaptureInfo(side, &a, &ia) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    if (a == cudaStreamCaptureStatusNone) return true;
    if (cudaStreamGetCaptureInfo(stream, &b, &ib) != cudaSuccess) cudaGetLastError();
    return a == cudaStreamCaptureStatusActive && b == a && ia == ib;
}

// Byte offset rounded up to 256 for staging sub-buffers.
static inline size_t align_up(size_t v, size_t a = 256) { return (v + a - 1) / a * a; }

// Packs `rows` rows of `row_bytes` from a strided host buffer into `dst`.
void pack_rows(uint8_t *dst, const void *src, intptr_t src_stride_bytes, int row_bytes, int rows);
void unpack_rows(void *dst, intptr_t dst_stride_bytes, const uint8_t *src, int row_bytes, int rows);

// ---- device helpers ---------------------------------------------------------
__device__ __forceinline__ int iabs_d(int v) { return v < 0 ? -v : v; }
// c + sum over the four bytes of |a - b|
__device__ __forceinline__ uint32_t sad4_acc(uint32_t a, uint32_t b, uint32_t c)
{
    uint32_t d;
    asm("vabsdiff4.u32.u32.u32.add %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
__device__ __forceinline__ int clip3_d(int lo, int hi, int v) { return min(max(v, lo), hi); }
__device__ __forceinline__ uint8_t clip_pel_d(int v) { return (uint8_t)min(max(v, 0), 255); }

// The 4 bytes at any address from the aligned word or two words that hold
// them (no word without one of the bytes is read: a block may end at the end
// of its allocation).
__device__ __forceinline__ uint32_t ld4_in(const uint8_t *p)
{
    const uintptr_t a = reinterpret_cast<uintptr_t>(p);
    const uint32_t *w = reinterpret_cast<const uint32_t *>(a & ~(uintptr_t)3);
    const uint32_t lo = w[0];
    return a & 3 ? __funnelshift_r(lo, w[1], 8 * (int)(a & 3)) : lo;
}
// byte k of a minus byte k of b
__device__ __forceinline__ int byte_diff(uint32_t a, uint32_t b, int k)
{
    return (int)__byte_perm(a, 0, 0x4440 + k) - (int)__byte_perm(b, 0, 0x4440 + k);
}

// 4-point Walsh-Hadamard butterfly (unnormalised)
__device__ __forceinline__ void fwht4_d(int &a, int &b, int &c, int &d)
{
    int s0 = a + b, d0 = a - b, s1 = c + d, d1 = c - d;
    a = s0 + s1; b = d0 + d1; c = s0 - s1; d = d0 - d1;
}

// ---- two 4x4 blocks side by side ---------------------------------------------
// Differences of two 4x4 blocks in one integer each, hi * 2^16 + lo with both
// signed: plain 32-bit adds and subtracts are exact butterflies of both blocks
// at 123 lanes a clock per SM, where __vadd2 / __vsub2 run at 60 and __vabsss2
// at 12 (measured; 128 is full issue).  The Hadamard sum's last butterflies
// |a + b| + |a - b| are 2 max(|a|, |b|); with a and b (|a|, |b| <= 2040) biased
// by 2^11 their halves are unsigned 16-bit values and
//     max(|a|, |b|) = max(max(a', b'), 2^12 - min(a', b')) - 2^11,
// three native packed instructions and a subtraction.
constexpr uint32_t kPairBias = 0x08000800u;
__device__ __forceinline__ uint32_t max_abs_pair(uint32_t a, uint32_t b)   // a, b and the result biased
{
    return __vmaxu2(__vmaxu2(a, b), 0x10001000u - __vminu2(a, b));
}
// half the sum of |H D H^T| over both blocks (the sum is even)
__device__ __forceinline__ int satd_pairs(uint32_t (&d)[4][4])
{
#pragma unroll
    for (int r = 0; r < 4; r++) {
        const uint32_t s0 = d[r][0] + d[r][1], e0 = d[r][0] - d[r][1];
        const uint32_t s1 = d[r][2] + d[r][3], e1 = d[r][2] - d[r][3];
        d[r][0] = s0 + s1;
        d[r][1] = e0 + e1;
        d[r][2] = s0 - s1;
        d[r][3] = e0 - e1;
    }
    uint32_t s = 0;
#pragma unroll
    for (int c = 0; c < 4; c++)
        s += max_abs_pair(d[0][c] + d[1][c] + kPairBias, d[2][c] + d[3][c] + kPairBias) +
             max_abs_pair(d[0][c] - d[1][c] + kPairBias, d[2][c] - d[3][c] + kPairBias);
    return (int)(s & 0xFFFFu) + (int)(s >> 16) - 2 * 8 * 2048;
}
// sum of |d| over both blocks (|d| <= 255)
__device__ __forceinline__ int sad_pairs(uint32_t (&d)[4][4])
{
    uint32_t s = 0;
#pragma unroll
    for (int r = 0; r < 4; r++)
#pragma unroll
        for (int c = 0; c < 4; c++) s += max_abs_pair(d[r][c] + kPairBias, d[r][c] + kPairBias);
    return (int)(s & 0xFFFFu) + (int)(s >> 16) - 2 * 16 * 2048;
}

// sum of |H D H^T| over the 4x4 difference block at (p1, p2); WORDS: a row of
// a block as words, for blocks read once (20,000 SATD of 64x64 scattered over a
// plane 50 us, 85 by bytes); by bytes where a warp's rows come from the cache
// again and again (60,000 PUs refined at 17 positions 1640 us, 1700 by words)
template <bool WORDS>
__device__ __forceinline__ int hsum4_d(const uint8_t *p1, intptr_t s1, const uint8_t *p2, intptr_t s2)
{
    int m[4][4];
#pragma unroll
    for (int y = 0; y < 4; y++) {
        int v[4];
        if (WORDS) {
            const uint32_t q1 = ld4_in(p1 + y * s1), q2 = ld4_in(p2 + y * s2);
#pragma unroll
            for (int x = 0; x < 4; x++) v[x] = byte_diff(q1, q2, x);
        } else {
#pragma unroll
            for (int x = 0; x < 4; x++) v[x] = p1[y * s1 + x] - p2[y * s2 + x];
        }
        int a = v[0], b = v[1], c = v[2], d = v[3];
        fwht4_d(a, b, c, d);
        m[y][0] = a; m[y][1] = b; m[y][2] = c; m[y][3] = d;
    }
    int s = 0;
#pragma unroll
    for (int x = 0; x < 4; x++) {
        int a = m[0][x], b = m[1][x], c = m[2][x], d = m[3][x];
        fwht4_d(a, b, c, d);
        s += iabs_d(a) + iabs_d(b) + iabs_d(c) + iabs_d(d);
    }
    return s;
}

// sum of |H8 D H8^T| over one 8x8 difference block, by bytes: a lane waits for
// its own unit, and bytes are all in flight together (20,000 SA8D of 16x16 83 us,
// 115-143 by words; a 16x16 in host memory at an odd address 23 us, 36-40 by words)
__device__ __forceinline__ int hsum8_d(const uint8_t *p1, intptr_t s1, const uint8_t *p2, intptr_t s2)
{
    int m[8][8];
#pragma unroll
    for (int y = 0; y < 8; y++) {
        int v[8];
#pragma unroll
        for (int x = 0; x < 8; x++) v[x] = p1[y * s1 + x] - p2[y * s2 + x];
        int t[8];
#pragma unroll
        for (int i = 0; i < 4; i++) { t[i] = v[i] + v[i + 4]; t[i + 4] = v[i] - v[i + 4]; }
        fwht4_d(t[0], t[1], t[2], t[3]);
        fwht4_d(t[4], t[5], t[6], t[7]);
#pragma unroll
        for (int x = 0; x < 8; x++) m[y][x] = t[x];
    }
    int s = 0;
#pragma unroll
    for (int x = 0; x < 8; x++) {
        int t[8];
#pragma unroll
        for (int i = 0; i < 4; i++) { t[i] = m[i][x] + m[i + 4][x]; t[i + 4] = m[i][x] - m[i + 4][x]; }
        fwht4_d(t[0], t[1], t[2], t[3]);
        fwht4_d(t[4], t[5], t[6], t[7]);
#pragma unroll
        for (int i = 0; i < 8; i++) s += iabs_d(t[i]);
    }
    return s;
}

// SATD rounding units (pixel.c:354-407): 4x4 units for widths 4 and for
// 12x16, otherwise 8x4 units whose two halves share one rounding.
__host__ __device__ __forceinline__ bool satd_unit4(int w, int h) { return w == 4 || (w == 12 && h == 16); }

// Cost of one SATD unit whose top-left corner is (x, y) inside the block.
template <bool WORDS>
__device__ __forceinline__ int satd_unit_d(bool u4, const uint8_t *p1, intptr_t s1, const uint8_t *p2, intptr_t s2)
{
    if (u4) return hsum4_d<WORDS>(p1, s1, p2, s2) >> 1;
    return (hsum4_d<WORDS>(p1, s1, p2, s2) + hsum4_d<WORDS>(p1 + 4, s1, p2 + 4, s2)) >> 1;
}

// SA8D unit kind for a shape: 0 = alias of SATD, 1 = 8x8 units, 2 = 16x16 units
__host__ __device__ __forceinline__ int sa8d_kind(int w, int h)
{
    if (w == 4 || h == 4 || w == 12 || h == 12) return 0;
    if (w == 8 || h == 8 || (w == 32 && h == 24) || (w == 24 && h == 32)) return 1;
    return 2;
}

// mvbits (me.c:614-641): 1 for 0, else 2*bitlen(|d|)+1
__host__ __device__ __forceinline__ int mvbits_hd(int d)
{
    unsigned a = (unsigned)(d < 0 ? -d : d);
#ifdef __CUDA_ARCH__
    return a ? 2 * (32 - __clz((int)a)) + 1 : 1;
#else
    int bl = 0;
    while (a) { bl++; a >>= 1; }
    return d ? 2 * bl + 1 : 1;
#endif
}

__host__ __device__ __forceinline__ int mv_cost_hd(int lambda, int mvx, int mvy, int pmx, int pmy)
{
    return (int)(((int64_t)lambda * (mvbits_hd(mvx - pmx) + mvbits_hd(mvy - pmy))) >> 16);
}

}  // namespace xg
