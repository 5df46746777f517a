// fs_cu.cuh -- full search of the partitions of one CU together.
//
// PUs with their own predictors have their own search centres, but the
// partitions of one CU (2Nx2N, 2NxN, Nx2N and the four asymmetric modes, or
// the 8x8 / 8x4 / 4x8 / 4x4 PUs of an 8x8 CU) have predictors from the same
// neighbourhood, so most of their centres lie a few pixels apart.  Partitions
// of a CU and reference whose centres are within kCuReach pixels of each
// other are searched over the union of their windows: the SADs of the CU's
// column strips and row bands at a displacement are computed once, and every
// member's SAD is a sum of them (7 times the CU's area per displacement
// becomes once).  Each member keeps its own MV cost, window and limits, so its
// (cost, visit order) minimum is the one its own search finds.
//
// Grouping happens on the device, after the candidates have fixed the centres
// (cu_cluster_kernel: a thread per CU, greedy around the first member left):
// clusters that share enough go to a queue per CU size, the other PUs to the
// queues of the per-PU search.
//
// fs_cu_kernel<S>: a CTA per cluster, the union window in shared memory.  A
// thread takes 4 adjacent displacements in kRows rows: per window word one
// load and three byte permutes serve 4 * kRows SAD steps; the column strips'
// sums run over all rows, the row bands' totals are read off them at each
// band's end.  Per member the smallest SAD of the thread's displacements plus
// the smallest MV cost of its columns and rows is compared with the member's
// best cost; only then its displacements are priced one by one.
//
// Bound by integer issue (55-68 % issue active, the SAD steps and byte
// permutes on one 64-lane pipe).  A 720p picture, 2 references, R = 64, every
// PU with its own predictor (381k searches; whole pass with upload and
// refinement): 28.9 ms with the plain per-PU search, 21.8 ms with the bounded
// one alone, 11.1 ms with the clusters; R = 7..32 on 520x344..1664x648:
// 1.75-3.7 times faster.  Two displacement rows per thread: four need 127
// registers at 8x8 (2 CTAs per SM, 11.4 ms against 11.1 with 4 CTAs); three
// CTAs for the larger CUs spill (11.9 against 11.4 ms).
#pragma once

#ifndef XG_CU8_ROWS
#define XG_CU8_ROWS 2
#endif
#ifndef XG_CU8_MINB
#define XG_CU8_MINB 4
#endif
#ifndef XG_CU_MINB
#define XG_CU_MINB 2
#endif

namespace xg {

constexpr int kCuReach = 6;      // pixels between a cluster's first member's centre and the others'
constexpr int kCuOut = 0x3fffffff;   // above any sum of two lambda x bits (lambda < 2^23); twice it fits an int
constexpr int kCuThreads = 256;

struct CuWork {
    uint32_t cu, mask;           // members (slots) of the cluster
};
// queue counters: [0..3] clusters of 8x8 .. 64x64 CUs, [4] / [5] PUs with a
// side above 16 / others for the per-PU search; [6..9] clusters taken
constexpr int kCuCounters = 10;
struct CuQueues {
    int *count;
    CuWork *work[4];
    uint32_t *large, *small;
};

__global__ void __launch_bounds__(128) cu_cluster_kernel(const CuRec *__restrict__ cus, int n,
                                                         const SessView *__restrict__ views, CuQueues q)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const SessView &v = views[0];
    const CuRec &c = cus[k];
    const int lg = c.lg;
    int16_t cx[kCuMembers], cy[kCuMembers];
    unsigned left = 0;
#pragma unroll
    for (int m = 0; m < kCuMembers; m++) {
        const int pu = c.pu[m];
        cx[m] = cy[m] = 0;
        if (pu < 0) continue;
        const PuState st = v.state[pu];
        if (!st.valid) continue;
        cx[m] = st.cx;
        cy[m] = st.cy;
        left |= 1u << m;
    }
    while (left) {
        const unsigned first = left & (0u - left);
        int fx = 0, fy = 0;
#pragma unroll
        for (int m = 0; m < kCuMembers; m++)
            if (first >> m & 1) { fx = cx[m]; fy = cy[m]; }
        unsigned mask = 0;
        int area = 0;
#pragma unroll
        for (int m = 0; m < kCuMembers; m++)
            if ((left >> m & 1) && abs(cx[m] - fx) <= kCuReach && abs(cy[m] - fy) <= kCuReach) {
                mask |= 1u << m;
                const int part = v.pus[c.pu[m]].part;
                area += c_pu_w[part] * c_pu_h[part];
            }
        left &= ~mask;
        // up to 16x16 the per-PU search's fixed work outweighs the block's:
        // any two members are cheaper together; a larger CU's area once costs
        // about two thirds of the same area in PUs (1,070 against 1,660 warp
        // instructions per 32 displacements at 64x64)
        if (__popc(mask) >= 2 && (lg <= 4 || 3 * area >= 2 << (2 * lg))) {
            q.work[lg - 3][atomicAdd(&q.count[lg - 3], 1)] = CuWork{(uint32_t)k, mask};
        } else {
            for (unsigned b = mask; b; b &= b - 1) {
                const int pu = c.pu[__ffs(b) - 1], part = v.pus[pu].part;
                const bool small = max(c_pu_w[part], c_pu_h[part]) <= kSmallDim;
                (small ? q.small : q.large)[atomicAdd(&q.count[small ? 5 : 4], 1)] = (uint32_t)pu;
            }
        }
    }
}

template <int S> struct CuShape {
    static constexpr int kRows = S == 8 ? XG_CU8_ROWS : 2;         // displacement rows per thread
    static constexpr int kStrips = S == 8 ? 2 : 4, kBands = kStrips;
    static constexpr int kWords = S / 4;                  // words per block row
    static constexpr int kStripWords = kWords / kStrips;
    static constexpr int kBandRows = S / kBands;
    static constexpr int kTerms = S == 8 ? 4 : 7;
    static constexpr int kSlots = S == 8 ? 9 : 13;
};

// a window row against the block rows it meets: row r - a of displacement
// row a, from <= a < to (compile-time constants); cur at block row r
template <int S>
__device__ __forceinline__ void cu_row(const uint32_t *w, const uint32_t *cur,
                                       uint32_t (&c)[CuShape<S>::kRows][4][CuShape<S>::kStrips], int from, int to)
{
    using C = CuShape<S>;
    constexpr int V = S == 8 ? 2 : 4;   // block words per load
    uint32_t lo = w[0];
#pragma unroll
    for (int x0 = 0; x0 < C::kWords; x0 += V) {
        uint32_t cw[C::kRows][V];
#pragma unroll
        for (int a = 0; a < C::kRows; a++) {
            if (a < from || a >= to) continue;
            if (V == 4) {
                const uint4 q = *reinterpret_cast<const uint4 *>(cur + x0 - a * C::kWords);
                cw[a][0] = q.x; cw[a][1] = q.y; cw[a][V - 2] = q.z; cw[a][V - 1] = q.w;
            } else {
                const uint2 q = *reinterpret_cast<const uint2 *>(cur + x0 - a * C::kWords);
                cw[a][0] = q.x; cw[a][1] = q.y;
            }
        }
#pragma unroll
        for (int k = 0; k < V; k++) {
            const int s = (x0 + k) / C::kStripWords;
            const uint32_t hi = w[x0 + k + 1];
            const uint32_t b1 = __byte_perm(lo, hi, 0x4321), b2 = __byte_perm(lo, hi, 0x5432),
                           b3 = __byte_perm(lo, hi, 0x6543);
#pragma unroll
            for (int a = 0; a < C::kRows; a++) {
                if (a < from || a >= to) continue;
                c[a][0][s] = sad4_acc(cw[a][k], lo, c[a][0][s]);
                c[a][1][s] = sad4_acc(cw[a][k], b1, c[a][1][s]);
                c[a][2][s] = sad4_acc(cw[a][k], b2, c[a][2][s]);
                c[a][3][s] = sad4_acc(cw[a][k], b3, c[a][3][s]);
            }
            lo = hi;
        }
    }
}

// terms of the member sums of a thread's displacements
template <int S>
__device__ __forceinline__ void cu_terms(const uint32_t *w, int pitch, const uint32_t *cur,
                                         uint32_t (&t)[CuShape<S>::kRows][4][CuShape<S>::kTerms])
{
    using C = CuShape<S>;
    uint32_t c[C::kRows][4][C::kStrips];
#pragma unroll
    for (int a = 0; a < C::kRows; a++)
#pragma unroll
        for (int x = 0; x < 4; x++)
#pragma unroll
            for (int s = 0; s < C::kStrips; s++) c[a][x][s] = 0;
    if constexpr (S == 8) {
        // displacement row a's upper blocks end with window row 3 + a
#pragma unroll
        for (int r = 0; r < 7 + C::kRows; r++) {
            cu_row<S>(w + r * pitch, cur + 2 * r, c, r < 8 ? 0 : r - 7, r + 1 < C::kRows ? r + 1 : C::kRows);
            if (r >= 3 && r < 3 + C::kRows)
#pragma unroll
                for (int x = 0; x < 4; x++) {
                    t[r - 3][x][0] = c[r - 3][x][0];
                    t[r - 3][x][1] = c[r - 3][x][1];
                }
        }
#pragma unroll
        for (int a = 0; a < C::kRows; a++)
#pragma unroll
            for (int x = 0; x < 4; x++) {
                t[a][x][2] = c[a][x][0] - t[a][x][0];
                t[a][x][3] = c[a][x][1] - t[a][x][1];
            }
    } else {
        auto total = [&](int a, int x) { return c[a][x][0] + c[a][x][1] + c[a][x][2] + c[a][x][3]; };
#pragma unroll
        for (int band = 0; band < C::kBands; band++) {
            // the band's first window row still ends displacement row 1's previous band
            if (band == 0) cu_row<S>(w, cur, c, 0, 1);
            else cu_row<S>(w, cur, c, 0, 2);
            w += pitch;
            cur += C::kWords;
            if (band > 0)
#pragma unroll
                for (int x = 0; x < 4; x++) t[1][x][3 + band] = total(1, x);
#pragma unroll(S <= 16 ? C::kBandRows - 1 : 1)
            for (int r = 1; r < C::kBandRows; r++, w += pitch, cur += C::kWords) cu_row<S>(w, cur, c, 0, 2);
            if (band < 3)
#pragma unroll
                for (int x = 0; x < 4; x++) t[0][x][4 + band] = total(0, x);
        }
        cu_row<S>(w, cur, c, 1, 2);
#pragma unroll
        for (int a = 0; a < 2; a++)
#pragma unroll
            for (int x = 0; x < 4; x++)
#pragma unroll
                for (int s = 0; s < 4; s++) t[a][x][s] = c[a][x][s];
    }
}

// SAD of slot m from the terms, m known at compile time
template <int S>
__device__ __forceinline__ uint32_t cu_slot_sad(int m, const uint32_t (&t)[CuShape<S>::kTerms], uint32_t total)
{
    if (S == 8) {
        switch (m) {
        case 0: return total;
        case 1: return t[0] + t[1];
        case 2: return t[2] + t[3];
        case 3: return t[0] + t[2];
        case 4: return t[1] + t[3];
        default: return t[m - 5];
        }
    }
    switch (m) {
    case 0: return total;
    case 1: return t[CuShape<S>::kTerms - 2];
    case 2: return total - t[CuShape<S>::kTerms - 2];
    case 3: return t[0] + t[1];
    case 4: return t[2] + t[3];
    case 5: return t[CuShape<S>::kTerms - 3];
    case 6: return total - t[CuShape<S>::kTerms - 3];
    case 7: return t[CuShape<S>::kTerms - 1];
    case 8: return total - t[CuShape<S>::kTerms - 1];
    case 9: return t[0];
    case 10: return total - t[0];
    case 11: return total - t[3];
    default: return t[3];
    }
}

// the SADs of slot m (the same for the whole warp) at a thread's displacements
template <int S>
__device__ __forceinline__ void cu_slot_sads(int m, const uint32_t (&t)[CuShape<S>::kRows][4][CuShape<S>::kTerms],
                                             const uint32_t (&tot)[CuShape<S>::kRows][4],
                                             uint32_t (&s)[CuShape<S>::kRows][4])
{
#pragma unroll
    for (int k = 0; k < CuShape<S>::kSlots; k++)
        if (k == m) {
#pragma unroll
            for (int a = 0; a < CuShape<S>::kRows; a++)
#pragma unroll
                for (int x = 0; x < 4; x++) s[a][x] = cu_slot_sad<S>(k, t[a][x], tot[a][x]);
        }
}

struct CuMember {
    int px, py;              // predictor minus 4 x the union window's origin (quarter-pels)
    int x0, x1, y0, y1;      // displacements of the member's own window inside its limits
    unsigned order;          // visit order of the union window's origin in the member's window
    int pu;
};

__host__ __device__ __forceinline__ int cu_cols(int R) { return 2 * R + 2 * kCuReach; }
template <int S> __host__ __device__ __forceinline__ int cu_pitch(int R) { return ((cu_cols(R) + S + 10) >> 2) | 1; }
template <int S> __host__ __device__ __forceinline__ int cu_col_groups(int R) { return (cu_cols(R) + 3) >> 2; }
template <int S> __host__ __device__ __forceinline__ int cu_row_groups(int R)
{
    return (cu_cols(R) + CuShape<S>::kRows - 1) / CuShape<S>::kRows;
}
// ints of a member's MV-cost tables: every column and row (padded to the
// threads' groups), their minima per group
template <int S> __host__ __device__ __forceinline__ int cu_table(int R)
{
    return 5 * cu_col_groups<S>(R) + (CuShape<S>::kRows + 1) * cu_row_groups<S>(R) + 3 & ~3;
}
template <int S> __host__ __device__ __forceinline__ int cu_smem(int R)
{
    return S * S + 16 * (int)(sizeof(CuMember) + 8) + kCuMembers * (int)sizeof(int) * cu_table<S>(R) +
           (cu_cols(R) + S + 2 * CuShape<S>::kRows) * 4 * cu_pitch<S>(R);
}

template <int S>
__global__ void __launch_bounds__(kCuThreads, S == 8 ? XG_CU8_MINB : XG_CU_MINB)
    fs_cu_kernel(const CuWork *__restrict__ work, const int *__restrict__ count, int *__restrict__ taken,
                 const CuRec *__restrict__ cus, const SessView *__restrict__ views, int R, int lambda)
{
    using C = CuShape<S>;
    extern __shared__ __align__(16) uint8_t smem_pu[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int ngx = cu_col_groups<S>(R), ngy = cu_row_groups<S>(R), pitch = cu_pitch<S>(R);
    __shared__ int s_li;
    uint32_t *s_cur = reinterpret_cast<uint32_t *>(smem_pu);                                  // [S][S/4]
    unsigned long long *s_key = reinterpret_cast<unsigned long long *>(smem_pu + S * S);      // [13]
    CuMember *s_mem = reinterpret_cast<CuMember *>(s_key + 16);                               // [13]
    // per member lambda x MV bits of the columns [4 ngx] and rows [kRows ngy]
    // (kCuOut outside its window and limits), minima of 4 columns, kRows rows
    const int table = cu_table<S>(R);
    int *s_tab = reinterpret_cast<int *>(s_mem + 16);
    uint32_t *s_win = reinterpret_cast<uint32_t *>(s_tab + kCuMembers * table);
    const SessView &v = views[0];
    const Geometry g = v.g;
    const int n = *count;
    while (true) {
        if (tid == 0) s_li = atomicAdd(taken, 1);
        __syncthreads();
        const int li = s_li;
        if (li >= n) break;
        const CuWork wk = work[li];
        const CuRec &cu = cus[wk.cu];
        const uint8_t *ref = v.ref0[cu.ref];
        // centres of the members: the union window
        int cx = 0, cy = 0, fx = 32767, fy = 32767, lx = -32768, ly = -32768;
        const bool mine = lane < kCuMembers && (wk.mask >> lane & 1);
        const int pu = mine ? cu.pu[lane] : 0;
        if (mine) {
            const PuState st = v.state[pu];
            fx = lx = cx = st.cx;
            fy = ly = cy = st.cy;
        }
        fx = __reduce_min_sync(0xffffffffu, fx);
        fy = __reduce_min_sync(0xffffffffu, fy);
        lx = __reduce_max_sync(0xffffffffu, lx);
        ly = __reduce_max_sync(0xffffffffu, ly);
        __syncthreads();   // the previous cluster's readers are done
        int x0 = 1 << 20, x1 = -1, y0 = 1 << 20, y1 = -1;   // displacements any member may take
        CuMember me{};
        if (mine) {
            const xavs2gpu_pu_t p = v.pus[pu];
            const int ox = fx - R, oy = fy - R;   // union origin, absolute displacement
            me.px = p.mvp_x - 4 * ox;
            me.py = p.mvp_y - 4 * oy;
            x0 = me.x0 = max((int)p.min_x, cx - R) - ox;
            x1 = me.x1 = min((int)p.max_x, cx + R - 1) - ox;
            y0 = me.y0 = max((int)p.min_y, cy - R) - oy;
            y1 = me.y1 = min((int)p.max_y, cy + R - 1) - oy;
            // order of (ci, cj): 2 + (oy + cj - cy + R) * 2R + (ox + ci - cx + R)
            me.order = 2u + (unsigned)((oy - cy + R) * 2 * R + (ox - cx + R));
            me.pu = pu;
        }
        x0 = __reduce_min_sync(0xffffffffu, x0);
        x1 = __reduce_max_sync(0xffffffffu, x1);
        y0 = __reduce_min_sync(0xffffffffu, y0);
        y1 = __reduce_max_sync(0xffffffffu, y1);
        // the union window, cut to those displacements
        const int ni = x1 - x0 + 1, nj = y1 - y0 + 1;
        if (ni <= 0 || nj <= 0) continue;
        if (warp == 0 && mine) {
            me.px -= 4 * x0;
            me.py -= 4 * y0;
            me.x0 -= x0; me.x1 -= x0;
            me.y0 -= y0; me.y1 -= y0;
            me.order += (unsigned)(y0 * 2 * R + x0);
            s_mem[lane] = me;
            s_key[lane] = v.keys[pu];
        }
        const uint8_t *o = v.cur + (ptrdiff_t)cu.y * g.stride + cu.x;   // 8-byte aligned
        for (int k = tid; k < S * C::kWords; k += kCuThreads)
            s_cur[k] = *reinterpret_cast<const uint32_t *>(o + (ptrdiff_t)(k / C::kWords) * g.stride +
                                                           4 * (k % C::kWords));
        // window samples, word-aligned to the first column.  Where the CU
        // leaves the padded plane only members inside it are priced: rows are
        // clamped, columns read on into the neighbouring rows of the session's
        // plane pool (a reference plane has planes before and after it).
        {
            const int wx = cu.x + fx - R + x0, wy = cu.y + fy - R + y0;
            const int ylast = min(wy + nj + S - 2, g.H + kPad - 1);
            const int rows = (nj + C::kRows - 1) / C::kRows * C::kRows + S, nw = (ni + S + 6) >> 2;
            for (int r = warp; r < rows; r += kCuThreads / 32) {
                const uint8_t *q = ref + (ptrdiff_t)max(min(wy + r, ylast), -kPad) * g.stride + wx;
                const uint32_t *a = reinterpret_cast<const uint32_t *>(reinterpret_cast<uintptr_t>(q) & ~(uintptr_t)3);
                const int sh = 8 * (int)((uintptr_t)q & 3);
                for (int c = lane; c < nw; c += 32)
                    s_win[r * pitch + c] = __funnelshift_r(__ldg(a + c), __ldg(a + c + 1), sh);
            }
        }
        __syncthreads();
        // smallest MV cost of each member over a thread's columns / rows
        const int ncg = (ni + 3) >> 2, nrg = (nj + C::kRows - 1) / C::kRows;
        for (int m = warp; m < C::kSlots; m += kCuThreads / 32) {
            if (!(wk.mask >> m & 1)) continue;
            const CuMember mm = s_mem[m];
            int *tx = s_tab + m * table, *ty = tx + 4 * ngx, *mx = ty + C::kRows * ngy, *my = mx + ngx;
            for (int k = lane; k < ncg + nrg; k += 32) {
                const bool col = k < ncg;
                const int len = col ? 4 : C::kRows, first = col ? 4 * k : len * (k - ncg);
                const int lo = col ? mm.x0 : mm.y0, hi = col ? mm.x1 : mm.y1, p = col ? mm.px : mm.py;
                int low = kCuOut;
                for (int t = first; t < first + len; t++) {
                    const int l = t >= lo && t <= hi ? lambda * mvbits_hd(4 * t - p) : kCuOut;
                    (col ? tx : ty)[t] = l;
                    low = min(low, l);
                }
                if (col) mx[k] = low;
                else my[k - ncg] = low;
            }
        }
        __syncthreads();
        const int items = ncg * nrg, inv = ((1 << 20) + ncg - 1) / ncg;   // items < 2^14, ncg < 128
        // the window's middle rows first: a good predictor's match is there,
        // and the best cost it leaves prices few displacements elsewhere
        const int start = max(0, (items - kCuThreads) / 2);
        for (int k = tid; k - lane < items; k += kCuThreads) {
            const bool on = k < items;
            const int it = k + start < items ? k + start : k + start - items;
            const int rg = on ? (int)(((unsigned)it * (unsigned)inv) >> 20) : 0, cg = on ? it - rg * ncg : 0;
            uint32_t t[C::kRows][4][C::kTerms];
            cu_terms<S>(s_win + C::kRows * rg * pitch + cg, pitch, s_cur, t);
            uint32_t tot[C::kRows][4];
#pragma unroll
            for (int a = 0; a < C::kRows; a++)
#pragma unroll
                for (int x = 0; x < 4; x++) tot[a][x] = t[a][x][0] + t[a][x][1] + t[a][x][2] + t[a][x][3];
            unsigned pass = 0;
#pragma unroll
            for (int m = 0; m < C::kSlots; m++) {
                if (!(wk.mask >> m & 1)) continue;
                uint32_t low = 0xffffffffu;
#pragma unroll
                for (int a = 0; a < C::kRows; a++)
                    low = min(min(low, min(cu_slot_sad<S>(m, t[a][0], tot[a][0]), cu_slot_sad<S>(m, t[a][1], tot[a][1]))),
                              min(cu_slot_sad<S>(m, t[a][2], tot[a][2]), cu_slot_sad<S>(m, t[a][3], tot[a][3])));
                const int *mx = s_tab + m * table + 4 * ngx + C::kRows * ngy;
                const uint32_t mv = (uint32_t)((mx[cg] + mx[ngx + rg]) >> 16);
                const uint32_t best = reinterpret_cast<const volatile uint32_t *>(&s_key[m])[1];
                if (low + mv <= best) pass |= 1u << m;
            }
            if (!on) pass = 0;
            // members that may improve: their displacements one by one
            for (unsigned any = __reduce_or_sync(0xffffffffu, pass); any; any &= any - 1) {
                const int m = __ffs(any) - 1;
                if (!(pass >> m & 1)) continue;
                uint32_t sad[C::kRows][4], bc = 0xffffffffu, bo = 0;
                cu_slot_sads<S>(m, t, tot, sad);
                const int *tx = s_tab + m * table + 4 * cg, *ty = s_tab + m * table + 4 * ngx + C::kRows * rg;
                const int4 lx = *reinterpret_cast<const int4 *>(tx);
#pragma unroll
                for (int a = 0; a < C::kRows; a++) {
                    const int l = ty[a];
#pragma unroll
                    for (int x = 0; x < 4; x++) {
                        const int bits = (x == 0 ? lx.x : x == 1 ? lx.y : x == 2 ? lx.z : lx.w) + l;
                        const uint32_t cost = sad[a][x] + (uint32_t)(bits >> 16);
                        if (bits < kCuOut && cost < bc) {
                            bc = cost;
                            bo = (unsigned)(a * 2 * R + x);
                        }
                    }
                }
                bo += s_mem[m].order + (unsigned)(C::kRows * rg * 2 * R + 4 * cg);
                const unsigned long long key = ((unsigned long long)bc << 32) | bo;
                if (bc != 0xffffffffu && key < *reinterpret_cast<volatile unsigned long long *>(&s_key[m]))
                    atomicMin(&s_key[m], key);
            }
            __syncwarp();
        }
        __syncthreads();
        if (warp == 0 && mine) {
            const unsigned long long k = s_key[lane];
            if (k < v.keys[pu]) v.keys[pu] = k;
        }
    }
}

// Searches one queue: CTAs take clusters until it is empty.
template <int S>
static int cu_launch_one(const CuQueues &q, const CuRec *cus, const SessView *views, int R, int lambda, cudaStream_t st)
{
    static std::atomic<int> grid[64][129];   // CTAs that run at once, per device and range
    const int dev = current_device(), bytes = cu_smem<S>(R);
    if (dev < 0 || dev >= 64 || R < 1 || R > 128) return XAVS2GPU_ERR_ARG;
    int ctas = grid[dev][R].load(std::memory_order_relaxed);
    if (!ctas) {
        int per_sm = 0;
        XG_CUDA(cudaFuncSetAttribute(fs_cu_kernel<S>, cudaFuncAttributeMaxDynamicSharedMemorySize, cu_smem<S>(128)));
        XG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fs_cu_kernel<S>, kCuThreads, bytes));
        ctas = sm_count() * std::max(per_sm, 1);
        grid[dev][R].store(ctas, std::memory_order_relaxed);
    }
    constexpr int k = S == 8 ? 0 : S == 16 ? 1 : S == 32 ? 2 : 3;
    fs_cu_kernel<S><<<ctas, kCuThreads, bytes, st>>>(q.work[k], q.count + k, q.count + 6 + k, cus, views, R, lambda);
    count_launch();
    XG_CUDA(cudaGetLastError());
    return XAVS2GPU_OK;
}

// Groups the CUs' partitions into clusters and PUs searched one by one.
static void cu_cluster_launch(const CuQueues &q, const CuRec *cus, int n, const SessView *views, cudaStream_t st)
{
    XG_CUDA(cudaMemsetAsync(q.count, 0, sizeof(int) * kCuCounters, st));
    cu_cluster_kernel<<<(n + 127) / 128, 128, 0, st>>>(cus, n, views, q);
    count_launch();
}

}  // namespace xg
