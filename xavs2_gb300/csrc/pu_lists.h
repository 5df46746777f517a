// pu_lists.h -- how a PU list is laid out for the search: the slots of a 64x64
// CTU, the order of the per-PU list, and the CUs whose partitions it holds.
// Host code without device calls.  A caller with new predictors for each
// picture pays for it each picture, so it is a table lookup or two per PU: with
// the slots found by comparing geometries and the order by two stable sorts,
// the 381,600 PUs of a 720p quadtree with two references took 22 ms more.
#pragma once

#include <stdint.h>
#include <string.h>

#include <vector>

#include "../../include/xavs2_gb300.h"
#include "pu_shapes.h"

namespace xg {

// ---- slot geometry --------------------------------------------------------------
constexpr int kSlots = 849;
struct SlotGeom { int ox, oy, part; };

static inline int part_of(int w, int h)
{
    for (int i = 0; i < kNumParts; i++)
        if (h_pu_w[i] == w && h_pu_h[i] == h) return i;
    return -1;
}

// mode m of an N x N CU at (cx, cy): 0 2Nx2N, 1-2 2NxN, 3-4 Nx2N, 5-6 2NxnU,
// 7-8 2NxnD, 9-10 nLx2N, 11-12 nRx2N
static inline SlotGeom cu_mode_geom(int N, int cx, int cy, int m)
{
    const int h2 = N / 2, q = N / 4, q3 = 3 * N / 4;
    switch (m) {
    case 0: return {cx, cy, part_of(N, N)};
    case 1: return {cx, cy, part_of(N, h2)};
    case 2: return {cx, cy + h2, part_of(N, h2)};
    case 3: return {cx, cy, part_of(h2, N)};
    case 4: return {cx + h2, cy, part_of(h2, N)};
    case 5: return {cx, cy, part_of(N, q)};
    case 6: return {cx, cy + q, part_of(N, q3)};
    case 7: return {cx, cy, part_of(N, q3)};
    case 8: return {cx, cy + q3, part_of(N, q)};
    case 9: return {cx, cy, part_of(q, N)};
    case 10: return {cx + q, cy, part_of(q3, N)};
    case 11: return {cx, cy, part_of(q3, N)};
    default: return {cx + q3, cy, part_of(q, N)};
    }
}

static SlotGeom slot_geom(int s)
{
    if (s < 576) {
        int cu = s / 9, m = s % 9, cx = (cu % 8) * 8, cy = (cu / 8) * 8;
        switch (m) {
        case 0: return {cx, cy, part_of(8, 8)};
        case 1: return {cx, cy, part_of(8, 4)};
        case 2: return {cx, cy + 4, part_of(8, 4)};
        case 3: return {cx, cy, part_of(4, 8)};
        case 4: return {cx + 4, cy, part_of(4, 8)};
        case 5: return {cx, cy, 0};
        case 6: return {cx + 4, cy, 0};
        case 7: return {cx, cy + 4, 0};
        default: return {cx + 4, cy + 4, 0};
        }
    }
    if (s < 784) {
        int cu = (s - 576) / 13, m = (s - 576) % 13;
        return cu_mode_geom(16, (cu % 4) * 16, (cu / 4) * 16, m);
    }
    if (s < 836) {
        int cu = (s - 784) / 13, m = (s - 784) % 13;
        return cu_mode_geom(32, (cu % 2) * 32, (cu / 2) * 32, m);
    }
    return cu_mode_geom(64, 0, 0, s - 836);
}

// (part, ox/4, oy/4) -> slot, -1 if none
struct SlotTable {
    int16_t t[kNumParts][16][16];
    SlotTable()
    {
        memset(t, 0xff, sizeof(t));
        for (int s = 0; s < kSlots; s++) {
            SlotGeom g = slot_geom(s);
            t[g.part][g.oy >> 2][g.ox >> 2] = (int16_t)s;
        }
    }
};
static inline const SlotTable &slot_table()
{
    static const SlotTable table;
    return table;
}

// ---- the per-PU list -------------------------------------------------------------
constexpr int kSmallDim = 16;   // the small PUs of the bounded search: no side above it

// Places of the shapes in the per-PU list, equal ones sharing a place: those
// with a side above kSmallDim, those with a side of it, then the others, each
// by area (the longest searches start first).
struct ShapeOrder {
    uint8_t place[kNumParts];
    int first_small = 0, first_tiny = 0;   // places of the first shape of the second and third kind
    static int side(int p) { return h_pu_w[p] > h_pu_h[p] ? h_pu_w[p] : h_pu_h[p]; }
    static int kind(int p) { return side(p) > kSmallDim ? 0 : side(p) == kSmallDim ? 1 : 2; }
    ShapeOrder()
    {
        auto area = [](int p) { return h_pu_w[p] * h_pu_h[p]; };
        auto before = [&](int a, int b) { return kind(a) != kind(b) ? kind(a) < kind(b) : area(a) > area(b); };
        for (int p = 0; p < kNumParts; p++) {
            int at = 0;
            for (int q = 0; q < kNumParts; q++) at += before(q, p) ? 1 : 0;
            place[p] = (uint8_t)at;
            first_small += kind(p) == 0 ? 1 : 0;
            first_tiny += kind(p) < 2 ? 1 : 0;
        }
    }
};
static inline const ShapeOrder &shape_order()
{
    static const ShapeOrder order;
    return order;
}

struct PerPuCounts {
    int part[kNumParts] = {0};      // PUs of each shape
    int n_large = 0, n_mid = 0;     // of the first and of the second kind
};

// Puts a list of PU indices into that order, each place's in the order they
// come.
static inline PerPuCounts per_pu_order(const std::vector<xavs2gpu_pu_t> &pus, std::vector<int> &list)
{
    const ShapeOrder &order = shape_order();
    PerPuCounts c;
    int at[kNumParts + 1] = {0};
    for (int i : list) c.part[pus[i].part]++;
    for (int p = 0; p < kNumParts; p++) at[order.place[p] + 1] += c.part[p];
    for (int k = 0; k < kNumParts; k++) at[k + 1] += at[k];
    c.n_large = at[order.first_small];
    c.n_mid = at[order.first_tiny] - c.n_large;
    std::vector<int> out(list.size());
    for (int i : list) out[at[order.place[pus[i].part]]++] = i;
    list.swap(out);
    return c;
}

// ---- which search ----------------------------------------------------------------
// The plain per-PU search prices every displacement; the bounded one excludes
// most of them, after a pass over every reference for its block means; the
// clusters share the work of a CU's partitions, after a launch that forms them.
// All give the same results, so a list takes what is estimated to be shorter,
// from the plain search's time in ns on the whole GPU (152 SMs), fitted to
// long lists of one shape: ns a PU at R = 16 / 32 / 64, measured (by the
// formula): 4x4 11 / 15 / 33 (12 / 17 / 39), 16x16 24 / 37 / 122 (23 / 41 /
// 116), 64x64 166 / 350 / 1340 (190 / 423 / 1356).
static inline double plain_ns(int part, int R)
{
    const double area = h_pu_w[part] * h_pu_h[part];
    return 10 + 0.025 * area + (area + 80) * (4.0 * R * R) / 55000;
}
// the block means: 5 us and 0.55 us per MB of plane (a 720p picture with two
// references 7 us, a 2160p one with four 26)
static inline double means_ns(size_t means_bytes) { return 5000 + 5.5e-4 * (double)means_bytes; }
// What the others save of it, at the least (blocky content with noise, which
// the bound excludes little of), and what they take besides: launches and the
// tails of their longest PUs.  us plain / otherwise, on smooth content and on
// blocky: clusters, R = 64, 4,096 PUs of 16x16 CUs 370 / 150 and 370 / 165;
// 4,096 of 8x8 CUs at R = 8 65 / 64 and 65 / 68 (plain by the rule); bounded,
// 2160p with four references, 4,096 PUs of 32x32 at R = 32 435 / 221 and 435 /
// 430, 1,024 of 64x64 at R = 32 397 / 160 and 399 / 420 (plain by the rule).
constexpr double kClusterSaves = 0.5, kClusterNs = 75000, kBoundedSaves = 0.4, kBoundedNs = 150000;
// Shapes whose lone PUs the bounded search is for: the fixed work per PU
// outweighs the displacements of small ones (16,384 4x4 PUs at R = 64: 570 us
// plain, 750 bounded; 16x16 at R = 32 634 / 634, at R = 64 2020 / 790).
static inline bool bounded_shape(int part, int R)
{
    const int kind = ShapeOrder::kind(part);
    return kind == 0 ? R >= 8 : kind == 1 && R >= 48;
}

// The leading PUs of an ordered list that take the bounded search.
struct BoundedPart {
    int n_large = 0, n_small = 0;
};
static inline double bounded_saving_ns(const PerPuCounts &c, int R, BoundedPart &b)
{
    double ns = 0;
    b = BoundedPart{};
    for (int p = 0; p < kNumParts; p++)
        if (bounded_shape(p, R)) {
            ns += c.part[p] * plain_ns(p, R);
            (ShapeOrder::kind(p) == 0 ? b.n_large : b.n_small) += c.part[p];
        }
    const double saving = kBoundedSaves * ns - kBoundedNs;
    if (saving <= 0) b = BoundedPart{};
    return saving > 0 ? saving : 0;
}
// For lists searched without clusters (several sessions in a batch), whole
// pictures as a rule: all of it from 64 PUs on, unless the pass over the
// references outweighs the plain search.  us a batch plain / bounded, leaf CUs'
// PUs with their own predictors, smooth content and blocky: four of 640x360 at R
// = 7 946 / 727 and 946 / 788, at R = 64 5490 / 2020 and 5500 / 3350; one of
// 256x128 at R = 7 105 / 97 and 108 / 95 (at R = 32 128 / 111 and 128 / 162).
constexpr int kBatchMinPus = 64;
static inline BoundedPart bounded_batch(const PerPuCounts &c, int R, size_t means_bytes)
{
    BoundedPart b;
    double ns = 10000;
    int n = 0;
    for (int p = 0; p < kNumParts; p++) {
        ns += 0.5 * c.part[p] * plain_ns(p, R);
        n += c.part[p];
    }
    if (n < kBatchMinPus || means_ns(means_bytes) > ns) return b;
    b.n_large = c.n_large;
    b.n_small = n - c.n_large;
    return b;
}

// ---- CUs -------------------------------------------------------------------------
constexpr int kCuMembers = 13;

struct CuRec {                   // a CU with PUs in the per-PU search, one reference
    int16_t x, y;
    uint8_t lg, ref;             // size 1 << lg
    uint16_t pad_;
    int32_t pu[kCuMembers];      // PU of each partition slot (cu_mode_geom's order; 8x8 CUs as slot_geom's), -1 none
};

// Slot of a PU among the partitions of its CU (side 1 << lg), -1 when it is none
// of them.
struct SlotOfCu {
    uint8_t lg[kSlots], m[kSlots];
    uint8_t part[4][kCuMembers] = {};       // shape of each slot, per CU size
    SlotOfCu()
    {
        for (int s = 0; s < kSlots; s++) {
            lg[s] = s < 576 ? 3 : s < 784 ? 4 : s < 836 ? 5 : 6;
            m[s] = (uint8_t)(s < 576 ? s % 9 : (s - 576) % 13);   // the larger CUs' slots: 16 + 4 + 1 times 13
            part[lg[s] - 3][m[s]] = (uint8_t)slot_geom(s).part;
        }
    }
};
static inline const SlotOfCu &slot_of_cu()
{
    static const SlotOfCu slots;
    return slots;
}
static inline int cu_slot(const SlotTable &table, const SlotOfCu &slots, const xavs2gpu_pu_t &p, int &lg)
{
    if ((p.x | p.y) & 3) return -1;
    const int s = table.t[p.part][(p.y & 63) >> 2][(p.x & 63) >> 2];
    if (s < 0) return -1;
    lg = slots.lg[s];
    return slots.m[s];
}

// An ordered per-PU list with clusters: the dense CUs, and the other PUs, in the
// list's order.
struct CuLists {
    std::vector<CuRec> recs;
    int n_rec[4] = {0, 0, 0, 0};            // records per CU size
    int cap_large = 0, cap_small = 0;       // PUs in records, with and without a side above kSmallDim
    std::vector<uint32_t> rest;
    BoundedPart bounded;                    // of rest
    bool use = false;                       // whether this is shorter than the plain search of them all
};

// A CTA searches a cluster, in 420 us for a 64x64 CU at R = 64, however short
// the list is otherwise.  So a list has clusters from an area of this many of
// its largest CU on (416x240, the first 4,096 PUs of the quadtree, 130 of
// 64x64, at R = 64: 295-515 us by content, 358 plain; 16,384 of them, 500 of
// 64x64: 575-690, 1240 plain).
constexpr int kClusterAreas = 200;

// A CU is clustered with at least four of its PUs, and above 16x16 with three
// times its area in them (all partitions are seven times).  Fewer share too
// little: 4,096 random PUs of a 1280x720 quadtree at R = 64 took 480-710 us
// with every two of a CU together, 380 plain.
static inline bool cu_dense(int members, int area, int lg) { return members >= 4 && (lg <= 4 || area >= 3 << (2 * lg)); }

// Share of a list's work in dense CUs from which the others are clustered too.
constexpr double kClusterAll = 0.75;

static inline CuLists cu_lists(const std::vector<xavs2gpu_pu_t> &pus, const std::vector<uint32_t> &list,
                               const PerPuCounts &counts, int W, int H, int nrefs, int R, size_t means_bytes)
{
    CuLists c;
    double all_ns = 0;
    long long area = 0;
    for (int p = 0; p < kNumParts; p++) {
        all_ns += counts.part[p] * plain_ns(p, R);
        area += (long long)counts.part[p] * h_pu_w[p] * h_pu_h[p];
    }
    const double means = means_ns(means_bytes);
    if (kClusterSaves * all_ns <= means) return c;      // not worth looking at
    const SlotTable &table = slot_table();
    const SlotOfCu &slots = slot_of_cu();
    std::vector<int> at[4];                             // record of each CU position, per size
    for (int k = 0; k < 4; k++) at[k].assign((size_t)nrefs * ((W >> (3 + k)) + 1) * ((H >> (3 + k)) + 1), -1);
    std::vector<char> in(pus.size(), 0);                // whether a record holds the PU
    for (const uint32_t i : list) {
        const xavs2gpu_pu_t &p = pus[i];
        int lg = 0;
        const int slot = cu_slot(table, slots, p, lg);
        if (slot < 0) continue;
        const int cols = (W >> lg) + 1, rows = (H >> lg) + 1;
        int &r = at[lg - 3][((size_t)p.ref * rows + (p.y >> lg)) * cols + (p.x >> lg)];
        if (r < 0) {
            r = (int)c.recs.size();
            CuRec rec{};
            rec.x = (int16_t)(p.x >> lg << lg);
            rec.y = (int16_t)(p.y >> lg << lg);
            rec.lg = (uint8_t)lg;
            rec.ref = p.ref;
            for (int &u : rec.pu) u = -1;
            c.recs.push_back(rec);
        }
        int32_t &u = c.recs[r].pu[slot];
        if (u >= 0) continue;                           // a second PU of the same partition searches alone
        u = (int)i;
        in[i] = 1;
    }
    // what the dense CUs hold
    auto dense = [&](const CuRec &r) {
        int members = 0, covered = 0;
        for (int m = 0; m < kCuMembers; m++)
            if (r.pu[m] >= 0) {
                const int part = slots.part[r.lg - 3][m];
                members++;
                covered += h_pu_w[part] * h_pu_h[part];
            }
        return cu_dense(members, covered, r.lg);
    };
    PerPuCounts left = counts, lone;
    int lg_max = 0;
    for (const CuRec &r : c.recs) {
        const bool d = dense(r);
        if (d && r.lg > lg_max) lg_max = r.lg;
        for (int m = 0; m < kCuMembers; m++)
            if (r.pu[m] >= 0) (d ? left.part : lone.part)[slots.part[r.lg - 3][m]] += d ? -1 : 1;
    }
    double in_ns = all_ns;
    for (int p = 0; p < kNumParts; p++) in_ns -= left.part[p] * plain_ns(p, R);
    double saving = kClusterSaves * in_ns - kClusterNs;
    const bool clusters = saving > 0 && area >= (long long)kClusterAreas << (2 * lg_max);
    // the few others of a list of dense CUs go along
    const bool every = clusters && in_ns >= kClusterAll * all_ns;
    if (!clusters) {
        saving = 0;
        left = counts;
    } else if (every) {
        for (int p = 0; p < kNumParts; p++) left.part[p] -= lone.part[p];
    }
    saving += bounded_saving_ns(left, R, c.bounded);
    c.use = saving > means;
    if (!c.use || !clusters) {
        c.recs.clear();
        if (!c.use) c.bounded = BoundedPart{};
        c.rest = list;
        return c;
    }
    size_t kept = 0;
    for (const CuRec &r : c.recs) {
        if (every || dense(r)) {
            c.n_rec[r.lg - 3]++;
            c.recs[kept++] = r;
        } else {
            for (int u : r.pu)
                if (u >= 0) in[u] = 0;
        }
    }
    c.recs.resize(kept);
    for (int q = 0; q < (int)list.size(); q++) {
        if (!in[list[q]]) c.rest.push_back(list[q]);
        else (q < counts.n_large ? c.cap_large : c.cap_small)++;
    }
    return c;
}

}  // namespace xg
