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
// with a side above kSmallDim, then the others, by area (the longest searches
// start first).
struct ShapeOrder {
    uint8_t place[kNumParts];
    int first_small = 0;        // place of the first small shape
    ShapeOrder()
    {
        auto large = [](int p) { return h_pu_w[p] > kSmallDim || h_pu_h[p] > kSmallDim; };
        auto area = [](int p) { return h_pu_w[p] * h_pu_h[p]; };
        auto before = [&](int a, int b) { return large(a) != large(b) ? large(a) : area(a) > area(b); };
        for (int p = 0; p < kNumParts; p++) {
            int at = 0;
            for (int q = 0; q < kNumParts; q++) at += before(q, p) ? 1 : 0;
            place[p] = (uint8_t)at;
            first_small += large(p) ? 1 : 0;
        }
    }
};

// Puts a list of PU indices into that order, each place's in the order they
// come; returns how many are large.
static inline int per_pu_order(const std::vector<xavs2gpu_pu_t> &pus, std::vector<int> &list)
{
    static const ShapeOrder order;
    int at[kNumParts + 1] = {0}, n_large = 0;
    for (int i : list) at[order.place[pus[i].part] + 1]++;
    for (int k = 0; k < kNumParts; k++) at[k + 1] += at[k];
    n_large = at[order.first_small];
    std::vector<int> out(list.size());
    for (int i : list) out[at[order.place[pus[i].part]]++] = i;
    list.swap(out);
    return n_large;
}

// ---- CUs -------------------------------------------------------------------------
constexpr int kCuMembers = 13;

struct CuRec {                   // a CU with PUs in the per-PU search, one reference
    int16_t x, y;
    uint8_t lg, ref;             // size 1 << lg
    uint16_t pad_;
    int32_t pu[kCuMembers];      // PU of each partition slot (cu_mode_geom's order; 8x8 CUs as slot_geom's), -1 none
};

// Slot of a PU among the partitions of its CU (side 1 << lg, corner cx, cy),
// -1 when it is none of them.
static inline int cu_slot(const SlotTable &table, const xavs2gpu_pu_t &p, int &lg, int &cx, int &cy)
{
    if ((p.x | p.y) & 3) return -1;
    const int s = table.t[p.part][(p.y & 63) >> 2][(p.x & 63) >> 2];
    if (s < 0) return -1;
    lg = s < 576 ? 3 : s < 784 ? 4 : s < 836 ? 5 : 6;
    cx = p.x >> lg << lg;
    cy = p.y >> lg << lg;
    return s < 576 ? s % 9 : (s - 576) % 13;   // the larger CUs' slots: 16 + 4 + 1 times 13
}

// The CUs of the per-PU list `list` (large PUs first, n_large of them) and the
// PUs that are a partition of none of them.
struct CuLists {
    std::vector<CuRec> recs;
    std::vector<uint32_t> rest;
    int n_rec[4] = {0, 0, 0, 0};            // records per CU size
    int rest_large = 0;                     // large PUs of rest (they come first)
    int cap_large = 0, cap_small = 0;       // PUs in records
};
static inline CuLists cu_lists(const std::vector<xavs2gpu_pu_t> &pus, const std::vector<uint32_t> &list, int n_large,
                               int W, int H, int nrefs)
{
    CuLists c;
    const SlotTable &table = slot_table();
    std::vector<int> at[4];                 // record of each CU position, per size
    for (int k = 0; k < 4; k++) at[k].assign((size_t)nrefs * ((W >> (3 + k)) + 1) * ((H >> (3 + k)) + 1), -1);
    for (int q = 0; q < (int)list.size(); q++) {
        const int i = (int)list[q];
        const xavs2gpu_pu_t &p = pus[i];
        int lg = 0, cx = 0, cy = 0;
        const int slot = cu_slot(table, p, lg, cx, cy);
        bool in = slot >= 0;
        if (in) {
            const int k = lg - 3, cols = (W >> lg) + 1, rows = (H >> lg) + 1;
            int &r = at[k][((size_t)p.ref * rows + (cy >> lg)) * cols + (cx >> lg)];
            if (r < 0) {
                r = (int)c.recs.size();
                CuRec n{};
                n.x = (int16_t)cx;
                n.y = (int16_t)cy;
                n.lg = (uint8_t)lg;
                n.ref = p.ref;
                for (int &u : n.pu) u = -1;
                c.recs.push_back(n);
                c.n_rec[k]++;
            }
            int32_t &u = c.recs[r].pu[slot];
            in = u < 0;                     // a second PU of the same partition searches alone
            if (in) {
                u = i;
                (q < n_large ? c.cap_large : c.cap_small)++;
            }
        }
        if (!in) {
            c.rest.push_back((uint32_t)i);
            c.rest_large += q < n_large ? 1 : 0;
        }
    }
    return c;
}

}  // namespace xg
