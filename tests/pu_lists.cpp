// Compares the layout of PU lists (xavs2_gb300/csrc/pu_lists.h) with its
// definition worked out the long way -- slots by comparing geometries, the
// order by stable sorts, the rules one PU at a time -- over every shape and
// position of a CTU and over lists of every route, the last of a picture's size
// and timed.  Prints the first difference and returns 1, or the two times in ms
// and returns 0.
#include "pu_lists.h"

#include <algorithm>
#include <chrono>
#include <cstdio>
#include <random>

using namespace xg;

static int slot_by_geometry(const xavs2gpu_pu_t &p, int &lg, int &cx, int &cy)
{
    const int w = h_pu_w[p.part], h = h_pu_h[p.part], S = std::max(8, std::max(w, h));
    lg = S == 8 ? 3 : S == 16 ? 4 : S == 32 ? 5 : 6;
    cx = p.x & ~(S - 1);
    cy = p.y & ~(S - 1);
    for (int m = 0; m < (S == 8 ? 9 : 13); m++) {
        SlotGeom g;
        if (S == 8) {
            g = slot_geom(m);
            g.ox += cx;
            g.oy += cy;
        } else {
            g = cu_mode_geom(S, cx, cy, m);
        }
        if (g.part == p.part && g.ox == p.x && g.oy == p.y) return m;
    }
    return -1;
}

static int side(const xavs2gpu_pu_t &p) { return std::max(h_pu_w[p.part], h_pu_h[p.part]); }
static int pixels(const xavs2gpu_pu_t &p) { return h_pu_w[p.part] * h_pu_h[p.part]; }

static PerPuCounts order_by_sorts(const std::vector<xavs2gpu_pu_t> &pus, std::vector<int> &list)
{
    PerPuCounts c;
    auto large = [&](int i) { return side(pus[i]) > 16; };
    auto mid = [&](int i) { return side(pus[i]) == 16; };
    const auto a = std::stable_partition(list.begin(), list.end(), large);
    const auto b = std::stable_partition(a, list.end(), mid);
    auto larger = [&](int x, int y) { return pixels(pus[x]) > pixels(pus[y]); };
    std::stable_sort(list.begin(), a, larger);
    std::stable_sort(a, b, larger);
    std::stable_sort(b, list.end(), larger);
    c.n_large = (int)(a - list.begin());
    c.n_mid = (int)(b - a);
    for (int i : list) c.part[pus[i].part]++;
    return c;
}

// every CU with a PU, then the rules on them one PU at a time
static CuLists lists_by_geometry(const std::vector<xavs2gpu_pu_t> &pus, const std::vector<uint32_t> &list, int W, int H,
                                 int nrefs, int R, size_t means)
{
    CuLists c;
    std::vector<int> at[4], of(pus.size(), -1);
    for (int k = 0; k < 4; k++) at[k].assign((size_t)nrefs * ((W >> (3 + k)) + 1) * ((H >> (3 + k)) + 1), -1);
    for (uint32_t i : list) {
        const xavs2gpu_pu_t &p = pus[i];
        int lg = 0, cx = 0, cy = 0;
        const int slot = slot_by_geometry(p, lg, cx, cy);
        if (slot < 0) continue;
        int &r = at[lg - 3][((size_t)p.ref * ((H >> lg) + 1) + (cy >> lg)) * ((W >> lg) + 1) + (cx >> lg)];
        if (r < 0) {
            r = (int)c.recs.size();
            CuRec n{};
            n.x = (int16_t)cx; n.y = (int16_t)cy; n.lg = (uint8_t)lg; n.ref = p.ref;
            for (int &u : n.pu) u = -1;
            c.recs.push_back(n);
        }
        if (c.recs[r].pu[slot] >= 0) continue;
        c.recs[r].pu[slot] = (int)i;
        of[i] = r;
    }
    std::vector<char> keep(c.recs.size());
    int lg_max = 0;
    for (size_t r = 0; r < c.recs.size(); r++) {
        int members = 0, area = 0;
        for (int u : c.recs[r].pu)
            if (u >= 0) members++, area += pixels(pus[u]);
        keep[r] = members >= 4 && (c.recs[r].lg < 5 || area >= 3 * (1 << c.recs[r].lg) * (1 << c.recs[r].lg));
        if (keep[r]) lg_max = std::max(lg_max, (int)c.recs[r].lg);
    }
    double all = 0, in = 0;
    long long area = 0;
    for (uint32_t i : list) {
        all += plain_ns(pus[i].part, R);
        area += pixels(pus[i]);
        if (of[i] >= 0 && keep[of[i]]) in += plain_ns(pus[i].part, R);
    }
    const bool clusters = kClusterSaves * in > kClusterNs && area >= (long long)kClusterAreas << (2 * lg_max);
    if (clusters && in >= kClusterAll * all) std::fill(keep.begin(), keep.end(), 1);
    double bounded = 0;
    for (uint32_t i : list) {
        const bool kept = clusters && of[i] >= 0 && keep[of[i]];
        if (kept) {
            (side(pus[i]) > 16 ? c.cap_large : c.cap_small)++;
            continue;
        }
        c.rest.push_back(i);
        if (side(pus[i]) > 16 ? R >= 8 : side(pus[i]) == 16 && R >= 48) {
            bounded += plain_ns(pus[i].part, R);
            (side(pus[i]) > 16 ? c.bounded.n_large : c.bounded.n_small)++;
        }
    }
    const double saved = kBoundedSaves * bounded - kBoundedNs;
    if (saved <= 0) c.bounded = BoundedPart{};
    c.use = (clusters ? kClusterSaves * in - kClusterNs : 0) + std::max(saved, 0.0) > means_ns(means);
    std::vector<CuRec> recs;
    for (size_t r = 0; r < c.recs.size(); r++)
        if (c.use && clusters && keep[r]) {
            recs.push_back(c.recs[r]);
            c.n_rec[c.recs[r].lg - 3]++;
        }
    c.recs = recs;
    if (!c.use) {
        c.rest = list;
        c.bounded = BoundedPart{};
        c.cap_large = c.cap_small = 0;
    }
    return c;
}

static bool equal(const CuLists &a, const CuLists &b)
{
    return a.use == b.use && a.recs.size() == b.recs.size() && (!a.use || a.rest == b.rest) &&
           a.cap_large == b.cap_large && a.cap_small == b.cap_small && a.bounded.n_large == b.bounded.n_large &&
           a.bounded.n_small == b.bounded.n_small && std::equal(a.n_rec, a.n_rec + 4, b.n_rec) &&
           (a.recs.empty() || memcmp(a.recs.data(), b.recs.data(), sizeof(CuRec) * a.recs.size()) == 0);
}

// PUs of the CTUs' slots inside the picture, `share` percent of them in columns
// up to `split`, `other` beyond; one in sixteen then moved off its slot
static std::vector<xavs2gpu_pu_t> make_list(std::mt19937 &rng, int W, int H, int nrefs, int share, int split, int other,
                                            unsigned kinds)
{
    std::vector<xavs2gpu_pu_t> pus;
    for (int ref = 0; ref < nrefs; ref++)
        for (int y = 0; y < H; y += 64)
            for (int x = 0; x < W; x += 64)
                for (int s = 0; s < kSlots; s++) {
                    const SlotGeom g = slot_geom(s);
                    const int w = h_pu_w[g.part], h = h_pu_h[g.part];
                    if (x + g.ox + w > W || y + g.oy + h > H) continue;
                    const int lg = s < 576 ? 0 : s < 784 ? 1 : s < 836 ? 2 : 3;
                    if (!(kinds >> lg & 1) || (int)(rng() % 100) >= (x < split ? share : other)) continue;
                    xavs2gpu_pu_t p{};
                    p.x = (int16_t)(x + g.ox);
                    p.y = (int16_t)(y + g.oy);
                    p.part = (uint8_t)g.part;
                    p.ref = (uint8_t)ref;
                    if (rng() % 16 == 0) {
                        p.x = (int16_t)(rng() % (W - w + 1));
                        p.y = (int16_t)(rng() % (H - h + 1));
                    }
                    pus.push_back(p);
                    if (rng() % 50 == 0) pus.push_back(p);   // a partition twice
                }
    return pus;
}

int main()
{
    for (int part = 0; part < kNumParts; part++)
        for (int y = 0; y < 130; y++)
            for (int x = 0; x < 130; x++) {
                xavs2gpu_pu_t p{};
                p.part = (uint8_t)part;
                p.x = (int16_t)x;
                p.y = (int16_t)y;
                int a = 0, b = 0, cx = 0, cy = 0;
                const int s = cu_slot(slot_table(), slot_of_cu(), p, a), t = slot_by_geometry(p, b, cx, cy);
                if (s != t || (s >= 0 && a != b)) {
                    printf("slot of part %d at (%d, %d): %d, %d\n", part, x, y, s, t);
                    return 1;
                }
            }
    std::mt19937 rng(7);
    double ms[2] = {0, 0};
    int routes[4] = {0, 0, 0, 0};   // plain, bounded, clusters, clusters with others left
    struct { int W, H, nrefs, share, split, other; unsigned kinds; int R; } cases[] = {
        {64, 64, 1, 0, 0, 0, 15, 16},         {128, 72, 1, 100, 128, 0, 15, 64},   {416, 240, 1, 100, 416, 0, 15, 16},
        {416, 240, 1, 100, 416, 0, 15, 7},    {416, 240, 1, 20, 416, 0, 15, 64},   {416, 240, 2, 100, 128, 0, 15, 64},
        {416, 240, 2, 100, 416, 0, 1, 64},    {416, 240, 2, 100, 416, 0, 2, 8},    {640, 360, 2, 30, 640, 0, 15, 48},
        {640, 360, 2, 30, 640, 0, 15, 16},    {640, 360, 2, 100, 256, 30, 15, 48}, {640, 360, 2, 100, 256, 30, 15, 16},
        {640, 360, 2, 100, 256, 30, 3, 4},    {640, 360, 2, 60, 640, 0, 12, 32},   {1280, 720, 2, 5, 1280, 0, 15, 64},
        {1280, 720, 2, 5, 1280, 0, 1, 64},    {1280, 720, 2, 50, 64, 2, 15, 128},  {1280, 720, 2, 100, 1280, 0, 15, 64}};
    for (const auto &t : cases) {
        const std::vector<xavs2gpu_pu_t> pus = make_list(rng, t.W, t.H, t.nrefs, t.share, t.split, t.other, t.kinds);
        const size_t means = (size_t)((t.W + 223) / 64 * 64) * (t.H + 160) * t.nrefs;
        std::vector<int> a;
        for (int i = 0; i < (int)pus.size(); i++)
            if (rng() % 20) a.push_back(i);
        for (int rep = 0; rep < 3; rep++) {
            std::vector<int> x = a, y = a;
            const auto t0 = std::chrono::steady_clock::now();
            const PerPuCounts pa = per_pu_order(pus, x);
            const CuLists ca =
                cu_lists(pus, std::vector<uint32_t>(x.begin(), x.end()), pa, t.W, t.H, t.nrefs, t.R, means);
            const auto t1 = std::chrono::steady_clock::now();
            const PerPuCounts pb = order_by_sorts(pus, y);
            const CuLists cb = lists_by_geometry(pus, std::vector<uint32_t>(y.begin(), y.end()), t.W, t.H, t.nrefs, t.R, means);
            const auto t2 = std::chrono::steady_clock::now();
            if (x != y || pa.n_large != pb.n_large || pa.n_mid != pb.n_mid ||
                !std::equal(pa.part, pa.part + kNumParts, pb.part) || !equal(ca, cb)) {
                printf("lists of %d PUs of %dx%d at R = %d differ\n", (int)a.size(), t.W, t.H, t.R);
                return 1;
            }
            const double u[2] = {std::chrono::duration<double>(t1 - t0).count() * 1e3,
                                 std::chrono::duration<double>(t2 - t1).count() * 1e3};
            for (int k = 0; k < 2; k++) ms[k] = rep == 0 ? u[k] : std::min(ms[k], u[k]);
            if (rep == 0) routes[!ca.use ? 0 : ca.recs.empty() ? 1 : ca.rest.size() * 10 < a.size() ? 2 : 3]++;
        }
    }
    // lists that measured slower by clusters or bounded searches stay plain:
    // the first PUs of one to a few CTUs, few PUs on a large picture
    for (int n : {64, 256, 1024, 4096})
        for (int R : {4, 8, 16, 64}) {
            std::vector<xavs2gpu_pu_t> pus = make_list(rng, 320, 192, 1, 100, 320, 0, 15);
            pus.resize(n);
            std::vector<int> x(n);
            for (int i = 0; i < n; i++) x[i] = i;
            const PerPuCounts c = per_pu_order(pus, x);
            const std::vector<uint32_t> l(x.begin(), x.end());
            const BoundedPart b = bounded_batch(c, 8, (size_t)4 * 4032 * 2320);
            if (cu_lists(pus, l, c, 320, 192, 1, R, 512 * 352).use || (n <= 256 && b.n_large + b.n_small > 0)) {
                printf("%d PUs at R = %d not plain\n", n, R);
                return 1;
            }
        }
    for (int k = 0; k < 4; k++)
        if (!routes[k]) {
            printf("no list took route %d\n", k);
            return 1;
        }
    printf("%f %f\n", ms[0], ms[1]);
    return 0;
}
