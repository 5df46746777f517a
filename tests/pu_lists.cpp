// Compares the layout of PU lists (xavs2_gb300/csrc/pu_lists.h) with its
// definition worked out the long way -- slots by comparing geometries, the
// order by stable sorts -- over every shape and position of a CTU and over
// random lists, then times both on a list of a picture's size.  Prints the
// first difference and returns 1, or the two times in ms and returns 0.
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

static int order_by_sorts(const std::vector<xavs2gpu_pu_t> &pus, std::vector<int> &list)
{
    auto side = [&](int i) { return std::max(h_pu_w[pus[i].part], h_pu_h[pus[i].part]); };
    auto pixels = [&](int i) { return h_pu_w[pus[i].part] * h_pu_h[pus[i].part]; };
    const auto small = std::stable_partition(list.begin(), list.end(), [&](int i) { return side(i) > kSmallDim; });
    auto larger = [&](int a, int b) { return pixels(a) > pixels(b); };
    std::stable_sort(list.begin(), small, larger);
    std::stable_sort(small, list.end(), larger);
    return (int)(small - list.begin());
}

static CuLists lists_by_geometry(const std::vector<xavs2gpu_pu_t> &pus, const std::vector<uint32_t> &list, int n_large,
                                 int W, int H, int nrefs)
{
    CuLists c;
    std::vector<int> at[4];
    for (int k = 0; k < 4; k++) at[k].assign((size_t)nrefs * ((W >> (3 + k)) + 1) * ((H >> (3 + k)) + 1), -1);
    for (size_t q = 0; q < list.size(); q++) {
        const xavs2gpu_pu_t &p = pus[list[q]];
        int lg = 0, cx = 0, cy = 0;
        const int slot = slot_by_geometry(p, lg, cx, cy);
        int *r = nullptr;
        if (slot >= 0) {
            r = &at[lg - 3][((size_t)p.ref * ((H >> lg) + 1) + (cy >> lg)) * ((W >> lg) + 1) + (cx >> lg)];
            if (*r < 0) {
                *r = (int)c.recs.size();
                CuRec n{};
                n.x = (int16_t)cx; n.y = (int16_t)cy; n.lg = (uint8_t)lg; n.ref = p.ref;
                for (int &u : n.pu) u = -1;
                c.recs.push_back(n);
                c.n_rec[lg - 3]++;
            }
        }
        if (r && c.recs[*r].pu[slot] < 0) {
            c.recs[*r].pu[slot] = (int)list[q];
            ((int)q < n_large ? c.cap_large : c.cap_small)++;
        } else {
            c.rest.push_back(list[q]);
            c.rest_large += (int)q < n_large ? 1 : 0;
        }
    }
    return c;
}

static bool equal(const CuLists &a, const CuLists &b)
{
    return a.recs.size() == b.recs.size() && a.rest == b.rest && a.rest_large == b.rest_large &&
           a.cap_large == b.cap_large && a.cap_small == b.cap_small &&
           std::equal(a.n_rec, a.n_rec + 4, b.n_rec) &&
           (a.recs.empty() || memcmp(a.recs.data(), b.recs.data(), sizeof(CuRec) * a.recs.size()) == 0);
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
                int a[3] = {0, 0, 0}, b[3] = {0, 0, 0};
                const int s = cu_slot(slot_table(), p, a[0], a[1], a[2]), t = slot_by_geometry(p, b[0], b[1], b[2]);
                if (s != t || (s >= 0 && (a[0] != b[0] || a[1] != b[1] || a[2] != b[2]))) {
                    printf("slot of part %d at (%d, %d): %d, %d\n", part, x, y, s, t);
                    return 1;
                }
            }
    std::mt19937 rng(7);
    double ms[2] = {0, 0};
    for (int n : {0, 1, 5, 64, 3000, 400000}) {
        const int W = 1280, H = 720, nrefs = 2;
        std::vector<xavs2gpu_pu_t> pus(n);
        for (auto &p : pus) {   // on the grid of their size, or (one in eight) anywhere
            p = xavs2gpu_pu_t{};
            p.part = (uint8_t)(rng() % kNumParts);
            p.ref = (uint8_t)(rng() % nrefs);
            const int any = rng() % 8 == 0, w = h_pu_w[p.part], h = h_pu_h[p.part];
            p.x = (int16_t)(any ? rng() % (W - w + 1) : rng() % ((W - w) / 4 + 1) * 4);
            p.y = (int16_t)(any ? rng() % (H - h + 1) : rng() % ((H - h) / 4 + 1) * 4);
        }
        std::vector<int> a, b;
        for (int i = 0; i < n; i++)
            if (n < 10 || rng() % 10) a.push_back(i);
        b = a;
        for (int rep = 0; rep < 3; rep++) {
            std::vector<int> x = a, y = b;
            const auto t0 = std::chrono::steady_clock::now();
            const int la = per_pu_order(pus, x);
            const CuLists ca = cu_lists(pus, std::vector<uint32_t>(x.begin(), x.end()), la, W, H, nrefs);
            const auto t1 = std::chrono::steady_clock::now();
            const int lb = order_by_sorts(pus, y);
            const CuLists cb = lists_by_geometry(pus, std::vector<uint32_t>(y.begin(), y.end()), lb, W, H, nrefs);
            const auto t2 = std::chrono::steady_clock::now();
            if (x != y || la != lb || !equal(ca, cb)) {
                printf("lists of %d PUs differ\n", n);
                return 1;
            }
            const double u[2] = {std::chrono::duration<double>(t1 - t0).count() * 1e3,
                                 std::chrono::duration<double>(t2 - t1).count() * 1e3};
            for (int k = 0; k < 2; k++) ms[k] = rep == 0 ? u[k] : std::min(ms[k], u[k]);
        }
    }
    printf("%f %f\n", ms[0], ms[1]);
    return 0;
}
