// rtm_partition.h -- blocks of a resident pass (k_resident, rtm_resident.cu): host code only.
//
// The grid's updated cells [4, dimX-4) x [4, dimZ-4) are cut into PX x PZ blocks, at most one per
// SM, by straight cuts (a tensor grid: a side of a block faces exactly one neighbour).  A cell of a
// CPML strip costs more than a plain one, so the cuts run through equal weights, not equal widths;
// the search tries the factorisations of the SM count with a few strip weights and keeps the one
// whose most expensive block is cheapest and fits a block's shared and tensor memory.
#pragma once

#include <algorithm>
#include <cmath>
#include <map>
#include <tuple>
#include <vector>

#include "rtm_internal.h"

namespace rtm {

struct ResPart {
    std::vector<int> xcut, zcut;       // PX + 1, PZ + 1 bounds
    std::vector<ResCta> ctas;          // x-major
    int cw = 0;                        // the most columns of a chunk (at least 3: the general kernel is needed)
    size_t smem = 0;                   // dynamic shared memory (bytes)
    size_t xch_quads = 0;              // exchange buffer
    double cost = 0.0;
};

// Bounds of `parts` pieces of [lo, hi) (each a multiple of `step`) of about equal weight, cells of
// [lo, s0) and [s1, hi) weighing w, the others 1; empty when a piece would be narrower than 8.
inline std::vector<int> res_cuts(int lo, int hi, int s0, int s1, double w, int parts, int step)
{
    s0 = std::min(std::max(s0, lo), hi);
    s1 = std::min(std::max(s1, s0), hi);
    const double wa = w * (s0 - lo), wb = s1 - s0, wc = w * (hi - s1), all = wa + wb + wc;
    std::vector<int> c(parts + 1);
    c[0] = lo;
    for (int k = 1; k < parts; ++k) {
        const double t = all * k / parts;
        const double p = t < wa ? lo + t / w : t < wa + wb ? s0 + (t - wa) : s1 + (t - wa - wb) / w;
        c[k] = lo + (int)((p - lo) / step + 0.5) * step;
    }
    c[parts] = hi;
    if (parts > 1)
        for (int k = 0; k < parts; ++k)
            if (c[k + 1] - c[k] < 8) return {};
    return c;
}

// Time of a block's step in ns, from the phases' times on GB300 (clock64 around them, 400 x 200,
// 2000 x 600 and 3400 x 700 grids): a column of the leapfrog 330, and 100 to swap it into the tile; a
// column of a top or bottom strip 520, of a left or right one 500 (only the columns in it); psi 550
// (left, right) and 350 (top, bottom) a round of the threads over its quads; a halo round 400; the
// ring 800.  Scaling the strips', psi's, halo's or ring's share by 0.6 to 1.5 gained nothing over nine
// grids from 400 x 200 to 3400 x 700 (most stayed within 2 %, the worst lost 30 %).
// Double runs at the FP64 pipe's pace (2 operations a cycle and SM): 20 operations a cell and field
// and 36 more a strip, and half as long again when a thread's values do not fit its registers.
inline double res_cost(const ResShape &s, int fields, int es)
{
    if (es == 8) {
        const double ops = 20.0 * fields * s.W * s.H + 36.0 * (s.nl + s.nr) * s.H + 36.0 * (s.ht + s.hb) * s.W +
                           9.0 * ((s.nl ? 8 : 0) + (s.nr ? 8 : 0)) * s.H + 9.0 * ((s.ht ? 8 : 0) + (s.hb ? 8 : 0)) * s.W;
        return (ops / 3.8 + 1500.0) * (s.CW > 1 ? 1.5 : 1.0);
    }
    const int nx = std::max(s.nl, s.nr);
    double c = s.CW * fields * 430.0;
    if (s.zslot >= 0) c += 520.0 * s.CW;
    if (s.xslot >= 0) c += 500.0 * std::min(s.CW, nx);
    auto rounds = [](int cols, int rows) {
        const int per = kResThreads / std::max(rows, 1);
        return per > 0 ? (cols + per - 1) / per : 1 << 20;
    };
    if (s.nl) c += 250.0 + 550.0 * rounds(s.nl + 8, s.HQ);
    if (s.nr) c += 250.0 + 550.0 * rounds(s.nr + 8, s.HQ);
    if (s.ht) c += 250.0 + 350.0 * rounds(s.W, s.ht / 4 + 1);
    if (s.hb) c += 250.0 + 350.0 * rounds(s.W, s.hb / 4 + 1);
    const double halo = (s.xslot >= 0 ? 16.0 : 8.0) * s.HQ + (s.zslot >= 0 ? 4.0 : 2.0) * s.W + (fields - 1) * (8.0 * s.HQ + 2.0 * s.W);
    c += 800.0 * halo / kResThreads;
    if (s.ring) c += 800.0;
    return c;
}

inline size_t res_bytes(const ResShape &s, int es) { return es == 8 ? res_smem<double>(s) : res_smem<float>(s); }

// A step with two columns in registers (k_resident's NC), or more in tensor memory, against one:
// 400 x 200 2.84 us with one, 3.22 with two; 901 x 301 4.14 with two, 5.57 with more, 600 x 300
// 4.22 and 1600 x 100 4.50 with two (1.2 and any factor from 1.3 to 1.6 choose the better there
// and on 11 more grids; 2.0 takes 1201 x 403 from 6.04 to 6.38).
inline double res_kind(int cw) { return cw == 1 ? 1.0 : cw == 2 ? 1.2 : 1.5; }

// Halo quads of a block in one direction at most: 8 columns or 2 rows of quads of the first field
// across each side (a neighbour in a strip needs them), 4 and 1 of the second.
inline int res_halo_most(const ResShape &s) { return 2 * (8 + 4) * s.HQ + 2 * (2 + 1) * s.W; }

// es: bytes of a value; fields: 1 (u, or the receiver field) or 2 (with the source field).
inline bool res_fits(const ResShape &s, int es)
{
    return s.HQ >= 1 && s.HQ <= kResThreads && s.W <= kResThreads && 2 * s.W + 8 * s.HQ <= 2 * kResThreads &&
           s.CW <= kResCols && (s.CW * s.nslot + s.CW - 1) * es <= kResTmemWords &&
           res_halo_most(s) <= kResItems * kResThreads &&
           (s.nslot > 1 ? 2 : 1) * s.field < (1 << 17) && res_bytes(s, es) <= (size_t)kResSmem;
}

// Blocks of a pass on `sms` SMs; false when no partition fits.
inline bool res_partition(const Geom &g, int fields, int es, int sms, ResPart &out)
{
    const int X0 = 4, X1 = g.dimx - 4, Z0 = 4, Z1 = ((g.dimz - 4) + 3) & ~3;
    const double weights[7] = {1.0, 1.3, 1.7, 2.2, 2.8, 3.5, 4.5};
    bool found = false;
    // the pieces of one axis: of the plain ones (clear of the strips and of the ring, [s0, s1) and
    // [r0, r1)) one of each width, and all the others
    struct Kinds { int n, lo[64], hi[64]; std::vector<int> cut; };
    auto kinds = [](std::vector<int> cut, int s0, int s1, int r0, int r1, Kinds &k) {
        k.n = cut.empty() ? 64 : 0;
        const int p0 = std::max(s0, r0), p1 = std::min(s1, r1);
        int w[4] = {0, 0, 0, 0}, nw = 0;               // plain widths differ by rounding only
        for (size_t i = 0; i + 1 < cut.size() && k.n < 64; ++i) {
            if (cut[i] >= p0 && cut[i + 1] <= p1) {
                const int width = cut[i + 1] - cut[i];
                if (width == w[0] || width == w[1] || width == w[2] || width == w[3]) continue;
                if (nw < 4) w[nw++] = width;
            }
            k.lo[k.n] = cut[i];
            k.hi[k.n++] = cut[i + 1];
        }
        k.cut = std::move(cut);
    };
    // the most expensive block: false when one does not fit, or costs `most`
    auto measure = [&](const Kinds &kx, const Kinds &kz, double most, double &cost, int &cw, size_t &smem) {
        cost = 0.0;
        cw = 0;
        smem = 0;
        for (int i = 0; i < kx.n; ++i)
            for (int k = 0; k < kz.n; ++k) {
                const ResShape s = res_shape(g, kx.lo[i], kx.hi[i], kz.lo[k], kz.hi[k], fields, es);
                if (!res_fits(s, es)) return false;
                cost = std::max(cost, res_cost(s, fields, es));
                if (cost >= most) return false;
                // both strips of an axis in one block: the general kernel (NC = 0)
                cw = std::max(cw, (s.nl && s.nr) || (s.ht && s.hb) ? std::max(3, s.CW) : s.CW);
                smem = std::max(smem, res_bytes(s, es));
            }
        if (es == 4) cost *= res_kind(cw);
        return cost < most;
    };
    const double cells = (double)(X1 - X0) * (Z1 - Z0);
    std::vector<Kinds> kx(7), kz(7);
    int px_of_kx = -1;
    for (int pz = 1; pz <= std::min(sms, std::max(1, (Z1 - Z0) / 8)); ++pz) {
        const int px = std::min(sms / pz, std::max(1, (X1 - X0) / 8));
        const double quads = cells / (4.0 * kResThreads * px * pz);       // a thread's, of the mean block
        const int least = std::max(1, (int)std::ceil(quads - 1e-9));
        if (found && (es == 8 ? quads * fields : least * fields * 430.0 * res_kind(least)) > out.cost) continue;
        for (int w = 0; w < 7; ++w)
            kinds(res_cuts(Z0, Z1, g.thu - 4, g.dimz - g.thd + 4, weights[w], pz, 4), g.thu - 4, g.dimz - g.thd + 4, g.rz0,
                  g.rz1, kz[w]);
        for (int w = 0; w < 7 && px != px_of_kx; ++w)
            kinds(res_cuts(X0, X1, g.thl - 4, g.dimx - g.thr + 4, weights[w], px, 1), g.thl - 4, g.dimx - g.thr + 4, g.rx0,
                  g.rx1, kx[w]);
        px_of_kx = px;
        for (const Kinds &z : kz)
            for (const Kinds &x : kx) {
                double cost;
                int cw;
                size_t smem;
                if (x.n >= 64 || z.n >= 64 || !measure(x, z, found ? out.cost : 1e30, cost, cw, smem)) continue;
                found = true;
                out.xcut = x.cut;
                out.zcut = z.cut;
                out.cost = cost;
                out.cw = cw;
                out.smem = smem;
            }
    }
    if (!found) return false;
    // mailboxes: one a side with a neighbour, (field, parity) boxes of its depth
    const int px = (int)out.xcut.size() - 1, pz = (int)out.zcut.size() - 1;
    out.ctas.assign((size_t)px * pz, ResCta{});
    size_t off = 0;
    auto at = [&](int i, int k) -> ResCta & { return out.ctas[(size_t)i * pz + k]; };
    auto in_s = [&](const ResCta &c) {
        return c.xa < g.rx1 + 4 && c.xb > g.rx0 - 4 && c.za < g.rz1 + 4 && c.zb > g.rz0 - 4;
    };
    for (int i = 0; i < px; ++i)
        for (int k = 0; k < pz; ++k) {
            ResCta &c = at(i, k);
            c.xa = out.xcut[i]; c.xb = out.xcut[i + 1];
            c.za = out.zcut[k]; c.zb = out.zcut[k + 1];
        }
    for (int i = 0; i < px; ++i)
        for (int k = 0; k < pz; ++k) {
            ResCta &c = at(i, k);
            const ResShape s = res_shape(g, c.xa, c.xb, c.za, c.zb, fields, es);
            const int di[4] = {-1, 1, 0, 0}, dk[4] = {0, 0, -1, 1};
            for (int side = 0; side < 4; ++side) {
                const int ni = i + di[side], nk = k + dk[side];
                if (ni < 0 || ni >= px || nk < 0 || nk >= pz) continue;
                ResCta &n = at(ni, nk);
                const bool x = side < 2;
                c.din[side] = x ? (s.xslot >= 0 ? 8 : 4) : (s.zslot >= 0 ? 2 : 1);
                c.in_cap[side] = c.din[side] * (x ? s.HQ : s.W);
                c.in_off[side] = (unsigned)off;
                off += (size_t)c.in_cap[side] * 2 * fields;
                c.sx[side] = fields == 2 && in_s(c) && in_s(n);
                const int opp = side ^ 1;
                n.dout[opp] = c.din[side];
                n.out_off[opp] = c.in_off[side];
                n.out_cap[opp] = c.in_cap[side];
            }
        }
    out.xch_quads = off;
    return true;
}

// Partitions of the grids that a server's members have, by shape and SM share.  A search takes 0.02 to 0.7 ms
// on the host, so that what the members at hand use is kept however many they are (400 members of 600 x 300
// to 1797 x 300, 200 steps a pass: 933 ms, and 1612 when all were dropped at 256 entries); what went unused
// for kResKeepSteps steps goes once there are more than kResKeepParts.
constexpr size_t kResKeepParts = 256;
constexpr int kResKeepSteps = 16;
class ResPartCache {
    struct Kept { ResPart part; long long used; };
    std::map<std::tuple<int, int, int, int, int, int, int, int>, Kept> kept_;
    long long now_ = 0, searches_ = 0;

public:
    // A server step begins: pointers from get() end here.
    void step()
    {
        if (++now_ % kResKeepSteps != 0 || kept_.size() <= kResKeepParts) return;
        for (auto it = kept_.begin(); it != kept_.end();)
            it = it->second.used + kResKeepSteps < now_ ? kept_.erase(it) : std::next(it);
    }
    // Blocks of a pass in 32 bits on `sms` SMs, or NULL when they do not fit.
    const ResPart *get(const Geom &g, int fields, int sms)
    {
        const auto key = std::make_tuple(g.dimx, g.dimz, g.thl, g.thr, g.thu, g.thd, fields, sms);
        auto it = kept_.find(key);
        if (it == kept_.end()) {
            ResPart part;
            if (!res_partition(g, fields, 4, sms, part)) part = ResPart();
            it = kept_.emplace(key, Kept{std::move(part), 0}).first;
            ++searches_;
        }
        it->second.used = now_;
        return it->second.part.ctas.empty() ? nullptr : &it->second.part;
    }
    size_t size() const { return kept_.size(); }
    long long searches() const { return searches_; }
};

}  // namespace rtm
