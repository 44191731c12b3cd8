// Host check of a server's waves of resident members (csrc/rtm_waves.h), over simulated server steps:
// no member is in two waves or takes SMs that are not there, every wave's blocks exist, its mailboxes and
// staged slots fit the room it is given and hold what its steps touch, and no member falls behind what it
// is owed, whatever the mix of grids and the steps a launch.  Prints "ok <runs>" or the first fault.
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "rtm_waves.h"

using namespace rtm;

static Geom geom(int nx, int nz, int th, int nt)
{
    Geom g;
    memset(&g, 0, sizeof g);
    g.nx = nx; g.nz = nz; g.thl = g.thr = g.thu = g.thd = th;
    g.dimx = nx + 2 * th; g.dimz = nz + 2 * th;
    g.rx0 = th - 4; g.rx1 = g.dimx - th + 4;
    g.rz0 = (th - 4 + 3) & ~3; g.rz1 = (g.dimz - th + 4) & ~3;
    g.nt = nt; g.slices = 4;
    return g;
}

static ResPartCache parts;
static const ResPart *part_of(const Geom &g, int fields, int sms) { return parts.get(g, fields, sms); }

// Slots of the store that steps [t0, t1) of a pass write or read, from the kernel's own use of them.
static bool slot_used(const WaveMember &w, int t0, int t1, int slot)
{
    const int nt = w.g->nt, sl = w.g->slices;
    for (int t = t0; t < t1; ++t) {
        if (w.storage == RTM_STORE_RING) {
            if (!w.back && t + 1 < nt && t + 1 == slot) return true;       // the ring of u_{t+1}
            if (w.back && t >= 2 && nt - t == slot) return true;           // of u_{nt-t}
        } else {
            const int tau = w.back ? nt - 1 - t : t;
            if (tau % sl == 0 && tau / sl == slot) return true;
        }
    }
    return w.storage == RTM_STORE_RING && w.back && t1 > 3 && nt - t1 + 2 == slot;   // handed on at the end
}

struct Member {
    Geom g;
    int precision, storage;
};

// The members through `steps` server steps.  Passes start over when they end; room (0: what a
// whole chip of full blocks takes, and no bound of the staging) starts at the least that each needs alone.
static int run(const char *name, const std::vector<Member> &ms, int spl, int steps, int sms, WaveRoom room = {0, 0})
{
    const int n = (int)ms.size();
    const bool tight = room.stage_elems != 0;
    if (!tight) room = {(size_t)sms * kResMostXchQuads, (size_t)1 << 40};
    std::vector<WaveMember> w(n);
    std::vector<int> gap(n, 0);
    for (int m = 0; m < n; ++m) {
        const Geom &g = ms[m].g;
        const size_t slot = ms[m].storage == RTM_STORE_RING ? 8 * (size_t)(g.dimx + g.dimz) : (size_t)g.nx * g.dimz;
        w[m] = {m, &g, m & 1, 0, 0, 0, ms[m].precision, ms[m].storage, slot};
    }
    auto part = [&](int m, int back, int s) { return part_of(ms[m].g, back && ms[m].storage == RTM_STORE_RING ? 2 : 1, s); };
    for (int k = 1; k <= steps; ++k) {
        for (auto &x : w) x.due = wave_owe(x.due, spl);
        const auto waves = res_waves(w, sms, spl, room, part);
        if (waves.empty()) { printf("%s, %d steps a launch: nothing runs\n", name, spl); return 1; }
        std::vector<char> seen(n, 0);
        for (int &x : gap) ++x;
        for (const auto &wave : waves) {
            int used = 0;
            size_t xch = 0, stage = 0;
            for (const WaveItem &it : wave) {
                WaveMember &x = w[it.m];
                const ResPart *p = part(it.m, it.back, sms / it.share);
                if (seen[it.m]++ || !p) { printf("%s: member %d twice or without blocks\n", name, it.m); return 1; }
                used += (int)p->ctas.size();
                xch += p->xch_quads;
                stage += wave_stage(x, it);
                if (it.t0 != x.step || it.t1 <= it.t0 || it.t1 > x.g->nt || it.t1 - it.t0 > std::min(kResMostSteps, x.due)) {
                    printf("%s: steps %d-%d\n", name, it.t0, it.t1);
                    return 1;
                }
                if (x.precision != RTM_PREC_FP32 && x.g->nt < 4096)
                    for (int slot = 0; slot <= x.g->nt; ++slot)
                        if (slot_used(x, it.t0, it.t1, slot) && (slot < it.lo || slot > it.hi)) {
                            printf("%s: pass %d, steps %d-%d touch slot %d, staged %d-%d\n", name, x.back, it.t0, it.t1, slot, it.lo, it.hi);
                            return 1;
                        }
                x.due -= it.t1 - it.t0;
                x.step = it.t1;
                if (x.step == x.g->nt) { x.step = x.due = 0; x.back ^= 1; }
                x.ran = k;
                gap[it.m] = 0;
            }
            if (used > sms) { printf("%s: %d blocks on %d SMs\n", name, used, sms); return 1; }
            if (xch > room.xch_quads || stage > room.stage_elems) {
                printf("%s, %d steps a launch: %zu quads, %zu elements in a room of %zu, %zu\n", name, spl, xch, stage, room.xch_quads, room.stage_elems);
                return 1;
            }
        }
        // W waves, n of them a step with n / W >= 1/8 and n kResMostSteps >= W spl: a wave's turn comes after
        // ceil(W / n) <= 8 steps, its members then owed less than kResMostSteps + spl, and what a launch
        // leaves over is less than spl
        for (int m = 0; m < n; ++m)
            if (gap[m] > 8 || (!tight && w[m].due > kResMostSteps + 2 * spl)) {
                printf("%s, %d steps a launch, server step %d: member %d waits since %d steps, owed %d (done %d)\n", name, spl, k,
                       m, gap[m], w[m].due, w[m].step);
                return 1;
            }
    }
    return 0;
}

int main()
{
    const int nt = 1 << 24;
    auto fp32 = [](const Geom &g) { return Member{g, RTM_PREC_FP32, RTM_STORE_RING}; };
    const Member big = fp32(geom(3400, 700, 50, nt)), mid = fp32(geom(2000, 600, 50, nt)), small = fp32(geom(400, 200, 40, nt)),
                 tiny = fp32(geom(96, 64, 16, nt));
    std::vector<Member> mixed = {small, big, tiny, mid, small, big, mid, small, small, big, tiny, mid, big, small, mid, big, mid, tiny, small, mid, big, small, tiny, mid};
    int runs = 0;
    for (int spl : {1, 7, 16, 64, 96, 100, 128, 200, 256})
        for (int n : {1, 2, 3, 5, 8, 9, 17}) {
            if (run("large", std::vector<Member>(n, big), spl, 60, 152)) return 1;
            if (run("small", std::vector<Member>(n, small), spl, 40, 152)) return 1;
            if (run("mixed", std::vector<Member>(mixed.begin(), mixed.begin() + n), spl, 60, 152)) return 1;
            runs += 3;
        }
    for (int spl : {16, 128, 256}) {
        if (run("mixed", mixed, spl, 80, 152) || run("mixed, fewer SMs", std::vector<Member>(mixed.size(), small), spl, 80, 100)) return 1;
        runs += 2;
    }
    // 16-bit rings and snapshots, short passes, rooms from the least that one of them needs upwards
    std::vector<Member> half;
    for (int k = 0; k < 14; ++k) {
        const int g[4][3] = {{400, 200, 40}, {2000, 600, 50}, {97, 61, 17}, {1201, 403, 41}};
        Geom x = geom(g[k % 4][0], g[k % 4][1], g[k % 4][2], 60 + 4 * (k % 5));
        x.slices = k % 3 == 0 ? 1 : 4;
        half.push_back({x, k % 5 == 4 ? RTM_PREC_FP32 : k & 1 ? RTM_PREC_BF16 : RTM_PREC_FP16, k & 2 ? RTM_STORE_SNAPSHOT : RTM_STORE_RING});
    }
    size_t least = 0, most = 0;
    for (const Member &m : half) {
        least = std::max(least, wave_least_stage(m.precision, m.storage, m.storage == RTM_STORE_RING ? 8 * (size_t)(m.g.dimx + m.g.dimz) : (size_t)m.g.nx * m.g.dimz));
        for (int f = 1; f <= 2; ++f) most = std::max(most, part_of(m.g, f, 152)->xch_quads);
    }
    for (int spl : {1, 2, 16, 100, 256})
        for (size_t k : {1, 2, 5, 40}) {
            if (run("16-bit", half, spl, 60, 152, {most * std::min<size_t>(k, 3), least * k})) return 1;
            ++runs;
        }
    // partitions: what hundreds of members of different grids use is searched for once, and goes once they have
    ResPartCache c;
    for (int k = 0; k < 80; ++k) {
        c.step();
        for (int m = 0; m < 300; ++m)
            for (int f = 1; f <= 2; ++f) c.get(geom(64 + m, 48, 16, 8), f, 8);
    }
    if (c.searches() != 600) { printf("%lld partitions searched for 600\n", c.searches()); return 1; }
    for (int k = 0; k < 2 * kResKeepSteps + 1; ++k) {
        c.step();
        c.get(geom(64, 48, 16, 8), 1, 8);
    }
    if (c.size() > kResKeepParts) { printf("%zu partitions kept of grids long gone\n", c.size()); return 1; }
    printf("ok %d\n", runs);
    return 0;
}
