// Host check of a server's waves of resident members (csrc/rtm_waves.h), over simulated server steps:
// no member is in two waves or takes SMs that are not there, every wave's blocks exist, and no member
// falls behind what it is owed, whatever the mix of grids and the steps a launch.  Prints "ok <runs>" or
// the first fault.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <tuple>

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

static std::map<std::tuple<int, int, int, int, int>, ResPart> parts;
static const ResPart *part_of(const Geom &g, int fields, int sms)
{
    auto key = std::make_tuple(g.dimx, g.dimz, g.thl, fields, sms);
    auto it = parts.find(key);
    if (it == parts.end()) {
        ResPart p;
        if (!res_partition(g, fields, 4, sms, p)) p = ResPart();
        it = parts.emplace(key, p).first;
    }
    return it->second.ctas.empty() ? nullptr : &it->second;
}

// Members of the given grids through `steps` server steps; passes that outlast them.
static int run(const char *name, const std::vector<Geom> &grids, int spl, int steps, int sms)
{
    const int n = (int)grids.size();
    std::vector<WaveMember> w(n);
    std::vector<int> gap(n, 0);
    for (int m = 0; m < n; ++m) w[m] = {m, &grids[m], m & 1, 0, 0, 0, RTM_PREC_FP32, RTM_STORE_RING};
    auto part = [&](int m, int back, int s) { return part_of(grids[m], back ? 2 : 1, s); };
    for (int k = 1; k <= steps; ++k) {
        for (auto &x : w) x.due = wave_owe(x.due, spl);
        const auto waves = res_waves(w, sms, spl, part);
        if (waves.empty()) { printf("%s, %d steps a launch: nothing runs\n", name, spl); return 1; }
        std::vector<char> seen(n, 0);
        for (int &x : gap) ++x;
        for (const auto &wave : waves) {
            int used = 0;
            for (const WaveItem &it : wave) {
                const ResPart *p = part(it.m, it.back, sms / it.share);
                if (seen[it.m]++ || !p) { printf("%s: member %d twice or without blocks\n", name, it.m); return 1; }
                used += (int)p->ctas.size();
                if (it.t0 != w[it.m].step || it.t1 <= it.t0 || it.t1 - it.t0 > kResMostSteps) { printf("%s: steps %d-%d\n", name, it.t0, it.t1); return 1; }
                w[it.m].due -= it.t1 - it.t0;
                w[it.m].step = it.t1;
                w[it.m].ran = k;
                gap[it.m] = 0;
            }
            if (used > sms) { printf("%s: %d blocks on %d SMs\n", name, used, sms); return 1; }
        }
        // W waves, n of them a step with n / W >= 1/8 and n kResMostSteps >= W spl: a wave's turn comes after
        // ceil(W / n) <= 8 steps, its members then owed less than kResMostSteps + spl, and what a launch
        // leaves over is less than spl
        for (int m = 0; m < n; ++m)
            if (gap[m] > 8 || w[m].due > kResMostSteps + 2 * spl) {
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
    const Geom big = geom(3400, 700, 50, nt), mid = geom(2000, 600, 50, nt), small = geom(400, 200, 40, nt), tiny = geom(96, 64, 16, nt);
    std::vector<Geom> mixed = {small, big, tiny, mid, small, big, mid, small, small, big, tiny, mid, big, small, mid, big, mid, tiny, small, mid, big, small, tiny, mid};
    int runs = 0;
    for (int spl : {1, 7, 16, 64, 96, 100, 128, 200, 256})
        for (int n : {1, 2, 3, 5, 8, 9, 17}) {
            if (run("large", std::vector<Geom>(n, big), spl, 60, 152)) return 1;
            if (run("small", std::vector<Geom>(n, small), spl, 40, 152)) return 1;
            if (run("mixed", std::vector<Geom>(mixed.begin(), mixed.begin() + n), spl, 60, 152)) return 1;
            runs += 3;
        }
    for (int spl : {16, 128, 256}) {
        if (run("mixed", mixed, spl, 80, 152) || run("mixed, fewer SMs", std::vector<Geom>(mixed.size(), small), spl, 80, 100)) return 1;
        runs += 2;
    }
    printf("ok %d\n", runs);
    return 0;
}
