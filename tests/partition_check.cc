// Host check of the resident passes' partition (csrc/rtm_partition.h): every updated cell in exactly
// one block, blocks within a CTA's limits, each mailbox written by the neighbour that faces it with the
// depth its reader expects, mailboxes disjoint.  Prints "ok <grids>" or the first fault.
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "rtm_partition.h"

using namespace rtm;

static int fault(const char *what, const Geom &g, int fields, int es)
{
    printf("%s: %d x %d, CPML %d %d %d %d, fields %d, %d-byte values\n", what, g.nx, g.nz, g.thl, g.thr, g.thu, g.thd,
           fields, es);
    return 1;
}

static int check(int nx, int nz, int l, int r, int u, int d, int fields, int es, int sms, int &found)
{
    Geom g;
    memset(&g, 0, sizeof g);
    g.nx = nx; g.nz = nz; g.thl = l; g.thr = r; g.thu = u; g.thd = d;
    g.dimx = l + nx + r; g.dimz = u + nz + d;
    g.rx0 = l - 4; g.rx1 = g.dimx - r + 4;
    g.rz0 = (u - 4 + 3) & ~3; g.rz1 = (g.dimz - d + 4) & ~3;
    ResPart p;
    if (!res_partition(g, fields, es, sms, p)) return 0;
    ++found;
    const int px = (int)p.xcut.size() - 1, pz = (int)p.zcut.size() - 1;
    if ((int)p.ctas.size() != px * pz || px * pz > sms) return fault("block count", g, fields, es);
    if (p.xcut[0] != 4 || p.xcut[px] != g.dimx - 4 || p.zcut[0] != 4 || p.zcut[pz] < g.dimz - 4 || p.zcut[pz] > g.dimz + 3)
        return fault("cuts do not span the grid", g, fields, es);
    std::vector<char> used(p.xch_quads, 0);
    for (int i = 0; i < px; ++i)
        for (int k = 0; k < pz; ++k) {
            const ResCta &c = p.ctas[(size_t)i * pz + k];
            if (c.xa != p.xcut[i] || c.xb != p.xcut[i + 1] || c.za != p.zcut[k] || c.zb != p.zcut[k + 1] || c.za % 4 ||
                (c.zb - c.za) % 4 || c.xb <= c.xa || c.zb <= c.za)
                return fault("block bounds", g, fields, es);
            const ResShape s = res_shape(g, c.xa, c.xb, c.za, c.zb, fields, es);
            if (!res_fits(s, es) || res_bytes(s, es) > p.smem || s.CW > p.cw) return fault("block does not fit", g, fields, es);
            if (s.K * s.HQ > kResThreads || s.K * s.CW < s.W) return fault("threads do not cover a block", g, fields, es);
            int items = 0;
            for (int side = 0; side < 4; ++side) {
                const int ni = i + (side == 0 ? -1 : side == 1), nk = k + (side == 2 ? -1 : side == 3);
                const bool have = ni >= 0 && ni < px && nk >= 0 && nk < pz;
                if (have != (c.din[side] > 0) || have != (c.dout[side] > 0)) return fault("neighbour", g, fields, es);
                if (!have) continue;
                const ResCta &n = p.ctas[(size_t)ni * pz + nk];
                const int len = side < 2 ? s.HQ : s.W, room = side < 2 ? c.xb - c.xa : s.HQ;
                if (n.dout[side ^ 1] != c.din[side] || n.out_off[side ^ 1] != c.in_off[side] || n.out_cap[side ^ 1] != c.in_cap[side])
                    return fault("mailbox of another block", g, fields, es);
                if (c.in_cap[side] < c.din[side] * len || c.dout[side] > room || c.sx[side] != n.sx[side ^ 1])
                    return fault("mailbox too small", g, fields, es);
                for (size_t q = 0; q < (size_t)c.in_cap[side] * 2 * fields; ++q) {
                    const size_t at = c.in_off[side] + q;
                    if (at >= p.xch_quads || used[at]) return fault("mailboxes overlap", g, fields, es);
                    used[at] = 1;
                }
                items += (c.din[side] + (c.sx[side] ? (side < 2 ? 4 : 1) : 0)) * len;
            }
            if (items > kResItems * kResThreads) return fault("too many halo quads", g, fields, es);
        }
    return 0;
}

int main()
{
    const int nxs[] = {1, 7, 33, 96, 250, 401, 777, 1201, 2000, 3400}, nzs[] = {4, 9, 64, 131, 200, 403, 700};
    const int ths[][4] = {{12, 12, 12, 12}, {16, 16, 16, 16}, {17, 60, 13, 45}, {50, 50, 50, 50}, {12, 64, 120, 30}, {300, 12, 12, 120}};
    int grids = 0, found = 0;
    for (int nx : nxs)
        for (int nz : nzs)
            for (auto &t : ths)
                for (int fields = 1; fields <= 2; ++fields)
                    for (int es = 4; es <= 8; es += 4)
                        for (int sms : {152, 148, 20}) {
                            ++grids;
                            if (check(nx, nz, t[0], t[1], t[2], t[3], fields, es, sms, found)) return 1;
                        }
    if (found < grids / 3) { printf("only %d of %d grids have a partition\n", found, grids); return 1; }
    printf("ok %d\n", found);
    return 0;
}
