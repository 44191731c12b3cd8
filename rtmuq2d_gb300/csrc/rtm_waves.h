// rtm_waves.h -- which of a server's resident members run at a server step, beside one another and how
// far: host code only.
//
// Large members take the chip one after the other; small ones share a launch (a wave), each with its part
// of the SMs.  Every member is owed steps_per_launch steps a server step; of the waves an eighth runs,
// each for the steps its members are owed, so that with eight waves or more a member's fields are brought
// on and off the chip once in eight server steps, for the same progress.
#pragma once

#include <algorithm>
#include <tuple>
#include <vector>

#include "rtm_gpu.h"
#include "rtm_partition.h"

namespace rtm {

// A member that shares a launch takes about one SM per kResCells cells, in whole shares of the chip so
// that a few partitions serve every mix (and more where SMs are spare): the exchange and the strips of
// a step cost nearly the same whatever a block holds, so the fullest blocks that fit do the most cells a
// second.  24 mixed members of 400 x 200 to 3400 x 700: 8000 cells an SM 166 ms, 12000 154, 16000 147,
// 20000 146, and no less with 24000 or 48000 (what does not fit takes a larger share).
constexpr double kResCells = 20000.0;
constexpr int kResMostSteps = 512;        // steps of one launch at most
// Quads of a block's mailboxes at most: two parities of two fields, each 8 columns or 2 rows of quads
// across every side, 16 HQ + 4 W of the 24 HQ + 6 W that res_fits holds to kResItems kResThreads.
constexpr size_t kResMostXchQuads = (size_t)kResItems * kResThreads * 2 / 3 * 4 + 4;

// What a member is owed once another server step begins (a debt of more than a launch's steps waits for
// the next one; the bound keeps the sum from running over).
inline int wave_owe(int due, int steps_per_launch) { return std::min(due + steps_per_launch, 1 << 20); }

// A resident member as a server step finds it.
struct WaveMember {
    int m;                            // slot
    const Geom *g;
    int back;                         // pass: 0 forward, 1 backward
    int step;                         // steps of the pass done
    int due;                          // steps owed, this server step's included
    long long ran;                    // server step of its last launch (of its admission before the first)
    int precision, storage;
    size_t slot_elems;
};

// Device room of a wave: mailboxes (quads) and staging of 16-bit members (elements).
struct WaveRoom {
    size_t xch_quads, stage_elems;
};

// Its part in a wave.
struct WaveItem {
    int m, share;                     // slot; it takes sms / share SMs
    int t0, t1, back;
    int lo, hi;                       // 16-bit storage: slots its steps write or read
    int due;
    long long ran;
};

// Slots of 16-bit storage that steps [it.t0, it.t1) of a pass write or read.
inline void wave_slots(const WaveMember &w, WaveItem &it)
{
    it.lo = 0;
    it.hi = -1;
    if (w.precision == RTM_PREC_FP32) return;
    const int nt = w.g->nt, sl = w.g->slices;
    if (w.storage == RTM_STORE_RING) {
        it.lo = it.back ? nt - it.t1 + 1 : it.t0 + 1;
        it.hi = it.back ? nt - std::max(it.t0 - 1, 2) : std::min(it.t1, nt - 1);
    } else {
        it.lo = (it.back ? nt - it.t1 + sl - 1 : it.t0 + sl - 1) / sl;
        it.hi = it.back ? (nt - 1 - it.t0) / sl : (it.t1 - 1) / sl;
    }
}

// Elements of the staging area that its steps take, and that one step takes at most (a backward step of a
// ring hands on the slot before its own).
inline size_t wave_stage(const WaveMember &w, const WaveItem &it) { return it.hi < it.lo ? 0 : (size_t)(it.hi - it.lo + 1) * w.slot_elems; }
inline size_t wave_least_stage(int precision, int storage, size_t slot_elems)
{
    return precision == RTM_PREC_FP32 ? 0 : (storage == RTM_STORE_RING ? 2 : 1) * slot_elems;
}

// The share of the chip that a member asks for in a wave: its grid's, or the smallest larger one that
// fits(share) holds for; the whole chip (1) if none does.
template <typename F>
int wave_share(const Geom &g, int sms, F fits)
{
    const int want = std::max(1, (int)((double)g.dimx * g.dimz / kResCells + 0.999));
    int share = std::max(1, std::min(sms / want, 16));
    while (share > 1 && !fits(share)) --share;
    return share;
}

// The waves that run at this server step, in order.  part(m, back, sms): the blocks of a pass of member m
// on that many SMs, NULL when they do not fit.  Every member's blocks fit at its share (wave_share), and the
// room of a wave holds their mailboxes and one step's staging; members join a wave while it holds theirs, and
// a wave's 16-bit members take as many steps as it holds slots for (a member of 3400 x 700 with snapshots at
// every step takes 11 MB a step).
// An eighth: 12 members of 3400 x 700 spent 3.5 us of 10 a step on bringing fields on and off the chip at
// 16 steps a launch.  A quarter: 64 members 213.6 Gcell-updates/s on the GPU against 218.3, 12 members
// 202.6 ms against 200.9; a 32nd 196.5 but 24 mixed ones 146.4 -> 147.8.
template <typename F>
std::vector<std::vector<WaveItem>> res_waves(const std::vector<WaveMember> &members, int sms, int steps_per_launch,
                                             const WaveRoom &room, F part)
{
    std::vector<WaveItem> items;
    std::vector<const WaveMember *> of;           // by slot
    auto fits = [&](const WaveItem &it, int share) {
        const ResPart *p = part(it.m, it.back, sms / share);
        return p && p->xch_quads <= room.xch_quads;
    };
    for (const WaveMember &w : members) {
        WaveItem it;
        it.m = w.m;
        it.back = w.back;
        it.t0 = w.step;
        it.due = w.due;
        it.ran = w.ran;
        it.t1 = std::min(w.g->nt, it.t0 + std::min(w.due, kResMostSteps));
        wave_slots(w, it);
        it.share = wave_share(*w.g, sms, [&](int share) { return fits(it, share); });
        if (w.m >= (int)of.size()) of.resize(w.m + 1);
        of[w.m] = &w;
        items.push_back(it);
    }
    std::stable_sort(items.begin(), items.end(), [](const WaveItem &a, const WaveItem &b) { return a.share < b.share; });

    // the largest member left and those that fit beside it
    std::vector<std::vector<WaveItem>> waves;
    std::vector<char> taken(items.size(), 0);
    for (size_t first = 0; first < items.size(); ++first) {
        if (taken[first]) continue;
        std::vector<WaveItem> wave;
        int used = 0;
        size_t xch = 0, stage = 0;
        for (size_t i = first; i < items.size(); ++i) {
            const int need = sms / items[i].share;
            if (taken[i] || used + need > sms) continue;
            const WaveMember &w = *of[items[i].m];
            const size_t quads = part(w.m, w.back, need)->xch_quads, least = wave_least_stage(w.precision, w.storage, w.slot_elems);
            if (!wave.empty() && (xch + quads > room.xch_quads || stage + least > room.stage_elems)) continue;
            taken[i] = 1;
            used += need;
            xch += quads;
            stage += least;
            wave.push_back(items[i]);
        }
        // spare SMs to the member with the most cells an SM, which the others wait for, as long as there
        // are enough (four members of 400 x 200, 1000 steps a pass: 20 ms, 33 where the first took all it could)
        std::vector<int> share(wave.size());
        for (size_t i = 0; i < wave.size(); ++i) share[i] = wave[i].share;
        for (;;) {
            size_t slow = 0;
            double most = -1.0;
            for (size_t i = 0; i < wave.size(); ++i) {
                const Geom &g = *of[wave[i].m]->g;
                const double per = (double)g.dimx * g.dimz / (sms / share[i]);
                if (per > most) { most = per; slow = i; }
            }
            if (share[slow] == 1) break;
            const int more = sms / (share[slow] - 1) - sms / share[slow];
            if (used + more > sms) break;
            used += more;
            --share[slow];
        }
        for (size_t i = 0; i < wave.size(); ++i) {
            const ResPart *p = part(wave[i].m, wave[i].back, sms / share[i]);
            if (!p) continue;
            const size_t was = part(wave[i].m, wave[i].back, sms / wave[i].share)->xch_quads;
            if (xch - was + p->xch_quads > room.xch_quads) continue;
            xch = xch - was + p->xch_quads;
            wave[i].share = share[i];
        }
        // the most steps a launch for which the staging area holds its slots
        auto staged = [&](int most) {
            size_t n = 0;
            for (WaveItem it : wave) {
                it.t1 = std::min(it.t1, it.t0 + most);
                wave_slots(*of[it.m], it);
                n += wave_stage(*of[it.m], it);
            }
            return n;
        };
        int lo = 1, hi = kResMostSteps;
        while (lo < hi) {
            const int mid = (lo + hi + 1) / 2;
            if (staged(mid) <= room.stage_elems) lo = mid;
            else hi = mid - 1;
        }
        for (WaveItem &it : wave) {
            if (of[it.m]->precision == RTM_PREC_FP32) continue;
            it.t1 = std::min(it.t1, it.t0 + lo);
            wave_slots(*of[it.m], it);
        }
        waves.push_back(std::move(wave));
    }
    // the waves that have waited longest come first: by debt alone those that a launch cannot pay in full --
    // it ends at kResMostSteps, or where the staging area is full -- would win every time
    struct Turn { long long ran; int due; size_t k; };
    std::vector<Turn> turn;
    for (const auto &wave : waves) {
        Turn t{wave[0].ran, 0, turn.size()};
        for (const WaveItem &it : wave) { t.ran = std::min(t.ran, it.ran); t.due = std::max(t.due, it.due); }
        turn.push_back(t);
    }
    std::sort(turn.begin(), turn.end(), [](const Turn &a, const Turn &b) { return std::tie(a.ran, b.due, a.k) < std::tie(b.ran, a.due, b.k); });
    // an eighth, and as many as it takes to pay all that is owed in launches of kResMostSteps
    const size_t all = waves.size(), paid = (all * (size_t)steps_per_launch + kResMostSteps - 1) / kResMostSteps;
    turn.resize(std::min(all, std::max((all + 7) / 8, paid)));
    std::vector<std::vector<WaveItem>> out;
    for (const Turn &t : turn) out.push_back(std::move(waves[t.k]));
    return out;
}

}  // namespace rtm
