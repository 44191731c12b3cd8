// rtm_gate.h -- which cooperative launches of one device may run at the same time: host code only.
//
// A resident launch holds one SM a block until its last step, so launches that may run at the same time
// must fit the SMs together: of two that do not, each could wait for SMs that the other holds.  Launches of
// one stream, a chain, follow one another.  A launch waits for launches of other chains, the oldest first,
// until its blocks and the most that each chain may still run beside it fit the SMs.  Any set of launches
// that run at the same time then fits: they are of different chains, and all others were there before the
// latest of them, which counted them.
#pragma once

#include <algorithm>
#include <cstddef>
#include <deque>
#include <utility>
#include <vector>

namespace rtm {

template <typename Event>
struct ResBook {
    struct Run {                      // launches of one size in a row: none can be beside another, so only
        Event end;                    // the end of the last of them makes a difference
        int blocks;
        long long turn;
    };
    struct Chain {
        unsigned long long stream;    // (an id that no later stream gets again)
        bool shares;                  // could do with half the SMs or fewer
        std::deque<Run> runs;         // not known to have ended, in their order; never empty
    };
    std::vector<Chain> open;
    long long turns = 0;

    // Launches that one of `blocks` blocks on `stream` waits for: (chain, run), the last of a chain that it
    // needs to wait for.
    std::vector<std::pair<size_t, size_t>> before(unsigned long long stream, int blocks, int sms) const
    {
        std::vector<size_t> next(open.size(), 0);      // first run of each chain that is not waited for
        auto beside = [&](size_t c) {
            int most = 0;
            for (size_t k = next[c]; k < open[c].runs.size(); ++k) most = std::max(most, open[c].runs[k].blocks);
            return most;
        };
        int sum = blocks;
        for (size_t c = 0; c < open.size(); ++c) {
            if (open[c].stream != stream) sum += beside(c);
        }
        while (sum > sms) {
            size_t c = open.size();
            for (size_t k = 0; k < open.size(); ++k)
                if (open[k].stream != stream && next[k] < open[k].runs.size() && (c == open.size() || open[k].runs[next[k]].turn < open[c].runs[next[c]].turn)) c = k;
            if (c == open.size()) break;               // (more blocks than SMs: refused by the launch)
            sum -= beside(c);
            ++next[c];
            sum += beside(c);
        }
        std::vector<std::pair<size_t, size_t>> w;
        for (size_t c = 0; c < open.size(); ++c)
            if (next[c] > 0) w.emplace_back(c, next[c] - 1);
        return w;
    }
    // A launch is on its way: the event to record at its end, fresh() unless it extends a run.
    template <typename F>
    Event launched(unsigned long long stream, int blocks, bool shares, F fresh)
    {
        Chain *chain = nullptr;
        for (Chain &c : open)
            if (c.stream == stream) chain = &c;
        if (!chain) {
            open.push_back({stream, shares, {}});
            chain = &open.back();
        }
        chain->shares = shares;
        if (chain->runs.empty() || chain->runs.back().blocks != blocks) chain->runs.push_back({fresh(), blocks, 0});
        chain->runs.back().turn = turns++;
        return chain->runs.back().end;
    }
    // Takes out what has ended: over(event) of a launch says so.  Ends of a chain come in its order.
    template <typename F>
    void prune(F over)
    {
        for (size_t c = 0; c < open.size();) {
            auto &runs = open[c].runs;
            while (!runs.empty() && over(runs.front().end)) runs.pop_front();
            if (runs.empty()) open.erase(open.begin() + (std::ptrdiff_t)c);
            else ++c;
        }
    }
    // Chains other than `stream`'s that could run beside it on a share of the chip.
    int sharers(unsigned long long stream) const
    {
        int n = 0;
        for (const Chain &c : open) n += c.shares && c.stream != stream;
        return n;
    }
};

}  // namespace rtm
