// Host check of the order of cooperative launches (csrc/rtm_gate.h): random launches on a few streams, some
// of which end, and every set of launches that the order lets run at the same time fits the SMs.  Prints
// "ok <launches>" or the first fault.
#include <cstdio>
#include <random>

#include "rtm_gate.h"

using namespace rtm;

int main()
{
    const int sms = 152, streams = 6;
    std::mt19937 rng(7);
    long long launches = 0, together = 0;
    for (int trial = 0; trial < 400; ++trial) {
        struct Run { int blocks; unsigned after; bool ended; };   // after: launches it is ordered after (bits)
        std::vector<Run> runs;
        ResBook<int> book;                                        // an event is the launch's number
        for (int n = 0; n < 14; ++n) {
            // some launches have ended, those they were ordered after with them
            for (size_t j = 0; j < runs.size(); ++j)
                if (rng() % 8 == 0) {
                    runs[j].ended = true;
                    for (size_t k = 0; k < j; ++k)
                        if (runs[j].after >> k & 1) runs[k].ended = true;
                }
            book.prune([&](int e) { return runs[e].ended; });
            const int sizes[] = {19, 38, 50, 60, 76, 150, 152, 1 + (int)(rng() % sms)}, blocks = sizes[rng() % 8];
            const unsigned long long s = 100 + rng() % streams;
            Run r{blocks, 0, false};
            for (const auto &w : book.before(s, blocks, sms)) {
                const int e = book.open[w.first].runs[w.second].end;
                r.after |= 1u << e | runs[e].after;
            }
            // of its own stream it follows all; a run's event is that of its last launch so far
            for (const auto &c : book.open)
                if (c.stream == s) r.after |= 1u << c.runs.back().end | runs[c.runs.back().end].after;
            runs.push_back(r);
            book.launched(s, blocks, true, [] { return 0; });
            for (auto &c : book.open)
                if (c.stream == s) c.runs.back().end = n;
            ++launches;
            // sets of launches without an order between any two, none ended
            for (unsigned set = 1; set < 1u << runs.size(); ++set) {
                if (!(set >> n & 1)) continue;
                int sum = 0, count = 0;
                bool free_of_order = true;
                for (size_t j = 0; j < runs.size() && free_of_order; ++j)
                    if (set >> j & 1) {
                        if (runs[j].ended || (runs[j].after & set)) free_of_order = false;
                        sum += runs[j].blocks;
                        ++count;
                    }
                if (!free_of_order) continue;
                if (count > 1) ++together;
                if (sum > sms) { printf("launches %x hold %d of %d SMs together\n", set, sum, sms); return 1; }
            }
        }
    }
    if (together < launches / 4) { printf("only %lld pairs may run at the same time\n", together); return 1; }
    ResBook<int> book;
    int next = 0;
    for (int blocks : {152, 152, 60}) book.launched(7, blocks, true, [&] { return next++; });
    book.launched(8, 60, false, [&] { return next++; });
    // behind the launches that fill the chip, not behind the smaller one after them
    const auto w = book.before(9, 32, sms);
    if (next != 3 || book.open.size() != 2 || book.sharers(7) != 0 || book.sharers(8) != 1 || w.size() != 1 || w[0].first != 0 || w[0].second != 0) {
        printf("chains of two streams\n");
        return 1;
    }
    printf("ok %lld\n", launches);
    return 0;
}
