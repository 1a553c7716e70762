// Checks psdm::CoopLedger on the CPU (see tests/test_coop_order.py): launches
// of random sizes on random streams, each starting once its stream's last one
// and those that the ledger names have completed, in any order that this
// allows, as many at once as possible.  Prints the largest number of blocks
// that ran side by side, the launches that never started, the largest
// number of launches that ran side by side, and the ids in use.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <map>
#include <random>
#include <vector>

#include "rtm_internal.h"

using namespace psdm;

int main(int argc, char** argv) {
    const int cap = atoi(argv[1]), streams = atoi(argv[2]), most = atoi(argv[3]), launches = atoi(argv[4]);
    const int seed = atoi(argv[5]), wide = atoi(argv[6]);  // wide: every eighth launch takes the whole device
    std::mt19937 rng(seed);
    struct Launch {
        int blocks, state;  // 0 queued, 1 running, 2 done
        std::vector<int> after;
    };
    std::vector<Launch> all;
    std::vector<int> last(streams, -1), place(streams);
    std::map<int, int> newest;  // id -> its last launch
    CoopLedger l;
    int worst = 0, side = 0;
    auto running = [&] {
        int b = 0, n = 0;
        for (const Launch& x : all)
            if (x.state == 1) b += x.blocks, ++n;
        worst = std::max(worst, b);
        side = std::max(side, n);
    };
    auto start = [&] {
        for (Launch& x : all) {
            if (x.state != 0) continue;
            bool ready = true;
            for (int a : x.after) ready = ready && all[a].state == 2;
            if (ready) x.state = 1;
        }
        running();
    };
    auto finish = [&](int k) {  // up to k of the running launches, picked at random
        std::vector<int> r;
        for (size_t i = 0; i < all.size(); ++i)
            if (all[i].state == 1) r.push_back((int)i);
        std::shuffle(r.begin(), r.end(), rng);
        for (int i = 0; i < k && i < (int)r.size(); ++i) all[r[i]].state = 2;
    };
    for (int i = 0; i < launches; ++i) {
        const int st = (int)(rng() % streams), blocks = wide && rng() % 8 == 0 ? cap : 1 + (int)(rng() % most);
        if (rng() % 2)  // completions are seen late, or not at all
            l.prune([&](int id) { return all[newest[id]].state == 2; });
        Launch x{blocks, 0, {}};
        const auto follow = l.before(&place[st], blocks, cap);
        for (const auto& f : follow) x.after.push_back(newest[f.id]);
        if (last[st] >= 0) x.after.push_back(last[st]);
        const int id = l.new_id();
        l.queued(follow, id, &place[st], blocks);
        newest[id] = i;
        last[st] = i;
        all.push_back(x);
        start();
        if (rng() % 3 == 0) {
            finish(1 + (int)(rng() % 3));
            start();
        }
    }
    for (int i = 0; i < 2 * launches; ++i) {
        finish(1);
        start();
    }
    long never = 0;
    for (const Launch& x : all) never += x.state == 0;
    printf("%d %ld %d %d\n", worst, never, side, l.ids);
    return 0;
}
