// Checks psdm::KeyedSlots on the CPU (see tests/test_region_plan_slots.py):
// groups of keys take slots as a batch's shots take their plans, each first
// use filling the slot, and read them only once the whole group has taken
// its own.  Prints the slots that no longer hold their group's key.
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>

#include "rtm_internal.h"

using namespace psdm;

int main(int argc, char** argv) {
    const int keys = atoi(argv[1]), groups = atoi(argv[2]), fixed = argc > 3 ? atoi(argv[3]) : 0;
    constexpr int N = 2 * kMaxSlots;
    KeyedSlots<int, N> s;
    int content[N];
    for (int& c : content) c = -1;
    std::mt19937 rng(11);
    long lost = 0, made = 0;
    auto group = [&](const std::vector<int>& want) {
        std::vector<int> at;
        for (int k : want) {
            bool held = false;
            const int i = s.take(k, &held);
            if (held)
                lost += content[i] != k;
            else
                content[i] = k, ++made;
            at.push_back(i);
        }
        for (size_t j = 0; j < want.size(); ++j) lost += content[at[j]] != want[j];
    };
    if (fixed) {  // every slot taken once, then a group of the oldest key and new ones
        for (int k = 0; k < N; ++k) group({k});
        std::vector<int> g = {0};
        for (int k = 1; k < kMaxSlots; ++k) g.push_back(N + k);
        group(g);
    }
    for (int i = 0; i < groups; ++i) {
        std::vector<int> g(1 + rng() % kMaxSlots);
        for (int& k : g) k = (int)(rng() % keys);
        group(g);
    }
    printf("%ld %ld\n", lost, made);
    return 0;
}
