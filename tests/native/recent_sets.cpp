// Sets that are used in turn are kept, the one not used for longest makes room, and what an object that goes was part of is given back.
#include "../../aspen_b200/csrc/recent_sets.h"

int main() {
    RecentSets<int, 3> sets;
    typedef RecentSets<int, 3>::Key Key;
    std::vector<int> released;
    auto release = [&](int &v) { released.push_back(v); };
    const Key a{1, 2}, b{2, 1}, c{1, 2, 3}, d{4};
    if (sets.find(a)) return 1;
    sets.put(a, 10, release);
    sets.put(b, 20, release);
    for (int i = 0; i < 5; i++)
        if (!sets.find(a) || *sets.find(a) != 10 || !sets.find(b) || *sets.find(b) != 20) return 2;
    sets.put(c, 30, release);
    if (!released.empty() || !sets.find(a)) return 3;
    sets.put(d, 40, release);
    if (released != std::vector<int>{20} || sets.find(b) || !sets.find(c) || !sets.find(a) || !sets.find(d)) return 4;
    released.clear();
    sets.drop(2, release);
    if (released.size() != 2 || sets.find(a) || sets.find(c) || !sets.find(d)) return 5;
    sets.drop(0, release);
    return released.back() == 40 && !sets.find(d) ? 0 : 6;
}
