// Sets that are used in turn are kept, what was made for the one not used for longest is handed over for the next, and what an object that
// goes was part of is given back.
#include "../../aspen_b200/csrc/recent_sets.h"

int main() {
    RecentSets<int, 3> sets;
    typedef RecentSets<int, 3>::Key Key;
    std::vector<int> released;
    auto release = [&](int &v) { released.push_back(v); };
    const Key a{1, 2}, b{2, 1}, c{1, 2, 3}, d{4};
    if (sets.find(a)) return 1;
    int old = 0;
    if (sets.make_room(old)) return 7;
    sets.put(a, 10);
    sets.put(b, 20);
    for (int i = 0; i < 5; i++)
        if (!sets.find(a) || *sets.find(a) != 10 || !sets.find(b) || *sets.find(b) != 20) return 2;
    sets.put(c, 30);
    if (!sets.find(a)) return 3;
    if (!sets.make_room(old)) return 8;
    sets.put(d, 40);
    if (old != 20 || sets.find(b) || !sets.find(c) || !sets.find(a) || !sets.find(d)) return 4;
    sets.drop(2, release);
    if (released.size() != 2 || sets.find(a) || sets.find(c) || !sets.find(d)) return 5;
    sets.drop(0, release);
    return released.back() == 40 && !sets.find(d) ? 0 : 6;
}
