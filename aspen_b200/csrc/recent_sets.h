// What was made for a set of objects (their serial numbers, in order), for the N sets used last.
#pragma once
#include <algorithm>
#include <vector>

template <typename T, unsigned N>
class RecentSets {
    struct Set {
        std::vector<unsigned long long> of;
        T made;
    };
    std::vector<Set> sets;       // used last first

public:
    typedef std::vector<unsigned long long> Key;
    T *find(const Key &of) {
        for (size_t i = 0; i < sets.size(); i++)
            if (sets[i].of == of) { std::rotate(sets.begin(), sets.begin() + i, sets.begin() + i + 1); return &sets[0].made; }
        return nullptr;
    }
    // With N sets kept the one not used for longest goes: true, and what was made for it is the caller's to use again.
    bool make_room(T &made) {
        if (sets.size() < N) return false;
        made = sets.back().made;
        sets.pop_back();
        return true;
    }
    void put(const Key &of, const T &made) { sets.insert(sets.begin(), Set{of, made}); }
    // `release(T &)` for what was made for the sets with this object; all of them if it is 0.
    template <typename F>
    void drop(unsigned long long object, F release) {
        for (size_t i = sets.size(); i-- > 0;)
            if (object == 0 || std::count(sets[i].of.begin(), sets[i].of.end(), object)) { release(sets[i].made); sets.erase(sets.begin() + i); }
    }
};
