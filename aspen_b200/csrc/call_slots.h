// Numbers for calls that run at the same time: a call has one to itself from take() to give().  No locks, no memory of its own.
#pragma once
#include <atomic>

template <unsigned N>
class CallSlots {
    static_assert(N % 64 == 0, "whole words");
    std::atomic<unsigned long long> taken[N / 64] = {};

public:
    // A free number below N, or -1.
    int take() {
        for (unsigned w = 0; w < N / 64; w++) {
            unsigned long long old = taken[w].load(std::memory_order_relaxed);
            while (~old) {
                const int bit = __builtin_ctzll(~old);
                if (taken[w].compare_exchange_weak(old, old | 1ull << bit, std::memory_order_acquire, std::memory_order_relaxed)) return (int)(w * 64) + bit;
            }
        }
        return -1;
    }
    void give(int slot) { taken[slot / 64].fetch_and(~(1ull << (slot % 64)), std::memory_order_release); }
};
