// Calls that run at the same time have numbers of their own; with all taken there is none, and what is given back is taken again.
#include "../../aspen_b200/csrc/call_slots.h"
#include <thread>
#include <vector>

static CallSlots<128> slots;
static std::atomic<int> holder[128];
static std::atomic<int> failures{0};

int main() {
    std::vector<std::thread> threads;
    for (int t = 1; t <= 16; t++)
        threads.emplace_back([t]() {
            int mine[12];                                     // 16 x 12 are more than there are
            for (int round = 0; round < 3000; round++) {
                for (int &s : mine) {
                    s = slots.take();
                    if (s < 0) continue;
                    if (s >= 128 || holder[s].exchange(t) != 0) failures++;
                }
                for (int s : mine)
                    if (s >= 0) { if (holder[s].exchange(0) != t) failures++; slots.give(s); }
            }
        });
    for (std::thread &t : threads) t.join();
    std::vector<bool> seen(128, false);
    for (int i = 0; i < 128; i++) {
        const int s = slots.take();
        if (s < 0 || seen[s]) return 2;
        seen[s] = true;
    }
    if (slots.take() != -1) return 3;
    slots.give(77);
    if (slots.take() != 77) return 4;
    return failures ? 1 : 0;
}
