// The table of cluster capacities (csrc/cuda/cluster_table.h) with a driver made up here: two devices of different layouts, a query that fails
// once, threads that ask at the same time.
#include <cstdio>
#include <thread>
#include <vector>

#include "cluster_table.h"

static int fails = 0;
#define EXPECT(c)                                                     \
    do {                                                              \
        if (!(c)) { std::printf("line %d: %s\n", __LINE__, #c); ++fails; } \
    } while (0)

int main() {
    ovb::ClusterTable t;
    int asked = 0;
    auto answer = [&](int n) { return [&asked, n] { ++asked; return n; }; };
    EXPECT(t.get(-1, 4, answer(9)) == 35 && asked == 0);            // no device: nothing is kept for the first one
    EXPECT(t.get(0, 4, answer(33)) == 33 && asked == 1);
    EXPECT(t.get(1, 4, answer(30)) == 30 && asked == 2);            // another device is asked, whoever came first
    EXPECT(t.get(0, 4, answer(7)) == 33 && t.get(1, 4, answer(7)) == 30 && asked == 2);
    EXPECT(t.get(2, 8, answer(0)) == 16 && asked == 3);             // no answer: a figure to go on with, which is not kept
    EXPECT(t.get(2, 8, answer(14)) == 14 && asked == 4 && t.get(2, 8, answer(0)) == 14 && asked == 4);
    EXPECT(t.get(3, 1, answer(5)) == 148 && asked == 4);

    ovb::ClusterTable shared;
    std::vector<std::thread> threads;
    std::vector<int> got(16);
    for (int i = 0; i < 16; ++i) threads.emplace_back([&, i] { got[i] = shared.get(i % 2, 2, [i] { return 60 + i % 2; }); });
    for (auto& th : threads) th.join();
    for (int i = 0; i < 16; ++i) EXPECT(got[i] == 60 + i % 2);
    if (fails == 0) std::printf("CLUSTER_TABLE_OK\n");
    return fails != 0;
}
