// Clusters of 1 .. 8 CTAs (one CTA per SM) that a device holds at a time, as its driver answers. Plain C++: also built into a test.
#pragma once
#include <mutex>

namespace ovb {

class ClusterTable {
public:
    // `ask()`: the driver's answer for the current device, 0 where it gives none. An answer is kept for its device alone; without one the figure of
    // a whole B200 serves, and the next call asks again. device < 0: there is none.
    template <class Ask>
    int get(int device, int size, Ask&& ask) {
        static constexpr int whole[9] = {0, 148, 74, 45, 35, 27, 22, 18, 16};
        if (device < 0 || size == 1) return whole[size];
        std::lock_guard<std::mutex> lk(mu_);
        int& n = known_[device & 63][size];
        if (n == 0) n = ask();
        return n > 0 ? n : whole[size];
    }

private:
    std::mutex mu_;
    int known_[64][9] = {};
};

}  // namespace ovb
