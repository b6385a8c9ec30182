// Host build of the parcel protocol (circlepacking_b200/csrc/cp_parcel.cuh) for the CPU tests.
#include "cp_parcel.cuh"

#include <atomic>
#include <thread>
#include <vector>

using namespace cpb;

extern "C" {
int p_claim(ParcelFlag* flag, unsigned long long epoch, unsigned d) { return parcel_claim(flag, epoch, d); }
// Threads claim, mark and leave `slots` slots `each` times; returns how often a slot had two owners.
long p_stress(int threads, unsigned slots, int each) {
    std::vector<ParcelFlag> flag(slots, 0);
    std::vector<std::atomic<int>> owners(slots);
    for (auto& o : owners) o = 0;
    std::atomic<unsigned> next{0};
    std::atomic<long> clashes{0};
    std::vector<std::thread> ts;
    for (int t = 0; t < threads; ++t)
        ts.emplace_back([&] {
            for (int k = 0; k < each; ++k) {
                const unsigned d = next++, s = d % slots;
                if (!parcel_claim(&flag[s], 7, d)) continue;
                if (owners[s].fetch_add(1) != 0) ++clashes;
                std::this_thread::yield();
                owners[s].fetch_sub(1);
                __atomic_fetch_or(&flag[s], (ParcelFlag)kParcelTaken, __ATOMIC_SEQ_CST);
            }
        });
    for (auto& t : ts) t.join();
    return clashes;
}
}
