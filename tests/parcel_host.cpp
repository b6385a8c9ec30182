// Host build of the parcel protocol (circlepacking_b200/csrc/cp_parcel.cuh) for the CPU tests.
#include "cp_parcel.cuh"

#include <pthread.h>

#include <atomic>
#include <chrono>
#include <thread>
#include <vector>

using namespace cpb;

namespace {
constexpr int kLanes = 4;
// A warp of host threads.  Lanes other than the first come late to each copy, as lanes of
// a warp may.
struct HostWarp {
    pthread_barrier_t* bar;
    int lane;
    bool first() const { return lane == 0; }
    void acquire() const { pthread_barrier_wait(bar); }
    void release() const { pthread_barrier_wait(bar); }
    void late() const {
        if (lane) std::this_thread::sleep_for(std::chrono::microseconds(200 * lane));
    }
};
template <class F>
void warp(pthread_barrier_t* bar, F f) {
    std::vector<std::thread> ts;
    for (int l = 0; l < kLanes; ++l) ts.emplace_back([=] { f(HostWarp{bar, l}); });
    for (auto& t : ts) t.join();
}
}  // namespace

extern "C" {
int p_claim(ParcelFlag* flag, unsigned long long epoch, unsigned d, unsigned slots) {
    return parcel_claim(flag, epoch, d, slots);
}
unsigned p_ready(unsigned long long f, unsigned long long epoch, unsigned d) { return parcel_ready(f, epoch, d); }
unsigned p_left(unsigned long long f, unsigned long long epoch) { return parcel_left(f, epoch); }
// Refinements of `launches` launches each on one handle; returns how many launches had
// an epoch (24 bits) at or below one that an uncleared flag may carry.
long p_epochs(long refinements, int launches) {
    long again = 0;
    unsigned long long last = 0, highest = 0;  // highest: of the flags since they were cleared
    for (long k = 0; k < refinements; ++k) {
        bool clear;
        last = parcel_epoch(last, clear);
        if (clear) highest = 0;
        if (((last - 1) & 0xFFFFFF) < highest) ++again;  // (a first launch looks back by one)
        for (int l = 0; l < launches; ++l, ++last) {
            if ((last & 0xFFFFFF) <= highest) ++again;
            highest = last & 0xFFFFFF;
        }
    }
    return again;
}
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
                if (!parcel_claim(&flag[s], 7, d, slots)) continue;
                if (owners[s].fetch_add(1) != 0) ++clashes;
                std::this_thread::yield();
                owners[s].fetch_sub(1);
                flag_set(&flag[s], parcel_tag(7, d) << 8 | kParcelTaken);
            }
        });
    for (auto& t : ts) t.join();
    return clashes;
}
// One giver and one taker hand `parcels` parcels over through one slot; returns how many
// parents arrived wrong.
long p_hand_over(int parcels) {
    ParcelFlag flag = 0;
    std::atomic<int> slot[kLanes] = {};
    std::atomic<long> wrong{0};
    pthread_barrier_t give, take;
    pthread_barrier_init(&give, nullptr, kLanes);
    pthread_barrier_init(&take, nullptr, kLanes);
    const auto see = [&](int d) { return flag_read(&flag) == (parcel_tag(1, d) << 8 | kLanes); };
    std::thread giver([&] {
        warp(&give, [&](HostWarp w) {
            for (int d = 0; d < parcels; ++d) {
                while (w.first() && !parcel_claim(&flag, 1, d, 1)) std::this_thread::yield();
                parcel_give(w, &flag, 1, d, kLanes, d > 0, [&] {
                    w.late();
                    slot[w.lane] = kLanes * d + w.lane;
                });
            }
        });
    });
    warp(&take, [&](HostWarp w) {
        for (int d = 0; d < parcels; ++d) {
            while (w.first() && !see(d)) std::this_thread::yield();
            parcel_take(w, &flag, [&] {
                w.late();
                if (slot[w.lane] != kLanes * d + w.lane) ++wrong;
            });
        }
    });
    giver.join();
    pthread_barrier_destroy(&give);
    pthread_barrier_destroy(&take);
    return wrong;
}
}
