// Parcels: how a warp of the depth-first refinement (cp_refine.cuh) hands parents to a
// warp that has run out.  Parcel d lies in slot d % slots, whose flag says which
// parcel it holds and how far that has come:
//
//     epoch (24 bits) | d (32 bits) | state (8 bits)
//
// state 0: claimed, its giver is writing the parents; 1 to 32: that many parents, ready;
// kParcelTaken: read, the slot is free.  The epoch is the launch's; a flag of another
// launch leaves its slot free.  Epochs come back after 2^24 launches, so the flags are
// cleared ahead of that (parcel_epoch).
//
// Givers run ahead of takers (about four warps give per missing parcel), so two of them can
// want one slot at a time: parcels d and d + slots.  A slot's first parcel of the launch
// (d < slots) has it without asking.  A later one claims it by compare-and-swap before it
// writes, and only where this launch's flag says taken: its giver finds the slot untouched,
// claimed or ready otherwise, and keeps its parents.
//
// A warp reads and writes a slot with all of its lanes, but one lane works its flag.  So
// the lanes' copies stand between an acquire() and a release() of the warp: no lane
// touches the slot before the lane at the flag has seen it in the warp's hands, and the
// flag passes the slot on when every lane is done with it.
//
// Host code too, so that the protocol is tested without a GPU.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define CPP_HD __host__ __device__ __forceinline__
#else
#define CPP_HD inline
#endif

namespace cpb {

typedef unsigned long long ParcelFlag;

constexpr unsigned kParcels = 1u << 12;  // slots
constexpr unsigned kParcelTaken = 0xFF;

CPP_HD ParcelFlag parcel_tag(unsigned long long epoch, unsigned d) { return (epoch & 0xFFFFFFull) << 32 | d; }

CPP_HD ParcelFlag flag_read(const ParcelFlag* flag) { return *(const volatile ParcelFlag*)flag; }
CPP_HD bool flag_swap(ParcelFlag* flag, ParcelFlag from, ParcelFlag to) {
#ifdef __CUDA_ARCH__
    return atomicCAS(flag, from, to) == from;
#else
    return __atomic_compare_exchange_n(flag, &from, to, false, __ATOMIC_SEQ_CST, __ATOMIC_SEQ_CST);
#endif
}

// No parcel of this launch lies in the slot.
CPP_HD bool parcel_free(ParcelFlag f, unsigned long long epoch) {
    return f >> 40 != (epoch & 0xFFFFFFull) || (f & 0xFF) == kParcelTaken;
}
// Parents ready in the slot for the ticket of parcel d; 0: not yet.
CPP_HD unsigned parcel_ready(ParcelFlag f, unsigned long long epoch, unsigned d) {
    const unsigned n = (unsigned)(f & 0xFF);
    return f >> 8 == parcel_tag(epoch, d) && n != kParcelTaken ? n : 0u;
}
// Parents that the launch of this epoch left over in the slot.
CPP_HD unsigned parcel_left(ParcelFlag f, unsigned long long epoch) {
    return parcel_free(f, epoch) ? 0u : (unsigned)(f & 0xFF);
}
// The epoch of a refinement's first launch, `last` being the epoch after the handle's
// latest launch.  No flag carries it or the one before: the next one but one, or, when
// half of the epochs are used up, epoch 1 over cleared flags (clear).  The other half is
// left to the further launches of a refinement.
CPP_HD unsigned long long parcel_epoch(unsigned long long last, bool& clear) {
    clear = last + 2 >= 1ull << 23;
    return clear ? 1 : last + 2;
}
// The giver's: true when slot d % slots is the caller's to write.  (The first parcels of a
// launch spread its work over the device, one hand-over after the other, so they go without
// the look at the flag and the swap.)
CPP_HD bool parcel_claim(ParcelFlag* flag, unsigned long long epoch, unsigned d, unsigned slots) {
    if (d < slots) return true;
    const ParcelFlag f = flag_read(flag);
    return f >> 40 == (epoch & 0xFFFFFFull) && (f & 0xFF) == kParcelTaken &&
           flag_swap(flag, f, parcel_tag(epoch, d) << 8);
}

#ifdef __CUDACC__
// The warp that handles a slot; all of its lanes make each call.  One lane's fence orders
// the whole warp's accesses, through the warp's barrier; start proof, half of its seeds, on
// a B200: 26.4 ms with a fence of every lane, 25.9 ms so.
struct SlotWarp {
    __device__ __forceinline__ bool first() const { return (threadIdx.x & 31) == 0; }
    __device__ __forceinline__ void acquire() const {
        if (first()) __threadfence();
        __syncwarp();
    }
    __device__ __forceinline__ void release() const {
        __syncwarp();
        if (first()) __threadfence();
    }
};
#endif
CPP_HD void flag_set(ParcelFlag* flag, ParcelFlag to) {
#ifdef __CUDA_ARCH__
    atomicExch(flag, to);
#else
    __atomic_store_n(flag, to, __ATOMIC_SEQ_CST);
#endif
}
CPP_HD void flag_or(ParcelFlag* flag, ParcelFlag bits) {
#ifdef __CUDA_ARCH__
    atomicOr(flag, bits);
#else
    __atomic_fetch_or(flag, bits, __ATOMIC_SEQ_CST);
#endif
}

// Writes the n parents of parcel d into its slot, which the warp has claimed: write() is a
// lane's part.  again: the slot has held another parcel of this launch (d >= slots).
template <class Warp, class Write>
CPP_HD void parcel_give(const Warp& w, ParcelFlag* flag, unsigned long long epoch, unsigned d, unsigned n, bool again,
                        const Write& write) {
    if (again) w.acquire();
    write();
    w.release();
    if (w.first()) flag_set(flag, parcel_tag(epoch, d) << 8 | n);
}
// Reads the parents of a slot whose flag, as the warp's first lane saw it, holds a parcel:
// read() is a lane's part.  The slot is free afterwards.
template <class Warp, class Read>
CPP_HD void parcel_take(const Warp& w, ParcelFlag* flag, const Read& read) {
    w.acquire();
    read();
    w.release();
    if (w.first()) flag_or(flag, kParcelTaken);
}

}  // namespace cpb
