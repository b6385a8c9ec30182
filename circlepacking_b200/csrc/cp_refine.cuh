// Warp-local refinement: the loop in which one warp evaluates boxes and refines
// the ones that are not proved, keeping as much of their subtrees as it can in
// shared memory.  Shared by the level kernel of the host-driven loop (cp_engine.cu;
// DEEP = false: the children that are evaluated once, at the depth limit, stay
// on chip, the others go to the next level) and by the depth-first kernel of the
// graph engine (cp_graph_kernels.cuh; DEEP = true: whole subtrees stay on chip).
//
// Why: with the filter a box costs about 700 warp instructions, less than writing
// its children to a level (65 B each, a division and two dependent table loads per
// child) and reading them back cost.  A refinement's last level holds most of its
// boxes.  B200, middle, 64^4 lattice and two uniform levels, graph engine: 188 -> 76 ms,
// the filter reading its boxes from shared memory included; half of the start proof 34 ->
// 26 ms; 31^4 start_end_3d lattice with the FP32 pre-pass 74 -> 50 ms.
//
// A warp holds, in shared memory:
//   * a stack of parents: boxes evaluated, not proved and above the depth limit,
//     whose children have not been made yet;
//   * a buffer of boxes ready for evaluation.
// A step takes the 32 youngest ready boxes; while there are fewer, the children of
// the top parents are made (2 to 16 parents fill a warp), clipped and appended, and
// when no parent is left, boxes of the input.  So steps have no idle lanes while
// there is work, whatever clipping drops.
//
// The stack is bounded.  Where a step evaluates nothing but the children just made
// ("strict"), its at most 32 parents are all deeper than the shallowest parent it
// came from, so the pushes on the stack have strictly increasing least depths from
// bottom to top: at most max_depth of them, 32 (max_depth + 1) parents in all.  Ready
// boxes left over from earlier parents break that order; a warp with `strict` spilled
// parents works strictly until it has fewer, so that the stack never holds more than
// those and the bound.  kParents of it fit on chip; more move to the
// warp's part of a spill list in global memory.  In the level kernel (DEEP = false)
// only input boxes become parents, and they enter when no parent is left, at most 32
// besides 31 ready ones: 63 parents.
#pragma once
#include "cp_level.cuh"
#include "cp_parcel.cuh"

namespace cpb {

constexpr int kParents = 64;  // parents per warp on chip
constexpr int kReady = 64;    // ready boxes: fewer than 32 before up to 32 are added

template <int D>
struct WarpBoxes {
    double plo[D][kParents], phi[D][kParents];
    double rlo[D][kReady], rhi[D][kReady];
    unsigned long long dig_sum[32], dig_xor[32];  // digest words per lane
    uint32_t pmeta[kParents];  // depth | axis << 8
    uint32_t rdepth[kReady];
};
// Box list with a meta word per box (depth | axis << 8).
struct MetaList {
    double* lo;
    double* hi;
    uint32_t* meta;
    size_t cap;
};

// Work sharing of a depth-first refinement.  Warps draw tickets: the first ones are
// pieces of the input, ticket `inputs` + d is the d-th parcel of up to 32 parents that
// some warp gives away (cp_parcel.cuh).  A warp whose ticket's parcel does not exist yet waits for it (a
// bounded wait); warps with enough parents give a parcel away per step while there
// are more tickets than parcels.  Parcels that nobody waited for to the end are the
// input of the next kernel launch ("round"); there are hardly ever any.
//
// Without sharing the trees below the seeds are too uneven: on the last slab of the
// start_end_3d proof (2.9e7 boxes, 26010 seeds) warps that stopped as soon as a
// quarter of them were idle, for a new round to spread the rest, needed 13 rounds and
// 4.2 ms, where parcels needed one round of 3.5 ms; the smallest slabs of the start
// and start_end_3d proofs took 0.10 to 0.2 ms instead of 0.2 to 0.4 (a level each).
struct DeepSched {
    unsigned long long count;  // seed boxes
    unsigned long long epoch;  // of this round; a parcel's flag carries it
    unsigned int inputs;       // tickets that are input
    unsigned int ticket;       // tickets drawn
    unsigned int parcels;      // parcels given away, or being written
    unsigned int filled, taken;
    unsigned int idle;         // warps waiting or gone
    unsigned int done;         // blocks finished
    unsigned int rounds;
    unsigned int left;         // parcels left over: another round is needed
    int status;                // 0 ok, 1 spill overflow
    unsigned long long given;  // over all rounds: parcels given, parents spilled
    unsigned long long spilled;
};
// A warp with fewer parents keeps them.  FP32: its steps take ten times as long, so
// that warps give from small stacks too and look after every step.
template <int PREC>
constexpr unsigned kMinGive = PREC == CP_FP32_PREFILTER ? 4 : 8;
constexpr int kWaitPolls = 1 << 17, kWaitNs = 200;  // polls of a wait (it ends after some 30 ms), pause between them
constexpr unsigned kStrict = 128;                   // RefineArgs::strict (512 was no faster)

struct RefineArgs {
    LevelArgs level;            // policy, limits, counters, input list
    unsigned long long* claim;  // DEEP = false: boxes of the chunk handed out
    unsigned per;               // input boxes per claim or ticket at most
    // DEEP
    DeepSched* sched;
    MetaList lists[2];          // parcels: round r gives to lists[r & 1], its input (r > 0) is the other
    unsigned long long* flags[2];
    MetaList spill;             // warp w: entries [w * seg, (w + 1) * seg)
    size_t seg;
    unsigned strict;            // spilled parents from which a warp works strictly
    unsigned slots;             // parcel slots in use, at most kParcels
    int polls;                  // of a wait for a parcel
};

// A warp's counts, in registers: per lane 10-bit fields for the five verdicts and the
// unresolved boxes, per warp a run of boxes of one depth (a step holds boxes of one
// or two depths).  Shared memory sees one atomic per field and 1023 steps.
struct WarpTally {
    unsigned long long fields = 0;
    unsigned steps = 0, fp32 = 0, run_depth = 0, run = 0;
};
__device__ __forceinline__ void tally_flush(WarpTally& t, LevelCounts& sm) {
    const bool first = (threadIdx.x & 31) == 0;
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        const unsigned n = __reduce_add_sync(0xffffffffu, (unsigned)(t.fields >> (10 * k)) & 1023u);
        if (first && n) atomicAdd(&sm.hist[k], (unsigned long long)n);  // k = 5: C_UNRESOLVED
    }
    t.fields = 0;
    t.steps = 0;
}
__device__ __forceinline__ void tally_run(WarpTally& t, LevelCounts& sm) {
    if (t.run && (threadIdx.x & 31) == 0)
        atomicAdd(&sm.depth[t.run_depth < kDepthBins ? t.run_depth : kDepthBins - 1], (unsigned long long)t.run);
    t.run = 0;
}
__device__ __forceinline__ void tally_step(WarpTally& t, LevelCounts& sm, int v, bool unresolved, unsigned depth) {
    if (v >= 0) t.fields += 1ull << (10 * v);
    if (unresolved) t.fields += 1ull << 50;
    if (++t.steps == 1023) tally_flush(t, sm);
    unsigned left = __ballot_sync(0xffffffffu, v >= 0);
    while (left) {
        const unsigned d0 = __shfl_sync(0xffffffffu, depth, __ffs(left) - 1);
        if (d0 != t.run_depth) {
            tally_run(t, sm);
            t.run_depth = d0;
        }
        const unsigned same = __ballot_sync(0xffffffffu, v >= 0 && depth == d0);
        t.run += __popc(same);
        left &= ~same;
    }
}

template <int D>
__device__ __forceinline__ void box_copy(const BoxRef<D>& box, double* lo, double* hi) {
#pragma unroll
    for (int d = 0; d < D; ++d) {
        lo[d] = box.lo[d * box.stride];
        hi[d] = box.hi[d * box.stride];
    }
}

__device__ __forceinline__ unsigned lanes_below() { return (1u << (threadIdx.x & 31)) - 1u; }

template <int FAM, int PREC, bool DEEP, class Smem>
__device__ __forceinline__ void refine_warp(const RefineArgs& r, Smem& sm, WarpBoxes<family_dims(FAM)>& wb,
                                            unsigned nwarps, unsigned warp_id, unsigned& handles) {
    constexpr int D = family_dims(FAM);
    const LevelArgs& a = r.level;
    const unsigned lane = threadIdx.x & 31, full = 0xffffffffu;
    const int flog = a.policy == SPLIT_UNIFORM ? D : 1;  // log2 of the children per parent
    const unsigned group = 32u >> flog;                  // parents that fill a warp
    unsigned round = 0, inputs = 0, ticket = warp_id, per;
    bool drawn = DEEP;  // DEEP: `ticket` has been drawn and not used up
    {
        // small inputs are spread over all warps
        const unsigned long long count = DEEP ? r.sched->count : a.count, share = (count + nwarps - 1) / nwarps;
        per = share < r.per ? (unsigned)(share ? share : 1) : r.per;
        if (DEEP) {
            round = r.sched->rounds;
            inputs = round ? r.sched->inputs : (unsigned)((count + per - 1) / per);
        }
    }
    unsigned long long cur = 0, end = 0;
    bool more = true;
    if (!DEEP) {  // the first pieces are the warps' by number
        cur = (unsigned long long)warp_id * per;
        end = cur + per < a.count ? cur + per : a.count;
        more = a.count > (unsigned long long)nwarps * per;
    }
    unsigned np = 0, nr = 0, nspill = 0, nclip = 0;
    WarpTally t;
    wb.dig_sum[lane] = wb.dig_xor[lane] = 0;
    for (;;) {
        const bool strict = DEEP && nspill >= r.strict;  // evaluate the next children made, and nothing else
        unsigned made = 0;
        while (nr < 32 && !(strict && made)) {
            double lo[4] = {0, 0, 0, 0}, hi[4] = {0, 0, 0, 0};
            int depth = 0;
            bool have = false, clipped = false;
            if (DEEP && np == 0 && nspill > 0) {  // the youngest spilled parents
                np = nspill < 32 ? nspill : 32;
                nspill -= np;
                if (lane < np) {
                    const size_t e = (size_t)warp_id * r.seg + nspill + lane;
#pragma unroll
                    for (int d = 0; d < D; ++d) {
                        wb.plo[d][lane] = r.spill.lo[d * r.spill.cap + e];
                        wb.phi[d][lane] = r.spill.hi[d * r.spill.cap + e];
                    }
                    wb.pmeta[lane] = r.spill.meta[e];
                }
                __syncwarp();
            }
            if (np > 0) {  // children of the top parents
                const unsigned k = np < group ? np : group;
                np -= k;
                if (lane < (k << flog)) {
                    const unsigned p = np + (lane >> flog);
                    double plo[4], phi[4];
#pragma unroll
                    for (int d = 0; d < D; ++d) {
                        plo[d] = wb.plo[d][p];
                        phi[d] = wb.phi[d][p];
                    }
                    const uint32_t m = wb.pmeta[p];
                    make_child<D>(plo, phi, a.policy, (int)((m >> 8) & 3u), (int)(lane & ((1u << flog) - 1u)), lo, hi);
                    depth = (int)(m & 0xFFu) + 1;
                    have = clip_child<FAM>(lo, hi, a.tab);
                    clipped = !have;
                }
            } else if (cur < end) {  // input boxes
                const size_t i = a.begin + (size_t)(cur + lane);
                if (lane < end - cur) {
                    depth = a.in.depth[i];
                    have = depth != 0xFF;
                    clipped = !have;
                    if (have) {
#pragma unroll
                        for (int d = 0; d < D; ++d) {
                            lo[d] = a.in.lo[d * a.in.cap + i];
                            hi[d] = a.in.hi[d * a.in.cap + i];
                        }
                    }
                }
                cur += end - cur < 32 ? end - cur : 32;
            } else if (!DEEP && more) {
                unsigned long long start = 0;
                if (lane == 0) start = atomicAdd(r.claim, (unsigned long long)per);
                cur = __shfl_sync(full, start, 0) + (unsigned long long)nwarps * per;
                more = cur < a.count;
                end = !more ? cur : cur + per < a.count ? cur + per : a.count;
                continue;
            } else if (DEEP && more) {
                if (!drawn) {
                    // the ready boxes first, unless there is input left to join them
                    unsigned seen = 0;
                    if (nr > 0) {
                        seen = *(volatile unsigned*)&r.sched->ticket;
                        seen = __shfl_sync(full, seen, 0);
                    }
                    if (nr > 0 && seen >= inputs) break;
                    if (lane == 0) ticket = atomicAdd(&r.sched->ticket, 1u);
                    ticket = __shfl_sync(full, ticket, 0);
                    drawn = true;
                }
                if (ticket < inputs && round == 0) {
                    const unsigned long long count = r.sched->count;
                    cur = (unsigned long long)ticket * per;
                    end = cur + per < count ? cur + per : count;
                    drawn = false;
                    continue;
                }
                unsigned n = 0, p;  // parents of the parcel, its slot
                const bool given_now = ticket >= inputs;
                unsigned long long* flag;
                if (!given_now) {  // a parcel left over from the last round
                    p = ticket;
                    flag = r.flags[(round + 1) & 1] + p;
                    n = parcel_left(flag_read(flag), r.sched->epoch - 1);
                    n = __shfl_sync(full, n, 0);
                    drawn = false;
                    if (n == 0) continue;
                } else {
                    if (nr > 0) break;  // (the last input went to another warp meanwhile)
                    p = (ticket - inputs) % r.slots;
                    flag = r.flags[round & 1] + p;
                    if (lane == 0) {
                        const unsigned long long epoch = r.sched->epoch;
                        atomicAdd(&r.sched->idle, 1u);
                        for (int k = 0; k < r.polls; ++k) {
                            const bool over = *(volatile unsigned*)&r.sched->idle >= nwarps;
                            __threadfence();
                            n = parcel_ready(flag_read(flag), epoch, ticket - inputs);
                            if (n || over) break;
                            __nanosleep(kWaitNs);
                        }
                        if (n) atomicSub(&r.sched->idle, 1u);
                    }
                    n = __shfl_sync(full, n, 0);
                    if (n == 0) {  // nobody gives any more, or not in time
                        more = false;
                        continue;
                    }
                    drawn = false;
                }
                const MetaList& from = r.lists[(given_now ? round : round + 1) & 1];
                parcel_take(SlotWarp{}, flag, [&] {
                    if (lane >= n) return;
                    const size_t e = (size_t)p * 32 + lane;
#pragma unroll
                    for (int d = 0; d < D; ++d) {
                        wb.plo[d][lane] = __ldcg(from.lo + d * from.cap + e);
                        wb.phi[d][lane] = __ldcg(from.hi + d * from.cap + e);
                    }
                    wb.pmeta[lane] = __ldcg(from.meta + e);
                });
                np = n;
                if (lane == 0 && given_now) atomicAdd(&r.sched->taken, 1u);
                continue;
            } else {
                break;
            }
            const unsigned mh = __ballot_sync(full, have);
            nclip += __popc(__ballot_sync(full, clipped));
            if (have) {
                const unsigned e = nr + __popc(mh & lanes_below());
#pragma unroll
                for (int d = 0; d < D; ++d) {
                    wb.rlo[d][e] = lo[d];
                    wb.rhi[d][e] = hi[d];
                }
                wb.rdepth[e] = (uint32_t)depth;
            }
            made = __popc(mh);
            nr += made;
            __syncwarp();
        }
        if (nr == 0) break;
        // the youngest ready boxes
        const unsigned take = strict ? made : nr < 32 ? nr : 32;
        nr -= take;
        const bool have = lane < take;
        const unsigned slot = nr + lane;  // (read by idle lanes too: below kReady)
        const BoxRef<D> box{&wb.rlo[0][slot], &wb.rhi[0][slot], kReady};
        int v = -1;
        bool left = false;
        if (have) {
            if (PREC == CP_FP32_PREFILTER) {
                uint8_t pmask;
                double lo[4], hi[4];
                box_copy<D>(box, lo, hi);
                const int pre = prefilter_box<FAM>(lo, hi, 0, false, &pmask);
                if (pre != PF_UNDECIDED) {
                    v = pre == PF_PROVED ? V_PROVED : pre == PF_EMPTY ? V_EMPTY : pre == PF_NOFIT ? V_NOFIT : V_CRITICAL;
                    if (pre != PF_EMPTY) ++t.fp32;
                }
            }
            if (v < 0) {
                Verdict q;
                left = !verdict_fast<FAM, DECIDE, flt::NEED_HANDLES>(box, 0, q);
                v = q.verdict;
                if (!left) handles += q.handles;
            }
        }
        if (__any_sync(full, left)) {  // boxes the filter leaves to the directed evaluation
            if (left) {
                const Verdict q = verdict_slow<FAM, DECIDE>(box, 0);
                v = q.verdict;
                handles += q.handles;
            }
            __syncwarp();
        }
        asm volatile("" ::: "memory");  // depth and box are read again, not kept in registers
        const int depth = (int)wb.rdepth[slot];
        const bool open = v >= 0 && v != V_PROVED && v != V_EMPTY;
        const bool split = open && depth < a.max_depth;
        tally_step(t, sm, v, open && !split, (unsigned)depth);
        if (a.digest) {
            double lo[4], hi[4];
            box_copy<D>(box, lo, hi);
            if (v >= 0) {
                const unsigned long long h = box_hash<D>(lo, hi, v);
                wb.dig_sum[lane] += h;
                wb.dig_xor[lane] ^= digest_xor_word(h);
            }
        }
        if (!__any_sync(full, split)) {
            if (!DEEP) continue;
        } else {
            double lo[4], hi[4];
            box_copy<D>(box, lo, hi);
            const int axis = split ? split_axis<D>(a.policy, a.lambda_scale, lo, hi) : 0;
            const bool local = split && (DEEP || depth + 1 >= a.max_depth);
            const unsigned mp = __ballot_sync(full, local);
            const unsigned cnt = __popc(mp);
            if (DEEP && np + cnt > kParents) {
                if (nspill + np <= r.seg) {
                    for (unsigned k = lane; k < np; k += 32) {
                        const size_t e = (size_t)warp_id * r.seg + nspill + k;
#pragma unroll
                        for (int d = 0; d < D; ++d) {
                            r.spill.lo[d * r.spill.cap + e] = wb.plo[d][k];
                            r.spill.hi[d * r.spill.cap + e] = wb.phi[d][k];
                        }
                        r.spill.meta[e] = wb.pmeta[k];
                    }
                    nspill += np;
                    if (lane == 0) atomicAdd(&r.sched->spilled, (unsigned long long)np);
                } else if (lane == 0) {
                    r.sched->status = 1;  // (beyond the bound)
                }
                np = 0;
                __syncwarp();
            }
            if (local) {
                const unsigned e = np + __popc(mp & lanes_below());
#pragma unroll
                for (int d = 0; d < D; ++d) {
                    wb.plo[d][e] = lo[d];
                    wb.phi[d][e] = hi[d];
                }
                wb.pmeta[e] = (uint32_t)depth | ((uint32_t)axis << 8);
            }
            np += cnt;
            __syncwarp();
            if constexpr (!DEEP)
                emit_children<FAM>(a, sm, lo, hi, depth, axis, split && !local ? 1u << flog : 0u);
        }
        constexpr bool eager = PREC == CP_FP32_PREFILTER;
        if (DEEP && np + nspill >= kMinGive<PREC> && (eager || (t.steps & 3u) == 0)) {
            // more tickets than parcels: give parents away, the older ones.  About four
            // warps per missing parcel do so at a time (a hash of warp and step picks
            // them), those with small stacks only when an eighth of the warps is waiting.
            const unsigned wanted = *(volatile unsigned*)&r.sched->ticket, given = *(volatile unsigned*)&r.sched->parcels;
            const unsigned missing = wanted > inputs + given ? wanted - inputs - given : 0u;
            const unsigned pick = (warp_id * 2654435761u + t.steps * 0x9E3779B9u) >> 16;
            bool give = (unsigned long long)pick * nwarps < (unsigned long long)missing * (4u << 16) &&
                        (eager || np + nspill >= 48 || missing * 8u > nwarps);
            give = __shfl_sync(full, (int)give, 0) != 0;
            unsigned d = 0, n = 0;
            bool room = false;  // the slot is this warp's
            if (give) {
                if (lane == 0) {
                    d = atomicAdd(&r.sched->parcels, 1u);
                    room = parcel_claim(r.flags[round & 1] + d % r.slots, r.sched->epoch, d, r.slots);
                }
                d = __shfl_sync(full, d, 0);
                room = __shfl_sync(full, (int)room, 0) != 0;
            }
            if (room) {
                const unsigned p = d % r.slots;
                const MetaList& out = r.lists[round & 1];
                // the youngest spilled parents, else half of those on chip.  (Three copies: with
                // one for both kinds the 64^4 middle lattice takes 77.6 ms instead of 75.7.)
                n = nspill >= 32 ? 32 : nspill > 0 ? nspill : np / 2;
                const bool chip = nspill == 0;
                if (!chip) nspill -= n;
                parcel_give(SlotWarp{}, r.flags[round & 1] + p, r.sched->epoch, d, n, d >= r.slots, [&] {
                    const size_t o = (size_t)p * 32 + lane;
                    const size_t e = (size_t)warp_id * r.seg + nspill + lane;
                    if (!chip && n == 32) {
#pragma unroll
                        for (int d = 0; d < D; ++d) {
                            out.lo[d * out.cap + o] = r.spill.lo[d * r.spill.cap + e];
                            out.hi[d * out.cap + o] = r.spill.hi[d * r.spill.cap + e];
                        }
                        out.meta[o] = r.spill.meta[e];
                    } else if (!chip) {
                        if (lane < n) {
#pragma unroll
                            for (int d = 0; d < D; ++d) {
                                out.lo[d * out.cap + o] = r.spill.lo[d * r.spill.cap + e];
                                out.hi[d * out.cap + o] = r.spill.hi[d * r.spill.cap + e];
                            }
                            out.meta[o] = r.spill.meta[e];
                        }
                    } else {
                        if (lane < n) {
#pragma unroll
                            for (int d = 0; d < D; ++d) {
                                out.lo[d * out.cap + o] = wb.plo[d][lane];
                                out.hi[d * out.cap + o] = wb.phi[d][lane];
                            }
                            out.meta[o] = wb.pmeta[lane];
                        }
                    }
                });
                if (lane == 0) atomicAdd(&r.sched->filled, 1u);
                if (chip) {  // entries n .. np move down to 0 (two rounds of 32 lanes)
                    for (unsigned b = 0; b < np - n; b += 32) {
                        const unsigned to = b + lane, q = n + to;
                        const bool move = q < np;
                        uint32_t m = 0;
                        double l[D], h[D];
                        if (move) {
                            m = wb.pmeta[q];
#pragma unroll
                            for (int d = 0; d < D; ++d) {
                                l[d] = wb.plo[d][q];
                                h[d] = wb.phi[d][q];
                            }
                        }
                        __syncwarp();
                        if (move) {
                            wb.pmeta[to] = m;
#pragma unroll
                            for (int d = 0; d < D; ++d) {
                                wb.plo[d][to] = l[d];
                                wb.phi[d][to] = h[d];
                            }
                        }
                        __syncwarp();
                    }
                    np -= n;
                }
            }
            __syncwarp();
        }
    }
    tally_flush(t, sm);
    tally_run(t, sm);
    if (a.digest) {
        atomicAdd(&sm.dig_sum, wb.dig_sum[lane]);
        atomicXor(&sm.dig_xor, wb.dig_xor[lane]);
    }
    if (PREC == CP_FP32_PREFILTER) {
        const unsigned n = __reduce_add_sync(full, t.fp32);
        if (lane == 0 && n) atomicAdd(&sm.hist[C_FP32], (unsigned long long)n);
    }
    if (lane == 0 && nclip) atomicAdd(&sm.hist[C_CLIPPED], (unsigned long long)nclip);
}

}  // namespace cpb
