// Placement solver: per-expert token counts -> hot-expert replication plan, for one
// NVLink domain, executed by one CTA (>= 4 warps).
//
// Results are bit-identical to the reference solver
// (csrc/kernels/placement.cu:788-1482 of the reference): same fp32 threshold
// arithmetic, same tie-breaks, same probe schedule of the threshold search, same
// largest-remainder splits. The execution is different:
//   * the ranks wait in the lanes of a warp, which finds the next source and the next taker by a reduction, and an expert is drained
//     once, from its one home rank, so a build sorts no ranks and keeps no occupancy table and no exported sums;
//   * the three builds of the fast path and the capacity pre-check run side by side on four
//     warps (the serial search takes the first that is feasible), while the other warps write
//     the outputs of all experts as they are without replicas;
//   * an export carries its redundant slot and so its physical id: behind the build the experts with replicas are written
//     over side by side, a warp or two each;
//   * each rank's masters are ranked by counting instead of a serial insertion sort;
//   * the loads come in shared memory from the caller, and with one domain the per-rank load matrix
//     too where it fits (plan.cu); else the few entries of it that are needed are read through L2.
// All of it is latency of one CTA: what counts is how many dependent instructions follow one another, how many of them branch, and
// how much code there is, since each line of it is fetched once a launch. Calls of uep_solve_placement among others on one B200: 64
// ranks x 4 experts x 2 slots 15.5 us; plan and reroute of eight ranks, 33 tokens of 64 experts each, 10.9. (With sorted lists of ranks,
// which one lane walked, and all else as it then was, 20.6 for 18.6 and 15.6 for 13.1.)
#pragma once

#include <climits>

#include "common.cuh"

namespace uep {

// The threads of a CTA that solve a problem together: their number among them, how many, and their barrier (0 to 15). A CTA can hold
// two of them; the second one has its shared memory behind the first one's, and what is out of line (below) takes the first one's, so
// it is closed to the second. (With the place as an argument it was open, and the plan's registers spilled: step of eight ranks of 8192
// bool rows of 128 with bf16 experts of 9 MB 57.7 us like this and 59.5.)
constexpr int kSecondCrewBarrier = 2;
struct Crew {
    int tid, threads, barrier;
    __device__ __forceinline__ bool second() const { return barrier == kSecondCrewBarrier; }
    __device__ __forceinline__ void sync() const { asm volatile("bar.sync %0, %1;" ::"r"(barrier), "r"(threads) : "memory"); }
};

// An export: tokens moved to a redundant slot. `place`: the slot's physical id inside the domain << 8 | its rank.
struct alignas(8) ExportEntry {
    int quota;
    int place;
};

// All the exports of one expert, which follow one another in the plan: expert, first entry, entries, rank of the master.
__device__ __forceinline__ uint32_t pack_batch(int expert, int first, int count, int rank) {
    return static_cast<uint32_t>(expert | first << 9 | count << 18) | static_cast<uint32_t>(rank) << 25;
}
static_assert(kMaxExpertsPerDomain <= 1 << 9 && kMaxExportsPerDomain <= 1 << 9 && kMaxRanksPerDomain < 1 << 7, "pack_batch");

struct SolveArgs {
    const int32_t* global_loads;    // [L]
    const int32_t* loads_per_rank;  // [N, L]
    int32_t* p2l;                   // [P]
    int32_t* l2p;                   // [L, D]
    int32_t* lcnts;                 // [L]
    int32_t* quota;                 // [L, D]
    int32_t* quota_prefix;          // [L, D]
    int32_t* rank_quota_prefix;     // [L, D]
    int32_t* physical_loads;        // [P] quota of every physical slot, 0 when empty (optional: may be null)
    int N, G, M, R, D;
    float balance_threshold;
    int min_tokens;
    int allow_zero_master;
    int locality;
    float eps;
    int my_rank;
    const int32_t* staged_loads;  // loads_per_rank[N, L] in shared memory, or null
    int preloaded;  // 1: the shared-memory loads and my_loads of the (only) domain are in place already
    unsigned long long* trace;  // optional: 8 globaltimer stamps of the solver phases (tuning aid), or null
};

// The arguments may lie in shared memory, where a pointer does not show that it is of global memory.
template <typename T>
__device__ __forceinline__ T* as_global(T* p) {
    return static_cast<T*>(__cvta_global_to_generic(__cvta_generic_to_global(p)));
}

constexpr int kSolverProbeWarps = 4;
constexpr int kSolverBuffers = 2 * kSolverProbeWarps;  // plans: one the search may end with, and those of the present round

// Control words in shared memory. kCtlBuilt0: of a buffer's plan, 0 if it is not feasible, else its batches plus one.
enum SolverCtrl { kCtlFitting = 0, kCtlHi, kCtlTotal, kCtlLargest, kCtlStop0, kCtlBuilt0 = kCtlStop0 + kSolverProbeWarps, kCtlCount = kCtlBuilt0 + kSolverBuffers };
static_assert(kCtlCount <= 32, "control words");

struct SolverSmem {
    int32_t* loads;      // [E]
    int32_t* my_loads;   // [E]
    int2* masters;       // [E] rank after rank: {load, expert}, largest load first, ties to the lower expert
    int32_t* rank_load;  // [G]
    ExportEntry* plan;   // [kSolverBuffers][slots]
    uint32_t* batches;   // [kSolverBuffers][slots]
    int* ctrl;           // [kCtlCount]
    int slots;           // redundant slots of the domain, the most exports of a plan (rounded up)
};

__host__ __device__ inline int solver_ns(int G) { return (G + 31) / 32; }
__host__ __device__ inline int solver_pad(int n) { return (n + 3) / 4 * 4; }
__host__ __device__ inline size_t solver_smem_bytes(int E, int G, int R) {
    return sizeof(int32_t) * (4 * static_cast<size_t>(solver_pad(E)) + solver_pad(G)) +
           kSolverBuffers * (sizeof(ExportEntry) + sizeof(uint32_t)) * solver_pad(G * R) + sizeof(int) * 32;
}

__device__ inline SolverSmem carve_solver_smem(char* raw, int E, int G, int R) {
    const int ep = solver_pad(E), gp = solver_pad(G), slots = solver_pad(G * R);
    SolverSmem s;
    int32_t* p = reinterpret_cast<int32_t*>(raw);
    s.loads = p; p += ep;
    s.my_loads = p; p += ep;
    s.masters = reinterpret_cast<int2*>(p); p += 2 * ep;
    s.rank_load = p; p += gp;
    s.plan = reinterpret_cast<ExportEntry*>(p); p += kSolverBuffers * 2 * slots;
    s.batches = reinterpret_cast<uint32_t*>(p); p += kSolverBuffers * slots;
    s.ctrl = reinterpret_cast<int*>(p);
    s.slots = slots;
    return s;
}

// Over the first n lanes.
__device__ __forceinline__ int warp_inclusive_scan(int v, int lane, int n) {
#pragma unroll 1
    for (int off = 1; off < n; off <<= 1) {
        const int t = __shfl_up_sync(kFullMask, v, off);
        if (lane >= off) v += t;
    }
    return v;
}

// Greedy export plan for one threshold, by one warp. Returns feasibility (uniform over
// the warp). Semantics of csrc/kernels/placement.cu:337-667 of the reference.
//
// The ranks above the threshold give experts away, largest load first, ties to the lower rank, and of each its masters, likewise. An
// expert's exports go to the ranks below it by slack, largest first, ties to the lower rank, each rank once; every one of them is
// filled up except the last, which comes back with the slack it has left once the expert is placed. A chain of dependent steps by
// nature. A lane holds the ranks lane, lane + 32, .. as keys, amount << 7 | 127 - rank, -1 where there is none, so that the next rank is
// the warp's largest key: one reduction, and its lane notices by itself that it was chosen. All the rest of an export is the same few
// instructions in every lane, with one branch, and the next source and its master are asked for beside the exports of this one.
// An export takes some 55 cycles, a source 290. (Sorted lists in shared memory, walked by one lane: several loads and selects an
// export; ranks x experts x slots, calls among others with the lists and when they were replaced by this (us), 72 x 7 x 4 28.1 and 23.9,
// 32 x 4 x 2 12.5 and 10.6, with rounds of probes, 16 x 2 x 1, 21.3 both.)
// kKeys: keys a lane. kWide: a key is the amount alone, where amount << 7 does not fit 31 bits, and the rank is a second reduction.
// kProbe: the floor is static, and nobody stops the build; else `stop` is raised by a warp whose result makes it pointless.
template <int kKeys, bool kWide, bool kProbe>
__device__ __forceinline__ bool drain_sources(const SolverSmem& sm, int buffer, int& num_batches, int thr, int G, int M, int R, int min_tokens,
                                              bool allow_zero_master, bool dynamic_floor, int lane, const volatile int* stop) {
    ExportEntry* const plan = sm.plan + buffer * sm.slots;
    uint32_t* const batches = sm.batches + buffer * sm.slots;
    const int keep = allow_zero_master ? 0 : 1, Lp = M + R;
    auto encode = [](int amount, int rank) { return kWide ? amount : amount << 7 | (127 - rank); };
    auto amount_of = [](int key) { return kWide ? key : key >> 7; };
    auto largest = [&](const int (&key)[kKeys]) {
        int mine = key[0];
#pragma unroll
        for (int k = 1; k < kKeys; ++k) mine = max(mine, key[k]);
        return __reduce_max_sync(kFullMask, mine);
    };
    auto rank_of = [&](const int (&key)[kKeys], int best) {
        if (!kWide) return 127 - (best & 127);
        int r = INT_MAX;  // the lowest one that has it
#pragma unroll
        for (int k = kKeys - 1; k >= 0; --k) r = key[k] == best ? lane + k * kWarp : r;
        return __reduce_min_sync(kFullMask, r);
    };
    int above[kKeys], below[kKeys];  // keys of the excess, of the slack
    int place[kKeys], last[kKeys];   // of the rank's next redundant slot, as the plan has it, and of the one behind its last
#pragma unroll
    for (int k = 0; k < kKeys; ++k) {
        const int rank = lane + k * kWarp, load = rank < G ? sm.rank_load[rank] : thr;
        above[k] = load > thr ? encode(load - thr, rank) : -1;
        below[k] = load < thr ? encode(thr - load, rank) : -1;
        place[k] = (rank * Lp + M) << 8 | rank;
        last[k] = place[k] + (R << 8);
    }
    const int first_source = largest(above);
    int need = amount_of(first_source), from = rank_of(above, first_source), at_master = from * M;
    int2 master = sm.masters[at_master];
    int num_exports = 0, left = M, stopped = 0;
    num_batches = 0;
    while (true) {
        // what only the next expert needs: its source if this one is the source's last, its master; and whether to go on at all
#pragma unroll
        for (int k = 0; k < kKeys; ++k) above[k] = from == lane + k * kWarp ? -1 : above[k];
        const int next_source = largest(above);
        int count = 0;  // ranks with slack and slots
        if (!kProbe) {
#pragma unroll
            for (int k = 0; k < kKeys; ++k) count += __popc(__ballot_sync(kFullMask, below[k] >= 0));
            if (__any_sync(kFullMask, stopped != 0)) return false;
            stopped = *stop;
        }
        const int next_from = next_source >= 0 ? rank_of(above, next_source) : 0;
        const int2 next_master = sm.masters[next_from * M], follow = sm.masters[min(at_master + 1, G * M - 1)];

        const int give = min(need, max(master.x - keep, 0));
        if (give == 0) return false;  // the masters come by load: no later one of this source has anything to give
        // an export is of at least min_tokens, or (dynamic) of ceil(what is still needed / the ranks that could still take part)
        const int by_count = !kProbe && dynamic_floor ? 1 : 0;
        int times = by_count != 0 ? count : 1, floor = by_count != 0 ? need : max(min_tokens, 0);
        int move = give, made = 0, best, q;
        bool small, hit[kKeys];
        do {
            best = largest(below);
            const int slack = amount_of(best), rank = kWide ? rank_of(below, best) : 0;
            q = min(slack, move);
            small = kWide ? static_cast<long long>(q) * times < floor : q * times < floor;  // with no rank left, too
            int at = -1;
#pragma unroll
            for (int k = 0; k < kKeys; ++k) {
                hit[k] = kWide ? rank == lane + k * kWarp : below[k] == best;
                at = hit[k] ? place[k] : at;
                place[k] += hit[k] ? 1 << 8 : 0;
                below[k] = hit[k] ? -1 : below[k];
            }
            if (at >= 0) plan[num_exports + made] = ExportEntry{q, at};
            ++made;
            times -= by_count;
            floor -= by_count * q;
            move -= slack;
        } while (move > 0 && !small);
        const int rest = -move;  // of the last one's slack
        if (small) {
            // The last one is too small, and is taken back. No later master of this source has more to give: where this one has made
            // no export, or the best rank's slack is what is too small, the others fail in the same way. (A threshold with the
            // static floor fails at its first source mostly; the walk over the other masters was the longest of the four builds.)
            if (made == 1 || rest <= 0) return false;
            --made;
            need += q;
#pragma unroll
            for (int k = 0; k < kKeys; ++k) {
                if (hit[k]) {
                    below[k] = best;
                    place[k] -= 1 << 8;
                }
            }
        } else {
#pragma unroll
            for (int k = 0; k < kKeys; ++k) {
                if (hit[k]) below[k] = rest > 0 && place[k] < last[k] ? encode(rest, lane + k * kWarp) : -1;
            }
        }
        if (lane == 0) batches[num_batches] = pack_batch(master.y, num_exports, made, from);
        ++num_batches;
        num_exports += made;
        need -= give;
        if (need > 0) {
            if (--left == 0) return false;
            ++at_master;
            master = follow;
            continue;
        }
        if (next_source < 0) return true;
        left = M;
        need = amount_of(next_source);
        from = next_from;
        at_master = from * M;
        master = next_master;
    }
}

// Out of line: groups and loads that need it are rare where the plan is short of time, and code that is jumped over is fetched all the
// same (below).
template <int kKeys, bool kWide, bool kProbe>
__device__ __noinline__ bool drain_sources_apart(int buffer, int& num_batches, int thr, int G, int M, int R, int min_tokens, bool allow_zero_master,
                                                 bool dynamic_floor, int lane, const volatile int* stop) {
    extern __shared__ __align__(128) char smem_raw[];  // the kernel's: as an argument its address would not be known to be shared
    const SolverSmem sm = carve_solver_smem(smem_raw, G * M, G, R);
    return drain_sources<kKeys, kWide, kProbe>(sm, buffer, num_batches, thr, G, M, R, min_tokens, allow_zero_master, dynamic_floor, lane, stop);
}
constexpr int kMostKeys = (kMaxRanksPerDomain + kWarp - 1) / kWarp;

// By one warp, into plan buffer `buffer`. `total`, `largest`: of the ranks' loads. kProbe: a static floor, and nobody stops it.
template <bool kProbe>
__device__ __forceinline__ bool warp_build_plan(const Crew& crew, const SolverSmem& sm, int buffer, int& num_batches, int thr, int total, int largest, int G, int M, int R,
                                                int min_tokens, bool allow_zero_master, bool dynamic_floor, int lane, const volatile int* stop) {
    num_batches = 0;
    if (largest <= thr) return true;
    // The excess has to fit the slack, and their difference is the sum of (load - threshold). Every export takes the same from
    // both, so the slack left always covers the excess left.
    if (total > static_cast<long long>(G) * thr) return false;
    const bool narrow = largest < 1 << 24;  // (then a slack times a number of ranks is below 2^31, too)
    if (narrow && G <= kWarp) {
        return drain_sources<1, false, kProbe>(sm, buffer, num_batches, thr, G, M, R, min_tokens, allow_zero_master, dynamic_floor, lane, stop);
    }
    if (crew.second()) return false;
    if (!narrow) return drain_sources_apart<kMostKeys, true, kProbe>(buffer, num_batches, thr, G, M, R, min_tokens, allow_zero_master, dynamic_floor, lane, stop);
    if (G <= 2 * kWarp) return drain_sources_apart<2, false, kProbe>(buffer, num_batches, thr, G, M, R, min_tokens, allow_zero_master, dynamic_floor, lane, stop);
    return drain_sources_apart<kMostKeys, false, kProbe>(buffer, num_batches, thr, G, M, R, min_tokens, allow_zero_master, dynamic_floor, lane, stop);
}

// The first warp of a round whose plan is feasible, -1: none; its batches go to num_batches.
__device__ __forceinline__ int first_feasible(const SolverSmem& sm, int buffer0, int& num_batches) {
    int first = -1;
#pragma unroll
    for (int w = kSolverProbeWarps - 1; w >= 0; --w) {
        const int built = sm.ctrl[kCtlBuilt0 + buffer0 + w];
        if (built != 0) {
            first = w;
            num_batches = built - 1;
        }
    }
    return first;
}

// The probes of the search: four a round. Every thread follows the interval, and a round's results are read behind its one barrier: the
// next round builds into the four buffers that do not hold the best plan so far, and the results of the round after that are
// written behind the next barrier. (Four barriers a round and the best threshold built again: 16 ranks x 2 experts x 1 slot
// 20.0 us, 18.8 like this.) Returns the plan's buffer and its batches. All threads of the CTA; the first four warps' buffers hold nothing that counts.
// Out of line, with a build of its own that knows its floor (one build, in one loop, for these and for the four in front of them: 16
// ranks x 2 experts x 1 slot 27.4 us for 21.9).
__device__ __noinline__ int2 probe_thresholds(Crew crew, int fitting, int hi0, int total, int largest, int G, int M, int R, int min_tokens,
                                              bool allow_zero_master) {
    extern __shared__ __align__(128) char smem_raw[];  // the kernel's: as an argument its address would not be known to be shared
    const SolverSmem sm = carve_solver_smem(smem_raw, G * M, G, R);
    const int warp = crew.tid >> 5, lane = crew.tid & 31;
    int lo = min(fitting + 1, hi0), hi = hi0, winner = -1, num_batches = 0;
    for (int set = kSolverProbeWarps; lo < hi;) {
        const int range = hi - lo;
        const bool each = range <= kSolverProbeWarps;
        auto probe = [&](int w) {
            return lo + (each ? w : static_cast<int>((static_cast<long long>(range) * (w + 1)) / (kSolverProbeWarps + 1)));
        };
        if (warp < kSolverProbeWarps) {
            int n = 0;
            const bool ok = (!each || warp < range) &&
                            warp_build_plan<true>(crew, sm, set + warp, n, probe(warp), total, largest, G, M, R, min_tokens, allow_zero_master, false, lane, nullptr);
            if (lane == 0) sm.ctrl[kCtlBuilt0 + set + warp] = ok ? n + 1 : 0;
        }
        crew.sync();
        const int first = first_feasible(sm, set, num_batches);
        if (first >= 0) {
            hi = probe(first);
            winner = set + first;
            lo = each ? hi : (first > 0 ? probe(first - 1) + 1 : lo);
            set ^= kSolverProbeWarps;
        } else {
            lo = each ? hi : probe(kSolverProbeWarps - 1) + 1;
            crew.sync();  // the same buffers again
        }
    }
    // no probe succeeded: at the largest load nothing is to be moved
    return winner >= 0 ? make_int2(winner, num_batches) : make_int2(0, 0);
}

// x = a * b over d, for a, b >= 0 and d > 0: quotient and remainder. A float estimate of a quotient below 2^20 is off by
// one at most (six roundings of 2^-24 each), which the remainder shows.
__device__ __forceinline__ void product_over(int a, int b, int d, int& quotient, int& remainder) {
    const long long x = static_cast<long long>(a) * b;
    const float estimate = static_cast<float>(a) * static_cast<float>(b) * __frcp_rn(static_cast<float>(d));
    if (estimate < 1048576.f) {
        int q = static_cast<int>(estimate);
        long long r = x - static_cast<long long>(q) * d;
        if (r < 0) {
            --q;
            r += d;
        } else if (r >= d) {
            ++q;
            r -= d;
        }
        quotient = q;
        remainder = static_cast<int>(r);
    } else {
        quotient = static_cast<int>(x / d);
        remainder = static_cast<int>(x % d);
    }
}

// Outputs of an expert with more than 32 replicas, by one thread: the split of this rank's tokens over the expert's replicas,
// as an inclusive prefix. Semantics of csrc/kernels/placement.cu:1342-1481 / :669-786 of the reference. Not inlined: its
// arrays and its code are for one rare case.
__device__ __noinline__ void write_many_replicas(SolveArgs a, int first_rank, int e, int C, int load, int my_load, const ExportEntry* exports) {
    constexpr int MAXC = kMaxRanksPerDomain;
    const int Lp = a.M + a.R, L = a.N * a.M, l_global = first_rank * a.M + e;
    const int64_t row = static_cast<int64_t>(l_global) * a.D;
    int phys[MAXC], q[MAXC];
    phys[0] = (first_rank + e / a.M) * Lp + e % a.M;
    q[0] = load;
    for (int j = 1; j < C; ++j) {
        phys[j] = first_rank * Lp + (exports[j - 1].place >> 8);
        q[j] = exports[j - 1].quota;
        q[0] -= q[j];
        a.p2l[phys[j]] = l_global;
        a.l2p[row + j] = phys[j];
    }
    int upto = 0;
    for (int j = 0; j < C; ++j) {
        upto += q[j];
        a.quota[row + j] = q[j];
        a.quota_prefix[row + j] = upto;
        if (a.physical_loads != nullptr) a.physical_loads[phys[j]] = q[j];
    }
    int host_rank[MAXC], my_alloc[MAXC];
    long long remainders[MAXC];
    for (int j = 0; j < C; ++j) {
        host_rank[j] = phys[j] / Lp;
        my_alloc[j] = 0;
        remainders[j] = -1;
    }
    if (!a.locality) {
        const int rem_my = my_load;
        int assigned = 0, total_quota = 0;
        for (int j = 0; j < C; ++j) total_quota += q[j];
        if (rem_my > 0 && total_quota > 0) {
            for (int j = 0; j < C; ++j) {
                const long long scaled = static_cast<long long>(rem_my) * q[j];
                const int share = static_cast<int>(scaled / total_quota);
                my_alloc[j] = share;
                remainders[j] = scaled % total_quota;
                assigned += share;
            }
            int remaining = rem_my - assigned;
            while (remaining > 0) {
                int best_j = -1;
                for (int j = 0; j < C; ++j) {
                    if (best_j < 0 || remainders[j] > remainders[best_j]) best_j = j;  // ties keep the lower j
                }
                my_alloc[best_j] += 1;
                remainders[best_j] = -1;
                --remaining;
            }
        }
    } else {
        int remote_cap[MAXC];
        int host_left[MAXC];  // remaining own load of host_rank[j]'s rank, shared between equal hosts via `first`
        int first[MAXC];
        int rem_my = my_load;
        int total_remote_cap = 0;
        for (int j = 0; j < C; ++j) {
            int f = j;
            for (int u = 0; u < j; ++u) {
                if (host_rank[u] == host_rank[j]) {
                    f = first[u];
                    break;
                }
            }
            first[j] = f;
            if (f == j) {
                host_left[j] = __ldcg(a.loads_per_rank + static_cast<int64_t>(host_rank[j]) * L + l_global);
            }
            const int qj = q[j];
            const int local_fill = min(host_left[f], qj);
            host_left[f] -= local_fill;
            remote_cap[j] = qj - local_fill;
            total_remote_cap += remote_cap[j];
            if (host_rank[j] == a.my_rank) {
                my_alloc[j] += local_fill;
                rem_my -= local_fill;
            }
        }
        rem_my = max(rem_my, 0);
        if (rem_my > 0 && total_remote_cap > 0) {
            int assigned = 0;
            for (int j = 0; j < C; ++j) {
                if (host_rank[j] == a.my_rank || remote_cap[j] <= 0) continue;
                const long long scaled = static_cast<long long>(rem_my) * remote_cap[j];
                const int share = static_cast<int>(scaled / total_remote_cap);
                my_alloc[j] += share;
                remainders[j] = scaled % total_remote_cap;
                assigned += share;
            }
            int remaining = rem_my - assigned;
            while (remaining > 0) {
                int best_j = -1;
                for (int j = 0; j < C; ++j) {
                    if (host_rank[j] == a.my_rank || remote_cap[j] <= 0) continue;
                    if (best_j < 0 || remainders[j] > remainders[best_j] ||
                        (remainders[j] == remainders[best_j] &&
                         (host_rank[j] < host_rank[best_j] || (host_rank[j] == host_rank[best_j] && j < best_j)))) {
                        best_j = j;
                    }
                }
                if (best_j < 0) break;
                my_alloc[best_j] += 1;
                remainders[best_j] = -1;
                --remaining;
            }
        }
    }
    int prefix = 0;
    for (int j = 0; j < C; ++j) {
        prefix += my_alloc[j];
        a.rank_quota_prefix[row + j] = prefix;
    }
}

// The same split for an expert with 2..32 replicas, by one warp: lane j
// holds replica j on rank `host`, which has `own` tokens for the expert itself, and the sums and
// arg-max searches are warp reductions. The hosts differ: an export never goes to a rank that
// holds the expert already.
__device__ __forceinline__ void warp_rank_quota_prefix(const SolveArgs& a, int l_global, int C, int my_load, int host,
                                                       int q, int own, int lane) {
    const bool active = lane < C;
    int my_alloc = 0;
    if (!a.locality) {
        const int total_quota = __reduce_add_sync(kFullMask, active ? q : 0);
        if (my_load > 0 && total_quota > 0) {
            int share, rem;
            product_over(my_load, active ? q : 0, total_quota, share, rem);
            if (!active) rem = INT_MIN;
            my_alloc = share;
            int remaining = my_load - __reduce_add_sync(kFullMask, share);  // < C: a sum of C fractional parts
            for (int it = 0; it < C && remaining > 0; ++it) {
                const int best = __reduce_max_sync(kFullMask, rem);
                const int pick = __ffs(__ballot_sync(kFullMask, active && rem == best)) - 1;  // ties: the lower j
                if (lane == pick) {
                    my_alloc += 1;
                    rem = -1;
                }
                --remaining;
            }
        }
    } else {
        const int local_fill = active ? min(own, q) : 0;
        const int remote_cap = active ? q - local_fill : 0;
        const int total_remote_cap = __reduce_add_sync(kFullMask, remote_cap);
        const bool mine = active && host == a.my_rank;
        if (mine) my_alloc = local_fill;
        const int rem_my = max(my_load - __reduce_add_sync(kFullMask, mine ? local_fill : 0), 0);
        if (rem_my > 0 && total_remote_cap > 0) {
            const bool eligible = active && !mine && remote_cap > 0;
            int share, rem;
            product_over(rem_my, eligible ? remote_cap : 0, total_remote_cap, share, rem);
            if (!eligible) rem = INT_MIN;
            my_alloc += share;
            int remaining = rem_my - __reduce_add_sync(kFullMask, share);  // < number of eligible replicas
            for (int it = 0; it < C && remaining > 0; ++it) {
                const int best = __reduce_max_sync(kFullMask, rem);
                if (best == INT_MIN) break;  // nobody can take a unit
                // ties: the lower host rank, then the lower j
                const bool cand = eligible && rem == best;
                const int best_host = __reduce_min_sync(kFullMask, cand ? host : INT_MAX);
                const int pick = __ffs(__ballot_sync(kFullMask, cand && host == best_host)) - 1;
                if (lane == pick) {
                    my_alloc += 1;
                    rem = -1;
                }
                --remaining;
            }
        }
    }
    const int prefix = warp_inclusive_scan(my_alloc, lane, C);
    if (active) as_global(a.rank_quota_prefix)[static_cast<int64_t>(l_global) * a.D + lane] = prefix;
}

// Solve one NVLink domain. All threads of the crew must call it (128 at least,
// multiple of 32). smem_raw must hold solver_smem_bytes(E, G, R) bytes, 16-byte aligned; of a first crew it is the start of the CTA's dynamic
// shared memory. A second crew leaves a problem as it is that needs more than 32 ranks, loads from 2^24 on or probes.
__device__ __forceinline__ void solve_domain(const SolveArgs& a, const Crew& crew, int domain, char* smem_raw, DeviceStatus* status) {
    const int tid = crew.tid, nthreads = crew.threads;
    const int warp = tid >> 5, lane = tid & 31;
    const int G = a.G, M = a.M, R = a.R, D = a.D;
    const int E = G * M, Lp = M + R, L = a.N * M;
    const int domain_start_rank = domain * G;
    const int domain_start_log = domain_start_rank * M;
    SolverSmem sm = carve_solver_smem(smem_raw, E, G, R);
    auto stamp = [&](int slot) {
        if (a.trace != nullptr && tid == 0) a.trace[slot] = global_timer_ns();
    };
    stamp(0);
    int32_t *const out_p2l = as_global(a.p2l), *const out_l2p = as_global(a.l2p), *const out_lcnts = as_global(a.lcnts);
    int32_t *const out_quota = as_global(a.quota), *const out_quota_prefix = as_global(a.quota_prefix);
    int32_t *const out_rank_quota_prefix = as_global(a.rank_quota_prefix);
    int32_t* const out_physical_loads = a.physical_loads != nullptr ? as_global(a.physical_loads) : nullptr;

    // Every output of this domain as it is without replicas (an expert then keeps all of this rank's tokens: every branch of
    // the split reduces to that); run by `n` threads once the loads are in place. The experts with replicas are written over.
    auto write_masters = [&](int t, int n) {
        for (int i = t; i < G * Lp; i += n) {
            const int rank = i / Lp, local = i - rank * Lp, e = rank * M + local;
            out_p2l[domain_start_rank * Lp + i] = local < M ? domain_start_log + e : -1;
            if (out_physical_loads != nullptr) out_physical_loads[domain_start_rank * Lp + i] = local < M ? sm.loads[e] : 0;
        }
        for (int e = t; e < E; e += n) out_lcnts[domain_start_log + e] = 1;
        const int64_t first = static_cast<int64_t>(domain_start_log) * D;
        auto master = [&](int e) { return (domain_start_rank + e / M) * Lp + e % M; };
        const uintptr_t align = reinterpret_cast<uintptr_t>(out_l2p) | reinterpret_cast<uintptr_t>(out_quota) |
                                reinterpret_cast<uintptr_t>(out_quota_prefix) | reinterpret_cast<uintptr_t>(out_rank_quota_prefix);
        if (D % 4 == 0 && (align & 15u) == 0) {
            const int vecs = D / 4;
            for (int i = t; i < E * vecs; i += n) {
                const int e = i / vecs;
                const bool head = i - e * vecs == 0;
                const int4 load = make_int4(head ? sm.loads[e] : 0, 0, 0, 0);
                reinterpret_cast<int4*>(out_l2p + first)[i] = make_int4(head ? master(e) : -1, -1, -1, -1);
                reinterpret_cast<int4*>(out_quota + first)[i] = load;
                reinterpret_cast<int4*>(out_quota_prefix + first)[i] = load;
                reinterpret_cast<int4*>(out_rank_quota_prefix + first)[i] = make_int4(head ? sm.my_loads[e] : 0, 0, 0, 0);
            }
        } else {
            for (int i = t; i < E * D; i += n) {
                const int e = i / D;
                const bool head = i - e * D == 0;
                out_l2p[first + i] = head ? master(e) : -1;
                out_quota[first + i] = head ? sm.loads[e] : 0;
                out_quota_prefix[first + i] = head ? sm.loads[e] : 0;
                out_rank_quota_prefix[first + i] = head ? sm.my_loads[e] : 0;
            }
        }
    };
    if (!a.preloaded) {
        for (int i = tid; i < E; i += nthreads) {
            sm.loads[i] = __ldcg(a.global_loads + domain_start_log + i);
            sm.my_loads[i] = __ldcg(a.loads_per_rank + static_cast<int64_t>(a.my_rank) * L + domain_start_log + i);
        }
    }
    if (tid < kSolverProbeWarps) sm.ctrl[kCtlStop0 + tid] = 0;
    const bool do_search = (R > 0 && G > 1);
    stamp(1);
    crew.sync();
    if (do_search) {
        // each rank's masters by load descending, ties to the lower index, and its load; four masters a load where they lie so
        const bool fours = (M & 3) == 0;
        for (int i = tid; i < E; i += nthreads) {
            const int rank = i / M, base = rank * M;
            const unsigned mine = static_cast<unsigned>(sm.loads[i]);
            int pos = 0, sum = 0;
            auto look = [&](int j, int other) {
                pos += static_cast<unsigned>(other) + (j < i ? 1u : 0u) > mine ? 1 : 0;
                sum += other;
            };
            if (fours) {
#pragma unroll 4
                for (int j = base; j < base + M; j += 4) {
                    const int4 v = *reinterpret_cast<const int4*>(sm.loads + j);
                    look(j, v.x);
                    look(j + 1, v.y);
                    look(j + 2, v.z);
                    look(j + 3, v.w);
                }
            } else {
#pragma unroll 8
                for (int j = base; j < base + M; ++j) look(j, sm.loads[j]);
            }
            sm.masters[base + pos] = make_int2(static_cast<int>(mine), i);
            if (i == base) sm.rank_load[rank] = sum;
        }
        crew.sync();
    }
    stamp(2);
    const bool allow0 = a.allow_zero_master != 0;
    // Without a search by all threads; else by the warps that build no plans (where there are any).
    const int builders = do_search && nthreads > kSolverProbeWarps * kWarp ? kSolverProbeWarps * kWarp : 0;
    if (tid >= builders) write_masters(tid - builders, nthreads - builders);
    int winner = 0, num_batches = 0;  // the buffer whose plan is taken
    if (do_search) {
        // The serial search is: up to three builds with the dynamic floor at rising thresholds; then one build at the
        // smallest threshold the capacities allow; then the probes. The first four run at once, one warp each; one that
        // succeeds stops those behind it.
        // Mostly this code comes from DRAM, a line after the other, and what is jumped over comes too: so what a call seldom needs is
        // out of line (the probes, the wide and the many keys, more than 32 replicas), and the outputs are compiled in once.
        // Plan of eight ranks behind an L2 flush, on the device (us), with all builds and widths inlined and when that was changed: 33
        // tokens of 64 experts 19.3 and 13.3, 4096 tokens 17.8 and 15.7; among other plans 10.3 and 9.5, 12.8 and 11.8.
        if (warp < kSolverProbeWarps) {
            int total = 0, largest = 0;
            for (int r = lane; r < G; r += kWarp) {
                total += sm.rank_load[r];
                largest = max(largest, sm.rank_load[r]);
            }
            total = warp_sum(total);
            largest = warp_max(largest);
            // fp32, in the reference's order: ceilf((float(total) / G) * bt). A power of two divides by a multiplication.
            const float bt = fmaxf(a.balance_threshold, 1.0f), sum = static_cast<float>(total), ranks = static_cast<float>(G);
            const float mean = (G & (G - 1)) == 0 ? __fmul_rn(sum, __uint_as_float(0x7F000000u - __float_as_uint(ranks))) : __fdiv_rn(sum, ranks);
            const int lo0 = static_cast<int>(ceilf(__fmul_rn(mean, bt))), hi0 = max(largest, lo0);
            const bool fast = warp < kSolverProbeWarps - 1;
            int thr;
            if (fast) {
                const float eps = fmaxf(a.eps, 0.0f);
                thr = max(static_cast<int>(ceilf(__fmul_rn(static_cast<float>(lo0), __fadd_rn(1.0f, eps)))), lo0);
                const int step = max(1, (hi0 + 99) / 100);
                for (int i = 0; i < warp; ++i) thr = min(hi0, thr + step);
            } else {
                // The smallest threshold from lo0 to hi0 whose excess fits its slack. Excess minus slack is the sum of (load - threshold):
                // it fits from the mean load on. (The reference bisects, csrc/kernels/placement.cu:76-84.)
                thr = min(max(lo0, static_cast<int>((static_cast<unsigned>(total) + G - 1) / G)), hi0);
                if (lane == 0) {
                    sm.ctrl[kCtlFitting] = thr;
                    sm.ctrl[kCtlHi] = hi0;
                    sm.ctrl[kCtlTotal] = total;
                    sm.ctrl[kCtlLargest] = largest;
                }
            }
            int n = 0;
            const bool ok = warp_build_plan<false>(crew, sm, warp, n, thr, total, largest, G, M, R, a.min_tokens, allow0, fast, lane, sm.ctrl + kCtlStop0 + warp);
            if (lane == 0) sm.ctrl[kCtlBuilt0 + warp] = ok ? n + 1 : 0;
            if (ok && lane > warp && lane < kSolverProbeWarps) *(sm.ctrl + kCtlStop0 + lane) = 1;
        }
        crew.sync();
        winner = first_feasible(sm, 0, num_batches);
        if (__builtin_expect(winner < 0, 0)) {
            if (crew.second()) return;
            const int2 found = probe_thresholds(crew, sm.ctrl[kCtlFitting], sm.ctrl[kCtlHi], sm.ctrl[kCtlTotal], sm.ctrl[kCtlLargest], G, M, R, a.min_tokens, allow0);
            winner = found.x;
            num_batches = found.y;
        }
    }
    stamp(3);
    // The experts with replicas, one per warp at a time, over what was written without them: lane 0 is the master, lane j the
    // j-th export in the order of their creation.
    const ExportEntry* plan = sm.plan + winner * sm.slots;
    const uint32_t* batches = sm.batches + winner * sm.slots;
    // Where there are warps enough, one of its own splits this rank's tokens, which takes longest, and the others write the rows.
    const int warps = nthreads / kWarp;
    const bool apart = num_batches < warps, split_only = apart && warp < num_batches, emit_only = apart && !split_only;
    for (int task = emit_only ? warp - num_batches : warp; task < num_batches; task += emit_only ? warps - num_batches : warps) {
        const uint32_t batch = batches[task];
        const bool emits = !split_only, splits = !emit_only;
        const int e = batch & 511, first = batch >> 9 & 511, C = static_cast<int>(batch >> 18 & 127) + 1, home = batch >> 25;
        const int l_global = domain_start_log + e;
        const int64_t row = static_cast<int64_t>(l_global) * D;
        const int my_load = sm.my_loads[e];
        if (C > D) {
            if (lane == 0) report_error(status, UEP_DEV_BAD_PLAN, l_global);
            continue;
        }
        if (lane == 0 && emits) out_lcnts[l_global] = C;
        if (C <= kWarp) {
            const bool active = lane < C;
            const ExportEntry entry = lane > 0 && active ? plan[first + lane - 1] : ExportEntry{0, 0};
            const int moved = warp_sum(entry.quota);
            const int host = domain_start_rank + (lane == 0 ? home : entry.place & 255);
            const int q = lane == 0 ? sm.loads[e] - moved : entry.quota;
            if (emits) {
                const int phys = lane == 0 ? host * Lp + e - home * M : domain_start_rank * Lp + (entry.place >> 8);
                const int prefix = warp_inclusive_scan(q, lane, C);
                if (active) {
                    out_quota[row + lane] = q;
                    out_quota_prefix[row + lane] = prefix;
                    if (out_physical_loads != nullptr) out_physical_loads[phys] = q;
                    if (lane > 0) {
                        out_p2l[phys] = l_global;
                        out_l2p[row + lane] = phys;
                    }
                }
            }
            if (splits) {
                int own = 0;
                if (a.locality && active) {
                    const int64_t at = static_cast<int64_t>(host) * L + l_global;
                    own = a.staged_loads != nullptr ? a.staged_loads[at] : __ldcg(a.loads_per_rank + at);
                }
                warp_rank_quota_prefix(a, l_global, C, my_load, active ? host : -1 - lane, q, own, lane);
            }
        } else if (lane == 0 && emits) {
            write_many_replicas(a, domain_start_rank, e, C, sm.loads[e], my_load, plan + first);
        }
    }
    crew.sync();
    stamp(4);
}

// ---------------------------------------------------------------------------------------------
// Legacy placement (legacy_placement=True). The reference solves this mode on the host after copying the
// loads back and synchronising the stream (csrc/kernels/legacy/placement_cpu.cpp:17-241); here it is one
// warp of the plan kernel, so the mode costs no host round trip. Same greedy, same doubles (IEEE
// division and addition, never contracted), same tie-breaks:
//   1. redundant slots are granted one at a time to the expert with the largest load per instance
//      (ties: lower id; at most G-1 extra instances per expert; with balance_threshold > 1 the granting
//      stops once the best load per instance is within threshold x the mean load per master slot);
//   2. the extra instances, ordered by load per instance descending then expert id, go to the rank
//      with the smallest accumulated load (ties: lower rank) that has a free slot and does not hold
//      the expert; an instance that finds no rank is dropped.
// Quotas are not used in this mode: the reroute is round-robin over an expert's instances.
// Shared memory: legacy_smem_bytes(E, G). All threads of the CTA must call it.
// ---------------------------------------------------------------------------------------------
__host__ __device__ inline size_t legacy_smem_bytes(int E, int G) {
    return sizeof(double) * (static_cast<size_t>(E) + 2 * kMaxExportsPerDomain + solver_pad(G)) +
           sizeof(int32_t) * (3 * static_cast<size_t>(E) + 2 * kMaxExportsPerDomain + solver_pad(G) + 8) +
           sizeof(uint32_t) * static_cast<size_t>(E) * solver_ns(G);
}

// Inlined where it is all that the kernel does, and out of line in the plan. Calls of uep_legacy_solve_placement, out of line and inlined
// (us): 8 ranks x 16 experts x 4 slots 59.4 and 55.4, 64 x 8 x 8 1129 and 1101; legacy plans of 128 experts 61.5 and 62.6.
__device__ __forceinline__ void legacy_solve(const SolveArgs& a, int domain, char* smem_raw, DeviceStatus* status) {
    const int tid = threadIdx.x, nthreads = blockDim.x, lane = tid & 31, warp = tid >> 5;
    const int G = a.G, M = a.M, R = a.R, D = a.D, E = G * M, Lp = M + R, ns = solver_ns(G);
    const int rank0 = domain * G, log0 = rank0 * M;
    double* score = reinterpret_cast<double*>(smem_raw);        // [E] load per instance
    double* xkey = score + E;                                    // [512] extras: load per instance
    double* xkey_sorted = xkey + kMaxExportsPerDomain;           // [512]
    double* rank_load = xkey_sorted + kMaxExportsPerDomain;      // [Gpad]
    int32_t* loads = reinterpret_cast<int32_t*>(rank_load + solver_pad(G));  // [E]
    int32_t* cnt = loads + E;                                    // [E] instances
    int32_t* placed = cnt + E;                                   // [E] instances placed so far (incl. master)
    int32_t* xid = placed + E;                                   // [512] extras: expert
    int32_t* xid_sorted = xid + kMaxExportsPerDomain;            // [512]
    int32_t* used = xid_sorted + kMaxExportsPerDomain;           // [Gpad] redundant slots used per rank
    int32_t* ctl = used + solver_pad(G);                        // [8]
    uint32_t* holds = reinterpret_cast<uint32_t*>(ctl + 8);      // [E][ns] ranks that hold the expert

    for (int i = tid; i < G * Lp; i += nthreads) {
        a.p2l[rank0 * Lp + i] = -1;
        if (a.physical_loads != nullptr) a.physical_loads[rank0 * Lp + i] = 0;
    }
    for (int i = tid; i < E * D; i += nthreads) {
        const int64_t idx = static_cast<int64_t>(log0) * D + i;
        a.l2p[idx] = -1;
        a.quota[idx] = 0;
        a.quota_prefix[idx] = 0;
        a.rank_quota_prefix[idx] = 0;
    }
    __syncthreads();
    for (int e = tid; e < E; e += nthreads) {
        const int l = log0 + e;
        loads[e] = __ldcg(a.global_loads + l);
        cnt[e] = 1;
        placed[e] = 1;
        score[e] = static_cast<double>(loads[e]);
        const int phys = (rank0 + e / M) * Lp + e % M;
        a.p2l[phys] = l;
        a.l2p[static_cast<int64_t>(l) * D] = phys;
        for (int w = 0; w < ns; ++w) holds[e * ns + w] = 0;
        holds[e * ns + ((e / M) >> 5)] = 1u << ((e / M) & 31);
    }
    __syncthreads();
    const bool search = R > 0 && G > 1;
    if (warp == 0 && search) {
        // 1. grant the slots
        double total = 0.0;
        for (int e = lane; e < E; e += kWarp) total = __dadd_rn(total, static_cast<double>(loads[e]));  // integers: exact in any order
        for (int off = 16; off > 0; off >>= 1) total = __dadd_rn(total, __shfl_xor_sync(kFullMask, total, off));
        const double mean_per_slot = total > 0.0 ? __ddiv_rn(total, static_cast<double>(G * M)) : 0.0;
        const double stop_at = __dmul_rn(mean_per_slot, static_cast<double>(a.balance_threshold));
        for (int slot = 0; slot < G * R; ++slot) {
            double best = -1.0;
            int best_e = -1;
            for (int e = lane; e < E; e += kWarp) {
                if (cnt[e] - 1 >= G - 1) continue;
                if (score[e] > best) {  // ascending scan: equal scores keep the lower id
                    best = score[e];
                    best_e = e;
                }
            }
            for (int off = 16; off > 0; off >>= 1) {
                const double ob = __shfl_xor_sync(kFullMask, best, off);
                const int oe = __shfl_xor_sync(kFullMask, best_e, off);
                if (oe >= 0 && (best_e < 0 || ob > best || (ob == best && oe < best_e))) {
                    best = ob;
                    best_e = oe;
                }
            }
            if (a.balance_threshold > 1.0f && mean_per_slot > 0.0 && best <= stop_at) break;
            if (best_e < 0) break;
            if (lane == 0) {
                cnt[best_e] += 1;
                score[best_e] = __ddiv_rn(static_cast<double>(loads[best_e]), static_cast<double>(cnt[best_e]));
            }
            __syncwarp();
        }
        // the extra instances, expert after expert
        int n = 0;
        for (int e0 = 0; e0 < E; e0 += kWarp) {
            const int e = e0 + lane;
            const int extra = e < E ? cnt[e] - 1 : 0;
            int incl = extra;
            for (int off = 1; off < kWarp; off <<= 1) {
                const int t = __shfl_up_sync(kFullMask, incl, off);
                if (lane >= off) incl += t;
            }
            for (int j = 0; j < extra; ++j) {
                const int o = n + incl - extra + j;
                if (o < kMaxExportsPerDomain) {
                    xid[o] = e;
                    xkey[o] = score[e];
                }
            }
            n += __shfl_sync(kFullMask, incl, kWarp - 1);
        }
        if (lane == 0) ctl[0] = n < kMaxExportsPerDomain ? n : kMaxExportsPerDomain;
    }
    __syncthreads();
    if (search) {
        // order the extras: larger load per instance first, then the lower expert; instances of one expert are
        // identical, their mutual order is their list order. Rank by counting, all threads.
        const int n = ctl[0];
        for (int i = tid; i < n; i += nthreads) {
            const double k = xkey[i];
            const int e = xid[i];
            int pos = 0;
            for (int j = 0; j < n; ++j) {
                const double kj = xkey[j];
                const int ej = xid[j];
                pos += (kj > k || (kj == k && (ej < e || (ej == e && j < i)))) ? 1 : 0;
            }
            xkey_sorted[pos] = k;
            xid_sorted[pos] = e;
        }
        for (int r = tid; r < G; r += nthreads) {
            double sum = 0.0;
            for (int m = 0; m < M; ++m) sum = __dadd_rn(sum, score[r * M + m]);  // load / instances, masters in order
            rank_load[r] = sum;
            used[r] = 0;
        }
    }
    __syncthreads();
    if (warp == 0 && search) {
        // 2. place them
        const int n = ctl[0];
        for (int i = 0; i < n; ++i) {
            const int e = xid_sorted[i];
            double best = 0.0;
            int target = -1;
            for (int r = lane; r < G; r += kWarp) {
                if (used[r] >= R || ((holds[e * ns + (r >> 5)] >> (r & 31)) & 1u)) continue;
                if (target < 0 || rank_load[r] < best) {  // ascending scan: equal loads keep the lower rank
                    best = rank_load[r];
                    target = r;
                }
            }
            for (int off = 16; off > 0; off >>= 1) {
                const double ob = __shfl_xor_sync(kFullMask, best, off);
                const int ot = __shfl_xor_sync(kFullMask, target, off);
                if (ot >= 0 && (target < 0 || ob < best || (ob == best && ot < target))) {
                    best = ob;
                    target = ot;
                }
            }
            if (lane == 0) {
                if (target < 0) {
                    cnt[e] -= 1;
                } else {
                    const int l = log0 + e;
                    const int phys = (rank0 + target) * Lp + M + used[target];
                    const int slot = placed[e];
                    if (slot < D) {
                        a.p2l[phys] = l;
                        a.l2p[static_cast<int64_t>(l) * D + slot] = phys;
                    } else {
                        report_error(status, UEP_DEV_BAD_PLAN, l);
                    }
                    placed[e] = slot + 1;
                    rank_load[target] = __dadd_rn(rank_load[target], xkey_sorted[i]);
                    used[target] += 1;
                    holds[e * ns + (target >> 5)] |= 1u << (target & 31);
                }
            }
            __syncwarp();
        }
    }
    __syncthreads();
    for (int e = tid; e < E; e += nthreads) a.lcnts[log0 + e] = cnt[e];
    __syncthreads();
}
__device__ __noinline__ void legacy_solve_apart(const SolveArgs& a, int domain, char* smem_raw, DeviceStatus* status) {
    legacy_solve(a, domain, smem_raw, status);
}

}  // namespace uep
