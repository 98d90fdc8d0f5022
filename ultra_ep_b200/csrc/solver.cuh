// Placement solver: per-expert token counts -> hot-expert replication plan, for one
// NVLink domain, executed by one CTA (>= 4 warps).
//
// Results are bit-identical to the reference solver
// (csrc/kernels/placement.cu:788-1482 of the reference): same fp32 threshold
// arithmetic, same tie-breaks, same probe schedule of the threshold search, same
// largest-remainder splits. The execution is different:
//   * the ranks with slack are kept sorted in the lanes of a warp (1-3 per lane), and one step
//     makes all the exports of an expert;
//   * an expert is drained once, from its one home rank, so a build keeps no occupancy table
//     and no exported sums: a source's masters sit in the lanes, and the walk over the sources
//     ends at the first one below the threshold;
//   * the three builds of the fast path and the capacity pre-check run side by side on four
//     warps (the serial search takes the first that is feasible), while the other warps clear
//     the outputs;
//   * each rank's masters are ranked by counting instead of a serial insertion sort;
//   * the loads come in shared memory from the caller, and with one domain the per-rank load matrix
//     too where it fits (plan.cu); else the few entries of it that are needed are read through L2.
//     Without the matrix shared memory stays under 48 KB at the static limits.
// All of it is latency of one CTA. Kernel time of uep_solve_placement on one B200: 64 ranks x 4 experts x 2 slots 25.3 us
// (39.5 with the outputs cleared first, one build after another and one warp maximum per export), of which the build 14.
#pragma once

#include <climits>

#include "common.cuh"

namespace uep {

struct ExportEntry {
    int expert_local;
    int target_rank_local;
    int quota;
};

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
    int legacy;  // 1: legacy placement (counts-only greedy, round-robin reroute) instead of the quota solver
    unsigned long long* trace;  // optional: 8 globaltimer stamps of the solver phases (tuning aid), or null
};

constexpr int kSolverProbeWarps = 4;

// Control words in shared memory.
enum SolverCtrl {
    kCtlLo = 0, kCtlHi, kCtlStop0, kCtlNumExports = kCtlStop0 + kSolverProbeWarps, kCtlSmallRange,
    kCtlProbe0, kCtlValid0 = kCtlProbe0 + kSolverProbeWarps, kCtlFeasible0 = kCtlValid0 + kSolverProbeWarps,
    kCtlExports0 = kCtlFeasible0 + kSolverProbeWarps, kCtlMultiCount = kCtlExports0 + kSolverProbeWarps, kCtlCount
};
static_assert(kCtlCount <= 32, "control words");

struct SolverSmem {
    int32_t* loads;           // [E]
    int32_t* my_loads;        // [E]
    int32_t* sorted_experts;  // [E]
    int32_t* expert_slot;     // [E]
    int32_t* rank_load;       // [Gp]
    int32_t* source_order;    // [Gp] ranks by load, largest first, ties to the lower one
    int32_t* sink_order;      // [Gp] smallest first, likewise
    int32_t* next_slot;       // [Gp]
    int32_t* export_sum;      // [4][E] of the four warps that build plans
    ExportEntry* plan;        // [4][kMaxExportsPerDomain]
    int* ctrl;                // [kCtlCount]
};

__host__ __device__ inline int solver_ns(int G) { return (G + 31) / 32; }
__host__ __device__ inline int solver_gpad(int G) { return (G + 3) / 4 * 4; }
__host__ __device__ inline size_t solver_smem_bytes(int E, int G) {
    return sizeof(int32_t) * (4 * static_cast<size_t>(E) + 4 * solver_gpad(G) + kSolverProbeWarps * static_cast<size_t>(E)) +
           kSolverProbeWarps * sizeof(ExportEntry) * kMaxExportsPerDomain + sizeof(int) * 32;
}

__device__ inline SolverSmem carve_solver_smem(char* raw, int E, int G) {
    const int gp = solver_gpad(G);
    SolverSmem s;
    int32_t* p = reinterpret_cast<int32_t*>(raw);
    s.loads = p; p += E;
    s.my_loads = p; p += E;
    s.sorted_experts = p; p += E;
    s.expert_slot = p; p += E;
    s.rank_load = p; p += gp;
    s.source_order = p; p += gp;
    s.sink_order = p; p += gp;
    s.next_slot = p; p += gp;
    s.export_sum = p; p += kSolverProbeWarps * E;
    s.plan = reinterpret_cast<ExportEntry*>(p); p += kSolverProbeWarps * 3 * kMaxExportsPerDomain;
    s.ctrl = reinterpret_cast<int*>(p);
    return s;
}

__device__ __forceinline__ int warp_inclusive_scan(int v, int lane) {
#pragma unroll
    for (int off = 1; off < kWarp; off <<= 1) {
        const int t = __shfl_up_sync(kFullMask, v, off);
        if (lane >= off) v += t;
    }
    return v;
}

// Greedy export plan for one threshold, by one warp. Returns feasibility (uniform over
// the warp). Semantics of csrc/kernels/placement.cu:337-667 of the reference.
//
// An expert's exports go to the ranks by slack, largest first, ties to the lower rank, each rank once; every one of them is
// filled up except the last. So the ranks are kept sorted in the lanes (slot 32 s + lane), with inclusive sums of their
// slack, and one step per expert finds all its exports: lane i takes part while the slack in front of it is less than what
// is to be moved and its share passes the floor. The filled ranks leave at the front, and the last one, if slack and
// slots are left, moves back to its place. (One export at a time, a warp maximum each: 325 ns an export.)
// `stop`: raised by a warp whose result makes this build pointless.
template <int NS, bool STORE>
__device__ bool warp_build_plan(const SolverSmem& sm, int32_t* export_sum, ExportEntry* plan, int& num_exports, int thr, int E,
                                int G, int M, int R, int min_tokens, bool allow_zero_master, bool dynamic_floor, int lane,
                                const volatile int* stop = nullptr) {
    num_exports = 0;
    if (STORE) {
        __syncwarp();  // an earlier build of this warp may still be storing its sums
        for (int e = lane; e < E; e += kWarp) export_sum[e] = 0;
        __syncwarp();
    }
    int slack[NS], meta[NS], upto[NS];  // meta: free slots << 8 | rank; upto: slack of this slot and all in front of it
    int order[NS], order_load[NS];      // the sources
    int end = 0;                        // slots with slack are [head, end)
    int local_excess = 0, total_slack = 0;
#pragma unroll
    for (int s = 0; s < NS; ++s) {
        const int i = lane + kWarp * s;
        const int sink = i < G ? sm.sink_order[i] : 0;
        slack[s] = i < G ? max(thr - sm.rank_load[sink], 0) : 0;
        meta[s] = R << 8 | sink;
        order[s] = i < G ? sm.source_order[i] : 0;
        order_load[s] = i < G ? sm.rank_load[order[s]] : thr;
        local_excess += max(order_load[s] - thr, 0);
        end += __popc(__ballot_sync(kFullMask, slack[s] > 0));
        upto[s] = warp_inclusive_scan(slack[s], lane) + total_slack;
        total_slack = __shfl_sync(kFullMask, upto[s], kWarp - 1);
    }
    const int total_excess = warp_sum(local_excess);
    if (total_excess == 0) return true;
    // Every export takes the same from both, so the slack left always covers the excess left.
    if (total_excess > total_slack) return false;

    auto at = [&](const int (&v)[NS], int slot) {
        int x = __shfl_sync(kFullMask, v[0], slot & 31);
#pragma unroll
        for (int s = 1; s < NS; ++s) {
            const int y = __shfl_sync(kFullMask, v[s], slot & 31);
            x = slot >> 5 == s ? y : x;
        }
        return x;
    };
    auto masters = [&](int src, int base, int& e, int& load) {  // 32 of the source's masters, one per lane
        e = base + lane < M ? sm.sorted_experts[src * M + base + lane] : 0;
        load = base + lane < M ? sm.loads[e] : 0;
    };
    int head = 0, gone = 0;  // gone: slack in front of slot `head`, as `upto` counts it
    int src = at(order, 0), src_load = at(order_load, 0), first_e, first_load;
    masters(src, 0, first_e, first_load);
    for (int ord = 0; ord < G; ++ord) {
        int need = src_load - thr;
        if (need <= 0) break;  // sources come by load: no later one is above the threshold
        if (stop != nullptr && __shfl_sync(kFullMask, *stop, 0) != 0) return false;
        const int this_src = src;
        int my_e = first_e, my_load = first_load;
        const int next_ord = min(ord + 1, G - 1);  // fetched while this one is drained
        src = at(order, next_ord);
        src_load = at(order_load, next_ord);
        masters(src, 0, first_e, first_load);
        bool drained = false;  // the masters come by load too: no later one has anything to give
        for (int base = 0; base < M && need > 0 && !drained; base += kWarp) {
            if (base > 0) masters(this_src, base, my_e, my_load);
            const int in_chunk = min(M - base, kWarp);
            for (int pos = 0; pos < in_chunk && need > 0; ++pos) {
                const int load_e = __shfl_sync(kFullMask, my_load, pos);
                const int avail = load_e - ((!allow_zero_master && load_e > 0) ? 1 : 0);
                if (avail <= 0) {
                    drained = true;
                    break;
                }
                const int move = min(need, avail);
                int q[NS], next_slack[NS], next_meta[NS], next_upto[NS];
                int first_out = kWarp * NS;  // the first slot from `head` on that takes nothing
#pragma unroll
                for (int s = NS - 1; s >= 0; --s) {
                    const int slot = lane + kWarp * s;
                    const int before = upto[s] - gone - slack[s];
                    q[s] = min(slack[s], move - before);
                    // dynamic floor: ceil(what is still needed / the ranks that could still take part)
                    const bool enough = dynamic_floor ? static_cast<long long>(q[s]) * (end - slot) >= need - before : q[s] >= min_tokens;
                    const unsigned out = __ballot_sync(kFullMask, slot >= head && !(slot < end && before < move && enough));
                    if (out != 0u) first_out = kWarp * s + __ffs(out) - 1;
                    next_slack[s] = __shfl_down_sync(kFullMask, slack[s], 1);
                    next_meta[s] = __shfl_down_sync(kFullMask, meta[s], 1);
                    next_upto[s] = __shfl_down_sync(kFullMask, upto[s], 1);
                    if (s + 1 < NS) {
                        const int a = __shfl_sync(kFullMask, slack[s + 1 < NS ? s + 1 : s], 0), b = __shfl_sync(kFullMask, meta[s + 1 < NS ? s + 1 : s], 0),
                                  c = __shfl_sync(kFullMask, upto[s + 1 < NS ? s + 1 : s], 0);
                        if (lane == kWarp - 1) {
                            next_slack[s] = a;
                            next_meta[s] = b;
                            next_upto[s] = c;
                        }
                    }
                }
                const int exports = first_out - head;
                if (exports == 0) continue;
                const int last = first_out - 1;
                const int last_upto = at(upto, last), last_meta = at(meta, last);
                const int moved = min(last_upto - gone, move);
                const int rest = last_upto - gone - moved;  // slack that the last rank keeps
                const bool stays = rest > 0 && last_meta >> 8 > 1;
                if (STORE) {
                    if (num_exports + exports > kMaxExportsPerDomain) return false;
                    const int e = __shfl_sync(kFullMask, my_e, pos);
#pragma unroll
                    for (int s = 0; s < NS; ++s) {
                        const int slot = lane + kWarp * s;
                        if (slot >= head && slot < first_out) plan[num_exports + slot - head] = ExportEntry{e, meta[s] & 255, q[s]};
                    }
                    if (lane == 0) export_sum[e] = moved;
                    num_exports += exports;
                }
                int ahead = 0;  // slots that come in front of the last rank now
#pragma unroll
                for (int s = 0; s < NS; ++s) {
                    const int slot = lane + kWarp * s;
                    ahead += __popc(__ballot_sync(kFullMask, slot > last && slot < end && (slack[s] > rest || (slack[s] == rest &&
                                                                                           (meta[s] & 255) < (last_meta & 255)))));
                }
#pragma unroll
                for (int s = 0; s < NS; ++s) {
                    const int slot = lane + kWarp * s;
                    if (stays && slot >= last && slot < last + ahead) {
                        slack[s] = next_slack[s];
                        meta[s] = next_meta[s];
                        upto[s] = next_upto[s] - rest;
                    } else if (stays && slot == last + ahead) {
                        slack[s] = rest;
                        meta[s] = last_meta - 256;
                    }
                }
                head = stays ? last : first_out;
                gone = stays ? gone + moved : last_upto;
                need -= moved;
            }
        }
        if (need > 0) return false;
    }
    return true;
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

// Split of this rank's tokens of one expert over the expert's replicas, as an inclusive
// prefix. Semantics of csrc/kernels/placement.cu:1342-1481 / :669-786 of the reference.
template <int MAXC>
__device__ void build_rank_quota_prefix(const SolveArgs& a, int l_global, int C, int my_load, const int* phys,
                                        const int* q, int Lp, int L) {
    // phys[j] / q[j]: physical id and quota of replica j (j = 0 is the master), handed over from
    // shared memory by the caller so that no plan row has to be read back from global memory.
    const int64_t row = static_cast<int64_t>(l_global) * a.D;
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

// The split of build_rank_quota_prefix for an expert with 2..32 replicas, by one warp: lane j
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
    const int prefix = warp_inclusive_scan(my_alloc, lane);
    if (active) a.rank_quota_prefix[static_cast<int64_t>(l_global) * a.D + lane] = prefix;
}

// Solve one NVLink domain. All threads of the CTA must call it (blockDim.x >= 128,
// multiple of 32). smem_raw must hold solver_smem_bytes(E, G) bytes, 16-byte aligned.
template <int NS>
__device__ void solve_domain(const SolveArgs& a, int domain, char* smem_raw, DeviceStatus* status) {
    const int tid = threadIdx.x, nthreads = blockDim.x;
    const int warp = tid >> 5, lane = tid & 31;
    const int G = a.G, M = a.M, R = a.R, D = a.D;
    const int E = G * M, Lp = M + R, L = a.N * M;
    const int domain_start_rank = domain * G;
    const int domain_start_log = domain_start_rank * M;
    SolverSmem sm = carve_solver_smem(smem_raw, E, G);
    auto stamp = [&](int slot) {
        if (a.trace != nullptr && tid == 0) a.trace[slot] = global_timer_ns();
    };
    stamp(0);

    // Every output of this domain as it is without replicas; run by `n` threads.
    auto clear_outputs = [&](int t, int n) {
        for (int i = t; i < G * Lp; i += n) {
            const int local = i % Lp;
            a.p2l[domain_start_rank * Lp + i] = local < M ? domain_start_log + i / Lp * M + local : -1;
            if (a.physical_loads != nullptr) a.physical_loads[domain_start_rank * Lp + i] = 0;
        }
        const int64_t first = static_cast<int64_t>(domain_start_log) * D;
        auto master = [&](int e) { return (domain_start_rank + e / M) * Lp + e % M; };
        const uintptr_t align = reinterpret_cast<uintptr_t>(a.l2p) | reinterpret_cast<uintptr_t>(a.quota) |
                                reinterpret_cast<uintptr_t>(a.quota_prefix) | reinterpret_cast<uintptr_t>(a.rank_quota_prefix);
        if (D % 4 == 0 && (align & 15u) == 0) {
            const int vecs = D / 4;
            const int4 none = make_int4(0, 0, 0, 0);
            for (int i = t; i < E * vecs; i += n) {
                const int e = i / vecs;
                reinterpret_cast<int4*>(a.l2p + first)[i] = make_int4(i - e * vecs == 0 ? master(e) : -1, -1, -1, -1);
                reinterpret_cast<int4*>(a.quota + first)[i] = none;
                reinterpret_cast<int4*>(a.quota_prefix + first)[i] = none;
                reinterpret_cast<int4*>(a.rank_quota_prefix + first)[i] = none;
            }
        } else {
            for (int i = t; i < E * D; i += n) {
                const int e = i / D;
                a.l2p[first + i] = i - e * D == 0 ? master(e) : -1;
                a.quota[first + i] = 0;
                a.quota_prefix[first + i] = 0;
                a.rank_quota_prefix[first + i] = 0;
            }
        }
    };
    for (int i = tid; i < E; i += nthreads) {
        if (!a.preloaded) {
            sm.loads[i] = __ldcg(a.global_loads + domain_start_log + i);
            sm.my_loads[i] = __ldcg(a.loads_per_rank + static_cast<int64_t>(a.my_rank) * L + domain_start_log + i);
        }
        sm.expert_slot[i] = 1;
    }
    if (tid == 0) sm.ctrl[kCtlNumExports] = 0;
    if (tid < kSolverProbeWarps) sm.ctrl[kCtlStop0 + tid] = 0;
    const bool do_search = (R > 0 && G > 1);
    stamp(1);
    if (!do_search) {
        clear_outputs(tid, nthreads);
    } else {
        __syncthreads();
        for (int r = tid; r < G; r += nthreads) {
            int sum = 0;
#pragma unroll 8
            for (int m = 0; m < M; ++m) sum += sm.loads[r * M + m];
            sm.rank_load[r] = sum;
            sm.next_slot[r] = 0;
        }
        for (int i = tid; i < E; i += nthreads) {  // each rank's masters by load descending, ties to the lower index
            const int base = (i / M) * M;
            const int mine = sm.loads[i];
            int pos = 0;
#pragma unroll 8
            for (int j = base; j < base + M; ++j) {
                const int other = sm.loads[j];
                pos += (other > mine || (other == mine && j < i)) ? 1 : 0;
            }
            sm.sorted_experts[base + pos] = i;
        }
        __syncthreads();
        for (int i = tid; i < G; i += nthreads) {  // the ranks likewise
            const int mine = sm.rank_load[i];
            int above = 0, below = 0, equal = 0;
#pragma unroll 8
            for (int j = 0; j < G; ++j) {
                const int other = sm.rank_load[j];
                above += other > mine ? 1 : 0;
                below += other < mine ? 1 : 0;
                equal += (other == mine && j < i) ? 1 : 0;
            }
            sm.source_order[above + equal] = i;
            sm.sink_order[below + equal] = i;
        }
        if (warp == 0) {
            int total = 0, mx = 0;
            for (int r = lane; r < G; r += kWarp) {
                total += sm.rank_load[r];
                mx = max(mx, sm.rank_load[r]);
            }
            total = warp_sum(total);
            mx = warp_max(mx);
            // fp32, in the reference's order: ceilf((float(total) / G) * bt)
            const float bt = fmaxf(a.balance_threshold, 1.0f);
            const float mean = __fdiv_rn(static_cast<float>(total), static_cast<float>(G));
            const int lo = static_cast<int>(ceilf(__fmul_rn(mean, bt)));
            if (lane == 0) {
                sm.ctrl[kCtlLo] = lo;
                sm.ctrl[kCtlHi] = max(mx, lo);
            }
        }
        __syncthreads();
    }
    stamp(2);
    const bool allow0 = a.allow_zero_master != 0;
    int winner = 0;  // the warp whose plan is taken
    if (do_search) {
        // The serial search is: up to three builds with the dynamic floor at rising thresholds; then one build at the
        // smallest threshold the capacities allow; then the probes below. The first four run at once, one warp each; one that
        // succeeds stops those behind it.
        const int lo0 = sm.ctrl[kCtlLo], hi0 = sm.ctrl[kCtlHi];
        if (warp < kSolverProbeWarps) {
            int thr;
            const volatile int* stop = sm.ctrl + kCtlStop0 + warp;
            const bool fast = warp < kSolverProbeWarps - 1;
            if (fast) {
                const float eps = fmaxf(a.eps, 0.0f);
                thr = max(static_cast<int>(ceilf(__fmul_rn(static_cast<float>(lo0), __fadd_rn(1.0f, eps)))), lo0);
                const int step = max(1, (hi0 + 99) / 100);
                for (int i = 0; i < warp; ++i) thr = min(hi0, thr + step);
            } else {
                int lo = lo0, hi = hi0;
                while (lo < hi && __shfl_sync(kFullMask, *stop, 0) == 0) {  // capacity bisection
                    const int probe = lo + ((hi - lo) >> 1);
                    int ex = 0, sl = 0;
                    for (int r = lane; r < G; r += kWarp) {
                        ex += max(sm.rank_load[r] - probe, 0);
                        sl += max(probe - sm.rank_load[r], 0);
                    }
                    if (warp_sum(ex) <= warp_sum(sl)) hi = probe;
                    else lo = probe + 1;
                }
                thr = lo;
            }
            int n = 0;
            const bool ok = warp_build_plan<NS, true>(sm, sm.export_sum + warp * E, sm.plan + warp * kMaxExportsPerDomain, n, thr, E, G,
                                                      M, R, a.min_tokens, allow0, fast, lane, stop);
            if (ok && lane > warp && lane < kSolverProbeWarps) *(sm.ctrl + kCtlStop0 + lane) = 1;
            if (lane == 0) {
                sm.ctrl[kCtlProbe0 + warp] = thr;
                sm.ctrl[kCtlFeasible0 + warp] = ok ? 1 : 0;
                sm.ctrl[kCtlExports0 + warp] = n;
            }
        } else {
            clear_outputs(tid - kSolverProbeWarps * kWarp, nthreads - kSolverProbeWarps * kWarp);
        }
        if (nthreads == kSolverProbeWarps * kWarp) clear_outputs(tid, nthreads);
        __syncthreads();
        winner = -1;
        for (int w = kSolverProbeWarps - 1; w >= 0; --w) {
            if (sm.ctrl[kCtlFeasible0 + w]) winner = w;
        }
        const int precheck_thr = sm.ctrl[kCtlProbe0 + kSolverProbeWarps - 1];
        const int num_exports = winner >= 0 ? sm.ctrl[kCtlExports0 + winner] : 0;
        __syncthreads();  // everyone has read the four results
        if (winner >= 0) {
            if (tid == 0) sm.ctrl[kCtlNumExports] = num_exports;
        } else {
            if (tid == 0) sm.ctrl[kCtlLo] = min(precheck_thr + 1, hi0);
            winner = 0;
            __syncthreads();
            while (true) {
                if (sm.ctrl[kCtlLo] >= sm.ctrl[kCtlHi]) break;
                __syncthreads();  // everyone has read lo/hi before thread 0 rewrites the probe table
                if (tid == 0) {
                    const int lo = sm.ctrl[kCtlLo], hi = sm.ctrl[kCtlHi];
                    const int range = hi - lo;
                    const int small_range = (range <= kSolverProbeWarps) ? 1 : 0;
                    sm.ctrl[kCtlSmallRange] = small_range;
                    for (int w = 0; w < kSolverProbeWarps; ++w) {
                        if (small_range) {
                            sm.ctrl[kCtlProbe0 + w] = lo + w;
                            sm.ctrl[kCtlValid0 + w] = (lo + w < hi) ? 1 : 0;
                        } else {
                            sm.ctrl[kCtlProbe0 + w] =
                                lo + static_cast<int>((static_cast<long long>(range) * (w + 1)) / (kSolverProbeWarps + 1));
                            sm.ctrl[kCtlValid0 + w] = 1;
                        }
                        sm.ctrl[kCtlFeasible0 + w] = 0;
                    }
                }
                __syncthreads();
                if (warp < kSolverProbeWarps && sm.ctrl[kCtlValid0 + warp]) {
                    int n = 0;
                    const bool ok = warp_build_plan<NS, false>(sm, nullptr, nullptr, n, sm.ctrl[kCtlProbe0 + warp], E, G, M, R,
                                                               a.min_tokens, allow0, false, lane);
                    if (lane == 0) sm.ctrl[kCtlFeasible0 + warp] = ok ? 1 : 0;
                }
                __syncthreads();
                if (tid == 0) {
                    if (sm.ctrl[kCtlSmallRange]) {
                        int best = -1;
                        for (int w = 0; w < kSolverProbeWarps; ++w) {
                            if (sm.ctrl[kCtlValid0 + w] && sm.ctrl[kCtlFeasible0 + w]) {
                                best = sm.ctrl[kCtlProbe0 + w];
                                break;
                            }
                        }
                        if (best >= 0) {
                            sm.ctrl[kCtlLo] = best;
                            sm.ctrl[kCtlHi] = best;
                        } else {
                            sm.ctrl[kCtlLo] = sm.ctrl[kCtlHi];
                        }
                    } else {
                        int first = -1;
                        for (int w = 0; w < kSolverProbeWarps; ++w) {
                            if (sm.ctrl[kCtlFeasible0 + w]) {
                                first = w;
                                break;
                            }
                        }
                        if (first >= 0) {
                            sm.ctrl[kCtlHi] = sm.ctrl[kCtlProbe0 + first];
                            if (first > 0) sm.ctrl[kCtlLo] = sm.ctrl[kCtlProbe0 + first - 1] + 1;
                        } else {
                            sm.ctrl[kCtlLo] = sm.ctrl[kCtlProbe0 + kSolverProbeWarps - 1] + 1;
                        }
                    }
                }
                __syncthreads();
            }
            if (warp == 0) {
                int n = 0;
                const bool ok = warp_build_plan<NS, true>(sm, sm.export_sum, sm.plan, n, sm.ctrl[kCtlLo], E, G, M, R, a.min_tokens,
                                                          allow0, false, lane);
                if (lane == 0) {
                    sm.ctrl[kCtlNumExports] = ok ? n : 0;
                    if (!ok) report_error(status, UEP_DEV_SOLVER_INFEASIBLE, sm.ctrl[kCtlLo]);
                }
            }
        }
    }
    __syncthreads();
    const int32_t* export_sum = sm.export_sum + winner * E;
    ExportEntry* plan = sm.plan + winner * kMaxExportsPerDomain;

    stamp(3);
    // Emit: master quotas, then replicas in plan order. Two tables of the search are free by now
    // and are reused: sorted_experts becomes "first plan entry of this expert" (an expert's
    // exports are consecutive in the plan: they are all made while its one source rank is being
    // drained), and another warp's sums become the list of experts that have replicas.
    int* first_entry = sm.sorted_experts;
    int* multi_list = sm.export_sum + (winner + 1) % kSolverProbeWarps * E;
    for (int e = tid; e < E; e += nthreads) {
        const int64_t row = static_cast<int64_t>(domain_start_log + e) * D;
        const int master_quota = do_search ? (sm.loads[e] - export_sum[e]) : sm.loads[e];
        a.quota[row] = master_quota;
        if (a.physical_loads != nullptr) a.physical_loads[(domain_start_rank + e / M) * Lp + e % M] = master_quota;
    }
    if (tid == 0) sm.ctrl[kCtlMultiCount] = 0;
    __syncthreads();
    if (warp == 0) {
        // 32 plan entries at a time: an entry's replica slot (and its target's redundant slot) is
        // the counter left by the earlier chunks plus the number of lower lanes that name the same
        // expert (the same target), which is exactly the creation order of a serial walk.
        const int n = sm.ctrl[kCtlNumExports];
        for (int base = 0; base < n; base += kWarp) {
            const int k = base + lane;
            const bool active = k < n;
            const unsigned amask = __ballot_sync(kFullMask, active);
            if (active) {
                const ExportEntry entry = plan[k];
                const unsigned same_e = __match_any_sync(amask, entry.expert_local);
                const unsigned same_t = __match_any_sync(amask, entry.target_rank_local);
                const unsigned below = (1u << lane) - 1u;
                const int slot = sm.expert_slot[entry.expert_local] + __popc(same_e & below);
                const int tslot = sm.next_slot[entry.target_rank_local] + __popc(same_t & below);
                __syncwarp(amask);  // every lane has read the counters
                if ((same_e >> lane) == 1u) sm.expert_slot[entry.expert_local] = slot + 1;  // highest lane of its group
                if ((same_t >> lane) == 1u) sm.next_slot[entry.target_rank_local] = tslot + 1;
                if (slot == 1) first_entry[entry.expert_local] = k;
                const int l_global = domain_start_log + entry.expert_local;
                const int64_t row = static_cast<int64_t>(l_global) * D;
                const int phys = (domain_start_rank + entry.target_rank_local) * Lp + M + tslot;
                if (slot >= D || phys >= (domain_start_rank + entry.target_rank_local + 1) * Lp) {
                    report_error(status, UEP_DEV_BAD_PLAN, k);
                } else {
                    a.p2l[phys] = l_global;
                    a.l2p[row + slot] = phys;
                    a.quota[row + slot] = entry.quota;
                    if (a.physical_loads != nullptr) a.physical_loads[phys] = entry.quota;
                    plan[k].target_rank_local = phys;  // from here on the entry carries the physical id
                }
            }
            __syncwarp();
        }
    }
    __syncthreads();
    stamp(4);
    // Counts and prefixes. An expert without replicas keeps all of this rank's tokens (every
    // branch of the split reduces to that), so one thread writes its row; the others go to the
    // warps, one expert per warp at a time.
    for (int e = tid; e < E; e += nthreads) {
        const int l_global = domain_start_log + e;
        const int64_t row = static_cast<int64_t>(l_global) * D;
        const int C = min(sm.expert_slot[e], D);
        a.lcnts[l_global] = C;
        if (C == 1) {
            a.quota_prefix[row] = do_search ? (sm.loads[e] - export_sum[e]) : sm.loads[e];
            a.rank_quota_prefix[row] = sm.my_loads[e];
        } else {
            multi_list[atomicAdd(&sm.ctrl[kCtlMultiCount], 1)] = e;
        }
    }
    __syncthreads();
    const int n_multi = sm.ctrl[kCtlMultiCount];
    // A lane's replica of the warp's next expert, its host's own load already on the way from L2.
    struct Replica {
        int e, C, phys, host, q, own;
    };
    auto fetch = [&](int idx) {
        Replica r{-1, 0, 0, -1 - lane, 0, 0};
        if (idx >= n_multi) return r;
        r.e = multi_list[idx];
        r.C = min(sm.expert_slot[r.e], D);
        if (lane == 0) {
            r.phys = (domain_start_rank + r.e / M) * Lp + r.e % M;
            r.q = sm.loads[r.e] - export_sum[r.e];
        } else if (lane < r.C && r.C <= kWarp) {
            const ExportEntry entry = plan[first_entry[r.e] + lane - 1];
            r.phys = entry.target_rank_local;
            r.q = entry.quota;
        }
        if (lane < r.C && r.C <= kWarp) {
            r.host = r.phys / Lp;
            const int64_t at = static_cast<int64_t>(r.host) * L + domain_start_log + r.e;
            if (a.locality) r.own = a.staged_loads != nullptr ? a.staged_loads[at] : __ldcg(a.loads_per_rank + at);
        }
        return r;
    };
    Replica next = fetch(warp);
    for (int idx = warp; idx < n_multi; idx += nthreads / kWarp) {
        const Replica r = next;
        next = fetch(idx + nthreads / kWarp);
        const int e = r.e, C = r.C;
        const int l_global = domain_start_log + e;
        const int64_t row = static_cast<int64_t>(l_global) * D;
        if (C <= kWarp) {
            const int qp = warp_inclusive_scan(r.q, lane);
            if (lane < C) a.quota_prefix[row + lane] = qp;
            warp_rank_quota_prefix(a, l_global, C, sm.my_loads[e], r.host, r.q, r.own, lane);
        } else if (lane == 0) {  // more than 32 replicas: the serial version
            int phys[kMaxRanksPerDomain], q[kMaxRanksPerDomain];
            phys[0] = r.phys;
            q[0] = r.q;
            int prefix = 0;
            const int first = first_entry[e];
            for (int j = 0; j < C; ++j) {
                if (j > 0) {
                    phys[j] = plan[first + j - 1].target_rank_local;
                    q[j] = plan[first + j - 1].quota;
                }
                prefix += q[j];
                a.quota_prefix[row + j] = prefix;
            }
            build_rank_quota_prefix<kMaxRanksPerDomain>(a, l_global, C, sm.my_loads[e], phys, q, Lp, L);
        }
        __syncwarp();
    }
    __syncthreads();
    stamp(5);
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
    return sizeof(double) * (static_cast<size_t>(E) + 2 * kMaxExportsPerDomain + solver_gpad(G)) +
           sizeof(int32_t) * (3 * static_cast<size_t>(E) + 2 * kMaxExportsPerDomain + solver_gpad(G) + 8) +
           sizeof(uint32_t) * static_cast<size_t>(E) * solver_ns(G);
}

__device__ __noinline__ void legacy_solve_domain(const SolveArgs& a, int domain, char* smem_raw, DeviceStatus* status) {
    const int tid = threadIdx.x, nthreads = blockDim.x, lane = tid & 31, warp = tid >> 5;
    const int G = a.G, M = a.M, R = a.R, D = a.D, E = G * M, Lp = M + R, ns = solver_ns(G);
    const int rank0 = domain * G, log0 = rank0 * M;
    double* score = reinterpret_cast<double*>(smem_raw);        // [E] load per instance
    double* xkey = score + E;                                    // [512] extras: load per instance
    double* xkey_sorted = xkey + kMaxExportsPerDomain;           // [512]
    double* rank_load = xkey_sorted + kMaxExportsPerDomain;      // [Gpad]
    int32_t* loads = reinterpret_cast<int32_t*>(rank_load + solver_gpad(G));  // [E]
    int32_t* cnt = loads + E;                                    // [E] instances
    int32_t* placed = cnt + E;                                   // [E] instances placed so far (incl. master)
    int32_t* xid = placed + E;                                   // [512] extras: expert
    int32_t* xid_sorted = xid + kMaxExportsPerDomain;            // [512]
    int32_t* used = xid_sorted + kMaxExportsPerDomain;           // [Gpad] redundant slots used per rank
    int32_t* ctl = used + solver_gpad(G);                        // [8]
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

__device__ inline void solve_domain_dispatch(const SolveArgs& a, int domain, char* smem_raw, DeviceStatus* status) {
    if (a.legacy) {
        legacy_solve_domain(a, domain, smem_raw, status);
        return;
    }
    const int ns = solver_ns(a.G);
    if (ns == 1) solve_domain<1>(a, domain, smem_raw, status);
    else if (ns == 2) solve_domain<2>(a, domain, smem_raw, status);
    else solve_domain<3>(a, domain, smem_raw, status);
}

}  // namespace uep
