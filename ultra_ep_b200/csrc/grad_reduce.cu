// Kernel 4 — replica Wgrad reduce: for every local master that has replicas,
//     master = ((master + g_1) + g_2) + ...      (fp32, replicas in plan slot order)
// where g_j is read from the peer that hosts replica j, and every consumed replica region
// is overwritten with zeros. The order is fixed, so the result is bit-exact and equal to
// the reference's deterministic kernel (csrc/kernels/grad_reduce.cu:289-394 of the
// reference; task order :41-69).
//
// The reference builds a task list with a single-thread kernel, then per tile loads one
// replica sub-tile at a time through a single shared-memory buffer (load, wait, add, zero
// with per-thread stores, repeat). Here:
//   * no task list: every CTA derives the pull list from the plan rows with a block scan;
//   * a replica region consumed from another device is not zeroed over the link. Pulling 75 MB and pushing 75 MB of
//     zeros back at the same time measured 450 GB/s against 660 GB/s for the pull alone (the link
//     is full duplex, but one kernel reading from a peer and writing to it through the same SMs
//     did not get both directions at full rate). Instead the rank that HOSTS a replica
//     zeroes it in its own memory: the master's launch reports its progress in 16 segments
//     (a counter per segment that every CTA bumps when it has consumed its items of the segment;
//     the CTA that completes a segment stores "epoch, segments done" into a flag word on every
//     rank it pulls from), and the host rank's launch clears each segment of each used slot as
//     soon as its flag allows, from a warp of its own that runs beside that launch's pulls (bulk
//     stores from a zero tile into local memory). A replica that lies on a rank of the same launch
//     needs none of that: the CTA that pulled a tile clears it;
//   * roles are split. Two producer warps (one lane each) only issue bulk loads: one feeds the
//     ring of replica tiles, the other the ring of master tiles. Eight
//     consumer warps wait on a stage's "full" mbarrier, add it into accumulators in registers
//     (16 floats per thread per tile) and arrive on its "empty" mbarrier: there is no CTA-wide
//     barrier per stage;
//   * two rings of 16 KiB stages: nine for the REMOTE replica tiles (144 KiB in flight per CTA,
//     6 MB over the default 42 CTAs: the bandwidth-delay product of NVLink reads under load is
//     several MB) and three for the local master tiles. In one common ring a master tile would
//     hold a stage as long as a remote tile does, and with one replica per master half of the
//     ring would be taken away from the remote loads;
//   * tiles are interleaved over masters so that concurrent CTAs pull from different peers; they go
//     expert by expert where all replicas lie in this device's memory, and long streams of those
//     are handed out as CTAs ask for more.
// The CTA budget (SMs used while the backward pass runs next to it) is the caller's knob
// (grad_reduce_num_sms); each CTA holds about 225 KB of shared memory (twelve stages and the zero tile are 200 KiB).

#include <climits>

#include "internal.h"

namespace uep {

namespace {

constexpr int kReduceConsumers = 256;
constexpr int kReduceThreads = kReduceConsumers + 128;  // eight consumer warps, two producer warps (replica ring, master ring),
                                                        // one clearing warp, one reporting warp
constexpr int kReduceZeroBytes = 8192;                 // zero tile the clearing warp stores from
constexpr int kReduceTileElems = 4096;                 // 16 KiB
constexpr int kReduceTileBytes = kReduceTileElems * 4;
constexpr int kReduceStages = 9;                       // ring of remote replica tiles
constexpr int kMasterStages = 3;                       // ring of local master tiles
constexpr int kReduceVecPerThread = kReduceTileElems / 4 / kReduceConsumers;  // float4 per thread per tile
constexpr int kMaxPulls = kMaxExportsPerDomain;
// Items handed out as CTAs ask for them, in runs: a CTA keeps those that it took, for the clearing, at most so many; half as many is its
// even share.
constexpr int kMaxRuns = 1024, kLeastRun = 2, kRunsAhead = 2;
constexpr int kHandOutItems = 64;    // of a CTA's even share, at least
constexpr int kHandOutTiles = 2048;  // of an expert, at least
constexpr int kItemRing = 32;  // items between the thread that takes them and the warps that add them up: at most the stages of both rings and two
static_assert(kItemRing >= kReduceStages + kMasterStages + 4, "an item is not overwritten while it is looked up");
constexpr int kMaxOwned = 64;  // used replica slots of the hosted ranks (a lane of a warp asks for two)

struct ReduceShared {
    int n_active, total_reps, vector_ok;
    volatile int error;
    int n_owned;
    volatile long long done_items;                 // items of this CTA whose replica tiles have all been consumed
    volatile int pull_finished;                    // the pull phase of this CTA is over (all items, or given up)
    int2 items[kItemRing];                         // handed out: {active, tile} of the k-th item of this CTA at k mod its size; active -1 behind the last one
    volatile int items_ready;                      // how many of them there are so far
    int runs[kMaxRuns];                            // the first items of the runs that this CTA took
    int n_hosted;                                  // replicas that lie on ranks of this launch
    int n_away;                                    // replicas on other devices
    unsigned long long epoch;
    int w_a[kReduceThreads / 32], w_r[kReduceThreads / 32];
    unsigned pull_mask[kMaxLocalRanks][3];         // per hosted rank: ranks on other devices it pulls replica gradients from
    float* own_base[kMaxOwned];                    // used local replica slots: base of the slot ...
    const uint64_t* own_flag[kMaxOwned];           // ... and the progress word its master's rank writes
    short rep_start[kMaxExpertsPerDomain + 1];
    float* rep_base[kMaxPulls];                    // replica slot base in the peer's grad buffer (null: skip)
    unsigned char rep_hosted[kMaxPulls];           // 1: that peer is a rank of this launch, so the pulling CTA clears what it read
    float* master[kMaxExpertsPerDomain][2];        // [n_active][fc1, fc2] master gradient base
    __align__(8) uint64_t full[kReduceStages];     // a remote tile has landed in the stage
    __align__(8) uint64_t empty[kReduceStages];    // all eight consumer warps are done with the stage
    __align__(8) uint64_t m_full[kMasterStages];   // the same for the ring of master tiles
    __align__(8) uint64_t m_empty[kMasterStages];
};

struct ReduceItem {
    int active;       // index into active_master
    int shard;        // 0 fc1, 1 fc2
    int64_t offset;   // element offset inside the shard
    int elems;
};

// Where a CTA's items lie, one after another: additions only. The threads that feed the rings have some 700 ns an item, and
// each division by a number that the compiler does not know, or of 64 bits, is a tenth of that. Backward of eight ranks with divisions
// for items and stages and like this: 128 experts of 4.7 M elements 95.6 us and 89.8, of 18.9 M 276 both.
struct ItemCursor {
    int active, tile, active_step, tile_step;
    // item `first`, then every step-th one: expert by expert (expert_tiles each), or (0) in turn over n_active masters
    __device__ __forceinline__ ItemCursor(int first, int step, int n_active, int expert_tiles) {
        const int d = max(expert_tiles > 0 ? expert_tiles : n_active, 1);
        const int q = first / d, r = first - q * d, dq = step / d, dr = step - dq * d;
        const bool whole = expert_tiles > 0;
        active = whole ? q : r;
        tile = whole ? r : q;
        active_step = whole ? dq : dr;
        tile_step = whole ? dr : dq;
    }
    __device__ __forceinline__ void advance(int n_active, int expert_tiles) {
        active += active_step;
        tile += tile_step;
        if (expert_tiles > 0) {
            if (tile >= expert_tiles) {
                tile -= expert_tiles;
                ++active;
            }
        } else if (active >= n_active) {
            active -= n_active;
            ++tile;
        }
    }
    __device__ __forceinline__ ReduceItem item(int64_t fc1_numel, int64_t fc2_numel, int tiles_fc1) const {
        ReduceItem it;
        it.active = active;
        it.shard = tile < tiles_fc1 ? 0 : 1;
        const int t = it.shard == 0 ? tile : tile - tiles_fc1;
        it.offset = static_cast<int64_t>(t) * kReduceTileElems;
        const int64_t left = (it.shard == 0 ? fc1_numel : fc2_numel) - it.offset;
        it.elems = static_cast<int>(left < kReduceTileElems ? left : kReduceTileElems);
        return it;
    }
};

// A place in a ring of kStages and the parity of its next completion.
template <int kStages>
struct RingPlace {
    int stage = 0;
    uint32_t parity = 0;
    __device__ __forceinline__ void advance() {
        if (++stage == kStages) {
            stage = 0;
            parity ^= 1u;
        }
    }
};

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}

// kHandOut: items may be handed out to CTAs as they ask for them. A kernel of its own, because short streams lose by the code for it
// (backward of eight ranks, 20 and 15 items a CTA 46.5 and 47.9 us without it, 46.8 and 48.2 with it there and not taken).
template <bool kHandOut>
__global__ void __launch_bounds__(kReduceThreads, 1) grad_reduce_kernel(ReduceCall call) {
    extern __shared__ __align__(128) char smem_raw[];  // kReduceStages replica tiles, kMasterStages master tiles, the zero tile
    __shared__ ReduceShared sm;

    const GroupDev& group = call.group;
    const int M = call.M, R = call.R, D = call.D, Lp = M + R, N = call.N, nlocal = call.nlocal;
    const int tid = threadIdx.x;
    const int64_t fc1 = call.fc1_numel, fc2 = call.fc2_numel, total_numel = fc1 + fc2;
    char* master_ring = smem_raw + kReduceStages * kReduceTileBytes;
    char* zero_tile = master_ring + kMasterStages * kReduceTileBytes;
    DeviceStatus* status0 = group.status[0];
    auto stamp = [&](int slot) {
        if (call.trace != nullptr && tid == 0) call.trace[blockIdx.x * 8 + slot] = global_timer_ns();
    };
    stamp(0);

    // Every global read of the set-up is asked for here, before anything depends on one of them: a master's count, its row of
    // instances (up to eight of them) and its gradients' addresses by a thread each, the owner of a redundant slot, the epoch. One
    // memory round trip then, where the count, each instance, the addresses and the owner came one behind the other.
    const int total_masters = nlocal * M;
    const bool row_cached = D <= 8;
    int pre_reps = 0, pre_row[7], pre_owner = -1;
    uintptr_t pre_grad[2] = {0, 0};
    {
        const bool valid = tid < total_masters;
        const int lr = valid ? tid / M : 0, m = valid ? tid % M : 0, l = group.my_rank[lr] * M + m;
        const PlanPtrs& plan = call.plan[lr];
        if (valid) pre_reps = plan.lcnts[l] - 1;
#pragma unroll
        for (int j = 0; j < 7; ++j) pre_row[j] = valid && row_cached && j < D - 1 ? plan.l2p[static_cast<int64_t>(l) * D + 1 + j] : -1;
        if (valid) {
            pre_grad[0] = static_cast<uintptr_t>(call.fc1_grad_ptrs[lr][m]);
            pre_grad[1] = static_cast<uintptr_t>(call.fc2_grad_ptrs[lr][m]);
        }
        if (tid < nlocal * R && nlocal * R <= kMaxOwned) pre_owner = call.plan[tid / R].p2l[group.my_rank[tid / R] * Lp + M + tid % R];
    }
    unsigned long long pre_epoch = 0;
    if (tid == 0) pre_epoch = *call.reduce_epoch;
    if (tid == 0) {
        sm.n_active = 0;
        sm.total_reps = 0;
        sm.vector_ok = ((fc1 & 3) == 0 && (fc2 & 3) == 0) ? 1 : 0;
        sm.error = 0;
        sm.n_owned = 0;
        sm.n_hosted = 0;
        sm.n_away = 0;
        sm.done_items = 0;
        sm.pull_finished = 0;
        sm.items_ready = 0;
        sm.epoch = pre_epoch + 1;  // ranks hosted together share the first one's counter
        for (int s = 0; s < kReduceStages; ++s) {
            mbar_init(&sm.full[s], 1);
            mbar_init(&sm.empty[s], kReduceConsumers / 32);
        }
        for (int s = 0; s < kMasterStages; ++s) {
            mbar_init(&sm.m_full[s], 1);
            mbar_init(&sm.m_empty[s], kReduceConsumers / 32);
        }
        fence_mbar_init();
    }
    for (int i = tid; i < kMaxLocalRanks * 3; i += blockDim.x) sm.pull_mask[i / 3][i % 3] = 0;
    for (int i = tid; i < kReduceZeroBytes / 4; i += blockDim.x) reinterpret_cast<float*>(zero_tile)[i] = 0.f;
    fence_proxy_async_smem();
    __syncthreads();

    auto hosted_here = [&](int rank) {
        if (call.owners_clear) return false;
        for (int lr = 0; lr < nlocal; ++lr) {
            if (group.my_rank[lr] == rank) return true;
        }
        return false;
    };
    // pull list: masters of the hosted ranks with replicas, and where each replica lives.
    // Hosted ranks pool their tiles over all CTAs of the launch.
    for (int g0 = 0; g0 < total_masters; g0 += blockDim.x) {
        const int gm = g0 + tid;
        const int lr = gm < total_masters ? gm / M : 0;
        const int m = gm < total_masters ? gm % M : 0;
        const PlanPtrs& plan = call.plan[lr];
        const int me = group.my_rank[lr];
        int reps = 0;
        if (gm < total_masters) {
            reps = g0 == 0 ? pre_reps : plan.lcnts[me * M + m] - 1;
            reps = reps < 0 ? 0 : (reps > D - 1 ? D - 1 : reps);
        }
        const int act = reps > 0 ? 1 : 0;
        int a_incl = act, r_incl = reps;
        const int lane = tid & 31, warp = tid >> 5;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int oa = __shfl_up_sync(kFullMask, a_incl, d), orr = __shfl_up_sync(kFullMask, r_incl, d);
            if (lane >= d) {
                a_incl += oa;
                r_incl += orr;
            }
        }
        if (lane == 31) {
            sm.w_a[warp] = a_incl;
            sm.w_r[warp] = r_incl;
        }
        __syncthreads();
        int a_off = sm.n_active, r_off = sm.total_reps;
        for (int w = 0; w < warp; ++w) {
            a_off += sm.w_a[w];
            r_off += sm.w_r[w];
        }
        if (act) {
            const int ai = a_off + a_incl - 1;
            const int rs = r_off + r_incl - reps;
            sm.rep_start[ai] = static_cast<short>(rs);
            const int l = me * M + m;
            auto place = [&](int j, int phys) {
                const int prank = phys / Lp, pslot = phys % Lp - M;
                if (phys < 0 || prank >= N || pslot < 0 || pslot >= R) {
                    report_error(group.status[lr], UEP_DEV_BAD_PLAN, l);
                    sm.rep_base[rs + j] = nullptr;
                } else {
                    const bool hosted = hosted_here(prank);
                    sm.rep_base[rs + j] = group.grad_of(prank) + static_cast<int64_t>(pslot) * total_numel;
                    sm.rep_hosted[rs + j] = hosted ? 1 : 0;
                    if (!hosted) atomicOr(&sm.pull_mask[lr][prank >> 5], 1u << (prank & 31));
                    atomicAdd(hosted ? &sm.n_hosted : &sm.n_away, 1);
                }
            };
            if (g0 == 0 && row_cached) {
#pragma unroll
                for (int j = 0; j < 7; ++j) {
                    if (j < reps && rs + j < kMaxPulls) place(j, pre_row[j]);
                }
            } else {
                for (int j = 0; j < reps && rs + j < kMaxPulls; ++j) place(j, plan.l2p[static_cast<int64_t>(l) * D + 1 + j]);
            }
            const uintptr_t p1 = g0 == 0 ? pre_grad[0] : static_cast<uintptr_t>(call.fc1_grad_ptrs[lr][m]);
            const uintptr_t p2 = g0 == 0 ? pre_grad[1] : static_cast<uintptr_t>(call.fc2_grad_ptrs[lr][m]);
            sm.master[ai][0] = reinterpret_cast<float*>(p1);
            sm.master[ai][1] = reinterpret_cast<float*>(p2);
            if ((p1 & 15u) || (p2 & 15u)) atomicAnd(&sm.vector_ok, 0);
        }
        __syncthreads();
        if (tid == blockDim.x - 1) {
            sm.n_active = a_off + a_incl;
            sm.total_reps = r_off + r_incl;
        }
        __syncthreads();
    }
    if (tid == 0) sm.rep_start[sm.n_active] = static_cast<short>(sm.total_reps < kMaxPulls ? sm.total_reps : kMaxPulls);
    // The used replica slots of the hosted ranks whose master's rank is on another device: this launch clears them once that
    // rank has pulled them.
    {
        const int i = tid;
        const bool in = i < nlocal * R && nlocal * R <= kMaxOwned;
        const int l = pre_owner;
        const bool used = in && l >= 0 && l / M < N && !hosted_here(l / M);
        const unsigned has = __ballot_sync(kFullMask, used);
        const int lane = tid & 31, warp = tid >> 5;
        if (lane == 0) sm.w_a[warp] = __popc(has);
        __syncthreads();
        int f = __popc(has & ((1u << lane) - 1u));
        for (int w = 0; w < warp; ++w) f += sm.w_a[w];
        if (used) {
            const int lr = i / R, me = group.my_rank[lr];
            sm.own_base[f] = group.grad_of(me) + static_cast<int64_t>(i % R) * total_numel;
            sm.own_flag[f] = group.reduce_flags_of(me) + l / M;
        }
        if (tid == 0) {
            int n = 0;
            for (int w = 0; w < kReduceThreads / 32; ++w) n += sm.w_a[w];
            sm.n_owned = n;
        }
    }
    __syncthreads();
    stamp(1);

    const int n_active = sm.n_active;
    const uint64_t epoch = sm.epoch;
    const int tiles_fc1 = static_cast<int>((fc1 + kReduceTileElems - 1) / kReduceTileElems);
    const int tiles_fc2 = static_cast<int>((fc2 + kReduceTileElems - 1) / kReduceTileElems);
    const int tiles_total = tiles_fc1 + tiles_fc2;
    // Items go expert by expert where every replica is in this device's memory: at any time the CTAs of the launch then read
    // and write a contiguous stretch of one expert, which suits the DRAM better than a tile of every expert at once (kernel
    // time 86 and 78 us with 128 experts of 4.7 M elements on eight ranks, 294 and 257 with 18.9 M). Replicas on other devices
    // are interleaved over the masters, so that concurrent CTAs pull from different peers.
    const int expert_tiles = sm.n_away == 0 ? tiles_total : 0;
    const int64_t total_items = static_cast<int64_t>(n_active) * tiles_total;
    const int64_t first = blockIdx.x, step = gridDim.x;
    const int64_t count = first < total_items ? (total_items - first + step - 1) / step : 0;
    // Where all replicas lie in this device's memory, and there are items enough, CTAs take them as they get on: of even shares the median
    // CTA was through after 169 us and the last one after 202, like this after 173 and 176 (128 experts of 18.9 M elements). Backward of
    // eight ranks, even shares and like this (us): 192 items a CTA of 4608 tiles an expert 276 and 259, 140 of 3240 211 and 191, 80 of 2304
    // 146.2 and 144.8; below the lines 60 of 1620 98.7 and 99.3, 1536 tiles 102.0 and 102.7, 20 of 576 48.2 and 48.7, 15 of 384 46.4 and
    // 46.8. (One item at a time 282 for 259, four the same.) Ranks of other devices are told how far each CTA has come in an order that
    // they know: there the shares are fixed.
    const bool handed_out = kHandOut && sm.n_away == 0 && sm.n_owned == 0 && sm.vector_ok != 0 && total_items >= kHandOutItems * step && total_items < 1 << 30;
    int run = kLeastRun;  // items at a time
    if (handed_out && total_items > step * (kLeastRun * kMaxRuns / 2)) {
        run = static_cast<int>((static_cast<unsigned>(total_items) + gridDim.x * (kMaxRuns / 2) - 1) / (gridDim.x * (kMaxRuns / 2)));
    }
    const ItemCursor start(static_cast<int>(first), static_cast<int>(step), n_active, expert_tiles);
    // segment s covers the tiles [seg_end(s-1), seg_end(s)) of an expert; items come tile after tile
    auto seg_end = [&](int s) -> int { return static_cast<int>(static_cast<int64_t>(s + 1) * tiles_total / kReduceSegments); };

    // One thread per CTA reports progress: `done` of this CTA's items are consumed. When the CTA has passed a
    // segment it bumps that segment's counter; the CTA that completes the count tells every rank the launch pulls
    // from, and the one that completes the last segment closes the epoch.
    int seg_next = sm.n_away > 0 ? 0 : kReduceSegments - 1;  // nobody to tell: only the epoch is left to close
    auto report_progress = [&](int64_t done) {
        while (seg_next < kReduceSegments) {
            const int64_t boundary = static_cast<int64_t>(seg_end(seg_next)) * n_active;  // first item index behind the segment
            if (done < count && first + done * step < boundary) break;
            __threadfence();
            int* counters = call.counters;
            if (atomicAdd(&counters[seg_next], 1) == static_cast<int>(gridDim.x) - 1) {
                counters[seg_next] = 0;
                const uint64_t word = epoch * kReduceFlagRadix + static_cast<uint64_t>(seg_next + 1);
                for (int lr = 0; lr < nlocal; ++lr) {
                    if (group.my_rank[lr] == call.withhold_rank) continue;
                    for (int p = 0; p < N; ++p) {
                        if (sm.pull_mask[lr][p >> 5] & (1u << (p & 31))) st_relaxed_sys_u64(group.reduce_flags_of(p) + group.my_rank[lr], word);
                    }
                }
                if (seg_next == kReduceSegments - 1) *call.reduce_epoch = epoch;
            }
            ++seg_next;
        }
    };

    auto replica_ptr = [&](const ReduceItem& it, int r) -> float* {
        return sm.rep_base[r] + (it.shard == 0 ? 0 : fc1) + it.offset;
    };
    auto master_ptr = [&](const ReduceItem& it) -> float* { return sm.master[it.active][it.shard] + it.offset; };

    // One thread, 16-byte aligned. The zeros stay in L2 like any other line: what accumulates into a slot next finds some of
    // them there (replicas of 8 MB each 74 us for reduce and accumulation with the zeros first to leave, 65 like this; of 19 MB
    // 154 and 150, of 75 MB 527 and 525; the reduce alone the same either way).
    auto clear_tile = [&](float* dst, int elems) {
        const uint32_t bytes = static_cast<uint32_t>(elems) * 4u;
        for (uint32_t o = 0; o < bytes; o += kReduceZeroBytes) {
            bulk_store(reinterpret_cast<char*>(dst) + o, zero_tile, bytes - o < kReduceZeroBytes ? bytes - o : kReduceZeroBytes);
        }
        bulk_commit();
    };

    // ---- clearing warp: the used replica slots hosted here, segment by segment as their master's rank releases
    //      them; runs beside the pulls of this CTA (every CTA of the launch takes every gridDim-th tile) ----------
    if (handed_out && tid >= kReduceConsumers + 64) {
        // nothing to report and nothing to wait for: the thread that takes items closes the epoch, and clears
    } else if (tid >= kReduceConsumers + 96) {
        // ---- reporting warp: keeps the atomics and the flag stores of the progress report off the threads that
        //      feed the rings (each costs a round trip to memory) -----------------------------------------------
        if (tid == kReduceConsumers + 96) {
            // waits for threads of its own CTA only, whose waits are all bounded; bounded itself all the same
            const uint64_t t_begin = global_timer_ns();
            while (true) {
                const int fin = sm.pull_finished;
                const long long done = fin || sm.n_away == 0 ? static_cast<long long>(count) : sm.done_items;
                report_progress(done);
                if (fin || seg_next >= kReduceSegments) break;
                if (global_timer_ns() - t_begin > 4 * call.timeout_ns) {
                    report_error(status0, UEP_DEV_TIMEOUT_COPY, blockIdx.x);
                    break;
                }
                __nanosleep(200);
            }
            report_progress(count);  // whatever happened, the counter of every segment sees this CTA exactly once
        }
    } else if (tid >= kReduceConsumers + 64) {
        const int lane = tid & 31;
        const int n_owned = sm.n_owned;
        const bool vec_zero = ((fc1 & 3) == 0) && ((fc2 & 3) == 0);
        // Every slot at its own pace: whatever its master's rank has released since the last look, so that what holds one rank up,
        // or ends it, holds back that rank's slots only. One lane asks for two slots: a look at all of them costs one round
        // trip. (Slot by slot, the last segment of the first slot held the clearing of all the others back until the pulls were
        // over: backward of eight hosted ranks that clear as ranks of other devices do, 128 experts of 4.7 M elements, 189 us
        // against 143. Segment by segment over all slots, the slowest rank held them back; where all keep the same pace it
        // takes as long as this, the reduce alone 96.1 and 97.2 us, with experts of 18.9 M 267 and 264.)
        auto clear_segment = [&](int u, int sg) {
            float* base = sm.own_base[u];
            const int t0 = sg == 0 ? 0 : seg_end(sg - 1), t1 = seg_end(sg);
            for (int t = t0 + static_cast<int>(blockIdx.x); t < t1; t += static_cast<int>(gridDim.x)) {
                const bool in1 = t < tiles_fc1;
                const int64_t off = in1 ? static_cast<int64_t>(t) * kReduceTileElems
                                        : fc1 + static_cast<int64_t>(t - tiles_fc1) * kReduceTileElems;
                const int64_t left = (in1 ? fc1 : total_numel) - off;
                const int elems = static_cast<int>(left < kReduceTileElems ? left : kReduceTileElems);
                float* dst = base + off;
                if (vec_zero) {
                    if (lane == 0) clear_tile(dst, elems);
                } else {
                    for (int i = lane; i < elems; i += 32) dst[i] = 0.f;
                }
            }
        };
        constexpr int kSlotsPerLane = kMaxOwned / kWarp;
        int cleared[kSlotsPerLane];  // segments done with, of slot 32 * h + lane; all of them where there is no slot
        uint64_t since[kSlotsPerLane];  // when that last changed
#pragma unroll
        for (int h = 0; h < kSlotsPerLane; ++h) {
            cleared[h] = kWarp * h + lane < n_owned ? 0 : kReduceSegments;
            since[h] = global_timer_ns();
        }
        while (true) {
            bool open = false;
#pragma unroll
            for (int h = 0; h < kSlotsPerLane; ++h) open = open || cleared[h] < kReduceSegments;
            if (!__any_sync(kFullMask, open)) break;
            int released[kSlotsPerLane];
#pragma unroll
            for (int h = 0; h < kSlotsPerLane; ++h) {
                released[h] = cleared[h];
                if (cleared[h] < kReduceSegments) {
                    const int64_t told = static_cast<int64_t>(ld_relaxed_sys_u64(sm.own_flag[kWarp * h + lane]) - epoch * kReduceFlagRadix);
                    if (told > cleared[h]) released[h] = static_cast<int>(told < kReduceSegments ? told : kReduceSegments);
                }
            }
            unsigned any_news = 0;
#pragma unroll
            for (int h = 0; h < kSlotsPerLane; ++h) {
                const unsigned news = __ballot_sync(kFullMask, released[h] > cleared[h]);
                any_news |= news;
                for (unsigned rest = news; rest != 0; rest &= rest - 1) {
                    const int src = __ffs(rest) - 1;
                    const int s0 = __shfl_sync(kFullMask, cleared[h], src), s1 = __shfl_sync(kFullMask, released[h], src);
                    for (int sg = s0; sg < s1; ++sg) clear_segment(kWarp * h + src, sg);
                }
                if (released[h] > cleared[h]) {
                    cleared[h] = released[h];
                    since[h] = global_timer_ns();
                }
            }
            if (any_news != 0) continue;
            const uint64_t now = global_timer_ns();
#pragma unroll
            for (int h = 0; h < kSlotsPerLane; ++h) {
                if (cleared[h] < kReduceSegments && now - since[h] > call.timeout_ns) {
                    report_error(status0, UEP_DEV_TIMEOUT_SYNC, kWarp * h + lane);
                    cleared[h] = kReduceSegments;  // given up: the slot keeps what it holds
                }
            }
            __nanosleep(100);
        }
        if (lane == 0) bulk_wait_all<0>();
    } else if (!sm.vector_ok) {
        // element-wise path for sizes / pointers that are not multiples of 16 bytes
        ItemCursor cursor = start;
        for (int64_t k = 0; k < count; ++k, cursor.advance(n_active, expert_tiles)) {
            const ReduceItem it = cursor.item(fc1, fc2, tiles_fc1);
            float* mp = master_ptr(it);
            const int r0 = sm.rep_start[it.active], r1 = sm.rep_start[it.active + 1];
            for (int i = tid; i < it.elems; i += kReduceConsumers + 64) {  // every thread but the clearing and reporting warps
                float acc = mp[i];
                for (int r = r0; r < r1; ++r) {
                    if (sm.rep_base[r] == nullptr) continue;
                    float* from = replica_ptr(it, r) + i;
                    acc = __fadd_rn(acc, __ldcg(from));
                    if (sm.rep_hosted[r]) *from = 0.f;
                }
                mp[i] = acc;
            }
        }
        // every thread's loads of the replicas have returned (the clearing and reporting warps are not part of this path: named barrier)
        asm volatile("bar.sync 1, %0;" ::"r"(kReduceConsumers + 64) : "memory");
        if (tid == 0) sm.pull_finished = 1;
    } else if (tid >= kReduceConsumers + 32) {
        // ---- producer of the master ring: one load per item, in item order -----------------------
        if (tid == kReduceConsumers + 32) {
            int64_t m_issued = 0;
            ItemCursor cursor = start;
            RingPlace<kMasterStages> place;
            for (; handed_out || m_issued < count; ++m_issued, place.advance(), cursor.advance(n_active, expert_tiles)) {
                const int s = place.stage;
                if (handed_out) {
                    const uint64_t t_begin = global_timer_ns();
                    bool there = sm.items_ready > m_issued;
                    while (!there) {  // (the thread that takes them ends with a -1, whatever happens)
                        if (global_timer_ns() - t_begin > 2 * call.timeout_ns) break;
                        there = sm.items_ready > m_issued;
                    }
                    __threadfence_block();
                    const int2 next = there ? sm.items[m_issued % kItemRing] : make_int2(-1, 0);
                    cursor.active = next.x;
                    cursor.tile = next.y;
                }
                const bool end = cursor.active < 0;
                ReduceItem it{};
                const float* from = nullptr;
                if (!end) {
                    it = cursor.item(fc1, fc2, tiles_fc1);
                    from = master_ptr(it);
                }
                if (m_issued >= kMasterStages) {  // the stage's previous tile has been read by every consumer warp
                    if (!mbar_wait(&sm.m_empty[s], place.parity ^ 1u, sm.error ? 0 : call.timeout_ns)) {
                        sm.error = 1;
                        break;
                    }
                }
                if (end) {  // the consumers find it where an item would be
                    sm.items[m_issued % kItemRing] = make_int2(-1, 0);
                    mbar_arrive(&sm.m_full[s]);
                    break;
                }
                const uint32_t bytes = static_cast<uint32_t>(it.elems) * 4u;
                mbar_expect_tx(&sm.m_full[s], bytes);
                bulk_load(master_ring + s * kReduceTileBytes, from, bytes, &sm.m_full[s]);
            }
            if (sm.error) {  // loads that never completed must not find the shared memory released under them
                for (int64_t j = m_issued > kMasterStages ? m_issued - kMasterStages : 0; j < m_issued; ++j) {
                    mbar_wait(&sm.m_full[j % kMasterStages], static_cast<uint32_t>((j / kMasterStages) & 1), call.timeout_ns);
                }
            }
        }
    } else if (tid >= kReduceConsumers) {
        // ---- producer of the replica ring: every remote load; reports this CTA's progress ------------
        if (tid == kReduceConsumers) {
            // (item, replica) pairs in the order the consumers take them
            int64_t k_rep = 0;
            int r_issue = -1, r_issue_end = -1;
            ReduceItem it_rep{};
            ItemCursor cursor = start;
            RingPlace<kReduceStages> fill, drain;
            bool last_of_item = false;
            // Handed out: the first run is the CTA's own number, the next ones are asked for ahead. Items without a replica to add (a plan with
            // bad entries) stay as they are.
            int taken = 0, left = 0, published = 0, asked = 1;
            int ahead[kRunsAhead];  // runs asked for
            auto ask = [&]() { return handed_out && asked++ < kMaxRuns ? static_cast<int>(gridDim.x) + atomicAdd(call.counters, 1) : INT_MAX; };
            ahead[0] = static_cast<int>(blockIdx.x);
#pragma unroll
            for (int i = 1; i < kRunsAhead; ++i) ahead[i] = ask();
            auto publish = [&](int active, int tile) {
                sm.items[published % kItemRing] = make_int2(active, tile);
                __threadfence_block();
                sm.items_ready = ++published;
            };
            // The next item of this CTA into it_rep; false: none.
            auto next_item = [&]() -> bool {
                if (!handed_out) {
                    if (k_rep >= count) return false;
                    it_rep = cursor.item(fc1, fc2, tiles_fc1);
                    cursor.advance(n_active, expert_tiles);
                    return true;
                }
                while (true) {
                    if (left > 0) {
                        if (++cursor.tile == expert_tiles) {
                            cursor.tile = 0;
                            ++cursor.active;
                        }
                    } else {
                        const int64_t at = static_cast<int64_t>(ahead[0]) * run;
                        if (at >= total_items) return false;
                        cursor.active = static_cast<int>(at) / expert_tiles;
                        cursor.tile = static_cast<int>(at) - cursor.active * expert_tiles;
                        left = min(run, static_cast<int>(total_items - at));
                        sm.runs[taken++] = static_cast<int>(at);
#pragma unroll
                        for (int i = 0; i + 1 < kRunsAhead; ++i) ahead[i] = ahead[i + 1];
                        ahead[kRunsAhead - 1] = ask();  // (whoever has twice an even share asks for no more: the others have room for the rest)
                    }
                    --left;
                    bool any = false;
                    for (int r = sm.rep_start[cursor.active]; r < sm.rep_start[cursor.active + 1] && !any; ++r) any = sm.rep_base[r] != nullptr;
                    if (!any) continue;
                    publish(cursor.active, cursor.tile);
                    it_rep = cursor.item(fc1, fc2, tiles_fc1);
                    return true;
                }
            };
            auto next_replica = [&](float*& src, int& elems) -> bool {
                while (true) {
                    if (r_issue < 0) {
                        if (!next_item()) return false;
                        r_issue = sm.rep_start[it_rep.active];
                        r_issue_end = sm.rep_start[it_rep.active + 1];
                    }
                    while (r_issue < r_issue_end && sm.rep_base[r_issue] == nullptr) ++r_issue;
                    if (r_issue >= r_issue_end) {
                        ++k_rep;
                        r_issue = -1;
                        continue;
                    }
                    src = replica_ptr(it_rep, r_issue);
                    elems = it_rep.elems;
                    ++r_issue;
                    int nxt = r_issue;  // is another replica of this item still to come?
                    while (nxt < r_issue_end && sm.rep_base[nxt] == nullptr) ++nxt;
                    last_of_item = nxt >= r_issue_end;
                    return true;
                }
            };
            uint32_t ring_last = 0;  // a bit a stage: the last tile of an item
            int64_t issued = 0, retired = 0, done_items = 0;
            bool more = true;
            while (true) {
                while (more && issued - retired < kReduceStages) {
                    float* src = nullptr;
                    int elems = 0;
                    more = next_replica(src, elems);
                    if (!more) break;
                    const int s = fill.stage;
                    fill.advance();
                    ring_last = last_of_item ? ring_last | 1u << s : ring_last & ~(1u << s);
                    const uint32_t bytes = static_cast<uint32_t>(elems) * 4u;
                    mbar_expect_tx(&sm.full[s], bytes);
                    bulk_load(smem_raw + s * kReduceTileBytes, src, bytes, &sm.full[s]);
                    ++issued;
                }
                if (retired == issued) break;  // every replica tile has been consumed
                // the oldest stage: every consumer warp has read it
                const int s = drain.stage;
                if (!mbar_wait(&sm.empty[s], drain.parity, sm.error ? 0 : call.timeout_ns)) {
                    sm.error = 1;
                    break;
                }
                ++retired;
                drain.advance();
                if (ring_last >> s & 1u) sm.done_items = ++done_items;  // the reporting warp turns this into segment counts
            }
            if (sm.error) {
                report_error(status0, UEP_DEV_TIMEOUT_COPY, static_cast<int>(retired));
                for (int64_t j = issued > kReduceStages ? issued - kReduceStages : 0; j < issued; ++j) {
                    mbar_wait(&sm.full[j % kReduceStages], static_cast<uint32_t>((j / kReduceStages) & 1), call.timeout_ns);
                }
            }
            if (handed_out) {
                publish(-1, 0);
                // When everybody has asked for the last time, the counters go back and the epoch is closed. (The fence: what was
                // asked for ahead and never looked at must have been counted before.)
                __threadfence();
                if (atomicAdd(&call.counters[kReduceSegments - 1], 1) == static_cast<int>(gridDim.x) - 1) {
                    __threadfence();
                    call.counters[0] = 0;
                    call.counters[kReduceSegments - 1] = 0;
                    *call.reduce_epoch = epoch;
                }
            }
            sm.pull_finished = 1;
            // Replicas of ranks of this launch: the CTA that pulled a tile clears it, once it has pulled all of its tiles. The
            // clearing is then mostly a phase of writes behind the phase of pulls; clearing a tile as soon as it has been read
            // took 273 us for 257, in batches of 16 items 273, of 64 268 (18.9 M elements; at 4.7 M 78 us each).
            if (sm.n_hosted > 0 && !sm.error) {
                auto clear_item = [&]() {
                    const ReduceItem it = cursor.item(fc1, fc2, tiles_fc1);
                    const int r0 = sm.rep_start[it.active], r1 = sm.rep_start[it.active + 1];
                    for (int r = r0; r < r1; ++r) {
                        if (sm.rep_base[r] != nullptr && sm.rep_hosted[r]) clear_tile(replica_ptr(it, r), it.elems);
                    }
                };
                if (handed_out) {
                    for (int k = 0; k < taken; ++k) {
                        const int at = sm.runs[k];
                        cursor.active = at / expert_tiles;
                        cursor.tile = at - cursor.active * expert_tiles;
                        for (int i = min(run, static_cast<int>(total_items) - at); i > 0; --i) {
                            clear_item();
                            if (++cursor.tile == expert_tiles) {
                                cursor.tile = 0;
                                ++cursor.active;
                            }
                        }
                    }
                } else {
                    cursor = start;
                    for (int64_t k = 0; k < count; ++k, cursor.advance(n_active, expert_tiles)) clear_item();
                }
                bulk_wait_all<0>();
            }
        }
    } else {
        // ---- consumer warps ---------------------------------------------------------------------
        const int lane = tid & 31;
        ItemCursor cursor = start;
        RingPlace<kMasterStages> m_place;
        const uint64_t wait_ns = handed_out ? 2 * call.timeout_ns : call.timeout_ns;
        RingPlace<kReduceStages> place;
        stamp(2);
        for (int64_t k = 0; handed_out || k < count; ++k, m_place.advance(), cursor.advance(n_active, expert_tiles)) {
            ReduceItem it{};
            if (!handed_out) it = cursor.item(fc1, fc2, tiles_fc1);  // beside the wait
            const bool there = mbar_wait(&sm.m_full[m_place.stage], m_place.parity, sm.error ? 0 : wait_ns);
            if (!there) sm.error = 1;  // keep the control flow uniform; the result of this tile is void
            if (handed_out) {  // an item is there before its master's tile is
                const int2 next = __all_sync(kFullMask, there) ? sm.items[k % kItemRing] : make_int2(-1, 0);
                if (next.x < 0) break;
                cursor.active = next.x;
                cursor.tile = next.y;
                it = cursor.item(fc1, fc2, tiles_fc1);
            }
            const int nvec = it.elems >> 2;
            float4 acc[kReduceVecPerThread];
            {
                const int s = m_place.stage;
                const float4* stage = reinterpret_cast<const float4*>(master_ring + s * kReduceTileBytes);
#pragma unroll
                for (int u = 0; u < kReduceVecPerThread; ++u) {
                    const int i = tid + u * kReduceConsumers;
                    acc[u] = i < nvec ? stage[i] : make_float4(0.f, 0.f, 0.f, 0.f);
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&sm.m_empty[s]);
            }
            const int r0 = sm.rep_start[it.active], r1 = sm.rep_start[it.active + 1];
            for (int r = r0; r < r1; ++r) {
                if (sm.rep_base[r] == nullptr) continue;
                const int s = place.stage;
                if (!mbar_wait(&sm.full[s], place.parity, sm.error ? 0 : call.timeout_ns)) {
                    sm.error = 1;
                }
                const float4* stage = reinterpret_cast<const float4*>(smem_raw + s * kReduceTileBytes);
#pragma unroll
                for (int u = 0; u < kReduceVecPerThread; ++u) {
                    const int i = tid + u * kReduceConsumers;
                    if (i < nvec) {
                        const float4 v = stage[i];
                        acc[u].x = __fadd_rn(acc[u].x, v.x); acc[u].y = __fadd_rn(acc[u].y, v.y);
                        acc[u].z = __fadd_rn(acc[u].z, v.z); acc[u].w = __fadd_rn(acc[u].w, v.w);
                    }
                }
                place.advance();
                __syncwarp();
                if (lane == 0) mbar_arrive(&sm.empty[s]);  // this warp no longer reads the stage
            }
            float4* mp = reinterpret_cast<float4*>(master_ptr(it));
#pragma unroll
            for (int u = 0; u < kReduceVecPerThread; ++u) {
                const int i = tid + u * kReduceConsumers;
                if (i < nvec) mp[i] = acc[u];
            }
        }
        stamp(3);
    }

    stamp(5);
}

}  // namespace

cudaError_t launch_grad_reduce(const ReduceCall& call, cudaStream_t stream) {
    const dim3 grid(call.nlocal * call.ctas_per_rank), block(kReduceThreads);
    // Whether items may be handed out goes by the size of an expert (how many experts have replicas is not known here) and by the CTAs: six
    // sevenths of the SMs at least. Fewer of them bound the kernel and not the memory, and keep pace with each other, and each
    // run that is asked for is a wait. Reduce of 28.3 M elements an expert, even shares and handed out (us): two ranks, a replica, on 84 CTAs 92
    // and 117, four ranks, four replicas, on 80 317 and 400, on 112 269 and 291, on 128 264 and 258, on 144 272 and 247; three ranks of 42 M on 126
    // 165 and 170.
    const int64_t tiles = (call.fc1_numel + kReduceTileElems - 1) / kReduceTileElems + (call.fc2_numel + kReduceTileElems - 1) / kReduceTileElems;
    const bool hand_out = call.nlocal == call.N && !call.owners_clear && tiles >= kHandOutTiles && static_cast<int>(grid.x) * 7 >= device_sm_count() * 6;
    void (*const kernel)(ReduceCall) = hand_out ? grad_reduce_kernel<true> : grad_reduce_kernel<false>;
    const size_t smem = static_cast<size_t>(kReduceStages + kMasterStages) * kReduceTileBytes + kReduceZeroBytes;
    cudaError_t e = allow_smem(reinterpret_cast<const void*>(kernel), smem);
    if (e != cudaSuccess) return e;
    if (call.nlocal * call.R > kMaxOwned) return cudaErrorInvalidValue;  // more replica slots per launch than the kernel's table holds
    count_launch();
    if (call.nlocal > 1 && call.owners_clear) {
        // hosted ranks clear their slots behind other hosted ranks' pulls inside this one launch: the CTAs that
        // wait and the CTAs they wait for must be resident together. (Else no CTA waits for another one of its launch.)
        ReduceCall copy = call;
        void* args[] = {&copy};
        return cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(kernel), grid, block, args, smem, stream);
    }
    kernel<<<grid, block, smem, stream>>>(call);
    return cudaGetLastError();
}

}  // namespace uep
