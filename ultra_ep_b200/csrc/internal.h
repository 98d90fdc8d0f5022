// Host-side declarations shared by the kernel translation units and the manager.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <string>

#include "../../include/uep_b200.h"
#include "common.cuh"

namespace uep {

constexpr int kMaxLocalRanks = 8;  // ranks one manager can host on one device (simulated EP)
constexpr int kMaxPeers = kMaxRanksPerDomain;
constexpr int kReduceSegments = 16;  // a replica's gradient is released for zeroing in this many pieces
constexpr unsigned long long kReduceFlagRadix = 64;  // progress word = epoch * radix + segments done

constexpr int kPlanMaxCtas = 32;  // CTAs of one rank in the plan kernel
constexpr int kRehearsalOut = 512;  // words that the rehearsal of a plan writes

// Where the group's buffers are. By value in the kernels' parameters, so that the first load of a kernel is of data and not
// of a pointer to it (each of the two is a miss: the tables were last read a layer ago). Fixed once connected. With a table
// per rank in device memory, and the plan's epoch and weight_sync's first unit waited for before the first load of data, the
// step of eight ranks (8192 tokens, 128 experts, fp8 weights of 19 MB) took 67.2 us, 63.2 like this; plan kernel 19.0 and
// 17.3.
struct GroupDev {
    uint8_t* arena[kMaxPeers];  // of every rank of the group, as the hosted ranks see them (all of them the same)
    int64_t gather, sync_flags, relay_flags, reduce_flags, replica_weight, replica_scale, replica_grad;  // offsets in an arena
    int my_rank[kMaxLocalRanks];
    DeviceStatus* status[kMaxLocalRanks];  // mapped pinned host memory

    // [2][N][Lpad] words, (epoch tag << 32) | token count
    __device__ __forceinline__ uint64_t* gather_of(int rank) const { return reinterpret_cast<uint64_t*>(arena[rank] + gather); }
    // [N], entry [src] = last epoch src finished sending to that rank
    __device__ __forceinline__ uint64_t* sync_flags_of(int rank) const { return reinterpret_cast<uint64_t*>(arena[rank] + sync_flags); }
    // [R][relay_cap], entry [slot][chunk] = epoch in which the master delivered that chunk
    __device__ __forceinline__ uint64_t* relay_flags_of(int rank) const { return reinterpret_cast<uint64_t*>(arena[rank] + relay_flags); }
    // [N], entry [src] = epoch * 64 + segments of its pulls master rank src has finished
    __device__ __forceinline__ uint64_t* reduce_flags_of(int rank) const { return reinterpret_cast<uint64_t*>(arena[rank] + reduce_flags); }
    __device__ __forceinline__ uint8_t* weight_of(int rank) const { return arena[rank] + replica_weight; }
    __device__ __forceinline__ uint8_t* scale_of(int rank) const { return arena[rank] + replica_scale; }
    __device__ __forceinline__ float* grad_of(int rank) const { return reinterpret_cast<float*>(arena[rank] + replica_grad); }
};

struct PlanPtrs {
    int32_t *p2l, *l2p, *lcnts, *quota, *quota_prefix, *rank_quota_prefix;
    int32_t* physical_loads;  // [P] tokens per physical slot under this plan (may be null)
};

struct ShardLayout {  // bytes of the four weight shards and their place inside a replica slot
    int64_t bytes[4];        // fc1, fc2, fc1 scale, fc2 scale
    int64_t slot_offset[4];  // offset inside the weight slot (0,1) / scale slot (2,3)
    int64_t weight_slot_stride, scale_slot_stride;
    int num_shards;          // 2 or 4
};

// ---- launchers (defined in the .cu files; every launch bumps the launch counter) ----
void count_launch(int n = 1);

struct PlanCall {
    GroupDev group;
    uint64_t* hist_parts[kMaxLocalRanks];    // [kPlanMaxCtas][Lpad] words, (epoch tag << 32) | partial count of one CTA
    // Counted on the device (by one CTA of every launch), not passed by value, so that a captured CUDA graph can be
    // replayed: every replay is a new epoch. The same for the epochs of weight_sync and of the Wgrad reduce.
    uint64_t* epoch[kMaxLocalRanks];
    int32_t* global_loads[kMaxLocalRanks];   // [L]
    int32_t* loads_per_rank[kMaxLocalRanks]; // [N][L] latest gathered matrix (contiguous copy)
    const void* input[kMaxLocalRanks];
    int T[kMaxLocalRanks];
    PlanPtrs plan[kMaxLocalRanks];
    int nlocal;
    int input_kind;  // 0 bool map, 1 ids32, 2 ids64
    int K_or_L;
    int N, G, M, R, D;
    uep_solver_params params;
    uint64_t timeout_ns;
    int ctas_per_rank, threads;
    int rehearsal_smem;      // where its crew's shared memory begins (set by launch_plan)
    int32_t* rehearsal_out;  // [hosted ranks][kRehearsalOut]
    int in_cluster;          // 1: the ranks hand each other their rows through the shared memory of their cluster (set by launch_plan)
    int withhold_rank;  // test hook: this rank does not publish its flags (-1: none)
    int withhold_row;   // test hook: in a cluster, this rank does not hand over its row (-1: none)
    int hard_rehearsal; // test hook: the rehearsal comes to the probes (1) or the wide keys (2)
    int legacy;         // 1: legacy placement solver (counts only; the reroute is then round-robin)
    unsigned long long* trace;  // optional: 8 globaltimer stamps per hosted rank (tuning aid), or null
};
// Whether the ranks hand their rows over inside a cluster: a group hosted whole. With the hook that withholds a rank they do it through
// memory, like ranks of several devices.
inline bool plan_in_cluster(int nlocal, int N, int withhold_rank) { return nlocal == N && withhold_rank < 0; }
// Whether the owners' CTAs rehearse the solver: a group hosted whole. Of one rank among ranks on other devices it is not measured, and its
// CTAs keep their size.
inline bool plan_rehearses(int nlocal, int N, int R, bool legacy) { return nlocal == N && N > 1 && R > 0 && !legacy; }
cudaError_t launch_plan(const PlanCall& call, cudaStream_t stream);
cudaError_t plan_most_ctas(int nlocal, int N, int G, int M, int R, int* ctas);
int plan_ctas_per_rank(int input_kind, int max_T, int K_or_L, int cap);

int plan_threads(int input_kind, int max_T, int K_or_L, int ctas);

struct SyncCall {
    GroupDev group;
    PlanPtrs plan[kMaxLocalRanks];
    const int64_t* src_ptrs[kMaxLocalRanks][4];  // device int64[M] tables; scale tables may be null
    int nlocal;
    int N, M, R, D;
    ShardLayout shards;
    uint64_t timeout_ns;
    int ctas_per_rank;
    int withhold_rank;  // test hook, as in PlanCall
    int relay_min_replicas;  // 0: every master writes all its replicas itself; else experts with at least this many
                             // replicas are scattered over them and forwarded replica to replica
    int relay_adaptive;      // 1: also relay the experts of ranks that send more than any rank receives (see weight_sync.cu)
    int relay_cap;           // chunks per slot the ready-flag table has room for
    uint64_t* sync_epoch;    // the sync epoch counter of the first hosted rank
    int* ticket;             // [2], zero between calls: CTAs that have finished, units handed out
    unsigned long long* trace;  // optional: 8 globaltimer stamps per CTA (tuning aid), or null
};
cudaError_t launch_weight_sync(const SyncCall& call, cudaStream_t stream);
int weight_sync_max_ctas_per_rank(int nlocal, int num_sms);

struct ReduceCall {
    GroupDev group;
    PlanPtrs plan[kMaxLocalRanks];
    const int64_t* fc1_grad_ptrs[kMaxLocalRanks];
    const int64_t* fc2_grad_ptrs[kMaxLocalRanks];
    int nlocal;
    int N, M, R, D;
    int64_t fc1_numel, fc2_numel;
    uint64_t timeout_ns;
    int ctas_per_rank;
    int owners_clear;           // test hook: replicas of hosted ranks are cleared by their owners too, as on other devices
    int withhold_rank;          // test hook: this rank reports no progress (-1: off)
    uint64_t* reduce_epoch;     // the reduce epoch counter of the first hosted rank
    int* counters;              // [kReduceSegments]: CTAs of this launch that have passed each segment; zero between calls
    unsigned long long* trace;  // optional: 8 globaltimer stamps per CTA (tuning aid), or null
};
cudaError_t launch_grad_reduce(const ReduceCall& call, cudaStream_t stream);

// Reroute launchers. One launch serves every hosted rank (blockIdx.y selects the rank).
struct DenseFwdArgs {
    const uint8_t* map;
    const float* probs;
    const int32_t *l2p, *lcnts, *rqp;
    int32_t* scratch;  // [dense tiles][L]
    uint8_t* out_map;
    float* out_probs;
    int T;
};
struct DenseBwdArgs {
    const float* grad_expanded;
    const uint8_t *map, *expanded_map;
    const int32_t *l2p, *lcnts;
    float* grad_probs;
    int T;
};
struct SparseArgs {
    const void* ids;
    void* out;
    const int32_t *l2p, *lcnts, *rqp;
    int32_t* scratch;  // [sparse tiles][L]
    int T;
};
template <typename A>
struct Batch {
    A a[kMaxLocalRanks];
    int n;
};
int64_t dense_scratch_elems(int T, int L);
int64_t sparse_scratch_elems(int64_t entries, int L);
// Kernels are launched as dependents of whatever is in front of them in their stream, and wait for it before they read anything but
// parameters (it may as well be a kernel of the caller's that starts its dependents early and writes the ids after that). An ordinary
// launch starts on the next tick of some 2 us from the start of the kernel in front, 1.8 us at least behind its end; a dependent one is
// past its wait 0.8 us behind that end whether or not the kernel in front says when it may start. So no kernel here says it, except to
// one that has something to do before its wait: CTAs that only wait take the place of others. Plan and reroute of eight ranks among
// others, before every launch was a dependent one and right behind that change (us): 33 tokens of 64 experts 13.5 and
// 11.4, 4096 tokens 25.1 and 16.9, bool rows 4096 of 128 experts 28.6 and 24.3; one rank's sparse, dense and backward, 8191 x 256,
// 28.5 and 25.4. beside_sync, beside_bytes: several ranks and a weight_sync of the plan was launched, which writes at most so many
// bytes: where its CTAs' first microseconds count, the reroute's launches are ordinary ones (reroute.cu).
cudaError_t launch_dense_forward(const Batch<DenseFwdArgs>& b, int L, int P, int D, int quota_mode, int interleave,
                                 bool beside_sync, cudaStream_t stream);
cudaError_t launch_dense_backward(const Batch<DenseBwdArgs>& b, int L, int P, int D, cudaStream_t stream);
cudaError_t launch_sparse_reroute(const Batch<SparseArgs>& b, int ids_kind, int K, int L, int D, int interleave, int64_t beside_bytes,
                                  cudaStream_t stream);

bool pdl_enabled();      // programmatic dependent launches are on (UEP_DISABLE_PDL=1 turns them off)
int device_sm_count();  // of the current device; launch sizes are multiples of it
// Lets a kernel use that much dynamic shared memory on the current device (and, once, ask for the largest carve-out).
cudaError_t allow_smem(const void* fn, size_t bytes, bool largest_carveout = false);
void set_error(const std::string& msg);
int fail(int code, const std::string& msg);
int fail_cuda(cudaError_t e, const char* what);

}  // namespace uep

#define UEP_CUDA_TRY(expr)                                         \
    do {                                                           \
        cudaError_t _e = (expr);                                   \
        if (_e != cudaSuccess) return ::uep::fail_cuda(_e, #expr); \
    } while (0)
