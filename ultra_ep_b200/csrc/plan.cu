// Kernel 1 — the plan: per-expert token counts, load all-gather over peer memory,
// reduction and placement solve in ONE launch per layer.
//
// What the reference does with about a dozen stream operations (memset + histogram,
// device copy, NVSHMEM fcollect, reduce kernel, six memsets, solver kernel;
// csrc/ultra_ep.cpp:676-745 and csrc/kernels/placement.cu:1602-1663 of the reference)
// is one kernel here:
//   * every CTA of a rank counts a slice of the routing input into shared memory; all but the
//     rank's first CTA store their partial counts as self-validating 64-bit words (epoch
//     tag << 32 | count; an aligned 8-byte store is single-copy atomic, so a word needs neither
//     a fence nor a flag) into a row of their own and are done;
//   * the rank's first CTA owns the rest: it adds up the partials (bounded wait on words of
//     its own launch's CTAs, none of which waits for it), stores the row into every peer's
//     gather buffer as the same kind of words, polls its own buffer (bounded) until every
//     rank's words carry this epoch's tag, reduces the matrix and runs the solver (solver.cuh).
// The gather buffers are double-buffered by epoch parity: a peer can be at most one
// call ahead, because it cannot pass call e+1 without this rank's row for e+1.
//
// With several ranks hosted on one device (simulated EP) the same kernel runs all of them in one launch of clusters, a CTA of
// every rank in each: the first CTAs of the ranks, the only ones that wait for each other, are one cluster and so co-resident,
// and hand their rows over through its shared memory.

#include <atomic>

#include <algorithm>
#include <cstring>

#include "internal.h"
#include "solver.cuh"

namespace uep {

namespace {

constexpr int kHistThreads = 256;
constexpr int kPlanThreads = 256;       // of a CTA of the plan kernel
constexpr int kRehearsalThreads = 128;  // and, where the solver is rehearsed, of its second crew
constexpr int kIdLoads = 4;  // 16-byte loads of ids that a thread has in flight
constexpr int kSolveThreads = 512;
constexpr size_t kSolveMaxSmem = 220 * 1024;
// Of the load matrix, where the plan kernel keeps it in shared memory: eight ranks of 512 experts, the largest group that one
// device can host and the plan kernel could be timed with. The solver's own kernel has its SM to itself and takes what fits.
constexpr size_t kPlanMatrixBytes = 16 * 1024;
// Partial counts a thread asks for at once. The CTAs behind a rank's first one are shared by as many threads as an expert can have: 14
// of them at most (eight hosted ranks) by two of 256 threads or four of 512 up to 128 experts, 31 (one rank) by four of 256 up to 64, one
// round each; more experts take more rounds.
constexpr int kPartBatch = 9;

__device__ __forceinline__ void hist_add_swar(uint32_t word, int32_t* hist, int col) {
    // four byte-wide counters packed in `word`
    const int c0 = word & 0xFF, c1 = (word >> 8) & 0xFF, c2 = (word >> 16) & 0xFF, c3 = word >> 24;
    if (c0) atomicAdd(hist + col, c0);
    if (c1) atomicAdd(hist + col + 1, c1);
    if (c2) atomicAdd(hist + col + 2, c2);
    if (c3) atomicAdd(hist + col + 3, c3);
}

// Bytes [begin, end) of a map whose rows are not whole vectors, into the counts at the start of the CTA's shared memory; `begin` is a row's
// first. Eight loads in flight, the column by additions. Out of line: most maps do not come here. (One load and a division at a time: plan of
// six ranks of 4000 x 120 33.5 us and 14.3, of eight of 8192 x 120 46.8 and 23.0, of three of 5561 x 120 37.1 and 19.5.)
__device__ __noinline__ void count_bytes(const uint8_t* __restrict__ map, int64_t begin, int64_t end, int L, int tid, int nthreads) {
    extern __shared__ __align__(128) char smem_raw[];
    int32_t* const hist = reinterpret_cast<int32_t*>(smem_raw);
    const int step = nthreads % L;
    int column = tid % L;
    for (int64_t i = begin + tid; i < end; i += 8 * nthreads) {
        uint8_t v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) v[u] = i + u * nthreads < end ? map[i + u * nthreads] : 0;
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            if (v[u] != 0) atomicAdd(hist + column, 1);
            column += step;
            column -= column >= L ? L : 0;
        }
    }
}

// Count this CTA's slice of the input into hist[L] (the start of its shared memory, zeroed by the caller).
// part / nparts split the rows (dense) or the entries (sparse) evenly.
// Inlined, so that a cold kernel does not jump for it first. Counts of 33 tokens of 64 experts behind an L2 flush, out of line and like
// this: 4.2 us after the start and 2.2, 4096 tokens 5.1 and 3.6; among other plans 1.9 and 1.6, 3.4 and 3.0.
__device__ __forceinline__ void histogram_slice(int input_kind, const void* input, int T, int K_or_L, int L, int part, int nparts,
                                int32_t* hist, int nthreads) {
    const int tid = threadIdx.x;
    if (input_kind == 0) {
        const uint8_t* map = static_cast<const uint8_t*>(input);
        const int rows_per = ceil_div_i(T, nparts);
        const int r0 = min(part * rows_per, T), r1 = min(r0 + rows_per, T);
        const int groups = L / 16;
        const bool vec_ok = (L % 16 == 0) && ((reinterpret_cast<uintptr_t>(map) & 15u) == 0) && groups <= nthreads;
        if (vec_ok) {
            // one thread owns a 16-column group and walks rows, eight loads in flight; 0/1 bytes are summed four at a
            // time inside 32-bit words and spilled to the histogram before a byte can overflow. (One load at a time: the
            // plan kernel of eight ranks of 8192 x 128 took 28 us, against 22 with this and the present solver.)
            const int g = tid % groups;
            const int row_lane = tid / groups, row_lanes = nthreads / groups;
            const int most = 8 * ceil_div_i(max(r1 - r0, 0), 8 * row_lanes);  // of a byte of a thread's sums
            uint4 acc = make_uint4(0, 0, 0, 0);
            int pending = 0;
            for (int r = row_lane < row_lanes ? r0 + row_lane : r1; r < r1; r += 8 * row_lanes) {
                uint4 v[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const int row = r + u * row_lanes;
                    v[u] = row < r1 ? ld_global_nc_v4(map + static_cast<int64_t>(row) * L + g * 16) : make_uint4(0, 0, 0, 0);
                }
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    acc.x += v[u].x; acc.y += v[u].y; acc.z += v[u].z; acc.w += v[u].w;
                }
                if ((pending += 8) == 248) {
                    hist_add_swar(acc.x, hist, g * 16); hist_add_swar(acc.y, hist, g * 16 + 4);
                    hist_add_swar(acc.z, hist, g * 16 + 8); hist_add_swar(acc.w, hist, g * 16 + 12);
                    acc = make_uint4(0, 0, 0, 0);
                    pending = 0;
                }
            }
            if (groups <= 32 && (groups & (groups - 1)) == 0 && most * (32 / groups) < 256) {
                // the lanes with the same columns add their bytes up first and then share the words: a fourth of the shared
                // additions at 128 experts, and no two of a warp's at one address
                for (int d = groups; d < 32; d <<= 1) {
                    acc.x += __shfl_xor_sync(kFullMask, acc.x, d); acc.y += __shfl_xor_sync(kFullMask, acc.y, d);
                    acc.z += __shfl_xor_sync(kFullMask, acc.z, d); acc.w += __shfl_xor_sync(kFullMask, acc.w, d);
                }
                const int subs = 32 / groups, sub = (tid & 31) / groups;
                const uint32_t words[4] = {acc.x, acc.y, acc.z, acc.w};
#pragma unroll
                for (int w = 0; w < 4; ++w) {
                    if ((w & (subs - 1)) == sub) hist_add_swar(words[w], hist, g * 16 + 4 * w);
                }
            } else {
                hist_add_swar(acc.x, hist, g * 16); hist_add_swar(acc.y, hist, g * 16 + 4);
                hist_add_swar(acc.z, hist, g * 16 + 8); hist_add_swar(acc.w, hist, g * 16 + 12);
            }
        } else {
            count_bytes(map, static_cast<int64_t>(r0) * L, static_cast<int64_t>(r1) * L, L, tid, nthreads);
        }
    } else {
        const int64_t n = static_cast<int64_t>(T) * K_or_L;
        // slices start at multiples of four entries so that aligned inputs can be read 16 bytes at a time;
        // a thread issues all of its vector loads before it touches the first result
        const int64_t per = ((n + nparts - 1) / nparts + 3) & ~static_cast<int64_t>(3);
        const int64_t begin = min(static_cast<int64_t>(part) * per, n), end = min(begin + per, n);
        if (input_kind == 1) {
            const int32_t* ids = static_cast<const int32_t*>(input);
            int64_t i0 = begin;
            if ((reinterpret_cast<uintptr_t>(ids) & 15u) == 0) {
                const int64_t nvec = (end - begin) / 4;
                const int4* v = reinterpret_cast<const int4*>(ids + begin);
                for (int64_t j0 = 0; j0 < nvec; j0 += kIdLoads * nthreads) {
                    int4 x[kIdLoads];
#pragma unroll
                    for (int u = 0; u < kIdLoads; ++u) {
                        const int64_t j = j0 + tid + static_cast<int64_t>(u) * nthreads;
                        x[u] = j < nvec ? __ldg(v + j) : make_int4(-1, -1, -1, -1);
                    }
#pragma unroll
                    for (int u = 0; u < kIdLoads; ++u) {
                        const int e[4] = {x[u].x, x[u].y, x[u].z, x[u].w};
#pragma unroll
                        for (int c = 0; c < 4; ++c) {
                            if (e[c] >= 0 && e[c] < L) atomicAdd(hist + e[c], 1);
                        }
                    }
                }
                i0 = begin + nvec * 4;
            }
            for (int64_t i = i0 + tid; i < end; i += nthreads) {
                const int32_t e = ids[i];
                if (e >= 0 && e < L) atomicAdd(hist + e, 1);
            }
        } else {
            const int64_t* ids = static_cast<const int64_t*>(input);
            int64_t i0 = begin;
            if ((reinterpret_cast<uintptr_t>(ids) & 15u) == 0) {
                const int64_t nvec = (end - begin) / 2;
                const longlong2* v = reinterpret_cast<const longlong2*>(ids + begin);
                for (int64_t j0 = 0; j0 < nvec; j0 += kIdLoads * nthreads) {
                    longlong2 x[kIdLoads];
#pragma unroll
                    for (int u = 0; u < kIdLoads; ++u) {
                        const int64_t j = j0 + tid + static_cast<int64_t>(u) * nthreads;
                        x[u] = j < nvec ? __ldg(v + j) : make_longlong2(-1, -1);
                    }
#pragma unroll
                    for (int u = 0; u < kIdLoads; ++u) {
                        if (x[u].x >= 0 && x[u].x < L) atomicAdd(hist + static_cast<int>(x[u].x), 1);
                        if (x[u].y >= 0 && x[u].y < L) atomicAdd(hist + static_cast<int>(x[u].y), 1);
                    }
                }
                i0 = begin + nvec * 2;
            }
            for (int64_t i = i0 + tid; i < end; i += nthreads) {
                const int64_t e = ids[i];
                if (e >= 0 && e < L) atomicAdd(hist + static_cast<int>(e), 1);
            }
        }
    }
}

__global__ void __launch_bounds__(kHistThreads) histogram_kernel(int input_kind, const void* input, int T, int K_or_L,
                                                                 int L, int32_t* loads) {
    extern __shared__ __align__(128) char smem_raw[];
    int32_t* hist = reinterpret_cast<int32_t*>(smem_raw);
    for (int i = threadIdx.x; i < L; i += blockDim.x) hist[i] = 0;
    __syncthreads();
    histogram_slice(input_kind, input, T, K_or_L, L, blockIdx.x, gridDim.x, hist, blockDim.x);
    __syncthreads();
    for (int i = threadIdx.x; i < L; i += blockDim.x) {
        if (hist[i]) atomicAdd(loads + i, hist[i]);
    }
}

// Stateless solve: one CTA per NVLink domain.
template <bool kLegacy>
__global__ void __launch_bounds__(kSolveThreads, 1) solve_kernel(SolveArgs a, int32_t* global_loads_out, int reduce_loads, int staged,
                                                                 DeviceStatus* status) {
    extern __shared__ __align__(128) char smem_raw[];
    const int domain = blockIdx.x;
    const int E = a.G * a.M, L = a.N * a.M;
    pdl_wait();  // ahead of every read
    if (reduce_loads) {
        // Total load of this domain's experts over all ranks, and this rank's own, straight to where the solver keeps
        // them. The rows are shared by all the threads an expert, or four of them, can have, 16 or 8 loads of each in flight.
        // Rows by single words and, where they are aligned, 16 bytes at a time (us): 64 ranks of 4 experts, two round trips and one, 17.0 and
        // 16.3, 72 of 7 experts 23.2 and 21.6, 48 of 7 18.9 and 17.6, 32 of 4 9.3 and 9.1.
        const SolverSmem sm = carve_solver_smem(smem_raw, E, a.G, a.R);
        int32_t* matrix = reinterpret_cast<int32_t*>(smem_raw + solver_smem_bytes(E, a.G, a.R));
        for (int i = threadIdx.x; i < E; i += blockDim.x) sm.loads[i] = 0;
        __syncthreads();
        const bool vec = (E & 3) == 0 && (reinterpret_cast<uintptr_t>(a.loads_per_rank) & 15u) == 0;
        const int columns = vec ? E / 4 : E, parts = max(static_cast<int>(blockDim.x) / columns, 1);
        for (int i = threadIdx.x; i < columns * parts; i += blockDim.x) {
            const int part = i / columns, e = (i - part * columns) * (vec ? 4 : 1);
            const int32_t* column = a.loads_per_rank + domain * E + e;
            if (vec) {
                int4 total = make_int4(0, 0, 0, 0);
                for (int r0 = part; r0 < a.N; r0 += 8 * parts) {
                    int4 v[8];
#pragma unroll
                    for (int u = 0; u < 8; ++u) {
                        v[u] = r0 + u * parts < a.N ? __ldcg(reinterpret_cast<const int4*>(column + static_cast<int64_t>(r0 + u * parts) * L)) : make_int4(0, 0, 0, 0);
                    }
#pragma unroll
                    for (int u = 0; u < 8; ++u) {
                        const int r = r0 + u * parts;
                        total.x += v[u].x; total.y += v[u].y; total.z += v[u].z; total.w += v[u].w;
                        if (staged && r < a.N) *reinterpret_cast<int4*>(matrix + r * L + e) = v[u];
                        if (r == a.my_rank) *reinterpret_cast<int4*>(sm.my_loads + e) = v[u];
                    }
                }
                atomicAdd(sm.loads + e, total.x); atomicAdd(sm.loads + e + 1, total.y);
                atomicAdd(sm.loads + e + 2, total.z); atomicAdd(sm.loads + e + 3, total.w);
                continue;
            }
            if (part == 0) sm.my_loads[e] = __ldcg(column + static_cast<int64_t>(a.my_rank) * L);
            int32_t total = 0;
            for (int r0 = part; r0 < a.N; r0 += 16 * parts) {
                int32_t v[16];
#pragma unroll
                for (int u = 0; u < 16; ++u) v[u] = r0 + u * parts < a.N ? __ldcg(column + static_cast<int64_t>(r0 + u * parts) * L) : 0;
#pragma unroll
                for (int u = 0; u < 16; ++u) {
                    total += v[u];
                    if (staged && r0 + u * parts < a.N) matrix[(r0 + u * parts) * L + e] = v[u];
                }
            }
            atomicAdd(sm.loads + e, total);
        }
        __syncthreads();
        for (int i = threadIdx.x; i < E; i += blockDim.x) global_loads_out[domain * E + i] = sm.loads[i];
        a.preloaded = 1;
        a.staged_loads = staged ? matrix : nullptr;
    }
    if (kLegacy) legacy_solve(a, domain, smem_raw, status);
    else solve_domain(a, Crew{static_cast<int>(threadIdx.x), static_cast<int>(blockDim.x), 0}, domain, smem_raw, status);
}

__global__ void __launch_bounds__(256) init_master_kernel(int32_t* p2l, int32_t* l2p, int32_t* lcnts, int32_t* quota,
                                                          int32_t* quota_prefix, int32_t* rqp, int N, int M, int R,
                                                          int D) {
    const int Lp = M + R, L = N * M, P = N * Lp;
    const int gtid = blockIdx.x * blockDim.x + threadIdx.x, gsize = gridDim.x * blockDim.x;
    for (int i = gtid; i < P; i += gsize) {
        const int local = i % Lp;
        p2l[i] = local < M ? (i / Lp) * M + local : -1;
    }
    for (int i = gtid; i < L * D; i += gsize) {
        const int l = i / D, j = i % D;
        l2p[i] = j == 0 ? (l / M) * Lp + l % M : -1;
        quota[i] = 0;
        quota_prefix[i] = 0;
        rqp[i] = 0;
    }
    for (int i = gtid; i < L; i += gsize) lcnts[i] = 1;
}

__host__ __device__ inline size_t plan_matrix_bytes(int N, int L) {
    const size_t bytes = sizeof(int32_t) * N * static_cast<size_t>(L);
    return bytes <= kPlanMatrixBytes ? bytes : 0;
}

// The solver's code runs once a layer, and what runs between two layers (weight copies, expanded outputs, the model) leaves none of
// it in L2: its instructions came from DRAM one line after another, and from L2 to the SM likewise where they were still there. So the
// CTA that owns a rank has a second crew of threads, which solves a small problem from the kernel's start, while the first one counts
// and exchanges, with the same instructions. Nobody waits for it. It takes the way of the default parameters: the sort, the four
// builds side by side with an expert of two exports and ranks that come back, outputs and splits of experts with replicas; not the rounds
// of probes nor more than 32 replicas, nor masters and replicas that do not come in fours. Its outputs go to a place of their own. Step of eight ranks among others without it and like
// this (us): bf16 experts of 9 MB, 8192 bool rows of 128 64.3 and 59.2; fp8 experts of 19 MB, 8192 int32 tokens of 128 56.1 and 54.4; plan and
// reroute of 4096 tokens of 64 18.8 and 18.1, of 33 11.6 and 11.4. (A CTA of its own warms L2 alone: the plan's builds 2.2 us instead of
// 1.8; half of the ranks with the outputs first 59.2 and 59.3.)
constexpr int kRehearsalRanks = 4, kRehearsalMasters = 4, kRehearsalSlots = 2, kRehearsalD = 4;
constexpr int kRehearsalExperts = kRehearsalRanks * kRehearsalMasters;
constexpr int kRehearsalPhysical = kRehearsalRanks * (kRehearsalMasters + kRehearsalSlots);
static_assert(4 * kRehearsalExperts * kRehearsalD + kRehearsalExperts + 2 * kRehearsalPhysical <= kRehearsalOut, "room for its outputs");
__host__ __device__ inline size_t rehearsal_smem_bytes() {
    return solver_smem_bytes(kRehearsalExperts, kRehearsalRanks, kRehearsalSlots) + sizeof(int32_t) * kRehearsalRanks * kRehearsalExperts;
}
// Two ranks above the mean and two below. The parameters are its own: a caller's threshold or floor could leave it without exports.
// (Test hook: a problem that comes to what is out of line. Three ranks of equal masters above the mean need more exports than the
// fourth has slots at every threshold below their load, so no build succeeds, and 1 << 24 needs wide keys.)
__device__ __forceinline__ void rehearsal_args(const PlanCall& call, const Crew& crew, int local, char* smem_raw, SolveArgs& a) {
    const SolverSmem sm = carve_solver_smem(smem_raw, kRehearsalExperts, kRehearsalRanks, kRehearsalSlots);
    int32_t* matrix = reinterpret_cast<int32_t*>(smem_raw + solver_smem_bytes(kRehearsalExperts, kRehearsalRanks, kRehearsalSlots));
    for (int i = crew.tid; i < kRehearsalExperts; i += crew.threads) {
        const int rank = i / kRehearsalMasters;
        int load = i % kRehearsalMasters != 0 ? 100 : (rank < 2 ? 6000 : 375 >> 2 * (rank - 2));
        if (call.hard_rehearsal) load = rank < 3 ? (call.hard_rehearsal == 1 ? 1 << 10 : 1 << 24) : 0;
        sm.loads[i] = load;
        sm.my_loads[i] = load / 4;
        for (int r = 0; r < kRehearsalRanks; ++r) matrix[r * kRehearsalExperts + i] = load / 4;
    }
    if (crew.tid == 0) {
        int32_t* out = call.rehearsal_out + local * kRehearsalOut;
        a.l2p = out; out += kRehearsalExperts * kRehearsalD;
        a.quota = out; out += kRehearsalExperts * kRehearsalD;
        a.quota_prefix = out; out += kRehearsalExperts * kRehearsalD;
        a.rank_quota_prefix = out; out += kRehearsalExperts * kRehearsalD;
        a.lcnts = out; out += kRehearsalExperts;
        a.p2l = out; out += kRehearsalPhysical;
        a.physical_loads = out;
        a.global_loads = nullptr;
        a.loads_per_rank = nullptr;
        a.N = a.G = kRehearsalRanks; a.M = kRehearsalMasters; a.R = kRehearsalSlots; a.D = kRehearsalD;
        a.balance_threshold = 1.f;
        a.min_tokens = 1;
        a.allow_zero_master = 0;
        a.locality = call.params.locality_aware;
        a.eps = 0.01f;
        a.my_rank = 0;
        a.preloaded = 1;
        a.staged_loads = matrix;
        a.trace = nullptr;
    }
    crew.sync();
}

// Steps 1 to 3 of a rank: counts, exchange, reduction. False: this CTA has handed its counts over and is done, or the loads did not
// come; else `a` says what to solve.
template <bool kLegacy>
__device__ __forceinline__ bool gather_loads(const PlanCall& call, const Crew& crew, int local, int part, char* smem_raw, SolveArgs& a) {
    __shared__ int s_timeout_peer;
    __shared__ uint64_t s_epoch;
    __shared__ __align__(8) uint64_t s_rows[kMaxLocalRanks];  // a barrier for each other rank's row, where they are pushed
    const GroupDev& group = call.group;
    uint64_t* const hist_parts = call.hist_parts[local];
    const int N = call.N, M = call.M;
    const int L = N * M;
    const int Lpad = (L + 3) / 4 * 4;
    const int tid = crew.tid;
    const unsigned long long t_start = call.trace != nullptr ? global_timer_ns() : 0ull;
    auto stamp = [&](int slot) {
        if (call.trace != nullptr && tid == 0) call.trace[local * 8 + slot] = global_timer_ns();
    };

    // 1. histogram slice -> shared. The rank's first CTA owns the rest of the kernel; the others hand it their
    //    partial counts as self-validating words (epoch tag << 32 | count) in a row of their own and are done:
    //    no atomics on a common row, no fence, no ticket, and the owner sees a partial one memory round trip
    //    after it was stored. The owner waits (bounded) for CTAs of its own launch; none of them waits for it,
    //    so they need not be resident at the same time.
    int32_t* hist = reinterpret_cast<int32_t*>(smem_raw);
    const int me = group.my_rank[local];
    const bool preload = !kLegacy;
    const bool staged = preload && plan_matrix_bytes(N, L) > 0;
    int32_t* matrix = reinterpret_cast<int32_t*>(smem_raw + solver_smem_bytes(L, N, call.R));
    for (int i = tid; i < L; i += crew.threads) hist[i] = 0;
    const bool owner = part == 0, pushes = call.in_cluster != 0;
    if (tid == 0) s_timeout_peer = -1;
    if (owner && pushes && tid < N && tid != local) {
        mbar_init(&s_rows[tid], 1);
        fence_mbar_init();
        mbar_expect_tx(&s_rows[tid], static_cast<uint32_t>(L * sizeof(int32_t)));
    }
    if (owner && pushes) cluster_arrive();  // (the owners are a cluster of their own)
    pdl_wait();  // ahead of every read: what is in front may still be writing the input
    // the epoch this launch opens: the owner stores it once it holds every partial, so every CTA of the launch reads the
    // same value here
    uint64_t last_epoch = 0;
    if (tid == 0) last_epoch = ld_relaxed_sys_u64(call.epoch[local]);  // on its way while the slice is counted
    crew.sync();
    histogram_slice(call.input_kind, call.input[local], call.T[local], call.K_or_L, L, part, call.ctas_per_rank, hist, crew.threads);
    if (tid == 0) s_epoch = last_epoch + 1;
    crew.sync();
    const uint64_t epoch = s_epoch;
    // never zero (the buffers start zeroed), period 2^32 - 1: an odd period, so the word that carried the same
    // tag one period ago sat in the other parity slot and cannot be mistaken for this epoch's
    const uint32_t tag = static_cast<uint32_t>(epoch % 0xFFFFFFFFull) + 1u;
    if (part != 0) {
        uint64_t* row = hist_parts + static_cast<int64_t>(part) * Lpad;
        for (int i = tid; i < L; i += crew.threads) st_relaxed_sys_u64(row + i, tag_word(tag, static_cast<uint32_t>(hist[i])));
        return false;
    }
    if (call.trace != nullptr && tid == 0) call.trace[local * 8 + 5] = t_start;  // when this CTA started
    if (pushes) cluster_wait();  // every owner has started and its barrier for the rows is there
    // An owner that gives up stays until nobody can push to it any more.
    auto leave = [&]() {
        if (pushes) {
            cluster_arrive();
            cluster_wait();
        }
    };
    // What the solver needs of the parameters goes into shared memory while this CTA waits for the others: of one rank they were last
    // read a layer ago, and each line of them comes from memory.
    if (tid == crew.threads - 1) {
        a.global_loads = call.global_loads[local];
        a.loads_per_rank = call.loads_per_rank[local];
        const PlanPtrs& pp = call.plan[local];
        a.p2l = pp.p2l; a.l2p = pp.l2p; a.lcnts = pp.lcnts; a.quota = pp.quota; a.quota_prefix = pp.quota_prefix;
        a.rank_quota_prefix = pp.rank_quota_prefix;
        a.physical_loads = pp.physical_loads;
        a.N = N; a.G = N; a.M = M; a.R = call.R; a.D = call.D;
        a.balance_threshold = call.params.balance_threshold;
        a.min_tokens = call.params.min_tokens_per_replica;
        a.allow_zero_master = call.params.allow_zero_master_quota;
        a.locality = call.params.locality_aware;
        a.eps = call.params.oracle_eps;
        a.my_rank = me;
        a.preloaded = preload ? 1 : 0;
        a.staged_loads = staged ? matrix : nullptr;
        a.trace = call.trace != nullptr ? call.trace + (kMaxLocalRanks + local) * 8 : nullptr;
    }
    {   // an expert's partials are shared by all the threads it can have, so that one round of loads fetches them
        const int rest = call.ctas_per_rank - 1;
        const int parts = max(min(crew.threads / L, rest), 1);
        for (int idx = tid; idx < L * parts; idx += crew.threads) {
            const int i = idx % L, part = idx / L;
            int32_t total = 0;
            for (int c0 = 1 + part; c0 <= rest; c0 += kPartBatch * parts) {
                uint64_t w[kPartBatch];
#pragma unroll
                for (int u = 0; u < kPartBatch; ++u) {
                    const int c = c0 + u * parts;
                    if (c <= rest) w[u] = ld_relaxed_sys_u64(hist_parts + static_cast<int64_t>(c) * Lpad + i);
                }
#pragma unroll
                for (int u = 0; u < kPartBatch; ++u) {
                    const int c = c0 + u * parts;
                    if (c <= rest) {
                        if (static_cast<uint32_t>(w[u] >> 32) != tag &&
                            !wait_tagged_word(hist_parts + static_cast<int64_t>(c) * Lpad + i, tag,
                                              *reinterpret_cast<volatile int*>(&s_timeout_peer) >= 0 ? 0 : call.timeout_ns, w[u])) {
                            atomicMax(&s_timeout_peer, group.my_rank[local]);
                            w[u] = 0;
                        }
                        total += static_cast<int32_t>(static_cast<uint32_t>(w[u]));
                    }
                }
            }
            if (rest > 0) atomicAdd(hist + i, total);
        }
    }
    crew.sync();
    if (tid == 0) *call.epoch[local] = epoch;  // every CTA of the launch has read the old value: its partial carried the tag
    if (s_timeout_peer >= 0) {  // a CTA of this very launch never delivered
        if (tid == 0) report_error(group.status[local], UEP_DEV_TIMEOUT_GATHER, s_timeout_peer);
        leave();
        return false;
    }
    stamp(0);

    // With one domain the solver finds the loads in shared memory where it keeps them: its loads are where hist was.
    const SolverSmem solver_sm = carve_solver_smem(smem_raw, L, N, call.R);
    if (pushes) {
        // 2, 3. The ranks of one cluster write their rows straight into each other's matrix, a warp per rank; the bytes are counted
        //    where they land, row by row, so that a rank whose row does not come can be named. (Words through memory, as below, take a store, a look and their two ways through L2: 1.5 us more.)
        const int warp = tid >> 5, lane = tid & 31, warps = crew.threads / kWarp;
        const bool vec = (L & 3) == 0;
        int32_t* row = matrix + me * L;
        for (int p = warp; p < N; p += warps) {
            if (p == local) {
                for (int i = lane; i < L; i += kWarp) row[i] = hist[i];
                continue;
            }
            if (me == call.withhold_row) continue;
            const uint32_t to = cluster_addr(row, p), bar = cluster_addr(&s_rows[local], p);
            if (vec) {
                for (int i = lane * 4; i < L; i += kWarp * 4) push_v4(to + i * 4, *reinterpret_cast<const int4*>(hist + i), bar);
            } else {
                for (int i = lane; i < L; i += kWarp) push_word(to + i * 4, hist[i], bar);
            }
        }
        crew.sync();  // hist has been read by every thread, this rank's own row is there
        stamp(1);
        if (tid < N && tid != local && !mbar_wait(&s_rows[tid], 0, call.timeout_ns)) atomicMax(&s_timeout_peer, group.my_rank[tid]);
        crew.sync();
        if (s_timeout_peer >= 0) {
            if (tid == 0) report_error(group.status[local], UEP_DEV_TIMEOUT_GATHER, s_timeout_peer);
            leave();
            return false;
        }
        for (int i = tid; i < L; i += crew.threads) {
            int32_t total = 0;
#pragma unroll
            for (int r = 0; r < kMaxLocalRanks; ++r) {
                if (r < N) {
                    const int32_t v = matrix[r * L + i];
                    call.loads_per_rank[local][r * L + i] = v;
                    total += v;
                }
            }
            call.global_loads[local][i] = total;
            if (preload) {
                solver_sm.my_loads[i] = hist[i];
                solver_sm.loads[i] = total;  // (hist[i] itself)
            }
        }
        __threadfence_block();
        crew.sync();
    } else {
        const int slot = static_cast<int>(epoch & 1ull);
        // 2. publish the row to every rank (itself included). Every 64-bit word carries the epoch beside its
        //    count, so a row needs neither a fence nor a flag: one NVLink crossing, and the reader knows a word
        //    is this layer's when it sees it.
        if (me != call.withhold_rank) {
            for (int i = tid; i < L; i += crew.threads) {
                const uint64_t word = tag_word(tag, static_cast<uint32_t>(hist[i]));
                for (int p = 0; p < N; ++p) st_relaxed_sys_u64(group.gather_of(p) + (static_cast<int64_t>(slot) * N + me) * Lpad + i, word);
            }
        }

        crew.sync();  // hist has been read by every thread
        stamp(1);
        // 3. collect every rank's row (bounded), expose the matrix, reduce. A thread owns one expert:
        //    it first issues the loads of eight ranks' words together and only then looks at them,
        //    so the common case (all rows already here) costs one memory round trip.
        const uint64_t* gathered = group.gather_of(me) + static_cast<int64_t>(slot) * N * Lpad;
        for (int i = tid; i < L; i += crew.threads) {
            int32_t total = 0;
            for (int r0 = 0; r0 < N; r0 += 8) {
                uint64_t w[8];
    #pragma unroll
                for (int u = 0; u < 8; ++u) {
                    if (r0 + u < N) w[u] = ld_relaxed_sys_u64(gathered + static_cast<int64_t>(r0 + u) * Lpad + i);
                }
    #pragma unroll
                for (int u = 0; u < 8; ++u) {
                    if (r0 + u < N) {
                        // one time limit for the whole gather: once a wait has run out, no other word is waited for
                        if (static_cast<uint32_t>(w[u] >> 32) != tag &&
                            !wait_tagged_word(gathered + static_cast<int64_t>(r0 + u) * Lpad + i, tag,
                                              *reinterpret_cast<volatile int*>(&s_timeout_peer) >= 0 ? 0 : call.timeout_ns, w[u])) {
                            atomicMax(&s_timeout_peer, r0 + u);
                            w[u] = 0;
                        }
                        const int32_t v = static_cast<int32_t>(static_cast<uint32_t>(w[u]));
                        call.loads_per_rank[local][static_cast<int64_t>(r0 + u) * L + i] = v;
                        if (staged) matrix[(r0 + u) * L + i] = v;
                        total += v;
                    }
                }
            }
            call.global_loads[local][i] = total;
            if (preload) {
                solver_sm.my_loads[i] = hist[i];
                solver_sm.loads[i] = total;  // (hist[i] itself)
            }
        }
        __threadfence_block();
        crew.sync();
        if (s_timeout_peer >= 0) {
            if (tid == 0) report_error(group.status[local], UEP_DEV_TIMEOUT_GATHER, s_timeout_peer);
            return false;  // plan of this layer is left as it was; the host raises on the status word
        }
    }
    stamp(2);
    stamp(3);
    return true;
}

// The fused per-layer plan kernel: ctas_per_rank clusters of a CTA of every hosted rank. The ranks' first CTAs come last, behind those that
// they wait for. The threads behind kThreads are there where it is rehearsed.
template <int kThreads, bool kLegacy>
__global__ void __launch_bounds__(kThreads + kRehearsalThreads, 1) plan_kernel(PlanCall call) {
    extern __shared__ __align__(128) char smem_raw[];
    const int local = cluster_cta();
    const int part = call.ctas_per_rank - 1 - (call.nlocal > 1 ? static_cast<int>(blockIdx.x) / call.nlocal : static_cast<int>(blockIdx.x));
    const bool rehearses = !kLegacy && threadIdx.x >= kThreads;
    const Crew crew = rehearses ? Crew{static_cast<int>(threadIdx.x) - kThreads, kRehearsalThreads, kSecondCrewBarrier} : Crew{static_cast<int>(threadIdx.x), kThreads, 1};
    char* const smem = rehearses ? smem_raw + call.rehearsal_smem : smem_raw;
    __shared__ SolveArgs args[2];  // of each crew
    SolveArgs& a = args[rehearses ? 1 : 0];
    if (rehearses) {
        if (part != 0) return;
        if (call.in_cluster) cluster_arrive();  // the other crew's barrier counts every thread
        rehearsal_args(call, crew, local, smem, a);
    } else if (!gather_loads<kLegacy>(call, crew, local, part, smem, a)) {
        return;
    }
    DeviceStatus* const status = rehearses ? nullptr : call.group.status[local];
    if (kLegacy) legacy_solve_apart(a, 0, smem, status);
    else solve_domain(a, crew, 0, smem, status);
    if (!rehearses && call.trace != nullptr && threadIdx.x == 0) call.trace[local * 8 + 4] = global_timer_ns();
}

size_t plan_smem_bytes(int N, int G, int M, int R) {
    const size_t solver = std::max(solver_smem_bytes(G * M, G, R) + (G == N ? plan_matrix_bytes(N, N * M) : 0), legacy_smem_bytes(G * M, G));
    const size_t hist = sizeof(int32_t) * static_cast<size_t>(N) * M;
    return (std::max(solver, hist) + 15) / 16 * 16;
}

std::atomic<int64_t> g_launches{0};

}  // namespace

void count_launch(int n) { g_launches.fetch_add(n, std::memory_order_relaxed); }

// Twice the threads where a CTA's slice of the input is long enough to pay for the larger block. Step of eight ranks with 256 threads and
// 512 (us), below the line: 2200 bool rows of 128 experts (18.3 KB a CTA) 36.5 and 38.2, 2600 (21.7 KB) 35.3 and 36.4, 8192 int32 tokens of 128
// (17 KB) 52.5 and 52.7, 9600 (20 KB) 39.65 and 39.6, 4800 int64 tokens of 64 (20 KB) 27.9 and 28.1; above it 11000 int32 tokens (23 KB) 40.75
// and 40.3, 2600 bool rows of 256 (43 KB) 53.4 and 51.8, 16384 int64 tokens of 256 (68 KB) 106.8 and 104.5. Legacy plans the same: with the
// dense reroute 8192 rows of 256 191.4 and 188.5, of 512 180.5 and 175.6; one rank's plan of 8192 x 256 9.5 and 8.1, of 16384 x 64 6.3 and 6.7.
// Maps that are counted byte by byte take longer: 512 threads from 16 KB on (plan of six ranks of 4000 x 120, 20.9 KB, 17.3 and 14.3; of seven of
// 4000 x 70 15.2 and 13.1).
constexpr int kFewThreadsBytes = 22 * 1024, kFewThreadsBytesSingle = 16 * 1024;
int plan_threads(int input_kind, int max_T, int K_or_L, int ctas) {
    const int64_t bytes = static_cast<int64_t>(max_T) * K_or_L * (input_kind == 0 ? 1 : (input_kind == 1 ? 4 : 8));
    const int line = input_kind == 0 && K_or_L % 16 != 0 ? kFewThreadsBytesSingle : kFewThreadsBytes;
    return bytes > static_cast<int64_t>(ctas) * line ? 2 * kPlanThreads : kPlanThreads;
}

int plan_ctas_per_rank(int input_kind, int max_T, int K_or_L, int cap) {
    const int64_t bytes = static_cast<int64_t>(max_T) * K_or_L * (input_kind == 0 ? 1 : (input_kind == 1 ? 4 : 8));
    const int64_t ctas = (bytes + 16 * 1024 - 1) / (16 * 1024);
    return static_cast<int>(std::max<int64_t>(std::min<int64_t>(ctas, std::min(cap, kPlanMaxCtas)), 1));
}

namespace {

const void* plan_kernel_of(bool legacy, int threads) {
    if (threads == kPlanThreads) {
        return legacy ? reinterpret_cast<const void*>(plan_kernel<kPlanThreads, true>) : reinterpret_cast<const void*>(plan_kernel<kPlanThreads, false>);
    }
    return legacy ? reinterpret_cast<const void*>(plan_kernel<2 * kPlanThreads, true>) : reinterpret_cast<const void*>(plan_kernel<2 * kPlanThreads, false>);
}

cudaLaunchAttribute dependent_launch() {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    return attr;
}

cudaLaunchAttribute plan_cluster(int nlocal) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = nlocal;
    attr.val.clusterDim.y = 1;
    attr.val.clusterDim.z = 1;
    return attr;
}

}  // namespace

// The most CTAs of a rank that the device holds at once, a CTA of every hosted rank being a cluster (clusters of eight: 15 of the 18 that
// 148 SMs could hold, since a cluster's SMs are of one GPC).
cudaError_t plan_most_ctas(int nlocal, int N, int G, int M, int R, int* ctas) {
    *ctas = kPlanMaxCtas;
    if (nlocal == 1) return cudaSuccess;
    const void* kernel = plan_kernel_of(false, kPlanThreads);
    const size_t smem = plan_smem_bytes(N, G, M, R) + rehearsal_smem_bytes();
    cudaError_t e = allow_smem(kernel, smem);
    if (e != cudaSuccess) return e;
    cudaLaunchAttribute attr[1] = {plan_cluster(nlocal)};
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(nlocal);
    cfg.blockDim = dim3(kPlanThreads + kRehearsalThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int clusters = 0;
    e = cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg);
    if (e != cudaSuccess) return e;
    *ctas = std::max(clusters, 1);
    return cudaSuccess;
}

cudaError_t launch_plan(const PlanCall& call, cudaStream_t stream) {
    const bool rehearses = plan_rehearses(call.nlocal, call.N, call.R, call.legacy != 0);
    PlanCall copy = call;
    copy.rehearsal_smem = static_cast<int>(plan_smem_bytes(call.N, call.G, call.M, call.R));
    copy.in_cluster = plan_in_cluster(call.nlocal, call.N, call.withhold_rank) ? 1 : 0;
    const size_t smem = copy.rehearsal_smem + (rehearses ? rehearsal_smem_bytes() : 0);
    const void* kernel = plan_kernel_of(call.legacy != 0, call.threads);
    cudaError_t e = allow_smem(kernel, smem);
    if (e != cudaSuccess) return e;
    cudaLaunchAttribute attr[2];
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(call.nlocal * call.ctas_per_rank);
    cfg.blockDim = dim3(call.threads + (rehearses ? kRehearsalThreads : 0));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = attr;
    if (call.nlocal > 1) attr[cfg.numAttrs++] = plan_cluster(call.nlocal);
    if (pdl_enabled()) attr[cfg.numAttrs++] = dependent_launch();
    void* args[] = {&copy};
    count_launch();
    return cudaLaunchKernelExC(&cfg, kernel, args);
}

}  // namespace uep

// ------------------------------------------------------------------------------------
// C ABI: stateless entry points
// ------------------------------------------------------------------------------------
using namespace uep;

extern "C" {

int64_t uep_launch_count(void) { return g_launches.load(); }
void uep_reset_launch_count(void) { g_launches.store(0); }

static int histogram_common(int kind, const void* input, int T, int K_or_L, int L, int32_t* loads, void* stream_) {
    if (L <= 0 || L > 65536 || T < 0 || K_or_L < 0 || loads == nullptr) return fail(UEP_ERR_INVALID, "histogram: bad sizes");
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    UEP_CUDA_TRY(cudaMemsetAsync(loads, 0, sizeof(int32_t) * L, stream));
    const int64_t n = static_cast<int64_t>(T) * K_or_L;
    if (n == 0) return UEP_OK;
    if (input == nullptr) return fail(UEP_ERR_INVALID, "histogram: null input");
    const int ctas = plan_ctas_per_rank(kind, T, K_or_L, kPlanMaxCtas);
    const size_t smem = sizeof(int32_t) * L;
    UEP_CUDA_TRY(allow_smem(reinterpret_cast<const void*>(histogram_kernel), smem));
    count_launch();
    histogram_kernel<<<ctas, kHistThreads, smem, stream>>>(kind, input, T, K_or_L, L, loads);
    UEP_CUDA_TRY(cudaGetLastError());
    return UEP_OK;
}

int uep_histogram_ids32(const int32_t* ids, int64_t num_entries, int L, int32_t* loads, void* stream) {
    if (num_entries < 0 || num_entries > INT32_MAX) return fail(UEP_ERR_INVALID, "histogram: too many entries");
    return histogram_common(1, ids, static_cast<int>(num_entries), 1, L, loads, stream);
}
int uep_histogram_ids64(const int64_t* ids, int64_t num_entries, int L, int32_t* loads, void* stream) {
    if (num_entries < 0 || num_entries > INT32_MAX) return fail(UEP_ERR_INVALID, "histogram: too many entries");
    return histogram_common(2, ids, static_cast<int>(num_entries), 1, L, loads, stream);
}
int uep_histogram_map(const uint8_t* routing_map, int T, int L, int32_t* loads, void* stream) {
    return histogram_common(0, routing_map, T, L, L, loads, stream);
}

int uep_solve_placement(const int32_t* loads_per_rank, int32_t* global_loads_out, int32_t* p2l, int32_t* l2p,
                        int32_t* lcnts, int32_t* quota, int32_t* quota_prefix, int32_t* rank_quota_prefix,
                        int num_ranks, int nvl_ranks, int M, int R, int D, const uep_solver_params* params,
                        int my_rank, int32_t* status, void* stream_) {
    if (params == nullptr || loads_per_rank == nullptr || global_loads_out == nullptr)
        return fail(UEP_ERR_INVALID, "solve_placement: null argument (global_loads_out is required as workspace)");
    if (nvl_ranks <= 0 || num_ranks <= 0 || num_ranks % nvl_ranks != 0 || M <= 0 || R < 0 || D < 1)
        return fail(UEP_ERR_INVALID, "solve_placement: bad group shape");
    if (nvl_ranks * M > kMaxExpertsPerDomain || nvl_ranks > kMaxRanksPerDomain || nvl_ranks * R > kMaxExportsPerDomain)
        return fail(UEP_ERR_INVALID, "solve_placement: domain exceeds the static limits (512 experts, 72 ranks, 512 replicas)");
    if (D < (nvl_ranks < num_ranks ? nvl_ranks : num_ranks))
        return fail(UEP_ERR_INVALID, "solve_placement: max_replicas_dim smaller than the NVLink domain");
    if (my_rank < 0 || my_rank >= num_ranks) return fail(UEP_ERR_INVALID, "solve_placement: my_rank out of range");
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    SolveArgs a;
    a.global_loads = global_loads_out;
    a.loads_per_rank = loads_per_rank;
    a.p2l = p2l; a.l2p = l2p; a.lcnts = lcnts; a.quota = quota; a.quota_prefix = quota_prefix;
    a.rank_quota_prefix = rank_quota_prefix;
    a.physical_loads = nullptr;
    a.N = num_ranks; a.G = nvl_ranks; a.M = M; a.R = R; a.D = D;
    a.balance_threshold = params->balance_threshold;
    a.min_tokens = params->min_tokens_per_replica;
    a.allow_zero_master = params->allow_zero_master_quota;
    a.locality = params->locality_aware;
    a.eps = params->oracle_eps;
    a.my_rank = my_rank;
    a.preloaded = 0;
    a.staged_loads = nullptr;
    a.trace = nullptr;
    size_t smem = solver_smem_bytes(nvl_ranks * M, nvl_ranks, R) + 16;
    // with one domain the solver also keeps the load matrix it adds up, where that fits
    const size_t matrix = sizeof(int32_t) * num_ranks * num_ranks * static_cast<size_t>(M);
    const int staged = nvl_ranks == num_ranks && smem + matrix <= kSolveMaxSmem ? 1 : 0;
    if (staged) smem += matrix;
    UEP_CUDA_TRY(allow_smem(reinterpret_cast<const void*>(solve_kernel<false>), smem));
    count_launch();
    cudaLaunchAttribute attr[1] = {dependent_launch()};
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(num_ranks / nvl_ranks);
    cfg.blockDim = dim3(kSolveThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 1 : 0;
    UEP_CUDA_TRY(cudaLaunchKernelEx(&cfg, solve_kernel<false>, a, global_loads_out, 1, staged, reinterpret_cast<DeviceStatus*>(status)));
    return UEP_OK;
}

int uep_legacy_solve_placement(const int32_t* global_loads, int32_t* p2l, int32_t* l2p, int32_t* lcnts, int32_t* quota,
                               int32_t* quota_prefix, int32_t* rank_quota_prefix, int num_ranks, int nvl_ranks, int M,
                               int R, int D, float balance_threshold, int32_t* status, void* stream_) {
    if (global_loads == nullptr) return fail(UEP_ERR_INVALID, "legacy_solve_placement: null loads");
    if (nvl_ranks <= 0 || num_ranks <= 0 || num_ranks % nvl_ranks != 0 || M <= 0 || R < 0 || D < 1)
        return fail(UEP_ERR_INVALID, "legacy_solve_placement: bad group shape");
    if (nvl_ranks * M > kMaxExpertsPerDomain || nvl_ranks > kMaxRanksPerDomain || nvl_ranks * R > kMaxExportsPerDomain)
        return fail(UEP_ERR_INVALID, "legacy_solve_placement: domain exceeds the static limits (512 experts, 72 ranks, 512 replicas)");
    if (D < (nvl_ranks < num_ranks ? nvl_ranks : num_ranks))
        return fail(UEP_ERR_INVALID, "legacy_solve_placement: max_replicas_dim smaller than the NVLink domain");
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    SolveArgs a;
    std::memset(&a, 0, sizeof(a));
    a.global_loads = global_loads;
    a.p2l = p2l; a.l2p = l2p; a.lcnts = lcnts; a.quota = quota; a.quota_prefix = quota_prefix;
    a.rank_quota_prefix = rank_quota_prefix;
    a.N = num_ranks; a.G = nvl_ranks; a.M = M; a.R = R; a.D = D;
    a.balance_threshold = balance_threshold;
    const size_t smem = legacy_smem_bytes(nvl_ranks * M, nvl_ranks) + 16;
    UEP_CUDA_TRY(allow_smem(reinterpret_cast<const void*>(solve_kernel<true>), smem));
    count_launch();
    solve_kernel<true><<<num_ranks / nvl_ranks, kSolveThreads, smem, stream>>>(a, nullptr, 0, 0, reinterpret_cast<DeviceStatus*>(status));
    UEP_CUDA_TRY(cudaGetLastError());
    return UEP_OK;
}

int uep_init_master_placement(int32_t* p2l, int32_t* l2p, int32_t* lcnts, int32_t* quota, int32_t* quota_prefix,
                              int32_t* rank_quota_prefix, int num_ranks, int M, int R, int D, void* stream) {
    if (num_ranks <= 0 || M <= 0 || R < 0 || D < 1) return fail(UEP_ERR_INVALID, "init_master_placement: bad shape");
    const int work = num_ranks * M * D;
    const int grid = work / 256 + 1 > 64 ? 64 : work / 256 + 1;
    count_launch();
    init_master_kernel<<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(p2l, l2p, lcnts, quota, quota_prefix,
                                                                           rank_quota_prefix, num_ranks, M, R, D);
    UEP_CUDA_TRY(cudaGetLastError());
    return UEP_OK;
}

}  // extern "C"
