// Kernel 2 — reroute: logical expert ids -> physical replica ids under the rank's
// quota split, in dense ([T,L] -> [T,P]) and sparse ([T,K]) form, the dense backward
// gather, and the token-gradient row gather.
//
// The reference resolves the ordinal of a token inside its expert with one warp per
// (expert, 128-token tile) reading the bool map column-wise, and writes the [T,P]
// outputs twice (zero-fill, then scatter): csrc/kernels/reroute.cu:21-51, 138-264 and
// csrc/ultra_ep.cpp:891-892 of the reference. Here:
//   * sparse: one launch (ordinals.cuh); a cluster of CTAs keeps its entries in registers and
//     counts again what lies in front of it, where there is more than one. In place, with several ranks or with very many
//     entries a count kernel goes in front;
//   * dense: pass 1 counts per (tile, expert) from coalesced row reads; pass 2 turns the counts of
//     the preceding tiles into a base per expert, holds the tile as bit columns, turns logical
//     columns into physical ones and writes every output element exactly once out of registers
//     (zeros included), so no pre-zeroing pass exists.
// Results equal the reference's dense rule bit for bit; the sparse form applies the same
// rule per (token, k) entry and therefore is deterministic, which the reference's
// atomic-counter sparse kernel (reroute.cu:492-515) is not.

#include <algorithm>
#include <climits>
#include <cstdlib>
#include <mutex>
#include <string>
#include <utility>

#include "internal.h"
#include "ordinals.cuh"

namespace uep {

namespace {

constexpr int kRerouteThreads = 256;
constexpr size_t kMaxCtaSmem = 225 * 1024;  // of a CTA
constexpr size_t kSmemLimit = 227 * 1024;   // what the device gives to one
constexpr int kDenseTileRows = 64;
constexpr int kSparseTileEntries = 2048;  // entries of a row of the count table (at least)

// The interleave's stride for a total of two or more: the first number from total/2 + 1 upwards that has no factor in
// common with the total (csrc/kernels/reroute.cu:21-51 of the reference searches for it). With h = total/2,
// gcd(h + 1, 2h + 1) = 1 and gcd(h + 1, 2h) = gcd(h + 1, 2): only an odd h of an even total needs the next number, and
// gcd(h + 2, 2h) = gcd(h + 2, 4) = 1 then. A total of two leaves 1.
__device__ __forceinline__ int interleave_stride(int total) {
    const int h = total / 2;
    return total == 2 ? 1 : h + 1 + (((total & 1) == 0 && (h & 1)) ? 1 : 0);
}

// The first kStagedReps entries of every expert's plan rows (rank-quota prefixes and physical ids) are copied
// into shared memory once per CTA: resolving an entry then costs no global load. Experts with more instances
// than that read their rows from global memory.
constexpr int kStagedReps = 8;

// Routing parameters of an expert as the resolution wants them: a reciprocal for the remainder, and a staged prefix row
// whose unused entries are never reached, so that the replica index is eight comparisons without a loop bound.
struct FastRouter {
    int C;              // instances
    int total, stride, offset;  // stride 0: no interleave
    uint32_t recip;     // floor((2^32 - 1) / total)
};

// Rows of the plan of every expert into shared memory, asynchronously: all of them are asked for at once, whether
// the expert has that many instances or not (the rows are there), so that they cost one round trip beside the
// entries' own. The instance counts go where the routers will stand.
__device__ __forceinline__ void stage_plan_rows_async(const int32_t* __restrict__ lcnts, const int32_t* __restrict__ rqp,
                                                      const int32_t* __restrict__ l2p, int L, int D, bool quota_mode,
                                                      FastRouter* routers, int32_t* prefix_s, int32_t* l2p_s) {
    const int tid = threadIdx.x, nt = blockDim.x;
    for (int e = tid; e < L; e += nt) cp_async_4(&routers[e].C, lcnts + e);
    const bool vec = D >= kStagedReps && (D % 4) == 0 &&
                     ((reinterpret_cast<uintptr_t>(l2p) | reinterpret_cast<uintptr_t>(quota_mode ? rqp : l2p)) & 15u) == 0;
    if (vec) {
        for (int i = tid; i < L * (kStagedReps / 4); i += nt) {
            const int e = i / (kStagedReps / 4), j = i % (kStagedReps / 4) * 4;
            cp_async_16(l2p_s + e * kStagedReps + j, l2p + static_cast<int64_t>(e) * D + j);
            if (quota_mode) cp_async_16(prefix_s + e * kStagedReps + j, rqp + static_cast<int64_t>(e) * D + j);
        }
        return;
    }
    for (int i = tid; i < L * kStagedReps; i += nt) {
        const int e = i / kStagedReps, j = i % kStagedReps;
        if (j < D) {
            cp_async_4(l2p_s + i, l2p + static_cast<int64_t>(e) * D + j);
            if (quota_mode) cp_async_4(prefix_s + i, rqp + static_cast<int64_t>(e) * D + j);
        }
    }
}

// prefix_row: the expert's staged row (rewritten here), or null where rows are not staged.
__device__ __forceinline__ FastRouter make_fast_router(int e, int C, const int32_t* __restrict__ rqp, int D, bool quota_mode,
                                                       bool interleave, int32_t* prefix_row) {
    FastRouter r{C, 0, 0, 0, 0};
    if (C <= 1 || !quota_mode) return r;
    if (prefix_row != nullptr && C <= kStagedReps) {
        r.total = C <= D ? prefix_row[C - 1] : 0;
#pragma unroll
        for (int j = 0; j < kStagedReps; ++j) {
            if (j >= C - 1) prefix_row[j] = INT_MAX;  // the index ends at C - 1 whatever the last prefix says
            else if (j >= D) prefix_row[j] = 0;
        }
    } else {
        r.total = rqp[static_cast<int64_t>(e) * D + C - 1];
    }
    if (interleave && r.total > 1) {
        r.stride = interleave_stride(r.total);
        r.offset = e % r.total;
        r.recip = 0xFFFFFFFFu / static_cast<uint32_t>(r.total);
    }
    return r;
}

__device__ __noinline__ int mod_wide(unsigned long long x, int total) { return static_cast<int>(x % static_cast<unsigned long long>(total)); }

// ordinal -> replica index, for an expert with two or more instances.
__device__ __forceinline__ int fast_replica_index(const FastRouter& r, int ordinal, const int32_t* prefix_row,
                                                  const int32_t* __restrict__ rqp_row, bool quota_mode) {
    if (!quota_mode) return ordinal % r.C;
    int qr = ordinal;
    if (r.stride != 0) {
        const unsigned long long prod = static_cast<unsigned long long>(static_cast<unsigned>(ordinal)) * static_cast<unsigned>(r.stride) +
                                        static_cast<unsigned>(r.offset);
        if ((prod >> 32) == 0) {
            // x * recip >> 32 is the quotient or one less: 2^32 / total - recip <= 1, so the product falls short by less than 2^32
            const uint32_t x = static_cast<uint32_t>(prod), t = static_cast<uint32_t>(r.total);
            uint32_t rem = x - __umulhi(x, r.recip) * t;
            if (rem >= t) rem -= t;
            qr = static_cast<int>(rem);
        } else {
            qr = mod_wide(prod, r.total);
        }
    }
    int idx = 0;
    if (prefix_row != nullptr && r.C <= kStagedReps) {
        const int4 a = reinterpret_cast<const int4*>(prefix_row)[0], b = reinterpret_cast<const int4*>(prefix_row)[1];
        idx = (qr >= a.x) + (qr >= a.y) + (qr >= a.z) + (qr >= a.w) + (qr >= b.x) + (qr >= b.y) + (qr >= b.z) + (qr >= b.w);
    } else {
        for (int j = 0; j < r.C - 1; ++j) idx += (qr >= rqp_row[j]) ? 1 : 0;
    }
    return idx;
}

// ----------------------------------------------------------------------------- dense
// A tile is 64 rows. Its bool map is held as bit columns: byte [s][c] has bit i set where row 8s + i marks column c.
// Four columns of eight rows come from eight independent 4-byte loads and fit one word, so the map is read once,
// coalesced, and never staged; the rank of a cell among its column's marked rows is a population count.
constexpr int kDenseSegs = kDenseTileRows / 8;
static_assert(kDenseTileRows == 64, "a byte of counts and the 64-bit columns rely on it");

__device__ __forceinline__ uint32_t nonzero_bytes(uint32_t w) {  // 0x01 where a byte of w is not zero
    return ((((w & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | w) >> 7) & 0x01010101u;
}

__host__ __device__ __forceinline__ int pad4(int n) { return (n + 3) & ~3; }

// Rows 8s .. 8s+7 (those below `rows`) of columns 4q .. 4q+3 as four bytes of row bits, read with loads of W's size, which
// the address of the tile's first row and `cols` are multiples of.
template <typename W>
__device__ __forceinline__ uint32_t segment_bits(const uint8_t* __restrict__ tile, int rows, int cols, int s, int q) {
    constexpr int kLoads = 4 / sizeof(W);
    uint32_t acc = 0;
#pragma unroll
    for (int k = 0; k < kLoads; ++k) {
        const int c = 4 * q + k * static_cast<int>(sizeof(W));
        W w[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            w[i] = (8 * s + i < rows && c < cols) ? __ldg(reinterpret_cast<const W*>(tile + static_cast<int64_t>(8 * s + i) * cols + c)) : W(0);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) acc |= nonzero_bytes(static_cast<uint32_t>(w[i]) << (8 * sizeof(W) * k)) << i;
    }
    return acc;
}
__device__ __forceinline__ int map_load_bytes(const uint8_t* map, int cols) {
    const uintptr_t bits = reinterpret_cast<uintptr_t>(map) | static_cast<uintptr_t>(cols);
    return (bits & 3u) == 0 ? 4 : ((bits & 1u) == 0 ? 2 : 1);
}
__device__ __forceinline__ uint32_t segment_bits_any(int load_bytes, const uint8_t* __restrict__ tile, int rows, int cols, int s, int q) {
    if (load_bytes == 4) return segment_bits<uint32_t>(tile, rows, cols, s, q);
    if (load_bytes == 2) return segment_bits<uint16_t>(tile, rows, cols, s, q);
    return segment_bits<uint8_t>(tile, rows, cols, s, q);
}

// The bit columns of a tile of up to 8 * segs rows into bits[segs][pad4(cols)] (shared memory), all threads of the CTA.
__device__ __forceinline__ void tile_bit_columns(const uint8_t* __restrict__ tile, int rows, int segs, int cols, uint8_t* bits) {
    const int quads = pad4(cols) / 4, load_bytes = map_load_bytes(tile, cols);
    for (int i = threadIdx.x; i < quads * segs; i += blockDim.x) {
        const int s = i / quads, q = i - s * quads;
        reinterpret_cast<uint32_t*>(bits)[i] = segment_bits_any(load_bytes, tile, rows, cols, s, q);
    }
}

// The count of a (tile, expert) pair is at most kDenseTileRows = 64: it is kept in ONE BYTE of the scratch buffer, an expert's
// tiles side by side, so that a warp of the second kernel adds up the tiles in front of its own four to a load and four to an
// instruction, and only for the experts that need it. Rows of four tiles and more are padded to 16 bytes (the scratch has an
// int32 for each pair).
__host__ __device__ __forceinline__ int count_stride(int tiles) { return tiles >= 4 ? (tiles + 15) & ~15 : 4; }
__host__ __device__ __forceinline__ int dense_tiles(int T) { return (T + kDenseTileRows - 1) / kDenseTileRows; }

// L is a multiple of 16 with L/16 in {1,2,4,...,32} and the map 16-byte aligned: a thread then always meets the same sixteen
// columns and can add map bytes as packed words.
__device__ __forceinline__ bool dense_fast_path(const uint8_t* map, int L) {
    const int G = L / 16;
    return (L % 16 == 0) && G <= 32 && (G & (G - 1)) == 0 && (reinterpret_cast<uintptr_t>(map) & 15u) == 0;
}

// TILES tiles a CTA: one or four (launch_dense_forward).
constexpr int kCountCtasPerSm = 5;  // at 48 registers
template <int TILES>
__global__ void __launch_bounds__(kRerouteThreads, kCountCtasPerSm) dense_count_kernel(Batch<DenseFwdArgs> batch, int L, int wait_first, int next_early) {
    if (wait_first) pdl_wait();  // ahead of every read: the kernel in front may still be writing the map
    if (next_early) pdl_launch_dependents();  // the scatter kernel may start its prologue now
    extern __shared__ __align__(128) char smem_raw[];  // [TILES][pad4(L)] counts, one byte each
    constexpr int kThreads = kRerouteThreads / TILES;  // of a tile: whole warps
    const DenseFwdArgs& a = batch.a[blockIdx.y];
    const int T = a.T, tiles = dense_tiles(T), words = pad4(L) / 4;
    const int first = blockIdx.x * TILES;
    if (first >= tiles) return;
    const int mine = threadIdx.x / kThreads, tid = threadIdx.x % kThreads;
    const int r0 = min((first + mine) * kDenseTileRows, T), rows = min(T - r0, kDenseTileRows);
    const uint8_t* src = a.map + static_cast<int64_t>(r0) * L;
    for (int i = threadIdx.x; i < words * TILES; i += blockDim.x) reinterpret_cast<uint32_t*>(smem_raw)[i] = 0;
    __syncthreads();
    uint32_t* cnt = reinterpret_cast<uint32_t*>(smem_raw) + mine * words;
    // a byte never exceeds 64, so the packed adds below cannot carry into the next byte
    if (dense_fast_path(a.map, L)) {
        constexpr int kFlight = TILES == 1 ? 4 : 8;
        const int G = L / 16;
        // vector i of the tile covers row i / G, columns 16 * (i % G) ..; kThreads is a multiple of G, so a
        // thread always meets the same column group and adds the 0/1 bytes of its rows as packed words
        const int nvec = rows * G;
        uint4 acc = make_uint4(0, 0, 0, 0);
        for (int i = tid; i < nvec; i += kFlight * kThreads) {
            uint4 v[kFlight];
#pragma unroll
            for (int u = 0; u < kFlight; ++u) {
                const int at = i + u * kThreads;
                v[u] = at < nvec ? ld_global_nc_v4(src + static_cast<int64_t>(at) * 16) : make_uint4(0, 0, 0, 0);
            }
#pragma unroll
            for (int u = 0; u < kFlight; ++u) {
                acc.x += v[u].x; acc.y += v[u].y; acc.z += v[u].z; acc.w += v[u].w;
            }
        }
        // lanes with the same column group inside the warp
        for (int d = G; d < 32; d <<= 1) {
            acc.x += __shfl_xor_sync(kFullMask, acc.x, d); acc.y += __shfl_xor_sync(kFullMask, acc.y, d);
            acc.z += __shfl_xor_sync(kFullMask, acc.z, d); acc.w += __shfl_xor_sync(kFullMask, acc.w, d);
        }
        const int lane = threadIdx.x & 31;
        if (lane < G) {
            atomicAdd(cnt + lane * 4 + 0, acc.x); atomicAdd(cnt + lane * 4 + 1, acc.y);
            atomicAdd(cnt + lane * 4 + 2, acc.z); atomicAdd(cnt + lane * 4 + 3, acc.w);
        }
    } else {
        const int load_bytes = map_load_bytes(src, L);
        for (int i = tid; i < words * kDenseSegs; i += kThreads) {
            const int s = i / words, q = i - s * words;
            const uint32_t b = segment_bits_any(load_bytes, src, rows, L, s, q);
            uint32_t packed = 0;
#pragma unroll
            for (int k = 0; k < 4; ++k) packed |= static_cast<uint32_t>(__popc((b >> (8 * k)) & 0xFFu)) << (8 * k);
            if (packed) atomicAdd(cnt + q, packed);
        }
    }
    __syncthreads();
    const uint8_t* bytes = reinterpret_cast<const uint8_t*>(smem_raw);
    const int stride = count_stride(tiles);
    uint8_t* counts = reinterpret_cast<uint8_t*>(a.scratch) + first;
    for (int e = threadIdx.x; e < L; e += blockDim.x) {
        if (TILES == 1) {
            counts[static_cast<int64_t>(e) * stride] = bytes[e];
        } else {
            uint32_t w = 0;
#pragma unroll
            for (int k = 0; k < TILES; ++k) w |= static_cast<uint32_t>(bytes[k * 4 * words + e]) << (8 * k);
            *reinterpret_cast<uint32_t*>(counts + static_cast<int64_t>(e) * stride) = w;
        }
    }
}

// Tokens of the tiles in front of `tile` in an expert's row of counts, by one warp.
__device__ __forceinline__ int sum_earlier_tiles(const uint8_t* counts, int tile, int lane) {
    uint32_t sum = 0;
    for (int t = 4 * lane; t < tile; t += 4 * kWarp) {
        uint32_t w = __ldcg(reinterpret_cast<const uint32_t*>(counts + t));
        if (tile - t < 4) w &= (1u << (8 * (tile - t))) - 1u;
        sum = __dp4a(w, 0x01010101u, sum);
    }
    return warp_sum(static_cast<int>(sum));
}

// Second kernel: one CTA per tile of 64 tokens. The logical bit columns become physical ones (an expert with one
// instance: its column is copied; with several: a warp resolves the column's marked rows), and then a thread owns four
// physical columns of four rows and writes them out of its registers: a probability is read where its bit is set,
// zeros are written elsewhere. Outputs wider than kDenseMaxChunkCols go in column chunks.
// What is done for every expert is little: its one physical column, or that it
// has several. Plan rows, the router and the tiles in front are looked up for an expert with several that the tile routes to, by
// the warp that resolves it, in a few words of its own; shared memory is 4 KB at 128 experts. With all plan rows staged, all
// experts' tiles added up by every CTA (15 KB) and eight rows a thread, and like this (us): the pair for eight ranks of 8192 tokens
// and 128 experts 30.0 and 27.3, of 4096 17.0 and 13.7; step of 8192 x 128 with bf16 experts of 9 MB 67.1 and 64.2, of 2000 x 256 with
// 3 MB 52.3 and 49.4; one rank of 8191 x 256, sparse, dense and backward, 31.9 and 27.9. 64 registers and three spilled words: with 40 (six CTAs an SM) 17.7,
// with 32 28. Marked cells written over zeros in memory are partial sectors, and rows gathered in shared memory and sent as
// bulk stores wait too long for each other: both slower. So were all experts with several resolved together, marks shared by the lanes
// (38.0 to 38.9), though that is fewer instructions. A tile's 9.8 us among 591 others: 4 until its bits are physical, 5 to write.
constexpr int kDenseMaxChunkCols = 4096;
constexpr int kDenseMaxExperts = 1340;
constexpr int kDenseMaxThreads = 512;
constexpr int kNoPlace = -1, kSeveralPlaces = -2;

struct DenseRows {  // of the expert that a warp resolves
    int32_t prefix[kStagedReps], l2p[kStagedReps];
};
struct DenseShared {
    DenseRows* rows;      // [warps]
    int32_t* place;       // [pad4(L)] physical id of an expert with one instance, or one of the constants above
    uint8_t* bits;        // [kDenseSegs][pad4(L)]
    uint8_t* phys_bits;   // [kDenseSegs][pad4(chunk)]
    uint16_t* expert_of;  // [pad4(chunk)] valid where a bit is set
    uint16_t* several;    // [L] experts with several instances that the tile routes to
};
__host__ __device__ inline size_t dense_smem_bytes(int L, int chunk_cols, int threads) {
    const size_t Lq = pad4(L), Cq = pad4(chunk_cols);
    return sizeof(DenseRows) * (threads / kWarp) + Lq * (4 + kDenseSegs + 2) + Cq * (kDenseSegs + 2);
}
__device__ __forceinline__ DenseShared carve_dense_smem(char* raw, int L, int chunk_cols) {
    const int Lq = pad4(L), Cq = pad4(chunk_cols);
    DenseShared s;
    s.rows = reinterpret_cast<DenseRows*>(raw);
    s.place = reinterpret_cast<int32_t*>(s.rows + blockDim.x / kWarp);
    s.bits = reinterpret_cast<uint8_t*>(s.place + Lq);
    s.phys_bits = s.bits + Lq * kDenseSegs;
    s.expert_of = reinterpret_cast<uint16_t*>(s.phys_bits + Cq * kDenseSegs);
    s.several = s.expert_of + Cq;
    return s;
}

template <int V>
struct DenseVec;
template <>
struct DenseVec<4> {
    using F = float4;
    using B = uint32_t;
};
template <>
struct DenseVec<2> {
    using F = float2;
    using B = uint16_t;
};
template <>
struct DenseVec<1> {
    using F = float;
    using B = uint8_t;
};

// Columns [p_lo, p_lo + cols) of the tile's rows, V columns and four rows per thread and turn.
template <int V>
__device__ __forceinline__ void write_dense_chunk(const DenseShared& s, const float* __restrict__ probs, float* __restrict__ out_probs,
                                                  uint8_t* __restrict__ out_map, int rows, int L, int P, int p_lo, int cols) {
    using F = typename DenseVec<V>::F;
    using B = typename DenseVec<V>::B;
    constexpr int kRows = 4;
    const int groups = cols / V, Cq = pad4(cols);
    const int turns = groups * ((rows + kRows - 1) / kRows);
    const uint32_t per_group = 0xFFFFFFFFu / static_cast<uint32_t>(groups) + 1u;  // i / groups, exact for i < 2^16; 0: one group
    for (int i = threadIdx.x; i < turns; i += blockDim.x) {
        const int strip = per_group != 0 ? static_cast<int>(__umulhi(static_cast<uint32_t>(i), per_group)) : i;
        const int c = (i - strip * groups) * V, r0 = strip * kRows;
        // byte k: the rows of column c + k
        const uint32_t bits = static_cast<uint32_t>(*reinterpret_cast<const B*>(s.phys_bits + r0 / 8 * Cq + c)) >> r0 % 8;
        unsigned from[V];
#pragma unroll
        for (int k = 0; k < V; ++k) from[k] = static_cast<unsigned>(r0 * L) + s.expert_of[c + k];
        float v[kRows][V];
#pragma unroll
        for (int r = 0; r < kRows; ++r) {
#pragma unroll
            for (int k = 0; k < V; ++k) v[r][k] = (bits >> (8 * k + r)) & 1u ? __ldg(probs + (from[k] + static_cast<unsigned>(r * L))) : 0.f;
        }
        float* to = out_probs + static_cast<int64_t>(r0) * P + p_lo + c;
        uint8_t* to_map = out_map + static_cast<int64_t>(r0) * P + p_lo + c;
#pragma unroll
        for (int r = 0; r < kRows; ++r) {
            if (r0 + r < rows) {
                F f;
#pragma unroll
                for (int k = 0; k < V; ++k) reinterpret_cast<float*>(&f)[k] = v[r][k];
                *reinterpret_cast<F*>(to) = f;
                *reinterpret_cast<B*>(to_map) = static_cast<B>((bits >> r) & 0x01010101u);
            }
            to += P;
            to_map += P;
        }
    }
}

__global__ void __launch_bounds__(kDenseMaxThreads, 2)
dense_scatter_kernel(Batch<DenseFwdArgs> batch, int L, int P, int D, int quota_mode, int interleave, int chunk_cols,
                     int overlapped, int wait_first) {
    if (wait_first) pdl_wait();  // the count kernel waited for what was in front of it, this one for both
    const DenseFwdArgs& a = batch.a[blockIdx.y];
    const int T = a.T;
    const int tile = blockIdx.x;
    const int r0 = tile * kDenseTileRows, rows = min(T - r0, kDenseTileRows);
    if (rows <= 0) return;
    extern __shared__ __align__(128) char smem_raw[];
    __shared__ int n_several;
    const DenseShared s = carve_dense_smem(smem_raw, L, chunk_cols);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, warps = blockDim.x / kWarp, Lq = pad4(L);

    // ---- nothing here depends on the count kernel ------------------------------------------------
    for (int i = tid; i < pad4(chunk_cols) / 4 * kDenseSegs; i += blockDim.x) reinterpret_cast<uint32_t*>(s.phys_bits)[i] = 0;
    if (tid == 0) n_several = 0;
    {
        auto place_of = [&](int C, int p) { return C > 1 ? kSeveralPlaces : (C == 1 && p >= 0 && p < P ? p : kNoPlace); };
        int C = 0, p = 0;  // asked for beside the map
        if (tid < L) {
            C = a.lcnts[tid];
            p = a.l2p[static_cast<int64_t>(tid) * D];
        }
        tile_bit_columns(a.map + static_cast<int64_t>(r0) * L, rows, kDenseSegs, L, s.bits);
        if (tid < L) s.place[tid] = place_of(C, p);
        for (int e = tid + blockDim.x; e < L; e += blockDim.x) s.place[e] = place_of(a.lcnts[e], a.l2p[static_cast<int64_t>(e) * D]);
    }
    __syncthreads();

    const float* probs = a.probs + static_cast<int64_t>(r0) * L;
    float* out_probs = a.out_probs + static_cast<int64_t>(r0) * P;
    uint8_t* out_map = a.out_map + static_cast<int64_t>(r0) * P;
    const uint8_t* counts = reinterpret_cast<const uint8_t*>(a.scratch);
    const int stride = count_stride(dense_tiles(T));
    for (int p_lo = 0; p_lo < P; p_lo += chunk_cols) {
        const int cols = min(chunk_cols, P - p_lo), Cq = pad4(cols);
        if (p_lo > 0) {
            __syncthreads();
            for (int i = tid; i < Cq / 4 * kDenseSegs; i += blockDim.x) reinterpret_cast<uint32_t*>(s.phys_bits)[i] = 0;
            __syncthreads();
        }
        for (int e = tid; e < L; e += blockDim.x) {  // experts with one instance; the first time also the list of the others
            const int place = s.place[e], p = place - p_lo;
            const bool single = place >= 0 && p >= 0 && p < cols;
            if (!single && (p_lo > 0 || place != kSeveralPlaces)) continue;
            uint32_t b[kDenseSegs], any = 0;
#pragma unroll
            for (int g = 0; g < kDenseSegs; ++g) {
                b[g] = s.bits[g * Lq + e];
                any |= b[g];
            }
            if (any == 0) continue;  // a caller's table may have the column for another expert too, which the tile routes to
            if (!single) {
                s.several[atomicAdd(&n_several, 1)] = static_cast<uint16_t>(e);
                continue;
            }
#pragma unroll
            for (int g = 0; g < kDenseSegs; ++g) {
                if (b[g] != 0) s.phys_bits[g * Cq + p] = static_cast<uint8_t>(b[g]);
            }
            s.expert_of[p] = static_cast<uint16_t>(e);
        }
        if (p_lo == 0 && overlapped) pdl_wait();
        __syncthreads();  // the list of experts with several; the bytes above share words with the atomics below
        for (int i = warp; i < n_several; i += warps) {
            const int e = s.several[i];
            const int64_t row = static_cast<int64_t>(e) * D;
            DenseRows& plan = s.rows[warp];
            const int C = a.lcnts[e];
            const int prefix = lane < min(D, kStagedReps) && quota_mode ? a.rqp[row + lane] : 0;
            const int phys = lane < min(D, kStagedReps) ? a.l2p[row + lane] : -1;
            int before = sum_earlier_tiles(counts + static_cast<int64_t>(e) * stride, tile, lane);
            __syncwarp();  // the expert before this one has been resolved
            if (lane < kStagedReps) {
                plan.prefix[lane] = prefix;
                plan.l2p[lane] = phys;
            }
            __syncwarp();
            FastRouter router{};
            if (lane == 0) router = make_fast_router(e, C, a.rqp, D, quota_mode != 0, interleave != 0, plan.prefix);
            router.C = C;
            router.total = __shfl_sync(kFullMask, router.total, 0);
            router.stride = __shfl_sync(kFullMask, router.stride, 0);
            router.offset = __shfl_sync(kFullMask, router.offset, 0);
            router.recip = __shfl_sync(kFullMask, router.recip, 0);
            __syncwarp();
#pragma unroll
            for (int half = 0; half < 2; ++half) {  // lane t: row 32 * half + t
                uint32_t m = 0;
#pragma unroll
                for (int g = 0; g < 4; ++g) m |= static_cast<uint32_t>(s.bits[(4 * half + g) * Lq + e]) << (8 * g);
                if ((m >> lane) & 1u) {
                    const int ordinal = before + __popc(m & ((1u << lane) - 1u));
                    const int j = fast_replica_index(router, ordinal, plan.prefix, a.rqp + row, quota_mode != 0);
                    const int p = (j < kStagedReps ? plan.l2p[j] : a.l2p[row + j]) - p_lo;
                    if (p >= 0 && p < cols) {
                        const int seg = 4 * half + lane / 8;
                        atomicOr(reinterpret_cast<uint32_t*>(s.phys_bits + seg * Cq) + p / 4, 1u << (8 * (p & 3) + (lane & 7)));
                        s.expert_of[p] = static_cast<uint16_t>(e);
                    }
                }
                before += __popc(m);
            }
        }
        __syncthreads();
        const uintptr_t fp = reinterpret_cast<uintptr_t>(out_probs), mp = reinterpret_cast<uintptr_t>(out_map);
        if (P % 4 == 0 && (fp & 15u) == 0 && (mp & 3u) == 0) write_dense_chunk<4>(s, probs, out_probs, out_map, rows, L, P, p_lo, cols);
        else if (P % 2 == 0 && (fp & 7u) == 0 && (mp & 1u) == 0) write_dense_chunk<2>(s, probs, out_probs, out_map, rows, L, P, p_lo, cols);
        else write_dense_chunk<1>(s, probs, out_probs, out_map, rows, L, P, p_lo, cols);
    }
}

__device__ __forceinline__ float routed_grad(const float* __restrict__ grad_expanded, const uint8_t* __restrict__ expanded_map,
                                             const int32_t* __restrict__ l2p, const int32_t* __restrict__ lcnts, int64_t t,
                                             int l, int P, int D) {
    const int C = lcnts[l];
    for (int r = 0; r < C; ++r) {
        const int phys = l2p[static_cast<int64_t>(l) * D + r];
        if (expanded_map[t * P + phys]) return grad_expanded[t * P + phys];
    }
    return 0.f;
}

// The marked cells of a warp's 32 words of row bits (one word per lane), 32 cells at a time: every lane gets the lane that
// holds its cell and the bit there. The few marked cells are so shared evenly by the lanes; a loop over the bits of the own
// word runs as long as the fullest of 32 words.
template <typename F>
__device__ __forceinline__ void for_each_marked(uint32_t word, F&& cell) {
    const int lane = threadIdx.x & 31;
    int upto = __popc(word);
#pragma unroll
    for (int d = 1; d < kWarp; d <<= 1) {
        const int x = __shfl_up_sync(kFullMask, upto, d);
        if (lane >= d) upto += x;
    }
    const int total = __shfl_sync(kFullMask, upto, kWarp - 1);
    for (int first = 0; first < total; first += kWarp) {
        int n = first + lane, src = 0;  // the first lane whose inclusive sum is above n
#pragma unroll
        for (int d = kWarp / 2; d > 0; d >>= 1) src += __shfl_sync(kFullMask, upto, src + d - 1) <= n ? d : 0;
        const bool active = n < total;
        const uint32_t w = __shfl_sync(kFullMask, word, src);
        n -= __shfl_sync(kFullMask, upto, src) - __popc(w);
        int bit = 0;  // of the n-th marked cell of w
#pragma unroll
        for (int width = 16; width > 0; width >>= 1) {
            const int c = __popc((w >> bit) & ((1u << width) - 1u));
            if (n >= c) {
                n -= c;
                bit += width;
            }
        }
        cell(active, src, bit & 31);
    }
}

// Zeros by all threads of the CTA, 16 bytes a store: `where` is 16-byte aligned.
__device__ __forceinline__ void zero_fill(void* where, int vecs) {
    uint4* v = static_cast<uint4*>(where) + threadIdx.x;
    int left = vecs - static_cast<int>(threadIdx.x);
    for (; left > 3 * static_cast<int>(blockDim.x); left -= 4 * blockDim.x, v += 4 * blockDim.x) {
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u * blockDim.x] = make_uint4(0, 0, 0, 0);
    }
    for (; left > 0; left -= blockDim.x, v += blockDim.x) *v = make_uint4(0, 0, 0, 0);
}

// `bytes` bytes into shared memory (16-byte aligned there), asynchronously where the source is aligned.
__device__ __forceinline__ void stage_bytes(uint8_t* dst, const uint8_t* __restrict__ src, int bytes) {
    const uintptr_t bits = reinterpret_cast<uintptr_t>(src) | static_cast<uintptr_t>(bytes);
    if ((bits & 15u) == 0) {
        for (int i = threadIdx.x * 16; i < bytes; i += blockDim.x * 16) cp_async_16(dst + i, src + i);
    } else if ((bits & 3u) == 0) {
        for (int i = threadIdx.x * 4; i < bytes; i += blockDim.x * 4) cp_async_4(dst + i, src + i);
    } else {
        for (int i = threadIdx.x; i < bytes; i += blockDim.x) dst[i] = __ldg(src + i);
    }
}

// Which of the 32 columns from `c` on are marked in a row of `cols` bytes, a multiple of four, in shared memory.
__device__ __forceinline__ uint32_t row_bits(const uint8_t* row, int c, int cols) {
    uint32_t bits = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const uint32_t marks = c + 4 * k < cols ? nonzero_bytes(*reinterpret_cast<const uint32_t*>(row + c + 4 * k)) : 0u;
        bits |= (marks * 0x10204080u) >> 28 << (4 * k);  // four bytes of 0 or 1 to four bits
    }
    return bits;
}

// Backward of a tile of `tile_rows` tokens: the rows of both maps are copied to shared memory, the output is filled with
// zeros, and the marked cells (topk of them a token) are shared by the lanes: a cell looks its instances up in the expanded
// row, fetches one gradient and stores it over the zero. L is a multiple of four and the output 16-byte aligned. Every step
// waits for memory, so occupancy counts: 32 registers, and eight CTAs an SM up to 28 KB of staged rows (23 KB at 128 experts
// and 160 slots; four CTAs at the 56 KB that the dispatch allows rows of more than eight tokens).
// Both maps as bit columns and four columns of eight rows per thread took 14 M instructions a call of eight ranks of 8192
// tokens and 128 experts, two thirds of the issue slots: 24.8 us a call, 18.3 like this (20.7 with four CTAs an SM); one
// rank of 16384 tokens and 256 experts 12.3 (a thread per four cells 19.3).
constexpr int kDenseBwdThreads = 256;

__host__ __device__ inline size_t dense_bwd_smem_bytes(int L, int P, int tile_rows) {
    return static_cast<size_t>(pad4(L)) * (kStagedReps + 1) * 4 + static_cast<size_t>(tile_rows) * (L + P) + 16;
}
__global__ void __launch_bounds__(kDenseBwdThreads, 8)
dense_backward_tile_kernel(Batch<DenseBwdArgs> batch, int L, int P, int D, int tile_rows, int wait_first) {
    if (wait_first) pdl_wait();  // ahead of every read
    const DenseBwdArgs& a = batch.a[blockIdx.y];
    const int first = static_cast<int>(blockIdx.x) * tile_rows;
    const int rows = min(a.T - first, tile_rows);
    if (rows <= 0) return;
    const int64_t r0 = first;
    extern __shared__ __align__(128) char smem_raw[];
    int32_t* l2p_s = reinterpret_cast<int32_t*>(smem_raw);
    int32_t* count_s = l2p_s + pad4(L) * kStagedReps;
    uint8_t* map_s = reinterpret_cast<uint8_t*>(count_s + pad4(L));
    uint8_t* expanded_s = map_s + (tile_rows * L + 15) / 16 * 16;
    const float* grads = a.grad_expanded + r0 * P;
    float* out = a.grad_probs + r0 * L;
    stage_bytes(map_s, a.map + r0 * L, rows * L);
    stage_bytes(expanded_s, a.expanded_map + r0 * P, rows * P);
    for (int e = threadIdx.x; e < L; e += blockDim.x) cp_async_4(count_s + e, a.lcnts + e);
    if (D >= kStagedReps && D % 4 == 0 && (reinterpret_cast<uintptr_t>(a.l2p) & 15u) == 0) {
        for (int i = threadIdx.x; i < L * (kStagedReps / 4); i += blockDim.x) {
            cp_async_16(l2p_s + i * 4, a.l2p + static_cast<int64_t>(i / (kStagedReps / 4)) * D + i % (kStagedReps / 4) * 4);
        }
    } else {
        for (int i = threadIdx.x; i < L * kStagedReps; i += blockDim.x) {
            if (i % kStagedReps < D) cp_async_4(l2p_s + i, a.l2p + static_cast<int64_t>(i / kStagedReps) * D + i % kStagedReps);
        }
    }
    zero_fill(out, rows * L / 4);
    cp_async_wait();
    __syncthreads();  // the zeros are in front of the stores below, too
    const int groups = (L + 31) / 32, tasks = rows * groups, lane = threadIdx.x & 31;
    float held = 0.f;  // a lane's last gradient, stored once its next one is on the way
    int held_at = -1;
    for (int i0 = threadIdx.x - lane; i0 < tasks; i0 += blockDim.x) {
        const int i = i0 + lane, my_row = i / groups, my_group = i - my_row * groups;
        const uint32_t word = i < tasks ? row_bits(map_s + my_row * L, 32 * my_group, L) : 0u;
        for_each_marked(word, [&](bool active, int src, int bit) {
            const int place = __shfl_sync(kFullMask, my_row << 16 | my_group, src);
            float g = 0.f;
            int at = -1;
            if (active) {
                const int row = place >> 16, l = 32 * (place & 0xFFFF) + bit, C = count_s[l];
                const uint8_t* took = expanded_s + row * P;
                int phys = -1;
                for (int j = 0; j < C && phys < 0; ++j) {
                    const int p = j < kStagedReps ? l2p_s[l * kStagedReps + j] : __ldg(a.l2p + static_cast<int64_t>(l) * D + j);
                    if (p >= 0 && p < P && took[p] != 0) phys = p;
                }
                if (phys >= 0) {
                    g = __ldg(grads + row * P + phys);
                    at = row * L + l;
                }
            }
            if (held_at >= 0) out[held_at] = held;
            held = g;
            held_at = at;
        });
    }
    if (held_at >= 0) out[held_at] = held;
}

// One thread per four logical experts of a token when the rows allow it (L a multiple of 4, map rows 4-byte and
// gradient rows 16-byte aligned): the routing map is read a word at a time and the gradients leave as float4.
// Most entries are not routed, so the kernel is a zero fill plus a few gathers.
__global__ void __launch_bounds__(kRerouteThreads) dense_backward_kernel(Batch<DenseBwdArgs> batch, int L, int P, int D, int wait_first) {
    if (wait_first) pdl_wait();  // ahead of every read
    const DenseBwdArgs& a = batch.a[blockIdx.y];
    const float* __restrict__ grad_expanded = a.grad_expanded;
    const uint8_t* __restrict__ map = a.map;
    const uint8_t* __restrict__ expanded_map = a.expanded_map;
    const int32_t* __restrict__ l2p = a.l2p;
    const int32_t* __restrict__ lcnts = a.lcnts;
    float* __restrict__ grad_probs = a.grad_probs;
    const int64_t total = static_cast<int64_t>(a.T) * L;
    const int64_t gtid = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    const int64_t gsize = static_cast<int64_t>(gridDim.x) * blockDim.x;
    const bool vec = (L % 4 == 0) && ((reinterpret_cast<uintptr_t>(map) & 3u) == 0) &&
                     ((reinterpret_cast<uintptr_t>(grad_probs) & 15u) == 0);
    if (vec) {
        const int groups = L / 4;
        for (int64_t q = gtid; q < total / 4; q += gsize) {
            const uint32_t m = __ldg(reinterpret_cast<const uint32_t*>(map) + q);
            float4 g = make_float4(0.f, 0.f, 0.f, 0.f);
            if (m != 0) {
                const int64_t t = q / groups;
                const int l0 = static_cast<int>(q % groups) * 4;
                if (m & 0x000000FFu) g.x = routed_grad(grad_expanded, expanded_map, l2p, lcnts, t, l0, P, D);
                if (m & 0x0000FF00u) g.y = routed_grad(grad_expanded, expanded_map, l2p, lcnts, t, l0 + 1, P, D);
                if (m & 0x00FF0000u) g.z = routed_grad(grad_expanded, expanded_map, l2p, lcnts, t, l0 + 2, P, D);
                if (m & 0xFF000000u) g.w = routed_grad(grad_expanded, expanded_map, l2p, lcnts, t, l0 + 3, P, D);
            }
            reinterpret_cast<float4*>(grad_probs)[q] = g;
        }
        return;
    }
    for (int64_t idx = gtid; idx < total; idx += gsize) {
        float g = 0.f;
        if (map[idx]) g = routed_grad(grad_expanded, expanded_map, l2p, lcnts, idx / L, static_cast<int>(idx % L), P, D);
        grad_probs[idx] = g;
    }
}

// ---------------------------------------------------------------------------- sparse
template <typename IdT>
__global__ void __launch_bounds__(kOrdThreads) sparse_count_kernel(Batch<SparseArgs> batch, int K, int L, int tile_entries, int wait_first,
                                                                   int next_early) {
    if (wait_first) pdl_wait();  // ahead of every read: the kernel in front may still be writing the ids
    if (next_early) pdl_launch_dependents();  // the reroute kernel may start on everything that does not read the table
    const SparseArgs& a = batch.a[blockIdx.y];
    count_tile<IdT>(static_cast<const IdT*>(a.ids), static_cast<int64_t>(a.T) * K, L, false, tile_entries, a.scratch);
}

// shared memory: prefix rows [L][8] i32 | l2p rows [L][8] i32 (both only where they fit) | ordinals | routers[L]
size_t sparse_smem_bytes(int L, bool rows_staged) {
    return (rows_staged ? static_cast<size_t>(L) * 2 * kStagedReps * 4 : 0) + ord_smem_bytes(L, kOrdThreads) + sizeof(FastRouter) * static_cast<size_t>(L);
}

// ids may alias out (every entry is read and written by the same thread, and nobody else reads it once the first is written).
// 512 threads at <= 96 registers and ~144*L bytes of shared memory leave room for this CTA on an SM that a weight_sync
// CTA occupies.
template <int EPT, typename IdT>
__global__ void __launch_bounds__(kOrdThreads) __maxnreg__(EPT > 4 ? 96 : 64)
sparse_reroute_kernel(Batch<SparseArgs> batch, int ctas, int K, int L, int D, int interleave, int rows_staged, int use_table, int wait_first) {
    extern __shared__ __align__(128) char smem_raw[];
    if (wait_first) pdl_wait();  // ahead of every read
    const SparseArgs& a = batch.a[blockIdx.y];
    const IdT* ids = static_cast<const IdT*>(a.ids);
    IdT* out = static_cast<IdT*>(a.out);
    const int64_t n = static_cast<int64_t>(a.T) * K;
    if (n == 0) return;  // every CTA of the rank
    const bool quota_mode = interleave != 2;  // 2: round-robin (legacy placement)
    int32_t* prefix_s = reinterpret_cast<int32_t*>(smem_raw);
    int32_t* l2p_s = prefix_s + static_cast<size_t>(L) * kStagedReps;
    const OrdShared o = carve_ord_smem(rows_staged ? reinterpret_cast<char*>(l2p_s + static_cast<size_t>(L) * kStagedReps) : smem_raw, L);
    FastRouter* routers = reinterpret_cast<FastRouter*>(o.counters + kOrdWarps * ord_row(L));
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (rows_staged) stage_plan_rows_async(a.lcnts, a.rqp, a.l2p, L, D, quota_mode, routers, prefix_s, l2p_s);

    int64_t begin, end;
    int iters;
    uint32_t packed[EPT];
    cluster_ordinals<EPT, false, IdT>(
        ids, n, L, false, ctas, use_table ? a.scratch : nullptr, o, begin, end, iters, packed,
        [&]() {
            for (int e = tid; e < L; e += kOrdThreads) {
                const int C = rows_staged ? routers[e].C : a.lcnts[e];
                routers[e] = make_fast_router(e, C, a.rqp, D, quota_mode, interleave == 1, rows_staged ? prefix_s + e * kStagedReps : nullptr);
            }
        },
        [&](int b, int base, int) { o.base[b] = base; });
    if (ctas > 1) cluster_arrive();
#pragma unroll
    for (int i = 0; i < EPT; ++i) {
        const int64_t at = begin + i * kWarp + lane;
        if (i >= iters || at >= end) continue;
        const uint32_t p = packed[i];
        const int b = static_cast<int>(p & 0xFFFFu);
        const int C = p != 0xFFFFFFFFu ? routers[b].C : 0;
        if (C <= 0) {  // an id outside [0, L), or an expert that maps nothing: the id stays
            if (out != ids) out[at] = ids[at];
            continue;
        }
        int j = 0;
        if (C > 1) {
            const int ordinal = o.base[b] + o.counters[warp * ord_row(L) + b] + static_cast<int>(p >> 16);
            j = fast_replica_index(routers[b], ordinal, rows_staged ? prefix_s + b * kStagedReps : nullptr,
                                   a.rqp + static_cast<int64_t>(b) * D, quota_mode);
        }
        out[at] = static_cast<IdT>(rows_staged && j < kStagedReps ? l2p_s[b * kStagedReps + j] : a.l2p[static_cast<int64_t>(b) * D + j]);
    }
    if (ctas > 1) cluster_wait();
}

// Several ranks in one launch beside weight_sync: a warp walks its entries, 32 at a time. Slower by itself than the kernel
// above, but thin: plain loads where they are needed, one after another. The kernel above finishes within the microseconds in
// which weight_sync's CTAs read their tables, and its burst of loads and asynchronous copies made that set-up 6.5 us
// instead of 4.2 (walk 4.9), and everything behind it slower. Whole step of eight ranks, 128 experts, fp8 weights (us):
// 8192 int32 ids a rank 70.0 with the walk, 75.0 without (the same with 256 threads and eight entries each, and with the
// reroute held back until weight_sync's launch), 4096 tokens 71.1 and 74.6.
constexpr int kWalkThreads = 256, kWalkWarps = kWalkThreads / kWarp;
__host__ __device__ __forceinline__ size_t walk_smem_bytes(int L) {
    return static_cast<size_t>(L) * (2 * kStagedReps * 4 + sizeof(FastRouter) + 4 + kWalkWarps * 4);
}
template <typename IdT>
__global__ void __launch_bounds__(kWalkThreads) sparse_walk_count_kernel(Batch<SparseArgs> batch, int K, int L, int wait_first) {
    extern __shared__ __align__(128) char smem_raw[];
    if (wait_first) pdl_wait();  // ahead of every read
    const SparseArgs& a = batch.a[blockIdx.y];
    const IdT* keys = static_cast<const IdT*>(a.ids);
    const int64_t n = static_cast<int64_t>(a.T) * K;
    const int64_t begin = static_cast<int64_t>(blockIdx.x) * kSparseTileEntries;
    if (begin >= n) return;  // a tile behind this rank's entries is read by nobody
    int32_t* hist = reinterpret_cast<int32_t*>(smem_raw);
    for (int i = threadIdx.x; i < L; i += blockDim.x) hist[i] = 0;
    __syncthreads();
    const int64_t end = min(begin + kSparseTileEntries, n);
    for (int64_t i = begin + threadIdx.x; i < end; i += blockDim.x) {
        const int b = key_bucket<IdT>(keys[i], L, false);
        if (b >= 0) atomicAdd(hist + b, 1);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < L; i += blockDim.x) a.scratch[static_cast<int64_t>(blockIdx.x) * L + i] = hist[i];
}

template <typename IdT>
__global__ void __launch_bounds__(kWalkThreads) sparse_walk_kernel(Batch<SparseArgs> batch, int K, int L, int D, int interleave, int wait_first) {
    extern __shared__ __align__(128) char smem_raw[];
    if (wait_first) pdl_wait();
    const SparseArgs& a = batch.a[blockIdx.y];
    const IdT* ids = static_cast<const IdT*>(a.ids);
    IdT* out = static_cast<IdT*>(a.out);
    const int64_t n = static_cast<int64_t>(a.T) * K;
    const int64_t tile_begin = static_cast<int64_t>(blockIdx.x) * kSparseTileEntries;
    if (tile_begin >= n) return;
    const bool quota_mode = interleave != 2;
    int32_t* prefix_s = reinterpret_cast<int32_t*>(smem_raw);
    int32_t* l2p_s = prefix_s + static_cast<size_t>(L) * kStagedReps;
    FastRouter* routers = reinterpret_cast<FastRouter*>(l2p_s + static_cast<size_t>(L) * kStagedReps);
    int32_t* base = reinterpret_cast<int32_t*>(routers + L);
    int32_t* warp_base = base + L;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    constexpr int kPerWarp = kSparseTileEntries / kWalkWarps;
    const int64_t begin = min(tile_begin + warp * kPerWarp, n), end = min(begin + kPerWarp, n);
    for (int e = tid; e < L; e += kWalkThreads) {
        int b = 0;
#pragma unroll 8
        for (int t = 0; t < static_cast<int>(blockIdx.x); ++t) b += __ldcg(a.scratch + static_cast<int64_t>(t) * L + e);
        base[e] = b;
    }
    for (int e = tid; e < L; e += kWalkThreads) {
        const int C = a.lcnts[e];
        const int m = min(min(C, D), kStagedReps);
        int32_t pre[kStagedReps], phys[kStagedReps];
#pragma unroll
        for (int j = 0; j < kStagedReps; ++j) {
            pre[j] = (j < m && quota_mode) ? a.rqp[static_cast<int64_t>(e) * D + j] : 0;
            phys[j] = j < m ? a.l2p[static_cast<int64_t>(e) * D + j] : -1;
        }
#pragma unroll
        for (int j = 0; j < kStagedReps; ++j) {
            prefix_s[e * kStagedReps + j] = pre[j];
            l2p_s[e * kStagedReps + j] = phys[j];
        }
        routers[e] = make_fast_router(e, C, a.rqp, D, quota_mode, interleave == 1, prefix_s + e * kStagedReps);
    }
    for (int i = tid; i < kWalkWarps * L; i += kWalkThreads) warp_base[i] = 0;
    __syncthreads();
    int32_t* mine = warp_base + warp * L;
    for (int64_t i = begin + lane; i < end; i += kWarp) {
        const int b = key_bucket<IdT>(ids[i], L, false);
        if (b >= 0) atomicAdd(mine + b, 1);
    }
    __syncthreads();
    for (int e = tid; e < L; e += kWalkThreads) {  // exclusive scan over the warps, behind the tiles in front
        int run = base[e];
#pragma unroll
        for (int w = 0; w < kWalkWarps; ++w) {
            const int c = warp_base[w * L + e];
            warp_base[w * L + e] = run;
            run += c;
        }
    }
    __syncthreads();
    for (int64_t i0 = begin; i0 < end; i0 += kWarp) {
        const int64_t i = i0 + lane;
        const bool in = i < end;
        const IdT id = in ? ids[i] : static_cast<IdT>(-1);
        const int b = key_bucket<IdT>(id, L, false);
        const unsigned active = __ballot_sync(kFullMask, b >= 0);
        int ordinal = 0;
        if (b >= 0) {
            const unsigned peers = __match_any_sync(active, b);
            const int before = __popc(peers & ((1u << lane) - 1u));
            ordinal = mine[b] + before;
            __syncwarp(active);
            if (before == 0) mine[b] += __popc(peers);
        }
        __syncwarp();
        if (!in) continue;
        const int C = b >= 0 ? routers[b].C : 0;
        if (C <= 0) {
            out[i] = id;
            continue;
        }
        const int j = C > 1 ? fast_replica_index(routers[b], ordinal, prefix_s + b * kStagedReps, a.rqp + static_cast<int64_t>(b) * D, quota_mode) : 0;
        out[i] = static_cast<IdT>(j < kStagedReps ? l2p_s[b * kStagedReps + j] : a.l2p[static_cast<int64_t>(b) * D + j]);
    }
}

// Experts with C <= 0 keep their id but still consume ordinals; the reference skips them before taking an ordinal
// (reroute.cu:505-509), which is equivalent because such an expert never maps anything.

// ------------------------------------------------------------- dispatch positions
__global__ void __launch_bounds__(kOrdThreads) dispatch_count_kernel(const int32_t* __restrict__ phys, int64_t n, int P, int tile_entries,
                                                                     int32_t* __restrict__ table) {
    pdl_wait();  // ahead of every read
    pdl_launch_dependents();
    count_tile<int32_t>(phys, n, P, true, tile_entries, table);
}

// Positions of the (token, k) entries once grouped by physical expert (stable) and the experts' row offsets: the
// same ordinals, plus a scan of the grand totals over the experts. Keys outside [0, P) go to a group at the end. pos may be
// phys itself, as in the sparse reroute.
template <int EPT>
__global__ void __launch_bounds__(kOrdThreads) __maxnreg__(EPT > 4 ? 128 : 80)
dispatch_positions_kernel(const int32_t* phys, int64_t n, int ctas, int P, const int32_t* __restrict__ table, int32_t* pos,
                          int32_t* __restrict__ expert_offsets) {
    if (table == nullptr) pdl_wait();  // ahead of every read; the count kernel in front waited, and its table is waited for where it is read
    extern __shared__ __align__(128) char smem_raw[];
    __shared__ int warp_tot[kOrdWarps];
    const int nb = P + 1;
    const OrdShared o = carve_ord_smem(smem_raw, nb);
    int32_t* all_of = o.behind;  // free once the totals are out
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nthreads = blockDim.x;
    int64_t begin, end;
    int iters;
    uint32_t packed[EPT];
    cluster_ordinals<EPT, true, int32_t>(
        phys, n, P, true, ctas, table, o, begin, end, iters, packed, []() {},
        [&](int b, int base, int all) {
            o.base[b] = base;
            all_of[b] = all;
        });
    if (ctas > 1) cluster_arrive();
    int carry = 0;
    for (int b0 = 0; b0 < nb; b0 += nthreads) {
        const int b = b0 + tid;
        const int all = b < nb ? all_of[b] : 0;
        int incl = all;
#pragma unroll
        for (int d = 1; d < kWarp; d <<= 1) {
            const int t = __shfl_up_sync(kFullMask, incl, d);
            if (lane >= d) incl += t;
        }
        if (lane == kWarp - 1) warp_tot[warp] = incl;
        __syncthreads();
        const int wt = lane < nthreads / kWarp ? warp_tot[lane] : 0;
        const int excl = carry + __reduce_add_sync(kFullMask, lane < warp ? wt : 0) + incl - all;
        if (b < nb) {
            o.base[b] += excl;
            if (blockIdx.x == 0 && expert_offsets != nullptr) expert_offsets[b] = excl;
        }
        carry += __reduce_add_sync(kFullMask, wt);
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < EPT; ++i) {
        const int64_t at = begin + i * kWarp + lane;
        if (i >= iters || at >= end) continue;
        const int b = static_cast<int>(packed[i] & 0xFFFFu);
        pos[at] = o.base[b] + o.counters[warp * ord_row(nb) + b] + static_cast<int>(packed[i] >> 16);
    }
    if (ctas > 1) cluster_wait();
}

// ------------------------------------------------------------------- row gather (HBM)
// out[i,:] = in[pos[i],:]. One warp per CTA drives a ring of bulk copies: global -> shared (mbarrier) -> global. An item is
// up to 32 consecutive output rows of together at most kGatherChunk bytes (a lane per row loads, one store writes them),
// or a chunk of that size of a longer row. Positions are fetched a batch of items ahead: a thread that read the position
// of the row it was about to load waited a memory round trip for every row. 65536 rows of 8 KiB: the
// step with its positions 217 -> 189 us.
constexpr int kGatherChunk = 16 * 1024;
constexpr int kGatherStages = 6;
constexpr int kGatherBatch = 256;  // positions

__global__ void __launch_bounds__(32) gather_rows_kernel(const uint8_t* __restrict__ in, const int32_t* __restrict__ pos,
                                                         uint8_t* __restrict__ out, int64_t num_rows,
                                                         int64_t row_bytes, int rows_per_item, int chunks_per_row,
                                                         int64_t num_src_rows, uint64_t timeout_ns, DeviceStatus* status) {
    extern __shared__ __align__(128) char smem_raw[];
    __shared__ __align__(8) uint64_t bars[kGatherStages];
    __shared__ int32_t pos_s[2][kGatherBatch];
    const int lane = threadIdx.x;
    if (lane == 0) {
        for (int s = 0; s < kGatherStages; ++s) mbar_init(&bars[s], 1);
        fence_mbar_init();
    }

    // either several rows per item or several items (chunks) per row; rows_per_item is a power of two
    const int shift = 31 - __clz(rows_per_item);
    const int64_t total = chunks_per_row > 1 ? num_rows * chunks_per_row : (num_rows + rows_per_item - 1) >> shift;
    const int64_t first = blockIdx.x, step = gridDim.x;
    const int count = first < total ? static_cast<int>((total - first + step - 1) / step) : 0;
    const int items = kGatherBatch >> shift;  // of a batch
    // Where an item lies. A cursor goes from item to item by additions: the divisions (64 bits, several an item) made rows of
    // two chunks 1.27 times as slow as one thread without them.
    struct Cursor {
        int64_t row;
        int chunk;
    };
    const bool whole = chunks_per_row == 1;
    const int64_t row_step = whole ? step << shift : step / chunks_per_row;
    const int chunk_step = whole ? 0 : static_cast<int>(step % chunks_per_row);
    auto advance = [&](Cursor& c) {
        c.row += row_step;
        c.chunk += chunk_step;
        if (c.chunk >= chunks_per_row) {
            c.chunk -= chunks_per_row;
            ++c.row;
        }
    };
    auto offset = [&](const Cursor& c) { return static_cast<int64_t>(c.chunk) * kGatherChunk; };
    auto row_part = [&](const Cursor& c) -> uint32_t {  // bytes of each of its rows
        return static_cast<uint32_t>(min(row_bytes - offset(c), static_cast<int64_t>(kGatherChunk)));
    };
    auto rows_of = [&](const Cursor& c) { return static_cast<int>(min(num_rows - c.row, static_cast<int64_t>(rows_per_item))); };

    auto fetch = [&](int batch, int32_t (&p)[kGatherBatch / 32]) {
#pragma unroll
        for (int u = 0; u < kGatherBatch / 32; ++u) {
            const int i = u * 32 + lane;
            const int k = batch * items + (i >> shift);
            int64_t row = num_rows;
            if (k < count) {
                const int64_t item = first + k * step;
                row = whole ? (item << shift) + (i & (rows_per_item - 1)) : item / chunks_per_row;
            }
            p[u] = row < num_rows ? __ldcg(pos + row) : 0;
        }
    };
    auto keep = [&](int batch, const int32_t (&p)[kGatherBatch / 32]) {
#pragma unroll
        for (int u = 0; u < kGatherBatch / 32; ++u) pos_s[batch & 1][u * 32 + lane] = p[u];
    };
    Cursor load = whole ? Cursor{first << shift, 0} : Cursor{first / chunks_per_row, static_cast<int>(first % chunks_per_row)};
    Cursor store = load;
    int issued = 0, load_stage = 0, load_slot = 0, load_half = 0;
    // (Loads whose lines are the first to leave L2: the gather alone 178.5 -> 176.4 us, 65536 rows of 8 KiB, and gather and a
    // kernel that reads its output 335 -> 340, 16384 rows 95 -> 96.)
    auto issue_load = [&]() {
        const int n = rows_of(load);
        const uint32_t bytes = row_part(load);
        if (lane == 0) mbar_expect_tx(&bars[load_stage], n * bytes);
        __syncwarp();
        if (lane < n) {
            int64_t src_row = pos_s[load_half][(load_slot << shift) + lane];
            if (src_row < 0 || src_row >= num_src_rows) {  // never read out of bounds: record and clamp
                report_error(status, UEP_DEV_BAD_PLAN, static_cast<int>(load.row + lane));
                src_row = 0;
            }
            bulk_load(smem_raw + load_stage * kGatherChunk + lane * bytes, in + src_row * row_bytes + offset(load), bytes, &bars[load_stage]);
        }
        advance(load);
        ++issued;
        if (++load_stage == kGatherStages) load_stage = 0;
        if (++load_slot == items) {
            load_slot = 0;
            load_half ^= 1;
        }
    };

    int32_t ahead[kGatherBatch / 32];
    pdl_wait();  // the positions may be the output of the kernel in front
    fetch(0, ahead);
    keep(0, ahead);
    __syncwarp();
    // Loads run at most kGatherStages - 1 items ahead: the first ones stay within batch 0, and batch b + 1 is in shared memory
    // while the items of batch b are stored.
    static_assert(kGatherBatch / 32 >= kGatherStages - 1, "the loads of a batch's items stay within the next batch");
    while (issued < count && issued < kGatherStages - 1) issue_load();
    fetch(1, ahead);
    keep(1, ahead);
    __syncwarp();
    int k = 0, stage = 0;
    uint32_t parity = 0;
    bool ok = true;
    for (int batch = 0; ok && k < count; ++batch) {
        fetch(batch + 2, ahead);
        const int batch_end = min((batch + 1) * items, count);
        for (; k < batch_end; ++k) {
            ok = __all_sync(kFullMask, mbar_wait(&bars[stage], parity, timeout_ns));
            if (!ok) break;
            if (lane == 0) {
                bulk_store(out + store.row * row_bytes + offset(store), smem_raw + stage * kGatherChunk, rows_of(store) * row_part(store));
                bulk_commit();
                if (issued < count && k >= 1) bulk_wait_read<1>();
            }
            __syncwarp();
            advance(store);
            if (++stage == kGatherStages) {
                stage = 0;
                parity ^= 1u;
            }
            if (issued < count) issue_load();
        }
        __syncwarp();
        keep(batch + 2, ahead);  // over batch b, whose loads have all been issued
        __syncwarp();
    }
    if (lane == 0) bulk_wait_all<0>();
    if (k < count) {
        // a load did not land in time: report, then give every load still in flight one more
        // bounded wait so that shared memory is not released under it
        if (lane == 0) report_error(status, UEP_DEV_TIMEOUT_COPY, k);
        for (int j = k; j < issued; ++j) {
            mbar_wait(&bars[j % kGatherStages], static_cast<uint32_t>((j / kGatherStages) & 1), timeout_ns);
        }
    }
}

// Plain vector-load variant for rows that are not 16-byte sized/aligned multiples.
__global__ void __launch_bounds__(256) gather_rows_plain_kernel(const uint8_t* __restrict__ in,
                                                                const int32_t* __restrict__ pos,
                                                                uint8_t* __restrict__ out, int64_t num_rows,
                                                                int64_t row_bytes, int64_t num_src_rows,
                                                                DeviceStatus* status) {
    for (int64_t row = blockIdx.x; row < num_rows; row += gridDim.x) {
        int64_t src = pos[row];
        if (src < 0 || src >= num_src_rows) {
            if (threadIdx.x == 0) report_error(status, UEP_DEV_BAD_PLAN, static_cast<int>(row));
            src = 0;
        }
        for (int64_t b = threadIdx.x; b < row_bytes; b += blockDim.x) out[row * row_bytes + b] = in[src * row_bytes + b];
    }
}

// These kernels also ask for the largest shared-memory carve-out: they run next to weight_sync, whose CTAs need most of an
// SM's shared memory, and an SM that was set up with a small carve-out for a reroute CTA cannot take a weight_sync CTA
// until it has drained.
cudaError_t ensure_smem_attr(const void* fn, size_t bytes) { return allow_smem(fn, bytes, true); }

int64_t sparse_tiles(int64_t n) { return (n + kSparseTileEntries - 1) / kSparseTileEntries; }

}  // namespace

int64_t dense_scratch_elems(int T, int L) { return static_cast<int64_t>(dense_tiles(T)) * L + 4; }
int64_t sparse_scratch_elems(int64_t entries, int L) { return sparse_tiles(entries) * L + 4; }

// Launch of a kernel that may start before the kernel in front of it in the stream has finished
// (programmatic dependent launch); the kernel calls pdl_wait() before it reads that kernel's output.
// UEP_DISABLE_PDL=1 turns the attribute off (the pair then runs strictly one after the other).
bool pdl_enabled() {
    static const bool disabled = [] {
        const char* e = std::getenv("UEP_DISABLE_PDL");
        return e != nullptr && e[0] == '1';
    }();
    return !disabled;
}

template <typename... Params, typename... Args>
cudaError_t launch_dependent(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                             bool overlap, Args&&... args) {
    const bool disabled = !pdl_enabled();
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = (disabled || !overlap) ? 0 : 1;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

cudaError_t launch_dense_forward(const Batch<DenseFwdArgs>& b, int L, int P, int D, int quota_mode, int interleave,
                                 bool beside_sync, cudaStream_t stream) {
    int max_T = 0;
    for (int i = 0; i < b.n; ++i) max_T = b.a[i].T > max_T ? b.a[i].T : max_T;
    if (max_T == 0) return cudaSuccess;
    // (the limit dates from a kernel that staged the map; a wider one is still refused)
    if (L > kDenseMaxExperts) return cudaErrorInvalidValue;
    const dim3 grid(dense_tiles(max_T), b.n);
    const int chunk = P > kDenseMaxChunkCols ? kDenseMaxChunkCols : P;
    const int sms = std::max(device_sm_count(), 1);
    // Four tiles a CTA where one each would be more CTAs than the device holds at once (kCountCtasPerSm) and four tiles are one round
    // of loads. Plan and pair of eight ranks of 128 experts, tile by tile and by four, among others / each alone (us): 4096 rows
    // 30.8/38.7 and 31.2/38.5, 5500 37.6/46.0 and 38.3/45.5, above the line 6000 38.7/47.6 and 38.8/46.5, 7000 42.6/51.4 and 42.4/49.6,
    // 8000 45.5/54.8 and 45.2/52.2; beside a weight_sync 6000 53.6/62.7 and 53.4/61.0, 7000 56.6/65.2 and 55.5/64.0. 8192 x 256 (two rounds)
    // 71.6 and 72.7.
    const bool by_four = L <= 128 && static_cast<int64_t>(grid.x) * b.n > kCountCtasPerSm * sms;
    const auto count = by_four ? dense_count_kernel<4> : dense_count_kernel<1>;
    // Up to two tiles an SM the scatter kernel is a chain of phases: more threads shorten each. Of 256 threads (64 registers) an SM
    // holds four tiles, of 128 eight: between the two all tiles are under way at once with 128, and their phases, of which only the last one
    // writes, fill each other's gaps; with 256 the first wave writes when the second one has not begun. Plan and pair of eight ranks, 256 and
    // 128 threads (us): 4800 rows of 128 experts 29.8 and 27.8, 8192 40.1 and 38.0, of 64 experts 28.5 and 25.7, of 256 61.2 and 60.5; beside
    // a weight_sync 8192 x 128 with bf16 experts of 9 MB 58.0 and 56.8, 6500 x 64 with fp8 of 5 MB 41.6 and 39.6. In one wave either way, 4096
    // x 128 25.3 and 25.9; in two, 12000 x 128 52.7 and 54.1. With more experts the tiles are longer and the last wave of 256 threads is filled
    // from seven tiles an SM on: pair of eight ranks, 256 and 128 threads, 8169 x 192 (6.9 tiles) 39.8 and 39.1, 8643 x 192 (7.3) 41.2 and 41.4,
    // 9353 x 256 (7.9) 50.5 and 51.0, quota plans, 51.9 and 52.9, legacy ones. One rank: 73000 x 192 (7.7) 38.2 and 37.2, 44000 x 256 30.5 and
    // 31.1, 57000 x 256 38.5 and 39.9, 55000 x 512 64.0 and 66.4 (50000 x 256 35.4 and 34.2).
    const int64_t all_tiles = static_cast<int64_t>(grid.x) * b.n;
    const int one_wave = L <= 128 ? 8 : (b.n > 1 ? 7 : (L < 256 ? 8 : 0));  // tiles an SM
    const int threads = all_tiles <= 2 * sms ? kDenseMaxThreads : (all_tiles > 4 * sms && all_tiles <= one_wave * sms ? kRerouteThreads / 2 : kRerouteThreads);
    const size_t smem_count = static_cast<size_t>(pad4(L)) * (by_four ? 4 : 1), smem = dense_smem_bytes(L, chunk, threads);
    // Both kernels are dependents of whatever is in front of them, as internal.h says; several ranks not beside a weight_sync, whose set-up
    // the early CTAs disturb (step of 8192 bool rows of 128 experts with bf16 experts of 9 MB 59.5 us, first kernel, second and both
    // as dependents 60.1, 60.2 and 60.3; of 8000 with 5 MB 54.0, 54.9, 54.0 and 54.5; of 1000 of 64 with 3 MB 29.9, 29.6, 30.0 and 30.7).
    const bool dependent = pdl_enabled() && (b.n == 1 || !beside_sync);
    // One rank's pair is latency: the second kernel has its prologue beside the first one. Several ranks fill the device with the
    // first kernel alone; their second one starts behind it and waits first (started early it does nothing but wait: plan and
    // pair of eight ranks, 4096 rows of 128 experts, 24.4 us and 25.6, 8192 rows 38.4 and 39.7).
    const bool prologue = dependent && b.n == 1;
    cudaError_t e = ensure_smem_attr(reinterpret_cast<const void*>(dense_scatter_kernel), smem);
    if (e != cudaSuccess) return e;
    e = ensure_smem_attr(reinterpret_cast<const void*>(count), smem_count);
    if (e != cudaSuccess) return e;
    count_launch(2);
    e = launch_dependent(count, dim3(by_four ? (grid.x + 3) / 4 : grid.x, b.n), dim3(kRerouteThreads), smem_count, stream, dependent, b, L,
                         dependent ? 1 : 0, prologue ? 1 : 0);
    if (e != cudaSuccess) return e;
    return launch_dependent(dense_scatter_kernel, grid, dim3(threads), smem, stream, dependent, b, L, P, D, quota_mode,
                            interleave, chunk, prologue ? 1 : 0, dependent && !prologue ? 1 : 0);
}

cudaError_t launch_dense_backward(const Batch<DenseBwdArgs>& b, int L, int P, int D, cudaStream_t stream) {
    int max_T = 0;
    for (int i = 0; i < b.n; ++i) max_T = b.a[i].T > max_T ? b.a[i].T : max_T;
    if (max_T == 0) return cudaSuccess;
    // The tile kernel pays where a launch is more than a few waves of latency, and where a row of the map is more than two
    // words, so that a tile keeps all of its threads busy (events around calls over 11 states, tiles against cells: one rank
    // of 4096 x 128 6.3 and 6.3, 8191 x 128 8.3 and 8.3, 4096 x 256 6.3 and 8.5, 8191 x 256 8.4 and 12.6, 16384 x 128 10.4
    // and 12.5; eight ranks of 1024 x 128 8.1 and 8.3, 2048 x 128 9.4 and 12.9; 64 experts: eight ranks of 2048 tokens 10.4
    // and 8.3, of 8192 14.0 and 16.5 with the kernel before). Very wide layers: the staged plan rows are more than the few
    // rows that share them.
    int64_t cells = 0;
    for (int i = 0; i < b.n; ++i) cells += static_cast<int64_t>(b.a[i].T) * L;
    const int groups = (L + 31) / 32;
    // a word of a row a thread: 64 rows at 128 experts (32 rows 18.6 us for 18.3, 128 20.9); fewer where that leaves SMs
    // without two CTAs (8191 x 256: 16 rows 8.4 us, 64 rows 10.4), or where wide rows fill the shared memory
    const int sms = std::max(device_sm_count(), 1);
    int rows = groups <= 4 ? 64 : (groups <= 8 ? 32 : 16);
    while (rows > 16 && static_cast<int64_t>((max_T + rows - 1) / rows) * b.n < 2 * sms) rows /= 2;
    while (rows > 8 && dense_bwd_smem_bytes(L, P, rows) > kMaxCtaSmem / 4) rows /= 2;
    const size_t smem = dense_bwd_smem_bytes(L, P, rows);
    bool tiles = cells >= (L > 64 ? 1 << 20 : 1 << 22) && L % 4 == 0 && L <= 512 && smem <= kMaxCtaSmem;
    for (int i = 0; i < b.n; ++i) {
        tiles = tiles && ((reinterpret_cast<uintptr_t>(b.a[i].map) & 3u) == 0) && ((reinterpret_cast<uintptr_t>(b.a[i].grad_probs) & 15u) == 0);
    }
    count_launch();
    if (tiles) {
        cudaError_t e = ensure_smem_attr(reinterpret_cast<const void*>(dense_backward_tile_kernel), smem);
        if (e != cudaSuccess) return e;
        return launch_dependent(dense_backward_tile_kernel, dim3((max_T + rows - 1) / rows, b.n), dim3(kDenseBwdThreads), smem, stream, true, b, L, P,
                                D, rows, 1);
    }
    int64_t blocks = (static_cast<int64_t>(max_T) * L / 4 + kRerouteThreads - 1) / kRerouteThreads + 1;
    const int64_t cap = std::max(sms * 16 / b.n, 1);
    if (blocks > cap) blocks = cap;
    return launch_dependent(dense_backward_kernel, dim3(static_cast<unsigned>(blocks), b.n), dim3(kRerouteThreads), 0, stream, true, b, L, P, D, 1);
}

// How an input of n entries is cut: a cluster of CTAs with at most per_lane entries a thread, and as many clusters as it
// takes. Measured on one rank's int32 ids, 128 experts (us; the count + reroute pair that this replaces: 14.8 at 65536):
//   * the cluster grows to eight CTAs before a thread takes a second entry: 2048 entries 4.5 on four CTAs, 5.7 on one;
//   * up to 16384 entries one cluster (6.9; two clusters the same), behind it two entries a thread up to eight clusters
//     (65536 entries 7.8; four entries a thread 8.5, one 9.6) and four beyond (131072: 9.6 against 11.4 with two);
//   * behind kOrdRecountMax entries, or in place behind one cluster's, a count kernel in front instead of the repeated
//     counting. The reroute then goes in single CTAs of four entries a thread: they find room anywhere beside weight_sync,
//     which leaves every SM a quarter of its shared memory. (524288 entries alone and beside weight_sync: 19.5 and 25, with
//     clusters of sixteen entries a thread 33.8 and 49; 131072 in place 13.3 and 16.4, 17.4 and 18.6 with clusters of four.) The tiles in front of
//     a CTA are a sum that grows with the square of the input: behind kOrdShortTiles entries tiles of sixteen entries
//     (2^21 entries 50, tiles of four 58). The positions need every tile's counts: sixteen entries in clusters at any size
//     (524288 entries 21.5; four 44, single CTAs 30).
constexpr int64_t kOrdRecountMax = 1 << 18;
constexpr int64_t kOrdShortTiles = 1 << 20;

struct OrdGrid {
    int threads, ctas, clusters, per_lane;
    bool table;
};
// `totals`: the grand totals are wanted too (the positions). Every CTA of a cluster then reads every other one's totals: with
// many buckets a thread takes four entries before the cluster grows (4096 entries, 320 and 1024 buckets: 10.2 and 12.3 us,
// on eight CTAs 12.3 and 19.7).
// one_cluster: up to eight entries a thread in one cluster (launch_sparse_typed).
OrdGrid ord_grid(int64_t n, int buckets, int ranks, bool in_place, int threads, bool totals, bool one_cluster = false) {
    OrdGrid g{threads, 1, 1, 1, false};
    const int64_t grow = static_cast<int64_t>(threads) * (totals && buckets > 256 ? 4 : 1);
    while (g.ctas < kOrdMaxCluster && n > g.ctas * grow) g.ctas *= 2;
    int64_t row = static_cast<int64_t>(g.ctas) * threads;  // one entry per thread of a cluster
    if (n <= row) return g;
    if (one_cluster && n > 4 * row && n <= 8 * row) {
        g.per_lane = 8;
        return g;
    }
    g.per_lane = 4;
    g.table = n > 4 * row && (in_place || ranks > 1 || n > kOrdRecountMax);
    if (g.table && totals) {
        g.per_lane = 16;
    } else if (g.table) {
        g.ctas = 1;
        row = threads;
        g.per_lane = n > kOrdShortTiles ? 16 : 4;
    }
    // (tiles of the table: per_lane entries a thread, at least kSparseTileEntries a tile)
    const int64_t chunk = row * (g.table ? g.per_lane : (n > 4 * row && n <= 16 * row ? 2 : 4));
    g.clusters = static_cast<int>((n + chunk - 1) / chunk);
    return g;
}

// Launch of clusters of `g.ctas` CTAs; `overlap`: as a programmatic dependent launch behind the count kernel.
template <typename... Params, typename... Args>
cudaError_t launch_clusters(void (*kernel)(Params...), const OrdGrid& g, int ranks, size_t smem, cudaStream_t stream, bool overlap, Args&&... args) {
    cudaError_t e = ensure_smem_attr(reinterpret_cast<const void*>(kernel), smem);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(static_cast<unsigned>(g.ctas) * g.clusters, ranks);
    cfg.blockDim = dim3(g.threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int na = 0;
    if (g.ctas > 1) {
        attr[na].id = cudaLaunchAttributeClusterDimension;
        attr[na].val.clusterDim.x = g.ctas;
        attr[na].val.clusterDim.y = 1;
        attr[na].val.clusterDim.z = 1;
        ++na;
    }
    if (overlap) {
        attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[na].val.programmaticStreamSerializationAllowed = 1;
        ++na;
    }
    cfg.attrs = attr;
    cfg.numAttrs = na;
    count_launch();
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

// `launch` with the compile-time number of entries a thread holds.
template <typename Launch>
cudaError_t with_lanes(const OrdGrid& g, Launch launch) {
    if (g.per_lane == 1) return launch(std::integral_constant<int, 1>{});
    if (g.per_lane == 4) return launch(std::integral_constant<int, 4>{});
    if (g.per_lane == 8) return launch(std::integral_constant<int, 8>{});
    return launch(std::integral_constant<int, 16>{});
}

// Several ranks in one launch, n entries of the longest (up to one cluster's the other kernel is one launch, and up to two beside a
// weight_sync that is not long): does the walk pay? Beside weight_sync while the walk's sums over the earlier tiles stay short, n / 2048 * L up to 4096 (whole step, walk
// and table: 128 experts, 65536 entries 72.5 and 75.2, 131072 80 and 74; 256 experts, 32768 entries 76.7 and 78.7, 65536 int64
// 84.9 and 81.3; 64 experts, 131072 entries 57.8 and 60.1). Alone from 65536 entries on, where the launch fills the device
// either way (131072 entries of 128 experts 27.6 and 31.7; 32768 entries 18 and 14.3). Behind kOrdRecountMax always
// (524288 entries 69 and 87).
bool walk_pays(int64_t n, int L, bool beside_sync) {
    if (n <= 4LL * kOrdMaxCluster * kOrdThreads) return false;
    return n > kOrdRecountMax || (beside_sync ? n * L <= 1 << 23 : n > 1 << 16);
}

// Several ranks beside a weight_sync of at most so many bytes: the reroute is then the longer one of the two, and both of its kernels
// are dependents like elsewhere; beside a longer one their early CTAs disturb its set-up. Step of eight ranks, ordinary launches and
// dependents (us): fp8 experts in 16 slots of 3 MB, 3000 tokens of 64 31.0 and 28.6; above the line 32 slots of 19 MB, 8192 tokens 54.3 and
// 54.9, 64 of 44 MB, 16384 of 256 104.0 and 107.4.
constexpr int64_t kShortSyncBytes = 64ll << 20;

// Several ranks of up to 32768 entries beside a weight_sync of at most so many bytes: one cluster a rank with up to eight entries a
// thread, one launch where the walk is two, each of which starts on a tick of 2 us. Step of eight ranks, walk and one cluster (us): 4000
// tokens of 256 experts with 71 MB 36.7 and 30.6, 4096 of 64 with 201 MB of bf16 31.0 and 27.1. Above the line the reroute is over before the
// weight_sync, whose set-up the cluster's burst of loads disturbs: 302 MB in 16 slots 51.6 and 52.0, 2.4 GB 80.5 and 81.3. With sixteen
// entries a thread longer inputs lose too: 8000 of 128 with 25 MB 30.9 and 34.4. Alone the pair with its counts is the better one, 16.9
// and 18.9.
constexpr int64_t kOneClusterSyncBytes = 256ll << 20;
constexpr int64_t kOneClusterEntries = 8LL * kOrdMaxCluster * kOrdThreads;

template <typename IdT>
static cudaError_t launch_sparse_typed(const Batch<SparseArgs>& b, int K, int L, int D, int interleave, int64_t beside_bytes,
                                       cudaStream_t stream) {
    const bool beside_sync = beside_bytes > 0;
    const bool dependent = pdl_enabled() && (b.n == 1 || beside_bytes <= kShortSyncBytes);
    int64_t max_n = 0;
    bool in_place = false;
    for (int i = 0; i < b.n; ++i) {
        const int64_t n = static_cast<int64_t>(b.a[i].T) * K;
        max_n = n > max_n ? n : max_n;
        const uintptr_t x = reinterpret_cast<uintptr_t>(b.a[i].ids), y = reinterpret_cast<uintptr_t>(b.a[i].out);
        const uintptr_t bytes = static_cast<uintptr_t>(n) * sizeof(IdT);
        in_place = in_place || (n > 0 && x < y + bytes && y < x + bytes);
    }
    if (max_n == 0) return cudaSuccess;
    const bool one_cluster = b.n > 1 && beside_sync && beside_bytes <= kOneClusterSyncBytes && max_n <= kOneClusterEntries;
    if (b.n > 1 && !one_cluster && walk_pays(max_n, L, beside_sync) && walk_smem_bytes(L) <= kMaxCtaSmem) {
        const dim3 grid(static_cast<unsigned>(sparse_tiles(max_n)), b.n);
        cudaError_t e = ensure_smem_attr(reinterpret_cast<const void*>(sparse_walk_count_kernel<IdT>), sizeof(int32_t) * L);
        if (e != cudaSuccess) return e;
        e = ensure_smem_attr(reinterpret_cast<const void*>(sparse_walk_kernel<IdT>), walk_smem_bytes(L));
        if (e != cudaSuccess) return e;
        count_launch(2);
        e = launch_dependent(sparse_walk_count_kernel<IdT>, grid, dim3(kWalkThreads), sizeof(int32_t) * L, stream, dependent, b, K, L,
                             dependent ? 1 : 0);
        if (e != cudaSuccess) return e;
        return launch_dependent(sparse_walk_kernel<IdT>, grid, dim3(kWalkThreads), walk_smem_bytes(L), stream, dependent, b, K, L, D, interleave,
                                dependent ? 1 : 0);
    }
    const int staged = sparse_smem_bytes(L, true) <= kMaxCtaSmem ? 1 : 0;
    const size_t smem = sparse_smem_bytes(L, staged != 0);
    const OrdGrid g = ord_grid(max_n, L, b.n, in_place, kOrdThreads, false, one_cluster);
    // The second kernel has its ids, its plan rows and its positions inside the warps while the first one counts: single CTAs, of
    // which few fill the device. Plan and reroute of eight ranks, second kernel behind the first and beside it (us): 2100 int64 tokens, top 8 of 64
    // 17.8 and 16.5, 4096 int32 of 64 17.9 and 16.8, 5000 top 6 of 128 18.5 and 17.4, 8192 of 128 22.9 and 22.1, of 256 25.3 and 24.4; with a
    // weight_sync of 25 MB 6000 of 256 32.8 and 31.2.
    const bool prologue = dependent && g.table;
    if (g.table) {
        cudaError_t e = ensure_smem_attr(reinterpret_cast<const void*>(sparse_count_kernel<IdT>), sizeof(int32_t) * L);
        if (e != cudaSuccess) return e;
        count_launch();
        e = launch_dependent(sparse_count_kernel<IdT>, dim3(g.ctas * g.clusters, b.n), dim3(kOrdThreads), sizeof(int32_t) * L, stream, dependent, b,
                             K, L, g.per_lane * kOrdThreads, dependent ? 1 : 0, prologue ? 1 : 0);
        if (e != cudaSuccess) return e;
    }
    return with_lanes(g, [&](auto per_lane) {
        return launch_clusters(sparse_reroute_kernel<decltype(per_lane)::value, IdT>, g, b.n, smem, stream, dependent, b, g.ctas, K, L, D,
                               interleave, staged, g.table ? 1 : 0, dependent && !prologue ? 1 : 0);
    });
}

cudaError_t launch_sparse_reroute(const Batch<SparseArgs>& b, int ids_kind, int K, int L, int D, int interleave, int64_t beside_bytes,
                                  cudaStream_t stream) {
    if (ids_kind == 2) return launch_sparse_typed<long long>(b, K, L, D, interleave, beside_bytes, stream);
    return launch_sparse_typed<int32_t>(b, K, L, D, interleave, beside_bytes, stream);
}

}  // namespace uep

using namespace uep;

extern "C" {

int64_t uep_reroute_scratch_elems(int64_t T, int K_or_0, int L) {
    if (K_or_0 <= 0) return dense_scratch_elems(static_cast<int>(T), L);
    return sparse_scratch_elems(T * K_or_0, L);
}

int uep_dense_reroute_forward(const uint8_t* routing_map, const float* probs, const int32_t* l2p,
                              const int32_t* lcnts, const int32_t* rank_quota_prefix, uint8_t* expanded_map,
                              float* expanded_probs, int32_t* scratch, int T, int L, int P, int D, int quota_mode,
                              int interleave, void* stream_) {
    if (T < 0 || L <= 0 || P <= 0 || D < 1) return fail(UEP_ERR_INVALID, "dense_reroute_forward: bad sizes");
    if (T == 0) return UEP_OK;
    if (!routing_map || !probs || !l2p || !lcnts || !expanded_map || !expanded_probs || !scratch ||
        (quota_mode && !rank_quota_prefix))
        return fail(UEP_ERR_INVALID, "dense_reroute_forward: null pointer");
    if (D > 255) return fail(UEP_ERR_INVALID, "dense_reroute_forward: more than 255 replicas per expert");
    Batch<DenseFwdArgs> b{};
    b.n = 1;
    b.a[0] = DenseFwdArgs{routing_map, probs, l2p, lcnts, rank_quota_prefix, scratch, expanded_map, expanded_probs, T};
    UEP_CUDA_TRY(launch_dense_forward(b, L, P, D, quota_mode, interleave, false, static_cast<cudaStream_t>(stream_)));
    return UEP_OK;
}

int uep_dense_reroute_backward(const float* grad_expanded, const uint8_t* routing_map, const uint8_t* expanded_map,
                               const int32_t* l2p, const int32_t* lcnts, float* grad_probs, int T, int L, int P, int D,
                               void* stream_) {
    if (T < 0 || L <= 0 || P <= 0 || D < 1) return fail(UEP_ERR_INVALID, "dense_reroute_backward: bad sizes");
    if (T == 0) return UEP_OK;
    if (!grad_expanded || !routing_map || !expanded_map || !l2p || !lcnts || !grad_probs)
        return fail(UEP_ERR_INVALID, "dense_reroute_backward: null pointer");
    Batch<DenseBwdArgs> b{};
    b.n = 1;
    b.a[0] = DenseBwdArgs{grad_expanded, routing_map, expanded_map, l2p, lcnts, grad_probs, T};
    UEP_CUDA_TRY(launch_dense_backward(b, L, P, D, static_cast<cudaStream_t>(stream_)));
    return UEP_OK;
}

// One message for what would otherwise end in a failed launch.
static int check_width(size_t smem, const char* what) {
    return smem <= kSmemLimit ? UEP_OK : fail(UEP_ERR_INVALID, std::string(what) + ": too many experts for the kernel's shared memory");
}

static int sparse_common(int kind, const void* ids, void* out, int T, int K, int L, const int32_t* l2p,
                         const int32_t* lcnts, const int32_t* rqp, int D, int interleave, int32_t* scratch,
                         void* stream_) {
    if (T < 0 || K < 0 || L <= 0 || D < 1) return fail(UEP_ERR_INVALID, "sparse_reroute: bad sizes");
    if (static_cast<int64_t>(T) * K == 0) return UEP_OK;
    if (!ids || !out || !scratch || !l2p || !lcnts || (interleave != 2 && !rqp)) return fail(UEP_ERR_INVALID, "sparse_reroute: null pointer");
    if (const int rc = check_width(sparse_smem_bytes(L, false), "sparse_reroute")) return rc;
    Batch<SparseArgs> b{};
    b.n = 1;
    b.a[0] = SparseArgs{ids, out, l2p, lcnts, rqp, scratch, T};
    UEP_CUDA_TRY(launch_sparse_reroute(b, kind, K, L, D, interleave, 0, static_cast<cudaStream_t>(stream_)));
    return UEP_OK;
}

int uep_sparse_reroute_i32(const int32_t* ids, int32_t* out, int T, int K, int L, const int32_t* l2p,
                           const int32_t* lcnts, const int32_t* rank_quota_prefix, int D, int interleave,
                           int32_t* scratch, void* stream) {
    return sparse_common(1, ids, out, T, K, L, l2p, lcnts, rank_quota_prefix, D, interleave, scratch, stream);
}
int uep_sparse_reroute_i64(const int64_t* ids, int64_t* out, int T, int K, int L, const int32_t* l2p,
                           const int32_t* lcnts, const int32_t* rank_quota_prefix, int D, int interleave,
                           int32_t* scratch, void* stream) {
    return sparse_common(2, ids, out, T, K, L, l2p, lcnts, rank_quota_prefix, D, interleave, scratch, stream);
}

// ---------------------------------------------------------------------------------------
// Sparse reroute for callers that must not allocate.
//
// Some hosts of this library cannot call cudaMalloc on the path where routing happens: an
// inference server that has handed the whole device to its own memory pool, a caller inside
// a region where the allocator is frozen, or a plugin boundary that only passes the tensors
// it was given. The regular entry point needs a caller-provided scratch buffer (per-tile
// expert counts); this variant keeps that scratch in a fixed array that is part of the
// loaded library image on every device, so the caller passes inputs and outputs only.
//
// Limits and rules:
//   * the per-tile counts must fit the array: ceil(T*K / 2048) * L + 4 <= 262144 int32 (1 MiB);
//     e.g. 131072 entries (16384 tokens x top-8) with as many experts as the kernel takes (about 3050, whose counters
//     fill a CTA's shared memory), or 511 tiles (1,046,528 entries) with 512 experts: the four spare words count against
//     the limit. Larger problems are refused with UEP_ERR_INVALID and a message, nothing is launched;
//   * the array is shared by every call on a device and keeps the previous call's counts. The
//     count pass overwrites every element the second pass reads, so nothing has to start at
//     zero; but two calls that can overlap on the GPU (different streams without an ordering
//     between them) would race on it: order them;
//   * the first call on a device resolves the array's device address (once per device, with
//     that device current). It launches nothing else extra, but it should be made before any
//     stream capture begins.
static constexpr int64_t kStaticRerouteScratchElems = 256 * 1024;
static __device__ __align__(256) int32_t g_static_reroute_scratch[kStaticRerouteScratchElems];

int uep_sparse_reroute_i32_static(const int32_t* ids, int32_t* out, int T, int K, int L, const int32_t* l2p,
                                  const int32_t* lcnts, const int32_t* rank_quota_prefix, int D, int interleave,
                                  void* stream) {
    if (T < 0 || K < 0 || L <= 0 || D < 1) return fail(UEP_ERR_INVALID, "sparse_reroute_static: bad sizes");
    const int64_t need = sparse_scratch_elems(static_cast<int64_t>(T) * K, L);
    if (need > kStaticRerouteScratchElems) {
        return fail(UEP_ERR_INVALID, "sparse_reroute_static: needs " + std::to_string(need) +
                                         " int32 of scratch, the built-in array holds " +
                                         std::to_string(kStaticRerouteScratchElems) +
                                         " (use uep_sparse_reroute_i32 with your own scratch)");
    }
    if (const int rc = check_width(sparse_smem_bytes(L, false), "sparse_reroute_static")) return rc;
    // In host code the array's name is only a handle for the runtime: the address a kernel can
    // use has to be asked for, per device, while that device is current.
    constexpr int kMaxDevices = 64;
    static std::mutex mu;
    static int32_t* device_ptr[kMaxDevices] = {nullptr};
    int dev = -1;
    UEP_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDevices) return fail(UEP_ERR_UNSUPPORTED, "sparse_reroute_static: device index above 63");
    int32_t* scratch = nullptr;
    {
        std::lock_guard<std::mutex> lock(mu);
        if (device_ptr[dev] == nullptr) {
            void* p = nullptr;
            UEP_CUDA_TRY(cudaGetSymbolAddress(&p, g_static_reroute_scratch));
            device_ptr[dev] = static_cast<int32_t*>(p);
        }
        scratch = device_ptr[dev];
    }
    return sparse_common(1, ids, out, T, K, L, l2p, lcnts, rank_quota_prefix, D, interleave, scratch, stream);
}

int64_t uep_dispatch_scratch_elems(int64_t num_entries, int P) { return sparse_tiles(num_entries) * (P + 1) + 4; }

int uep_dispatch_positions(const int32_t* phys_ids, int64_t num_entries, int P, int32_t* pos,
                           int32_t* expert_offsets, int32_t* scratch, void* stream_) {
    if (num_entries < 0 || P <= 0) return fail(UEP_ERR_INVALID, "dispatch_positions: bad sizes");
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    if (num_entries == 0) {
        if (expert_offsets) UEP_CUDA_TRY(cudaMemsetAsync(expert_offsets, 0, sizeof(int32_t) * (P + 1), stream));
        return UEP_OK;
    }
    if (!phys_ids || !pos || !scratch) return fail(UEP_ERR_INVALID, "dispatch_positions: null pointer");
    if (const int rc = check_width(ord_smem_bytes(P + 1, kOrdFewThreads) + sizeof(int32_t) * kOrdWarps, "dispatch_positions")) return rc;
    const uintptr_t x = reinterpret_cast<uintptr_t>(phys_ids), y = reinterpret_cast<uintptr_t>(pos), bytes = sizeof(int32_t) * num_entries;
    const bool in_place = x < y + bytes && y < x + bytes;
    const OrdGrid g = ord_grid(num_entries, P + 1, 1, in_place, ord_smem_bytes(P + 1, kOrdThreads) <= kMaxCtaSmem ? kOrdThreads : kOrdFewThreads, true);
    const size_t smem = ord_smem_bytes(P + 1, g.threads), smem1 = sizeof(int32_t) * (P + 1);
    if (g.table) {
        UEP_CUDA_TRY(ensure_smem_attr(reinterpret_cast<const void*>(dispatch_count_kernel), smem1));
        count_launch();
        UEP_CUDA_TRY(launch_dependent(dispatch_count_kernel, dim3(g.ctas * g.clusters), dim3(g.threads), smem1, stream, true, phys_ids, num_entries, P,
                                      g.per_lane * g.threads, scratch));
    }
    const int32_t* table = g.table ? scratch : nullptr;
    UEP_CUDA_TRY(with_lanes(g, [&](auto per_lane) {
        return launch_clusters(dispatch_positions_kernel<decltype(per_lane)::value>, g, 1, smem, stream, pdl_enabled(), phys_ids, num_entries, g.ctas, P,
                               table, pos, expert_offsets);
    }));
    return UEP_OK;
}

int uep_gather_rows(const void* in, const int32_t* pos, void* out, int64_t num_rows, int64_t num_src_rows,
                    int64_t row_bytes, int32_t* status, void* stream_) {
    if (num_rows < 0 || row_bytes <= 0 || num_src_rows < 0) return fail(UEP_ERR_INVALID, "gather_rows: bad sizes");
    if (num_rows == 0) return UEP_OK;
    if (!in || !pos || !out) return fail(UEP_ERR_INVALID, "gather_rows: null pointer");
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    DeviceStatus* st = reinterpret_cast<DeviceStatus*>(status);
    const bool aligned = (row_bytes % 16 == 0) && ((reinterpret_cast<uintptr_t>(in) & 15u) == 0) &&
                         ((reinterpret_cast<uintptr_t>(out) & 15u) == 0);
    count_launch();
    if (aligned) {
        const int chunks = static_cast<int>((row_bytes + kGatherChunk - 1) / kGatherChunk);
        const size_t smem = static_cast<size_t>(kGatherStages) * kGatherChunk;
        UEP_CUDA_TRY(ensure_smem_attr(reinterpret_cast<const void*>(gather_rows_kernel), smem));
        const int64_t sms = device_sm_count() > 0 ? device_sm_count() : 1;
        // as many rows an item as fit its stage, as long as every CTA still gets four items
        int rows = 1;
        while (rows < 32 && 2 * rows * row_bytes <= kGatherChunk && num_rows >= 8 * rows * 2 * sms) rows *= 2;
        int64_t ctas = chunks > 1 ? num_rows * chunks : (num_rows + rows - 1) / rows;
        if (ctas > 2 * sms) ctas = 2 * sms;  // two CTAs of one warp per SM
        UEP_CUDA_TRY(launch_dependent(gather_rows_kernel, dim3(static_cast<unsigned>(ctas)), dim3(32), smem, stream, true,
                                      static_cast<const uint8_t*>(in), pos, static_cast<uint8_t*>(out), num_rows, row_bytes, rows, chunks,
                                      num_src_rows, static_cast<uint64_t>(2000000000ull), st));
    } else {
        const int64_t sms = device_sm_count() > 0 ? device_sm_count() : 1;
        int64_t ctas = num_rows > sms * 8 ? sms * 8 : num_rows;
        gather_rows_plain_kernel<<<static_cast<int>(ctas), 256, 0, stream>>>(
            static_cast<const uint8_t*>(in), pos, static_cast<uint8_t*>(out), num_rows, row_bytes, num_src_rows, st);
    }
    UEP_CUDA_TRY(cudaGetLastError());
    return UEP_OK;
}

}  // extern "C"
