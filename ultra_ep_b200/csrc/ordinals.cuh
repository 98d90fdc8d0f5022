// Ordinals of keys inside their buckets: for every entry of an id array, how many entries in front of it (row-major)
// name the same expert. The sparse reroute and the dispatch positions are this plus a look-up.
//
// The entries of a rank are cut into chunks, one thread-block cluster per chunk; a warp takes `iters` x 32 entries in
// a row, in cluster, CTA, warp order. What lies in front of a chunk is counted again by its own cluster (its CTAs
// share that work): up to a few hundred thousand entries the repeated counting is one or two microseconds against a
// launch and the gap behind it. Where it is not allowed (the ids are replaced in place, a neighbour may already have
// been overwritten) or too much (it grows with the square of the input), a count kernel in front leaves a table of
// tile counts, a tile being one CTA's entries. The CTAs of a cluster hand each other their totals through
// distributed shared memory; no CTA waits for another cluster.
//
// All of it is latency, not bandwidth: 4*T*K bytes are a few hundred KB. So a warp issues the loads of all its
// entries at once, keeps the entries in registers, and takes the positions inside the warp with ballots and one
// shared-memory counter per (warp, bucket).
#pragma once

#include "common.cuh"

namespace uep {

constexpr int kOrdThreads = 512;                   // threads of a CTA ...
constexpr int kOrdWarps = kOrdThreads / kWarp;
constexpr int kOrdFewThreads = 128;                // ... or, where 16 rows of counters do not fit shared memory, these
constexpr int kOrdMaxCluster = 8;  // the portable limit

__device__ __forceinline__ void cp_async_16(void* smem_dst, const void* gsrc) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(smem_dst)), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async_4(void* smem_dst, const void* gsrc) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_addr(smem_dst)), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// the four words at the same place of another CTA's shared memory
__device__ __forceinline__ int4 ld_cluster_v4(const int4* own, int cta) {
    uint32_t a;
    int4 v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_addr(own)), "r"(cta));
    asm volatile("ld.shared::cluster.v4.s32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
    return v;
}

// bucket of a key: itself when in [0,nb_valid), else the last bucket (if there is one) or none
template <typename IdT>
__device__ __forceinline__ int key_bucket(IdT key, int nb_valid, bool tail_bucket) {
    if (key >= 0 && key < nb_valid) return static_cast<int>(key);
    return tail_bucket ? nb_valid : -1;
}

__host__ __device__ __forceinline__ int ord_row(int nb) { return (nb + 7) / 8 * 8; }  // a warp's row of 16-bit counters

struct OrdShared {
    int4* totals;        // what the other CTAs of the cluster read: {front, front + own, front + own + behind, 0}
    int32_t* base;       // this CTA's share of the entries in front of the chunk, then the caller's from finish() on
    int32_t* behind;     // ... and behind the chunk, likewise (only where the grand totals are wanted)
    uint16_t* counters;  // [warps][ord_row(nb)]
};
__host__ __device__ __forceinline__ size_t ord_smem_bytes(int nb, int threads) {
    return static_cast<size_t>(ord_row(nb)) * (16 + 2 * 4 + threads / kWarp * 2);
}
__device__ __forceinline__ OrdShared carve_ord_smem(char* raw, int nb) {  // raw: 16-byte aligned
    const int row = ord_row(nb);
    OrdShared o;
    o.totals = reinterpret_cast<int4*>(raw);
    o.base = reinterpret_cast<int32_t*>(o.totals + row);
    o.behind = o.base + row;
    o.counters = reinterpret_cast<uint16_t*>(o.behind + row);
    return o;
}

// Counts keys[begin, end) into hist (shared memory), all threads of the CTA.
template <typename IdT>
__device__ __forceinline__ void count_keys(const IdT* __restrict__ keys, int64_t begin, int64_t end, int nb_valid, bool tail_bucket,
                                           int32_t* hist) {
    constexpr int kVec = 16 / sizeof(IdT);
    const int nthreads = blockDim.x;
    struct alignas(16) Vec {
        IdT k[kVec];
    };
    int64_t i0 = begin;
    if (((reinterpret_cast<uintptr_t>(keys + begin)) & 15u) == 0) {
        const int64_t nvec = (end - begin) / kVec;
        const uint4* src = reinterpret_cast<const uint4*>(keys + begin);
        for (int64_t j0 = threadIdx.x; j0 < nvec; j0 += 4 * nthreads) {
            uint4 raw[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                if (j0 + u * nthreads < nvec) raw[u] = __ldg(src + j0 + u * nthreads);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                if (j0 + u * nthreads < nvec) {
                    const Vec v = *reinterpret_cast<const Vec*>(&raw[u]);
#pragma unroll
                    for (int c = 0; c < kVec; ++c) {
                        const int b = key_bucket<IdT>(v.k[c], nb_valid, tail_bucket);
                        if (b >= 0) atomicAdd(hist + b, 1);
                    }
                }
            }
        }
        i0 = begin + nvec * kVec;
    }
    for (int64_t i = i0 + threadIdx.x; i < end; i += nthreads) {
        const int b = key_bucket<IdT>(keys[i], nb_valid, tail_bucket);
        if (b >= 0) atomicAdd(hist + b, 1);
    }
}

// The table of the two-launch form: row `tile` holds the bucket counts of entries [tile * tile_entries, + tile_entries).
template <typename IdT>
__device__ __forceinline__ void count_tile(const IdT* keys, int64_t n, int nb_valid, bool tail_bucket, int tile_entries, int32_t* table) {
    extern __shared__ __align__(128) char smem_raw[];
    int32_t* hist = reinterpret_cast<int32_t*>(smem_raw);
    const int nthreads = blockDim.x;
    const int nb = nb_valid + (tail_bucket ? 1 : 0);
    const int64_t begin = static_cast<int64_t>(blockIdx.x) * tile_entries;
    if (begin >= n) return;  // a tile behind this rank's entries is read by nobody
    for (int b = threadIdx.x; b < nb; b += nthreads) hist[b] = 0;
    __syncthreads();
    count_keys<IdT>(keys, begin, min(begin + tile_entries, n), nb_valid, tail_bucket, hist);
    __syncthreads();
    for (int b = threadIdx.x; b < nb; b += nthreads) table[static_cast<int64_t>(blockIdx.x) * nb + b] = hist[b];
}

// Adds the table's rows first, first + step, ... < end to acc (shared memory). The whole CTA shares the rows so that one or
// two memory round trips do: next to weight_sync each takes several microseconds, and a thread per bucket that walked
// 63 rows eight at a time made this 40 us.
__device__ __forceinline__ void add_rows(const int32_t* __restrict__ table, int nb, int64_t first, int64_t end, int step, int32_t* acc) {
    const int nthreads = blockDim.x;
    if ((nb & 3) == 0 && (reinterpret_cast<uintptr_t>(table) & 15u) == 0 && nb / 4 <= nthreads) {
        const int groups = nb / 4, parts = nthreads / groups;
        const int g = threadIdx.x % groups, part = threadIdx.x / groups;
        if (part >= parts) return;
        int4 sum = make_int4(0, 0, 0, 0);
        for (int64_t t0 = first + static_cast<int64_t>(part) * step; t0 < end; t0 += 8LL * parts * step) {
            int4 v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int64_t t = t0 + static_cast<int64_t>(u) * parts * step;
                v[u] = t < end ? __ldcg(reinterpret_cast<const int4*>(table + t * nb) + g) : make_int4(0, 0, 0, 0);
            }
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                sum.x += v[u].x; sum.y += v[u].y; sum.z += v[u].z; sum.w += v[u].w;
            }
        }
        if (sum.x) atomicAdd(acc + g * 4, sum.x);
        if (sum.y) atomicAdd(acc + g * 4 + 1, sum.y);
        if (sum.z) atomicAdd(acc + g * 4 + 2, sum.z);
        if (sum.w) atomicAdd(acc + g * 4 + 3, sum.w);
        return;
    }
    for (int b = threadIdx.x; b < nb; b += nthreads) {
        int sum = 0;
#pragma unroll 8
        for (int64_t t = first; t < end; t += step) sum += __ldcg(table + t * nb + b);
        acc[b] = sum;
    }
}

// Run by all threads of every CTA of the rank's clusters (`ctas` CTAs each). Fills packed[i] of the calling thread's entries
// begin + i * 32 + lane < end: (position among the warp's entries of the bucket) << 16 | bucket, 0xFFFFFFFF for an
// entry without a bucket; and, once finish(b, base, all) has been called for every bucket by one thread of the CTA, the
// ordinal of an entry is base + counters[warp][b] + position. `staged` runs once the caller's own cp.async copies have
// landed, all threads. With kAll, `all` is the number of entries of the bucket in the whole input (else 0).
// `table`: the counts of the kernel in front (tiles of EPT entries a thread), or null. Without a table and with more than
// one cluster the keys must not be overwritten. Ends with a CTA barrier.
// No CTA may leave while another one may still read its totals: with ctas > 1 the caller arrives on the cluster barrier
// behind this and waits on it before it exits.
template <int EPT, bool kAll, typename IdT, typename Staged, typename Finish>
__device__ __forceinline__ void cluster_ordinals(const IdT* keys, int64_t n, int nb_valid, bool tail_bucket, int ctas,
                                                 const int32_t* __restrict__ table, const OrdShared& o, int64_t& begin,
                                                 int64_t& end, int& iters, uint32_t (&packed)[EPT], Staged staged, Finish finish) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nthreads = blockDim.x, warps = nthreads / kWarp;
    const int nb = nb_valid + (tail_bucket ? 1 : 0), row = ord_row(nb);
    const int clusters = gridDim.x / ctas, chunk = blockIdx.x / ctas, cta = blockIdx.x % ctas;
    const int64_t cta_threads = static_cast<int64_t>(ctas) * nthreads;
    iters = table != nullptr ? EPT : static_cast<int>((n + clusters * cta_threads - 1) / (clusters * cta_threads));
    const int64_t chunk_entries = cta_threads * iters;
    begin = min(chunk * chunk_entries + (static_cast<int64_t>(cta) * warps + warp) * iters * kWarp, n);
    end = min(begin + static_cast<int64_t>(iters) * kWarp, n);
    uint16_t* mine = o.counters + warp * row;

    IdT key[EPT];
#pragma unroll
    for (int i = 0; i < EPT; ++i) {
        const int64_t at = begin + i * kWarp + lane;
        key[i] = (i < iters && at < end) ? keys[at] : static_cast<IdT>(-1);
    }
    for (int b = lane; b < nb; b += kWarp) mine[b] = 0;
    if (clusters > 1) {
        for (int b = tid; b < nb; b += nthreads) {
            o.base[b] = 0;
            if (kAll) o.behind[b] = 0;
        }
        __syncthreads();
    }
    if (table == nullptr && clusters > 1) {
        // this CTA's share of the other chunks: shares are multiples of the CTA's threads, so aligned inputs stay aligned
        const int64_t front_share = chunk_entries / ctas * chunk;
        count_keys<IdT>(keys, min(cta * front_share, n), min((cta + 1) * front_share, n), nb_valid, tail_bucket, o.base);
        if (kAll) {
            const int64_t first = min((chunk + 1) * chunk_entries, n);
            const int64_t share = ((n - first + ctas - 1) / ctas + 3) / 4 * 4;
            count_keys<IdT>(keys, min(first + cta * share, n), min(first + (cta + 1) * share, n), nb_valid, tail_bucket, o.behind);
        }
    }
    __syncwarp();
    // Lanes with the same bucket: one ballot per bit of the bucket number, the entries of a lane side by side. Entries
    // without a bucket carry the number nb; the tail bucket is for keys outside [0, nb_valid), not for entries behind the end.
    int bucket[EPT];
    unsigned peers[EPT];
#pragma unroll
    for (int i = 0; i < EPT; ++i) {
        const int b = begin + i * kWarp + lane < end ? key_bucket<IdT>(key[i], nb_valid, tail_bucket) : -1;
        bucket[i] = b >= 0 ? b : nb;
        peers[i] = kFullMask;
    }
    for (int bit = 31 - __clz(nb); bit >= 0; --bit) {
#pragma unroll
        for (int i = 0; i < EPT; ++i) {
            const bool set = (bucket[i] >> bit) & 1;
            const unsigned with = __ballot_sync(kFullMask, set);
            peers[i] &= set ? with : ~with;
        }
    }
    // only the counter update is a chain
#pragma unroll
    for (int i = 0; i < EPT; ++i) {
        packed[i] = 0xFFFFFFFFu;
        if (i < iters) {
            const bool valid = bucket[i] < nb;
            const int before = __popc(peers[i] & ((1u << lane) - 1u));
            const int c = valid ? mine[bucket[i]] : 0;
            __syncwarp();
            if (valid && before == 0) mine[bucket[i]] = static_cast<uint16_t>(c + __popc(peers[i]));
            __syncwarp();
            if (valid) packed[i] = static_cast<uint32_t>(c + before) << 16 | static_cast<uint32_t>(bucket[i]);
        }
    }
    if (table != nullptr) {
        pdl_wait();  // the table is complete, and nobody else reads the keys any more, from here on
        const int64_t tiles = (n + EPT * nthreads - 1) / (EPT * nthreads);
        add_rows(table, nb, cta, min(static_cast<int64_t>(chunk) * ctas, tiles), ctas, o.base);
        if (kAll) add_rows(table, nb, static_cast<int64_t>(chunk + 1) * ctas + cta, tiles, ctas, o.behind);
    }
    cp_async_wait();
    __syncthreads();
    staged();
    // exclusive scan of the warps' counters, bucket by bucket
    for (int b = tid; b < nb; b += nthreads) {
        int c[kOrdWarps];
#pragma unroll
        for (int w = 0; w < kOrdWarps; ++w) c[w] = w < warps ? o.counters[w * row + b] : 0;
        int run = 0;
#pragma unroll
        for (int w = 0; w < kOrdWarps; ++w) {
            if (w < warps) o.counters[w * row + b] = static_cast<uint16_t>(run);
            run += c[w];
        }
        const int f = clusters > 1 ? o.base[b] : 0, h = kAll && clusters > 1 ? o.behind[b] : 0;
        if (ctas > 1) o.totals[b] = make_int4(f, f + run, f + run + h, 0);
        else finish(b, f, f + run + h);
    }
    if (ctas > 1) {
        cluster_arrive();
        cluster_wait();
        for (int b = tid; b < nb; b += nthreads) {
            int before = 0, all = 0;
#pragma unroll
            for (int c = 0; c < kOrdMaxCluster; ++c) {
                if (c < ctas) {
                    const int4 t = ld_cluster_v4(o.totals + b, c);
                    before += c < cta ? t.y : t.x;
                    all += t.z;
                }
            }
            finish(b, before, kAll ? all : 0);
        }
    }
    __syncthreads();
}

}  // namespace uep
