// The candidate leaf pairs of a CG_DFS_ORDER step in the order of the
// reference's recursion (OBBtree::IntersectOBBtreesRecursive,
// src/Geometry/OBBtree.cpp:414-476): grouped by query, each query's by the
// 128-bit descent paths that leaf_keys_kernel (cg_contacts.cu) found. Ordered
// when they are first read: their numbers are known by then, so that only the
// launches that the list needs are made, none for an empty one (in the step,
// with launches for the longest possible list, one pair's mid phase without
// leaf pairs took 76 us instead of 60).
//
//   leaf_few      a list of at most a tile: one block sorts it by query and path
//                 and writes it out
//
// A longer one:
//
//   leaf_offsets  one block: the queries' places (prefix sums of their counts,
//                 which leaf_keys counted) and their tiles of kLeafTile
//   leaf_group    a thread per leaf pair: its path and list index into its
//                 query's place
//   leaf_tiles    a block per tile: a bitonic sort in shared memory; a query
//                 of one tile is written out
//   leaf_merge    a thread per leaf pair of the larger queries: its place among
//                 32 sorted runs is its place in its own plus its lower bounds
//                 in the others (independent binary searches), so each launch
//                 makes runs 32 times longer; a query that is one run is
//                 written out. As many launches as the query with the most
//                 needs
//
// Of the two buffers of paths the first is the output's own memory (a record
// has a path's size) and the second the list-ordered paths', done with once
// they are grouped; the second buffer of indexes is the places'. So a leaf pair
// takes 24 bytes beside the list and the output (60 with buffers of their own).
// A tile is read before its block writes it out; a merge that reads the first
// buffer leaves the query for the next one, which reads the second, to write
// out.
//
// All of it is memory latency: 155,000 leaf pairs of 250 queries take 67 us
// (tiles 32, merges 26) where reading paths and pairs back and sorting them on
// the host took 3.6 ms.
#include <cuda_runtime.h>

#include "cg_internal.h"

namespace cg {

namespace {

constexpr uint32_t kLeafTile = 1024, kLeafWays = 32;

static_assert(sizeof(cg_leaf_pair) == sizeof(ulonglong2), "the output's memory holds a path per leaf pair");
__device__ __forceinline__ bool before(ulonglong2 a, ulonglong2 b) { return a.x < b.x || (a.x == b.x && a.y < b.y); }

// Leaf pair i of the list, as read back, to place pos.
__device__ __forceinline__ void emit(const LeafOrderParams& P, uint32_t pos, uint32_t i) {
    const uint4 e = P.leaf_list[i];
    const PackedQuery* Q = P.q + e.x;
    cg_leaf_pair lp;
    lp.query = e.x;
    lp.offset_a = e.y - __ldg(&Q->tri_base_a);
    lp.offset_b = e.z - __ldg(&Q->tri_base_b);
    lp.count_a = uint16_t(e.w & 0xffffu);
    lp.count_b = uint16_t(e.w >> 16);
    P.out[pos] = lp;
}

// Entry of leaf_few's sort.
struct FewKey {
    ulonglong2 path;
    uint32_t query, id;
};
__device__ __forceinline__ bool before(const FewKey& a, const FewKey& b) {
    if (a.query != b.query) return a.query < b.query;
    if (a.path.x != b.path.x) return a.path.x < b.path.x;
    return a.path.y != b.path.y ? a.path.y < b.path.y : a.id < b.id;
}

__global__ void __launch_bounds__(512) leaf_few_kernel(const LeafOrderParams P) {
    __shared__ FewKey key[kLeafTile];
    const uint32_t tid = threadIdx.x;
    uint32_t size = 1;
    while (size < P.n) size <<= 1;
    for (uint32_t k = tid; k < size; k += 512u)
        key[k] = k < P.n ? FewKey{P.keys[k], P.leaf_list[k].x, k} : FewKey{make_ulonglong2(~0ull, ~0ull), ~0u, ~0u};
    __syncthreads();
    for (uint32_t width = 2; width <= size; width <<= 1)
        for (uint32_t step = width >> 1; step; step >>= 1) {
            for (uint32_t p = tid; p < size / 2u; p += 512u) {
                const uint32_t i = 2u * p - (p & (step - 1u)), j = i + step;
                const FewKey x = key[i], y = key[j];
                if (before(y, x) == ((i & width) == 0u)) key[i] = y, key[j] = x;
            }
            __syncthreads();
        }
    for (uint32_t k = tid; k < P.n; k += 512u) emit(P, k, key[k].id);
}

__global__ void __launch_bounds__(1024) leaf_offsets_kernel(const LeafOrderParams P) {
    __shared__ unsigned long long warp_sum[32];
    const uint32_t tid = threadIdx.x, lane = tid & 31u, w = tid >> 5;
    unsigned long long carry = 0;  // leaf pairs | tiles << 32
    for (uint32_t q0 = 0; q0 < P.n_queries; q0 += 1024u) {
        const uint32_t q = q0 + tid;
        const uint32_t c = q < P.n_queries ? P.count[q] : 0u;
        const unsigned long long own = c | (unsigned long long)((c + kLeafTile - 1u) / kLeafTile) << 32;
        unsigned long long inc = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long t = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= uint32_t(o)) inc += t;
        }
        if (lane == 31u) warp_sum[w] = inc;
        __syncthreads();
        if (w == 0u) {
            unsigned long long v = warp_sum[lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned long long t = __shfl_up_sync(0xffffffffu, v, o);
                if (lane >= uint32_t(o)) v += t;
            }
            warp_sum[lane] = v;
        }
        __syncthreads();
        const unsigned long long before_me = carry + (w ? warp_sum[w - 1u] : 0ull) + (inc - own);
        if (q < P.n_queries) {
            P.first[q] = uint32_t(before_me);
            P.tile[q] = uint32_t(before_me >> 32);
        }
        carry += warp_sum[31];
        __syncthreads();
    }
    if (tid == 0u) P.tile[P.n_queries] = uint32_t(carry >> 32);
}

__global__ void __launch_bounds__(256) leaf_group_kernel(const LeafOrderParams P) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < P.n; i += gridDim.x * blockDim.x) {
        const uint32_t pos = P.first[P.leaf_list[i].x] + P.place[i];
        P.key[0][pos] = P.keys[i];
        P.index[0][pos] = i;
    }
}

__global__ void __launch_bounds__(512) leaf_tiles_kernel(const LeafOrderParams P) {
    __shared__ ulonglong2 key[kLeafTile];
    __shared__ uint32_t id[kLeafTile];
    const uint32_t tid = threadIdx.x, tiles = P.tile[P.n_queries];
    for (uint32_t t = blockIdx.x; t < tiles; t += gridDim.x) {
        // the tile's query: the last whose first tile is at or before it (a
        // query without leaf pairs has the next one's)
        uint32_t a = 0, b = P.n_queries - 1u;
        while (a < b) {
            const uint32_t m = (a + b + 1u) >> 1;
            if (P.tile[m] <= t)
                a = m;
            else
                b = m - 1u;
        }
        const uint32_t count = P.count[a], at = (t - P.tile[a]) * kLeafTile, base = P.first[a] + at;
        const uint32_t m = min(count - at, kLeafTile);
        uint32_t size = 1;
        while (size < m) size <<= 1;
        for (uint32_t k = tid; k < size; k += 512u) {
            key[k] = k < m ? P.key[0][base + k] : make_ulonglong2(~0ull, ~0ull);
            id[k] = k < m ? P.index[0][base + k] : 0xffffffffu;
        }
        __syncthreads();
        for (uint32_t width = 2; width <= size; width <<= 1)
            for (uint32_t step = width >> 1; step; step >>= 1) {
                for (uint32_t p = tid; p < size / 2u; p += 512u) {
                    const uint32_t i = 2u * p - (p & (step - 1u)), j = i + step;
                    const ulonglong2 x = key[i], y = key[j];
                    const uint32_t u = id[i], v = id[j];
                    const bool swap = before(y, x) || (x.x == y.x && x.y == y.y && v < u);
                    if (swap == ((i & width) == 0u)) {
                        key[i] = y, key[j] = x;
                        id[i] = v, id[j] = u;
                    }
                }
                __syncthreads();
            }
        for (uint32_t k = tid; k < m; k += 512u) {
            if (count <= kLeafTile) {
                emit(P, base + k, id[k]);
            } else {
                P.key[1][base + k] = key[k];
                P.index[1][base + k] = id[k];
            }
        }
        __syncthreads();
    }
}

// Merges runs of `run` leaf pairs, from buffer `from` into the other.
__global__ void __launch_bounds__(256) leaf_merge_kernel(const LeafOrderParams P, uint64_t run, uint32_t from) {
    const ulonglong2* key = P.key[from];
    for (uint32_t pos = blockIdx.x * blockDim.x + threadIdx.x; pos < P.n; pos += gridDim.x * blockDim.x) {
        // its query: the last whose first place is at or before pos
        uint32_t a = 0, b = P.n_queries - 1u;
        while (a < b) {
            const uint32_t m = (a + b + 1u) >> 1;
            if (P.first[m] <= pos)
                a = m;
            else
                b = m - 1u;
        }
        const uint32_t first = P.first[a], count = P.count[a];
        if (count <= run) {  // written out already, or one run since the merge before this one
            if (from == 1u && run > kLeafTile && count > run / kLeafWays) emit(P, pos, P.index[1][pos]);
            continue;
        }
        const uint32_t i = P.index[from][pos];
        const ulonglong2 k = key[pos];
        const uint64_t wide = run * kLeafWays, local = pos - first, group = local / wide * wide;
        const uint32_t mine = uint32_t((local - group) / run);
        const uint64_t end = min(uint64_t(count), group + wide);
        uint64_t rank = local - group - mine * run;
        for (uint32_t s = 0; s < kLeafWays && group + s * run < end; ++s) {
            if (s == mine) continue;
            const ulonglong2* r = key + first + group + s * run;
            uint32_t lo = 0, hi = uint32_t(min(run, end - (group + s * run)));
            while (lo < hi) {  // a tie goes to the earlier run
                const uint32_t m = (lo + hi) >> 1;
                const bool left = s < mine ? !before(k, r[m]) : before(r[m], k);
                if (left)
                    lo = m + 1u;
                else
                    hi = m;
            }
            rank += lo;
        }
        const uint32_t to = uint32_t(first + group + rank);
        if (from == 1u && count <= wide) {
            emit(P, to, i);
        } else {
            P.key[from ^ 1u][to] = k;
            P.index[from ^ 1u][to] = i;
        }
    }
}

}  // namespace

cudaError_t launch_leaf_order(const LeafOrderParams& p, uint32_t sm_count, cudaStream_t s) {
    if (p.n == 0) return cudaSuccess;
    if (p.n <= kLeafTile) {
        leaf_few_kernel<<<1, 512, 0, s>>>(p);
        return cudaGetLastError();
    }
    leaf_offsets_kernel<<<1, 1024, 0, s>>>(p);
    leaf_group_kernel<<<8u * sm_count, 256, 0, s>>>(p);
    leaf_tiles_kernel<<<4u * sm_count, 512, 0, s>>>(p);
    uint32_t from = 1;
    // (the last merge is one that writes out)
    for (uint64_t run = kLeafTile; run < p.most || (from == 1u && run > kLeafTile); run *= kLeafWays, from ^= 1u)
        leaf_merge_kernel<<<8u * sm_count, 256, 0, s>>>(p, run, from);
    return cudaGetLastError();
}

}  // namespace cg
