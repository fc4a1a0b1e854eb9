// Collision kernels for sm_103a: query packing, counter reset, record surfaces,
// the persistent warp-cooperative OBB-tree traversal, and the persistent
// triangle-pair (Moller) narrow phase.
//
// Traversal. A worker is a block of one, two or four warps that share a deque of
// items in shared memory and advance it a step at a time: up to 32 items per
// warp, an item being a split node whose two children are tested against the
// other tree's box. A step loads the box records (four 16-byte loads each) and
// the query's matrix, moves B's box into A's space, runs the 15-axis SAT (the
// filter of cg_sat.cuh) and applies the reference's descent rule
// (OBBtree::IntersectOBBtreesRecursive, src/Geometry/OBBtree.cpp:414-476): two
// inner nodes -> split the one with the larger surface, ties to the first
// tree; one leaf -> split the other; two leaves -> a candidate leaf pair.
// Surviving child pairs are pushed with __ballot_sync/__popc compaction;
// candidate leaf pairs are buffered per worker and appended to a global list
// in batches.
//
// Load balance uses a global task queue. Tasks are the root items of the
// queries, which the workers take first, and chunks of up to 32 items. A
// worker whose deque runs dry claims the next chunk slot and waits for it; a
// worker with surplus gives chunks from the bottom (shallowest) part of its
// deque to waiting workers, with one atomic per donation. Every wait is
// bounded by wait_ns (globaltimer), after which the kernel records
// ERR_TIMEOUT and returns.
//
// Narrow phase. Each warp takes 32 leaf pairs of the list at a time and runs
// their triangle pairs, one pair per lane.
#include <cuda_runtime.h>

#include <algorithm>

#include "cg_device.cuh"
#include "cg_internal.h"
#include "cg_sat.cuh"

namespace cg {

namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr unsigned kPollSleepMaxNs = 256;  // longest sleep of a waiting warp between two looks at its slot

__device__ __forceinline__ unsigned long long gtimer() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ unsigned ld_relaxed(const unsigned* p) {
    unsigned v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ unsigned long long ld_relaxed64(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release(unsigned* p, unsigned v) {
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ uint4 ld_relaxed4(const uint4* p) {
    uint4 v;
    asm volatile("ld.relaxed.gpu.global.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p)
                 : "memory");
    return v;
}
__device__ __forceinline__ unsigned lanemask_lt() {
    unsigned m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// head in the low 32 bits, tail in the high 32 bits.
__device__ __forceinline__ unsigned long long* ht_of(Counters* c) {
    return reinterpret_cast<unsigned long long*>(&c->head);
}
__device__ __forceinline__ uint32_t ht_head(unsigned long long v) { return uint32_t(v); }
__device__ __forceinline__ uint32_t ht_tail(unsigned long long v) { return uint32_t(v >> 32); }

// True once every task (the queries' roots and the donated chunks) has
// finished. `done` is read (acquire) before the tail: done(t1) == n_queries +
// tail(t2) with t1 < t2 implies no task was running at t1 and none could be
// reserved afterwards.
__device__ __forceinline__ bool all_done(const TraverseParams& P) {
    const unsigned d = ld_acquire(&P.ctr->done);
    return d == P.n_queries + ht_tail(ld_relaxed64(ht_of(P.ctr)));
}

struct Rec {
    Box box;
    uint32_t ref;
    uint32_t meta;
    float surf;
};

__device__ __forceinline__ Rec load_rec(const float4* recs, uint32_t r) {
    const float4* p = recs + 4ull * r;
    const float4 a = __ldg(p), b = __ldg(p + 1), c = __ldg(p + 2), d = __ldg(p + 3);
    Rec R;
    R.box.c = make_float3(a.x, a.y, a.z);
    R.box.u = make_float3(a.w, b.x, b.y);
    R.box.v = make_float3(b.z, b.w, c.x);
    R.box.w = make_float3(c.y, c.z, c.w);
    R.ref = __float_as_uint(d.x);
    R.meta = __float_as_uint(d.y);
    R.surf = d.z;
    return R;
}

__device__ __forceinline__ Mat4 load_mat(const PackedQuery* Q) {
    Mat4 M;
    M.c0 = __ldg(&Q->m[0]);
    M.c1 = __ldg(&Q->m[1]);
    M.c2 = __ldg(&Q->m[2]);
    M.c3 = __ldg(&Q->m[3]);
    return M;
}

__device__ __forceinline__ void load_tri(const float4* tris, uint32_t i, float3& p0, float3& p1, float3& p2) {
    const float4* p = tris + 3ull * i;
    const float4 a = __ldg(p), b = __ldg(p + 1), c = __ldg(p + 2);
    p0 = make_float3(a.x, a.y, a.z);
    p1 = make_float3(b.x, b.y, b.z);
    p2 = make_float3(c.x, c.y, c.z);
}

// Whether boxes a and b overlap on every axis of `open` (bits as sat_axis
// numbers them): the filter's undecided axes, 1 in 3,000 box pairs.
__device__ __noinline__ bool overlap_on_axes(const Box& a, const Box& b, unsigned open) {
    do {
        const uint32_t k = uint32_t(__ffs(int(open))) - 1u;
        if (!sat_axis(a, b, k)) return false;
        open &= open - 1u;
    } while (open);
    return true;
}
__device__ __noinline__ float surface_of(const Box& b) { return surface(b); }

// What a child pair gives: an item, a candidate leaf pair or (kNone) nothing,
// with its three words.
enum : int { kNone = 0, kItem = 1, kLeaf = 2 };
struct Out {
    int what;
    uint32_t q, s, o;
};

// The reference descent rule (OBBtree.cpp:414-476) for a child pair whose
// boxes overlap: split the inner node with the larger box surface (the first
// tree's on ties), else the inner one, or report a leaf pair. C is the child
// record (record rc) of the split node, O the other box (record io), bx the
// child pair's box of the second tree as transformed for the SAT; `surf` is
// within `surf_err` of its surface (the surface itself is computed only where
// that does not settle the comparison).
__device__ __forceinline__ Out descend(const TraverseParams& P, bool ok, bool sideB, const Rec& O, const Rec& C,
                                       uint32_t rc, uint32_t io, uint32_t qi, const Box& bx, float surf,
                                       float surf_err) {
    const uint32_t a_ref = sideB ? O.ref : C.ref;
    const uint32_t a_meta = sideB ? O.meta : C.meta;
    const float a_surf = sideB ? O.surf : C.surf;
    const uint32_t b_ref = sideB ? C.ref : O.ref;
    const uint32_t b_meta = sideB ? C.meta : O.meta;
    const bool la = (a_meta & kLeafFlag) != 0;
    const bool lb = (b_meta & kLeafFlag) != 0;
    const float diff = a_surf - surf;
    bool larger = diff > 0.0f;
    if (ok && !la && !lb && !(fabsf(diff) > surf_err)) larger = a_surf >= surface_of(bx);
    const bool split_a = !la && (lb || larger);
    const bool both = la && lb;
    Out r;
    r.what = !ok ? kNone : (both ? kLeaf : kItem);
    // a leaf pair: first triangles of both leaves, counts packed; an item: the
    // split node's first child, the other record, the query and side
    r.q = both ? (a_meta & 0xffffu) | (b_meta << 16) : (split_a ? qi : (qi | kItemSideB));
    r.s = (both || split_a) ? a_ref : b_ref;
    r.o = both ? b_ref : (split_a == sideB ? rc : io);
    // the split node's two child records share one 128-byte line: fetch it
    // into L1 for the step that tests them
    if (r.what == kItem) asm volatile("prefetch.global.L1 [%0];" ::"l"(P.recs + 4ull * r.s));
    return r;
}

struct Deque {
    uint32_t* q;
    uint32_t* a;
    uint32_t* b;
    uint32_t mask;
};

// One look at donated slot `slot`: 1 with r = its chunk size + 1 when it can
// be read, 0 with r = 0 when all work finished, an error was raised or the
// wait limit (counted from t0) passed, -1 when it is not ready yet.
__device__ int poll_ready(const TraverseParams& P, uint32_t slot, unsigned long long t0, unsigned& r) {
    r = 0;
    if (slot < P.slot_alloc) {
        r = ld_acquire(P.ready + slot);
        if (r) return 1;
    }
    // past every slot a donor could publish, only the end of the work or an
    // error releases the block
    if (all_done(P) || ld_relaxed(&P.ctr->error) != 0) return 0;
    if (gtimer() - t0 > P.wait_ns) {
        atomicOr(&P.ctr->error, ERR_TIMEOUT);
        return 0;
    }
    return -1;
}

// Adds v busy lanes in `steps` warps' steps to the bucket of the present time.
__device__ __forceinline__ void trace_add(unsigned int* trace, uint32_t trace_ns, unsigned long long t_base, int field,
                                          unsigned v, unsigned steps) {
    const unsigned long long b = (gtimer() - t_base) / trace_ns;
    if (b < kTraceBuckets) {
        atomicAdd(trace + 4 * b + field, v);
        atomicAdd(trace + 4 * b + field + 1, steps);
    }
}

__device__ __forceinline__ unsigned long long trace_base(Counters* ctr) {
    const unsigned long long now = gtimer();
    const unsigned long long old = atomicCAS(&ctr->t_start, 0ull, now);
    return old ? old : now;
}

// One warp's survivors of the plane tests: whole triangle tests still to run.
struct NarrowQueue {
    uint4* e;      // (first triangle, second triangle, leaf-list index, query), 64 places
    uint32_t n;    // the same in every lane
};
struct NarrowCounts {
    unsigned long long tests = 0, fragile = 0, rechecked = 0, disagree = 0;  // lane 0's
};

// Runs the last m (<= 32) tests of the queue, a lane each, and writes the
// colliding pairs.
template <int kMode>
__device__ __forceinline__ void narrow_run(const NarrowParams& P, NarrowQueue& Q, uint32_t m, int lane, NarrowCounts& N) {
    Q.n -= m;
    __syncwarp();
    int res = TT_MISS;
    uint4 e = make_uint4(0u, 0u, 0u, 0u);
    float3 src = make_float3(0.f, 0.f, 0.f), tgt = src;
    Recheck rck;
    if (uint32_t(lane) < m) {
        e = Q.e[Q.n + lane];
        const Mat4 M = load_mat(P.q + e.w);
        float3 a0, a1, a2, b0, b1, b2;
        load_tri(P.tris, e.x, a0, a1, a2);
        load_tri(P.tris, e.y, b0, b1, b2);
        b0 = xform(M, b0, 1.0f);
        b1 = xform(M, b1, 1.0f);
        b2 = xform(M, b2, 1.0f);
        res = tri_tri_mode<kMode>(a0, a1, a2, b0, b1, b2, src, tgt, rck);
    }
    const unsigned hitmask = __ballot_sync(kFull, res == TT_HIT);
    const unsigned fragmask = __ballot_sync(kFull, res == TT_FRAGILE);
    if (kMode != 0) {
        const unsigned nchk = __reduce_add_sync(kFull, rck.checked);
        const unsigned ndis = __popc(__ballot_sync(kFull, rck.disagree));
        if (lane == 0) {
            N.rechecked += nchk;
            N.disagree += ndis;
        }
    }
    if (hitmask) {
        unsigned long long obase = 0;
        if (lane == 0) obase = atomicAdd(&P.ctr->n_pairs, (unsigned long long)__popc(hitmask));
        obase = __shfl_sync(kFull, obase, 0);
        if (res == TT_HIT && !(P.flags & CG_NO_TRI_PAIRS)) {
            const unsigned long long o = obase + __popc(hitmask & lanemask_lt());
            if (o < P.pairs_cap) {
                const PackedQuery* K = P.q + e.w;
                cg_tri_pair r;
                r.query = e.w;
                r.tri_a = e.x - __ldg(&K->tri_base_a);
                r.tri_b = e.y - __ldg(&K->tri_base_b);
                r.source[0] = src.x;
                r.source[1] = src.y;
                r.source[2] = src.z;
                r.target[0] = tgt.x;
                r.target[1] = tgt.y;
                r.target[2] = tgt.z;
                P.pairs[o] = r;
                if (P.pair_aux) P.pair_aux[o] = e;
            }
        }
    }
    if (lane == 0) N.fragile += __popc(fragmask);
    __syncwarp();
}

// The narrow phase of leaf pairs [first, first + nl) of the list (nl <= 32),
// staged in `stage`; all 32 lanes call it. The entries must be visible to the
// calling warp. Each round runs the plane tests of 32 triangle pairs
// (planes_miss, about 180 instructions with the moving of the second triangle);
// the pairs that they do not reject, 1 in 8, wait in the warp's queue for a
// whole test of 32 at a time: in place, its long rest ran for 4 of 32 lanes in
// every round. 52 M pairs of 10,000 uneven queries: 860 us in place, 716 so
// (a lane per second triangle, its plane kept for the first leaf's: 822).
template <int kMode>
__device__ __forceinline__ void narrow_block(const NarrowParams& P, uint32_t* stage, uint32_t first, uint32_t nl,
                                             int lane, NarrowQueue& Q, NarrowCounts& N, unsigned long long t_base) {
    uint32_t* lq = stage;
    uint32_t* loa = lq + 32;
    uint32_t* lob = loa + 32;
    uint32_t* lcn = lob + 32;
    uint32_t* lrc = lcn + 32;  // ceil(2^16 / count_b), or 0 where the division is done in full
    uint32_t* pre = lrc + 32;  // 33 entries
    uint32_t c0 = 0;
    if (uint32_t(lane) < nl) {
        const uint4 e = P.leaf_list[first + lane];
        lq[lane] = e.x;
        loa[lane] = e.y;
        lob[lane] = e.z;
        lcn[lane] = e.w;
        const uint32_t cb = e.w >> 16;
        c0 = (e.w & 0xffffu) * cb;
        // local / cb == (local * ceil(2^16 / cb)) >> 16 for local < 256, cb <= 16
        lrc[lane] = (cb <= 16u && c0 < 256u) ? (65536u + cb - 1u) / cb : 0u;
        if ((P.flags & CG_KEEP_LEAF_PAIRS) && first + lane < P.leafs_cap) {
            const PackedQuery* Q = P.q + e.x;
            cg_leaf_pair lp;
            lp.query = e.x;
            lp.offset_a = e.y - __ldg(&Q->tri_base_a);
            lp.offset_b = e.z - __ldg(&Q->tri_base_b);
            lp.count_a = uint16_t(e.w & 0xffffu);
            lp.count_b = uint16_t(e.w >> 16);
            P.leafs[first + lane] = lp;
        }
    }
    uint32_t s0 = c0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t0 = __shfl_up_sync(kFull, s0, o);
        if (lane >= o) s0 += t0;
    }
    const uint32_t total = (P.flags & CG_MID_ONLY) ? 0u : __shfl_sync(kFull, s0, 31);
    const uint32_t my_pre = s0 - c0;  // first test of this lane's leaf pair
    pre[lane] = my_pre;
    if (lane == 0) pre[32] = total;
    __syncwarp();

    // The leaf pair of test t: each round, the leaf pairs that start inside
    // the round's 32 tests set their bit, and a lane counts the starts at or
    // below it from the leaf pair that holds the round's first test. A leaf
    // pair without tests (an empty leaf) starts where the next one does; a
    // block with one looks the leaf pair up by binary search instead.
    const bool counted = __all_sync(kFull, uint32_t(lane) >= nl || c0 != 0u);
    uint32_t own0 = 0;
    for (uint32_t base = 0; base < total; base += 32) {
        const uint32_t t = base + lane;
        const int d = int(my_pre) - int(base);
        const bool mine = uint32_t(lane) < nl;
        const unsigned starts = __reduce_or_sync(kFull, (mine && d >= 1 && d <= 31) ? (1u << d) : 0u);
        const bool next_at_32 = __any_sync(kFull, mine && d == 32);
        uint32_t lo = own0 + __popc(starts & ((2u << lane) - 1u));
        own0 += __popc(starts) + (next_at_32 ? 1u : 0u);
        bool keep = false;
        uint4 e = make_uint4(0u, 0u, 0u, 0u);
        if (t < total) {
            if (!counted) {
                int l = 0, h = int(nl) - 1;
                while (l < h) {
                    const int mid = (l + h + 1) >> 1;
                    if (pre[mid] <= t)
                        l = mid;
                    else
                        h = mid - 1;
                }
                lo = uint32_t(l);
            }
            const uint32_t local = t - pre[lo];
            const uint32_t cn = lcn[lo];
            const uint32_t cb = cn >> 16;
            const uint32_t rc = lrc[lo];
            const uint32_t i = rc ? (local * rc) >> 16 : local / cb;
            const uint32_t j = local - i * cb;
            e = make_uint4(loa[lo] + i, lob[lo] + j, first + lo, lq[lo]);
            const Mat4 M = load_mat(P.q + e.w);
            float3 a0, a1, a2, b0, b1, b2;
            load_tri(P.tris, e.x, a0, a1, a2);
            load_tri(P.tris, e.y, b0, b1, b2);
            b0 = xform(M, b0, 1.0f);
            b1 = xform(M, b1, 1.0f);
            b2 = xform(M, b2, 1.0f);
            keep = !planes_miss<kMode>(a0, a1, a2, tri_plane(a0, a1, a2), b0, b1, b2, tri_plane(b0, b1, b2));
        }
        const unsigned kept = __ballot_sync(kFull, keep);
        if (keep) Q.e[Q.n + __popc(kept & lanemask_lt())] = e;
        Q.n += __popc(kept);
        if (lane == 0 && P.trace) trace_add(P.trace, P.trace_ns, t_base, 2, min(32u, total - base), 1u);
        if (Q.n >= 32u) narrow_run<kMode>(P, Q, 32u, lane, N);
    }
    if (lane == 0) N.tests += total;
    __syncwarp();
}

// The words a block's threads share beside its deque and leaf buffer.
struct TraverseShared {
    unsigned push[2];             // this step's pushes so far: items | leaf pairs << 16 (by step parity)
    unsigned long long qs[2];     // the queue's head and tail as read in the step (by step parity)
    unsigned long long leaf_base; // where a flush goes in the list
    uint32_t claim;               // first root or donated slot taken, roots or chunk size taken; 0: the end
    uint32_t claim_n;
    uint32_t claim_root;
    int mode;                     // the donation: slots reserved (1), none (0), queue full (-1)
    uint32_t slot;
};

// Appends the block's buffered leaf pairs to the list (all threads).
__device__ __forceinline__ void flush_leafs(const TraverseParams& P, TraverseShared& sh, const uint32_t* lq,
                                            const uint32_t* loa, const uint32_t* lob, const uint32_t* lcn,
                                            uint32_t nl) {
    if (threadIdx.x == 0) sh.leaf_base = atomicAdd(&P.ctr->n_leafs, (unsigned long long)nl);
    __syncthreads();
    const unsigned long long base = sh.leaf_base;
    for (uint32_t e = threadIdx.x; e < nl; e += blockDim.x)
        if (base + e < P.leaf_cap) P.leaf_list[base + e] = make_uint4(lq[e], loa[e], lob[e], lcn[e]);
}

}  // namespace

constexpr uint32_t kWorkerMax = 4;  // warps of the widest worker block

// A block of W warps is one worker: its warps share a deque of items in
// shared memory and advance it together, one step (two barriers) at a time.
__global__ void __launch_bounds__(kWorkerMax * 32, 2) traverse_kernel(const TraverseParams P) {
    extern __shared__ uint32_t smem[];
    __shared__ TraverseShared sh;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t NT = blockDim.x, W = NT >> 5;
    const uint32_t S = deque_entries(P.stack_cap, W);
    Deque D;
    D.q = smem;
    D.a = D.q + S;
    D.b = D.a + S;
    D.mask = S - 1u;
    uint32_t* lq = D.b + S;
    uint32_t* loa = lq + kLeafCap * W;
    uint32_t* lob = loa + kLeafCap * W;
    uint32_t* lcn = lob + kLeafCap * W;
    unsigned long long* ht = ht_of(P.ctr);

    // the block's state, the same in every thread
    uint32_t top = 0, bot = 0, nl = 0, held_tasks = 0, par = 0;
    bool roots_left = true;
    unsigned long long st_nodes = 0, st_don = 0, st_steps = 0;
    unsigned long long t_base = 0;
    if (P.trace && tid == 0) t_base = trace_base(P.ctr);
    if (tid < 2u) sh.push[tid] = 0u;

    for (;;) {
        if (top == bot) {
            // Out of work: take the next roots, or claim the next donated slot
            // and wait for it (thread 0 looks and sleeps between looks, the
            // others wait at the barrier).
            if (tid == 0) {
                uint32_t n = 0, at = 0, root = 0;
                if (roots_left) {
                    at = atomicAdd(&P.ctr->root_next, P.root_batch);
                    if (at < P.n_queries) {
                        n = min(P.root_batch, P.n_queries - at);
                        root = 1u;
                    }
                }
                if (!root) {
                    at = ht_head(atomicAdd(ht, 1ull));
                    unsigned r = 0;
                    const unsigned long long t0 = gtimer();
                    unsigned ns = 32;
                    while (poll_ready(P, at, t0, r) < 0) {
                        __nanosleep(ns);
                        if (ns < kPollSleepMaxNs) ns <<= 1;
                    }
                    n = r ? r - 1u : 0u;
                }
                sh.claim = at;
                sh.claim_n = n;
                sh.claim_root = root;
            }
            __syncthreads();
            const uint32_t at = sh.claim, cn = sh.claim_n;
            if (cn == 0u) break;
            roots_left = sh.claim_root != 0u;
            held_tasks = roots_left ? cn : 1u;
            if (roots_left) {
                // the first items of queries [at, at + cn), made by the pack kernel
                for (uint32_t k = tid; k < cn; k += NT) {
                    const PackedQuery* Q = P.q + at + k;
                    const uint32_t iq = __ldg(&Q->item_q);
                    if (iq != kNoItem) {
                        const uint32_t pos = atomicAdd(&sh.push[par], 1u) & D.mask;  // the deque is empty: top is 0
                        D.q[pos] = iq;
                        D.a[pos] = __ldg(&Q->item_split);
                        D.b[pos] = __ldg(&Q->item_other);
                    }
                }
                __syncthreads();
                bot = 0;
                top = sh.push[par];
                __syncthreads();
                if (tid == 0) sh.push[par] = 0u;
                if (top == 0u) {
                    if (tid == 0) atomicAdd(&P.ctr->done, held_tasks);
                    __syncthreads();
                    continue;
                }
            } else {
                // thread 0 observed the slot's release; the barrier orders the
                // other threads' pool reads after that acquire
                if (tid < cn) {
                    const uint4 e = ld_relaxed4(P.pool + size_t(kChunk) * at + tid);
                    D.q[tid] = e.x;
                    D.a[tid] = e.y;
                    D.b[tid] = e.z;
                }
                bot = 0;
                top = cn;
            }
            __syncthreads();
        }

        // Queue state, read early so its latency overlaps the step's loads.
        unsigned long long qs = 0;
        if (tid == 0) qs = ld_relaxed64(ht);

        // ---- one step over up to 32 W items from the top of the deque. An item
        // tests both children of a split node against the other box: the
        // other record is loaded (and, for the second tree, transformed) once,
        // the two child records come from one 128-byte line. With more than
        // 16 W items a lane tests an item's two children, with fewer a lane
        // tests one child, both through the SAT filter: about 280
        // instructions a box pair against 900 for the 15 axes as the
        // reference writes them (DRAM and L2 are idle here; issue and the
        // dependent latency of a step bound the launch). With an item per
        // warp or fewer, 16 lanes share a child, an axis each as written (75
        // instructions), so that the single chains at a launch's start and
        // end step fastest. Every verdict is the conjunction of the same 15
        // axes.
        const uint32_t size = top - bot;
        const uint32_t n = min(size, NT);
        // log2 of lanes per item
        const uint32_t lg = n <= W ? 5u : (n <= NT / 2u ? 1u : 0u);
        const uint32_t slot_i = tid >> lg;
        const uint32_t sub = tid & ((1u << lg) - 1u);
        const bool active = slot_i < n;
        uint32_t iq = 0, is = 0, io = 0;
        if (active) {
            const uint32_t pos = (top - n + slot_i) & D.mask;
            iq = D.q[pos];
            is = D.a[pos];
            io = D.b[pos];
        }
        top -= n;
        __syncthreads();  // the popped places are rewritten below
        if (tid == 0) sh.push[par ^ 1u] = 0u;

        // Per lane, per child: a new item (split node, other record, query
        // word) or a candidate leaf pair (triangle offsets and counts).
        Out out0{kNone, 0u, 0u, 0u}, out1 = out0;
        const uint32_t qi = iq & ~kItemSideB;
        const bool sideB = (iq & kItemSideB) != 0;
        if (lg <= 1u) {
            if (active) {
                const Mat4 M = load_mat(P.q + qi);
                const uint32_t first = is + sub;  // the lane's (first) child
                const Rec O = load_rec(P.recs, io);
                const Rec C0 = load_rec(P.recs, first);
                const Box moved = xform_box(M, sideB ? C0.box : O.box);
                const SatBox so = sat_box(sideB ? O.box : moved);
                const Box cb0 = sideB ? moved : C0.box;
                unsigned open0 = 0, open1 = 0;
                float err0, err1;
                if (lg == 0u) {
                    const Rec C1 = load_rec(P.recs, first + 1u);
                    Box cb1 = C1.box;
                    if (sideB) cb1 = xform_box(M, C1.box);
                    const SatBox s0 = sat_box(cb0), s1 = sat_box(cb1);
                    bool ok0 = !sat_filter(so, s0, open0);
                    bool ok1 = !sat_filter(so, s1, open1);
                    const float surf0 = sat_surface(sideB ? s0 : so, err0);
                    const float surf1 = sat_surface(sideB ? s1 : so, err1);
                    if (ok0 && open0) ok0 = overlap_on_axes(so.b, cb0, open0);
                    if (ok1 && open1) ok1 = overlap_on_axes(so.b, cb1, open1);
                    out0 = descend(P, ok0, sideB, O, C0, first, io, qi, sideB ? cb0 : so.b, surf0, err0);
                    out1 = descend(P, ok1, sideB, O, C1, first + 1u, io, qi, sideB ? cb1 : so.b, surf1, err1);
                } else {
                    const SatBox s0 = sat_box(cb0);
                    bool ok0 = !sat_filter(so, s0, open0);
                    const float surf0 = sat_surface(sideB ? s0 : so, err0);
                    if (ok0 && open0) ok0 = overlap_on_axes(so.b, cb0, open0);
                    out0 = descend(P, ok0, sideB, O, C0, first, io, qi, sideB ? cb0 : so.b, surf0, err0);
                }
            }
        } else {
            const uint32_t kc = sub >> 4;   // the child this lane tests
            const uint32_t ax = sub & 15u;  // its axis
            bool ok = true;
            Rec O, C;
            Box bx;
            if (active) {
                const Mat4 M = load_mat(P.q + qi);
                O = load_rec(P.recs, io);
                C = load_rec(P.recs, is + kc);
                bx = xform_box(M, sideB ? C.box : O.box);
                if (ax < 15u) ok = sat_axis(sideB ? O.box : C.box, bx, ax);
            }
            // the child's verdict: none of its 16 lanes found a separating axis
            const unsigned fail = __ballot_sync(kFull, !ok);
            ok = (fail & (0xffffu << (lane & 16u))) == 0u;
            if (active && ax == 0u)
                out0 = descend(P, ok, sideB, O, C, is + kc, io, qi, bx, 0.0f, __int_as_float(0x7f800000));
        }

        // pushes: the warp's places from one shared counter, the lanes' by ballot
        const unsigned i0 = __ballot_sync(kFull, out0.what == kItem), i1 = __ballot_sync(kFull, out1.what == kItem);
        const unsigned l0 = __ballot_sync(kFull, out0.what == kLeaf), l1 = __ballot_sync(kFull, out1.what == kLeaf);
        if (i0 | i1 | l0 | l1) {
            unsigned off = 0;
            if (lane == 0)
                off = atomicAdd(&sh.push[par], (__popc(i0) + __popc(i1)) | (__popc(l0) + __popc(l1)) << 16);
            off = __shfl_sync(kFull, off, 0);
            const unsigned lt = lanemask_lt();
            uint32_t r = top + (off & 0xffffu) + __popc(i0 & lt) + __popc(i1 & lt);
            uint32_t l = nl + (off >> 16) + __popc(l0 & lt) + __popc(l1 & lt);
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const Out& out = k ? out1 : out0;
                if (out.what == kItem) {
                    const uint32_t p = r & D.mask;
                    D.q[p] = out.q;
                    D.a[p] = out.s;
                    D.b[p] = out.o;
                    ++r;
                }
                if (out.what == kLeaf) {
                    lq[l] = qi;
                    loa[l] = out.s;
                    lob[l] = out.o;
                    lcn[l] = out.q;
                    ++l;
                }
            }
        }
        if (tid == 0) {
            sh.qs[par] = qs;
            st_nodes += 2u * n;
            const uint32_t steps = ((n << lg) + 31u) >> 5;  // of warps that hold items
            st_steps += steps;
            if (P.trace) trace_add(P.trace, P.trace_ns, t_base, 0, n, steps);
        }
        __syncthreads();
        const unsigned pushed = sh.push[par];
        top += pushed & 0xffffu;
        nl += pushed >> 16;
        qs = sh.qs[par];
        par ^= 1u;

        if (nl > (P.leaf_flush - 1u) * W) {
            flush_leafs(P, sh, lq, loa, lob, lcn, nl);
            nl = 0;
        }

        // ---- balance: give chunks from the bottom of the deque to the blocks
        // that wait (one chunk per waiting block, keeping at least a chunk; a
        // full chunk when the deque is nearly full). A block does not take
        // queued chunks while it has work: that costs a contended atomic per
        // step and measured slower.
        const uint32_t held = top - bot;
        const bool forced = held + 64u * W > S;
        const int waiting = int(ht_head(qs) - ht_tail(qs));
        if (forced || (waiting > 0 && held >= P.donate_min)) {
            const uint32_t c = held >= 2u * kChunk ? uint32_t(kChunk) : (held >> 1);
            const uint32_t want = max(uint32_t(max(waiting, 1)), forced ? W : 1u);
            const uint32_t nch = max(1u, min(want, min(held / c - 1u, 8u * W)));
            if (tid == 0) {
                int mode = 0;
                if (ht_tail(qs) + nch <= P.slot_cap) {
                    sh.slot = ht_tail(atomicAdd(ht, (unsigned long long)nch << 32));
                    mode = 1;
                } else if (forced) {
                    atomicOr(&P.ctr->error, ERR_QUEUE);
                    mode = -1;
                }
                sh.mode = mode;
            }
            __syncthreads();
            if (sh.mode == -1) break;
            if (sh.mode == 1) {
                const uint32_t slot = sh.slot;
                for (uint32_t k = tid; k < nch * c; k += NT) {
                    const uint32_t ch = k / c, pos = (bot + k) & D.mask;
                    P.pool[size_t(kChunk) * (slot + ch) + (k - ch * c)] = make_uint4(D.q[pos], D.a[pos], D.b[pos], 0u);
                }
                __threadfence();
                __syncthreads();
                for (uint32_t k = tid; k < nch; k += NT) st_release(P.ready + slot + k, c + 1u);
                if (tid == 0) st_don += c * nch;
                bot += c * nch;
            }
        }

        if (top == bot) {
            // every thread has read the shared words of this step's end
            __syncthreads();
            if (tid == 0) atomicAdd(&P.ctr->done, held_tasks);
            held_tasks = 0;
        }
    }

    // remaining buffered leaf pairs
    __syncthreads();
    if (nl) flush_leafs(P, sh, lq, loa, lob, lcn, nl);
    if (tid == 0) {
        if (st_nodes) atomicAdd(&P.ctr->node_pairs, st_nodes);
        if (st_don) atomicAdd(&P.ctr->donations, st_don);
        if (st_steps) atomicAdd(&P.ctr->warp_steps, st_steps);
    }
}

// Runs the triangle pairs of the leaf-pair list, 32 leaf pairs per warp and
// one triangle pair per lane, in the order of the reference's pair loop per
// leaf pair (CreateUncollideRays.cpp:78-86): B's triangle is moved into A's
// space with TrianglePosition::MultiplyBy4x4Matrix arithmetic, then tested.
template <int kMode>
__global__ void __launch_bounds__(256, 3) narrow_kernel(const NarrowParams P) {
    __shared__ uint4 queue[8][64];
    __shared__ uint32_t sm[8 * kNarrowWarpWords];
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    uint32_t* stage = sm + warp * kNarrowWarpWords;
    NarrowQueue Q{queue[warp], 0u};
    NarrowCounts N;

    const unsigned long long n_all = *reinterpret_cast<volatile unsigned long long*>(&P.ctr->n_leafs);
    const uint32_t n = uint32_t(n_all < P.leaf_cap ? n_all : P.leaf_cap);
    unsigned long long t_base = 0;
    if (P.trace && lane == 0) t_base = trace_base(P.ctr);

    // Each warp's first `per` leaf pairs are fixed by its index; later ones
    // come from the shared counter, past all first rounds. A small list
    // costs no atomic to the warps it does not reach, and is spread over all
    // warps (per < 32 leaf pairs each) so that its rounds run side by side.
    const uint32_t n_warps = gridDim.x * (blockDim.x >> 5);
    const uint32_t per = n >= 32u * n_warps ? 32u : max(1u, (n + n_warps - 1u) / n_warps);
    uint32_t first = per * (blockIdx.x * (blockDim.x >> 5) + uint32_t(warp));
    while (first < n) {
        const uint32_t nl = min(per, n - first);
        narrow_block<kMode>(P, stage, first, nl, lane, Q, N, t_base);
        uint32_t next = 0;
        if (lane == 0) next = per * n_warps + atomicAdd(&P.ctr->narrow_lp, per);
        first = __shfl_sync(kFull, next, 0);
    }
    if (Q.n) narrow_run<kMode>(P, Q, Q.n, lane, N);
    if (lane == 0) {
        if (N.tests) atomicAdd(&P.ctr->tri_tests, N.tests);
        if (N.fragile) atomicAdd(&P.ctr->fragile, N.fragile);
        if (kMode != 0) {
            if (N.rechecked) atomicAdd(&P.ctr->rechecked, N.rechecked);
            if (N.disagree) atomicAdd(&P.ctr->disagreements, N.disagree);
        }
    }
}

// One thread per query: packs the relative matrix and runs the root pair the
// way the traversal runs every pair (SAT, then the descent rule), so that the
// query enters the work queue as its first item; a leaf-leaf root goes
// straight to the leaf-pair list.
__global__ void pack_kernel(const cg_query* in, uint32_t n, const DevTree* trees, uint32_t n_trees,
                            const float4* recs, PackedQuery* out, Counters* ctr, uint4* leaf_list, uint32_t leaf_cap) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const cg_query Q = in[i];
    PackedQuery p;
    p.m[0] = make_float4(Q.relative[0], Q.relative[1], Q.relative[2], Q.relative[3]);
    p.m[1] = make_float4(Q.relative[4], Q.relative[5], Q.relative[6], Q.relative[7]);
    p.m[2] = make_float4(Q.relative[8], Q.relative[9], Q.relative[10], Q.relative[11]);
    p.m[3] = make_float4(Q.relative[12], Q.relative[13], Q.relative[14], Q.relative[15]);
    p.item_q = kNoItem;
    p.item_split = p.item_other = p.pad = 0u;
    p.tri_base_a = p.tri_base_b = 0u;
    p.tree_a = Q.tree_a;
    p.tree_b = Q.tree_b;
    const bool ok = Q.tree_a < n_trees && Q.tree_b < n_trees && trees[Q.tree_a].live && trees[Q.tree_b].live;
    if (!ok) {
        atomicOr(&ctr->error, ERR_BAD_QUERY);
        out[i] = p;
        return;
    }
    p.tri_base_a = trees[Q.tree_a].tri_base;
    p.tri_base_b = trees[Q.tree_b].tri_base;
    const uint32_t ra = trees[Q.tree_a].rec_base + 1u;
    const uint32_t rb = trees[Q.tree_b].rec_base + 1u;
    const Mat4 M{p.m[0], p.m[1], p.m[2], p.m[3]};
    const Rec A = load_rec(recs, ra);
    const Rec B = load_rec(recs, rb);
    const Box bb = xform_box(M, B.box);
    {
        // one atomic per group of converged lanes
        const unsigned m = __activemask();
        if ((threadIdx.x & 31u) == unsigned(__ffs(m) - 1)) atomicAdd(&ctr->node_pairs, (unsigned long long)__popc(m));
    }
    if (sat(A.box, bb)) {
        const bool la = (A.meta & kLeafFlag) != 0;
        const bool lb = (B.meta & kLeafFlag) != 0;
        if (la && lb) {
            const unsigned long long idx = atomicAdd(&ctr->n_leafs, 1ull);
            if (idx < leaf_cap) leaf_list[idx] = make_uint4(i, A.ref, B.ref, (A.meta & 0xffffu) | ((B.meta & 0xffffu) << 16));
        } else {
            const bool split_a = (!la && !lb) ? (A.surf >= surface(bb)) : !la;
            p.item_q = split_a ? i : (i | kItemSideB);
            p.item_split = split_a ? A.ref : B.ref;
            p.item_other = split_a ? rb : ra;
        }
    }
    out[i] = p;
}

// Resets the counters for a launch over n_queries and clears the ready flags
// of the slots the previous launch reserved (their count is still in the
// counters), and the trace when it is kept.
__global__ void init_kernel(Counters* ctr, unsigned int* ready, uint32_t slot_alloc, uint32_t n_queries,
                            unsigned int* trace) {
    __shared__ uint32_t used;
    if (threadIdx.x == 0) used = min(ctr->tail, slot_alloc);
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < used; i += blockDim.x) ready[i] = 0u;
    if (trace)
        for (uint32_t i = threadIdx.x; i < 4u * kTraceBuckets; i += blockDim.x) trace[i] = 0u;
    __syncthreads();
    if (threadIdx.x == 0) {
        Counters c = {};
        c.n_queries = n_queries;
        // vertex-set slots stay taken until a contacts launch empties them
        c.prev_vertices = ctr->prev_vertices + ctr->n_vertices;
        *ctr = c;
    }
}

// Paralgram::GetSurface of records [first, first + n_recs), written into q3.z.
__global__ void surfaces_kernel(float4* recs, uint32_t first, uint32_t n_recs) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_recs) return;
    float4* p = recs + 4ull * (first + i);
    const float4 a = p[0], b = p[1], c = p[2];
    Box box;
    box.c = make_float3(a.x, a.y, a.z);
    box.u = make_float3(a.w, b.x, b.y);
    box.v = make_float3(b.z, b.w, c.x);
    box.w = make_float3(c.y, c.z, c.w);
    p[3].z = surface(box);
}

cudaError_t launch_pack(const cg_query* in, uint32_t n, const DevTree* trees, uint32_t n_trees, const float4* recs,
                        PackedQuery* out, Counters* ctr, uint4* leaf_list, uint32_t leaf_cap, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    pack_kernel<<<(n + 127) / 128, 128, 0, s>>>(in, n, trees, n_trees, recs, out, ctr, leaf_list, leaf_cap);
    return cudaGetLastError();
}

cudaError_t launch_init(Counters* ctr, unsigned int* ready, uint32_t slot_alloc, uint32_t n_queries,
                        unsigned int* trace, cudaStream_t s) {
    init_kernel<<<1, 1024, 0, s>>>(ctr, ready, slot_alloc, n_queries, trace);
    return cudaGetLastError();
}

cudaError_t launch_surfaces(float4* recs, uint32_t first, uint32_t n_recs, cudaStream_t s) {
    if (n_recs == 0) return cudaSuccess;
    surfaces_kernel<<<(n_recs + 255) / 256, 256, 0, s>>>(recs, first, n_recs);
    return cudaGetLastError();
}

namespace {
// Warps of a worker block. Two: a worker's steps are wide enough to advance a
// query's whole frontier in most of them, and an SM holds four workers that
// hide one another's latency; a launch of at most one query per eight warps
// has no other work for them, and four warps widen the step further.
// Traversal alone, 1, 2, 4 and 8 warps (us): 1 query of 2 x 2,048 triangles
// 59, 51, 48, 47; 64 of these 85, 67, 58, 64; 150 queries of 2 x 20,000 213,
// 180, 190, 202; the 256-entity scene 131, 103, 110, 119; 10,000 uneven
// queries 1310, 1288, 1392, 1587. The line is where a worker of four warps still
// has a query of its own to itself; from 64 queries up to it two warps are
// somewhat faster for large trees (150 queries: 180 against 190), four for small
// ones.
//
// With the smallest stacks (256 entries) a worker is one warp and takes one root
// at a time: donations that a full stack forces are then the rule, and how many
// of the queue's slots they take decides whether a launch fits its queue. Two
// 32,768-triangle meshes fit 256 slots so and not 64; those of wider workers fit
// 64, or, with half the entries per warp, need 512.
constexpr uint32_t kPoolStack = 512;
uint32_t worker_warps(uint32_t n_queries, uint32_t total_warps, uint32_t stack_cap) {
    if (stack_cap < kPoolStack) return 1u;
    return uint64_t(n_queries) * 8u <= total_warps && total_warps >= 4u ? 4u : (total_warps >= 2u ? 2u : 1u);
}
constexpr uint32_t kStackMax = 4096;  // cg_config.stack_entries' limit
}  // namespace

cudaError_t traverse_occupancy(uint32_t warps_per_block, uint32_t stack_cap, int* blocks_per_sm) {
    // the widest worker's deque at the largest stack: one limit for every
    // context of the process
    cudaError_t e = cudaFuncSetAttribute(traverse_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         int(traverse_smem_words(kStackMax, 4u) * sizeof(uint32_t)));
    if (e != cudaSuccess) return e;
    int device = 0, limit = 0, two = 0, four = 0;
    if ((e = cudaGetDevice(&device)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&limit, cudaDevAttrMaxSharedMemoryPerBlockOptin, device)) != cudaSuccess) return e;
    *blocks_per_sm = 0;
    // a setting whose warps' stacks together are more than a block may hold
    if (size_t(warps_per_block) * (3u * stack_cap + 4u * kLeafCap) * sizeof(uint32_t) > size_t(limit))
        return cudaSuccess;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&two, traverse_kernel, 64,
                                                      traverse_smem_words(stack_cap, 2u) * sizeof(uint32_t));
    if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&four, traverse_kernel, 128,
                                                          traverse_smem_words(stack_cap, 4u) * sizeof(uint32_t));
    const int warps = std::min(2 * two, 4 * four);
    *blocks_per_sm = warps ? std::max(1, warps / int(warps_per_block)) : 0;
    return e;
}

cudaError_t narrow_occupancy(uint32_t warps_per_block, int* blocks_per_sm) {
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, narrow_kernel<0>, int(32 * warps_per_block), 0);
}

cudaError_t launch_traverse(const TraverseParams& p_in, uint32_t blocks, uint32_t warps_per_block, cudaStream_t s) {
    TraverseParams p = p_in;
    const uint32_t total = blocks * warps_per_block, W = worker_warps(p.n_queries, total, p.stack_cap),
                   workers = total / W;
    p.donate_min *= W;
    // all roots start at once where they fit a step of the workers
    p.root_batch = p.stack_cap < kPoolStack
                       ? 1u
                       : std::min(std::max((p.n_queries + workers - 1u) / workers, 1u), 32u * W);
    const size_t smem = size_t(traverse_smem_words(p.stack_cap, W)) * sizeof(uint32_t);
    traverse_kernel<<<workers, 32 * W, smem, s>>>(p);
    return cudaGetLastError();
}

cudaError_t launch_narrow(const NarrowParams& p, uint32_t blocks, uint32_t warps_per_block, cudaStream_t s) {
    if (p.flags & CG_ROBUST)
        narrow_kernel<2><<<blocks, 32 * warps_per_block, 0, s>>>(p);
    else if (p.flags & CG_RECHECK)
        narrow_kernel<1><<<blocks, 32 * warps_per_block, 0, s>>>(p);
    else
        narrow_kernel<0><<<blocks, 32 * warps_per_block, 0, s>>>(p);
    return cudaGetLastError();
}

}  // namespace cg
