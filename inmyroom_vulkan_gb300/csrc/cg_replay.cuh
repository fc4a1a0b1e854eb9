// A sequential FP64 sum (s = s + t[0], s + t[1], ..., each add rounded to
// nearest even) computed in parallel segments with the same bits.
//
// A dependent FP64 add takes 63 cycles on this part and a warp's FP64
// instruction holds the pipe that long whether one or 32 lanes are active, so
// a long chain of adds runs at one term per 64 cycles. Here the terms are cut
// into segments that start from predicted sums (an FP64 prefix sum in another
// order, off by a few last places), all at once, 4 candidates per segment:
// the prediction with its last two mantissa bits set to 0, 1, 2 and 3. When
// the true sum s at the segment's start is known, the candidate with s's last
// two bits differs from it by d, a multiple of 4 ulps of s. If every state of
// the candidate's chain lies at most one binade above s (its rounding
// granularity g is at most 2 ulps, so d is a multiple of 2 g) and farther
// than |d| from the ends of its binade, the chain from s visits the same
// binades, each add rounds the same way (ties to even included: d / g is
// even), and the end is the candidate's end plus d, exactly. Else the
// segment is added term by term.
//
// The functions here are the rule; the kernels of cg_build.cu arrange the
// segments.
#pragma once

#include <cstdint>

namespace cg {

__device__ __forceinline__ unsigned long long dbits(double x) {
#ifdef __CUDA_ARCH__
    return (unsigned long long)__double_as_longlong(x);
#else
    unsigned long long b;
    __builtin_memcpy(&b, &x, 8);
    return b;
#endif
}
__device__ __forceinline__ double bits_double(unsigned long long b) {
#ifdef __CUDA_ARCH__
    return __longlong_as_double((long long)b);
#else
    double x;
    __builtin_memcpy(&x, &b, 8);
    return x;
#endif
}
__device__ __forceinline__ int clz32(uint32_t x) {  // x > 0
#ifdef __CUDA_ARCH__
    return __clz(int(x));
#else
    return __builtin_clz(x);
#endif
}

// Candidate r (0..3) of a segment predicted to start at p.
__device__ __forceinline__ double replay_candidate(double p, unsigned r) { return bits_double((dbits(p) & ~3ull) | r); }

// What a candidate's chain has visited: the smallest distance of its states
// from the ends of their binades (2^(margin - 1043) or more; 0: no distance)
// and the largest exponent field of its states. Every state is seen, the
// start among them.
struct ReplayChain {
    int margin = 0x7fffffff, top = 0;
};
__device__ __forceinline__ void replay_see(ReplayChain& c, double v) {
    const uint32_t hi = uint32_t(dbits(v) >> 32);
    const int e = int(hi >> 20) & 0x7ff;
    const uint32_t m = hi & 0xfffffu, far = 0xfffffu - m, d = m < far ? m : far;
    const int k = d ? e + 31 - clz32(d) : 0;
    c.margin = k < c.margin ? k : c.margin;
    c.top = e > c.top ? e : c.top;
}

// A candidate's end, moved by d ulps of its start where |d| <= limit: as an
// offset from the following segment's base (that prediction with its last two
// bits cleared), next + (d / 2) mul, mul being plus or minus 2^(1 + es - ee)
// (the exponents of start and end; minus when the signs differ). `limit` is
// -1 where such an offset does not stay within 32 bits.
struct alignas(16) ReplayLink {
    int next, limit, mul, pad;
};
constexpr long long kReplayNear = 1ll << 29;
__device__ __forceinline__ unsigned long long replay_base(double pred) { return dbits(pred) & ~3ull; }
__device__ __forceinline__ ReplayLink replay_end(double start, const ReplayChain& c, double v, double next_pred) {
    const unsigned long long sb = dbits(start), ev = dbits(v);
    const int es = int(sb >> 52) & 0x7ff, ee = int(ev >> 52) & 0x7ff, sh = es - ee;
    const long long next = (long long)(ev - replay_base(next_pred));
    // (|d| + 4) 2^(es - 1075) < 2^(margin - 1043)
    const int x = c.margin - es + 32;
    const bool moves = es > 0 && ee > 0 && c.top <= es + 1 && c.top < 0x7ff && x > 2 && sh < 4;
    ReplayLink r;
    r.next = int(next);
    r.limit = moves ? (1 << (x < 25 ? x : 25)) - 5 : 0;
    r.mul = moves ? ((ev ^ sb) >> 63 ? -1 : 1) * (1 << (sh + 1)) : 0;
    if (next < -kReplayNear || next > kReplayNear) r.limit = -1;
    r.pad = 0;
    return r;
}

// The sum that starts at s (pred[0] exactly): segment g predicted to start at
// pred[g] (pred[n]: the whole sum) and ended by its four candidates as
// end[4 g + r]; add(g, s) adds segment g's terms to s one by one. The running
// sum is kept as its offset o from the segment's base (a dozen dependent
// operations a segment); where a segment cannot be linked or the offset is
// out of range, as the double itself.
template <class Add>
__device__ __forceinline__ double replay_chain(double s, const double* pred, const ReplayLink* end, uint32_t n, Add add) {
    int o = int(dbits(s) & 3ull);
    uint32_t g = 0;
    for (;;) {
        for (; g < n; ++g) {
            const ReplayLink e = end[4u * g + (unsigned(o) & 3u)];
            const int d = o & ~3;
            if ((d < 0 ? -d : d) > e.limit) break;
            o = e.next + (d >> 1) * e.mul;
        }
        s = bits_double(replay_base(pred[g]) + (unsigned long long)(long long)o);
        for (;;) {
            if (g == n) return s;
            s = add(g, s);
            ++g;
            const long long off = (long long)(dbits(s) - replay_base(pred[g]));
            if (g < n && off >= -kReplayNear && off <= kReplayNear) {
                o = int(off);
                break;
            }
        }
    }
}

}  // namespace cg
