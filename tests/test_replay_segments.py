"""The rule by which the tree build adds up a sequential FP64 sum in parallel
segments (csrc/cg_replay.cuh), compiled for the host: whatever the predicted
starts, the linked sum must have the sequential sum's bits.
Terms: covariance-like products, oscillating sums, ties, cancellation, signed
zeros, tiny and huge scales, non-finite terms; predictions off by 0 to 2^24
last places, or wrong altogether."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "inmyroom_vulkan_gb300", "csrc")

SOURCE = r"""
#include <algorithm>
#include <vector>
#define __device__
#define __forceinline__ inline
#include "cg_replay.cuh"
using namespace cg;
// segments of `len` terms; off[k] last places are added to the k-th segment's true start as its prediction.
// Returns the number of linked segments, or -1 when the sum is not the chain's.
extern "C" long replay(const double* t, long n, long len, const long long* off, long* segments) {
    std::vector<double> pred;
    double chain = 0.0;
    for (long b = 0; b < n; b += len) {
        pred.push_back(b ? bits_double(dbits(chain) + (unsigned long long)off[pred.size()]) : chain);
        for (long j = b; j < std::min(n, b + len); ++j) chain = chain + t[j];
    }
    const long k = long(pred.size());
    pred.push_back(bits_double(dbits(chain) + (unsigned long long)off[0]));
    std::vector<ReplayLink> end(4 * k);
    for (long g = 0; g < k; ++g)
        for (unsigned r = 0; r < 4; ++r) {
            const double first = replay_candidate(pred[g], r);
            double v = first;
            ReplayChain seen;
            for (long j = g * len; j < std::min(n, (g + 1) * len); ++j) {
                replay_see(seen, v);
                v = v + t[j];
            }
            replay_see(seen, v);
            end[4 * g + r] = replay_end(first, seen, v, pred[g + 1]);
        }
    long added = 0;
    const double got = replay_chain(0.0, pred.data(), end.data(), uint32_t(k), [&](uint32_t g, double s) {
        ++added;
        for (long j = g * len; j < std::min(n, (long(g) + 1) * len); ++j) s = s + t[j];
        return s;
    });
    *segments = k;
    return dbits(got) == dbits(chain) || (got != got && chain != chain) ? k - added : -1;
}
"""


@pytest.fixture(scope="module")
def replay(tmp_path_factory):
    d = tmp_path_factory.mktemp("replay")
    src, so = d / "replay.cpp", d / "replay.so"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-I", CSRC, str(src), "-o", str(so)],
                   check=True)
    lib = C.CDLL(str(so))
    lib.replay.restype = C.c_long

    def run(t, length, off):
        t, off = np.ascontiguousarray(t, np.float64), np.ascontiguousarray(off, np.int64)
        seg = C.c_long()
        got = lib.replay(C.c_void_p(t.ctypes.data), C.c_long(len(t)), C.c_long(length), C.c_void_p(off.ctypes.data),
                         C.byref(seg))
        return got, seg.value

    return run


def terms(kind, rng, n=6000):
    x, y = rng.normal(size=(2, n)).astype(np.float32).astype(np.float64) - rng.normal(size=2)[:, None]
    if kind == "squares":
        return x * x
    if kind == "products":
        return x * y
    if kind == "rings":  # sums that swing through zero
        return np.cos(np.arange(n) * 0.05) * (1 + 0.01 * x)
    if kind == "ties":  # few mantissa bits: ties at every binade
        return rng.integers(-3, 9, n) * 2.0 ** rng.integers(-54, -50, n) + (rng.random(n) < 0.01)
    if kind == "cancel":
        z = x * 10.0 ** rng.integers(-12, 6, n)
        z[1::2] = -z[::2] * (1 + 2.0 ** -50 * rng.integers(0, 2, n // 2))
        return z
    if kind == "zeros":
        return np.where(rng.random(n) < 0.9, np.where(rng.random(n) < 0.5, 0.0, -0.0), x)
    if kind == "tiny":
        return x * 10.0 ** rng.uniform(-320, -300, n)
    if kind == "huge":
        return x * 1e300
    z = x.copy()
    z[rng.integers(0, n, 5)] = rng.choice([np.nan, np.inf, -np.inf], 5)
    return z


@pytest.mark.parametrize("kind", ["squares", "products", "rings", "ties", "cancel", "zeros", "tiny", "huge", "nonfinite"])
def test_linked_segments_are_the_sequential_sum(replay, kind):
    rng = np.random.Generator(np.random.PCG64(23))
    good = total = 0
    for length in (1, 7, 64, 128, 500):
        n_seg = 6000 // length + 1
        for bits in (0, 2, 7, 12, 24, 60):
            off = rng.integers(-(2 ** bits), 2 ** bits + 1, n_seg) if bits else np.zeros(n_seg, np.int64)
            got, seg = replay(terms(kind, rng), length, off)
            assert got >= 0, (length, bits)
            if length == 128 and bits in (2, 7):
                good, total = good + got, total + seg
            if bits == 0 and np.isfinite(terms(kind, np.random.Generator(np.random.PCG64(1)))).all():
                assert got == seg
    if kind == "squares":  # and predictions a few places off are linked
        assert good > 0.8 * total
