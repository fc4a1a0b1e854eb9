// The eig3 eigensystem of a symmetric 3x3 (eig3/eig3.cpp:21-265), for any
// floating type: Householder reduction to tridiagonal form, implicit-shift QL,
// then the ascending selection sort of the eigenvalues with their eigenvector
// columns. Every operation is the published procedure's, in its order, so
// that in double without contraction the results are the CPU's bits (the
// tree build), and in float the refit's axes.
#pragma once

#include <cuda_runtime.h>

namespace cg {

template <typename R>
__device__ __forceinline__ R hyp(R x, R y) {
    return sqrt(x * x + y * y);
}

// Every loop below has its bounds at compile time and is unrolled, so that v, d
// and e stay in registers. With the published loops' bounds (and so the indexes)
// at run time they lay in local memory: the refit's axes of 64 trees of 12,000
// triangles took 50 us instead of 25, the eigensystems of all levels of a
// 5,003-triangle mesh's build 724 us instead of 644 (there FP64 instructions,
// about 64 cycles each, are the rest).

// How a matrix is worked on: by one thread (Alone), or by a group of lanes that
// all hold it (Group: 4 to 32 lanes of a warp, of which mask are this group's
// and base the first), where two quotients of one divisor take the time of one
// division, a lane each. kRows rows of v to a thread: a Group's lane turns one
// row in the QL sweeps.
struct Alone {
    static constexpr int kRows = 3;
    template <typename R>
    __device__ __forceinline__ void divide(R a, R b, R by, R& qa, R& qb) const {
        qa = a / by;
        qb = b / by;
    }
};
struct Group {
    static constexpr int kRows = 1;
    unsigned mask;
    uint32_t base;
    bool odd;  // this lane's is the second quotient
    template <typename R>
    __device__ __forceinline__ void divide(R a, R b, R by, R& qa, R& qb) const {
        const R q = (odd ? b : a) / by;
        qa = __shfl_sync(mask, q, base);
        qb = __shfl_sync(mask, q, base + 1u);
    }
};

// Householder reduction of the symmetric 3x3 in v to tridiagonal form
// (eig3.cpp:21-134): v becomes the accumulated transform, d the diagonal,
// e[1..2] the sub-diagonal.
template <class By, typename R>
__device__ __forceinline__ void tridiagonalize(const By& by, R v[3][3], R d[3], R e[3]) {
#pragma unroll
    for (int c = 0; c < 3; ++c) d[c] = v[2][c];
#pragma unroll
    for (int i = 2; i >= 1; --i) {
        R scale = R(0), h = R(0);
#pragma unroll
        for (int k = 0; k < i; ++k) scale = scale + fabs(d[k]);
        if (scale == R(0)) {
            e[i] = d[i - 1];
#pragma unroll
            for (int c = 0; c < i; ++c) {
                d[c] = v[i - 1][c];
                v[i][c] = R(0);
                v[c][i] = R(0);
            }
        } else {
            if (i == 2)
                by.divide(d[0], d[1], scale, d[0], d[1]);
            else
                d[0] = d[0] / scale;
#pragma unroll
            for (int k = 0; k < i; ++k) h = h + d[k] * d[k];
            R f = d[i - 1];
            R g = sqrt(h);
            if (f > 0) g = -g;
            e[i] = scale * g;
            h = h - f * g;
            d[i - 1] = f - g;
#pragma unroll
            for (int c = 0; c < i; ++c) e[c] = R(0);
#pragma unroll
            for (int c = 0; c < i; ++c) {
                f = d[c];
                v[c][i] = f;
                g = e[c] + v[c][c] * f;
#pragma unroll
                for (int k = c + 1; k <= i - 1; ++k) {
                    g = g + v[k][c] * d[k];
                    e[k] = e[k] + v[k][c] * f;
                }
                e[c] = g;
            }
            f = R(0);
            if (i == 2)
                by.divide(e[0], e[1], h, e[0], e[1]);
            else
                e[0] = e[0] / h;
#pragma unroll
            for (int c = 0; c < i; ++c) f = f + e[c] * d[c];
            const R hh = f / (h + h);
#pragma unroll
            for (int c = 0; c < i; ++c) e[c] = e[c] - hh * d[c];
#pragma unroll
            for (int c = 0; c < i; ++c) {
                f = d[c];
                g = e[c];
#pragma unroll
                for (int k = c; k <= i - 1; ++k) v[k][c] = v[k][c] - (f * e[k] + g * d[k]);
                d[c] = v[i - 1][c];
                v[i][c] = R(0);
            }
        }
        d[i] = h;
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        v[2][i] = v[i][i];
        v[i][i] = R(1);
        const R h = d[i + 1];
        if (h != R(0)) {
            if (i == 1)
                by.divide(v[0][2], v[1][2], h, d[0], d[1]);
            else
                d[0] = v[0][1] / h;
#pragma unroll
            for (int c = 0; c <= i; ++c) {
                R g = R(0);
#pragma unroll
                for (int k = 0; k <= i; ++k) g = g + v[k][i + 1] * v[k][c];
#pragma unroll
                for (int k = 0; k <= i; ++k) v[k][c] = v[k][c] - g * d[k];
            }
        }
#pragma unroll
        for (int k = 0; k <= i; ++k) v[k][i + 1] = R(0);
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        d[c] = v[2][c];
        v[2][c] = R(0);
    }
    v[2][2] = R(1);
    e[0] = R(0);
}

// Sweeps of the implicit-shift QL over rows L..M (eig3.cpp:160-227) until
// e[L] is negligible. A sweep count limit stops what only a non-finite input
// could run forever.
template <int L, int M, class By, typename R>
__device__ __forceinline__ void ql_sweeps(const By& by, R v[By::kRows][3], R d[3], R e[3], R& f, R small) {
    int sweeps = 0;
    do {
        ++sweeps;
        R g = d[L];
        R p = (d[L + 1] - g) / (R(2) * e[L]);
        R r = hyp(p, R(1));
        if (p < 0) r = -r;
        d[L] = e[L] / (p + r);
        d[L + 1] = e[L] * (p + r);
        const R dl1 = d[L + 1];
        R h = g - d[L];
#pragma unroll
        for (int i = L + 2; i < 3; ++i) d[i] = d[i] - h;
        f = f + h;
        p = d[M];
        R c = R(1), c2 = c, c3 = c;
        const R el1 = e[L + 1];
        R s = R(0), s2 = R(0);
#pragma unroll
        for (int i = M - 1; i >= L; --i) {
            c3 = c2;
            c2 = c;
            s2 = s;
            g = c * e[i];
            h = c * p;
            r = hyp(p, e[i]);
            e[i + 1] = s * r;
            by.divide(e[i], p, r, s, c);
            p = c * d[i] - s * g;
            d[i + 1] = h + s * (c * g + s * d[i]);
#pragma unroll
            for (int k = 0; k < By::kRows; ++k) {
                h = v[k][i + 1];
                v[k][i + 1] = s * v[k][i] + c * h;
                v[k][i] = c * v[k][i] - s * h;
            }
        }
        p = -s * s2 * c3 * el1 * e[L] / dl1;
        e[L] = s * p;
        d[L] = c * p;
    } while (fabs(e[L]) > small && sweeps < 10000);
}

// Implicit-shift QL on the tridiagonal form, then the ascending sort of the
// eigenvalues with their eigenvector columns (eig3.cpp:138-254), for the rows of
// v that the thread has. The last row
// with a negligible sub-diagonal is at most 2 (its e is 0).
template <class By, typename R>
__device__ __forceinline__ void ql_sort(const By& by, R v[By::kRows][3], R d[3], R e[3], R eps) {
    e[0] = e[1], e[1] = e[2];
    e[2] = R(0);
    R f = 0, tst1 = 0;
    auto top = [&](int l) {
        const R t = fabs(d[l]) + fabs(e[l]);
        tst1 = (tst1 > t) ? tst1 : t;
    };
    top(0);
    if (!(fabs(e[0]) <= eps * tst1)) {
        if (fabs(e[1]) <= eps * tst1)
            ql_sweeps<0, 1>(by, v, d, e, f, eps * tst1);
        else
            ql_sweeps<0, 2>(by, v, d, e, f, eps * tst1);
    }
    d[0] = d[0] + f;
    e[0] = R(0);
    top(1);
    if (!(fabs(e[1]) <= eps * tst1)) ql_sweeps<1, 2>(by, v, d, e, f, eps * tst1);
    d[1] = d[1] + f;
    e[1] = R(0);
    d[2] = d[2] + f;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        int k = i;
        R p = d[i];
#pragma unroll
        for (int j = i + 1; j < 3; ++j)
            if (d[j] < p) {
                k = j;
                p = d[j];
            }
#pragma unroll
        for (int j = i + 1; j < 3; ++j)
            if (k == j) {
                d[j] = d[i];
                d[i] = p;
#pragma unroll
                for (int r = 0; r < By::kRows; ++r) {
                    const R tmp = v[r][i];
                    v[r][i] = v[r][j];
                    v[r][j] = tmp;
                }
            }
    }
}

}  // namespace cg
