// G^2 in 64-bit fixed point, for tests whose decision is all that is asked (a skeleton's).
//
// With F(n) = n ln n, a test's statistic is twice
//     sum F(N_xyz) - sum F(N_xz) - sum F(N_yz) + sum F(N_z)
// (IndependenceTest.cpp:94-138 with ln(O N_z / (N_x N_y)) split into its logarithms).  F is a
// table of integers round(n ln n 2^k), so the sums are exact whatever their order and a test
// needs no logarithm, no division and no FP64 accumulation (an FP64 instruction holds a GB300
// scheduler for about 64 cycles).  Error: half a unit per count and FP64's in the table, below
// 1e-6 for tables in shared memory.  The decision compares the statistic with the quantiles at
// alpha +- kTight; what falls between is decided by the FP64 terms and their p-value.
#pragma once
#include "ci_device.cuh"

namespace fpgm {

constexpr int64_t kFixedMaxSamples = (int64_t)1 << 20;  // F's table stays in L2 and k above 34
constexpr double kTight = 1e-6;

struct Fixed {
    const long long *f;  // F(0 .. samples); null: not in use
    double unit;         // 2^-k
    const double *lo;    // G^2 below lo[df] => p > alpha + kTight
    const double *hi;    // G^2 above hi[df] => p < alpha - kTight
    int dfmax;
};

// 1 independent, 0 dependent, -1 undecided.  counts: table entries whose F was summed.
__device__ inline int fixed_decide(const Fixed &x, long long df, long long sum, int64_t counts, int64_t S, double *g2) {
    *g2 = 2.0 * x.unit * (double)sum;
    if (df == 0) return 1;
    if (df > x.dfmax) return -1;
    const double err = x.unit * (double)counts + 2e-14 * (double)S;
    if (*g2 + err < x.lo[df]) return 1;
    if (*g2 - err > x.hi[df]) return 0;
    return -1;
}

__device__ inline long long warp_sum_ll(long long v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ inline void group_sum_ll(const WarpGroup &, long long &a, long long &b, long long *) {
    a = warp_sum_ll(a);
    b = warp_sum_ll(b);
}
__device__ inline void group_sum_ll(const CtaGroup &, long long &a, long long &b, long long *scratch) {
    a = warp_sum_ll(a);
    b = warp_sum_ll(b);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) {
        scratch[2 * warp] = a;
        scratch[2 * warp + 1] = b;
    }
    __syncthreads();
    a = b = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
        a += scratch[2 * w];
        b += scratch[2 * w + 1];
    }
}

// A count table held by group g: cell (stratum k, x value i, y value j) at
// t[zoff[k] + i * sx + j * sy] (zoff null: k * dx * dy).  ni / nj / nk: dz*dx, dz*dy and dz ints
// of scratch.  hv: the sum of F over the cells, or null to have it summed here.  Every thread of
// g calls it; the verdict is valid in the group's first warp.  (p is that of a recheck only.)
template <class G>
__device__ inline Verdict score_fixed(const G &g, const int *t, const int *zoff, int sx, int sy, int dx, int dy, int dz,
                                      int *ni, int *nj, int *nk, const long long *hv, const Fixed &x, double alpha,
                                      int64_t S, Partial *scratch) {
    const int dxy = dx * dy;
    long long sum = 0, df = 0;
    for (int idx = g.t; idx < dz * dx; idx += g.n()) {
        const int k = idx / dx, i = idx - k * dx;
        const int *row = t + (zoff ? zoff[k] : k * dxy) + i * sx;
        int s = 0;
        for (int j = 0; j < dy; ++j) s += row[j * sy];
        ni[idx] = s;
        sum -= __ldg(&x.f[s]);
    }
    for (int idx = g.t; idx < dz * dy; idx += g.n()) {
        const int k = idx / dy, j = idx - k * dy;
        const int *base = t + (zoff ? zoff[k] : k * dxy) + j * sy;
        int s = 0;
        for (int i = 0; i < dx; ++i) s += base[i * sx];
        nj[idx] = s;
        sum -= __ldg(&x.f[s]);
    }
    if (hv) {
        if (g.t == 0) sum += *hv;
    } else {
        for (int c = g.t; c < dz * dxy; c += g.n()) sum += __ldg(&x.f[t[c]]);
    }
    g.sync();
    for (int k = g.t; k < dz; k += g.n()) {
        int alx = 0, aly = 0, tot = 0;
        for (int i = 0; i < dx; ++i) {
            const int v = ni[k * dx + i];
            alx += v > 0;
            tot += v;
        }
        for (int j = 0; j < dy; ++j) aly += nj[k * dy + j] > 0;
        nk[k] = tot;
        df += (long long)(max(alx, 1) - 1) * (max(aly, 1) - 1);
        sum += __ldg(&x.f[tot]);
    }
    g.sync();
    group_sum_ll(g, sum, df, reinterpret_cast<long long *>(scratch));
    Verdict v{df, 0.0, 1.0, 1, 0, 0.0, 0ull};
    const int dec = fixed_decide(x, df, sum, (int64_t)dz * (dxy + dx + dy + 1), S, &v.g2);
    v.indep = dec;
    if (dec >= 0) return v;
    // FP64 terms in the reference's formula, and their p-value
    Partial q{0, 0.0, 0.0, 0.0, 0ull};
    for (int c = g.t; c < dz * dxy; c += g.n()) {
        const int k = c / dxy, rem = c - k * dxy, i = rem / dy, j = rem - i * dy;
        const int o = t[(zoff ? zoff[k] : k * dxy) + i * sx + j * sy];
        if (o == 0) continue;
        const double expected = (double)nj[k * dy + j] * (double)ni[k * dx + i] / (double)nk[k];
        q.g2 += 2.0 * o * log(o / expected);
    }
    g.sync();  // scratch is free again
    const Partial r = group_sum(g, q, scratch);
    v.dp = fabs(v.g2 - r.g2);
    v.g2 = r.g2;
    v.rechecked = 1;
    if (g.t < 32) {
        v.p = chisq_pvalue(r.g2, df);
        v.indep = v.p > alpha;
        v.dp = df > 1 ? 0.5 * v.dp : v.dp;  // the density is at most 1/2 there
    }
    return v;
}

// F(n) = n ln n in units of 2^-k
__global__ void fixed_table_kernel(long long *f, int64_t n_max, double scale) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i <= n_max) f[i] = i < 2 ? 0 : __double2ll_rn((double)i * log((double)i) * scale);
}

}  // namespace fpgm
