// Tests whose joint tables fit shared memory, counted once per variable set.
//
// A test (x, y | Z) needs the joint table of the set {x, y} + Z whichever of its variables are
// x and y: the same set comes back under its other pairs, and under the same pair from the other
// side (CheckEdge tests Z from x's neighbours, then from y's, PCStable.cpp:399-494).  So a
// level keeps the tables it has counted, over the set's variables in ascending order, and a test
// is scored from its set's table with the strides of its own x, y and Z.
//   classify        enters the test's set (set_enter); a set met for the first time gets room
//                   for its table and goes to the list of sets to count
//   set_count_*     one to eight warps per new set
//   set_score_*     one warp or one CTA per test
// Tests per distinct set, duplicates of a pair included: 1.2 (1,041 variables, level 1), 1.6 to
// 2.0 (100 to 223 variables, level 1), 2 to 2.3 at level 2, 3.3 to 3.8 at level 3, 4.8 at level 4.
#pragma once
#include "ci_kernels.cuh"

namespace fpgm {

// Warp or CTA: the variables of an item in ascending order (rank of each of z.., x, y among
// them), their columns and state counts, and the stride of each in the set's table.
struct SetShape {
    const uint8_t *col[kMaxCols];
    uint32_t dim[kMaxCols];
    int32_t stride[kMaxCols];
    int32_t rank[kMaxCols];  // of the item's variable j (z1 .. zd, x, y)
};
__device__ inline void set_shape(const WaveArgs &a, int item, int lane, SetShape &s) {
    const int ncols = a.d + 2;
    const uint16_t *iv = a.item_vars + (int64_t)item * ncols;
    const int var = lane < ncols ? iv[lane] : 0x10000;
    int rank = 0;
    for (int j = 0; j < ncols; ++j) rank += __shfl_sync(0xffffffffu, var, j) < var;
    if (lane < ncols) {
        s.rank[lane] = rank;
        s.col[rank] = a.cols + a.var_off[var];
        s.dim[rank] = a.card[var];
    }
    __syncwarp();
    if (lane < ncols) {
        int st = 1;
        for (int j = lane + 1; j < ncols; ++j) st *= (int)s.dim[j];
        s.stride[lane] = st;
    }
    __syncwarp();
}

template <int kWarpsPer>
__device__ __forceinline__ void warps_sync(int group) {
    if (kWarpsPer == 1) __syncwarp();
    else if (kWarpsPer == kWarps) __syncthreads();
    else asm volatile("bar.sync %0, %1;" ::"r"((kWarpsPer == 4 ? 1 : 3) + group), "n"(32 * kWarpsPer) : "memory");
}

// Counts the set of entry e.x (shape of item e.y in sh) with n threads, and writes its table in
// the order of its ascending variables; returns the thread's share of the sum of F.
template <class Sync>
__device__ __forceinline__ long long count_set(const WaveArgs &a, const int2 e, const SetShape &sh, int64_t S, int *rep,
                                               int ints, int t, int n, const Sync &sync) {
    const int cells = sh.stride[0] * (int)sh.dim[0], lane = threadIdx.x & 31;
    const int lgR = set_replicas(cells, S, ints), R = 1 << lgR;
    for (int i = t; i < (cells << lgR); i += n) rep[i] = 0;
    sync();
    count_columns(rep, lgR, lane, sh.col, sh.dim, a.d + 2, S, t, n);
    sync();
    int *out = a.sets.pool + a.sets.off[e.x];
    long long h = 0;
    for (int c = t; c < cells; c += n) {
        int m = 0;
        for (int r = 0; r < R; ++r) m += rep[(c << lgR) + ((r + lane) & (R - 1))];
        out[c] = m;
        h += __ldg(&a.fx.f[m]);
    }
    return h;
}

// The sets of one class, kWarpsPer warps each.
template <int kWarpsPer>
__device__ inline void count_sets(const WaveArgs &a, int *smem, SetShape *s_shape, int2 *s_e, long long *s_h, int k) {
    const int group = (threadIdx.x >> 5) / kWarpsPer, t = threadIdx.x % (32 * kWarpsPer), lane = threadIdx.x & 31;
    const int first = group * kWarpsPer;  // the group's first warp: its shared memory is theirs
    int *rep = smem + first * kSetWarpInts;
    SetShape &sh = s_shape[first];
    const int n = a.counters[C_SET + k];
    auto sync = [&]() { warps_sync<kWarpsPer>(group); };
    for (;;) {
        if (t < 32) {
            int idx = 0;
            if (lane == 0) idx = atomicAdd(&a.counters[C_WSET + k], 1);
            idx = __shfl_sync(0xffffffffu, idx, 0);
            const int2 e = idx < n ? a.sets.fresh[k * a.list_cap + idx] : make_int2(-1, 0);
            if (e.x >= 0) set_shape(a, e.y, lane, sh);
            if (lane == 0) {
                s_e[first] = e;
                s_h[first] = 0;
            }
        }
        sync();
        const int2 e = s_e[first];
        if (e.x < 0) break;
        const int64_t S = a.var_S[a.item_vars[(int64_t)e.y * (a.d + 2)]];
        const long long h = warp_sum_ll(count_set(a, e, sh, S, rep, kSetWarpInts * kWarpsPer, t, 32 * kWarpsPer, sync));
        if (kWarpsPer == 1) {
            if (lane == 0) a.sets.h[e.x] = h;
        } else if (lane == 0) {
            atomicAdd(reinterpret_cast<unsigned long long *>(&s_h[first]), (unsigned long long)h);
        }
        sync();
        if (kWarpsPer > 1) {
            if (t == 0) a.sets.h[e.x] = s_h[first];
        }
    }
    sync();  // s_e and the group's shared memory are free
}

// New sets of tables of up to 8 * kSetWarpInts cells, 8, 4, 2 or 1 warps each (set_class); in a
// wave of few sets the whole CTA counts each, so that no warp is left alone with all samples of
// one.  Bound by the shared-memory atomics and instruction issue together; the samples come
// from L2.
__global__ void __launch_bounds__(kThreads, 3) set_count_kernel(WaveArgs a) {
    extern __shared__ int smem[];
    __shared__ SetShape s_shape[kWarps];
    __shared__ int2 s_e[kWarps];
    __shared__ long long s_h[kWarps];
    const int small = a.counters[C_SET] + a.counters[C_SET + 1] + a.counters[C_SET + 2];
    count_sets<8>(a, smem, s_shape, s_e, s_h, 3);
    if (small <= a.sets.few) {
        for (int k = 2; k >= 0; --k) count_sets<8>(a, smem, s_shape, s_e, s_h, k);
        return;
    }
    count_sets<4>(a, smem, s_shape, s_e, s_h, 2);
    count_sets<2>(a, smem, s_shape, s_e, s_h, 1);
    count_sets<1>(a, smem, s_shape, s_e, s_h, 0);
}

// One CTA per new set of a larger table.
__global__ void __launch_bounds__(kThreads, 2) set_count_big_kernel(WaveArgs a) {
    extern __shared__ int smem[];
    __shared__ SetShape sh;
    __shared__ int s_idx;
    __shared__ unsigned long long s_h;
    const int tid = threadIdx.x, lane = tid & 31;
    const int n = a.counters[C_SET + 4];
    for (;;) {
        if (tid == 0) {
            s_idx = atomicAdd(&a.counters[C_WSET + 4], 1);
            s_h = 0;
        }
        __syncthreads();
        const int idx = s_idx;
        if (idx >= n) break;
        const int2 e = a.sets.fresh[4 * a.list_cap + idx];
        const int64_t S = a.var_S[a.item_vars[(int64_t)e.y * (a.d + 2)]];
        if (tid < 32) set_shape(a, e.y, lane, sh);
        __syncthreads();
        const long long h =
            warp_sum_ll(count_set(a, e, sh, S, smem, kCtaInts, tid, kThreads, []() { __syncthreads(); }));
        if (lane == 0) atomicAdd(&s_h, (unsigned long long)h);
        __syncthreads();
        if (tid == 0) a.sets.h[e.x] = (long long)s_h;
        __syncthreads();
    }
}

// zoff[k]: offset of stratum k in the set's table, Z's digits taken from the last variable on
template <class G>
__device__ inline void stratum_offsets(const G &g, const SetShape &sh, int d, int dz, int *zoff) {
    for (int k = g.t; k < dz; k += g.n()) {
        int q = k, o = 0;
        for (int j = d - 1; j >= 0; --j) {
            const int r = sh.rank[j], m = (int)sh.dim[r], w = q / m;
            o += (q - w * m) * sh.stride[r];
            q = w;
        }
        zoff[k] = o;
    }
}

__device__ inline void set_missed(const WaveArgs &a, int item) {
    const int d = a.d;
    const uint16_t *iv = a.item_vars + (int64_t)item * (d + 2);
    int dz = 1;
    for (int k = 0; k < d; ++k) dz *= a.card[iv[k]];
    const int dx = a.card[iv[d]], dy = a.card[iv[d + 1]];
    const int tier = dz * dx * dy + dz * (dx + dy + 1) <= a.warp_ints - 32 ? 0 : 1;
    a.lists[tier * a.list_cap + atomicAdd(&a.counters[C_TIER0 + tier], 1)] = item;
    atomicAdd(&a.stats[ST_BYTES_SHARED], (unsigned long long)(d + 2) * (unsigned long long)a.var_S[iv[d]]);
}

// One warp per test, from its set's table.
template <int kSlice, int kMinBlocks>
__global__ void __launch_bounds__(kThreads, kMinBlocks) set_score_warp_kernel(WaveArgs a) {
    extern __shared__ int smem[];
    __shared__ SetShape s_shape[kWarps];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int *tab = smem + warp * kSlice;
    SetShape &sh = s_shape[warp];
    const int n0 = a.counters[C_SCOREW], d = a.d, ncols = d + 2;
    const WarpGroup g{lane};
    for (;;) {
        int idx = 0;
        if (lane == 0) idx = atomicAdd(&a.counters[C_WSCOREW], 1);
        idx = __shfl_sync(0xffffffffu, idx, 0);
        if (idx >= n0) break;
        const int2 e = a.sets.items[idx];  // set, item
        if (a.sets.off[e.x] < 0) {         // no room for the set's table: the test counts its own
            if (lane == 0) set_missed(a, e.y);
            continue;
        }
        const int64_t S = a.var_S[a.item_vars[(int64_t)e.y * ncols]];
        set_shape(a, e.y, lane, sh);
        const int rx = sh.rank[d], ry = sh.rank[d + 1];
        const int dx = sh.dim[rx], dy = sh.dim[ry], cells = sh.stride[0] * (int)sh.dim[0], dz = cells / (dx * dy);
        int *zoff = tab + cells, *ni = zoff + dz, *nj = ni + dz * dx, *nk = nj + dz * dy;
        const int *src = a.sets.pool + a.sets.off[e.x];
        for (int c = lane; c < cells; c += 32) tab[c] = __ldcg(src + c);
        stratum_offsets(g, sh, d, dz, zoff);
        __syncwarp();
        const Verdict v = score_fixed(g, tab, zoff, sh.stride[rx], sh.stride[ry], dx, dy, dz, ni, nj, nk,
                                      a.sets.h + e.x, a.fx, a.alpha, S, nullptr);
        if (lane == 0) {
            record(a, e.y, v, cells, 0, 0);
            if (d == 0 && a.pair_g2) keep_pair(a, a.item_vars[(int64_t)e.y * 2], a.item_vars[(int64_t)e.y * 2 + 1], v.g2);
        }
        __syncwarp();
    }
}

__global__ void __launch_bounds__(kThreads, 2) set_score_cta_kernel(WaveArgs a) {
    extern __shared__ int smem[];
    __shared__ SetShape sh;
    __shared__ int s_idx;
    __shared__ Partial scratch[kWarps];
    const int tid = threadIdx.x;
    const int n1 = a.counters[C_SCOREC], d = a.d, ncols = d + 2;
    const CtaGroup g{tid};
    for (;;) {
        if (tid == 0) s_idx = atomicAdd(&a.counters[C_WSCOREC], 1);
        __syncthreads();
        const int idx = s_idx;
        if (idx >= n1) break;
        const int2 e = a.sets.items[a.list_cap - 1 - idx];
        if (a.sets.off[e.x] < 0) {
            if (tid == 0) set_missed(a, e.y);
            __syncthreads();
            continue;
        }
        const int64_t S = a.var_S[a.item_vars[(int64_t)e.y * ncols]];
        if (tid < 32) set_shape(a, e.y, tid, sh);
        __syncthreads();
        const int rx = sh.rank[d], ry = sh.rank[d + 1];
        const int dx = sh.dim[rx], dy = sh.dim[ry], cells = sh.stride[0] * (int)sh.dim[0], dz = cells / (dx * dy);
        int *zoff = smem + cells, *ni = zoff + dz, *nj = ni + dz * dx, *nk = nj + dz * dy;
        const int *src = a.sets.pool + a.sets.off[e.x];
        for (int c = tid; c < cells; c += kThreads) smem[c] = __ldcg(src + c);
        stratum_offsets(g, sh, d, dz, zoff);
        __syncthreads();
        const Verdict v = score_fixed(g, smem, zoff, sh.stride[rx], sh.stride[ry], dx, dy, dz, ni, nj, nk,
                                      a.sets.h + e.x, a.fx, a.alpha, S, scratch);
        if (tid == 0) {
            record(a, e.y, v, cells, 0, 1);
            if (d == 0 && a.pair_g2) keep_pair(a, a.item_vars[(int64_t)e.y * 2], a.item_vars[(int64_t)e.y * 2 + 1], v.g2);
        }
        __syncthreads();
    }
}

// ---- level 2's bounds
// A level-2 test is bounded from below by the statistics of its sets of three variables
// (dependent_by_triples), which are far fewer than its tests: of a variable of k neighbours
// C(k, 2) against k C(k - 1, 2).  Before the level's first wave those of every edge and neighbour
// are completed from level 1's tables, which hold most of them counted, and the rest is counted
// now.  It leaves 22% of the tests run at level 2 to be counted with 100 variables x 50,000
// samples, 18% with 223 x 500,000 and 62% with 1,041 x 100,000 (tested_from_x included); the level
// takes 1.20, 7.96 and 13.3 ms where it took 1.68, 17.7 and 23.7.  The sets {y, z, w} with z and w
// neighbours of x alone would leave 3 to 11%, but they are as many as the sets of four.
constexpr int kTripleInts = 2048;  // the largest table taken (a warp's shared memory)

// One warp per edge of the level (a: level 1's sets; d = 1), a lane per neighbour of either end.
__global__ void __launch_bounds__(kThreads) triple_enter_kernel(WaveArgs a) {
    const int lane = threadIdx.x & 31, warps = gridDim.x * kWarps;
    for (int e = blockIdx.x * kWarps + (threadIdx.x >> 5); e < a.n_edges; e += warps) {
        const int x = a.ex[e], y = a.ey[e], nx = a.deg[x] - 1, ny = a.deg[y] - 1;
        const int dxy = (int)a.card[x] * a.card[y];
        for (int i = lane; i < nx + ny; i += 32) {
            const int from = i < nx ? x : y, skip = i < nx ? a.pxy[e] : a.pyx[e], k = i < nx ? i : i - nx;
            const int z = a.adjl[(int64_t)from * a.adj_stride + (k < skip ? k : k + 1)];
            if (i >= nx && tested_from_x(a, x, &z)) continue;
            const int cells = dxy * a.card[z];
            if (cells > kTripleInts) continue;
            const uint16_t sv[3] = {(uint16_t)min(x, z), (uint16_t)(z < x ? x : min(y, z)), (uint16_t)max(y, z)};
            bool fresh;
            const int at = set_enter(a.sets, sv, 3, &fresh);
            if (at < 0) continue;
            const bool list = atomicExch(&a.tri.listed[at], 1) == 0;
            if (!fresh && !list) continue;
            const int item = atomicAdd(&a.counters[C_TIER0], 1);
            const bool fits = item < a.list_cap;
            if (fresh) {
                const unsigned long long o = fits ? atomicAdd(a.sets.used, (unsigned long long)((cells + 3) & ~3)) : 0;
                const bool room = fits && o + cells <= a.sets.pool_cap;
                a.sets.off[at] = room ? (int32_t)o : -1;
                if (room) {
                    const int c = set_class(cells, a.var_S[x]);
                    a.sets.fresh[c * a.list_cap + atomicAdd(&a.counters[C_SET + c], 1)] = make_int2(at, item);
                }
            }
            if (!fits) continue;
            uint16_t *iv = a.item_vars + (int64_t)item * 3;
            iv[0] = (uint16_t)z;
            iv[1] = (uint16_t)x;
            iv[2] = (uint16_t)y;
            if (list) a.sets.items[atomicAdd(&a.counters[C_SCOREW], 1)] = make_int2(at, item);
        }
    }
}

// The three statistics of each listed set, from its table: a warp per set.
__global__ void __launch_bounds__(kThreads, 3) triple_score_kernel(WaveArgs a) {
    extern __shared__ int smem[];
    __shared__ SetShape s_shape[kWarps];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, n = a.counters[C_SCOREW];
    int *t = smem + warp * kTripleInts;
    SetShape &sh = s_shape[warp];
    for (int idx = blockIdx.x * kWarps + warp; idx < n; idx += gridDim.x * kWarps) {
        const int2 e = a.sets.items[idx];
        if (a.sets.off[e.x] < 0) continue;
        set_shape(a, e.y, lane, sh);
        const int m[3] = {(int)sh.dim[0], (int)sh.dim[1], (int)sh.dim[2]};
        const int st[3] = {m[1] * m[2], m[2], 1}, cells = m[0] * st[0];
        const int *src = a.sets.pool + a.sets.off[e.x];
        for (int c = lane; c < cells; c += 32) t[c] = __ldcg(src + c);
        __syncwarp();
        long long pair[3] = {0, 0, 0}, one[3] = {0, 0, 0};  // sums of F: without variable c, of variable c
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const int u = c == 0 ? 1 : 0, v = c == 2 ? 1 : 2;
            for (int q = lane; q < m[u] * m[v]; q += 32) {
                const int i = q / m[v], j = q - i * m[v];
                int s = 0;
                for (int k = 0; k < m[c]; ++k) s += t[i * st[u] + j * st[v] + k * st[c]];
                pair[c] += __ldg(&a.fx.f[s]);
            }
            for (int k = lane; k < m[c]; k += 32) {
                int s = 0;
                for (int i = 0; i < m[u]; ++i)
                    for (int j = 0; j < m[v]; ++j) s += t[k * st[c] + i * st[u] + j * st[v]];
                one[c] += __ldg(&a.fx.f[s]);
            }
        }
        __syncwarp();
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            pair[c] = warp_sum_ll(pair[c]);
            one[c] = warp_sum_ll(one[c]);
        }
        if (lane < 3) {
            const long long sum = a.sets.h[e.x] - (pair[0] + pair[1] + pair[2] - pair[lane]) + one[lane];
            a.tri.g[3 * (int64_t)e.x + lane] = (float)(2.0 * a.fx.unit * (double)sum);
        }
    }
}

}  // namespace fpgm
