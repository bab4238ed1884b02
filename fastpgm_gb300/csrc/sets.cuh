// Tests whose joint tables fit shared memory, counted once per variable set.
//
// A test (x, y | Z) needs the joint table of the set {x, y} + Z whichever of its variables are
// x and y: the same set comes back under its other pairs, and under the same pair from the other
// side (CheckEdge tests Z from x's neighbours, then from y's, PCStable.cpp:399-494).  So a
// level keeps the tables it has counted, over the set's variables in ascending order, and a test
// is scored from its set's table with the strides of its own x, y and Z.
//   classify        enters the test's set (set_enter); a set met for the first time gets room
//                   for its table and goes to the list of sets to count
//   set_count_*     one warp (tables of at most WaveArgs::warp_ints) or one CTA per new set
//   set_score_*     one warp or one CTA per test
// Tests per distinct set, duplicates of a pair included: 1.2 (1,041 variables, level 1), 1.6 to
// 2.0 (100 to 223 variables, level 1), 2 to 2.3 at level 2, 3.3 to 3.8 at level 3, 4.8 at level 4.
#pragma once
#include "ci_kernels.cuh"

namespace fpgm {

// Replicas (log2) of a counted table interleaved cell by cell, as many as fit `ints`.
__device__ __forceinline__ int replica_log(int cells, int extra, int ints) {
    for (int l = 5; l >= 1; --l)
        if ((cells << l) + extra <= ints) return l;
    return 0;
}

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

// One warp per new set.  Bound by instruction issue (4.5 per sample and set of three columns)
// and the shared-memory atomic unit; the samples come from L2.
template <int kSlice, int kMinBlocks>
__global__ void __launch_bounds__(kThreads, kMinBlocks) set_count_warp_kernel(WaveArgs a) {
    extern __shared__ int smem[];
    __shared__ SetShape s_shape[kWarps];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int *rep = smem + warp * kSlice;
    SetShape &sh = s_shape[warp];
    const int n0 = a.counters[C_SETW], ncols = a.d + 2;
    if (n0 <= a.sets.few) return;  // set_count_cta_kernel takes them
    for (;;) {
        int idx = 0;
        if (lane == 0) idx = atomicAdd(&a.counters[C_WSETW], 1);
        idx = __shfl_sync(0xffffffffu, idx, 0);
        if (idx >= n0) break;
        const int2 e = a.sets.fresh[idx];  // set, an item of it
        const int64_t S = a.var_S[a.item_vars[(int64_t)e.y * ncols]];
        set_shape(a, e.y, lane, sh);
        const int cells = sh.stride[0] * (int)sh.dim[0];
        const int lgR = replica_log(cells, 0, kSlice);
        for (int i = lane; i < (cells << lgR); i += 32) rep[i] = 0;
        __syncwarp();
        // lane l counts into replica l mod R: with 32 replicas every lane owns one bank
        count_columns<32>(rep, lgR, lane, sh.col, sh.dim, ncols, S, lane);
        __syncwarp();
        int *out = a.sets.pool + a.sets.off[e.x];
        long long h = 0;
        for (int c = lane; c < cells; c += 32) {
            int n = 0;
            for (int r = 0; r < (1 << lgR); ++r) n += rep[(c << lgR) + ((r + lane) & ((1 << lgR) - 1))];
            out[c] = n;
            h += __ldg(&a.fx.f[n]);
        }
        h = warp_sum_ll(h);
        if (lane == 0) a.sets.h[e.x] = h;
        __syncwarp();
    }
}

// One CTA per new set whose table is beyond a warp's slice, and for every new set of a wave with
// no more of them than CTAs: a warp would count 500,000 samples in about 100 us while the rest
// of the GPU waits.
__global__ void __launch_bounds__(kThreads, 2) set_count_cta_kernel(WaveArgs a) {
    extern __shared__ int smem[];
    __shared__ SetShape sh;
    __shared__ int s_idx;
    __shared__ long long s_h;
    const int tid = threadIdx.x, lane = tid & 31;
    const int n1 = a.counters[C_SETC], ncols = a.d + 2;
    const int n0 = a.counters[C_SETW] <= a.sets.few ? a.counters[C_SETW] : 0;
    for (;;) {
        if (tid == 0) {
            s_idx = atomicAdd(&a.counters[C_WSETC], 1);
            s_h = 0;
        }
        __syncthreads();
        const int idx = s_idx;
        if (idx >= n1 + n0) break;
        const int2 e = a.sets.fresh[idx < n1 ? a.list_cap - 1 - idx : idx - n1];
        const int64_t S = a.var_S[a.item_vars[(int64_t)e.y * ncols]];
        if (tid < 32) set_shape(a, e.y, lane, sh);
        __syncthreads();
        const int cells = sh.stride[0] * (int)sh.dim[0];
        const int lgR = replica_log(cells, 0, kCtaInts);
        for (int i = tid; i < (cells << lgR); i += kThreads) smem[i] = 0;
        __syncthreads();
        count_columns<kThreads>(smem, lgR, lane, sh.col, sh.dim, ncols, S, tid);
        __syncthreads();
        int *out = a.sets.pool + a.sets.off[e.x];
        long long h = 0;
        for (int c = tid; c < cells; c += kThreads) {
            int n = 0;
            for (int r = 0; r < (1 << lgR); ++r) n += smem[(c << lgR) + ((r + lane) & ((1 << lgR) - 1))];
            out[c] = n;
            h += __ldg(&a.fx.f[n]);
        }
        h = warp_sum_ll(h);
        if (lane == 0) atomicAdd(reinterpret_cast<unsigned long long *>(&s_h), (unsigned long long)h);
        __syncthreads();
        if (tid == 0) a.sets.h[e.x] = s_h;
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
        if (lane == 0) record(a, e.y, v, cells, 0, 0);
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
        if (tid == 0) record(a, e.y, v, cells, 0, 1);
        __syncthreads();
    }
}

}  // namespace fpgm
