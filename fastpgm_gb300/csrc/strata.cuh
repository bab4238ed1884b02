// Shared strata: the CI tests of a wave whose joint tables are too large for shared memory,
// counted through the variable sets they have in common.
//
// With F(n) = n ln n and, for a set V of variables, H(V) = sum of F over the counts of V's
// configurations, the statistic of a test (c, o | Z) is
//     G^2 = 2 [ H(Z + c + o) - H(Z + c) - H(Z + o) + H(Z) ]
// (the textbook G^2 with ln(O N_z / (N_x N_y)) split into its four logarithms), and its degrees
// of freedom are the sum over Z's strata of (a_c - 1)(a_o - 1), a_v the number of v's values
// that occur in the stratum (IndependenceTest.cpp:94-138).  The sets belong to many tests: c is
// the side whose neighbours Z are drawn from (CheckEdge, PCStable.cpp:399-494), so every o and
// every split of Z + o into Z and o share them.  At 1,041 variables x 100,000 samples, |Z| = 6,
// 19,922 tests share 2,849 sets Z + c + o and 3,767 sets Z.
//
// Strata of one sample add nothing to any H (F(1) = 0) nor to any degree of freedom, in Z or in
// any set that refines Z, so only strata of two or more samples are kept.  A set's strata are
// one 16-bit id per sample (kNoStratum: left out), refined variable by variable: the strata of
// P + v are the (id, v) pairs that two or more samples share, counted in shared memory with no
// hashing and no sorting.
//   strata_collect  a test's sets, found or entered in a trie (a node = its parent node and the
//                   next variable, ascending) and in a table of (node, variable) pairs
//   strata_build    a new node: its ids, H, number of strata (one CTA per node, one launch per
//                   set size, parents first)
//   strata_pair     a new pair (P, v): H(P + v) and a_v for every stratum of P
//   strata_test     a test: which values of o occur in every stratum of Z (one bit mask per
//                   stratum), the degrees of freedom, the decision
// Nodes and pairs live until the skeleton ends: the sets Z + o of level d are the sets Z of
// level d + 1, and the pairs (Z + o, c) its pairs (Z, c).
//
// F is the fixed-point table of fixed.cuh: exact sums, whatever their order.
#pragma once
#include "ci_kernels.cuh"

namespace fpgm {

constexpr int kStrataThreads = 512;
constexpr int kStrataInts = 27 * 1024;               // 108 KB of shared counters, two CTAs per SM
constexpr uint32_t kNoStratum = 0xffffu;
constexpr int kStrataMaxSets = kMaxCond + 2;         // sizes of built sets: 1 .. |Z| + 1
constexpr int kStrataMaxCard = 32;                   // states of the test's o (one mask word)

// counters, cleared for every wave: nodes to build per size, taken per size, pairs, tests
struct StrataCounters {
    int32_t n_build[kStrataMaxSets + 1], w_build[kStrataMaxSets + 1];
    int32_t n_pair, w_pair, w_test;
};

struct StrataArgs {
    uint64_t *node_key;    // trie: ((parent + 1) << 16 | variable) | 1 << 62; 0: free; a node's index is its place
    uint64_t *pair_key;    // (node << 16 | variable) | 1 << 62
    int32_t node_cap, pair_cap;  // powers of two
    int32_t *node_n;       // strata kept; -1: not built (out of room, or more than 65,534 strata)
    int32_t *node_max;     // samples of the largest
    long long *node_h;     // H
    int64_t *node_ids;     // its ids, an offset into the pool
    long long *pair_h;
    int64_t *pair_a;       // offset of a_v - 1 per stratum in the pool; -1: not counted
    char *pool;            // ids and a_v vectors
    unsigned long long *pool_used;  // [0] bytes handed out (past the capacity: out of room), [1] nodes, [2] pairs
    unsigned long long pool_cap;
    int32_t *build_list;   // [size][build_cap] node indices
    int32_t *pair_list;
    int32_t build_cap, pair_list_cap;
    int4 *item_ref;        // per listed test: nodes Z and Z + o, pairs (Z, c) and (Z + o, c)
    StrataCounters *sc;
};

// The trie node of a set of m ascending variables (entered with every prefix that is missing);
// -1 when there is no room.
__device__ inline int strata_node(const StrataArgs &s, const uint16_t *v, int m) {
    int at = -1;
    for (int i = 0; i < m; ++i) {
        bool fresh;
        at = table_enter(s.node_key, s.node_cap, kEnterProbe, ((uint64_t)(at + 1) << 16 | v[i]) | (1ull << 62), &fresh);
        if (at < 0) return -1;
        if (fresh) {
            s.node_n[at] = -1;
            atomicAdd(&s.pool_used[1], 1ull);
            const int q = atomicAdd(&s.sc->n_build[i + 1], 1);
            if (q < s.build_cap) s.build_list[(int64_t)(i + 1) * s.build_cap + q] = at;
        }
    }
    return at;
}

__device__ inline int strata_pair_of(const StrataArgs &s, int node, int v) {
    bool fresh;
    const int at = table_enter(s.pair_key, s.pair_cap, kEnterProbe, ((uint64_t)node << 16 | (uint64_t)v) | (1ull << 62), &fresh);
    if (fresh) {
        s.pair_a[at] = -1;
        atomicAdd(&s.pool_used[2], 1ull);
        const int q = atomicAdd(&s.sc->n_pair, 1);
        if (q < s.pair_list_cap) s.pair_list[q] = at;
    }
    return at;
}

// One thread per listed test: enters its sets; a test with no room goes to the per-test kernels.
__global__ void strata_collect_kernel(WaveArgs a, StrataArgs s) {
    const int n = a.counters[C_STRATA], d = a.d;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int e = a.lists[6 * a.list_cap + i], item = e >> 1;
        const uint16_t *iv = a.item_vars + (int64_t)item * (d + 2);
        const int c = iv[d + (e & 1)], o = iv[d + 1 - (e & 1)];
        uint16_t v[kMaxCond + 1];
        for (int k = 0; k < d; ++k) v[k] = iv[k];
        int4 r;
        r.x = strata_node(s, v, d);
        int k = d;
        for (; k > 0 && v[k - 1] > o; --k) v[k] = v[k - 1];
        v[k] = (uint16_t)o;
        r.y = strata_node(s, v, d + 1);
        r.z = r.x < 0 ? -1 : strata_pair_of(s, r.x, c);
        r.w = r.y < 0 ? -1 : strata_pair_of(s, r.y, c);
        s.item_ref[i] = r;
    }
}

// Ids of 16 consecutive samples (vector v; ids null: every sample of the dataset in stratum 0).
__device__ __forceinline__ void strata_ids16(uint32_t (&id)[8], const uint16_t *ids, int64_t v, int64_t S) {
    if (ids) {
        const uint4 p = __ldcg(reinterpret_cast<const uint4 *>(ids) + 2 * v);
        const uint4 q = __ldcg(reinterpret_cast<const uint4 *>(ids) + 2 * v + 1);
        id[0] = p.x; id[1] = p.y; id[2] = p.z; id[3] = p.w;
        id[4] = q.x; id[5] = q.y; id[6] = q.z; id[7] = q.w;
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int64_t s0 = 16 * v + 2 * i;
            id[i] = (s0 < S ? 0u : kNoStratum) | (s0 + 1 < S ? 0u : kNoStratum << 16);
        }
    }
}

__device__ __forceinline__ long long block_sum_ll(long long v, long long *scratch) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) scratch[threadIdx.x >> 5] = v;
    __syncthreads();
    long long r = 0;
    for (int w = 0; w < kStrataThreads / 32; ++w) r += scratch[w];
    return r;
}

// Counts the (stratum of P, value of v) pairs in shared memory, as many strata at a time as fit,
// and reads the counts row by row (a row = a stratum, a thread each).  kBuild: P + v becomes a
// node (its strata numbered in the order the counts are met, its ids written in a second sweep
// over the samples); else a pair (a_v - 1 per stratum).
// Counters are 32 bits wide, in up to 32 copies interleaved cell by cell while they fit (the
// lanes of a warp then hit different banks); 16 bits wide when the 32-bit ones would not fit
// and no stratum of P has more samples than they hold.
// What bounds it: shared-memory atomics, one per sample (a sweep reads 3 bytes per sample from
// L2).
template <bool kBuild>
__global__ void __launch_bounds__(kStrataThreads, 2) strata_count_kernel(WaveArgs a, StrataArgs s, int size) {
    extern __shared__ __align__(16) int smem[];
    __shared__ long long scratch[kStrataThreads / 32];
    __shared__ int s_idx, s_new, s_max;
    __shared__ long long s_off;
    const int tid = threadIdx.x, lane = tid & 31;
    const int n_list = kBuild ? min(s.sc->n_build[size], s.build_cap) : min(s.sc->n_pair, s.pair_list_cap);
    for (;;) {
        if (tid == 0) s_idx = atomicAdd(kBuild ? &s.sc->w_build[size] : &s.sc->w_pair, 1);
        __syncthreads();
        if (s_idx >= n_list) break;
        const int at = kBuild ? s.build_list[(int64_t)size * s.build_cap + s_idx] : s.pair_list[s_idx];
        const uint64_t key = (kBuild ? s.node_key[at] : s.pair_key[at]) & ~(1ull << 62);
        const int var = (int)(key & 0xffff), parent = (int)(key >> 16) - (kBuild ? 1 : 0);
        const int64_t S = a.var_S[var], nvec = (S + 15) >> 4;
        const int n = parent < 0 ? 1 : s.node_n[parent];
        const int pmax = parent < 0 ? (int)S : s.node_max[parent];
        const uint16_t *ids = parent < 0 || n < 0 ? nullptr : reinterpret_cast<const uint16_t *>(s.pool + s.node_ids[parent]);
        const uint8_t *col = a.cols + a.var_off[var];
        const int cv = a.card[var];
        if (tid == 0) {
            const unsigned long long need = kBuild ? (unsigned long long)(nvec * 32) : (unsigned long long)((n + 15) & ~15);
            s_off = -1;
            if (n >= 0) {
                const unsigned long long o = atomicAdd(s.pool_used, need);
                if (o + need <= s.pool_cap) s_off = (long long)o;
            }
            s_new = 0;
            s_max = 0;
        }
        __syncthreads();
        const int64_t off = s_off;
        if (off < 0) {  // the parent was not built, or no room: its tests go to the per-test kernels
            __syncthreads();
            continue;
        }
        const int64_t cells = (int64_t)n * cv;
        const bool wide = cells <= kStrataInts || pmax > 0xffff;  // 32-bit counters
        int lgR = 0;
        if (wide)
            while (lgR < 5 && (cells << (lgR + 1)) + (kBuild ? cells : 0) <= kStrataInts) ++lgR;
        const int rows = (int)min((int64_t)n, (int64_t)(wide ? kStrataInts : 2 * kStrataInts) / cv);
        uint16_t *out = reinterpret_cast<uint16_t *>(s.pool + off);
        uint8_t *av = reinterpret_cast<uint8_t *>(s.pool + off);
        int *names = lgR > 0 ? smem + (cells << lgR) : smem;  // kBuild: new ids, one word per cell (wide)
        uint16_t *half = reinterpret_cast<uint16_t *>(smem);
        long long h = 0;
        int big = 0;
        for (int r0 = 0; r0 < n; r0 += rows) {
            const int r1 = min(n, r0 + rows), nr = r1 - r0;
            const int words = wide ? (nr * cv) << lgR : (nr * cv + 1) >> 1;
            for (int i = tid; i < words; i += kStrataThreads) smem[i] = 0;
            __syncthreads();
            const int rep = lane & ((1 << lgR) - 1);
            for (int64_t v = tid; v < nvec; v += kStrataThreads) {
                uint32_t id[8];
                strata_ids16(id, ids, v, S);
                const uint4 w = __ldg(reinterpret_cast<const uint4 *>(col) + v);
                const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                for (int b = 0; b < 16; ++b) {
                    const uint32_t k = (id[b >> 1] >> (16 * (b & 1))) & 0xffffu;
                    if (k == kNoStratum || k - (uint32_t)r0 >= (uint32_t)nr) continue;
                    const uint32_t c = (k - r0) * cv + ((ww[b >> 2] >> (8 * (b & 3))) & 0xffu);
                    if (wide) atomicAdd(&smem[(c << lgR) + rep], 1);
                    else atomicAdd(&smem[c >> 1], 1 << (16 * (c & 1)));
                }
            }
            __syncthreads();
            // rows: F of every count, values met, strata kept
            const int rounds = (nr + kStrataThreads - 1) / kStrataThreads;
            for (int rd = 0; rd < rounds; ++rd) {
                const int r = rd * kStrataThreads + tid;
                int met = 0, kept = 0;
                if (r < nr) {
                    for (int j = 0; j < cv; ++j) {
                        const int c = r * cv + j;
                        int m = 0;
                        if (wide) {
                            for (int q = 0; q < (1 << lgR); ++q) m += smem[(c << lgR) + ((q + tid) & ((1 << lgR) - 1))];
                            if (kBuild) names[c] = m;  // lgR == 0: in place
                        } else {
                            m = half[c];
                        }
                        if (m == 0) continue;
                        ++met;
                        if (m >= 2) {
                            ++kept;
                            h += __ldg(&a.fx.f[m]);
                            big = max(big, m);
                        }
                    }
                    if (!kBuild) av[r0 + r] = (uint8_t)(met - 1);
                }
                if (kBuild) {
                    int incl = kept;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const int t = __shfl_up_sync(0xffffffffu, incl, o);
                        if (lane >= o) incl += t;
                    }
                    int first = 0;
                    if (lane == 31 && incl > 0) first = atomicAdd(&s_new, incl);
                    first = __shfl_sync(0xffffffffu, first, 31) + incl - kept;
                    if (r < nr)
                        for (int j = 0; j < cv; ++j) {
                            const int c = r * cv + j;
                            const int m = wide ? names[c] : half[c];
                            const int name = m >= 2 ? min(first++, (int)kNoStratum) : (int)kNoStratum;
                            if (wide) names[c] = name;
                            else half[c] = (uint16_t)name;
                        }
                }
            }
            __syncthreads();
            if (kBuild) {
                for (int64_t v = tid; v < nvec; v += kStrataThreads) {
                    uint32_t id[8];
                    strata_ids16(id, ids, v, S);
                    const uint4 w = __ldg(reinterpret_cast<const uint4 *>(col) + v);
                    const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
                    uint32_t o[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
                    for (int b = 0; b < 16; ++b) {
                        const uint32_t k = (id[b >> 1] >> (16 * (b & 1))) & 0xffffu;
                        uint32_t name = kNoStratum;
                        if (k != kNoStratum && k - (uint32_t)r0 < (uint32_t)nr) {
                            const uint32_t c = (k - r0) * cv + ((ww[b >> 2] >> (8 * (b & 3))) & 0xffu);
                            name = wide ? (uint32_t)names[c] : (uint32_t)half[c];
                            if (r0 > 0) out[16 * v + b] = (uint16_t)name;  // later rows: only their own samples
                        }
                        o[b >> 1] |= name << (16 * (b & 1));
                    }
                    if (r0 == 0) {
                        uint4 *dst = reinterpret_cast<uint4 *>(out) + 2 * v;
                        dst[0] = make_uint4(o[0], o[1], o[2], o[3]);
                        dst[1] = make_uint4(o[4], o[5], o[6], o[7]);
                    }
                }
                __syncthreads();
            }
        }
        if (kBuild) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) big = max(big, __shfl_xor_sync(0xffffffffu, big, o));
            if (lane == 0) atomicMax(&s_max, big);
        }
        h = block_sum_ll(h, scratch);  // its barriers make s_new and s_max final
        if (tid == 0) {
            if (kBuild) {
                s.node_h[at] = h;
                s.node_ids[at] = off;
                s.node_max[at] = s_max;
                s.node_n[at] = s_new <= 0xfffe ? s_new : -1;
            } else {
                s.pair_h[at] = h;
                s.pair_a[at] = off;
            }
        }
        __syncthreads();
    }
}

// One CTA per test: the values of o met in every stratum of Z as one mask word per stratum (a
// value already seen is not written again), the degrees of freedom, the statistic from the four
// sums, the decision.  Undecided within the error bound, or a set that was not counted: the
// per-test kernels take the test (C_TIER2 list).
__global__ void __launch_bounds__(kStrataThreads, 2) strata_test_kernel(WaveArgs a, StrataArgs s) {
    extern __shared__ __align__(16) int smem[];
    __shared__ long long scratch[kStrataThreads / 32];
    __shared__ int s_idx;
    const int tid = threadIdx.x;
    const int n_list = a.counters[C_STRATA], d = a.d;
    uint32_t *mask = reinterpret_cast<uint32_t *>(smem);
    for (;;) {
        if (tid == 0) s_idx = atomicAdd(&s.sc->w_test, 1);
        __syncthreads();
        const int i = s_idx;
        if (i >= n_list) break;
        const int e = a.lists[6 * a.list_cap + i], item = e >> 1;
        const int4 r = s.item_ref[i];
        const int n = r.x >= 0 ? s.node_n[r.x] : -1;
        const int64_t aoff = r.z >= 0 ? s.pair_a[r.z] : -1;
        const bool ok = n >= 0 && aoff >= 0 && r.y >= 0 && r.w >= 0 && s.node_n[r.y] >= 0 && s.pair_a[r.w] >= 0;
        long long df = 0;
        if (ok) {
            const int o = a.item_vars[(int64_t)item * (d + 2) + d + 1 - (e & 1)];
            const int64_t S = a.var_S[o], nvec = (S + 15) >> 4;
            const uint8_t *col = a.cols + a.var_off[o];
            const uint16_t *ids = reinterpret_cast<const uint16_t *>(s.pool + s.node_ids[r.x]);
            const uint8_t *av = reinterpret_cast<const uint8_t *>(s.pool + aoff);
            for (int r0 = 0; r0 < n; r0 += kStrataInts) {
                const int nr = min(n - r0, kStrataInts);
                for (int k = tid; k < nr; k += kStrataThreads) mask[k] = 0u;
                __syncthreads();
                for (int64_t v = tid; v < nvec; v += kStrataThreads) {
                    uint32_t id[8];
                    strata_ids16(id, ids, v, S);
                    const uint4 w = __ldg(reinterpret_cast<const uint4 *>(col) + v);
                    const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                    for (int b = 0; b < 16; ++b) {
                        const uint32_t k = ((id[b >> 1] >> (16 * (b & 1))) & 0xffffu) - (uint32_t)r0;
                        if (k >= (uint32_t)nr) continue;  // left out (n <= 65,534), or another round's
                        const uint32_t bit = 1u << ((ww[b >> 2] >> (8 * (b & 3))) & 0x1fu);
                        if (!(mask[k] & bit)) atomicOr(&mask[k], bit);
                    }
                }
                __syncthreads();
                for (int k = tid; k < nr; k += kStrataThreads)
                    df += (long long)__ldcg(av + r0 + k) * (__popc(mask[k]) - 1);
                __syncthreads();
            }
        }
        df = block_sum_ll(df, scratch);
        if (tid < 32) {
            int dec = -1;
            if (ok) {
                const long long hs = s.pair_h[r.w] - s.pair_h[r.z] - s.node_h[r.y] + s.node_h[r.x];
                const int64_t S = a.var_S[a.item_vars[(int64_t)item * (d + 2) + d]];
                // the four sums hold at most 2 S counts of two or more
                double g2;
                dec = fixed_decide(a.fx, df, hs, 2 * S, S, &g2);
                if (dec < 0) {
                    const double err = 2.0 * a.fx.unit * (double)S + 2e-14 * (double)S;
                    if (df > a.fx.dfmax) {
                        const double pw = chisq_pvalue_wh(g2, (double)df);
                        const double slack = kBand + kWhMargin + 2.0 * err * 0.3 / sqrt((double)df);
                        if (fabs(pw - a.alpha) > slack) dec = pw > a.alpha;
                    }
                    if (dec < 0) {  // the p-value, unless its error bound (a density of at most 1/2) reaches alpha
                        const double p = chisq_pvalue(fmax(g2, 0.0), df);
                        if (fabs(p - a.alpha) > 1e-7 + err && (df > 1 || g2 > 1.0)) dec = p > a.alpha;
                        if (dec >= 0 && tid == 0) atomicAdd(&a.stats[ST_RECHECK], 1ull);
                    }
                }
            }
            if (tid == 0) {
                if (dec >= 0) {
                    a.flag[item] = (uint8_t)dec;
                    atomicAdd(&a.stats[ST_LARGE], 1ull);
                } else {
                    const int q = atomicAdd(&a.counters[C_TIER2], 1);
                    a.lists[2 * a.list_cap + q] = item;
                }
            }
        }
        __syncthreads();
    }
}

}  // namespace fpgm
