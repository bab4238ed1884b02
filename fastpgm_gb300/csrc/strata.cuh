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
//   strata_pack     the tests of a pair (Z, c), in packs of up to four
//   strata_test     a pack of tests: which values of their o's
//                   occur in every stratum of Z (bit masks in one word per stratum), the degrees
//                   of freedom, the decisions
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
    int32_t n_pair, w_pair, n_group, n_pack, w_test;
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
    int32_t *item_next;    // ... and the next listed test of its pair (Z, c)
    int32_t *pair_head;    // per pair: the last listed test of the wave (1 + its place), 0: none
    int32_t *group_list;   // pairs (Z, c) of the wave's tests; -1 - place: a test without a pair
    int4 *pack_list;       // tests counted together: up to four places, -1: none
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
        // tests of a pair (Z, c) are linked; the first one to come lists the pair
        const int before = r.z >= 0 ? atomicExch(&s.pair_head[r.z], i + 1) : 0;
        s.item_next[i] = before;
        if (before == 0) s.group_list[atomicAdd(&s.sc->n_group, 1)] = r.z >= 0 ? r.z : -1 - i;
    }
}

// One thread per pair (Z, c) with tests: cut into packs whose o's states fit a 32-bit word (8, 16
// or 32 bits each), and of no more tests than leave a pack for every CTA of strata_test_kernel.
constexpr int kPack = 4;
__device__ inline int pack_bits(int states) { return states <= 8 ? 8 : states <= 16 ? 16 : 32; }
__global__ void strata_pack_kernel(WaveArgs a, StrataArgs s, int ctas) {
    const int n = s.sc->n_group, d = a.d, most = max(1, min(kPack, a.counters[C_STRATA] / ctas));
    for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < n; g += gridDim.x * blockDim.x) {
        const int pair = s.group_list[g];
        int at = pair >= 0 ? s.pair_head[pair] : -pair;  // places from 1
        if (pair >= 0) s.pair_head[pair] = 0;
        while (at > 0) {
            int place[kPack] = {-1, -1, -1, -1}, used = 0;
#pragma unroll
            for (int m = 0; m < kPack; ++m) {
                if (at <= 0 || m >= most) break;
                const int e = a.lists[6 * a.list_cap + at - 1];
                const int bits = pack_bits(a.card[a.item_vars[(int64_t)(e >> 1) * (d + 2) + d + 1 - (e & 1)]]);
                if (used + bits > 32) break;
                used += bits;
                place[m] = at - 1;
                at = s.item_next[at - 1];
            }
            s.pack_list[atomicAdd(&s.sc->n_pack, 1)] = make_int4(place[0], place[1], place[2], place[3]);
        }
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

// Where a (stratum, value) pair is counted: rows of cv words, a row per stratum.  Wide: 32-bit
// counters, in up to 32 copies interleaved word by word while they fit (the lanes of a warp then
// hit different banks).  Else 16-bit ones, two rows to one row of words: the lower half of the
// strata in the low halves (when 32-bit ones would not fit and no stratum of P has more samples
// than 16 bits hold).
struct StrataRows {
    uint32_t r0, nr;    // strata counted in this pass
    uint32_t split;     // strata of the round in low halves (wide: all)
    uint32_t cv, mul;   // values of v; bytes from one word's copy to the next word's
    uint32_t base;      // shared-memory address of this lane's copy
};

// Adds one sample (16 bits of id, a byte of v) when its stratum is of this pass.
__device__ __forceinline__ void strata_add(const StrataRows &g, uint32_t id, uint32_t value) {
    uint32_t k = id - g.r0;
    if (k >= g.nr) return;  // kNoStratum is past every round's last stratum (n <= 65,534)
    const bool high = k >= g.split;
    if (high) k -= g.split;
    asm volatile("red.shared.add.u32 [%0], %1;" ::"r"((k * g.cv + value) * g.mul + g.base), "r"(high ? 0x10000u : 1u)
                 : "memory");
}
__device__ __forceinline__ void strata_add16(const StrataRows &g, const uint32_t (&id)[8], const uint4 w) {
    const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int b = 0; b < 16; ++b)
        strata_add(g, __byte_perm(id[b >> 1], 0, b & 1 ? 0x4432 : 0x4410), __byte_perm(ww[b >> 2], 0, 0x4440 + (b & 3)));
}

// Counts the (stratum of P, value of v) pairs in shared memory, as many strata at a time as fit,
// and reads the counts row by row (a stratum, a thread each).  kBuild: P + v becomes a node (its
// strata numbered in the order the counts are met, its ids written in a second sweep over the
// samples); else a pair (a_v - 1 per stratum).
// Bound by instruction issue (55% active at 32 warps per SM; 7 per sample and sweep) and the
// shared-memory atomics, one per sample; a sweep reads 3 bytes per sample from L2.
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
        const int64_t S = a.var_S[var];
        const int nvec = (int)((S + 15) >> 4);
        const int n = parent < 0 ? 1 : s.node_n[parent];
        const int pmax = parent < 0 ? (int)S : s.node_max[parent];
        const uint16_t *ids = parent < 0 || n < 0 ? nullptr : reinterpret_cast<const uint16_t *>(s.pool + s.node_ids[parent]);
        const uint4 *col = reinterpret_cast<const uint4 *>(a.cols + a.var_off[var]);
        const int cv = a.card[var];
        if (tid == 0) {
            const unsigned long long need = kBuild ? (unsigned long long)nvec * 32 : (unsigned long long)((n + 15) & ~15);
            s_off = -1;
            if (n >= 0) {
                const unsigned long long o = atomicAdd(s.pool_used, need);
                if (o + need <= s.pool_cap) s_off = (long long)o;
            }
            s_new = 0;
            s_max = 0;
            if (s_off >= 0)  // ids and column read once, new ids written
                atomicAdd(&a.stats[ST_BYTES_LARGE], (unsigned long long)S * ((parent < 0 ? 1 : 3) + (kBuild ? 2 : 0)));
        }
        __syncthreads();
        const int64_t off = s_off;
        if (off < 0) {  // the parent was not built, or no room: its tests go to the per-test kernels
            __syncthreads();
            continue;
        }
        const int64_t cells = (int64_t)n * cv;
        const bool wide = cells <= kStrataInts || pmax > 0xffff;
        int lgR = 0;
        if (wide)
            while (lgR < 5 && (cells << (lgR + 1)) + (kBuild ? cells : 0) <= kStrataInts) ++lgR;
        const int R = 1 << lgR, rows = (int)min((int64_t)n, (int64_t)(wide ? 1 : 2) * (kStrataInts / cv));
        uint16_t *out = reinterpret_cast<uint16_t *>(s.pool + off);
        uint8_t *av = reinterpret_cast<uint8_t *>(s.pool + off);
        int *names = lgR > 0 ? smem + (cells << lgR) : smem;  // kBuild, wide: new ids, one word per cell
        uint16_t *half = reinterpret_cast<uint16_t *>(smem);
        StrataRows g;
        g.cv = cv;
        g.mul = 4u << lgR;
        g.base = (uint32_t)__cvta_generic_to_shared(smem + (lane & (R - 1)));
        long long h = 0;
        int big = 0;
        for (int r0 = 0; r0 < n; r0 += rows) {
            const int nr = min(n - r0, rows), split = wide ? nr : (nr + 1) >> 1;
            g.r0 = r0;
            g.nr = nr;
            g.split = split;
            for (int i = tid; i < (split * cv) << lgR; i += kStrataThreads) smem[i] = 0;
            __syncthreads();
            int v = tid;
            for (; v + kStrataThreads < nvec; v += 2 * kStrataThreads) {  // two vectors' loads in flight
                uint32_t i0[8], i1[8];
                strata_ids16(i0, ids, v, S);
                strata_ids16(i1, ids, v + kStrataThreads, S);
                const uint4 w0 = __ldg(col + v), w1 = __ldg(col + v + kStrataThreads);
                strata_add16(g, i0, w0);
                strata_add16(g, i1, w1);
            }
            if (v < nvec) {
                uint32_t i0[8];
                strata_ids16(i0, ids, v, S);
                strata_add16(g, i0, __ldg(col + v));
            }
            __syncthreads();
            // rows: F of every count, values met, strata kept
            const int rounds = (nr + kStrataThreads - 1) / kStrataThreads;
            for (int rd = 0; rd < rounds; ++rd) {
                const int r = rd * kStrataThreads + tid;
                const int word = (r < split ? r : r - split) * cv, upper = r < split ? 0 : 1;  // half: in the high halves
                int met = 0, kept = 0;
                if (r < nr) {
                    for (int j = 0; j < cv; ++j) {
                        int m = 0;
                        if (wide) {
                            for (int q = 0; q < R; ++q) m += smem[((word + j) << lgR) + ((q + tid) & (R - 1))];
                            if (kBuild) names[word + j] = m;  // lgR == 0: in place
                        } else {
                            m = half[2 * (word + j) + upper];
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
                            const int m = wide ? names[word + j] : half[2 * (word + j) + upper];
                            const int name = m >= 2 ? min(first++, (int)kNoStratum) : (int)kNoStratum;
                            if (wide) names[word + j] = name;
                            else half[2 * (word + j) + upper] = (uint16_t)name;
                        }
                }
            }
            __syncthreads();
            if (kBuild) {
                // a sample's new id: the low half of its cell's word in names (wide) or its half
                const uint16_t *look = wide ? reinterpret_cast<const uint16_t *>(names) : half;
                for (int u = tid; u < nvec; u += kStrataThreads) {
                    uint32_t id[8];
                    strata_ids16(id, ids, u, S);
                    const uint4 w = __ldg(col + u);
                    const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
                    uint32_t o[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
                    for (int b = 0; b < 16; ++b) {
                        uint32_t k = __byte_perm(id[b >> 1], 0, b & 1 ? 0x4432 : 0x4410) - (uint32_t)r0;
                        uint32_t name = kNoStratum;
                        if (k < (uint32_t)nr) {
                            const bool high = k >= (uint32_t)split;
                            if (high) k -= split;
                            name = look[2 * (k * cv + __byte_perm(ww[b >> 2], 0, 0x4440 + (b & 3))) + (high ? 1 : 0)];
                            if (r0 > 0) out[16 * (int64_t)u + b] = (uint16_t)name;  // later rows: only their own samples
                        }
                        o[b >> 1] |= name << (16 * (b & 1));
                    }
                    if (r0 == 0) {
                        uint4 *dst = reinterpret_cast<uint4 *>(out) + 2 * (int64_t)u;
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

constexpr int kTestThreads = 256;
constexpr int kTestInts = 10 * 1024;  // strata per round: 40 KB of masks, five CTAs per SM

// A pack of tests of one pair (Z, c): a stratum's word holds, for each test, which values of its
// o occur in it, so one shared-memory read per sample (and an atomic when a value is new to the
// stratum) serves them all.  Then the degrees of freedom, the statistic from the four sums and
// the decision, a warp per test.  Undecided within the error bound, or a set that was not
// counted: the per-test kernels take the test (C_TIER2 list).
// Bound by instruction issue: 10 instructions per sample and 2.5 for every test (one test at a
// time took 12, and 36 us of a CTA at 50,000 samples, a third of it for clearing and reading the
// masks and deciding).
__global__ void __launch_bounds__(kTestThreads, 5) strata_test_kernel(WaveArgs a, StrataArgs s) {
    extern __shared__ __align__(16) int smem[];
    __shared__ int s_idx;
    __shared__ int s_place[kPack], s_shift[kPack], s_bits[kPack];
    __shared__ const uint4 *s_col[kPack];
    __shared__ unsigned long long s_df[kPack];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n_pack = s.sc->n_pack, d = a.d;
    uint32_t *mask = reinterpret_cast<uint32_t *>(smem);
    for (;;) {
        if (tid < 32) {
            int idx = 0;
            if (lane == 0) idx = atomicAdd(&s.sc->w_test, 1);
            idx = __shfl_sync(0xffffffffu, idx, 0);
            if (lane == 0) s_idx = idx;
            int place = -1, bits = 0, o = 0;
            if (idx < n_pack && lane < kPack) {
                place = reinterpret_cast<const int *>(s.pack_list + idx)[lane];
                if (place >= 0) {
                    const int e = a.lists[6 * a.list_cap + place];
                    o = a.item_vars[(int64_t)(e >> 1) * (d + 2) + d + 1 - (e & 1)];
                    bits = pack_bits(a.card[o]);
                }
            }
            int shift = 0;  // bits of the tests before this one
#pragma unroll
            for (int j = 0; j < kPack - 1; ++j) {
                const int bj = __shfl_sync(0xffffffffu, bits, j);
                if (j < lane) shift += bj;
            }
            if (lane < kPack) {
                s_place[lane] = place;
                s_bits[lane] = bits;
                s_shift[lane] = shift;
                s_col[lane] = reinterpret_cast<const uint4 *>(a.cols + a.var_off[o]);
                s_df[lane] = 0;
            }
        }
        __syncthreads();
        if (s_idx >= n_pack) break;
        {
            const int m = 1 + (s_place[1] >= 0) + (s_place[2] >= 0) + (s_place[3] >= 0);
            const int e0 = a.lists[6 * a.list_cap + s_place[0]];
            const int64_t S = a.var_S[a.item_vars[(int64_t)(e0 >> 1) * (d + 2) + d]];
            const int4 r0 = s.item_ref[s_place[0]];
            const int n = r0.x >= 0 ? s.node_n[r0.x] : -1;
            const int64_t aoff = r0.z >= 0 ? s.pair_a[r0.z] : -1;
            if (n >= 0 && aoff >= 0) {
                const int nvec = (int)((S + 15) >> 4);
                if (tid == 0) atomicAdd(&a.stats[ST_BYTES_LARGE], (unsigned long long)S * (2 + m));
                const uint4 *ids = reinterpret_cast<const uint4 *>(s.pool + s.node_ids[r0.x]);
                const uint8_t *av = reinterpret_cast<const uint8_t *>(s.pool + aoff);
                const uint4 *c0 = s_col[0], *c1 = s_col[m > 1 ? 1 : 0], *c2 = s_col[m > 2 ? 2 : 0], *c3 = s_col[m > 3 ? 3 : 0];
                // the word's lowest bit of each test (0: no such test)
                const uint32_t b0 = 1u, b1 = m > 1 ? 1u << s_shift[1] : 0u, b2 = m > 2 ? 1u << s_shift[2] : 0u,
                               b3 = m > 3 ? 1u << s_shift[3] : 0u;
                for (int r = 0; r < n; r += kTestInts) {
                    const uint32_t nr = (uint32_t)min(n - r, kTestInts);
                    for (int k = tid; k < (int)nr; k += kTestThreads) mask[k] = 0u;
                    __syncthreads();
                    for (int v = tid; v < nvec; v += kTestThreads) {
                        const uint4 p = __ldcg(ids + 2 * v), q = __ldcg(ids + 2 * v + 1);
                        const uint32_t id[8] = {p.x, p.y, p.z, p.w, q.x, q.y, q.z, q.w};
                        const uint4 w0 = __ldg(c0 + v);
                        uint4 w1 = make_uint4(0, 0, 0, 0), w2 = w1, w3 = w1;
                        if (m > 1) w1 = __ldg(c1 + v);
                        if (m > 2) w2 = __ldg(c2 + v);
                        if (m > 3) w3 = __ldg(c3 + v);
                        const uint32_t x0[4] = {w0.x, w0.y, w0.z, w0.w}, x1[4] = {w1.x, w1.y, w1.z, w1.w},
                                       x2[4] = {w2.x, w2.y, w2.z, w2.w}, x3[4] = {w3.x, w3.y, w3.z, w3.w};
#pragma unroll
                        for (int b = 0; b < 16; ++b) {
                            const uint32_t k = __byte_perm(id[b >> 1], 0, b & 1 ? 0x4432 : 0x4410) - (uint32_t)r;
                            if (k >= nr) continue;  // left out (n <= 65,534), or another round's
                            const int pick = 0x4440 + (b & 3);
                            uint32_t bit = b0 << __byte_perm(x0[b >> 2], 0, pick);
                            if (m > 1) bit |= b1 << __byte_perm(x1[b >> 2], 0, pick);
                            if (m > 2) bit |= b2 << __byte_perm(x2[b >> 2], 0, pick);
                            if (m > 3) bit |= b3 << __byte_perm(x3[b >> 2], 0, pick);
                            if (bit & ~mask[k]) atomicOr(&mask[k], bit);
                        }
                    }
                    __syncthreads();
                    int df[kPack] = {0, 0, 0, 0};  // (a - 1)(a_o - 1) summed over at most 40 strata per thread
                    for (int k = tid; k < (int)nr; k += kTestThreads) {
                        const uint32_t w = mask[k];
                        const int ac = (int)__ldcg(av + r + k);
#pragma unroll
                        for (int j = 0; j < kPack; ++j)
                            if (j < m) {
                                const uint32_t part = s_bits[j] == 32 ? w : (w >> s_shift[j]) & ((1u << s_bits[j]) - 1u);
                                df[j] += ac * (__popc(part) - 1);
                            }
                    }
#pragma unroll
                    for (int j = 0; j < kPack; ++j)
                        if (j < m) {
                            const int t = __reduce_add_sync(0xffffffffu, df[j]);
                            if (lane == 0 && t) atomicAdd(&s_df[j], (unsigned long long)t);
                        }
                    __syncthreads();
                }
            }
            if (warp < m) {  // a warp decides a test
                const int place = s_place[warp], item = a.lists[6 * a.list_cap + place] >> 1;
                const int4 r = s.item_ref[place];
                const long long df = (long long)s_df[warp];
                int dec = -1;
                if (n >= 0 && aoff >= 0 && r.y >= 0 && r.w >= 0 && s.node_n[r.y] >= 0 && s.pair_a[r.w] >= 0) {
                    const long long hs = s.pair_h[r.w] - s.pair_h[r.z] - s.node_h[r.y] + s.node_h[r.x];
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
                            if (dec >= 0 && lane == 0) atomicAdd(&a.stats[ST_RECHECK], 1ull);
                        }
                    }
                }
                if (lane == 0) {
                    if (dec >= 0) {
                        a.flag[item] = (uint8_t)dec;
                        atomicAdd(&a.stats[ST_LARGE], 1ull);
                    } else {
                        const int q = atomicAdd(&a.counters[C_TIER2], 1);
                        a.lists[2 * a.list_cap + q] = item;
                        atomicAdd(&a.stats[ST_BYTES_LARGE], (unsigned long long)S * (2 + d));
                    }
                }
            }
        }
        __syncthreads();
    }
}

}  // namespace fpgm
