// wp_khits.cu -- the reference's k-hit set without replaying its priority
// queue, one warp per read.
//
// KBest (kd-tree/k-best.h:26-42) takes the entries in the walk's order,
// pushes those below the farthest kept one (once the hits have reached k) and
// pops at most one per push, while the others' hits still reach k.  Let A_t(m)
// be the hits of the m nearest entries offered up to t.  After the fill the
// kept set is always the M_t nearest offered, and a push leaves M_t as it is
// when A_t(M) >= k and adds one otherwise, so
//
//     M_t = max(M_{t-1}, m_t),   m_t = the shortest prefix with hits >= k,
//
// (one push lengthens m_t by at most one) and the set that KBest ends with is
// the M nearest of all entries, M = max(t_f - 1, max over t >= t_f of m_t),
// t_f the number of entries that fill the first k hits.  The same maximum,
// taken over distance levels instead of times, is
//
//     M = max(t_f - 1, 1 + max over levels x with t(x) > t_f of n(x)),
//
// where t(x) is the place in the walk where the hits of the entries within x
// reach k and n(x) the number of entries within x before it.  Levels do not
// depend on one another, so nothing has to be kept in a queue: the kernel
//
//   1. walks the tree and lists, in walk order, the entries that can matter
//      (those within an upper bound of KBest's threshold, from a histogram of
//      the listed distances: 64 bins per octave),
//   2. sorts the list into finer bins, takes them in groups of about 96
//      entries and moves one group down and some places up the list together
//      (each step passes entries once, 32 at a time), which gives n between
//      the groups and, per group, an upper bound for the levels inside it,
//   3. looks inside the groups whose bound exceeds the maximum found, those with
//      the largest bounds first (their entries ranked by FP64 distance, a lane per
//      level of a block of up to 64), the CTA's warps that are between reads
//      helping: groups do not depend on one another, and one read can have 280 of
//      them where the mean is 30, and
//   4. ranks the bin that holds the M-th nearest entry, KBest's final top, and
//      writes the read's candidate list as the brute-force passes would (wp_nn.cu:
//      the entries up to the end of the top's distance bin, in tree order, by
//      slices), the M kept ones with their positions, the others as -1.  The votes
//      are added in groups of that list, so both routes give the same bits.
//
// Exactness.  Only ranks inside the groups of 3 and 4 need FP64 distances; an
// entry whose FP32 distance lies within its rounding error of a bin edge is
// put in its bin by its FP64 distance too, so the bins are exact.  Entries of
// equal distance in a ranked group (KBest's answer then depends on when they
// were refused), lists beyond the scratch and reads that are not finite are
// flagged and left to the replay (wp_kbest.cu).
//
// The walk screens 128 entries per step: counts of at most 15 dyes, two to a
// byte, transposed per 128 tree positions (a lane's 16-byte load brings 8
// coordinates of four entries), against the read rounded to 16 bits, as two
// 8-bit integer dot products (dp4a); the rounding is covered by a margin of
// TC (NC - 1) steps.
//
// Bound by the latency of a read's chain of instructions: 16 warps per SM (128
// registers each) issue one every 7 to 9 cycles, with L2 at 4 % of its peak
// (3,700 tiles of 128 entries screened, 25,000 of 470,000 entries listed per read
// at k = 10,000: 57 % of the cycles in the walk, 10 % in the groups).  4,000 reads
// against 946,000 tracks, k = 10,000: 27 ms, 36 with each group's levels followed
// one by one by the read's own warp (the slowest read's groups alone took 27),
// against 132 ms for the replay (20,000 pushes per read, one at a time, and its
// table look-ups of 48 coordinates for every entry met) and 41 ms for the
// brute-force passes that then collected the entries (the list holds them all);
// 2,000 reads against 70,000 tracks, k = 1,000: 0.83 ms against 4.1 and 4.0 ms.
// Whole calls of 2,000 and of 100 reads against 470,000 tracks by k, with the replay
// in brackets: 30,000 57 and 33 ms (230 and 173), 100,000 271 and 77 (535 and 409),
// 400,000 761 and 123 (1,628 and 808): no k of this range is better off with it.
// Tried and left out: integer sums in place of the FP64 ones in the groups, no
// faster (39.9 against 41.4 ms for the whole call); warps that start from the
// reads with the fewest dyes so as to help sooner, 1.55 against 1.67 ms in the
// second case and 43.6 against 39.9 in the first.
#include <cuda_runtime.h>
#include <float.h>
#include <math.h>
#include <stdint.h>

#include "wp_common.cuh"

#define KH_NB 1024     // distance bins: 16 octaves below the first leaf's farthest corner
#define KH_SH 17       // float bits >> 17: exponent and 6 mantissa bits
#define KH_WARPS 4     // warps per CTA
#define KH_RANK 8192   // most entries of a group that are ranked (a power of two)
#define KH_EPS 2e-6f   // bound of the FP32 distances' relative error (27 roundings, all terms >= 0)
#define KH_GRP 96      // entries per group of bins, about
#define KH_MAXG 1024   // groups
#define KH_LATE 15     // a wait ran out (the largest of a read's fatal codes)
#define KH_CROWD 9     // kh_group: the group cannot be taken in FP32 order
#define KH_WAIT 4000000  // most turns of a wait (0.2 to 1 us each)

struct KHSmem {
    unsigned cnt[KH_NB];   // entries per bin
    unsigned hit[KH_NB];   // hits per bin; after the walk, the end of each bin in `order`
    int qpos[64];          // screened entries waiting for their distances
    float4 q32[16];        // the read
};

// The list of one read and the state of the two moving pointers.
struct KHList {
    int2* ent;        // (tree position, hits) in walk order
    float* d;         // squared distance (FP32)
    uint16_t* bin;    // fine bin
    int2* order;      // (list index, hits) by fine bin
    uint16_t* rank;   // within a ranked group: the entry's place, farthest first
    int4* state;      // per group: pointer state above it, bound inside it
    int4* group;      // per group: lowest and highest bin, first place and end in `order`
    int* pick;        // the groups to look into, those with the largest bounds first
    long long* mem_d; // a ranked group's FP64 distances (as bits: they order alike)
    unsigned* mem_k;  // the same relative to the nearest, in 32 bits
    int2* sorted;     // its (list index, hits), farthest first
    int n;
};

__device__ __forceinline__ unsigned kh_sum(unsigned v) { return __reduce_add_sync(0xffffffffu, v); }

// Lower edge of bin b (base: the bin 0 in units of float bits >> KH_SH).
__device__ __forceinline__ float kh_edge(int base, int b) {
    const int v = base + b;
    return v <= 0 ? 0.f : __uint_as_float((unsigned)v << KH_SH);
}

__device__ __forceinline__ int kh_clamp_bin(float d, int base) {
    const int b = (int)(__float_as_uint(d) >> KH_SH) - base;
    return b < 0 ? 0 : (b > KH_NB - 1 ? KH_NB - 1 : b);
}

// FP32 squared distance from the per-read table sq32[i][n].
template <int DP>
__device__ __forceinline__ float kh_d32(const uint8_t* __restrict__ cnt, long p, const float* sq32, int NC, int TC) {
    const uint4* src = reinterpret_cast<const uint4*>(cnt + p * DP);
    float a0 = 0.f, a1 = 0.f;
#pragma unroll
    for (int i = 0; i < DP / 16; i++) {
        const uint4 v = __ldg(src + i);
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int j = 0; j < 16; j += 2) {
            const int d = 16 * i + j;
            if (d < TC) a0 += sq32[d * NC + (int)((w[j >> 2] >> (8 * (j & 3))) & 255u)];
            if (d + 1 < TC) a1 += sq32[(d + 1) * NC + (int)((w[(j + 1) >> 2] >> (8 * ((j + 1) & 3))) & 255u)];
        }
    }
    return a0 + a1;
}

// The 32 entries of the list around T, one per lane (most moves end where the
// last one did, so they are loaded once and not for each move).
struct KHWindow {
    int base, bin, hits, rank;
};

// Moves T up the list until the hits of the entries counted reach k: entries
// in bins below b, and with after >= 0 those of bins b .. b1 ranked after it.
// False if the list ends first.
__device__ __forceinline__ bool kh_advance(const KHList& L, KHWindow& w, int lane, int b, int b1, int after, int k,
                                           int& T, int& c, int& H) {
    while (H < k) {
        if (T >= L.n) return false;
        if (T - w.base >= 32) {
            w.base = T & ~31;
            const int i = w.base + lane;
            w.bin = 0xffff;
            w.hits = w.rank = 0;
            if (i < L.n) {
                w.bin = L.bin[i];
                w.hits = L.ent[i].y;
                if (after >= 0) w.rank = L.rank[i];
            }
        }
        const bool counted = lane >= T - w.base && (w.bin < b || (after >= 0 && w.bin <= b1 && w.rank > after));
        int s = counted ? w.hits : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += t;
        }
        const unsigned in = __ballot_sync(0xffffffffu, counted);
        const unsigned hit = __ballot_sync(0xffffffffu, H + s >= k);
        if (hit) {
            const int l = __ffs(hit) - 1;
            T = w.base + l + 1;
            H += __shfl_sync(0xffffffffu, s, l);
            c += __popc(in & (0xffffffffu >> (31 - l)));
            return true;
        }
        H += __shfl_sync(0xffffffffu, s, 31);
        c += __popc(in);
        T = min(w.base + 32, L.n);
    }
    return true;
}

// FP64 squared distance as LeafNode::consider sums it, from the read's table
// sq64[i][n] = (q_i - coordinate(n))^2 (a third of the FP64 operations).
template <int DP>
__device__ __forceinline__ double kh_d64(const uint8_t* __restrict__ cnt, long p, const double* sq64, int NC, int TC) {
    const uint8_t* row = cnt + p * DP;
    double acc = 0.0;
    int i = 0;
    for (; i + 3 < TC; i += 4) {
        const uint32_t w = *reinterpret_cast<const uint32_t*>(row + i);
        const double* s = sq64 + i * NC;
        acc = __dadd_rn(acc, __dadd_rn(__dadd_rn(__dadd_rn(s[w & 255u], s[NC + ((w >> 8) & 255u)]),
                                                 s[2 * NC + ((w >> 16) & 255u)]),
                                       s[3 * NC + (w >> 24)]));
    }
    for (; i < TC; i++) acc = __dadd_rn(acc, sq64[i * NC + row[i]]);
    return acc;
}

// FP64 distances of the m entries from `start` of L.order into mem_d.
template <int DP>
__device__ __forceinline__ void kh_bin_d64(const KHArgs& a, const KHList& L, int lane, int start, int m,
                                           const double* sq64) {
    for (int j = lane; j < m; j += 32)
        L.mem_d[j] =
            __double_as_longlong(kh_d64<DP>(a.cnt, L.ent[L.order[start + j].x].x, sq64, a.NC, a.TC));
    __syncwarp();
}

// The m entries of mem_d ranked, farthest first: f(j, place) for each of a
// lane's entries j.  False if two are equal.  The distances' bits are compared
// as integers (this GPU's FP64 pipe takes 16 cycles to compare a warp), first
// by 32 bits below their common range: places that are all different add up
// to m (m - 1) / 2, and only if they don't are the full 64 bits compared.
template <class F>
__device__ __forceinline__ bool kh_rank(const KHList& L, int lane, int m, F f) {
    long long lo = 0x7fffffffffffffffll, hi = 0;
    for (int j = lane; j < m; j += 32) {
        const long long v = L.mem_d[j];
        lo = min(lo, v);
        hi = max(hi, v);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    const int sh = max(0, 32 - __clzll(hi - lo));
    for (int j = lane; j < m; j += 32) L.mem_k[j] = (unsigned)((L.mem_d[j] - lo) >> sh);
    __syncwarp();
    for (int wide = 0; wide < 2; wide++) {
        unsigned sum = 0;
        for (int j0 = 0; j0 < m; j0 += 128) {
            int place[4] = {0, 0, 0, 0};
            if (!wide) {
                unsigned d[4];
#pragma unroll
                for (int u = 0; u < 4; u++) d[u] = j0 + 32 * u + lane < m ? L.mem_k[j0 + 32 * u + lane] : 0xffffffffu;
#pragma unroll 8
                for (int v = 0; v < m; v++) {
                    const unsigned dv = L.mem_k[v];
#pragma unroll
                    for (int u = 0; u < 4; u++) place[u] += dv > d[u] ? 1 : 0;
                }
            } else {
                long long d[4];
#pragma unroll
                for (int u = 0; u < 4; u++)
                    d[u] = j0 + 32 * u + lane < m ? L.mem_d[j0 + 32 * u + lane] : 0x7fffffffffffffffll;
                for (int v = 0; v < m; v++) {
                    const long long dv = L.mem_d[v];
#pragma unroll
                    for (int u = 0; u < 4; u++) place[u] += dv > d[u] ? 1 : 0;
                }
            }
#pragma unroll
            for (int u = 0; u < 4; u++)
                if (j0 + 32 * u + lane < m) {
                    sum += (unsigned)place[u];
                    f(j0 + 32 * u + lane, place[u]);
                }
        }
        if (kh_sum(sum) == (unsigned)m * (unsigned)(m - 1) / 2u) return true;
    }
    return false;
}

// The list of warp gw of the grid, with the scratch of warp own.
__device__ __forceinline__ KHList kh_list(const KHArgs& a, long gw, long own) {
    KHList L;
    L.ent = a.ent + gw * a.cap;
    L.d = a.d + gw * a.cap;
    L.bin = a.bin + gw * a.cap;
    L.order = a.order + gw * a.cap;
    L.rank = a.rank + gw * a.cap;
    L.state = a.state + gw * 3 * KH_MAXG;
    L.group = L.state + KH_MAXG;
    L.pick = reinterpret_cast<int*>(L.state + 2 * KH_MAXG);
    L.mem_d = a.mem_d + own * KH_RANK;
    L.mem_k = a.mem_k + own * KH_RANK;
    L.sorted = a.sorted + own * KH_RANK;
    L.n = 0;
    return L;
}

// Looks inside group g of warp gw's list of n (its levels' n, from the state
// above it): the larger of M and the largest found, or minus a fatal code; KH_CROWD
// if more neighbours than a block takes lie within the FP32 error of one another.
// EXACT: for a group that came to that, in the order of the FP64 distances (sets
// dense at the top's distance: 9 of 150 reads at k = 200,000 of 470,000 tracks).
template <int DP, bool EXACT>
__device__ __noinline__ int kh_group(const KHArgs& a, long gw, long own, int n, int lane, int g, int tf, int k,
                                     const double* sq64, int M) {
    KHList L = kh_list(a, gw, own);
    L.n = n;
    const int4 st = L.state[g];
    int fatal = 0;
    KHWindow win = {-64, 0, 0, 0};
    const int4 gr = L.group[g];
    const int m = gr.w - gr.z;
    if (m > KH_RANK) return -5;
    if constexpr (EXACT) {
        kh_bin_d64<DP>(a, L, lane, gr.z, m, sq64);
    } else {
        // the group by FP32 distance (equal ones in any order)
        for (int j = lane; j < m; j += 32)
            L.mem_d[j] = (long long)__float_as_uint(L.d[L.order[gr.z + j].x]) * KH_RANK + j;
        __syncwarp();
    }
    const bool distinct = kh_rank(L, lane, m, [&](int j, int place) {
        const int2 x = L.order[gr.z + j];
        L.sorted[place] = x;
        L.rank[x.x] = (uint16_t)place;
    });
    if (EXACT && !distinct) return -6;
    __syncwarp();
    int Tx = st.x, cx = st.y, Hx = st.z;
    // blocks of up to 64 levels, cut where neighbours differ by more
    // than the FP32 error: n between the blocks and a bound inside,
    // as for the groups
    for (int j0 = 0; j0 < m && !fatal;) {
        int2 x[2];
        int len = 0;
        {
            float d[2];
            unsigned cut[2];
#pragma unroll
            for (int u = 0; u < 2; u++) {
                const int j = j0 + 32 * u + lane;
                x[u] = j < m ? L.sorted[j] : make_int2(0x7fffffff, 0);
                d[u] = j < m ? L.d[x[u].x] : 0.f;
            }
#pragma unroll
            for (int u = 0; u < 2; u++) {
                // the cut after this entry
                const int j = j0 + 32 * u + lane;
                const float next = u == 0 ? __shfl_sync(0xffffffffu, lane == 0 ? d[1] : d[0], (lane + 1) & 31)
                                          : __shfl_down_sync(0xffffffffu, d[1], 1);
                cut[u] = __ballot_sync(0xffffffffu, j == m - 1 || (j < m - 1 && (u == 0 || lane < 31) &&
                                                                   d[u] * (1.f - KH_EPS) > next * (1.f + KH_EPS)));
            }
            len = EXACT ? min(64, m - j0) : cut[0] ? 32 - __clz(cut[0]) : (cut[1] ? 32 + __ffs(cut[1]) : 0);
        }
        if (!EXACT && len == 0) {
            fatal = KH_CROWD;
            break;
        }
#pragma unroll
        for (int u = 0; u < 2; u++)
            if (32 * u + lane >= len) x[u] = make_int2(0x7fffffff, 0);
        const unsigned gone = kh_sum((x[0].x < Tx ? 1u : 0u) + (x[1].x < Tx ? 1u : 0u));
        int T1 = Tx, c1 = cx - (int)gone,
            H1 = Hx - (int)kh_sum((x[0].x < Tx ? (unsigned)x[0].y : 0u) + (x[1].x < Tx ? (unsigned)x[1].y : 0u));
        const bool reached = kh_advance(L, win, lane, gr.x, gr.y, j0 + len - 1, k, T1, c1, H1);
        const int lim = reached ? T1 - 1 : n;
        const int lt = (int)kh_sum((x[0].x < lim ? 1u : 0u) + (x[1].x < lim ? 1u : 0u));
        const int bound = !reached ? c1 + lt + 1 : (T1 > tf ? c1 + lt : -1);
        if (bound > M) {
            // level by level, by FP64 distance, a lane per level (two of them if
            // the block has more than 32).  A level's own entry and the farther
            // ones of the block are out.  The distances as 31-bit keys (the bits
            // below their common range, plus 1); only if two of those are equal
            // are the full 64 bits ranked.
            long long dd[2] = {0, 0};
            unsigned key[2] = {0u, 0u};
            {
                long long lo = 0x7fffffffffffffffll, hi = 0;
#pragma unroll
                for (int u = 0; u < 2; u++)
                    if (32 * u + lane < len) {
                        dd[u] = __double_as_longlong(kh_d64<DP>(a.cnt, L.ent[x[u].x].x, sq64, a.NC, a.TC));
                        lo = min(lo, dd[u]);
                        hi = max(hi, dd[u]);
                    }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
                    hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
                }
                const int sh = max(0, 33 - __clzll(hi - lo));
#pragma unroll
                for (int u = 0; u < 2; u++)
                    if (32 * u + lane < len) key[u] = (unsigned)((dd[u] - lo) >> sh) + 1u;
            }
            // the state at each level's start: what the block loses to it taken out
            int Hl[2], cl[2], Tl[2];
            bool need[2];
            for (int wide = 0; wide < 2; wide++) {
                unsigned gone_h[2] = {0u, 0u}, gone_c[2] = {0u, 0u}, same = 0u;
                const int in0 = x[0].x < Tx ? x[0].y : -1, in1 = x[1].x < Tx ? x[1].y : -1;
                for (int v = 0; v < len; v++) {
                    const unsigned kv = __shfl_sync(0xffffffffu, v < 32 ? key[0] : key[1], v & 31);
                    const int hv = __shfl_sync(0xffffffffu, v < 32 ? in0 : in1, v & 31);
#pragma unroll
                    for (int u = 0; u < 2; u++) {
                        const bool out = kv >= key[u];
                        same += kv == key[u] ? 1u : 0u;
                        if (out && hv >= 0) {
                            gone_h[u] += (unsigned)hv;
                            gone_c[u]++;
                        }
                    }
                }
#pragma unroll
                for (int u = 0; u < 2; u++) {
                    Hl[u] = Hx - (int)gone_h[u];
                    cl[u] = cx - (int)gone_c[u];
                    Tl[u] = Tx;
                    need[u] = 32 * u + lane < len && Hl[u] < k;
                }
                // each key meets itself and no other (a lane without a level has key
                // 0, no level has)
                if (kh_sum(same) == (unsigned)len) break;
                if (wide) {
                    fatal = 6;
                    break;
                }
                // equal keys: the ranks of the full distances in their place
                unsigned nearer[2] = {0u, 0u};
                for (int v = 0; v < len; v++) {
                    const long long dv = __shfl_sync(0xffffffffu, v < 32 ? dd[0] : dd[1], v & 31);
#pragma unroll
                    for (int u = 0; u < 2; u++) nearer[u] += dv < dd[u] ? 1u : 0u;
                }
#pragma unroll
                for (int u = 0; u < 2; u++)
                    if (32 * u + lane < len) key[u] = nearer[u] + 1u;
            }
            if (fatal) break;
            // the list from Tx until each level's hits reach k again, all levels
            // together: an entry nearer than the block counts for all of them (key 0),
            // one of the block for the levels farther than it
            const int end = reached ? T1 : n;
            for (int i0 = Tx & ~31; i0 < end; i0 += 32) {
                const int i = i0 + lane;
                int place = -1, h = 0;
                if (i >= Tx && i < end) {
                    const int bi = L.bin[i];
                    if (bi < gr.x) {
                        place = 64;
                    } else if (bi <= gr.y) {
                        const int rk = (int)L.rank[i] - j0;
                        place = rk < 0 ? -1 : (rk < len ? rk : 64);
                    }
                    if (place >= 0) h = L.ent[i].y;
                }
                unsigned ke = __shfl_sync(0xffffffffu, key[0], place & 31);
                const unsigned k1 = __shfl_sync(0xffffffffu, key[1], place & 31);
                if (place >= 32) ke = place == 64 ? 0u : k1;
                unsigned todo = __ballot_sync(0xffffffffu, place >= 0);
                while (todo) {
                    const int l = __ffs(todo) - 1;
                    todo &= todo - 1;
                    const unsigned kv = __shfl_sync(0xffffffffu, ke, l);
                    const int hl = __shfl_sync(0xffffffffu, h, l);
#pragma unroll
                    for (int u = 0; u < 2; u++)
                        if (need[u] && kv < key[u]) {
                            Hl[u] += hl;
                            cl[u]++;
                            if (Hl[u] >= k) {
                                need[u] = false;
                                Tl[u] = i0 + l + 1;
                            }
                        }
                }
                if (!__any_sync(0xffffffffu, need[0] || need[1])) break;
            }
            int most = -1;
#pragma unroll
            for (int u = 0; u < 2; u++)
                if (32 * u + lane < len) most = max(most, need[u] ? cl[u] + 1 : (Tl[u] > tf ? cl[u] : -1));
            M = max(M, __reduce_max_sync(0xffffffffu, most));
        }
        if (!reached) break;
        if (T1 > tf) M = max(M, c1);
        Tx = T1;
        cx = c1;
        Hx = H1;
        j0 += len;
    }
    return fatal ? -fatal : M;
}

// The np groups picked of warp gw's list again, by itself and in FP64 order: the
// largest n found, or minus a fatal code.
template <int DP>
__device__ __noinline__ int kh_exact_groups(const KHArgs& a, long gw, int lane, int np, int tf, int n, int k,
                                            const double* sq64, int M) {
    const int4* state = a.state + gw * 3 * KH_MAXG;
    const int* pick = reinterpret_cast<const int*>(state + 2 * KH_MAXG);
    for (int i = 0; i < np && state[pick[i]].w > M; i++) {
        const int found = kh_group<DP, true>(a, gw, gw, n, lane, pick[i], tf, k, sq64, M);
        if (found < 0) return found;
        M = found;
    }
    return M;
}

// One warp's groups, for the CTA's warps to take (kh_help).
struct KHShare {
    int open;   // groups can be taken
    int busy;   // other warps looking or at work
    int np, next, fatal, M, tf, n;
};

// Takes groups of the read that sh describes (its list is warp gw's) until none
// is left; own: the calling warp, for its scratch.
template <int DP>
__device__ __forceinline__ void kh_help(const KHArgs& a, long own, int lane, KHShare* sh, long gw,
                                        const double* sq64, int k) {
    const int* pick = reinterpret_cast<const int*>(a.state + gw * 3 * KH_MAXG + 2 * KH_MAXG);
    const int np = *(volatile int*)&sh->np, tf = *(volatile int*)&sh->tf, n = *(volatile int*)&sh->n;
    for (;;) {
        int g = 0;
        if (lane == 0) g = atomicAdd(&sh->next, 1);
        g = __shfl_sync(0xffffffffu, g, 0);
        if (g >= np) break;
        const int M = __shfl_sync(0xffffffffu, *(volatile int*)&sh->M, 0);
        g = pick[g];
        if (a.state[gw * 3 * KH_MAXG + g].w <= M) break;  // nor do the rest exceed it
        const int found = kh_group<DP, false>(a, gw, own, n, lane, g, tf, k, sq64, M);
        if (lane == 0) {
            if (found > M) atomicMax(&sh->M, found);
            if (found < 0) atomicMax(&sh->fatal, -found);
        }
        __syncwarp();
        if (found < 0) break;
    }
}

// The slots nobody has taken yet: left to the replay.
__device__ __noinline__ void kh_drain(const KHArgs& a) {
    for (int i = atomicAdd(a.next, 1); i < a.Rc; i = atomicAdd(a.next, 1)) a.kept_n[a.q0 + a.Rc - 1 - i] = -1;
}

template <int DP>
__global__ void __launch_bounds__(KH_WARPS * 32, 4) wp_khits_kernel(const __grid_constant__ KHArgs a) {
    extern __shared__ __align__(16) unsigned char kh_smem[];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const unsigned below = (1u << lane) - 1u;
    const size_t tab_bytes = ((size_t)a.TC * a.NC * (sizeof(double) + sizeof(float)) + 15) / 16 * 16;
    const size_t stack_bytes = ((size_t)a.stack_cap * (sizeof(int) + sizeof(double)) + 15) / 16 * 16;
    unsigned char* mine = kh_smem + (sizeof(KHSmem) + tab_bytes + stack_bytes) * wib;
    KHSmem* sm = reinterpret_cast<KHSmem*>(mine);
    double* sq64 = reinterpret_cast<double*>(mine + sizeof(KHSmem));
    float* sq32 = reinterpret_cast<float*>(sq64 + a.TC * a.NC);
    double* s_plane = reinterpret_cast<double*>(mine + sizeof(KHSmem) + tab_bytes);
    int* s_node = reinterpret_cast<int*>(s_plane + a.stack_cap);
    const long gw = (long)blockIdx.x * KH_WARPS + wib;
    KHList L = kh_list(a, gw, gw);
    __shared__ KHShare share[KH_WARPS];
    __shared__ int leaving;  // warps without further reads
    KHShare* const sh = share + wib;
    if (lane == 0) {
        sh->open = sh->busy = 0;
        if (wib == 0) leaving = 0;
    }
    __syncthreads();
    int2* seg = a.seg + gw * KH_MAXG;
    const int k = (int)a.k;

    // helps the CTA's other warps with the groups they have left
    auto help = [&]() {
        for (int v = 1; v < KH_WARPS; v++) {
            const int o = (wib + v) % KH_WARPS;
            KHShare* const so = share + o;
            int go = 0;
            if (lane == 0 && *(volatile int*)&so->open) {
                atomicAdd(&so->busy, 1);
                __threadfence_block();
                go = *(volatile int*)&so->open;
                if (!go) atomicSub(&so->busy, 1);
            }
            if (!__shfl_sync(0xffffffffu, go, 0)) continue;
            __threadfence_block();
            kh_help<DP>(a, gw, lane, so, gw - wib + o,
                        reinterpret_cast<const double*>(kh_smem + (sizeof(KHSmem) + tab_bytes + stack_bytes) * o +
                                                        sizeof(KHSmem)),
                        k);
            __threadfence_block();
            __syncwarp();
            if (lane == 0) atomicSub(&so->busy, 1);
        }
    };

    for (;;) {
        help();
        int slot = 0;
        if (lane == 0) slot = atomicAdd(a.next, 1);
        slot = __shfl_sync(0xffffffffu, slot, 0);
        if (slot >= a.Rc) break;
        // from the last (the reads are sorted, those with the most dyes, whose walks
        // are the longest, last) to the first
        slot = a.q0 + a.Rc - 1 - slot;
        const int r = a.qperm ? a.qperm[slot] : slot;
        const double* q64 = a.rads + (long)r * a.TC;
        // ---- the read: distance table, 16-bit rounding for the screen
        for (int i = a.TC + lane; i < DP; i += 32) reinterpret_cast<float*>(sm->q32)[i] = 0.f;
        float amax = 0.f, qn = 0.f;
        bool finite = true;
        for (int i = lane; i < a.TC; i += 32) {
            const float v = (float)q64[i];
            const float w = (float)(q64[i] * a.ctab[(i % a.C) * a.NC + 1]);
            reinterpret_cast<float*>(sm->q32)[i] = v;
            finite = finite && isfinite(v) && isfinite(w) && fabsf(v) < 1e6f && fabsf(w) < 1e6f;
            amax = fmaxf(amax, fabsf(w));
            qn = fmaf(v, v, qn);
        }
        for (int o = 16; o > 0; o >>= 1) {
            amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
            qn += __shfl_xor_sync(0xffffffffu, qn, o);
        }
        int fatal = __all_sync(0xffffffffu, finite) ? 0 : 1;
        for (int i = lane; i < a.TC * a.NC; i += 32) {
            const int dim = i / a.NC, n = i % a.NC;
            const double x = __dsub_rn(q64[dim], a.ctab[(dim % a.C) * a.NC + n]);
            const double s = __dmul_rn(x, x);
            sq64[i] = s;
            sq32[i] = (float)s;
        }
        const float step = fmaxf(amax, 1e-20f) * (1.f / 32000.f);
        int qh[DP / 4], ql[DP / 4];
#pragma unroll
        for (int g = 0; g < DP / 4; g++) {
            unsigned hi = 0u, lo = 0u;
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const int i = 4 * g + u;
                int W = 0;
                if (i < a.TC && !fatal) W = __float2int_rn((float)(q64[i] * a.ctab[(i % a.C) * a.NC + 1]) / step);
                const int l = ((W + 128) & 255) - 128;
                hi |= ((unsigned)((W - l) >> 8) & 255u) << (8 * u);
                lo |= ((unsigned)l & 255u) << (8 * u);
            }
            qh[g] = (int)hi;
            ql[g] = (int)lo;
        }
        const float slack = 1.02f * step * (float)(a.TC * (a.NC - 1)) - qn * (1.f - 1e-5f);
        for (int i = lane; i < KH_NB; i += 32) sm->cnt[i] = sm->hit[i] = 0u;
        if (lane == 0) {
            s_node[0] = 0;
            s_plane[0] = -1.0;
        }
        __syncwarp();

        // ---- 1. the walk: depth first, nearer child first
        int sp = 1, n = 0, tf = 0, base = 0, nseg = 0;
        bool fill = true, have_base = false;
        unsigned S = 0;                      // hits listed (until the fill ends)
        int Htf = 0;                         // hits of the first t_f entries
        int bh = KH_NB, Cb = 0, bc = KH_NB, Cc = 0, mub = 0, ub = KH_NB - 1;
        long long Sb = 0;                    // hits in bins below bh
        // entries are listed up to `reach`: KBest's threshold is at most the upper
        // edge of bin ub, and the candidate list ends within 1/16 octave and the
        // binning distance's margins beyond its last value
        float reach = INFINITY, rhs = INFINITY;
        while (sp > 0 && !fatal) {
            sp--;
            int node = s_node[sp];
            const double plane = s_plane[sp];
            __syncwarp();
            if (plane > (double)reach) continue;
            KDNode nd = a.nodes[node];
            while (!nd.leaf) {
                const double qv = q64[nd.s];
                int near, far;
                double dist;
                if (qv < nd.split) {
                    near = nd.left;
                    far = nd.right;
                    dist = nd.min_right - qv;
                } else {
                    near = nd.right;
                    far = nd.left;
                    dist = qv - nd.max_left;
                }
                if (sp >= a.stack_cap) {
                    fatal = 2;
                    break;
                }
                if (lane == 0) {
                    s_node[sp] = far;
                    s_plane[sp] = __dmul_rn(dist, dist);
                }
                __syncwarp();
                sp++;
                node = near;
                nd = a.nodes[node];
            }
            if (fatal) break;
            {
                // the leaf's box: nearest point, and farthest corner for the bins' origin
                float g2 = 0.f, f2 = 0.f;
                for (int i = lane; i < a.TC; i += 32) {
                    const float lo = a.llo[(long)node * DP + i], hi = a.lhi[(long)node * DP + i];
                    const float qq = (float)q64[i];
                    const float g = fmaxf(fmaxf(lo - qq, qq - hi), 0.f);
                    const float f = fmaxf(fabsf(qq - lo), fabsf(hi - qq));
                    g2 = fmaf(g, g, g2);
                    f2 = fmaf(f, f, f2);
                }
                for (int o = 16; o > 0; o >>= 1) {
                    g2 += __shfl_xor_sync(0xffffffffu, g2, o);
                    f2 += __shfl_xor_sync(0xffffffffu, f2, o);
                }
                if (!have_base) {
                    have_base = true;
                    base = (int)(__float_as_uint(f2 * (1.f + 1e-4f)) >> KH_SH) - (KH_NB - 1);
                }
                if (!fill && g2 > reach * (1.f + 1e-4f) + 1e-3f) continue;
            }
            const int n_leaf = n;
            const int g_lo = nd.begin >> 7, g_hi = (nd.end - 1) >> 7;
            int qn_ = 0;
            uint4 w[DP / 8];
            float en[4];
            {
                const uint4* src = a.nib + (long)g_lo * (DP / 8) * 32 + lane;
#pragma unroll
                for (int j = 0; j < DP / 8; j++) w[j] = __ldg(src + j * 32);
#pragma unroll
                for (int u = 0; u < 4; u++) en[u] = __ldg(a.enorm + (long)g_lo * 128 + 32 * u + lane);
            }
            for (int g = g_lo; g <= g_hi && !fatal; g++) {
                uint4 wn[DP / 8];
                float en_n[4];
                {
                    const int g1 = min(g + 1, g_hi);
                    const uint4* src = a.nib + (long)g1 * (DP / 8) * 32 + lane;
#pragma unroll
                    for (int j = 0; j < DP / 8; j++) wn[j] = __ldg(src + j * 32);
#pragma unroll
                    for (int u = 0; u < 4; u++) en_n[u] = __ldg(a.enorm + (long)g1 * 128 + 32 * u + lane);
                }
                int dh[4] = {0, 0, 0, 0}, dl[4] = {0, 0, 0, 0};
#pragma unroll
                for (int j = 0; j < DP / 8; j++) {
                    const uint32_t v[4] = {w[j].x, w[j].y, w[j].z, w[j].w};
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        const int x = (int)(v[u] & 0x0f0f0f0fu), y = (int)((v[u] >> 4) & 0x0f0f0f0fu);
                        dh[u] = __dp4a(qh[2 * j], x, dh[u]);
                        dl[u] = __dp4a(ql[2 * j], x, dl[u]);
                        dh[u] = __dp4a(qh[2 * j + 1], y, dh[u]);
                        dl[u] = __dp4a(ql[2 * j + 1], y, dl[u]);
                    }
                }
                float lhs[4];
#pragma unroll
                for (int u = 0; u < 4; u++)
                    lhs[u] = fmaf((float)(256 * dh[u] + dl[u]), -2.f * step, en[u] * (1.f - 1e-5f));
#pragma unroll
                for (int j = 0; j < DP / 8; j++) w[j] = wn[j];
#pragma unroll
                for (int u = 0; u < 4; u++) en[u] = en_n[u];
#pragma unroll 1
              for (int u = 0; u < 4; u++) {
                const float lu = u == 0 ? lhs[0] : (u == 1 ? lhs[1] : (u == 2 ? lhs[2] : lhs[3]));
                const int p = g * 128 + 32 * u + lane;
                const bool cand = p >= nd.begin && p < nd.end && (fill || lu <= rhs);
                const bool last = g == g_hi && u == 3;
                const unsigned m = __ballot_sync(0xffffffffu, cand);
                if (m == 0u && !last) continue;
                if (cand) sm->qpos[qn_ + __popc(m & below)] = p;
                qn_ += __popc(m);
                __syncwarp();
                while (qn_ >= 32 || (last && qn_ > 0)) {
                    const int cntb = min(32, qn_);
                    int pos = 0, h = 0, b = KH_NB;
                    float d = 0.f;
                    if (lane < cntb) {
                        pos = sm->qpos[lane];
                        h = a.hits[pos];
                        d = kh_d32<DP>(a.cnt, pos, sq32, a.NC, a.TC);
                        // within the FP32 error of a bin edge: the FP64 distance decides
                        if ((__float_as_uint(d * (1.f - KH_EPS)) >> KH_SH) != (__float_as_uint(d * (1.f + KH_EPS)) >> KH_SH))
                            d = __double2float_rd(kh_d64<DP>(a.cnt, pos, sq64, a.NC, a.TC));
                        b = kh_clamp_bin(d, base);
                    }
                    int rest = 0;
                    if (lane + cntb < qn_) rest = sm->qpos[lane + cntb];
                    __syncwarp();
                    if (lane + cntb < qn_) sm->qpos[lane] = rest;
                    qn_ -= cntb;
                    const bool keep = lane < cntb && (fill || d <= reach);
                    const unsigned km = __ballot_sync(0xffffffffu, keep);
                    if (km == 0u) {
                        __syncwarp();
                        continue;
                    }
                    const int at = n + __popc(km & below);
                    if (n + 32 > a.cap) {
                        fatal = 3;
                        break;
                    }
                    if (keep) {
                        L.ent[at] = make_int2(pos, h);
                        L.d[at] = d;
                        atomicAdd(&sm->cnt[b], 1u);
                        atomicAdd(&sm->hit[b], (unsigned)h);
                    }
                    n += __popc(km);
                    __syncwarp();
                    if (fill) {
                        int s = keep ? h : 0;
#pragma unroll
                        for (int o = 1; o < 32; o <<= 1) {
                            const int v = __shfl_up_sync(0xffffffffu, s, o);
                            if (lane >= o) s += v;
                        }
                        const unsigned full = __ballot_sync(0xffffffffu, (long long)S + s >= k);
                        if (full) {
                            const int l = __ffs(full) - 1;
                            tf = __shfl_sync(0xffffffffu, at, l) + 1;
                            Htf = (int)S + __shfl_sync(0xffffffffu, s, l);
                            fill = false;
                            mub = n;
                            Sb = (long long)S + __shfl_sync(0xffffffffu, s, 31);
                            Cb = Cc = n;
                        } else {
                            S += (unsigned)__shfl_sync(0xffffffffu, s, 31);
                            continue;
                        }
                    } else {
                        Sb += kh_sum(keep && b < bh ? (unsigned)h : 0u);
                        Cb += __popc(__ballot_sync(0xffffffffu, keep && b < bh));
                        Cc += __popc(__ballot_sync(0xffffffffu, keep && b < bc));
                        // no prefix since the last batch was longer than the
                        // entries now within the bin that then held it
                        mub = max(mub, Cb + (int)sm->cnt[bh]);
                    }
                    // bh: the bin where the hits reach k; bc: where the count
                    // reaches the longest prefix so far (its upper bound)
                    while (Sb >= k) {
                        bh--;
                        Sb -= (long long)sm->hit[bh];
                        Cb -= (int)sm->cnt[bh];
                    }
                    while (Cc >= mub) {
                        bc--;
                        Cc -= (int)sm->cnt[bc];
                    }
                    while (Cc + (int)sm->cnt[bc] < mub) {
                        Cc += (int)sm->cnt[bc];
                        bc++;
                    }
                    const int nub = max(bh, bc);
                    if (nub != ub) {
                        ub = nub;
                        reach = ub == KH_NB - 1 ? INFINITY
                                                : fmaf(1.05f, kh_edge(base, ub + 1), fmaf(2e-5f, qn, 2e-3f));
                        rhs = reach + slack;
                    }
                }
                if (fatal) break;
              }
            }
            if (n > n_leaf) {
                // the leaf's part of the list
                if (nseg == KH_MAXG) fatal = fatal ? fatal : 10;
                else if (lane == 0) seg[nseg] = make_int2(nd.begin, n_leaf);
                nseg++;
            }
        }
        if (!fatal && fill) fatal = 4;  // the hits never reached k: not for this kernel

        int M = 0;
        if (!fatal) {
            L.n = n;
            // ---- 2. the list by finer bins: the coarse bins from bh (where the
            // hits reach k) up to the highest listed, split as far as they fit;
            // bin 0 holds everything below
            int hb = 0;
            for (int g = KH_NB / 32 - 1; g >= 0; g--) {
                const unsigned some = __ballot_sync(0xffffffffu, sm->cnt[g * 32 + lane] != 0u);
                if (some) {
                    hb = g * 32 + 31 - __clz(some);
                    break;
                }
            }
            int fs = 0;
            while (fs < 5 && ((hb - bh + 1) << (fs + 1)) <= KH_NB - 1) fs++;
            const int fsh = KH_SH - fs, fbase = ((base + bh) << fs) - 1;
            __syncwarp();
            for (int i = lane; i < KH_NB; i += 32) sm->cnt[i] = 0u;
            __syncwarp();
            for (int i = lane; i < n; i += 32) {
                float d = L.d[i];
                if ((__float_as_uint(d * (1.f - KH_EPS)) >> fsh) != (__float_as_uint(d * (1.f + KH_EPS)) >> fsh))
                    d = __double2float_rd(kh_d64<DP>(a.cnt, L.ent[i].x, sq64, a.NC, a.TC));
                const int f = (int)(__float_as_uint(d) >> fsh) - fbase;
                const int fb = f < 0 ? 0 : (f > KH_NB - 1 ? KH_NB - 1 : f);
                L.bin[i] = (uint16_t)fb;
                atomicAdd(&sm->cnt[fb], 1u);
            }
            __syncwarp();
            {
                unsigned part = 0;
                for (int i = 0; i < KH_NB / 32; i++) part += sm->cnt[lane * (KH_NB / 32) + i];
                unsigned s = part;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const unsigned v = __shfl_up_sync(0xffffffffu, s, o);
                    if (lane >= o) s += v;
                }
                s -= part;
                for (int i = 0; i < KH_NB / 32; i++) {
                    const int b = lane * (KH_NB / 32) + i;
                    sm->hit[b] = s;
                    s += sm->cnt[b];
                }
            }
            __syncwarp();
            for (int i = lane; i < n; i += 32)
                L.order[atomicAdd(&sm->hit[L.bin[i]], 1u)] = make_int2(i, L.ent[i].y);
            __syncwarp();
            // down the groups, up the list
            const int gsize = max(KH_GRP, n / (KH_MAXG / 2) + 1);
            int T = tf, c = tf, H = Htf, ng = 0, e = n;
            M = tf - 1;
            KHWindow win = {-64, 0, 0, 0};
            while (e > 0) {
                // bin 0 (its hits are fewer than k, so the moves end above it) joins no group
                const int end0 = (int)sm->hit[0];
                const int b = L.bin[L.order[max(e - gsize, e > end0 ? end0 : 0)].x], b1 = L.bin[L.order[e - 1].x];
                const int start = (int)(sm->hit[b] - sm->cnt[b]);
                // a lane's first four entries stay in registers for the second pass
                int2 x[4];
                unsigned rc = 0, rh = 0;
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const int j = start + 32 * u + lane;
                    x[u] = j < e ? L.order[j] : make_int2(0x7fffffff, 0);
                }
#pragma unroll
                for (int u = 0; u < 4; u++)
                    if (x[u].x < T) {
                        rc++;
                        rh += (unsigned)x[u].y;
                    }
                for (int j = start + 128 + lane; j < e; j += 32) {
                    const int2 y = L.order[j];
                    if (y.x < T) {
                        rc++;
                        rh += (unsigned)y.y;
                    }
                }
                int T1 = T, c1 = c - (int)kh_sum(rc), H1 = H - (int)kh_sum(rh);
                const bool reached = kh_advance(L, win, lane, b, b, -1, k, T1, c1, H1);
                unsigned lt = 0;
                const int lim = reached ? T1 - 1 : n;
#pragma unroll
                for (int u = 0; u < 4; u++) lt += x[u].x < lim ? 1u : 0u;
                for (int j = start + 128 + lane; j < e; j += 32) lt += L.order[j].x < lim ? 1u : 0u;
                lt = kh_sum(lt);
                const int bound = !reached ? c1 + (int)lt + 1 : (T1 > tf ? c1 + (int)lt : -1);
                if (lane == 0) {
                    L.state[ng] = make_int4(T, c, H, bound);
                    L.group[ng] = make_int4(b, b1, start, e);
                }
                ng++;
                if (!reached) break;
                if (T1 > tf) M = max(M, c1);
                T = T1;
                c = c1;
                H = H1;
                e = start;
            }
            __syncwarp();
            // ---- 3. the groups whose bound exceeds the maximum, those with the
            // largest bounds first (they raise the maximum past most others' bounds),
            // with the CTA's other warps
            int np = 0;
            for (int g0 = 0; g0 < ng; g0 += 32) {
                const int bound = g0 + lane < ng ? L.state[g0 + lane].w : -1;
                const unsigned in = __ballot_sync(0xffffffffu, bound > M);
                if (bound > M) {
                    L.mem_k[np + __popc(in & below)] = (unsigned)bound;
                    L.sorted[np + __popc(in & below)].x = g0 + lane;
                }
                np += __popc(in);
            }
            __syncwarp();
            for (int j = lane; j < np; j += 32) {
                const unsigned mine_ = L.mem_k[j];
                int place = 0;
#pragma unroll 8
                for (int v = 0; v < np; v++) {
                    const unsigned o = L.mem_k[v];
                    place += o > mine_ || (o == mine_ && v < j) ? 1 : 0;
                }
                L.pick[place] = L.sorted[j].x;
            }
            __syncwarp();
            if (lane == 0) {
                sh->np = np;
                sh->next = 0;
                sh->fatal = 0;
                sh->M = M;
                sh->tf = tf;
                sh->n = n;
                __threadfence_block();
                *(volatile int*)&sh->open = 1;
            }
            __syncwarp();
            kh_help<DP>(a, gw, lane, sh, gw, sq64, k);
            if (lane == 0) {
                *(volatile int*)&sh->open = 0;
                __threadfence_block();
                // helpers still in a group (bounded: each ends its group and leaves)
                int wait = 0;
                while (*(volatile int*)&sh->busy > 0 && wait < KH_WAIT) {
                    __nanosleep(200);
                    wait++;
                }
                if (wait == KH_WAIT) sh->fatal = KH_LATE;
                __threadfence_block();
            }
            __syncwarp();
            M = *(volatile int*)&sh->M;
            fatal = max(fatal, *(volatile int*)&sh->fatal);
            __syncwarp();
            if (fatal == KH_CROWD) {
                const int found = kh_exact_groups<DP>(a, gw, lane, np, tf, n, k, sq64, M);
                fatal = max(-found, 0);
                M = max(found, 0);
            }
            // ---- 4. the M-th nearest entry
            if (!fatal) {
                int b = -1;
                for (int g = 0; g < KH_NB / 32 && b < 0; g++) {
                    const unsigned hit = __ballot_sync(0xffffffffu, (int)sm->hit[g * 32 + lane] >= M);
                    if (hit) b = g * 32 + __ffs(hit) - 1;
                }
                const int m = b < 0 ? 0 : (int)sm->cnt[b], start = b < 0 ? 0 : (int)sm->hit[b] - m;
                if (b < 0 || M < 1 || m > KH_RANK) {
                    fatal = 7;
                } else {
                    kh_bin_d64<DP>(a, L, lane, start, m, sq64);
                    const int want = start + m - M;  // its place, farthest first
                    int at = -1;
                    const bool distinct = kh_rank(L, lane, m, [&](int j, int place) {
                        L.rank[L.order[start + j].x] = (uint16_t)place;
                        if (place == want) at = j;
                    });
                    // (ranked twice where 32-bit keys tie: the second time counts)
                    if (at >= 0 && (int)L.rank[L.order[start + at].x] != want) at = -1;
                    const unsigned hit = __ballot_sync(0xffffffffu, at >= 0);
                    if (!distinct || !hit) fatal = 8;
                    __syncwarp();
                    // the brute-force passes' last candidate bin for this top (they
                    // move their bins up at most three times)
                    int bstar = WP_NN_BINS - 1, qbase = a.qbase[slot];
                    float lim = 0.f;
                    if (!fatal) {
                        const double td = __longlong_as_double(L.mem_d[__shfl_sync(0xffffffffu, at, __ffs(hit) - 1)]);
                        const float v = wp_nn_bound(td);
                        for (int u = 0; u < 4; u++) {
                            bstar = wp_nn_bin(v, qbase);
                            if (bstar < WP_NN_BINS - 1) break;
                            qbase += WP_NN_REDO_SHIFT;
                        }
                        if (bstar == WP_NN_BINS - 1) fatal = 12;
                        lim = wp_nn_bin_start(qbase, bstar + 1);
                    }
                    if (!fatal) {
                        // the leaves' parts in tree order, the kept entries of each
                        for (int j = lane; j < nseg; j += 32) {
                            const int2 s = seg[j];
                            int place = 0;
                            for (int v = 0; v < nseg; v++) place += seg[v].x < s.x ? 1 : 0;
                            L.sorted[place] = make_int2(s.y, j + 1 < nseg ? seg[j + 1].y : n);
                        }
                        __syncwarp();
                        const long out = (long)(slot - a.q0) * a.stride;
                        float qd = 0.f;
                        {
                            float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;  // as wp_nn.cu's nn_norm2_x2
#pragma unroll
                            for (int u = 0; u < DP / 4; u++) {
                                const float4 q = sm->q32[u];
                                a0 = fmaf(q.x, q.x, a0);
                                a1 = fmaf(q.y, q.y, a1);
                                a2 = fmaf(q.z, q.z, a2);
                                a3 = fmaf(q.w, q.w, a3);
                            }
                            qd = (a0 + a1) + (a2 + a3);
                        }
                        const float near = fmaf(1.001f, lim, fmaf(2e-5f, qn, 1e-4f));
                        int kept = 0, slice = -1, wrote = 0;
                        for (int s = 0; s < nseg && !fatal; s++) {
                            const int2 part = L.sorted[s];
                            for (int i0 = part.x; i0 < part.y && !fatal; i0 += 32) {
                                const int i = i0 + lane;
                                bool cand = false, keep = false;
                                int pos = 0;
                                float d2 = 0.f;
                                if (i < part.y && L.d[i] <= near) {
                                    const int bi = L.bin[i];
                                    keep = bi < b || (bi == b && (int)L.rank[i] >= want);
                                    pos = L.ent[i].x;
                                    // as wp_nn.cu's nn_d2_dot_x2 (the bin) and nn_d2_x2
                                    float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f, p0 = 0.f, p1 = 0.f, p2 = 0.f, p3 = 0.f;
                                    const float4* e = reinterpret_cast<const float4*>(a.coords + (long)pos * DP);
#pragma unroll
                                    for (int u = 0; u < DP / 4; u++) {
                                        const float4 v = __ldg(e + u), q = sm->q32[u];
                                        const float x0 = q.x - v.x, x1 = q.y - v.y, x2 = q.z - v.z, x3 = q.w - v.w;
                                        a0 = fmaf(x0, x0, a0);
                                        a1 = fmaf(x1, x1, a1);
                                        a2 = fmaf(x2, x2, a2);
                                        a3 = fmaf(x3, x3, a3);
                                        p0 = fmaf(q.x, v.x, p0);
                                        p1 = fmaf(q.y, v.y, p1);
                                        p2 = fmaf(q.z, v.z, p2);
                                        p3 = fmaf(q.w, v.w, p3);
                                    }
                                    d2 = (a0 + a1) + (a2 + a3);
                                    const float dot = fmaxf(fmaf(-2.f, (p0 + p1) + (p2 + p3), qd + a.enorm[pos]), 0.f);
                                    cand = wp_nn_bin(dot, qbase) <= bstar;
                                }
                                kept += __popc(__ballot_sync(0xffffffffu, keep));
                                // slice by slice, each from a multiple of 32
                                const int sl = pos / a.slice_len;
                                unsigned left = __ballot_sync(0xffffffffu, cand);
                                while (left) {
                                    const int now = __shfl_sync(0xffffffffu, sl, __ffs(left) - 1);
                                    if (now != slice) {
                                        const int up = (wrote + 31) / 32 * 32;
                                        if (wrote + lane < up && up <= a.stride) a.kept_pos[out + wrote + lane] = -1;
                                        wrote = up;
                                        slice = now;
                                    }
                                    const unsigned cm = __ballot_sync(0xffffffffu, cand && sl == now);
                                    if (wrote + __popc(cm) > a.stride) {
                                        fatal = 11;
                                        break;
                                    }
                                    if (cand && sl == now) {
                                        const long p = out + wrote + __popc(cm & below);
                                        a.kept_pos[p] = keep ? pos : -1;
                                        a.kept_d2[p] = d2;
                                    }
                                    wrote += __popc(cm);
                                    left &= ~cm;
                                }
                            }
                        }
                        if (kept != M && !fatal) fatal = 13;
                        M = wrote;
                    }
                }
            }
        }
        if (lane == 0) a.kept_n[slot] = fatal ? (fatal == KH_LATE ? WP_KH_LATE : -1) : M;
        if (fatal == KH_LATE) {
            // a helper may still be using this warp's list and record: the warp looks
            // into no more reads, and the call fails
            if (lane == 0) kh_drain(a);
            break;
        }
        __syncwarp();
    }
    // no reads left: help until the CTA's other warps are through (or, past the
    // limit, leave the rest to them)
    if (lane == 0) atomicAdd(&leaving, 1);
    for (int i = 0; i < KH_WAIT; i++) {
        int left = 0;
        if (lane == 0) left = *(volatile int*)&leaving;
        if (__shfl_sync(0xffffffffu, left, 0) == KH_WARPS) break;
        help();
        __nanosleep(1000);
    }
}

// Counts as nibbles, transposed per 128 positions (KHArgs::nib).
__global__ void wp_khits_pack_kernel(const uint8_t* __restrict__ cnt, int N, int DP, uint4* __restrict__ nib) {
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    const int W = DP / 8, lane = (int)(i & 31), j = (int)((i >> 5) % W);
    const long g = (i >> 5) / W;
    if (g * 128 >= N) return;
    uint32_t v[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
        const long p = g * 128 + 32 * u + lane;
        v[u] = 0u;
        if (p < N) {
            const uint2 w = *reinterpret_cast<const uint2*>(cnt + p * DP + 8 * j);
            v[u] = w.x | (w.y << 4);
        }
    }
    nib[i] = make_uint4(v[0], v[1], v[2], v[3]);
}

cudaError_t wp_launch_khits_pack(const uint8_t* cnt, int N, int DP, uint4* nib, cudaStream_t s) {
    const long n = (long)((N + 127) / 128) * (DP / 8) * 32;
    if (n == 0) return cudaSuccess;
    wp_khits_pack_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(cnt, N, DP, nib);
    return cudaGetLastError();
}

int wp_khits_warps_per_cta() { return KH_WARPS; }
int wp_khits_groups() { return KH_MAXG; }
int wp_khits_rank() { return KH_RANK; }

size_t wp_khits_smem_bytes(int TC, int NC, int stack_cap) {
    const size_t tab = ((size_t)TC * NC * (sizeof(double) + sizeof(float)) + 15) / 16 * 16;
    const size_t stk = ((size_t)stack_cap * (sizeof(int) + sizeof(double)) + 15) / 16 * 16;
    return (sizeof(KHSmem) + tab + stk) * KH_WARPS;
}

template <int DP>
static cudaError_t kh_launch(int grid, size_t smem, cudaStream_t s, const KHArgs& a) {
    int per_sm = 0, sms = 0;
    const cudaError_t e = wp_launch_shape(reinterpret_cast<const void*>(wp_khits_kernel<DP>), KH_WARPS * 32, smem,
                                          &per_sm, &sms);
    if (e != cudaSuccess) return e;
    wp_khits_kernel<DP><<<grid, KH_WARPS * 32, smem, s>>>(a);
    return cudaGetLastError();
}

cudaError_t wp_launch_khits(int grid, cudaStream_t s, const KHArgs& a) {
    const size_t smem = wp_khits_smem_bytes(a.TC, a.NC, a.stack_cap);
    if (grid <= 0 || a.Rc == 0) return cudaSuccess;
    switch (a.DP) {
        case 16: return kh_launch<16>(grid, smem, s, a);
        case 32: return kh_launch<32>(grid, smem, s, a);
        case 48: return kh_launch<48>(grid, smem, s, a);
        case 64: return kh_launch<64>(grid, smem, s, a);
    }
    return cudaErrorInvalidValue;
}
