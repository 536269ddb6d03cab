// wp_nnscore.cu -- NNClassifier's votes (classifiers/nn-classifier.cc:137-203)
// over a read's kept dye-tracks, one CTA per read: Gaussian weights
// exp(-d^2 / 2 sig^2), per-id scores sum(weight x hits / count), the total and
// the top h ids in ascending (score, id) order.
//
// The scores of all U source ids sit in shared memory (U up to about 23,000;
// wp_nn_select_kernel keeps them in global memory for larger sets).  512 kept
// places of the candidate list at a time get their weights, one per thread; the
// sources of every 32 places, flattened, are taken in batches of 32 whose terms
// are first added per id and then written down as (id, value); each of the 16
// warps adds the values of its ids (id mod 16), 32 at a time.  So every id's sum is
// formed in the list's order and grouping, the one of a warp that walks the list,
// whatever the timing.  The h-th score is found by a radix select over the ids
// touched (a bit each).
//
// Weights of the tracks near the read (within 18.5 x 2 sig^2 of the nearest, i.e.
// above 1e-8 of the largest weight) come from FP64 distances, as the reference
// forms them, the far ones' from FP32 (their error is below 1e-8 of the largest
// weight).  FP64 distances are summed from a per-read table of squared
// differences, for the near tracks of a chunk side by side; that and FP64 exp (108
// FP64 instructions per 32 near tracks at 16 cycles each on this GPU's FP64 pipe)
// and the chain of barriers are what bounds the kernel.  4,000 reads with 5,600
// kept tracks, 20,000 ids: 8.7 ms, 9.7 with near and far places mixed, against 22.1 ms for a
// warp per read with its scores in global memory (780 MB of scattered
// accumulators over the resident warps, beyond L2).
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "wp_common.cuh"

#define SC_THREADS 512
#define SC_WARPS (SC_THREADS / 32)
#define SC_SLAB 2048   // (id, value) pairs written down at a time
#define SC_HMAX 1024   // largest h

// Shared memory after the U scores and their bits.
struct SCSmem {
    double val[SC_SLAB];     // before them a chunk's near tracks (place, track), then the selected scores
    int id[SC_SLAB];         // then their ids
    double w[SC_THREADS];    // weights of the tracks in hand
    int s0[SC_THREADS];      // their first sources
    int pre[SC_THREADS];     // running number of sources
    int batch[SC_WARPS + 1]; // batches of 32 sources before each 32 tracks
    int queue[SC_WARPS][64];
    unsigned hist[256];
    double red[SC_WARPS];
    int redi[SC_WARPS];
    int item, digit, before, nsel, nnear;
};

__device__ __forceinline__ int sc_scan_incl(int v, int* redi) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    if (lane == 31) redi[w] = v;
    __syncthreads();
    int add = 0;
    for (int i = 0; i < w; i++) add += redi[i];
    __syncthreads();
    return v + add;
}

__device__ __forceinline__ double sc_sum(double v, double* red) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    double s = 0.0;
    for (int i = 0; i < SC_WARPS; i++) s += red[i];
    __syncthreads();
    return s;
}

// FP64 squared distance as LeafNode::consider sums it, from the read's table.
__device__ __forceinline__ double sc_d64(const uint8_t* __restrict__ row, const double* sq, int NC, int TC) {
    double acc = 0.0;
    int i = 0;
    for (; i + 3 < TC; i += 4) {
        const uint32_t c = *reinterpret_cast<const uint32_t*>(row + i);
        const double* s = sq + i * NC;
        acc = __dadd_rn(acc, __dadd_rn(__dadd_rn(__dadd_rn(s[c & 255u], s[NC + ((c >> 8) & 255u)]),
                                                 s[2 * NC + ((c >> 16) & 255u)]),
                                       s[3 * NC + (c >> 24)]));
    }
    for (; i < TC; i++) acc = __dadd_rn(acc, sq[i * NC + row[i]]);
    return acc;
}

// The digit (from the top) of the histogram where the running count reaches
// `want`; by warp 0, result in s.digit and the count above it in s.before.
__device__ __forceinline__ void sc_digit(SCSmem& s, int want) {
    const int lane = threadIdx.x & 31;
    int mine = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) mine += (int)s.hist[255 - (lane * 8 + i)];
    int incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    const unsigned hit = __ballot_sync(0xffffffffu, incl >= want);
    if (lane == __ffs(hit) - 1) {
        int c = incl - mine;
        for (int i = 0; i < 8; i++) {
            const int d = 255 - (lane * 8 + i);
            const int n = (int)s.hist[d];
            if (c + n >= want) {
                s.digit = d;
                s.before = c;
                break;
            }
            c += n;
        }
    }
}

__global__ void __launch_bounds__(SC_THREADS, 2) wp_nn_score_kernel(NNScoreArgs a) {
    extern __shared__ __align__(16) unsigned char sc_smem[];
    double* acc = reinterpret_cast<double*>(sc_smem);
    unsigned* bits = reinterpret_cast<unsigned*>(acc + a.U);
    const int nwords = (a.U + 31) / 32;
    double* sq = reinterpret_cast<double*>(sc_smem + (((size_t)a.U * 8 + (size_t)nwords * 4 + 15) / 16 * 16));
    const int ntab = a.table ? a.TC * a.NC : 0;
    SCSmem& s = *reinterpret_cast<SCSmem*>(sq + (ntab + 1) / 2 * 2);
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;

    for (;;) {
        if (tid == 0) s.item = atomicAdd(a.next, 1);
        __syncthreads();
        const int lq = s.item;
        if (lq >= a.R) break;
        const int gq = a.q0 + lq;
        const int n = a.kept_n[gq];
        if (n < 0) {
            __syncthreads();
            continue;
        }
        const int oq = a.qperm ? a.qperm[gq] : gq;
        const long long base = a.koff ? a.koff[lq] : (long long)lq * a.stride;
        for (int i = tid; i < a.U; i += SC_THREADS) acc[i] = 0.0;
        for (int i = tid; i < nwords; i += SC_THREADS) bits[i] = 0u;
        const double* q64 = a.rads ? a.rads + (long)oq * a.TC : nullptr;
        for (int i = tid; i < ntab; i += SC_THREADS) {
            const int dim = i / a.NC, c = i % a.NC;
            const double x = __dsub_rn(q64[dim], a.ctab[(dim % a.C) * a.NC + c]);
            sq[i] = __dmul_rn(x, x);
        }
        float dmin = INFINITY;
        if (q64) {
            for (int i = tid; i < n; i += SC_THREADS)
                if (a.kept_pos[base + i] >= 0) dmin = fminf(dmin, a.kept_d2[base + i]);
            dmin = __uint_as_float(__reduce_min_sync(0xffffffffu, __float_as_uint(dmin)));
            if (lane == 0) s.red[wid] = (double)dmin;
            __syncthreads();
            double m = s.red[0];
            for (int i = 1; i < SC_WARPS; i++) m = fmin(m, s.red[i]);
            dmin = (float)m;
        }
        __syncthreads();
        const double wlim = (double)dmin + 18.5 * a.two_sig_sq + 1e-3;

        // ---- the tracks' contributions
        double total_part = 0.0;
        int2* near_list = reinterpret_cast<int2*>(s.val);
        if (tid == 0) s.nnear = 0;
        __syncthreads();
        for (int c0 = 0; c0 < n; c0 += SC_THREADS) {
            const int i = c0 + tid;
            int ns = 0;
            const int e = i < n ? a.kept_pos[base + i] : -1;
            bool near = false;
            if (e >= 0) {
                const float d2 = a.kept_d2[base + i];
                near = q64 && (double)d2 < wlim;
                if (!near) {
                    // 2^x: exp2f of the fraction, the integer part applied in FP64 so
                    // far entries keep a non-zero weight
                    const float x = -d2 * a.inv_two_sig_sq * 1.4426950408889634f;
                    const float fl = floorf(x);
                    s.w[tid] = ldexp((double)exp2f(x - fl), (int)fl);
                }
                const int f = a.src_off[e];
                s.s0[tid] = f;
                ns = a.src_off[e + 1] - f;
            }
            // the near tracks in hand side by side, so that the FP64 work fills warps
            // (a list has gaps, and near and far places mixed)
            {
                const unsigned nm = __ballot_sync(0xffffffffu, near);
                int at = 0;
                if (lane == 0 && nm) at = atomicAdd(&s.nnear, __popc(nm));
                at = __shfl_sync(0xffffffffu, at, 0);
                if (near) near_list[at + __popc(nm & ((1u << lane) - 1u))] = make_int2(tid, e);
            }
            __syncthreads();
            const int nnear = s.nnear;
            if (tid < nnear) {
                const int2 t = near_list[tid];
                const double d64 = a.table ? sc_d64(a.cnt + (long)t.y * a.DP, sq, a.NC, a.TC)
                                           : wp_nn_exact_d2(q64, t.y, a.TC, a.C, a.DP, a.cnt, a.ctab, a.NC, a.ecoord);
                s.w[t.x] = exp(-d64 / a.two_sig_sq);
            }
            const int incl = sc_scan_incl(ns, s.redi);
            s.pre[tid] = incl;
            if (tid == 0) s.nnear = 0;  // everyone has read it (the scan's barriers)
            __syncthreads();
            if (wid == 0) {
                // batches of up to 32 sources, those of each 32 list places apart
                const int q = min(lane, SC_WARPS - 1), lo = q > 0 ? s.pre[32 * q - 1] : 0;
                int nb = lane < SC_WARPS ? (s.pre[32 * q + 31] - lo + 31) / 32 : 0;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int t = __shfl_up_sync(0xffffffffu, nb, o);
                    if (lane >= o) nb += t;
                }
                if (lane < SC_WARPS) s.batch[lane + 1] = nb;
                if (lane == 0) s.batch[0] = 0;
            }
            __syncthreads();
            const int nbatch = s.batch[SC_WARPS];
            for (int b0 = 0; b0 < nbatch; b0 += SC_SLAB / 32) {
                const int mb = min(SC_SLAB / 32, nbatch - b0), m = mb * 32;
                for (int b = wid; b < mb; b += SC_WARPS) {
                    // a batch per warp, one source per lane
                    int q = 0;
#pragma unroll
                    for (int step = SC_WARPS / 2; step > 0; step >>= 1)
                        if (s.batch[q + step] <= b0 + b) q += step;
                    const int first = q > 0 ? s.pre[32 * q - 1] : 0;
                    const int at = first + (b0 + b - s.batch[q]) * 32 + lane;
                    const bool act = at < s.pre[32 * q + 31];
                    // the track whose running number of sources first exceeds `at`
                    int L = 32 * q;
#pragma unroll
                    for (int step = 16; step > 0; step >>= 1)
                        if (s.pre[L + step - 1] <= at) L += step;
                    int id = -1;
                    double val = 0.0;
                    if (act) {
                        const int src = s.s0[L] + at - (L > 0 ? s.pre[L - 1] : 0);
                        const double w = s.w[L];
                        id = a.src_dense[src];
                        val = w * a.src_ratio[src];
                        total_part += w * (double)a.src_hits[src];
                    }
                    // an id's terms within the batch are added first, in order, and
                    // written by the first
                    s.val[b * 32 + lane] = val;
                    __syncwarp();
                    const unsigned grp = __match_any_sync(0xffffffffu, id);
                    const bool leader = act && lane == __ffs(grp) - 1;
                    double sum = 0.0;
                    if (leader) {
                        unsigned g = grp;
                        while (g) {
                            sum += s.val[b * 32 + __ffs(g) - 1];
                            g &= g - 1;
                        }
                    }
                    __syncwarp();
                    s.val[b * 32 + lane] = sum;
                    s.id[b * 32 + lane] = leader ? id : -1;
                }
                __syncthreads();
                // this warp's ids, 32 pairs at a time
                int* queue = s.queue[wid];
                int qn = 0;
                for (int j0 = 0; j0 < m || qn > 0; j0 += 32) {
                    const int j = j0 + lane;
                    const int idj = j < m ? s.id[j] : -1;
                    const bool mine = idj >= 0 && (idj & (SC_WARPS - 1)) == wid;
                    const unsigned mask = __ballot_sync(0xffffffffu, mine);
                    if (mine) queue[qn + __popc(mask & ((1u << lane) - 1u))] = j;
                    qn += __popc(mask);
                    __syncwarp();
                    if (qn < 32 && j0 + 32 < m) continue;
                    while (qn >= 32 || (qn > 0 && j0 + 32 >= m)) {
                        const int cnt = min(32, qn);
                        const int at = lane < cnt ? queue[lane] : -1;
                        const int rest = lane + cnt < qn ? queue[lane + cnt] : 0;
                        const int id = at >= 0 ? s.id[at] : -1;
                        const unsigned grp = __match_any_sync(0xffffffffu, id);
                        if (id >= 0 && lane == __ffs(grp) - 1) {
                            double v = acc[id];
                            unsigned g = grp;
                            while (g) {
                                v += s.val[queue[__ffs(g) - 1]];
                                g &= g - 1;
                            }
                            acc[id] = v;
                            atomicOr(&bits[id >> 5], 1u << (id & 31));
                        }
                        __syncwarp();
                        if (lane + cnt < qn) queue[lane] = rest;
                        qn -= cnt;
                        __syncwarp();
                    }
                }
                __syncthreads();
            }
        }
        const double tot = sc_sum(total_part, s.red);

        // ---- top h of the touched ids by (score, id)
        int nt = 0;
        for (int i = tid; i < nwords; i += SC_THREADS) nt += __popc(bits[i]);
        nt = (int)__reduce_add_sync(0xffffffffu, (unsigned)nt);
        if (lane == 0) s.redi[wid] = nt;
        if (tid == 0) s.nsel = 0;
        __syncthreads();
        nt = 0;
        for (int i = 0; i < SC_WARPS; i++) nt += s.redi[i];
        __syncthreads();
        const int h = a.h;
        const bool all = nt <= h;
        unsigned long long pre = 0ull, msk = 0ull;
        int id_thr = 0;  // of the ids scoring exactly `pre`, those from id_thr up
        if (!all) {
            int want = h;
            int same = nt;  // ids whose scores agree with `pre` in the digits found
            for (int shift = 56; shift >= 0; shift -= 8) {
                for (int i = tid; i < 256; i += SC_THREADS) s.hist[i] = 0u;
                __syncthreads();
                for (int i = tid; i < nwords; i += SC_THREADS) {
                    unsigned b = bits[i];
                    while (b) {
                        const int id = i * 32 + __ffs(b) - 1;
                        b &= b - 1;
                        const unsigned long long key = (unsigned long long)__double_as_longlong(acc[id]);
                        if ((key & msk) == pre) atomicAdd(&s.hist[(key >> shift) & 255ull], 1u);
                    }
                }
                __syncthreads();
                if (wid == 0) sc_digit(s, want);
                __syncthreads();
                pre |= (unsigned long long)s.digit << shift;
                msk |= 255ull << shift;
                want -= s.before;
                same = (int)s.hist[s.digit];
                __syncthreads();
                if (same == want) break;  // every id with these digits or larger ones is in
            }
            if (same > want) {
                // ties at the h-th score: the `want` largest ids
                unsigned ipre = 0u, imsk = 0u;
                for (int shift = 24; shift >= 0; shift -= 8) {
                    for (int i = tid; i < 256; i += SC_THREADS) s.hist[i] = 0u;
                    __syncthreads();
                    for (int i = tid; i < nwords; i += SC_THREADS) {
                        unsigned b = bits[i];
                        while (b) {
                            const unsigned id = i * 32 + __ffs(b) - 1;
                            b &= b - 1;
                            if ((unsigned long long)__double_as_longlong(acc[id]) == pre && (id & imsk) == ipre)
                                atomicAdd(&s.hist[(id >> shift) & 255u], 1u);
                        }
                    }
                    __syncthreads();
                    if (wid == 0) sc_digit(s, want);
                    __syncthreads();
                    ipre |= (unsigned)s.digit << shift;
                    imsk |= 255u << shift;
                    want -= s.before;
                    __syncthreads();
                }
                id_thr = (int)ipre;
            }
        }
        for (int i = tid; i < nwords; i += SC_THREADS) {
            unsigned b = bits[i];
            while (b) {
                const int id = i * 32 + __ffs(b) - 1;
                b &= b - 1;
                const double v = acc[id];
                const unsigned long long key = (unsigned long long)__double_as_longlong(v) & msk;
                if (all || key > pre || (key == pre && id >= id_thr)) {
                    const int at = atomicAdd(&s.nsel, 1);
                    if (at < SC_HMAX) {
                        s.val[at] = v;
                        s.id[at] = id;
                    }
                }
            }
        }
        __syncthreads();
        const int nsel = min(s.nsel, SC_HMAX);
        int n2 = 1;
        while (n2 < nsel) n2 <<= 1;
        for (int i = nsel + tid; i < n2; i += SC_THREADS) {
            s.val[i] = __longlong_as_double(-1ll);
            s.id[i] = 0x7fffffff;
        }
        __syncthreads();
        // bitonic sort ascending by (score, id); scores are never negative, so
        // their bits order as they do, and a NaN's (a read that is not finite) come
        // after all but the padding's, whatever its sign
        for (int size = 2; size <= n2; size <<= 1)
            for (int stride = size >> 1; stride > 0; stride >>= 1) {
                for (int i = tid; i < n2; i += SC_THREADS) {
                    const int j = i ^ stride;
                    if (j > i) {
                        const double vi = s.val[i], vj = s.val[j];
                        const int ii = s.id[i], ij = s.id[j];
                        const unsigned long long ki = (unsigned long long)__double_as_longlong(vi),
                                                 kj = (unsigned long long)__double_as_longlong(vj);
                        const bool gt = ki > kj || (ki == kj && ii > ij);
                        if (gt == ((i & size) == 0)) {
                            s.val[i] = vj;
                            s.val[j] = vi;
                            s.id[i] = ij;
                            s.id[j] = ii;
                        }
                    }
                }
                __syncthreads();
            }
        // outputs, at the read's own index
        for (int i = tid; i < nsel; i += SC_THREADS) {
            const int u = s.id[i];
            a.out_cand_id[(long)oq * h + i] = a.dense_id[u];
            a.out_cand_score[(long)oq * h + i] = s.val[i];
            if (a.out_cand_pep) a.out_cand_pep[(long)oq * h + i] = a.dense_pep[u];
            // HybridClassifier: sum of adjusted score x peptide count, in
            // candidate order (hybrid-classifier.cc:58-64); the terms formed in
            // parallel
            if (a.out_subfrac) s.val[i] = (s.val[i] / tot) * (double)a.dense_count[u];
        }
        for (int i = nsel + tid; i < h; i += SC_THREADS) {  // the places past them
            a.out_cand_id[(long)oq * h + i] = 0;
            a.out_cand_score[(long)oq * h + i] = 0.0;
        }
        if (a.out_subfrac) {
            __syncthreads();
            if (tid == 0) {
                double sf = 0.0;
#pragma unroll 8
                for (int i = 0; i < nsel; i++) sf += s.val[i];
                a.out_subfrac[oq] = sf;
            }
        }
        if (tid == 0) {
            a.out_ncand[oq] = nsel;
            a.out_total[oq] = tot;
        }
        __syncthreads();
    }
}

size_t wp_nn_score_smem_bytes(int U, int table_entries) {
    return ((size_t)U * 8 + (size_t)((U + 31) / 32) * 4 + 15) / 16 * 16 + (size_t)((table_entries + 1) / 2 * 2) * 8 +
           sizeof(SCSmem);
}

int wp_nn_score_ctas_per_sm(size_t smem) {
    int n = 0, sms = 0;
    if (wp_launch_shape(reinterpret_cast<const void*>(wp_nn_score_kernel), SC_THREADS, smem, &n, &sms) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n;
}

cudaError_t wp_launch_nn_score(int grid, size_t smem, cudaStream_t s, const NNScoreArgs& a) {
    if (a.R == 0) return cudaSuccess;
    int n = 0, sms = 0;
    cudaError_t e =
            wp_launch_shape(reinterpret_cast<const void*>(wp_nn_score_kernel), SC_THREADS, smem, &n, &sms);
    if (e == cudaSuccess) e = cudaMemsetAsync(a.next, 0, sizeof(int), s);
    if (e != cudaSuccess) return e;
    wp_nn_score_kernel<<<grid, SC_THREADS, smem, s>>>(a);
    return cudaGetLastError();
}
