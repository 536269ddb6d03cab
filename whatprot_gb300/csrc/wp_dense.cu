// wp_dense.cu -- dense warp-per-pair forward pass: the fallback for pairs
// whose pruned boxes exceed the pair engine's per-thread slab.
//
// One warp per (read, peptide) pair; the pair's two state tensors (normal
// and broken-N) are held over the full extents [0, D_c + 1) per channel in
// shared memory, lanes striding over states.  Instead of restricting each
// step to its pruned box, every state is computed and the emission factors
// are zero outside the read's emission box [cmin_t, cmax_t); because dye
// counts never increase this reproduces the reference's pruned result
// exactly (the only leak, the detached-state sum, is dropped by the
// allow-detached flags in the same timesteps as in the reference,
// hmm/step/peptide-emission.cc:218-223).  Same FP32 arithmetic and exact
// power-of-two rescaling as the pair engine.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <algorithm>

#include "wp_common.cuh"
#include "wp_engine.cuh"

#define WP_DENSE_WARPS 8

// Edman success coefficients by (dye count n, remaining dyes tot) at
// [n * 17 + tot], rounded as the kernel's own expression: the cut dye was
// another one (x), the state one dye up lost the cut dye (y).
struct DenseEdman {
    float x[16 * 17], y[16 * 17];
};

#define WP_DENSE_NONE 31u  // in an Edman position's word: no dye there

// Slab classes of a launch (see above).
struct DensePass {
    int S_small, S_cap;  // states per slice of a warp's slab in the two phases
    int big_warps;       // warps of the second phase (0: no pair is larger than S_small)
};

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ int warp_max_int(int v) {
    return __reduce_max_sync(0xffffffffu, v);
}

// In-place binomial transition along one channel axis for every fiber of
// the slices e < e_count (binomial-transition.cc:114-136):
// out[to] = sum_{from >= to} prob(from, to) * in[from].
template <int W>
__device__ void binomial_fibers(float* X, int S, int F, int nf, int stc,
                                const uint16_t* __restrict__ fib,
                                const float* __restrict__ tab, int lane) {
    float p[W * (W + 1) / 2];
#pragma unroll
    for (int i = 0; i < W * (W + 1) / 2; i++) p[i] = tab[i];
    int e = lane / F, r = lane - (lane / F) * F;
    const int de = 32 / F, dr = 32 - de * F;
    for (int f = lane; f < nf; f += 32) {
        int base = e * S + fib[r];
        float v[W];
#pragma unroll
        for (int i = 0; i < W; i++) v[i] = X[base + i * stc];
#pragma unroll
        for (int to = 0; to < W; to++) {
            float acc = 0.0f;
#pragma unroll
            for (int from = to; from < W; from++) acc = fmaf(p[from * (from + 1) / 2 + to], v[from], acc);
            X[base + to * stc] = acc;
        }
        r += dr;
        e += de;
        if (r >= F) {
            r -= F;
            e++;
        }
    }
}

// Same transition for W > 8: table entries read from shared memory (one
// broadcast load per multiply-add), in place with ascending `to`.
__device__ void binomial_fibers_wide(float* X, int S, int W, int F, int nf, int stc,
                                     const uint16_t* __restrict__ fib,
                                     const float* __restrict__ tab, int lane) {
    int e = lane / F, r = lane - (lane / F) * F;
    const int de = 32 / F, dr = 32 - de * F;
    for (int f = lane; f < nf; f += 32) {
        int base = e * S + fib[r];
        for (int to = 0; to < W; to++) {
            float acc = 0.0f;
            for (int from = to; from < W; from++)
                acc = fmaf(tab[from * (from + 1) / 2 + to], X[base + from * stc], acc);
            X[base + to * stc] = acc;
        }
        r += dr;
        e += de;
        if (r >= F) {
            r -= F;
            e++;
        }
    }
}

__device__ void binomial_step(float* X, int S, int W, int e_count, int stc,
                              const uint16_t* fib, const float* tab, int lane) {
    int F = S / W;
    int nf = e_count * F;
    switch (W) {
#define WP_BCASE(w) case w: binomial_fibers<w>(X, S, F, nf, stc, fib, tab, lane); break;
        WP_BCASE(2) WP_BCASE(3) WP_BCASE(4) WP_BCASE(5) WP_BCASE(6) WP_BCASE(7) WP_BCASE(8)
#undef WP_BCASE
        default: binomial_fibers_wide(X, S, W, F, nf, stc, fib, tab, lane); break;
    }
}

// Per-warp shared memory carve-up.
struct WarpBufs {
    uint32_t* code;  // [T - 1] Edman position: st << 16 | (D + 1) << 10 | tot << 5 | 4 c, WP_DENSE_NONE for no dye
    float* X;
    float* XB;
    float* em;
    uint16_t* coord;
    uint16_t* fib;  // [C][S_cap]
};

__host__ __device__ inline size_t wp_warp_bytes(int T, int S_cap, int C, bool has_block) {
    size_t f = (size_t)(has_block ? 2 : 1) * T * S_cap + S_cap;
    size_t h = (size_t)S_cap * (1 + C);
    size_t b = f * 4 + h * 2;
    return (b + 15) & ~(size_t)15;
}

// Forward pass of one (read, peptide) pair by one warp.  Returns the
// probability as mant * 2^expo (mant == 0: probability zero).
template <int C, bool HAS_BLOCK>
__device__ void pair_forward(const BatchArgs& a, const SmemModel& H, const DenseEdman& ed, int r,
                             const DevModel& m, const PeptideRec& pep,
                             const WarpBufs& wb, int S_cap, int lane,
                             float* out_mant, int* out_expo, int* err) {
    const int T = m.T;
    const int W_read = a.W;
    const EmitEntry* __restrict__ rtab = a.tab + (long)r * a.entries;
    const uint8_t* blo = a.lo + (long)r * T * C;
    const uint8_t* bhi = a.hi + (long)r * T * C;
    // widths D + 1 (one byte per channel) and strides (16 bits per channel)
    uint32_t wpk = 0;
    uint64_t spk = 0;
    int S = 1;
    bool empty = a.flags[r] != 0;
#pragma unroll
    for (int c = 0; c < C; c++) {
        wpk |= (uint32_t)(pep.D[c] + 1) << (8 * c);
        if (pep.D[c] < a.Lsuf[(long)r * T * C + c]) empty = true;  // some L_t > D_c
    }
    auto wid = [&](int c) { return (int)((wpk >> (8 * c)) & 255u); };
    auto str = [&](int c) { return (int)((spk >> (16 * c)) & 65535u); };
#pragma unroll
    for (int c = C - 1; c >= 0; c--) {
        spk |= (uint64_t)S << (16 * c);
        S *= wid(c);
    }
    if (empty) {
        *out_mant = 0.0f;
        *out_expo = 0;
        return;
    }
    if (S > S_cap) {
        if (lane == 0) atomicExch(err, 1);
        *out_mant = 0.0f;
        *out_expo = 0;
        return;
    }
    for (int e = lane; e < T - 1; e += 32) {
        const int c = pep.dye[e];
        wb.code[e] = c < 0 ? WP_DENSE_NONE
                           : (uint32_t)str(c) << 16 | (uint32_t)wid(c) << 10 | (uint32_t)pep.tot[e] << 5 |
                                     (uint32_t)(4 * c);
    }
    // Coordinates of each state of an Edman slice, 4 bits per channel.
    for (int j = lane; j < S; j += 32) {
        int code = 0, x = j;
#pragma unroll
        for (int c = C - 1; c >= 0; c--) {
            const int q = x / wid(c);
            code |= (x - q * wid(c)) << (4 * c);
            x = q;
        }
        wb.coord[j] = (uint16_t)code;
    }
    // Fiber base offsets per channel: the states with n_c == 0.
#pragma unroll 1
    for (int c = 0; c < C; c++) {
        if (wid(c) == 1) continue;
        const int F = S / wid(c), sc = str(c);
        for (int rr = lane; rr < F; rr += 32) {
            const int q = rr / sc;
            wb.fib[c * S_cap + rr] = (uint16_t)(q * sc * wid(c) + rr - q * sc);
        }
    }
    float* const X = wb.X;
    float* const XB = wb.XB;
    // t = 0: start state (0, D) (peptide-state-vector.cc:38-40), initial
    // block (block-transition.cc:33-62), then duds per channel.
    for (int j = lane; j < S; j += 32) {
        float a = (j == S - 1) ? 1.0f : 0.0f;
        if (HAS_BLOCK) {
            XB[j] = m.p_ib * a;
            a = (1.0f - m.p_ib) * a;
        }
        X[j] = a;
    }
    __syncwarp();
#pragma unroll 1
    for (int c = 0; c < C; c++) {
        if (wid(c) == 1) continue;
        binomial_step(X, S, wid(c), 1, str(c), wb.fib + c * S_cap, H.dud[c], lane);
        if (HAS_BLOCK) binomial_step(XB, S, wid(c), 1, str(c), wb.fib + c * S_cap, H.dud[c], lane);
        __syncwarp();
    }
    int expo = 0;       // log2 of the factor the stored state is scaled by
    float pd = 0.0f;    // detached state, in the rescaled frame
    int k_prev = 0;     // exponent removed at the last rescale
    float fac_prev = 1.0f;  // (1 - p_detach) pending from the last timestep
    for (int t = 0; t < T; t++) {
        if (t > 0) {
            // Cyclic block (block-transition.cc:33-62).
            if (HAS_BLOCK) {
                int n = t * S;
                for (int i = lane; i < n; i += 32) {
                    float a = X[i];
                    XB[i] = XB[i] + m.p_cb * a;
                    X[i] = (1.0f - m.p_cb) * a;
                }
                __syncwarp();
            }
            // Detach (detach-transition.cc:36-68) is folded into the
            // previous rescale (pd) and the pending factor fac_prev.
            // Bleach per channel.
#pragma unroll 1
            for (int c = 0; c < C; c++) {
                if (wid(c) == 1) continue;
                binomial_step(X, S, wid(c), t, str(c), wb.fib + c * S_cap, H.bleach[c], lane);
                if (HAS_BLOCK) binomial_step(XB, S, wid(c), t, str(c), wb.fib + c * S_cap, H.bleach[c], lane);
                __syncwarp();
            }
            // Edman (edman-transition.cc:62-162) as a gather, in place: state
            // i of slice e reads i, i - S and i - S + st[c], all at most i, so
            // the elements go from the last down, and those of one step are
            // read before any of them is written.
            {
                const float pf = m.pf, qf = 1.0f - m.pf;
                const int n = (t + 1) * S;
                const int de = 32 / S, dj = 32 - de * S;
                const int top = ((n + 31) & ~31) - 32;
                int e = (top + lane) / S, j = top + lane - e * S;
                for (int i0 = top; i0 >= 0; i0 -= 64) {
                    float v[2];
#pragma unroll
                    for (int u = 0; u < 2; u++) {
                        const int i = i0 - 32 * u + lane;
                        v[u] = 0.0f;
                        if (i >= 0 && i < n) {
                            if (e < t) v[u] = pf * X[i];
                            if (e >= 1) {
                                const uint32_t code = wb.code[e - 1];
                                const float xin = X[i - S];
                                if (code == WP_DENSE_NONE) {
                                    v[u] = fmaf(qf, xin, v[u]);
                                } else {
                                    const int nc = (wb.coord[j] >> (code & 31)) & 15, tot = (code >> 5) & 31;
                                    if (nc < tot) v[u] = fmaf(ed.x[nc * 17 + tot], xin, v[u]);
                                    if (nc + 1 < (int)((code >> 10) & 63))
                                        v[u] = fmaf(ed.y[nc * 17 + tot], X[i - S + (int)(code >> 16)], v[u]);
                                }
                            }
                        }
                        j -= dj;
                        e -= de;
                        if (j < 0) {
                            j += S;
                            e--;
                        }
                    }
                    __syncwarp();
#pragma unroll
                    for (int u = 0; u < 2; u++) {
                        const int i = i0 - 32 * u + lane;
                        if (i >= 0 && i < n) X[i] = v[u];
                    }
                    __syncwarp();
                }
                if (HAS_BLOCK)
                    for (int j2 = lane; j2 < S; j2 += 32) XB[t * S + j2] = 0.0f;
                __syncwarp();
            }
        }
        // Emission factors of this timestep for this pair, normalised by the
        // largest exponent over the pair's reachable box.
        int kmax;
        if (!m.interacting) {
            kmax = 0;
#pragma unroll
            for (int c = 0; c < C; c++) {
                // largest exponent over [cmin, min(cmax, D + 1)) of channel
                // c (at most 16 counts: a lane each)
                const int n1 = min((int)bhi[t * C + c], wid(c)), n = blo[t * C + c] + lane;
                int km = WP_EXPO_ZERO;
                if (n < n1) {
                    const EmitEntry en = rtab[(t * C + c) * W_read + n];
                    if (en.mant != 0.0f) km = en.expo;
                }
                km = warp_max_int(km);
                if (km == WP_EXPO_ZERO) kmax = WP_EXPO_ZERO;
                if (kmax != WP_EXPO_ZERO) kmax += km;
            }
        } else {
            int km = WP_EXPO_ZERO;
            for (int j = lane; j < S; j += 32) {
                int code = wb.coord[j], g = 0;
                for (int c = 0; c < C; c++) g = g * W_read + ((code >> (4 * c)) & 15);
                EmitEntry en = rtab[t * wp_ipow(W_read, C) + g];
                if (en.mant != 0.0f) km = max(km, en.expo);
            }
            kmax = warp_max_int(km);
        }
        if (kmax == WP_EXPO_ZERO) {  // no reachable state emits
            *out_mant = 0.0f;
            *out_expo = 0;
            return;
        }
        float em0 = 0.0f;
        for (int j = lane; j < S; j += 32) {
            int code = wb.coord[j];
            float mant = 1.0f;
            int ks = 0;
            if (!m.interacting) {
#pragma unroll
                for (int c = 0; c < C; c++) {
                    EmitEntry en = rtab[(t * C + c) * W_read + ((code >> (4 * c)) & 15)];
                    mant *= en.mant;
                    ks += en.expo;
                }
            } else {
                int g = 0;
                for (int c = 0; c < C; c++) g = g * W_read + ((code >> (4 * c)) & 15);
                EmitEntry en = rtab[t * wp_ipow(W_read, C) + g];
                mant = en.mant;
                ks = en.expo;
            }
            float ev = 0.0f;
            if (mant != 0.0f) {
                int d = ks - kmax;
                if (j == 0) em0 = mant * exp2i(max(d, -200));
                ev = (mant * fac_prev) * exp2i(max(min(d - k_prev, 127), -200));
            }
            wb.em[j] = ev;
        }
        em0 = __shfl_sync(0xffffffffu, em0, 0);
        __syncwarp();
        // Emission (peptide-emission.cc:212-243) over e <= t, with the
        // pending rescale folded in, and the state sum.
        float part = 0.0f;
        {
            int n = (t + 1) * S;
            int j = lane % S;
            const int dj = 32 % S;
            for (int i = lane; i < n; i += 32) {
                float w = wb.em[j];
                float a = X[i] * w;
                X[i] = a;
                part += a;
                if (HAS_BLOCK) {
                    float b = XB[i] * w;
                    XB[i] = b;
                    part += b;
                }
                j += dj;
                if (j >= S) j -= S;
            }
        }
        // The butterfly leaves lane-dependent rounding; take lane 0's value so
        // that every lane applies the same rescale.
        float sum_ab = __shfl_sync(0xffffffffu, warp_sum(part), 0);
        pd = a.allow[(long)r * T + t] ? pd * em0 : 0.0f;
        expo += kmax;
        float tot = sum_ab + pd;
        if (!(tot > 0.0f) || !isfinite(tot)) {
            *out_mant = 0.0f;
            *out_expo = 0;
            return;
        }
        int k;
        float fm = frexpf(tot, &k);
        if (t == T - 1) {
            *out_mant = fm;
            *out_expo = expo + k;
            return;
        }
        float f = exp2i(-k);
        expo += k;
        // Detach of the next timestep (detach-transition.cc:36-68), in the
        // rescaled frame; the stored state keeps its scale until the next
        // emission multiplies in f * (1 - p_detach).
        pd = (pd + H.p_det[t] * sum_ab) * f;
        k_prev = k;
        fac_prev = 1.0f - H.p_det[t];
        __syncwarp();
    }
}


// Persistent: warps take overflow pairs one at a time.  Both phases go
// through the whole list, each taking the pairs of its class.
template <int C, bool HAS_BLOCK>
__global__ void __launch_bounds__(WP_DENSE_WARPS * 32, 4) wp_dense_kernel(BatchArgs a, DensePass ps) {
    const int count = *a.ovf_count;
    if (count == 0) return;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    SmemModel& M = *reinterpret_cast<SmemModel*>(smem_raw);
    DenseEdman& ed = *reinterpret_cast<DenseEdman*>(smem_raw + ((sizeof(SmemModel) + 15) & ~(size_t)15));
    const DevModel& m = *a.model;
    load_smem_model(M, m);
    {
        const float qf = 1.0f - m.pf;
        for (int i = threadIdx.x; i < 16 * 17; i += blockDim.x) {
            const int n = i / 17;
            const float tot = (float)max(i % 17, 1);
            const float ratio = (float)n / tot, r1 = (float)(n + 1) / tot;
            ed.x[i] = qf * (1.0f - ratio);
            ed.y[i] = qf * r1;
        }
    }
    __syncthreads();
    const int T = m.T;
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    uint32_t* code = reinterpret_cast<uint32_t*>(reinterpret_cast<unsigned char*>(&ed) +
                                                 ((sizeof(DenseEdman) + 15) & ~(size_t)15));
    unsigned char* wbase = reinterpret_cast<unsigned char*>(code + WP_DENSE_WARPS * WP_MAX_TIMESTEPS);
    for (int phase = 0; phase < 2; phase++) {
        const int S_cap = phase == 0 ? ps.S_small : ps.S_cap;
        if (phase == 1) {
            if (ps.big_warps == 0) break;
            __syncthreads();  // the small slabs are done with
            if (warp >= ps.big_warps) break;
        }
        float* fb = reinterpret_cast<float*>(wbase + wp_warp_bytes(T, S_cap, C, HAS_BLOCK) * warp);
        const size_t slab = (size_t)T * S_cap;
        WarpBufs wb;
        wb.code = code + warp * WP_MAX_TIMESTEPS;
        wb.X = fb;
        wb.XB = HAS_BLOCK ? fb + slab : nullptr;
        wb.em = fb + (HAS_BLOCK ? 2 : 1) * slab;
        wb.coord = reinterpret_cast<uint16_t*>(wb.em + S_cap);
        wb.fib = wb.coord + S_cap;
        int* head = phase == 0 ? a.ovf_head : a.ovf_head2;
        for (;;) {
            int idx = 0;
            if (lane == 0) idx = atomicAdd(head, 1);
            idx = __shfl_sync(0xffffffffu, idx, 0);
            if (idx >= count) break;
            const int2 rg = a.ovf[idx];
            int vmax;
            const PeptideRec& pep = a.peps[slot_pep(a, rg.x, item_slot(a, rg, &vmax))];
            int S = 1;
            for (int c = 0; c < C; c++) S *= pep.D[c] + 1;
            if (ps.big_warps > 0 && (S > ps.S_small) != (phase == 1)) continue;
            float mant;
            int ex;
            pair_forward<C, HAS_BLOCK>(a, M, ed, rg.x, m, pep, wb, S_cap, lane, &mant, &ex, a.err);
            if (lane == 0) {
                a.res_mant[rg.y] = mant;
                a.res_expo[rg.y] = ex;
            }
            __syncwarp();
        }
    }
}

static size_t dense_fixed_bytes() {
    return ((sizeof(SmemModel) + 15) & ~(size_t)15) + ((sizeof(DenseEdman) + 15) & ~(size_t)15) +
           sizeof(uint32_t) * WP_DENSE_WARPS * WP_MAX_TIMESTEPS;
}

// Whether the dense kernel takes pairs of S_cap states per slice.  The limit
// (two copies of the state beside the model) is a property of the framework,
// not of this kernel's layout: larger pairs are refused.
bool wp_dense_fits(int T, int S_cap, int C, bool has_block, size_t smem_optin) {
    const size_t state = (size_t)(has_block ? 2 : 1) * T * S_cap * sizeof(float);
    return ((sizeof(SmemModel) + 15) & ~(size_t)15) + wp_warp_bytes(T, S_cap, C, has_block) + state <= smem_optin &&
           dense_fixed_bytes() + wp_warp_bytes(T, S_cap, C, has_block) <= smem_optin;
}

template <int C, bool HAS_BLOCK>
static cudaError_t launch_dense(int T, size_t smem_optin, cudaStream_t stream, const BatchArgs& a, long pairs) {
    // Small class: as many states as let 4 CTAs share an SM (228 KB, 1 KB of
    // it per CTA the system's).
    const size_t fixed = dense_fixed_bytes();
    const size_t quarter = (size_t)228 * 1024 / 4 - 1024 - fixed;
    DensePass ps;
    ps.S_cap = a.dense_S_cap;
    ps.S_small = ps.S_cap;
    while (ps.S_small > 4 && wp_warp_bytes(T, ps.S_small, C, HAS_BLOCK) * WP_DENSE_WARPS > quarter) ps.S_small -= 4;
    size_t arena = wp_warp_bytes(T, ps.S_small, C, HAS_BLOCK) * WP_DENSE_WARPS;
    ps.big_warps = 0;
    if (ps.S_small < ps.S_cap) {
        const size_t big = wp_warp_bytes(T, ps.S_cap, C, HAS_BLOCK);
        arena = std::max(arena, big);
        ps.big_warps = (int)std::min<size_t>(arena / big, WP_DENSE_WARPS);
    }
    const size_t smem = fixed + arena;
    if (smem > smem_optin) return cudaErrorInvalidConfiguration;
    int sms = 0, per_sm = 0;
    const cudaError_t e = wp_launch_shape(reinterpret_cast<const void*>(wp_dense_kernel<C, HAS_BLOCK>),
                                          WP_DENSE_WARPS * 32, smem, &per_sm, &sms);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorInvalidConfiguration;
    const int grid =
            std::max(1, (int)std::min<long>((long)sms * per_sm, (pairs + WP_DENSE_WARPS - 1) / WP_DENSE_WARPS));
    wp_dense_kernel<C, HAS_BLOCK><<<grid, WP_DENSE_WARPS * 32, smem, stream>>>(a, ps);
    return cudaGetLastError();
}

// Persistent grid over the dense list (BatchArgs::ovf, at most `pairs`).
cudaError_t wp_launch_dense(bool has_block, int T, int C, size_t smem_optin, cudaStream_t stream,
                            const BatchArgs& a, long pairs) {
    switch (C * 2 + (has_block ? 1 : 0)) {
        case 2: return launch_dense<1, false>(T, smem_optin, stream, a, pairs);
        case 3: return launch_dense<1, true>(T, smem_optin, stream, a, pairs);
        case 4: return launch_dense<2, false>(T, smem_optin, stream, a, pairs);
        case 5: return launch_dense<2, true>(T, smem_optin, stream, a, pairs);
        case 6: return launch_dense<3, false>(T, smem_optin, stream, a, pairs);
        case 7: return launch_dense<3, true>(T, smem_optin, stream, a, pairs);
        case 8: return launch_dense<4, false>(T, smem_optin, stream, a, pairs);
        case 9: return launch_dense<4, true>(T, smem_optin, stream, a, pairs);
        default: return cudaErrorInvalidValue;
    }
}
