// wp_fitw.cu -- Baum-Welch E-step (hmm/hmm/generic-hmm.h:60-109), one warp
// per read: the default where a read's two state vectors fit shared memory
// beside enough others.  Same sums as wp_fit.cu's kernels.
//
// Chain of timestep t >= 1: cyclic block, detach, bleach per channel, Edman,
// emission.  A backward pass keeps, per timestep, the vector x_t behind the
// detachment (before the bleach steps); the vector at the chain's input is an
// affine function of it (b = (1 - p) x + p pd, then the block's mix), so
// neither is formed.  A forward sweep then takes the expected counts:
//
//   * Bleach.  Losing dyes one by one, the expected losses from n are
//     q n (value with n - 1), and the channels' bleach steps commute, so both
//     sums of every channel come from the forward vector f behind the
//     detachment and x:  den_c = sum n_c f x,  num_c = q_c sum n_c f x(n_c - 1).
//     All terms are positive and no vector between the bleach steps is needed.
//   * Detach: sums of f and f x over the non-zero states.
//   * Edman: f behind the bleach steps against the backward vectors on both
//     sides of the cut, recomputed from x_{t+1} (two multiply-adds).
//   * Dud: the start is one state, so P is the dot product of the emission-weighted
//     vector at t = 0 with one fixed vector, and a channel's dud count the same
//     weighted by the dyes a state has lost, D_c - n_c.
//   * Emission statistics at t: column sums of f b at the next chain's input.
//
// Layout: rows of S = prod (D_c + 1) dye-count states per Edman cut.  Lanes own
// columns (32 at a time) and walk the rows, so weights and coefficients stay in
// registers and per-column sums need no communication; columns are taken in
// the order that leaves a cut's neighbour (one dye up or down) unmodified, and
// every step works in place.  The bleach steps take a channel's fibres, one per
// lane, in registers (up to six counts; longer ones in place).  x_t goes to a
// per-warp slab in global memory (38 KB at 3 channels of 4/3/3 dyes and 16
// timesteps: the resident warps' slabs stay in L2).
//
// Vectors are FP32 with powers of two carried as integers (backward after each
// step, forward in the next step's weights); sums over the states of one timestep
// are FP32, their frame factor 2^(exponents) / P and the sums over timesteps and
// reads FP64, in a fixed order.
//
// Bound by instruction issue and shared-memory bandwidth (about 150 issue slots
// per 32 states and timestep).  50,000 reads, 3 channels (4/3/3 dyes), 16
// timesteps: 5.6 ms, against 60.3 ms for a CTA per read, whose 500 block-wide
// barriers per read each waited for a handful of states per thread.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "wp_common.cuh"

#define FW_WARPS 8    // most warps per CTA
#define FW_MAXW 6     // fibres of up to this length are processed in registers
#define FW_LOW (-8)   // vectors 2^8 and more below their place are brought up at once
#define FW_TOP 96     // the forward vector's largest entry is kept near 2^96: where later
                      // timesteps contradict earlier ones the read's path can lie far below
                      // it (2^-33 per dark dye and cycle), and FP32 ends at 2^-149
#define FW_EMIS_N (WP_MAX_DYES_PER_CHANNEL + 1)

// The slots of wp_fit.cu.
__device__ __forceinline__ int fw_det(int t) { return 6 + 2 * t; }
__device__ __forceinline__ int fw_rate(int T, int c) { return 6 + 2 * (T - 1) + 4 * c; }
__device__ __forceinline__ int fw_emis(int T, int C, int kind, int c, int n) {
    return 6 + 2 * (T - 1) + 4 * C + (kind * C + c) * FW_EMIS_N + n;
}

__device__ __forceinline__ float fw_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// The lanes' sums of N values (a power of two): lane l gets that of value l mod N.
template <int N>
__device__ __forceinline__ float fw_sums(float (&v)[N], int lane) {
#pragma unroll
    for (int w = N / 2; w >= 1; w >>= 1) {
        const bool up = (lane & w) != 0;
#pragma unroll
        for (int i = 0; i < w; i++)
            v[i] = (up ? v[i + w] : v[i]) + __shfl_xor_sync(0xffffffffu, up ? v[i] : v[i + w], w);
    }
#pragma unroll
    for (int o = N; o < 32; o <<= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
    return v[0];
}

// Largest of the lanes' non-negative floats.
__device__ __forceinline__ float fw_max(float v) {
    return __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(v)));
}

// 2^e for any e an FP32 product can need, in two factors.
__device__ __forceinline__ float fw_exp2(float v, int e) {
    const int a = max(-126, min(126, e)), b = max(-126, min(126, e - a));
    return v * __int_as_float((a + 127) << 23) * __int_as_float((b + 127) << 23);
}

// 2^e, the frame of sums whose truth is a count: where e passes 1000 they have long
// underflowed to zero, and zero they stay.
__device__ __forceinline__ double fw_exp2d(int e) {
    return __hiloint2double((max(-1000, min(1000, e)) + 1023) << 20, 0);
}

// Exponent k with v = m 2^k, m in [0.5, 1); 0 for v = 0.
__device__ __forceinline__ int fw_expo(float v) {
    int k = 0;
    if (v > 0.f) frexpf(v, &k);
    return k;
}

// One channel's binomial step in place over nf fibres of W states (stride
// st): forward out[x] = sum_{from >= x} p(from, x) in[from], else its
// transpose out[x] = sum_{to <= x} p(x, to) in[to].  tab: p(i, j) at
// i (i + 1) / 2 + j.  Returns the largest value written; with `out`, also
// writes the result there.
template <int W, bool FORWARD, bool OUT>
__device__ __forceinline__ float fw_binomial_w(float* v, int nf, int st, unsigned magic, const float* tab, int lane,
                                               float* out) {
    float p[W * (W + 1) / 2];
#pragma unroll
    for (int i = 0; i < W * (W + 1) / 2; i++) p[i] = tab[i];
    float mx = 0.f;
    for (int f = lane; f < nf; f += 32) {
        const int q = st == 1 ? f : (int)__umulhi((unsigned)f, magic);
        const int base = q * (st * W) + (f - q * st);
        float x[W];
#pragma unroll
        for (int i = 0; i < W; i++) x[i] = v[base + i * st];
#pragma unroll
        for (int i = 0; i < W; i++) {
            float s = 0.f;
            if (FORWARD) {
#pragma unroll
                for (int k = i; k < W; k++) s = fmaf(p[k * (k + 1) / 2 + i], x[k], s);
            } else {
#pragma unroll
                for (int k = 0; k <= i; k++) s = fmaf(p[i * (i + 1) / 2 + k], x[k], s);
            }
            v[base + i * st] = s;
            if (OUT) out[base + i * st] = s;
            if (OUT) mx = fmaxf(mx, s);
        }
    }
    return mx;
}

template <bool FORWARD, bool OUT>
__device__ float fw_binomial(float* v, int n, int W, int st, unsigned magic, const float* tab, int lane, float* out) {
    const int nf = n / W;
    switch (W) {
        case 2: return fw_binomial_w<2, FORWARD, OUT>(v, nf, st, magic, tab, lane, out);
        case 3: return fw_binomial_w<3, FORWARD, OUT>(v, nf, st, magic, tab, lane, out);
        case 4: return fw_binomial_w<4, FORWARD, OUT>(v, nf, st, magic, tab, lane, out);
        case 5: return fw_binomial_w<5, FORWARD, OUT>(v, nf, st, magic, tab, lane, out);
        case 6: return fw_binomial_w<6, FORWARD, OUT>(v, nf, st, magic, tab, lane, out);
        default: break;
    }
    float mx = 0.f;
    for (int f = lane; f < nf; f += 32) {
        const int q = st == 1 ? f : (int)__umulhi((unsigned)f, magic);
        float* b = v + q * (st * W) + (f - q * st);
        // in place: forward results need the entries from theirs up, the
        // transpose's those up to theirs
        for (int u = 0; u < W; u++) {
            const int i = FORWARD ? u : W - 1 - u;
            float s = 0.f;
            if (FORWARD) {
                for (int k = i; k < W; k++) s = fmaf(tab[k * (k + 1) / 2 + i], b[k * st], s);
            } else {
                for (int k = 0; k <= i; k++) s = fmaf(tab[i * (i + 1) / 2 + k], b[k * st], s);
            }
            b[i * st] = s;
            if (OUT) out[(b - v) + i * st] = s;
            mx = fmaxf(mx, s);
        }
    }
    return mx;
}

// Shared memory of a CTA (floats): per e the Edman cut, the columns' dye
// counts, the dud vector, the binomial tables; then per warp its vectors.
struct FWLayout {
    int S, T, C, wsum;
    int tri;        // entries of the channels' binomial tables
    int cuts;       // dye counts per position of the cut table (most dyes + 2)
    int vec;        // floats of one padded vector
    int per_warp;   // floats per warp
    int shared;     // floats of the CTA's tables
};

__host__ __device__ inline FWLayout fw_layout(int T, int C, const int* D, bool hb, bool emission, int nslots) {
    FWLayout L;
    L.T = T;
    L.C = C;
    L.S = 1;
    L.wsum = 0;
    L.tri = 0;
    for (int c = 0; c < C; c++) {
        L.S *= D[c] + 1;
        L.wsum += D[c] + 1;
        L.tri += (D[c] + 1) * (D[c] + 2) / 2;
    }
    L.vec = (T * L.S + 32 + 3) / 4 * 4;
    // the vectors behind a front pad of S (a column's neighbour one dye down)
    int w = L.S + (hb ? 4 : 2) * L.vec;
    w += 2 * L.S + 32;          // front pad and weights of one timestep
    w += T * L.wsum;            // weights per (t, c, n)
    w += emission ? L.S : 0;    // column products (emission statistics)
    w += 7 * (T + 1);           // per timestep: kmx, exponents, pd, detach sums and their frame
    w = (w + 3) / 4 * 4;
    w += 2 * nslots;            // FP64 sums
    L.per_warp = (w + 3) / 4 * 4;
    L.cuts = 2;
    for (int c = 0; c < C; c++) L.cuts = D[c] + 2 > L.cuts ? D[c] + 2 : L.cuts;
    L.shared = (2 * T * L.cuts + T + L.S + L.S + L.tri + 3) / 4 * 4;
    return L;
}

template <int C, bool HB>
__global__ void __launch_bounds__(FW_WARPS * 32, 2) wp_fit_warp_kernel(FitArgs a, float* slab, long slab_stride) {
    extern __shared__ __align__(16) float fw_smem[];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, wpc = blockDim.x >> 5;
    const int inst = a.inst_ctas > 0 ? (int)(blockIdx.x / a.inst_ctas) : 0;
    const long lw = (a.inst_ctas > 0 ? (long)(blockIdx.x % a.inst_ctas) : (long)blockIdx.x) * wpc + wib;
    const long gw = (a.inst_ctas > 0 ? (long)a.inst_ctas : (long)gridDim.x) * wpc;
    const DevModel& m = a.model[inst];
    const int T = m.T;
    const FWLayout L = fw_layout(T, C, a.D, HB, a.emission != 0, a.nslots);
    const int S = L.S, NC = (S + 31) / 32;
    int W[C], st[C], woff[C];
    unsigned magic[C];
    {
        int s = 1;
#pragma unroll
        for (int c = C - 1; c >= 0; c--) {
            W[c] = a.D[c] + 1;
            st[c] = s;
            magic[c] = s > 1 ? 0xffffffffu / (unsigned)s + 1u : 0u;
            s *= W[c];
        }
        int o = 0;
#pragma unroll
        for (int c = 0; c < C; c++) {
            woff[c] = o;
            o += W[c];
        }
    }
    // ---- the CTA's tables
    // [T][cuts] (1 - p_fail) times {another dye is cut, the cut dye shows} with n dyes left
    float2* e_cut = reinterpret_cast<float2*>(fw_smem);
    // [T] the cut's channel: its stride and 4 c (<< 16); 0 without a dye
    int* e_ch = reinterpret_cast<int*>(e_cut + T * L.cuts);
    uint32_t* coord = reinterpret_cast<uint32_t*>(e_ch + T);  // [S] dye counts, 4 bits per channel
    float* dud0 = reinterpret_cast<float*>(coord + S);        // [S] start through the duds
    float* bleach = dud0 + S;                                 // the channels' binomial tables
    int boff[C];
    {
        int o = 0;
#pragma unroll
        for (int c = 0; c < C; c++) {
            boff[c] = o;
            o += W[c] * (W[c] + 1) / 2;
        }
    }
    const float pf = m.pf, qf = 1.0f - m.pf;
    for (int e = threadIdx.x; e < T; e += blockDim.x) {
        const int c = a.dye[e];
        for (int n = 0; n < L.cuts; n++) {
            const float x = c >= 0 ? (float)n / (float)a.tot[e] : 0.f;
            e_cut[e * L.cuts + n] = make_float2(x < 1.f ? qf * (1.f - x) : 0.f, qf * x);
        }
        int s = 0;
#pragma unroll
        for (int k = 0; k < C; k++)
            if (k == c) s = st[k];
        e_ch[e] = c >= 0 ? s | (4 * c) << 16 : 0;
    }
    for (int j = threadIdx.x; j < S; j += blockDim.x) {
        uint32_t pk = 0;
        float full = 1.f;
#pragma unroll
        for (int c = 0; c < C; c++) {
            const int n = (j / st[c]) % W[c], D = W[c] - 1;
            pk |= (uint32_t)n << (4 * c);
            full *= m.dud[c][D * (D + 1) / 2 + n];
        }
        coord[j] = pk;
        dud0[j] = full;
    }
#pragma unroll
    for (int c = 0; c < C; c++)
        for (int i = threadIdx.x; i < W[c] * (W[c] + 1) / 2; i += blockDim.x) bleach[boff[c] + i] = m.bleach[c][i];
    // ---- the warp's own
    float* mine = fw_smem + L.shared + (size_t)wib * L.per_warp;
    float* FA = mine + S;
    float* XA = FA + L.vec;
    float* FB = HB ? XA + L.vec : nullptr;
    float* XB = HB ? FB + L.vec : nullptr;
    float* wv = (HB ? XB : XA) + L.vec + S;      // weights of one timestep behind a pad of S
    float* wtab = wv + S + 32;                   // [T][wsum]
    float* colv = wtab + T * L.wsum;             // [S] with emission statistics
    int* kmx = reinterpret_cast<int*>(colv + (a.emission ? S : 0));  // [T + 1]
    int* Ebr = kmx + T + 1;                      // exponent of x_t (0: of P)
    int* kx = Ebr + T + 1;                       // its normalising exponent
    float* pdx = reinterpret_cast<float*>(kx + T + 1);  // detached state's backward value beside x_t
    float* dx = pdx + T + 1;                     // detach sums per timestep
    float* dn = dx + T + 1;
    int* dfr = reinterpret_cast<int*>(dn + T + 1);  // their frame's exponent
    double* acc = reinterpret_cast<double*>(mine + L.per_warp - 2 * a.nslots);
    for (int i = lane; i < L.per_warp; i += 32) mine[i] = 0.f;
    float* xs = slab + ((long)blockIdx.x * wpc + wib) * slab_stride;  // x_t at the sum of the earlier ones' sizes
    const int nv = HB ? 2 : 1;
    auto x_at = [&](int t) { return xs + (long)nv * S * (t * (t - 1) / 2); };
    __syncthreads();

    // weights of timestep t into wv
    auto weights = [&](int t) {
        for (int j = lane; j < S; j += 32) {
            const uint32_t pk = coord[j];
            float w = 1.f;
#pragma unroll
            for (int c = 0; c < C; c++) w *= wtab[t * L.wsum + woff[c] + ((pk >> (4 * c)) & 15u)];
            wv[j] = w;
        }
        __syncwarp();
    };

    // The timesteps' sums, value i of every timestep in lane i, FP64 over timesteps
    // and reads: a term's frame factor passes FP32's range where a read's earlier
    // and later timesteps favour different states, and an FP32 sum over timesteps
    // would add terms of different frames.  0, 1: the detach sums (FP64 at the read's
    // end); 2: the cyclic block's denominator; 3: the forward vector's sum; 4, 5:
    // Edman; from 6: bleach; then the block's numerator.
    constexpr int NV = 6 + 2 * C + (HB ? 1 : 0), NR = NV <= 8 ? 8 : 16;
    double all_reads = 0.0;

    double lp_m = 0.0;  // of the lane's read among the last 32: P = lp_m 2^lp_e
    int lp_e = 0;
    long lp_at = -1;
    int lp_n = 0;
    auto flush_logp = [&]() {
        if (lp_at >= 0) a.logp[lp_at] = lp_m > 0.0 ? log(lp_m) + (double)lp_e * 0.69314718055994530942 : -INFINITY;
        lp_at = -1;
        lp_n = 0;
    };

    for (long kr = lw; kr < a.R; kr += gw) {
        const long r = a.read_idx ? (long)a.read_idx[(long)inst * a.R + kr] : kr;
        const long ro = a.read_idx ? (long)inst * a.R + kr : kr;
        // ---- emission weights per (t, c, n), each channel's largest a power of two
        const EmitEntry* tab = a.tab + r * (long)T * C * a.W;
        bool dead = false;
        for (int t = lane; t < T; t += 32) {
            int ks = 0;
#pragma unroll
            for (int c = 0; c < C; c++) {
                const EmitEntry* en = tab + (t * C + c) * a.W;
                int km = WP_EXPO_ZERO;
                for (int n = 0; n < W[c]; n++)
                    if (en[n].mant != 0.0f) km = max(km, en[n].expo);
                if (km == WP_EXPO_ZERO) dead = true;
                for (int n = 0; n < W[c]; n++)
                    wtab[t * L.wsum + woff[c] + n] =
                        en[n].mant != 0.0f && km != WP_EXPO_ZERO ? fw_exp2(en[n].mant, max(en[n].expo - km, -200)) : 0.0f;
                ks += km;
            }
            kmx[t] = ks;
        }
        dead = __any_sync(0xffffffffu, dead);
        __syncwarp();

        float Ps = 0.f, ib = 0.f, dudn[C];
#pragma unroll
        for (int c = 0; c < C; c++) dudn[c] = 0.f;
        // The vector at the input of chain t + 1 from x_{t+1}: detachment q x + o,
        // then the block's mix, with the forward sweep's own coefficients (folded
        // into one factor they would round apart and bias every count).
        float q = 0.f, o = 1.f, cb0 = 1.f, cb1 = 0.f, pd = 1.f;
        int Eb = 0;
        auto affine = [&](int t, float scale) {  // of x_t, times scale
            q = scale * (1.f - m.p_det[t - 1]);
            o = scale * m.p_det[t - 1] * pdx[t];
            if (HB) {
                cb0 = 1.f - m.p_cb;
                cb1 = m.p_cb;
            }
        };
        auto in_a = [&](float xa, float xb) {
            return HB ? fmaf(cb1, fmaf(q, xb, o), cb0 * fmaf(q, xa, o)) : fmaf(q, xa, o);
        };
        if (!dead) {
            // ---- backward
            for (int i = lane; i < T * S; i += 32) {
                XA[i] = 0.f;
                if (HB) XB[i] = 0.f;
            }
            __syncwarp();
            for (int t = T - 1; t >= 1; t--) {
                weights(t);
                // emission and the cut's transpose, rows 0 .. t - 1 from 0 .. t
                for (int h = NC - 1; h >= 0; h--) {
                    const int j = 32 * h + lane;
                    const bool on = j < S;
                    const float w = on ? wv[j] : 0.f;
                    const uint32_t pk = on ? coord[j] : 0u;
                    float xb = HB ? XB[j] : 0.f;
                    float e3 = w * in_a(XA[j], xb);
                    for (int e = 0; e < t; e++) {
                        const int k = (e + 1) * S + j, ch = e_ch[e], s = ch & 0xffff;
                        const float xbn = HB ? XB[k] : 0.f;
                        const float n3 = w * in_a(XA[k], xbn);
                        float v = pf * e3;
                        if (s) {
                            const float2 ec = e_cut[e * L.cuts + ((pk >> (ch >> 16)) & 15u)];
                            const float d3 = wv[j - s] * in_a(XA[k - s], HB ? XB[k - s] : 0.f);
                            v = fmaf(ec.x, n3, fmaf(ec.y, d3, v));
                        } else {
                            v = fmaf(qf, n3, v);
                        }
                        __syncwarp();
                        if (on) {
                            XA[e * S + j] = v;
                            if (HB) XB[e * S + j] = w * fmaf(q, xb, o);
                        }
                        e3 = n3;
                        xb = xbn;
                    }
                    __syncwarp();
                }
                pd *= wv[0];
                float mx = pd;
                float* out = x_at(t);
#pragma unroll
                for (int c = C - 1; c >= 0; c--) {
                    if (c > 0) {
                        if (W[c] > 1) {
                            fw_binomial<false, false>(XA, t * S, W[c], st[c], magic[c], bleach + boff[c], lane, nullptr);
                            if (HB)
                                fw_binomial<false, false>(XB, t * S, W[c], st[c], magic[c], bleach + boff[c], lane, nullptr);
                        }
                    } else if (W[0] > 1) {
                        mx = fmaxf(mx, fw_binomial<false, true>(XA, t * S, W[0], st[0], magic[0], bleach, lane, out));
                        if (HB)
                            mx = fmaxf(mx, fw_binomial<false, true>(XB, t * S, W[0], st[0], magic[0], bleach, lane,
                                                                    out + t * S));
                    } else {
                        for (int i = lane; i < t * S; i += 32) {
                            out[i] = XA[i];
                            mx = fmaxf(mx, XA[i]);
                            if (HB) {
                                out[t * S + i] = XB[i];
                                mx = fmaxf(mx, XB[i]);
                            }
                        }
                    }
                    __syncwarp();
                }
                int k = fw_expo(fw_max(mx)), up = 0;
                if (k < FW_LOW) {
                    // left to the weights of the next step, so small a vector would
                    // cost its terms their low bits, and below 2^-127 the scale
                    // that undoes it would be infinite
                    up = k;
                    k = 0;
                    for (int i = lane; i < t * S; i += 32) {
                        out[i] = XA[i] = fw_exp2(XA[i], -up);
                        if (HB) out[t * S + i] = XB[i] = fw_exp2(XB[i], -up);
                    }
                    pd = fw_exp2(pd, -up);
                }
                if (lane == 0) {
                    pdx[t] = pd;
                    Ebr[t] = Eb + kmx[t] + up;
                    kx[t] = k;
                }
                __syncwarp();
                Eb = Ebr[t] + k;
                affine(t, fw_exp2(1.f, -k));
                pd = fw_exp2(pd, -k);
            }
            // t = 0: P and the dud counts
            weights(0);
            for (int h = 0; h < NC; h++) {
                const int j = 32 * h + lane;
                if (j < S) {
                    const float w = wv[j];
                    float b = w * in_a(XA[j], HB ? XB[j] : 0.f);
                    if (HB) {
                        const float bb = w * fmaf(q, XB[j], o);
                        ib = fmaf(dud0[j], bb, ib);
                        b = (1.f - m.p_ib) * b + m.p_ib * bb;
                    } else {
                        b *= 1.f - m.p_ib;
                    }
                    const float v = dud0[j] * b;
                    Ps += v;
                    const uint32_t pk = coord[j];
#pragma unroll
                    for (int c = 0; c < C; c++)
                        dudn[c] = fmaf((float)(a.D[c] - (int)((pk >> (4 * c)) & 15u)), v, dudn[c]);
                }
            }
            Ps = fw_sum(Ps);
            if (HB) ib = fw_sum(ib);
        }
        const bool live = !dead && Ps > 0.f;
        int EP = 0;
        float Pm = 0.f;
        if (live) {
            Pm = frexpf(Ps, &EP);
            EP += Eb + kmx[0];
        }
        if (a.logp) {
            if (lane == lp_n) {
                lp_m = live ? (double)Pm : 0.0;
                lp_e = EP;
                lp_at = ro;
            }
            if (++lp_n == 32) flush_logp();
        }
        if (!live) continue;
        const double invP = 1.0 / (double)Pm;
        double tsum = 0.0;  // times P

        // ---- forward sweep with the expected counts
        float fpd = 0.f;
        int Ea = kmx[0] - FW_TOP, kf;
        {
            float mx = 0.f;
            for (int j = lane; j < S; j += 32) {
                const float v = wv[j] * (dud0[j] * 0x1p96f);
                FA[j] = (1.f - m.p_ib) * v;
                if (HB) FB[j] = m.p_ib * v;
                mx = fmaxf(mx, v);
            }
            kf = fw_expo(fw_max(mx)) - FW_TOP;
        }
        // the same as above for the forward vector of n states
        auto bring_up = [&](int n) {
            if (kf >= FW_LOW) return;
            __syncwarp();
            for (int i = lane; i < n; i += 32) {
                FA[i] = fw_exp2(FA[i], -kf);
                if (HB) FB[i] = fw_exp2(FB[i], -kf);
            }
            __syncwarp();
            fpd = fw_exp2(fpd, -kf);
            Ea += kf;
            kf = 0;
        };
        bring_up(S);
        // emission statistics at t from the column products g in colv and the
        // detached state's gd, both in the frame 2^e / P
        auto emission = [&](int t, float gd, int e) {
            __syncwarp();
            const double sc = invP * fw_exp2d(e - EP);
            for (int b = lane; b < L.wsum; b += 32) {
                int c = 0, n = b;
#pragma unroll
                for (int k = 0; k < C - 1; k++)
                    if (c == k && n >= W[k]) {
                        n -= W[k];
                        c = k + 1;
                    }
                int s = 1, w = 1;
#pragma unroll
                for (int k = 0; k < C; k++)
                    if (k == c) {
                        s = st[k];
                        w = W[k];
                    }
                float g = n == 0 ? gd : 0.f;
                for (int hi = 0; hi < S; hi += s * w)
                    for (int lo = 0; lo < s; lo++) g += colv[hi + n * s + lo];
                const double x = a.rads[(r * T + t) * C + c], gs = (double)g * sc;
                acc[fw_emis(T, C, 0, c, n)] += gs;
                acc[fw_emis(T, C, 1, c, n)] += gs * x;
                acc[fw_emis(T, C, 2, c, n)] += gs * x * x;
            }
            __syncwarp();
        };
        if (T > 1) {  // x_1
            const float* src = x_at(1);
            for (int i = lane; i < S; i += 32) {
                XA[i] = src[i];
                if (HB) XB[i] = src[S + i];
            }
        }
        __syncwarp();
        for (int t = 1; t < T; t++) {
            const float p = m.p_det[t - 1], keep = 1.f - p;
            const float pdt = pdx[t];
            const int fr = Ea + Ebr[t] - EP;  // frame of f times backward values here
            float sum[NR];
#pragma unroll
            for (int i = 0; i < NR; i++) sum[i] = 0.f;
            // detachment, block and bleach sums, column by column
            float Fnz = 0.f, F0 = 0.f, Gnz = 0.f, G0 = 0.f, Fa = 0.f, Gaa = 0.f, Gab = 0.f;
            for (int h = 0; h < NC; h++) {
                const int j = 32 * h + lane;
                if (j < S) {
                    float fs = 0.f, H = 0.f, K[C];
#pragma unroll
                    for (int c = 0; c < C; c++) K[c] = 0.f;
                    for (int e = 0; e < t; e++) {
                        const int i = e * S + j;
                        float f = FA[i];
                        const float x = XA[i];
                        if (HB) {
                            const float xb = XB[i];
                            Fa += f;
                            Gaa = fmaf(f, x, Gaa);
                            Gab = fmaf(f, xb, Gab);
                            const float fb = fmaf(m.p_cb, f, FB[i]);
                            f *= 1.f - m.p_cb;
                            FA[i] = f;
                            FB[i] = fb;
                            fs += fb;
                            H = fmaf(fb, xb, H);
#pragma unroll
                            for (int c = 0; c < C; c++) K[c] = fmaf(fb, XB[i - st[c]], K[c]);
                        }
                        fs += f;
                        H = fmaf(f, x, H);
#pragma unroll
                        for (int c = 0; c < C; c++) K[c] = fmaf(f, XA[i - st[c]], K[c]);
                    }
                    const uint32_t pk = coord[j];
#pragma unroll
                    for (int c = 0; c < C; c++) {
                        const float n = (float)((pk >> (4 * c)) & 15u);
                        sum[6 + 2 * c] = fmaf(n, n != 0.f ? K[c] : 0.f, sum[6 + 2 * c]);
                        sum[7 + 2 * c] = fmaf(n, H, sum[7 + 2 * c]);
                    }
                    if (j == 0) {
                        F0 = fs;
                        G0 = H;
                    } else {
                        Fnz += fs;
                        Gnz += H;
                    }
                    if (a.emission) colv[j] = fmaf(keep, H, p * pdt * fs);
                }
            }
            if (a.emission) emission(t - 1, fpd * pdt, Ea + Ebr[t]);
            // a timestep's constants are multiplied into the sums one by one: folded
            // into one FP32 factor they would bias every term alike
#pragma unroll
            for (int c = 0; c < 2 * C; c++) sum[6 + c] *= keep;
            // (F0, G0: lane 0's, zero in the others)
            sum[0] = p * pdt * Fnz;
            sum[1] = fmaf(keep, Gnz, sum[0]);
            sum[3] = Fnz + F0;
            if (HB) {
                const float gb = fmaf(keep, Gab, p * pdt * Fa), ga = fmaf(keep, Gaa, p * pdt * Fa);
                sum[2] = fmaf(1.f - m.p_cb, ga, m.p_cb * gb);
                sum[NV - 1] = m.p_cb * gb;
            } else {
                sum[2] = (1.f - m.p_cb) * fmaf(keep, Gnz + G0, p * pdt * sum[3]);
            }
            __syncwarp();
            // the next chain's backward vector
            if (t + 1 < T) {
                const float* src = x_at(t + 1);
                const int n = (t + 1) * S;
                for (int i = lane; i < n; i += 32) {
                    XA[i] = src[i];
                    if (HB) XB[i] = src[n + i];
                }
                affine(t + 1, fw_exp2(1.f, -kx[t + 1]));
            } else {
                q = 0.f;
                o = cb0 = 1.f;
                cb1 = 0.f;
            }
#pragma unroll
            for (int c = 0; c < C; c++)
                if (W[c] > 1) {
                    fw_binomial<true, false>(FA, t * S, W[c], st[c], magic[c], bleach + boff[c], lane, nullptr);
                    if (HB) fw_binomial<true, false>(FB, t * S, W[c], st[c], magic[c], bleach + boff[c], lane, nullptr);
                    __syncwarp();
                }
            weights(t);
            // The cut and the emission, rows 0 .. t from 0 .. t - 1 (the forward
            // vector's scale goes into the weights), and with them the Edman sums: f
            // before the cut times the backward vector behind a failed and a
            // successful one.
            const float sc = fw_exp2(1.f, -kf);
            float mx = 0.f, en = 0.f, ed = 0.f;
            for (int h = 0; h < NC; h++) {
                const int j = 32 * h + lane;
                const bool on = j < S;
                const float wj = on ? wv[j] : 0.f, w = wj * keep * sc;
                const uint32_t pk = on ? coord[j] : 0u;
                float cur = 0.f, enj = 0.f, edj = 0.f;
                float next = wj * in_a(XA[t * S + j], HB ? XB[t * S + j] : 0.f);
                for (int e = t; e >= 0; e--) {
                    float v = pf * cur;
                    float prev = 0.f;
                    if (e > 0) {
                        const int k = (e - 1) * S + j, ch = e_ch[e - 1], s = ch & 0xffff;
                        prev = FA[k];
                        const float b = wj * in_a(XA[k], HB ? XB[k] : 0.f);
                        enj = fmaf(prev, b, enj);
                        float y;
                        if (s) {
                            const int n = (int)((pk >> (ch >> 16)) & 15u);
                            const float2* ec = e_cut + (e - 1) * L.cuts + n;
                            const float d3 = wv[j - s] * in_a(XA[k + S - s], HB ? XB[k + S - s] : 0.f);
                            y = fmaf(ec[0].x, next, ec[0].y * d3);
                            v = fmaf(ec[0].x, prev, v);
                            // from the state one dye up, if the channel has that many
                            if (n < a.D[ch >> 18]) v = fmaf(ec[1].y, FA[k + s], v);
                        } else {
                            y = qf * next;
                            v = fmaf(qf, prev, v);
                        }
                        edj = fmaf(prev, y, edj);
                        next = b;
                    }
                    v *= w;
                    __syncwarp();
                    if (on) FA[e * S + j] = v;
                    mx = fmaxf(mx, v);
                    if (HB && on) {
                        const float vb = e < t ? w * FB[e * S + j] : 0.f;
                        FB[e * S + j] = vb;
                        mx = fmaxf(mx, vb);
                    }
                    cur = prev;
                }
                if (on && j > 0) {
                    en += enj;
                    ed += edj;
                }
                __syncwarp();
            }
            sum[4] = pf * (keep * en);
            sum[5] = fmaf(keep, ed, sum[4]);
            const float mine_v = fw_sums<NR>(sum, lane);
            if (lane < 2) (lane == 0 ? dx : dn)[t - 1] = mine_v;
            if (lane == 0) dfr[t - 1] = fr;
            // (the Edman sums' backward vectors are those before x_t was brought up)
            const int fe = Ea + kmx[t] - EP + (t + 1 < T ? Ebr[t + 1] + kx[t + 1] : 0);
            tsum = fma((double)mine_v, fw_exp2d((lane & ~1) == 4 ? fe : fr), tsum);
            fpd = wv[0] * sc * fmaf(p, __shfl_sync(0xffffffffu, mine_v, 3), fpd);
            Ea += kf + kmx[t];
            kf = fw_expo(fw_max(fmaxf(mx, fpd))) - FW_TOP;
            bring_up((t + 1) * S);
        }
        if (a.emission) {
            __syncwarp();
            for (int j = lane; j < S; j += 32) {
                float s = 0.f;
                for (int e = 0; e < T; e++) s += HB ? FA[e * S + j] + FB[e * S + j] : FA[e * S + j];
                colv[j] = s;
            }
            emission(T - 1, fpd, Ea);
        }
        // ---- the read's sums into the warp's: value i in lane i
        {
            float mine_v = 0.f;
            double mine_q = 1.0;
            int slot = -1;
            auto put = [&](int i, int s, float v, double q = 1.0) {
                if (lane == i) {
                    mine_v = v;
                    mine_q = q;
                    slot = s;
                }
            };
            const double fp = invP * fw_exp2d(Eb + kmx[0] - EP);  // frame of P
            if (HB) put(2, 2, m.p_ib * ib, fp);
            put(3, 3, 1.f);
#pragma unroll
            for (int c = 0; c < C; c++) {
                put(8 + 4 * c, fw_rate(T, c) + 2, fw_sum(dudn[c]), fp);
                put(9 + 4 * c, fw_rate(T, c) + 3, (float)a.D[c]);
            }
            if (slot >= 0) acc[slot] += (double)mine_v * mine_q;
            all_reads = fma(tsum, invP, all_reads);
            for (int t = lane; t < T - 1; t += 32) {
                const double f = invP * fw_exp2d(dfr[t]);
                acc[fw_det(t)] += (double)dx[t] * f;
                acc[fw_det(t) + 1] += (double)dn[t] * f;
            }
            __syncwarp();
        }
    }
    flush_logp();
    {
        const int i = lane;
        if (i == 2) acc[5] += all_reads;
        if (i == 4 || i == 5) acc[i - 4] += all_reads;
        if (i >= 6 && i < 6 + 2 * C) {
            const int c = (i - 6) >> 1;
            acc[fw_rate(T, c) + (i & 1)] += (i & 1) ? all_reads : all_reads * m.q_bleach[c];
        }
        if (HB && i == NV - 1) acc[4] += all_reads;
    }
    __syncthreads();
    // the CTA's sums, its warps in order
    for (int k = threadIdx.x; k < a.nslots; k += blockDim.x) {
        double s = 0.0;
        for (int w = 0; w < wpc; w++)
            s += reinterpret_cast<double*>(fw_smem + L.shared + (size_t)(w + 1) * L.per_warp - 2 * a.nslots)[k];
        a.sums[(long)k * gridDim.x + blockIdx.x] = s;
    }
}

size_t wp_fit_warp_smem_bytes(int T, int C, const int* D, bool hb, bool emission, int nslots, int warps) {
    const FWLayout L = fw_layout(T, C, D, hb, emission, nslots);
    return sizeof(float) * ((size_t)L.shared + (size_t)warps * L.per_warp);
}

// Floats of one warp's slab: x_t of t rows, t = 1 .. T - 1.
long wp_fit_warp_slab_floats(int T, int S, bool hb) { return (hb ? 2l : 1l) * S * ((long)T * (T - 1) / 2); }

template <int C, bool HB>
static const void* fw_kernel() {
    return reinterpret_cast<const void*>(wp_fit_warp_kernel<C, HB>);
}

static const void* fw_pick(int C, bool hb) {
    switch (C) {
        case 1: return hb ? fw_kernel<1, true>() : fw_kernel<1, false>();
        case 2: return hb ? fw_kernel<2, true>() : fw_kernel<2, false>();
        case 3: return hb ? fw_kernel<3, true>() : fw_kernel<3, false>();
        case 4: return hb ? fw_kernel<4, true>() : fw_kernel<4, false>();
    }
    return nullptr;
}

int wp_fit_warp_max_warps() { return FW_WARPS; }

// Dyes of a channel up to which its fibres are processed in registers.
int wp_fit_warp_register_dyes() { return FW_MAXW - 1; }

// Resident CTAs per SM (0: the shape does not fit).
int wp_fit_warp_ctas_per_sm(int C, bool hb, size_t smem, int warps) {
    const void* k = fw_pick(C, hb);
    if (!k) return 0;
    int n = 0, sms = 0;
    if (wp_launch_shape(k, warps * 32, smem, &n, &sms) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n;
}

cudaError_t wp_launch_fit_warp(int C, bool hb, int grid, int warps, size_t smem, cudaStream_t s, const FitArgs& a,
                               float* slab, long slab_stride) {
    const void* k = fw_pick(C, hb);
    if (!k) return cudaErrorInvalidValue;
    FitArgs args = a;
    void* p[] = {&args, &slab, &slab_stride};
    int per_sm = 0, sms = 0;
    const cudaError_t e = wp_launch_shape(k, warps * 32, smem, &per_sm, &sms);
    if (e != cudaSuccess) return e;
    return cudaLaunchKernel(k, dim3(grid), dim3(warps * 32), p, smem, s);
}
