// wp_coop.cu -- the pair engine for pairs with large boxes: G lanes per
// (read, peptide) pair.
//
// wp_engine.cu gives each pair to one thread and each thread its own slab of
// shared memory, so the larger a pair's box the fewer threads fit an SM: at
// 430 states 64 of them, two warps, each a chain of dependent shared-memory
// loads.  Here G lanes share one pair and one slab, so the same shared
// memory keeps G times as many lanes in flight.  A state's arithmetic is the
// thread engine's, operation by operation, and the sum over the states that
// sets each timestep's rescale is formed in its order, so a pair's result
// has the same bits whichever kernel it goes to.
//
// Per timestep: the bleach steps with a lane per column (all states along
// the channel), Edman and emission with a lane per (state, slice), and the
// sum as one lane's serial chain, its odd slices' partial sums made by all
// lanes beforehand.  What a state needs of its own (its place in the
// bleached box, its packed dye counts, its emission factor) is worked out
// once, into a table of WP_COOP_STATES entries in shared memory; larger
// boxes go through it in chunks.
//
// Bound by issue slots, about three times the thread engine's per pair (the
// state table, index work per element and the serial sums): pays where the
// thread engine leaves an SM with 4 warps or fewer.  400 reads x 200
// peptides, 3 channels, 16 timesteps, no pruning: the two passes for boxes
// of 108 to 442 states 7.9 ms with a thread per pair, 1.06 here.
//
// The groups of a warp are pairs of one read or of neighbouring reads and
// move in step: every phase ends in a whole-warp __syncwarp, and a pair that
// has finished (or was never there) sits out its phases.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "wp_common.cuh"
#include "wp_engine.cuh"

#define WP_COOP_THREADS 128
#define WP_COOP_STATES 32  // states per chunk of the state table
#define WP_COOP_IDX 512    // largest slab half (index arithmetic below)

// One state of the chunk: X (packed counts, bit 7 of byte c: the bleached
// box has the state one dye up in channel c), its index in a slice of the
// bleached box, its emission factor and its second partial sum.
struct CoopState {
    uint32_t X;
    int ib;
    float w;
    float part2;
};

// x / d for x < WP_COOP_IDX, 1 <= d <= WP_COOP_IDX, rcp[d] = ceil(2^20 / d):
// exact, as x (rcp[d] d - 2^20) < x d <= 2^18 < 2^20.
__device__ __forceinline__ int cdiv20(int x, uint32_t r) { return (int)(((uint32_t)x * r) >> 20); }

// binomial_step (wp_engine.cu) with the columns over the group's lanes.  K:
// columns at most K states on both sides, in registers (0: any).
template <int K, class V>
__device__ __forceinline__ void coop_columns(const V* __restrict__ src, V* __restrict__ dst, int gl, int G, int ncol,
                                             int inner, uint32_t rin, int win, int wout, int from0, int to0,
                                             const float* __restrict__ tab) {
    if constexpr (K > 0) {
        float cf[K][K];
        const int d = from0 - to0;
#pragma unroll
        for (int k = 0; k < K; k++) {
            const int from = from0 + k;
            const int rb = from * (from + 1) / 2 + to0;
#pragma unroll
            for (int k2 = 0; k2 < K; k2++)
                cf[k2][k] = (k < win && k2 < wout && d + k - k2 >= 0) ? tab[rb + k2] : 0.0f;
        }
        for (int q = gl; q < ncol; q += G) {
            const int o = cdiv20(q, rin), i = q - o * inner;
            const V* s = src + o * win * inner + i;
            V* w = dst + o * wout * inner + i;
            V x[K];
#pragma unroll
            for (int k = 0; k < K; k++) x[k] = k < win ? s[k * inner] : vzero(V());
#pragma unroll
            for (int k2 = 0; k2 < K; k2++)
                if (k2 < wout) {
                    V acc = vmul(cf[k2][0], x[0]);
#pragma unroll
                    for (int k = 1; k < K; k++) acc = vfma(cf[k2][k], x[k], acc);
                    w[k2 * inner] = acc;
                }
        }
    } else {
        for (int q = gl; q < ncol; q += G) {
            const int o = cdiv20(q, rin), i = q - o * inner;
            const V* s = src + o * win * inner + i;
            V* w = dst + o * wout * inner + i;
            for (int k2 = 0; k2 < wout; k2++) {
                const int to = to0 + k2;
                V acc = vzero(V());
                for (int k = max(0, to - from0); k < win; k++) {
                    const int from = from0 + k;
                    acc = vfma(tab[from * (from + 1) / 2 + to], s[k * inner], acc);
                }
                w[k2 * inner] = acc;
            }
        }
    }
}

template <int C, bool HB, int G>
__global__ void __launch_bounds__(WP_COOP_THREADS) wp_coop_kernel(BatchArgs a, EngineLists L) {
    using V = typename StateOf<HB>::V;
    constexpr int NP = 32 / G;  // pairs per warp
    constexpr unsigned FULL = 0xffffffffu;
    const int count = *L.in_count;
    if (count == 0) return;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    SmemModel& M = *reinterpret_cast<SmemModel*>(smem_raw);
    const DevModel& m = *a.model;
    load_smem_model(M, m);
    uint32_t* rcp = reinterpret_cast<uint32_t*>(smem_raw + ((sizeof(SmemModel) + 15) & ~(size_t)15));
    for (int d = threadIdx.x; d <= WP_COOP_IDX; d += blockDim.x)
        rcp[d] = d ? ((1u << 20) + (uint32_t)d - 1u) / (uint32_t)d : 0u;
    __syncthreads();
    const int lane = threadIdx.x & 31, gl = lane & (G - 1), grp = threadIdx.x / G;
    const int half = L.slab_half;
    unsigned char* pair_base = reinterpret_cast<unsigned char*>(rcp + ((WP_COOP_IDX + 1 + 3) & ~3));
    const size_t pair_bytes = sizeof(CoopState) * WP_COOP_STATES + WP_ENGINE_CODES +
                              (((size_t)2 * half * sizeof(V) + 15) & ~(size_t)15);
    pair_base += pair_bytes * grp;
    CoopState* st = reinterpret_cast<CoopState*>(pair_base);
    uint8_t* codes = pair_base + sizeof(CoopState) * WP_COOP_STATES;
    V* const slab = reinterpret_cast<V*>(codes + WP_ENGINE_CODES);
    // model scalars
    const int T = m.T;
    const float pf = m.pf, qf = 1.0f - m.pf;
    const bool interacting = m.interacting != 0;
    const bool pk = T <= 17;
    const int W = a.W;
    const int IG = interacting ? wp_ipow(W, C) : 0;

    for (;;) {
        int base = 0;
        if (lane == 0) base = atomicAdd(L.in_head, NP);
        base = __shfl_sync(FULL, base, 0);
        if (base >= count) break;
        const int wi = base + lane / G;
        bool run = wi < count;
        const int2 rg = L.in[run ? wi : base];
        int vmax;
        const int p = slot_pep(a, rg.x, item_slot(a, rg, &vmax));
        if (run && vmax > half) {
            // not routed here by the compaction: to the next list
            if (gl == 0) {
                if (L.spill_error) {
                    atomicExch(a.err, 2);
                    a.res_mant[rg.y] = 0.0f;
                    a.res_expo[rg.y] = 0;
                } else {
                    const int q = atomicAdd(L.out_count, 1);
                    L.out[q] = rg;
                }
            }
            run = false;
        }
        const PeptideRec& pep = a.peps[p];
        const int r = rg.x;
        const EmitEntry* tab = a.tab + (long)r * a.entries;
        ReadEmit re;
        re.tab = tab;
        re.W = W;
        re.gt = a.gtab ? a.gtab + (long)r * a.entries : nullptr;
        re.gd = a.gdelta ? a.gdelta + (long)r * a.entries : nullptr;
        const int* gKr = a.gtab ? a.gK + (long)r * T : nullptr;
        const float4* gOr = a.gone ? a.gone + (long)r * T : nullptr;
        const uint32_t* Lpk = a.Lpk + (long)r * T;
        const uint32_t* Upk = a.Upk + (long)r * T;
        uint32_t D1 = 0;
#pragma unroll
        for (int c = 0; c < C; c++) D1 = bset(D1, c, pep.D[c] + 1);
        const uint64_t dye_pk = pep.dye_pk, tot_pk = pep.tot_pk;
        if (pk)
            for (int k = gl; k < WP_ENGINE_CODES; k += G)
                codes[k] = (uint8_t)(pep.ecode[k >> 3] >> (8 * (k & 7)));

        V* cur = slab;
        V* nxt = slab + half;
        PBox bx;
        bx.lo = 0;
        bx.w = 0;
        float bscale = 1.0f;
        int expo = 0;
        float pd = 0.0f;
        int k_prev = 0;
        float scale_prev = 1.0f, fac_prev = 1.0f;
        const float4 one_none = make_float4(0.0f, 0.0f, 0.0f, __int_as_float(WP_GK_NONE));

        for (int t = 0; t < T; t++) {
            // ---- this timestep's emission box [L_t, min(U_t, D + 1))
            const uint32_t lw = Lpk[t], uw = Upk[t];
            const int gk = gKr ? gKr[t] : WP_GK_NONE;
            const float4 one = gOr ? gOr[t] : one_none;
            PBox nx;
            nx.lo = lw & 0x7f7f7f7fu;
            const uint32_t msk = ((((uw | 0x80808080u) - D1) >> 7) & 0x01010101u) * 0xffu;
            nx.w = ((D1 & msk) | (uw & ~msk)) - nx.lo;
            const bool allow_t = (lw >> 31) != 0;
            const bool narrow = !interacting && ((nx.w + 0x7b7b7b7bu) & 0x80808080u) == 0;
            const int vn = run ? bvol<C>(nx.w) : 0;
            if (t == 0) {
                // start state, initial block and duds, straight into the box
                bx = nx;
                for (int j = gl; j < vn; j += G) {
                    V s;
                    if constexpr (HB) {
                        s = make_float2(1.0f - m.p_ib, m.p_ib);
                    } else {
                        s = 1.0f;
                    }
                    int jc[C];
                    int x = j;
#pragma unroll
                    for (int c = C - 1; c >= 0; c--) {
                        const int w = bget(nx.w, c);
                        const int q = cdiv20(x, rcp[w]);
                        jc[c] = x - q * w;
                        x = q;
                    }
#pragma unroll
                    for (int c = 0; c < C; c++) {
                        const int d = pep.D[c], n = bget(nx.lo, c) + jc[c];
                        s = vmul(M.dud[c][d * (d + 1) / 2 + n], s);
                    }
                    cur[j] = s;
                }
                __syncwarp();
            } else {
                bscale = 1.0f;
                if constexpr (HB) {
                    if (m.p_cb != 0.0f) {
                        const int n = run ? t * bvol<C>(bx.w) : 0;
                        for (int i = gl; i < n; i += G) {
                            const float2 s = cur[i];
                            cur[i] = make_float2((1.0f - m.p_cb) * s.x, s.y + m.p_cb * s.x);
                        }
                        __syncwarp();
                    }
                }
                // ---- bleach, one channel after another
                const bool fold = (bx.w & chan_mask<C>()) == (0x01010101u & chan_mask<C>()) &&
                                  ((bx.lo ^ nx.lo) & chan_mask<C>()) == 0;
                if (fold) {
#pragma unroll
                    for (int c = 0; c < C; c++) {
                        const int l = bget(nx.lo, c);
                        bscale *= M.bleach[c][l * (l + 3) / 2];
                    }
                }
#pragma unroll 1
                for (int c = 0; c < C; c++) {
                    bool pass = false;
                    if (run && !fold) {
                        const int ln = bget(nx.lo, c);
                        const int lo = bget(bx.lo, c), win = bget(bx.w, c);
                        const int wout = min(ln + bget(nx.w, c) + 1, lo + win) - ln;
                        if (win == 1 && wout == 1) {
                            bscale *= lo >= ln ? M.bleach[c][lo * (lo + 1) / 2 + ln] : 0.0f;
                        } else {
                            int outer = t, inner = 1;
#pragma unroll
                            for (int c2 = 0; c2 < C; c2++) {
                                const int w = bget(bx.w, c2);
                                if (c2 < c) outer *= w;
                                if (c2 > c) inner *= w;
                            }
                            const uint32_t rin = rcp[inner];
                            if (win <= 2 && wout <= 2)
                                coop_columns<2, V>(cur, nxt, gl, G, outer * inner, inner, rin, win, wout, lo, ln,
                                                   M.bleach[c]);
                            else if (win <= 4 && wout <= 4)
                                coop_columns<4, V>(cur, nxt, gl, G, outer * inner, inner, rin, win, wout, lo, ln,
                                                   M.bleach[c]);
                            else
                                coop_columns<0, V>(cur, nxt, gl, G, outer * inner, inner, rin, win, wout, lo, ln,
                                                   M.bleach[c]);
                            pass = true;
                        }
                        bx.lo = bset(bx.lo, c, ln);
                        bx.w = bset(bx.w, c, wout);
                    }
                    __syncwarp();
                    if (pass) {
                        V* tmp = cur;
                        cur = nxt;
                        nxt = tmp;
                    }
                }
            }
            // ---- emission factors of the box: narrow, per channel in
            // registers, else from the table per state
            const bool fused = t > 0 && pk && narrow && (C <= 3 || bvol<C>(bx.w) <= 255);
            float g[C][4];
            int kmax = 0;
            float em0 = 0.0f;
            bool zero = false;
            if (run && narrow) {
                zero = !narrow_factors<C>(re, gk, one, t, nx, g, &kmax);
                if (allow_t) {
                    em0 = 1.0f;
#pragma unroll
                    for (int c = 0; c < C; c++) em0 *= g[c][0];
                }
            } else if (run) {
                float mm = 1.0f;
                int ks = 0;
                if (!interacting) {
#pragma unroll
                    for (int c = 0; c < C; c++) {
                        const EmitEntry* row = tab + (t * C + c) * W + bget(nx.lo, c);
                        int km = WP_EXPO_ZERO;
                        for (int k = 0; k < bget(nx.w, c); k++)
                            if (row[k].mant != 0.0f) km = max(km, row[k].expo);
                        if (km == WP_EXPO_ZERO) zero = true;
                        kmax += km;
                        const EmitEntry en = tab[(t * C + c) * W];
                        mm *= en.mant;
                        ks += en.expo;
                    }
                } else {
                    kmax = WP_EXPO_ZERO;
                    for (int j = 0; j < vn; j++) {
                        int gi = 0, x = j, mul = 1;
#pragma unroll
                        for (int c = C - 1; c >= 0; c--) {
                            const int w = bget(nx.w, c);
                            const int q = cdiv20(x, rcp[w]);
                            gi += (bget(nx.lo, c) + x - q * w) * mul;
                            mul *= W;
                            x = q;
                        }
                        const EmitEntry en = tab[t * IG + gi];
                        if (en.mant != 0.0f) kmax = max(kmax, en.expo);
                    }
                    zero = kmax == WP_EXPO_ZERO;
                    const EmitEntry en = tab[t * IG];
                    mm = en.mant;
                    ks = en.expo;
                }
                em0 = mm != 0.0f && allow_t ? mm * exp2i(max(ks - kmax, -200)) : 0.0f;
            }
            if (run && zero) {
                if (gl == 0) {
                    a.res_mant[rg.y] = 0.0f;
                    a.res_expo[rg.y] = 0;
                }
                run = false;
            }
            const int nst = run ? vn : 0;  // states to go through
            // strides of the bleached box
            int stb[C];
            int vb = 1;
#pragma unroll
            for (int c = C - 1; c >= 0; c--) {
                stb[c] = vb;
                vb *= bget(bx.w, c);
            }
            // failure plus success, rounded as edman_emit does (one rounding)
            // or as edman_gather (the product first)
            auto keep = [&](float x, float y, float z) {
                return fused ? fmaf(x, y, z) : __fadd_rn(__fmul_rn(x, y), z);
            };
            const float sf = fac_prev * bscale * scale_prev;
            const float sft = fac_prev * bscale;
            float part = 0.0f;
            for (int j0 = 0; __any_sync(FULL, j0 < nst); j0 += WP_COOP_STATES) {
                const int cn = max(0, min(WP_COOP_STATES, nst - j0));
                // the chunk's states
                for (int jj = gl; jj < cn; jj += G) {
                    CoopState s;
                    s.X = nx.lo;
                    s.ib = 0;
                    s.part2 = 0.0f;
                    int x = j0 + jj;
                    int jc[C];
#pragma unroll
                    for (int c = C - 1; c >= 0; c--) {
                        const int w = bget(nx.w, c);
                        const int q = cdiv20(x, rcp[w]);
                        const int k = x - q * w;
                        x = q;
                        jc[c] = k;
                        s.X += (uint32_t)k << (8 * c);
                        if (k + 1 < bget(bx.w, c)) s.X |= 0x80u << (8 * c);
                        s.ib += k * stb[c];
                    }
                    if (narrow) {
                        float w = sf;
#pragma unroll
                        for (int c = 0; c < C; c++) {
                            const int k = jc[c];
                            w *= k == 0 ? g[c][0] : k == 1 ? g[c][1] : k == 2 ? g[c][2] : g[c][3];
                        }
                        s.w = w;
                    } else {
                        float mm = sft;
                        int ks = 0;
                        if (!interacting) {
#pragma unroll
                            for (int c = 0; c < C; c++) {
                                const EmitEntry en = tab[(t * C + c) * W + bget(nx.lo, c) + jc[c]];
                                mm *= en.mant;
                                ks += en.expo;
                            }
                        } else {
                            int gi = 0;
#pragma unroll
                            for (int c = 0; c < C; c++) gi = gi * W + bget(nx.lo, c) + jc[c];
                            const EmitEntry en = tab[t * IG + gi];
                            mm *= en.mant;
                            ks = en.expo;
                        }
                        s.w = mm != 0.0f ? mm * exp2i(max(ks - kmax - k_prev, -200)) : 0.0f;
                    }
                    st[jj] = s;
                }
                __syncwarp();
                // Edman and emission, a lane per (slice, state)
                if (t == 0) {
                    for (int jj = gl; jj < cn; jj += G) cur[j0 + jj] = vmul(st[jj].w, cur[j0 + jj]);
                } else {
                    const int ne = (t + 1) * cn;
                    const uint32_t rc = rcp[max(cn, 1)];
                    for (int q = gl; q < ne; q += G) {
                        const int e = cdiv20(q, rc), jj = q - e * cn;
                        const uint32_t X = st[jj].X;
                        const int ib = st[jj].ib;
                        const float w = st[jj].w;
                        const V* col = cur + e * vb + ib;  // slice e of the state's column
                        float add = 0.0f;
                        if (e >= 1) {
                            const V* sp = col - vb;
                            float xin;
                            if constexpr (HB) {
                                xin = sp->x;
                            } else {
                                xin = *sp;
                            }
                            float cx, cy;
                            uint32_t up;
                            int sd;
                            if (pk) {
                                const uint32_t code = codes[e - 1];
                                const uint32_t b = prmt(X, 0u, code);
                                const int ci = (int)(b & 0x7fu) * 17 + (int)(code >> 4);
                                cx = M.edx[ci];
                                cy = M.edy[ci];
                                up = b & 0x80u;
                                sd = (int)(code & 7u);
                            } else {
                                const int dc = pep.dye[e - 1];
                                sd = dc < 0 ? 4 : dc;
                                const uint32_t b = prmt(X, 0u, (uint32_t)sd);
                                const int ci = (int)(b & 0x7fu) * 17 + (dc < 0 ? 0 : pep.tot[e - 1]);
                                cx = dc < 0 ? qf : M.edx[ci];
                                cy = M.edy[ci];
                                up = b & 0x80u;
                            }
                            add = cx * xin;
                            if (up) {
                                int so = 0;
#pragma unroll
                                for (int c = 0; c < C; c++)
                                    if (c == sd) so = stb[c];
                                if constexpr (HB) {
                                    add = fmaf(cy, sp[so].x, add);
                                } else {
                                    add = fmaf(cy, sp[so], add);
                                }
                            }
                        }
                        V v;
                        if (e == t) {
                            if constexpr (HB) {
                                v = make_float2(add, 0.0f);
                            } else {
                                v = add;
                            }
                        } else {
                            const V f = *col;
                            if constexpr (HB) {
                                v = make_float2(keep(pf, f.x, add), f.y);
                            } else {
                                v = keep(pf, f, add);
                            }
                        }
                        nxt[e * vn + j0 + jj] = vmul(w, v);
                    }
                }
                __syncwarp();
                V* const o = t == 0 ? cur : nxt;
                // the even slices' sums, a lane per state
                if (fused && t > 2)
                    for (int jj = gl; jj < cn; jj += G) {
                        float p2 = 0.0f;
                        const V* x = o + j0 + jj;
                        for (int e = 2; e < t; e += 2) p2 += vtotal(x[e * vn]);
                        st[jj].part2 = p2;
                    }
                __syncwarp();
                // the sum over the states, in the thread engine's order
                if (gl == 0) {
                    if (fused) {
                        for (int jj = 0; jj < cn; jj++) {
                            const V* x = o + j0 + jj;
                            part += vtotal(x[0]);
                            for (int e = 1; e < t; e += 2) part += vtotal(x[e * vn]);
                            part += st[jj].part2;
                            part += vtotal(x[t * vn]);
                        }
                    } else {
                        for (int jj = 0; jj < cn; jj++) {
                            const V* x = o + j0 + jj;
                            for (int e = 0; e <= t; e++) part += vtotal(x[e * vn]);
                        }
                    }
                }
                __syncwarp();
            }
            part = __shfl_sync(FULL, part, lane & ~(G - 1));
            if (t > 0) {
                V* tmp = cur;
                cur = nxt;
                nxt = tmp;
                bx = nx;
            }
            // ---- detached state, rescale and the next detach (close_step)
            if (run) {
                pd = allow_t ? pd * em0 : 0.0f;
                expo += kmax;
                const float tot = part + pd;
                if (!(tot > 0.0f) || !isfinite(tot)) {
                    if (gl == 0) {
                        a.res_mant[rg.y] = 0.0f;
                        a.res_expo[rg.y] = 0;
                    }
                    run = false;
                } else {
                    int k;
                    float fm;
                    const int bits = __float_as_int(tot);
                    if (bits >= 0x00800000) {
                        k = (bits >> 23) - 126;
                        fm = __int_as_float((bits & 0x007fffff) | 0x3f000000);
                    } else {
                        fm = frexpf(tot, &k);
                    }
                    if (t == T - 1) {
                        if (gl == 0) {
                            a.res_mant[rg.y] = fm;
                            a.res_expo[rg.y] = expo + k;
                        }
                    } else {
                        expo += k;
                        const float f = exp2i(-k);
                        pd = (pd + M.p_det[t] * part) * f;
                        k_prev = k;
                        scale_prev = f;
                        fac_prev = 1.0f - M.p_det[t];
                    }
                }
            }
            if (!__any_sync(FULL, run)) break;
        }
        __syncwarp();
    }
}

// Shared memory of one CTA: the model, the reciprocals and, per pair, the
// state table, the Edman codes and two slab halves.
size_t wp_coop_smem_bytes(int slab_half, bool has_block, int lanes) {
    const size_t elem = has_block ? sizeof(float2) : sizeof(float);
    const size_t pair = sizeof(CoopState) * WP_COOP_STATES + WP_ENGINE_CODES +
                        (((size_t)2 * slab_half * elem + 15) & ~(size_t)15);
    return ((sizeof(SmemModel) + 15) & ~(size_t)15) + sizeof(uint32_t) * ((WP_COOP_IDX + 1 + 3) & ~3) +
           pair * (WP_COOP_THREADS / lanes);
}

template <int C, bool HB, int G>
static cudaError_t launch_coop(cudaStream_t s, const BatchArgs& a, const EngineLists& L, long pairs) {
    const size_t smem = wp_coop_smem_bytes(L.slab_half, HB, G);
    int sms = 0, per_sm = 0;
    const cudaError_t e = wp_launch_shape(reinterpret_cast<const void*>(wp_coop_kernel<C, HB, G>), WP_COOP_THREADS,
                                          smem, &per_sm, &sms);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorInvalidConfiguration;
    constexpr int in_hand = WP_COOP_THREADS / G;  // pairs of a CTA
    const int grid = std::max(1, (int)std::min<long>((long)sms * per_sm, (pairs + in_hand - 1) / in_hand));
    wp_coop_kernel<C, HB, G><<<grid, WP_COOP_THREADS, smem, s>>>(a, L);
    return cudaGetLastError();
}

template <int C, bool HB>
static cudaError_t launch_coop_lanes(int lanes, cudaStream_t s, const BatchArgs& a, const EngineLists& L,
                                     long pairs) {
    switch (lanes) {
        case 8: return launch_coop<C, HB, 8>(s, a, L, pairs);
        case 16: return launch_coop<C, HB, 16>(s, a, L, pairs);
        default: return cudaErrorInvalidValue;
    }
}

// One pass over a work list of at most `pairs`, `lanes` lanes per pair (persistent
// grid).
cudaError_t wp_launch_coop(int C, bool has_block, int lanes, cudaStream_t s, const BatchArgs& a, const int2* in,
                           const int* in_count, int* in_head, int2* out, int* out_count, int slab_half,
                           int spill_error, long pairs) {
    if (slab_half > WP_COOP_IDX) return cudaErrorInvalidValue;
    EngineLists L{in, in_count, in_head, out, out_count, slab_half, 0, spill_error};
    switch (C * 2 + (has_block ? 1 : 0)) {
        case 2: return launch_coop_lanes<1, false>(lanes, s, a, L, pairs);
        case 3: return launch_coop_lanes<1, true>(lanes, s, a, L, pairs);
        case 4: return launch_coop_lanes<2, false>(lanes, s, a, L, pairs);
        case 5: return launch_coop_lanes<2, true>(lanes, s, a, L, pairs);
        case 6: return launch_coop_lanes<3, false>(lanes, s, a, L, pairs);
        case 7: return launch_coop_lanes<3, true>(lanes, s, a, L, pairs);
        case 8: return launch_coop_lanes<4, false>(lanes, s, a, L, pairs);
        case 9: return launch_coop_lanes<4, true>(lanes, s, a, L, pairs);
        default: return cudaErrorInvalidValue;
    }
}
