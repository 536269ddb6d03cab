// wp_engine.cuh -- what the pair engine's kernels share (wp_engine.cu: one
// thread per pair; wp_coop.cu: several lanes per pair): the state value, the
// packed box, a read's emission factors and a pass's lists.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "wp_common.cuh"

#define WP_ENGINE_CODES 16  // Edman code bytes per pair (positions 0..15)

template <bool HB>
struct StateOf;
template <>
struct StateOf<false> {
    using V = float;
};
template <>
struct StateOf<true> {
    using V = float2;
};

__device__ __forceinline__ float vzero(float) { return 0.0f; }
__device__ __forceinline__ float2 vzero(float2) { return make_float2(0.0f, 0.0f); }
__device__ __forceinline__ float vfma(float k, float v, float acc) { return fmaf(k, v, acc); }
__device__ __forceinline__ float2 vfma(float k, float2 v, float2 acc) {
    return make_float2(fmaf(k, v.x, acc.x), fmaf(k, v.y, acc.y));
}
__device__ __forceinline__ float vmul(float k, float v) { return k * v; }
__device__ __forceinline__ float2 vmul(float k, float2 v) { return make_float2(k * v.x, k * v.y); }
__device__ __forceinline__ float vtotal(float v) { return v; }
__device__ __forceinline__ float vtotal(float2 v) { return v.x + v.y; }

// Packed box: byte c of lo / w is channel c's lower corner / width.
struct PBox {
    uint32_t lo;
    uint32_t w;
};
__device__ __forceinline__ int bget(uint32_t v, int c) { return (int)((v >> (8 * c)) & 0xffu); }
// prmt.b32 in its default mode: byte n of the result is the byte of {y, x}
// (x: bytes 0-3, y: 4-7) that nibble n of s selects, its sign replicated
// where the nibble's bit 3 is set.
__device__ __forceinline__ uint32_t prmt(uint32_t x, uint32_t y, uint32_t s) {
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(x), "r"(y), "r"(s));
    return d;
}
__device__ __forceinline__ uint32_t bset(uint32_t v, int c, int x) {
    return (v & ~(0xffu << (8 * c))) | ((uint32_t)x << (8 * c));
}
// The bytes of a packed word that hold channels.
template <int C>
__device__ __forceinline__ uint32_t chan_mask() {
    return C >= 4 ? 0xffffffffu : (1u << (8 * C)) - 1u;
}

template <int C>
__device__ __forceinline__ int bvol(uint32_t w) {
    int v = 1;
#pragma unroll
    for (int c = 0; c < C; c++) v *= bget(w, c);
    return v;
}

// A read's emission factors as the engine reads them: the (mant, expo)
// table, and where present the window-normalised FP32 factors with their
// per-box exponent corrections (wp_prep_window_kernel).
struct ReadEmit {
    const EmitEntry* tab;  // [(t C + c) W + n]
    const float* gt;       // same layout, null when absent
    const uint8_t* gd;     // [(t C + c) W + u - 1]
    int W;
};

// Emission factors of the box nx at timestep t (at most 4 wide per channel,
// no interactions), per channel normalised by the box's largest exponent:
// g[c][k] for count L_c + k (0 beyond the box), and *kmax_out the sum of
// the normalising exponents.  gk is the (read, t)'s sum of window
// exponents: the window factors times 2^gdelta are these numbers exactly;
// with WP_GK_NONE they are normalised here from the table.  one: the
// (read, t)'s one-state factors (BatchArgs::gone).  Returns false
// when every factor of some channel is zero (only detected on the table
// path; on the other the zero factors give the pair P = 0 at this step's
// rescale).
template <int C>
__device__ __forceinline__ bool narrow_factors(const ReadEmit& re, int gk, float4 one, int t, PBox nx,
                                               float (&g)[C][4], int* kmax_out) {
    if constexpr (C <= 3) {
        // the read's box is one state in every channel: that state's factor
        // mantissas and exponent sum, as the two paths below would give
        if (__float_as_int(one.w) != WP_GK_NONE) {
            const float mv[3] = {one.x, one.y, one.z};
#pragma unroll
            for (int c = 0; c < C; c++) {
                g[c][0] = mv[c];
                g[c][1] = g[c][2] = g[c][3] = 0.0f;
            }
            *kmax_out = __float_as_int(one.w);
            return true;
        }
    }
    if (gk != WP_GK_NONE) {
        int kmax = gk;
#pragma unroll
        for (int c = 0; c < C; c++) {
            const int wc = bget(nx.w, c);
            const int base = (t * C + c) * re.W + bget(nx.lo, c);
            const int dl = re.gd[base + max(wc, 1) - 1];
            const float sc = exp2i(dl);
            const float* row = re.gt + base;
#pragma unroll
            for (int k = 0; k < 4; k++) g[c][k] = k < wc ? row[k] * sc : 0.0f;
            kmax -= dl;
        }
        *kmax_out = kmax;
        return true;
    }
    int kmax = 0;
#pragma unroll
    for (int c = 0; c < C; c++) {
        const EmitEntry* row = re.tab + (t * C + c) * re.W + bget(nx.lo, c);
        const int wc = bget(nx.w, c);
        EmitEntry en[4];
        int km = WP_EXPO_ZERO;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            en[k].mant = 0.0f;
            en[k].expo = WP_EXPO_ZERO;
            if (k < wc) en[k] = row[k];
            if (en[k].mant != 0.0f) km = max(km, en[k].expo);
        }
        if (km == WP_EXPO_ZERO) return false;
#pragma unroll
        for (int k = 0; k < 4; k++)
            g[c][k] = en[k].mant != 0.0f ? en[k].mant * exp2i(max(en[k].expo - km, -200)) : 0.0f;
        kmax += km;
    }
    *kmax_out = kmax;
    return true;
}

// Lists one engine pass reads and spills to.
struct EngineLists {
    const int2* in;
    const int* in_count;
    int* in_head;
    int2* out;
    int* out_count;
    int slab_half;
    int scr_floats;   // reserved per-thread scratch (floats), 0 when unused
    int spill_error;  // nonzero: nothing downstream takes spills; flag err
};
