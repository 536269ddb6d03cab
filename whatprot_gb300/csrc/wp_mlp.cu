// wp_mlp.cu -- the learned proposal network: an MLP from a radiometry
// (T*C intensities, zero-padded to 64) to logits over the peptide set,
//
//     x -> GELU(W1 x + b1) -> GELU(W2 h1 + b2) -> W3 h2 + b3     (1024 wide)
//
// with BF16 weights and activations and FP32 accumulation on the tensor
// cores (wp_gemm.cu), trained with softmax cross-entropy and Adam on reads
// simulated on the GPU (wp_sim.cu), used to propose the top-H peptides that
// the HMM then rescores, in place of the kNN stage of the hybrid classifier.
// The reference has no such network; this file has no reference
// counterpart.
//
// All products are C = A . B^T (wp_gemm_bf16); where an operand's reduction
// dimension is the strided one the tensor cores read it as it is (MN-major),
// so the backward pass needs no transposed copies:
//     dH2 = dL . W3         W3 [P][1024] MN-major
//     dW3 = dL^T . H2       both MN-major
//     dH1 = dZ2 . W2        W2 MN-major
//     dW2 = dZ2^T . H1      both
//     dW1 = dZ1^T . X       both
// Master weights, gradients and Adam moments are FP32.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <curand_kernel.h>
#include <math.h>
#include <stdint.h>

// wp_shape.cu
cudaError_t wp_launch_shape(const void* kernel, int threads, size_t smem, int* per_sm, int* sms);

typedef __nv_bfloat16 bf16;

// Radiometries (FP32 or FP64, [B][TC]) to BF16 inputs [B][64] (zero padded).
__global__ void wp_mlp_input_kernel(const float* __restrict__ xf, const double* __restrict__ xd, int B, int TC,
                                    bf16* __restrict__ X) {
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long)B * 64) return;
    const long b = i / 64;
    const int d = (int)(i % 64);
    float v = 0.f;
    if (d < TC) v = xf ? xf[b * TC + d] : (float)xd[b * TC + d];
    X[i] = __float2bfloat16_rn(v);
}

// Block-wide reductions in a fixed order (warp trees, then warp 0).
__device__ float block_max(float v, float* sh) {
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    __syncthreads();
    if (l == 0) sh[w] = v;
    __syncthreads();
    if (w == 0) {
        v = l < (int)(blockDim.x >> 5) ? sh[l] : -INFINITY;
        for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
        if (l == 0) sh[0] = v;
    }
    __syncthreads();
    return sh[0];
}

__device__ float block_sum(float v, float* sh) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    __syncthreads();
    if (l == 0) sh[w] = v;
    __syncthreads();
    if (w == 0) {
        v = l < (int)(blockDim.x >> 5) ? sh[l] : 0.f;
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (l == 0) sh[0] = v;
    }
    __syncthreads();
    return sh[0];
}

// One CTA per row: softmax over the first P logits, cross-entropy against
// the label (rows with label < 0 are skipped: loss 0, gradient 0; so are those
// with a label of P or more, which set *bad), and the
// logit gradient (softmax - onehot) * scale as BF16 (zero past P).  The row
// (ld a multiple of 4, 16-byte aligned) stays in shared memory, so HBM sees
// each logit once and each exponential is formed once.  Bound by issue slots and
// the phases' latency at two CTAs per SM.  4,096 rows of 20,032: 139 us, 158
// with the label compared at every element of 4-byte stores, 365 for three
// passes over global memory.  Rows beyond the shared memory (`keep` 0) are read
// again for each pass.
__global__ void __launch_bounds__(256) wp_softmax_ce_kernel(const float* __restrict__ logits, int P, int ld,
                                                            const int* __restrict__ labels, float scale,
                                                            bf16* __restrict__ dL, double* __restrict__ loss, int keep,
                                                            int* __restrict__ bad) {
    extern __shared__ __align__(16) float ce_row[];
    __shared__ float sh[32];
    const long row = blockIdx.x;
    const float* l = logits + row * ld;
    int y = labels[row];
    if (y >= P) {  // from the caller's memory: no class, and no index
        y = -1;
        if (threadIdx.x == 0) atomicExch(bad, 1);
    }
    float mx = -INFINITY;
    if (keep) {
#pragma unroll 4
        for (int j = 4 * threadIdx.x; j < ld; j += 1024) {
            const float4 v = *reinterpret_cast<const float4*>(l + j);
            *reinterpret_cast<float4*>(ce_row + j) = v;
            if (j + 3 < P) {
                mx = fmaxf(fmaxf(fmaxf(mx, v.x), fmaxf(v.y, v.z)), v.w);
            } else {
                if (j < P) mx = fmaxf(mx, v.x);
                if (j + 1 < P) mx = fmaxf(mx, v.y);
                if (j + 2 < P) mx = fmaxf(mx, v.z);
            }
        }
    } else {
        for (int j = threadIdx.x; j < P; j += blockDim.x) mx = fmaxf(mx, l[j]);
    }
    mx = block_max(mx, sh);
    float s = 0.f;
    if (keep) {
#pragma unroll 4
        for (int j = threadIdx.x; j < P; j += 256) {
            const float e = expf(ce_row[j] - mx);
            ce_row[j] = e;
            s += e;
        }
    } else {
        for (int j = threadIdx.x; j < P; j += blockDim.x) s += expf(l[j] - mx);
    }
    s = block_sum(s, sh);
    const float inv = 1.0f / s;
    bf16* g = dL + row * ld;
    if (keep && y >= 0) {
#pragma unroll 2
        for (int j = 4 * threadIdx.x; j < ld; j += 1024) {
            float4 e = *reinterpret_cast<const float4*>(ce_row + j);
            if (j + 3 >= P) {
                if (j >= P) e.x = 0.f;
                if (j + 1 >= P) e.y = 0.f;
                if (j + 2 >= P) e.z = 0.f;
                e.w = 0.f;
            }
            const __nv_bfloat162 h0 = __floats2bfloat162_rn((e.x * inv) * scale, (e.y * inv) * scale);
            const __nv_bfloat162 h1 = __floats2bfloat162_rn((e.z * inv) * scale, (e.w * inv) * scale);
            uint2 u;
            u.x = *reinterpret_cast<const unsigned*>(&h0);
            u.y = *reinterpret_cast<const unsigned*>(&h1);
            *reinterpret_cast<uint2*>(g + j) = u;
        }
        // the label's element again, by the thread that wrote it
        if ((int)threadIdx.x == (y >> 2) % 256) g[y] = __float2bfloat16_rn(fmaf(ce_row[y], inv, -1.f) * scale);
    } else {
        for (int j = 2 * threadIdx.x; j < ld; j += 512) {
            float v[2] = {0.f, 0.f};
            if (y >= 0) {
#pragma unroll
                for (int u = 0; u < 2; u++)
                    if (j + u < P) v[u] = fmaf(expf(l[j + u] - mx), inv, j + u == y ? -1.f : 0.f) * scale;
            }
            *reinterpret_cast<__nv_bfloat162*>(g + j) = __floats2bfloat162_rn(v[0], v[1]);
        }
    }
    if (threadIdx.x == 0) loss[row] = y >= 0 ? (double)(logf(s) + mx - l[y]) : 0.0;
}

// dZ = dH * GELU'(Z), GELU(z) = z Phi(z):  GELU'(z) = Phi(z) + z phi(z).  Four
// elements per thread (n a multiple of 4, 16-byte aligned).
__global__ void wp_gelu_bwd_kernel(const float4* __restrict__ dH, const uint2* __restrict__ Z, long n4,
                                   uint2* __restrict__ dZ) {
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n4) return;
    const float4 h = dH[i];
    const uint2 zz = Z[i];
    const float hv[4] = {h.x, h.y, h.z, h.w};
    const unsigned zw[4] = {zz.x << 16, zz.x & 0xffff0000u, zz.y << 16, zz.y & 0xffff0000u};
    float o[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
        const float z = __uint_as_float(zw[u]);
        const float d = 0.5f * (1.0f + erff(z * 0.70710678118654752f)) + z * 0.39894228040143268f * expf(-0.5f * z * z);
        o[u] = hv[u] * d;
    }
    const __nv_bfloat162 h0 = __floats2bfloat162_rn(o[0], o[1]), h1 = __floats2bfloat162_rn(o[2], o[3]);
    dZ[i] = make_uint2(*reinterpret_cast<const unsigned*>(&h0), *reinterpret_cast<const unsigned*>(&h1));
}

// Column sums of a BF16 [rows][ld] matrix, each column's rows added in order
// (rows and columns multiples of 64).  A CTA takes 64 columns: all its threads
// bring tiles of 64 rows (128 bytes of each) into shared memory, four tiles in
// flight, 64 of them add.  The chain of `rows` additions bounds a column (4
// cycles each) and with it the narrow matrices, HBM the wide one.  4,096 x 20,032:
// 30 us, 68 us with 16 columns per CTA and one tile in flight (32-byte pieces of
// rows), 700 us for a thread per column that loads its own elements; 4,096 x
// 1,024: 18 us, 24 before.
#define CS_COLS 64
#define CS_ROWS 64
#define CS_STAGES 5
__global__ void __launch_bounds__(256) wp_colsum_bf16_kernel(const bf16* __restrict__ M, int rows, int ld,
                                                             float* __restrict__ out) {
    __shared__ __align__(16) bf16 tile[CS_STAGES][CS_ROWS * CS_COLS];
    const int c0 = blockIdx.x * CS_COLS, nt = rows / CS_ROWS;
    const int r = threadIdx.x >> 3, cc = (threadIdx.x & 7) * 8;  // rows r and r + 32, 8 columns from cc
    const bf16* src = M + (long)r * ld + c0 + cc;
    auto fetch = [&](int t) {
        if (t < nt) {
#pragma unroll
            for (int u = 0; u < 2; u++)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(
                                     &tile[t % CS_STAGES][(r + 32 * u) * CS_COLS + cc])),
                             "l"(src + (long)(t * CS_ROWS + 32 * u) * ld)
                             : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (int t = 0; t < CS_STAGES - 1; t++) fetch(t);
    float s = 0.f;
    for (int t = 0; t < nt; t++) {
        asm volatile("cp.async.wait_group %0;" ::"n"(CS_STAGES - 2) : "memory");
        __syncthreads();  // tile t is there, tile t - 1 has been added
        fetch(t + CS_STAGES - 1);
        if (threadIdx.x < CS_COLS) {
            const bf16* x = &tile[t % CS_STAGES][threadIdx.x];
#pragma unroll
            for (int i = 0; i < CS_ROWS; i++) s += __bfloat162float(x[i * CS_COLS]);
        }
    }
    if (threadIdx.x < CS_COLS) out[c0 + threadIdx.x] = s;
}

// Adam (Kingma & Ba 2015) on FP32 master weights; refreshes the BF16 copy.
// Four weights per thread (n a multiple of 4, 16-byte aligned).  Nothing is
// changed where *bad is set (a label without a class).  Bound by HBM (30
// bytes per weight): 20.5 million in 84 us, 113 with one weight per thread.
__global__ void wp_adam_kernel(float4* __restrict__ w, const float4* __restrict__ g, float4* __restrict__ m,
                               float4* __restrict__ v, long n4, float lr, float b1, float b2, float eps, float bc1,
                               float bc2, uint2* __restrict__ wb, const int* __restrict__ bad) {
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n4 || *bad) return;
    const float4 g4 = g[i], m4 = m[i], v4 = v[i], w4 = w[i];
    const float gi[4] = {g4.x, g4.y, g4.z, g4.w};
    float mi[4] = {m4.x, m4.y, m4.z, m4.w}, vi[4] = {v4.x, v4.y, v4.z, v4.w}, wi[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
    for (int u = 0; u < 4; u++) {
        // the rounding is spelled out: a weight's path must not depend on what the
        // compiler makes of the sums
        mi[u] = fmaf(1.f - b1, gi[u], __fmul_rn(b1, mi[u]));
        vi[u] = fmaf(__fmul_rn(1.f - b2, gi[u]), gi[u], __fmul_rn(b2, vi[u]));
        wi[u] = wi[u] - lr * (mi[u] / bc1) / (sqrtf(vi[u] / bc2) + eps);
    }
    m[i] = make_float4(mi[0], mi[1], mi[2], mi[3]);
    v[i] = make_float4(vi[0], vi[1], vi[2], vi[3]);
    w[i] = make_float4(wi[0], wi[1], wi[2], wi[3]);
    if (wb) {
        const __nv_bfloat162 h0 = __floats2bfloat162_rn(wi[0], wi[1]), h1 = __floats2bfloat162_rn(wi[2], wi[3]);
        wb[i] = make_uint2(*reinterpret_cast<const unsigned*>(&h0), *reinterpret_cast<const unsigned*>(&h1));
    }
}

__global__ void wp_f32_to_bf16_kernel(const float* __restrict__ in, long n, bf16* __restrict__ out) {
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = __float2bfloat16_rn(in[i]);
}

// Gaussian initialisation N(0, std^2) of rows [0, valid_rows) of a
// [rows][cols] matrix (others zero), Philox stream per element.
__global__ void wp_init_normal_kernel(float* __restrict__ w, long rows, long cols, long valid_rows, float std,
                                      unsigned long long seed) {
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= rows * cols) return;
    if (i / cols >= valid_rows) {
        w[i] = 0.f;
        return;
    }
    curandStatePhilox4_32_10_t st;
    curand_init(seed, (unsigned long long)i, 0ull, &st);
    w[i] = std * curand_normal(&st);
}

// Sortable unsigned key of a float (ascending order of the floats).
__device__ __forceinline__ unsigned fkey(float f) {
    const unsigned u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

// The exact fallback of the top-h selection, one CTA (256 threads) per read
// of the list rows[0 .. *nrows) (persistent over it): the h largest of the
// first P logits by (logit, index), by radix select on the sortable keys,
// then sorted ascending; writes peptide indices and softmax probabilities,
// and the sum of probability x peptide count over the candidates.
__global__ void wp_topk_kernel(const float* __restrict__ logits, int P, int ld, int h, const int* __restrict__ counts,
                               int* __restrict__ out_idx, float* __restrict__ out_prob, double* __restrict__ out_mass,
                               const int* __restrict__ rows, const int* __restrict__ nrows) {
    __shared__ unsigned hist[256];
    __shared__ float sh[32];
    __shared__ unsigned long long skey[1024];
    __shared__ int sidx[1024];
    __shared__ int nsel;
  for (int it = blockIdx.x; it < *nrows; it += gridDim.x) {
    const long row = rows[it];
    const float* l = logits + row * ld;
    // softmax normaliser
    float mx = -INFINITY;
    for (int j = threadIdx.x; j < P; j += blockDim.x) mx = fmaxf(mx, l[j]);
    mx = block_max(mx, sh);
    float s = 0.f;
    for (int j = threadIdx.x; j < P; j += blockDim.x) s += expf(l[j] - mx);
    s = block_sum(s, sh);
    // radix select of the h-th largest key (count based, from the top)
    unsigned prefix = 0u, mask = 0u;
    int want = min(h, P);
    for (int pass = 0; pass < 4; pass++) {
        const int shift = 24 - 8 * pass;
        for (int i = threadIdx.x; i < 256; i += blockDim.x) hist[i] = 0u;
        __syncthreads();
        for (int j = threadIdx.x; j < P; j += blockDim.x) {
            const unsigned k = fkey(l[j]);
            if ((k & mask) == prefix) atomicAdd(&hist[(k >> shift) & 255u], 1u);
        }
        __syncthreads();
        __shared__ int sdigit, sbefore;
        if (threadIdx.x == 0) {
            int c = 0, d = 255;
            for (; d > 0; d--) {
                if (c + (int)hist[d] >= want) break;
                c += (int)hist[d];
            }
            sdigit = d;
            sbefore = c;
        }
        __syncthreads();
        prefix |= (unsigned)sdigit << shift;
        mask |= 255u << shift;
        want -= sbefore;
        __syncthreads();
    }
    // keys above the threshold, plus `want` of those equal to it with the
    // largest indices (one thread walks the ties from the top index down)
    if (threadIdx.x == 0) nsel = 0;
    __syncthreads();
    for (int j = threadIdx.x; j < P; j += blockDim.x) {
        const unsigned k = fkey(l[j]);
        if (k > prefix) {
            const int pos = atomicAdd(&nsel, 1);
            skey[pos] = ((unsigned long long)k << 32) | (unsigned)j;
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int taken = 0;
        for (int j = P - 1; j >= 0 && taken < want; j--)
            if (fkey(l[j]) == prefix) {
                skey[nsel++] = ((unsigned long long)prefix << 32) | (unsigned)j;
                taken++;
            }
    }
    __syncthreads();
    const int n = nsel;
    int n2 = 1;
    while (n2 < n) n2 <<= 1;
    for (int i = n + threadIdx.x; i < n2; i += blockDim.x) skey[i] = ~0ull;
    __syncthreads();
    for (int size = 2; size <= n2; size <<= 1)
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            for (int i = threadIdx.x; i < n2; i += blockDim.x) {
                const int j = i ^ stride;
                if (j > i) {
                    const bool up = (i & size) == 0;
                    const unsigned long long a = skey[i], b = skey[j];
                    if ((a > b) == up) {
                        skey[i] = b;
                        skey[j] = a;
                    }
                }
            }
            __syncthreads();
        }
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const int j = (int)(skey[i] & 0xffffffffu);
        out_idx[row * h + i] = j;
        out_prob[row * h + i] = expf(l[j] - mx) / s;
        sidx[i] = j;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double mass = 0.0;
        for (int i = 0; i < n; i++) mass += (double)(expf(l[sidx[i]] - mx) / s) * (double)counts[sidx[i]];
        out_mass[row] = mass;
    }
    __syncthreads();
  }
}

// The top-h selection, one warp per read (persistent over the reads): a
// sample of TK_SAMPLE logits at a fixed stride gives, by a bitwise search
// for its order statistic, a threshold that about 2 h of the read's logits
// reach; one pass over the logits
// keeps those at or above it (composite key: sortable logit bits, then the
// index) in the warp's shared buffer and forms the softmax normaliser
// online; the buffer, sorted, yields the h largest, written ascending as the
// fallback kernel does.  A read whose kept set is smaller than h or larger
// than the buffer goes to fail_rows for the exact fallback kernel.
#define TK_WARPS 8
#define TK_CAP 1024
#define TK_SAMPLE 1024

// Bitonic sort, descending, of buf[0 .. n) (n a power of two) by one warp.
__device__ __forceinline__ void tk_warp_sort_desc(unsigned long long* buf, int n) {
    const int lane = threadIdx.x & 31;
    for (int size = 2; size <= n; size <<= 1)
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            for (int i = lane; i < n; i += 32) {
                const int j = i ^ stride;
                if (j > i) {
                    const bool desc = (i & size) == 0;
                    const unsigned long long a = buf[i], b = buf[j];
                    if ((a < b) == desc) {
                        buf[i] = b;
                        buf[j] = a;
                    }
                }
            }
            __syncwarp();
        }
}

__global__ void __launch_bounds__(TK_WARPS * 32) wp_topk_warp_kernel(const float* __restrict__ logits, int R, int P,
                                                                      int ld, int h, const int* __restrict__ counts,
                                                                      int* __restrict__ out_idx,
                                                                      float* __restrict__ out_prob,
                                                                      double* __restrict__ out_mass,
                                                                      int* __restrict__ fail_rows,
                                                                      int* __restrict__ fail_count, int vec4) {
    extern __shared__ unsigned long long tk_smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    unsigned long long* buf = tk_smem + (size_t)warp * TK_CAP;
    unsigned* hist = reinterpret_cast<unsigned*>(tk_smem + (size_t)TK_WARPS * TK_CAP) + warp * 256;
    const unsigned lt = (1u << lane) - 1u;
    for (long row = (long)blockIdx.x * TK_WARPS + warp; row < R; row += (long)gridDim.x * TK_WARPS) {
        const float* l = logits + row * ld;
        // threshold: the composite key that about 2.5 h logits reach
        unsigned long long tau = 0ull;
        if (P > TK_CAP) {
            // the rank-th largest sample key, bit by bit from the top: the
            // largest t with at least `rank` sample keys >= t
            // TK_SAMPLE / 4 blocks of four neighbouring logits at a fixed
            // stride (one 16-byte load each)
            unsigned sk[TK_SAMPLE / 32];
#pragma unroll
            for (int u = 0; u < TK_SAMPLE / 128; u++) {
                const int b = u * 32 + lane;
                int j = (int)(((long)b * P) / (TK_SAMPLE / 4)) & ~3;
                j = min(j, (P - 4) & ~3);  // a multiple of 4 (16-byte aligned), j + 3 < P
                float4 v;
                if (vec4) {
                    v = *reinterpret_cast<const float4*>(l + j);
                } else {
                    v = make_float4(l[j], l[j + 1], l[j + 2], l[j + 3]);
                }
                sk[4 * u] = fkey(v.x);
                sk[4 * u + 1] = fkey(v.y);
                sk[4 * u + 2] = fkey(v.z);
                sk[4 * u + 3] = fkey(v.w);
            }
            const int rank = min(TK_SAMPLE, (int)ceilf(2.0f * (float)h * (float)TK_SAMPLE / (float)P) + 4);
            unsigned t = 0u;
#pragma unroll 1
            for (int bit = 31; bit >= 0; bit--) {
                const unsigned cand = t | (1u << bit);
                int c = 0;
#pragma unroll
                for (int u = 0; u < TK_SAMPLE / 32; u++) c += sk[u] >= cand ? 1 : 0;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
                if (c >= rank) t = cand;
            }
            tau = (unsigned long long)t << 32;  // every index of a key at the threshold
        }
        // the float at the threshold key: x >= tf keeps every key >= tau
        // (and possibly -0.0 at +0.0, harmless: extra keys are sorted out)
        const unsigned th = (unsigned)(tau >> 32);
        const float tf = P > TK_CAP ? __uint_as_float((th & 0x80000000u) ? (th & 0x7fffffffu) : ~th) : -INFINITY;
        // one pass: keep keys >= tau; online max and sum of exp
        int cnt = 0;
        float m = -INFINITY, sum = 0.0f;
        // element j: online softmax, then kept when its key reaches tau
        // (the normaliser uses the fast exponential: relative error near
        // 1e-6 over the logit range; the probabilities written use expf)
        auto visit = [&](int j, float x, bool in) {
            if (in) {
                if (x > m) {
                    sum = sum * __expf(m - x) + 1.0f;
                    m = x;
                } else {
                    sum += __expf(x - m);
                }
            }
            const bool keep = in && x >= tf;
            const unsigned ball = __ballot_sync(0xffffffffu, keep);
            if (ball) {
                if (keep) {
                    const int pos = cnt + __popc(ball & lt);
                    if (pos < TK_CAP) buf[pos] = ((unsigned long long)fkey(x) << 32) | (unsigned)j;
                }
                cnt += __popc(ball);
            }
        };
        int j0 = 0;
        if (vec4) {  // 16-byte rows: eight float4 per lane in flight
            // eight independent online-softmax states (one per float4 slot,
            // so the exponentials do not form one long dependent chain),
            // merged below; the kept keys of a 1,024-logit chunk are placed
            // with one warp scan of the lanes' counts (their order in the
            // buffer does not matter: it is sorted)
            const float4* l4 = reinterpret_cast<const float4*>(l);
            float mu[8], su[8];
#pragma unroll
            for (int u = 0; u < 8; u++) {
                mu[u] = -INFINITY;
                su[u] = 0.0f;
            }
            for (; j0 + 1024 <= P; j0 += 1024) {
                float4 v[8];
#pragma unroll
                for (int u = 0; u < 8; u++) v[u] = l4[(j0 >> 2) + 32 * u + lane];
                unsigned km = 0u;
#pragma unroll
                for (int u = 0; u < 8; u++) {
                    const float mx = fmaxf(fmaxf(v[u].x, v[u].y), fmaxf(v[u].z, v[u].w));
                    if (mx > mu[u]) {
                        su[u] = su[u] * __expf(mu[u] - mx);
                        mu[u] = mx;
                    }
                    su[u] += (__expf(v[u].x - mu[u]) + __expf(v[u].y - mu[u])) +
                             (__expf(v[u].z - mu[u]) + __expf(v[u].w - mu[u]));
                    km |= (v[u].x >= tf ? 1u : 0u) << (4 * u);
                    km |= (v[u].y >= tf ? 1u : 0u) << (4 * u + 1);
                    km |= (v[u].z >= tf ? 1u : 0u) << (4 * u + 2);
                    km |= (v[u].w >= tf ? 1u : 0u) << (4 * u + 3);
                }
                const int mine = __popc(km);
                int incl = mine;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int t = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += t;
                }
                int pos = cnt + incl - mine;
#pragma unroll
                for (int u = 0; u < 8; u++) {
                    unsigned m4 = (km >> (4 * u)) & 15u;
                    while (m4) {
                        const int c = __ffs(m4) - 1;
                        m4 &= m4 - 1;
                        const float x = c == 0 ? v[u].x : c == 1 ? v[u].y : c == 2 ? v[u].z : v[u].w;
                        if (pos < TK_CAP)
                            buf[pos] = ((unsigned long long)fkey(x) << 32) | (unsigned)(j0 + 128 * u + 4 * lane + c);
                        pos++;
                    }
                }
                cnt += __shfl_sync(0xffffffffu, incl, 31);
            }
            // the lane's softmax state from its eight
#pragma unroll
            for (int u = 0; u < 8; u++) {
                if (mu[u] == -INFINITY) continue;
                if (mu[u] > m) {
                    sum = (m == -INFINITY ? 0.0f : sum * __expf(m - mu[u])) + su[u];
                    m = mu[u];
                } else {
                    sum += su[u] * __expf(mu[u] - m);
                }
            }
        }
        for (; j0 < P; j0 += 32) {
            const int j = j0 + lane;
            visit(j, j < P ? l[j] : -INFINITY, j < P);
        }
        // warp-wide softmax normaliser
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float m2 = __shfl_xor_sync(0xffffffffu, m, o), s2 = __shfl_xor_sync(0xffffffffu, sum, o);
            const float mm = fmaxf(m, m2);
            sum = (m == -INFINITY ? 0.0f : sum * __expf(m - mm)) + (m2 == -INFINITY ? 0.0f : s2 * __expf(m2 - mm));
            m = mm;
        }
        if (cnt < min(h, P) || cnt > TK_CAP) {
            if (lane == 0) fail_rows[atomicAdd(fail_count, 1)] = (int)row;
            __syncwarp();
            continue;
        }
        __syncwarp();
        const int hh0 = min(h, P);
        int nk = cnt;
        if (cnt > 256 && hh0 <= 256) {
            // only the h largest keys are needed: the h-th largest by a radix
            // select over the kept (unique) keys, eight 8-bit digits from the
            // top, then the keys at or above it moved to the front, so that
            // the sort below covers 256 keys instead of 512 or 1,024
            unsigned long long pre = 0ull, msk = 0ull;
            int want = hh0;
            for (int pass = 0; pass < 8; pass++) {
                const int shift = 56 - 8 * pass;
                for (int i = lane; i < 256; i += 32) hist[i] = 0u;
                __syncwarp();
                for (int i = lane; i < cnt; i += 32) {
                    const unsigned long long k = buf[i];
                    if ((k & msk) == pre) atomicAdd(&hist[(unsigned)(k >> shift) & 255u], 1u);
                }
                __syncwarp();
                // digits from 255 down: lane l holds [248 - 8 l, 256 - 8 l)
                int mine = 0;
#pragma unroll
                for (int i = 0; i < 8; i++) mine += (int)hist[255 - (lane * 8 + i)];
                int incl = mine;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int t = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += t;
                }
                const unsigned hit = __ballot_sync(0xffffffffu, incl >= want);
                const int L = __ffs(hit) - 1;
                int before = __shfl_sync(0xffffffffu, incl - mine, L);
                int digit = 0;
                if (lane == L) {
                    int c = before;
                    for (int i = 0; i < 8; i++) {
                        const int d = 255 - (L * 8 + i);
                        if (c + (int)hist[d] >= want) {
                            digit = d;
                            break;
                        }
                        c += (int)hist[d];
                    }
                    before = c;
                }
                digit = __shfl_sync(0xffffffffu, digit, L);
                before = __shfl_sync(0xffffffffu, before, L);
                want -= before;
                pre |= (unsigned long long)digit << shift;
                msk |= 255ull << shift;
                __syncwarp();
            }
            // pre is the h-th largest key: keep the keys >= it (exactly h),
            // compacted in place (a chunk is read before any lane writes)
            int out = 0;
            for (int i0 = 0; i0 < cnt; i0 += 32) {
                const int i = i0 + lane;
                const unsigned long long k = i < cnt ? buf[i] : 0ull;
                const bool keep = i < cnt && k >= pre;
                const unsigned bal = __ballot_sync(0xffffffffu, keep);
                __syncwarp();
                if (keep) buf[out + __popc(bal & ((1u << lane) - 1u))] = k;
                out += __popc(bal);
                __syncwarp();
            }
            nk = out;
        }
        int n2 = 1;
        while (n2 < nk) n2 <<= 1;
        for (int i = nk + lane; i < n2; i += 32) buf[i] = 0ull;
        __syncwarp();
        tk_warp_sort_desc(buf, n2);
        // the h largest, written ascending by (logit, index)
        const int hh = min(h, P);
        double part = 0.0;  // this lane's share of the candidate mass
        for (int i = lane; i < hh; i += 32) {
            const int j = (int)(buf[hh - 1 - i] & 0xffffffffu);
            const float pr = expf(l[j] - m) / sum;
            out_idx[row * h + i] = j;
            out_prob[row * h + i] = pr;
            part += (double)pr * (double)counts[j];
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) part += __shfl_down_sync(0xffffffffu, part, o);
        if (lane == 0) out_mass[row] = part;
        __syncwarp();
    }
}

// ------------------------------------------------------------------ launchers
cudaError_t wp_mlp_launch_input(const float* xf, const double* xd, int B, int TC, bf16* X, cudaStream_t s) {
    const long n = (long)B * 64;
    if (n == 0) return cudaSuccess;
    wp_mlp_input_kernel<<<(int)((n + 255) / 256), 256, 0, s>>>(xf, xd, B, TC, X);
    return cudaGetLastError();
}

// rows, cols multiples of 64; a CTA takes CS_COLS columns and all rows.
cudaError_t wp_mlp_launch_colsum(const bf16* M, int rows, int cols, int ld, float* out, cudaStream_t s) {
    if (rows % 64 || cols % 64) return cudaErrorInvalidValue;
    wp_colsum_bf16_kernel<<<cols / CS_COLS, 256, 0, s>>>(M, rows, ld, out);
    return cudaGetLastError();
}

cudaError_t wp_mlp_launch_softmax_ce(const float* logits, int B, int P, int ld, const int* labels, float scale,
                                     bf16* dL, double* loss, int* bad, cudaStream_t s) {
    // two CTAs per SM keep their rows up to 28,000 logits, one up to 56,000
    const size_t smem = sizeof(float) * ld;
    const bool keep = smem <= 220 * 1024;
    if (keep) {
        int per_sm = 0, sms = 0;
        const cudaError_t e =
                wp_launch_shape(reinterpret_cast<const void*>(wp_softmax_ce_kernel), 256, smem, &per_sm, &sms);
        if (e != cudaSuccess) return e;
    }
    wp_softmax_ce_kernel<<<B, 256, keep ? smem : 0, s>>>(logits, P, ld, labels, scale, dL, loss, keep ? 1 : 0, bad);
    return cudaGetLastError();
}

cudaError_t wp_mlp_launch_gelu_bwd(const float* dH, const bf16* Z, long n, bf16* dZ, cudaStream_t s) {
    if (n % 4) return cudaErrorInvalidValue;
    const long n4 = n / 4;
    wp_gelu_bwd_kernel<<<(int)((n4 + 255) / 256), 256, 0, s>>>(reinterpret_cast<const float4*>(dH),
                                                               reinterpret_cast<const uint2*>(Z), n4,
                                                               reinterpret_cast<uint2*>(dZ));
    return cudaGetLastError();
}

cudaError_t wp_mlp_launch_adam(float* w, const float* g, float* m, float* v, long n, float lr, float b1, float b2,
                               float eps, float bc1, float bc2, bf16* wb, const int* bad, cudaStream_t s) {
    if (n % 4) return cudaErrorInvalidValue;
    const long n4 = n / 4;
    wp_adam_kernel<<<(int)((n4 + 255) / 256), 256, 0, s>>>(
            reinterpret_cast<float4*>(w), reinterpret_cast<const float4*>(g), reinterpret_cast<float4*>(m),
            reinterpret_cast<float4*>(v), n4, lr, b1, b2, eps, bc1, bc2, reinterpret_cast<uint2*>(wb), bad);
    return cudaGetLastError();
}

cudaError_t wp_mlp_launch_to_bf16(const float* in, long n, bf16* out, cudaStream_t s) {
    wp_f32_to_bf16_kernel<<<(int)((n + 255) / 256), 256, 0, s>>>(in, n, out);
    return cudaGetLastError();
}

cudaError_t wp_mlp_launch_init(float* w, long rows, long cols, long valid_rows, float std, unsigned long long seed,
                               cudaStream_t s) {
    const long n = rows * cols;
    wp_init_normal_kernel<<<(int)((n + 255) / 256), 256, 0, s>>>(w, rows, cols, valid_rows, std, seed);
    return cudaGetLastError();
}

// fail: scratch of R + 1 ints (the fallback's row list, then its count).
cudaError_t wp_mlp_launch_topk(const float* logits, int R, int P, int ld, int h, const int* counts, int* idx,
                               float* prob, double* mass, int* fail, cudaStream_t s) {
    if (R == 0) return cudaSuccess;
    if (h > 1024) return cudaErrorInvalidValue;
    int* fail_count = fail + R;
    cudaError_t e = cudaMemsetAsync(fail_count, 0, sizeof(int), s);
    if (e != cudaSuccess) return e;
    const size_t smem = sizeof(unsigned long long) * TK_WARPS * TK_CAP + sizeof(unsigned) * TK_WARPS * 256;
    int sms = 0, per_sm = 0;
    e = wp_launch_shape(reinterpret_cast<const void*>(wp_topk_warp_kernel), TK_WARPS * 32, smem, &per_sm, &sms);
    if (e != cudaSuccess) return e;
    const int grid = std::max(1, std::min(sms * std::max(per_sm, 1), (R + TK_WARPS - 1) / TK_WARPS));
    const int vec4 = (ld % 4 == 0 && ((uintptr_t)logits & 15u) == 0) ? 1 : 0;
    wp_topk_warp_kernel<<<grid, TK_WARPS * 32, smem, s>>>(logits, R, P, ld, h, counts, idx, prob, mass, fail,
                                                         fail_count, vec4);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    // exact fallback for the reads the threshold missed (usually none)
    wp_topk_kernel<<<std::max(1, std::min(R, 2 * sms)), 256, 0, s>>>(logits, P, ld, h, counts, idx, prob, mass, fail,
                                                                       fail_count);
    return cudaGetLastError();
}
