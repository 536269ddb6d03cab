// wp_gemm.cu -- BF16 GEMM on the fifth-generation tensor cores (sm_103a):
//
//     C[M][N] = epilogue( A[M][K] . B[N][K]^T + bias[N] )
//
// with A and B BF16, each either row-major as written (K-major) or stored
// transposed ([K][M], [K][N]: MN-major, which the tensor cores read as it
// is), FP32 accumulation in tensor memory, and an epilogue that adds the bias, optionally applies GELU (and
// keeps the pre-activation), and stores BF16 or FP32.  This is the building
// block of the learned proposal network (forward layers, and with
// transposed operands its backward products).
//
// A persistent CTA per SM walks 128 x 256 output tiles with 6 warps:
//   warp 0 (one thread)  TMA producer: 64-wide K slices of A and B into a
//                        4-stage shared-memory ring (128-byte swizzle),
//                        signalled on the stage's `full` mbarrier;
//   warp 1 (one thread)  MMA issuer: four tcgen05.mma (M128 N256 K16) per
//                        stage into one of two 256-column TMEM accumulators,
//                        tcgen05.commit onto the stage's `empty` mbarrier so
//                        the producer can refill it, and onto the
//                        accumulator's `full` mbarrier after the last K
//                        slice; warp 1 also owns the TMEM allocation;
//   warps 2-5            epilogue: each reads its 32 TMEM lanes (rows) in
//                        32-column chunks with tcgen05.ld (the next chunk's
//                        load in flight), adds the bias (the tile's biases
//                        fetched to shared memory ahead), and stores from
//                        registers, a 32-byte sector of its row per lane and
//                        store; the accumulator is freed (its `empty`
//                        mbarrier) for the tile after next as soon as its
//                        last chunk is in registers.
// A tile's products at K = 1024 take 11,300 cycles, and the epilogue's 32,768
// outputs must take no longer or they set the time.  Shared memory is what
// they must stay off: the products keep it busy, and outputs staged through
// it for stores of whole rows took 24,000 cycles a tile.  4,096 x 20,000 x
// 1,024: BF16 output 171 -> 119 us, FP32 output 212 -> 154 (its 328 MB of
// stores bound it: 109 without them); 4,096 x 1,024 x 64 with GELU and
// pre-activation, 34 -> 18 us.
// Every mbarrier wait is bounded; on expiry the CTA records an error code,
// stops issuing work, waits (bounded) for what it issued and frees its TMEM.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <algorithm>

#define GEMM_BM 128
#define GEMM_BK 64
#define GEMM_THREADS 192
#define GEMM_A_STAGE (GEMM_BM * GEMM_BK * 2)  // 16 KB

// Tile width BN: 256, or 64 for products with few tiles.
template <int BN>
struct GemmShape {
    static constexpr int STAGES = BN == 256 ? 4 : 8;
    static constexpr int B_STAGE = BN * GEMM_BK * 2;  // 32 or 8 KB
    static constexpr size_t SMEM =
            1024 + STAGES * (GEMM_A_STAGE + B_STAGE) + 4 * BN * 4 + (2 * STAGES + 5) * 8 + 16;
};
#define GEMM_WAIT_LIMIT (1L << 22)

typedef __nv_bfloat16 bf16_t;

struct GemmParams {
    int M, N, K;
    void* C;            // [M][ldc] BF16 or FP32
    int ldc;
    int c_fp32;         // 1: FP32 output, 0: BF16
    const float* bias;  // [N] or null
    int act;            // 0 none, 1 GELU (erf form)
    __nv_bfloat16* Z;   // pre-activation [M][ldc] BF16, or null
    int* err;
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
            "{\n"
            ".reg .pred p;\n"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
            "selp.u32 %0, 1, 0, p;\n"
            "}\n"
            : "=r"(ok)
            : "r"(smem_u32(bar)), "r"(parity)
            : "memory");
    return ok != 0;
}

// Bounded wait for the phase of `parity`; false (and an error code) when
// the limit expires.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, int* err, int code) {
    for (long i = 0; i < GEMM_WAIT_LIMIT; i++)
        if (mbar_try_wait(bar, parity)) return true;
    atomicExch(err, code);
    return false;
}

__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
    asm volatile(
            "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
            ::"r"(smem_u32(dst)), "l"((uint64_t)map), "r"(x), "r"(y), "r"(smem_u32(bar))
            : "memory");
}

// Shared-memory matrix descriptor of a K-major tile written by TMA with the
// 128-byte swizzle: rows of 128 B, 8-row atoms 1024 B apart (stride byte
// offset), fixed field 0b001 at bit 46, swizzle mode 2 (128 B) at bit 61.
// The leading byte offset is unused for this layout.
__device__ __forceinline__ uint64_t sw128_desc(uint32_t saddr) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}

// The same of an MN-major tile: boxes of 64 (M or N) x 64 K, one after
// another along M or N.  A box is rows of 128 B, one per K; its 8-row atoms are
// 1024 B apart (stride byte offset), the boxes 8 KB (leading byte offset).
__device__ __forceinline__ uint64_t sw128_mn_desc(uint32_t saddr) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);
    d |= (uint64_t)(8192 >> 4) << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}

// Instruction descriptor, kind::f16: FP32 accumulator (bits 4-5 = 1), A and
// B BF16 (bits 7-9 = 1, 10-12 = 1), A and B K-major (bits 15, 16 = 0) or
// MN-major (1), N >> 3 at bits 17-22, M >> 4 at bits 24-28.
__host__ __device__ constexpr uint32_t gemm_idesc(int M, int N, bool a_mn, bool b_mn) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((a_mn ? 1u : 0u) << 15) | ((b_mn ? 1u : 0u) << 16) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void mma_bf16(uint32_t tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t acc) {
    asm volatile(
            "{\n"
            ".reg .pred p;\n"
            "setp.ne.b32 p, %4, 0;\n"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n"
            "}\n" ::"r"(tmem),
            "l"(adesc), "l"(bdesc), "r"(idesc), "r"(acc)
            : "memory");
}

__device__ __forceinline__ void mma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

__device__ __forceinline__ void tmem_ld32_start(uint32_t taddr, uint32_t* r) {
    asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
            "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
            "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
              "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
              "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]),
              "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]),
              "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
            : "r"(taddr));
}

// Waits for the loads started; the registers pass through, so that nothing
// reads them earlier.
__device__ __forceinline__ void tmem_ld32_wait(uint32_t* r) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]),
                   "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]),
                   "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]), "+r"(r[16]), "+r"(r[17]),
                   "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]),
                   "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]),
                   "+r"(r[30]), "+r"(r[31])
                 :
                 : "memory");
}

__device__ __forceinline__ float gelu_erf(float x) { return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f)); }

// 32 bytes to a 32-byte boundary in one store: a whole sector per lane.
__device__ __forceinline__ void store_32b(void* p, const uint32_t* u) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(u[0]), "r"(u[1]), "r"(u[2]),
                 "r"(u[3]), "r"(u[4]), "r"(u[5]), "r"(u[6]), "r"(u[7])
                 : "memory");
}

// A lane's 32 columns (the first `cols` of them) of one row.
__device__ __forceinline__ void store_f32(float* d, const float* v, int cols) {
    const int align = (int)(reinterpret_cast<uintptr_t>(d) & 31);
    if (cols == 32 && align == 0) {
#pragma unroll
        for (int j = 0; j < 32; j += 8) {
            uint32_t u[8];
#pragma unroll
            for (int i = 0; i < 8; i++) u[i] = __float_as_uint(v[j + i]);
            store_32b(d + j, u);
        }
    } else if (cols == 32 && (align & 15) == 0) {
#pragma unroll
        for (int j = 0; j < 32; j += 4)
            *reinterpret_cast<float4*>(d + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
    } else {
#pragma unroll
        for (int j = 0; j < 32; j++)
            if (j < cols) d[j] = v[j];
    }
}

__device__ __forceinline__ void store_bf16(bf16_t* d, const float* v, int cols) {
    const int align = (int)(reinterpret_cast<uintptr_t>(d) & 31);
    uint32_t u[16];
#pragma unroll
    for (int j = 0; j < 16; j++) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
        u[j] = *reinterpret_cast<const uint32_t*>(&h);
    }
    if (cols == 32 && align == 0) {
        store_32b(d, u);
        store_32b(d + 16, u + 8);
    } else if (cols == 32 && (align & 15) == 0) {
#pragma unroll
        for (int j = 0; j < 16; j += 4)
            *reinterpret_cast<uint4*>(d + 2 * j) = make_uint4(u[j], u[j + 1], u[j + 2], u[j + 3]);
    } else {
#pragma unroll
        for (int j = 0; j < 32; j++)
            if (j < cols) d[j] = __ushort_as_bfloat16((unsigned short)((j & 1) ? u[j >> 1] >> 16 : u[j >> 1] & 0xffffu));
    }
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// Persistent: CTA b takes tiles b, b + gridDim.x, ... (M blocks fastest, so
// the CTAs running at once share B tiles in L2).  Two TMEM accumulators
// (2 x 256 columns): the MMA thread fills one while the epilogue warps drain
// the other.
template <bool AMN, bool BMN, int BN>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
        wp_gemm_tn_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                          GemmParams p) {
    constexpr int STAGES = GemmShape<BN>::STAGES, B_STAGE = GemmShape<BN>::B_STAGE;
    extern __shared__ uint8_t gemm_smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(gemm_smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t* sA = smem;
    uint8_t* sB = smem + STAGES * GEMM_A_STAGE;
    float* bias_tile = reinterpret_cast<float*>(sB + STAGES * B_STAGE);  // [4 warps][BN]
    uint64_t* full = reinterpret_cast<uint64_t*>(bias_tile + 4 * BN);
    uint64_t* empty = full + STAGES;
    uint64_t* acc_full = empty + STAGES;  // [2]
    uint64_t* acc_empty = acc_full + 2;        // [2]
    uint64_t* done = acc_empty + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nk = p.K / GEMM_BK;
    const int mblocks = (p.M + GEMM_BM - 1) / GEMM_BM;
    const int nblocks = (p.N + BN - 1) / BN;
    const int ntiles = mblocks * nblocks;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; b++) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], 4);
        }
        mbar_init(done, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(2 * BN)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;

    if (warp == 0) {
        if (lane == 0) {
            // TMA producer over every (tile, k) of this CTA
            int it = 0;
            for (int t = blockIdx.x; t < ntiles && !*abort_flag; t += gridDim.x) {
                const int m0 = (t % mblocks) * GEMM_BM, n0 = (t / mblocks) * BN;
                for (int kt = 0; kt < nk; kt++, it++) {
                    const int s = it % STAGES, round = it / STAGES;
                    if (*abort_flag || !mbar_wait(&empty[s], (round & 1) ^ 1, p.err, 101)) {
                        *abort_flag = 1;
                        break;
                    }
                    mbar_expect_tx(&full[s], GEMM_A_STAGE + B_STAGE);
                    if constexpr (AMN) {
#pragma unroll
                        for (int i = 0; i < GEMM_BM / 64; i++)
                            tma_load_2d(sA + s * GEMM_A_STAGE + i * 8192, &tmA, m0 + 64 * i, kt * GEMM_BK, &full[s]);
                    } else {
                        tma_load_2d(sA + s * GEMM_A_STAGE, &tmA, kt * GEMM_BK, m0, &full[s]);
                    }
                    if constexpr (BMN) {
#pragma unroll
                        for (int i = 0; i < BN / 64; i++)
                            tma_load_2d(sB + s * B_STAGE + i * 8192, &tmB, n0 + 64 * i, kt * GEMM_BK, &full[s]);
                    } else {
                        tma_load_2d(sB + s * B_STAGE, &tmB, kt * GEMM_BK, n0, &full[s]);
                    }
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            // MMA issuer
            const uint32_t idesc = gemm_idesc(GEMM_BM, BN, AMN, BMN);
            int it = 0, li = 0;
            for (int t = blockIdx.x; t < ntiles && !*abort_flag; t += gridDim.x, li++) {
                const int b = li & 1, use = li >> 1;
                if (!mbar_wait(&acc_empty[b], (use & 1) ^ 1, p.err, 105)) {
                    *abort_flag = 1;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t acc = tmem + (uint32_t)(b * BN);
                bool ok = true;
                for (int kt = 0; kt < nk; kt++, it++) {
                    const int s = it % STAGES, round = it / STAGES;
                    if (*abort_flag || !mbar_wait(&full[s], round & 1, p.err, 102)) {
                        ok = false;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t a0 = smem_u32(sA + s * GEMM_A_STAGE), b0 = smem_u32(sB + s * B_STAGE);
#pragma unroll
                    for (int k = 0; k < GEMM_BK / 16; k++)
                        mma_bf16(acc, AMN ? sw128_mn_desc(a0 + k * 2048) : sw128_desc(a0 + k * 32),
                                 BMN ? sw128_mn_desc(b0 + k * 2048) : sw128_desc(b0 + k * 32), idesc,
                                 (kt | k) != 0 ? 1u : 0u);
                    mma_commit(&empty[s]);
                }
                if (!ok) {
                    *abort_flag = 1;
                    break;
                }
                mma_commit(&acc_full[b]);
            }
            mma_commit(done);  // every MMA this thread issued has completed when this arrives
        }
    } else {
        // epilogue: warp w reads TMEM lanes 32 (w % 4) .. + 31
        const int q = warp & 3;
        float* sb = bias_tile + q * BN;
        int li = 0;
        for (int t = blockIdx.x; t < ntiles; t += gridDim.x, li++) {
            const int b = li & 1, use = li >> 1;
            const int m0 = (t % mblocks) * GEMM_BM, n0 = (t / mblocks) * BN;
            const int rbase = m0 + 32 * q;
            if (p.bias) {
                // this tile's biases, while its products are formed
                __syncwarp();
                for (int j = lane; j < BN; j += 32) sb[j] = n0 + j < p.N ? p.bias[n0 + j] : 0.0f;
                __syncwarp();
            }
            if (*abort_flag || !mbar_wait(&acc_full[b], use & 1, p.err, 103)) {
                *abort_flag = 1;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int nch = rbase < p.M ? (min(BN, p.N - n0) + 31) / 32 : 0;
            const uint32_t tacc = tmem + (uint32_t)(b * BN) + ((uint32_t)(32 * q) << 16);
            // this accumulator may be refilled (after the last chunk is in registers)
            auto release = [&]() {
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&acc_empty[b]);
            };
            // one chunk: a lane's 32 columns of its row, straight from registers
            const int row = rbase + lane;
            const bool live = row < p.M;
            auto chunk = [&](const uint32_t* r, int ch) {
                const int c0 = n0 + ch * 32;
                const int cols = min(32, p.N - c0);
                float v[32];
#pragma unroll
                for (int j = 0; j < 32; j += 4) {
                    float4 bv = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    if (p.bias) bv = *reinterpret_cast<const float4*>(sb + ch * 32 + j);
                    const float w[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        v[j + u] = __uint_as_float(r[j + u]);
                        if (p.bias) v[j + u] += w[u];
                    }
                }
                const long at = (long)row * p.ldc + c0;
                if (p.Z && live) store_bf16(p.Z + at, v, cols);
                if (p.act == 1) {
#pragma unroll
                    for (int j = 0; j < 32; j++) v[j] = gelu_erf(v[j]);
                }
                if (live) {
                    if (p.c_fp32) store_f32(reinterpret_cast<float*>(p.C) + at, v, cols);
                    else store_bf16(reinterpret_cast<bf16_t*>(p.C) + at, v, cols);
                }
            };
            // two register buffers: the next chunk's load runs under this one's stores
            uint32_t r0[32], r1[32];
            if (nch > 0) tmem_ld32_start(tacc, r0);
            for (int ch = 0; ch < nch; ch += 2) {
                tmem_ld32_wait(r0);
                if (ch + 1 < nch) tmem_ld32_start(tacc + (uint32_t)(32 * (ch + 1)), r1);
                else release();
                chunk(r0, ch);
                if (ch + 1 < nch) {
                    tmem_ld32_wait(r1);
                    if (ch + 2 < nch) tmem_ld32_start(tacc + (uint32_t)(32 * (ch + 2)), r0);
                    else release();
                    chunk(r1, ch + 1);
                }
            }
            if (nch == 0) release();
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        // free the columns only after every issued MMA has completed
        mbar_wait(done, 0, p.err, 104);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * BN)
                     : "memory");
    }
}

// ------------------------------------------------------------------ host
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &q) ==
                    cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(f);
    }
    return fn;
}

// Row-major BF16 [rows][K] (row pitch ld elements; for an MN-major operand the
// rows are K and the columns M or N), boxes of 64 x box_rows.
static bool make_map(CUtensorMap* map, const void* ptr, int rows, int K, int ld, int box_rows) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
    cuuint32_t box[2] = {GEMM_BK, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

static int gemm_sms() {
    static int sms[64] = {0};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && sms[dev] == 0) cudaDeviceGetAttribute(&sms[dev], cudaDevAttrMultiProcessorCount, dev);
    return (dev >= 0 && dev < 64 && sms[dev] > 0) ? sms[dev] : 148;
}

static int gemm_tiles(int M, int N, int BN) { return ((M + GEMM_BM - 1) / GEMM_BM) * ((N + BN - 1) / BN); }

template <bool AMN, bool BMN, int BN>
static cudaError_t gemm_launch(const CUtensorMap& ma, const CUtensorMap& mb, const GemmParams& p, cudaStream_t s) {
    constexpr size_t smem = GemmShape<BN>::SMEM;
    cudaError_t e = cudaFuncSetAttribute(wp_gemm_tn_kernel<AMN, BMN, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)smem);
    if (e != cudaSuccess) return e;
    // as few CTAs as take the same number of tiles in turn: the SMs left over are
    // free for kernels on other streams
    const int tiles = gemm_tiles(p.M, p.N, BN), turns = (tiles + gemm_sms() - 1) / gemm_sms();
    const int grid = (tiles + turns - 1) / turns;
    wp_gemm_tn_kernel<AMN, BMN, BN><<<grid, GEMM_THREADS, smem, s>>>(ma, mb, p);
    return cudaGetLastError();
}

// C = act(A . B^T + bias).  A: [M][K] (pitch lda), or with a_mn [K][M]; B:
// [N][K] (pitch ldb), or with b_mn [K][N] (taken with a_mn or without; a_mn
// only with b_mn).  Both BF16, 16-byte aligned, K a multiple of 64, pitches
// multiples of 8 elements.  Returns cudaErrorInvalidValue on a shape the
// kernel does not take.
cudaError_t wp_gemm_bf16(const void* A, int lda, bool a_mn, const void* B, int ldb, bool b_mn, int M, int N, int K,
                         void* C, int ldc, int c_fp32, const float* bias, int act, void* Z, int* err,
                         cudaStream_t s) {
    if (M <= 0 || N <= 0 || K <= 0 || K % GEMM_BK != 0 || lda % 8 || ldb % 8 || lda < (a_mn ? M : K) ||
        ldb < (b_mn ? N : K) || ldc < N || ((uintptr_t)A & 15) || ((uintptr_t)B & 15) || (a_mn && !b_mn))
        return cudaErrorInvalidValue;
    CUtensorMap ma, mb;
    if (!(a_mn ? make_map(&ma, A, K, M, lda, GEMM_BK) : make_map(&ma, A, M, K, lda, GEMM_BM)) ||
        !(b_mn ? make_map(&mb, B, K, N, ldb, GEMM_BK) : make_map(&mb, B, N, K, ldb, 256)))
        return cudaErrorInvalidValue;
    GemmParams p;
    p.M = M;
    p.N = N;
    p.K = K;
    p.C = C;
    p.ldc = ldc;
    p.c_fp32 = c_fp32;
    p.bias = bias;
    p.act = act;
    p.Z = reinterpret_cast<__nv_bfloat16*>(Z);
    p.err = err;
    // Tiles 64 wide for the weight gradients of the small layers, whose few tiles
    // of 256 leave most SMs idle through a long K (both operands MN-major; no
    // other product of the network has fewer than 128 tiles): 1,024 x 1,024 x 4,096
    // 33 -> 28 us, 1,024 x 64 x 4,096 30 -> 27.
    if (a_mn && gemm_tiles(M, N, 256) <= gemm_sms() / 3) return gemm_launch<true, true, 64>(ma, mb, p, s);
    if (a_mn) return gemm_launch<true, true, 256>(ma, mb, p, s);
    if (b_mn) return gemm_launch<false, true, 256>(ma, mb, p, s);
    return gemm_launch<false, false, 256>(ma, mb, p, s);
}

// Both operands K-major.
cudaError_t wp_gemm_bf16_tn(const void* A, int lda, const void* B, int ldb, int M, int N, int K, void* C, int ldc,
                            int c_fp32, const float* bias, int act, void* Z, int accumulate, int* err,
                            cudaStream_t s) {
    if (accumulate) return cudaErrorInvalidValue;
    return wp_gemm_bf16(A, lda, false, B, ldb, false, M, N, K, C, ldc, c_fp32, bias, act, Z, err, s);
}
