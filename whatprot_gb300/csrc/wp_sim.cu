// wp_sim.cu -- seeded read simulator on the GPU (`simulate rad`):
// generate_dye_track (simulation/generate-dye-track.cc:29-110) and
// generate_radiometry (simulation/generate-radiometry.cc:28-62), one thread
// per read, counter-based Philox streams (read r uses subsequence r of the
// seed, so results do not depend on the launch shape).
//
// Per read: a peptide drawn with probability proportional to its count, its
// dyes made duds (per channel p_dud), an initial block, then per timestep:
// record the live dye counts; cyclic block; detach (the read is empty from
// then on); unless blocked, an Edman cycle that succeeds with
// 1 - p_edman_failure and removes the dye at the cut position; bleaching of
// every remaining dye past the cut.  A read whose timestep-0 counts are all
// zero is not detectable and gets peptide index -1 (the reference drops it).
// Intensities are Normal(adjusted_mu, sigma(adjusted_mu)) per (t, c), with
// ChannelModel's interactions (channel-model.h:35-70), drawn in FP64 (in
// FP32 when only FP32 reads are asked for, as for network training).  Each
// Bernoulli event is one 32-bit draw against a precomputed threshold: the
// track part of the kernel does no floating-point work.
//
// With per_peptide > 0 the kernel makes the dye-track instances of the kNN
// training set instead (generate-dye-tracks.cc:32-70): instance r belongs to
// peptide copy r / per_peptide, and only the tracks are written.
//
// The reference draws from std::default_random_engine in a different order,
// so parity with it is statistical (tests compare distributions).
#include <cuda_runtime.h>
#include <curand_kernel.h>
#include <math.h>
#include <stdint.h>

#include "wp_common.cuh"

#define SIM_MAX_LEN 256


__device__ double sim_adjusted_mu(const DevModel& m, int channel, const int* counts) {
    double amu = m.mu[channel] * (double)counts[channel];
    for (int c = 0; c < m.C; c++) {
        const double fi = m.flat[channel][c], ii = m.inter[channel][c];
        if (c == channel) {
            if (counts[c] > 1) {
                if (fi != 1.0) amu *= fi;
                if (ii != 1.0) amu *= pow(ii, (double)(counts[c] - 1));
            }
        } else if (counts[c] > 0) {
            if (fi != 1.0) amu *= fi;
            if (ii != 1.0) amu *= pow(ii, (double)counts[c]);
        }
    }
    return amu;
}

// The same in FP32, for the FP32 reads the proposal network trains on.
__device__ float sim_adjusted_mu_f(const DevModel& m, int channel, const int* counts) {
    float amu = (float)m.mu[channel] * (float)counts[channel];
    for (int c = 0; c < m.C; c++) {
        const float fi = (float)m.flat[channel][c], ii = (float)m.inter[channel][c];
        const int n = c == channel ? counts[c] - 1 : counts[c];
        if (n > 0) {
            if (fi != 1.0f) amu *= fi;
            if (ii != 1.0f) amu *= powf(ii, (float)n);
        }
    }
    return amu;
}

// A read's draws, ahead of their use: a ring of SIM_RING per thread in shared
// memory, filled four at a time.  The lanes of a warp use draws at different
// rates; taken one by one, some lane needs four new ones at nearly every
// draw, and the warp pays for the generator each time.
#define SIM_THREADS 128
#define SIM_RING 16
struct SimDraws {
    curandStatePhilox4_32_10_t* st;
    unsigned* ring;  // [SIM_RING][SIM_THREADS], this thread's column
    int head, tail;  // draws taken, draws made
    __device__ __forceinline__ void fill() {
        const uint4 x = curand4(st);
        ring[((tail) & (SIM_RING - 1)) * SIM_THREADS] = x.x;
        ring[((tail + 1) & (SIM_RING - 1)) * SIM_THREADS] = x.y;
        ring[((tail + 2) & (SIM_RING - 1)) * SIM_THREADS] = x.z;
        ring[((tail + 3) & (SIM_RING - 1)) * SIM_THREADS] = x.w;
        tail += 4;
    }
    // at least n draws (n <= SIM_RING - 3) for what follows
    __device__ __forceinline__ void want(int n) {
        while (tail - head < n) fill();
    }
    // one that want() has seen to, below a threshold in 1 .. 2^32
    __device__ __forceinline__ bool below(unsigned long long thr) {
        const unsigned x = ring[(head & (SIM_RING - 1)) * SIM_THREADS];
        head++;
        return x <= (unsigned)(thr - 1ull);
    }
    // bernoulli_distribution(p) with p as a 33-bit threshold; no draw for p = 0
    __device__ __forceinline__ bool event(unsigned long long thr) { return thr != 0ull && below(thr); }
};

__device__ __forceinline__ int sim_popc(uint32_t x) { return __popc(x); }
__device__ __forceinline__ int sim_popc(uint64_t x) { return __popcll((long long)x); }

// generate_dye_track for one instance, the live dyes as bits of one mask
// ordered by channel, then position (base: each channel's first bit, one byte
// per channel): a channel's live count is the population of its bits, the
// Edman cut clears the bit of the next dye of the cut position's channel, and
// bleaching draws once per set bit.  Writes the live counts [T][C] to trk.
template <class Mask>
__device__ __forceinline__ void sim_track(const SimParams& p, SimDraws& dr, const int8_t* seq, int L, uint32_t base,
                                          int nlab, uint8_t* trk) {
    auto first = [&](int c) { return (int)((base >> (8 * c)) & 255u); };
    Mask live = 0, chan[WP_MAX_CHANNELS];
#pragma unroll
    for (int c = 0; c < WP_MAX_CHANNELS; c++) {
        const int lo = first(c), hi = c + 1 < WP_MAX_CHANNELS ? first(c + 1) : nlab;
        const Mask up = hi >= (int)sizeof(Mask) * 8 ? ~(Mask)0 : (((Mask)1 << hi) - 1);
        chan[c] = lo >= (int)sizeof(Mask) * 8 ? (Mask)0 : (up & ~(((Mask)1 << lo) - 1));
    }
    uint32_t next = base;  // the next dye of each channel, as a bit
    for (int i = 0, k = 0; i < L && k < nlab; i++) {
        const int d = seq[i];
        if (d < 0) continue;
        k++;
        dr.want(2);
        if (!dr.event(p.thr_dud[d])) live |= (Mask)1 << ((next >> (8 * d)) & 255u);  // duds
        next += 1u << (8 * d);
    }
    next = base;
    int e = 0;
    Mask drawn = 0;  // dyes of the channels that bleach
#pragma unroll
    for (int c = 0; c < WP_MAX_CHANNELS; c++)
        if (c < p.C && p.thr_bleach[c] != 0ull) drawn |= chan[c];
    dr.want(1);
    bool block = dr.event(p.thr_initial_block), gone = false;
    for (int t = 0; t < p.T; t++) {
        if (!gone && e < L) {
            dr.want(min(3 + sim_popc(live), SIM_RING - 3));
#pragma unroll
            for (int c = 0; c < WP_MAX_CHANNELS; c++)
                if (c < p.C) trk[t * p.C + c] = (uint8_t)sim_popc((Mask)(live & chan[c]));
            if (dr.event(p.thr_cyclic_block)) block = true;
            if (dr.event(p.thr_detach[t])) {
                gone = true;
                continue;
            }
            if (!block && !dr.event(p.thr_fail)) {
                const int d = seq[e];
                if (d >= 0) {  // the cut removes the dye at position e
                    live &= ~((Mask)1 << ((next >> (8 * d)) & 255u));
                    next += 1u << (8 * d);
                }
                e++;
            }
            Mask m = live & drawn;
            while (m) {  // bleaching past the cut
                const Mask low = m & (~m + 1);
                m &= m - 1;
                const unsigned long long thr = (low & chan[0])   ? p.thr_bleach[0]
                                               : (low & chan[1]) ? p.thr_bleach[1]
                                               : (low & chan[2]) ? p.thr_bleach[2]
                                                                 : p.thr_bleach[3];
                dr.want(1);
                if (dr.below(thr)) live &= ~low;
            }
        } else {
            for (int c = 0; c < p.C; c++) trk[t * p.C + c] = 0;
        }
    }
}

// Bound by issue slots (the generator, the events and their divergence).  2e6
// tracks of 16 timesteps, 3 channels: 504 us, 846 us with a generator call per
// event.
__global__ void __launch_bounds__(SIM_THREADS, 8) wp_sim_reads_kernel(SimParams p) {
    __shared__ unsigned ring[SIM_RING * SIM_THREADS];
    const long r = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= p.R) return;
    curandStatePhilox4_32_10_t st;
    const unsigned long long seed =
            p.batch > 0 ? p.seed + (unsigned long long)(r / p.batch) * p.seed_step : p.seed;
    const unsigned long long seq_no = (unsigned long long)(p.batch > 0 ? r % p.batch : r);
    curand_init(seed, seq_no, 0ull, &st);
    // peptide by count weight (upper bound of u * total in the prefix sums),
    // or the peptide of copy r / per_peptide: generate_dye_tracks
    // (generate-dye-tracks.cc:40-47) makes per_peptide tracks for each of
    // the count copies of every dye-seq, in order
    const double total = p.cum[p.P - 1];
    const double u = p.per_peptide > 0 ? (double)(r / p.per_peptide) + 1.0
                                       : curand_uniform_double(&st) * total;  // (0, total]
    const long long ub = __double_as_longlong(u);
    int lo = 0, hi = p.P - 1;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        // both positive: their bits order as they do
        if (__double_as_longlong(p.cum[mid]) >= ub) hi = mid;
        else lo = mid + 1;
    }
    const int pep = lo;
    const int L = min(p.offsets[pep + 1] - p.offsets[pep], SIM_MAX_LEN);
    const int8_t* seq = p.seqs + p.offsets[pep];
    __align__(16) uint8_t trk[WP_MAX_TIMESTEPS * WP_MAX_CHANNELS];
    // uploaded dye-seqs carry at most 15 dyes on each of at most 4 channels,
    // so at most 60 labeled positions
    uint32_t per = 0;  // dyes of each channel, one byte each
    for (int i = 0; i < L; i++)
        if (seq[i] >= 0) per += 1u << (8 * seq[i]);
    const uint32_t base = (per << 8) + (per << 16) + (per << 24);  // sums of the channels before (60 at most)
    const int nlab = (int)((base >> 24) + (per >> 24));
    SimDraws dr;
    dr.st = &st;
    dr.ring = ring + threadIdx.x;
    dr.head = dr.tail = 0;
    if (nlab <= 32) sim_track<uint32_t>(p, dr, seq, L, base, nlab, trk);
    else sim_track<uint64_t>(p, dr, seq, L, base, nlab, trk);
    bool trivial = true;
    for (int c = 0; c < p.C; c++)
        if (trk[c] != 0) trivial = false;
    p.pep[r] = trivial ? -1 : pep;
    const int TC = p.T * p.C;
    if (p.tracks) {
        if (TC % 16 == 0) {  // rows on 16-byte boundaries
            uint4* dst = reinterpret_cast<uint4*>(p.tracks + r * TC);
            for (int q = 0; q < TC / 16; q++) dst[q] = reinterpret_cast<const uint4*>(trk)[q];
        } else {
            for (int i = 0; i < TC; i++) p.tracks[r * TC + i] = trk[i];
        }
    }
    if (!p.rads_f && !p.rads_d) return;  // dye-tracks only
    // the draws after the peptide's and those the track used
    curand_init(seed, seq_no, 0ull, &st);
    if (p.per_peptide == 0) curand_uniform_double(&st);
    skipahead((unsigned long long)dr.head, &st);
    const DevModel& m = *p.model;
    const bool fp32 = !p.rads_d;  // FP32 reads only: FP32 draws
    for (int t = 0; t < p.T; t++) {
        int cts[WP_MAX_CHANNELS] = {0, 0, 0, 0};
        for (int c = 0; c < p.C; c++) cts[c] = trk[t * p.C + c];
        for (int c = 0; c < p.C; c++) {
            if (fp32) {
                const float mu = sim_adjusted_mu_f(m, c, cts);
                const float bg = (float)m.bg_sig[c], sg1 = (float)m.sig[c];
                const float sg = sqrtf(bg * bg + mu * sg1 * sg1);
                p.rads_f[r * TC + t * p.C + c] = mu + sg * curand_normal(&st);
            } else {
                const double mu = sim_adjusted_mu(m, c, cts);
                const double sg = sqrt(m.bg_sig[c] * m.bg_sig[c] + mu * m.sig[c] * m.sig[c]);
                const double x = mu + sg * curand_normal_double(&st);
                if (p.rads_f) p.rads_f[r * TC + t * p.C + c] = (float)x;
                p.rads_d[r * TC + t * p.C + c] = x;
            }
        }
    }
}

cudaError_t wp_launch_sim_reads(const SimParams& p, cudaStream_t s) {
    if (p.R == 0) return cudaSuccess;
    wp_sim_reads_kernel<<<(p.R + SIM_THREADS - 1) / SIM_THREADS, SIM_THREADS, 0, s>>>(p);
    return cudaGetLastError();
}
