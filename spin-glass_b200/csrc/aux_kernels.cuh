// aux_kernels.cuh — set-up and section-end kernels (not on the sweep path).
//
// init_kernel     : bonds and initial spins from the seed (replaces the host
//                   cuRAND generation of eamsim.cu:562-652).
// bond_counts_kernel, overlap_planes_kernel : the integers of the current
//                   state the reference's records are formed from: unsatisfied
//                   bonds and spins up per (copy, temperature, sample), and the
//                   sites where the copies differ per coordinate plane, from
//                   which the Fourier overlaps of compute_q (eamsim.cu:451-511)
//                   follow.  Both count 32 samples at once in bit-sliced
//                   counters per lane, 4 temperatures of a quad per 16-byte load.
// records_kernel  : the reference's obs_s records from those integers.
// records_launch  : the three of them, queued on a stream.
// The kernels have internal linkage: each translation unit that launches
// them (the engine, the no-allocation records entry point) has its own copy
// of the same code.
#pragma once
#include <cstdint>

#include "philox.cuh"
#include "pt_kernel.cuh"

namespace csg {

static __global__ void init_kernel(uint32_t* spins, uint32_t* bonds, int L, int W, int C, int Q,
                            uint32_t k0, uint32_t k1, uint32_t word0) {
    const long N = (long)L * L * L;
    const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (long)W * N) return;
    const int w = (int)(idx / N);
    const int i = (int)(idx - (long)w * N);
    const int x = i % L, y = (i / L) % L, z = i / (L * L);
    const long slot = (long)((x + y + z) & 1) * (N / 2) + (long)(z * L + y) * (L / 2) + (x >> 1);
    const uint32_t wg = (uint32_t)w + word0;
    const u32x4 rb = philox4x32_10((uint32_t)i, 0u, wg, kTagBond, k0, k1);
    bonds[((long)w * 3 + 0) * N + slot] = rb.v0;
    bonds[((long)w * 3 + 1) * N + slot] = rb.v1;
    bonds[((long)w * 3 + 2) * N + slot] = rb.v2;
    uint4* sp = reinterpret_cast<uint4*>(spins);
    for (int c = 0; c < C; ++c)
        for (int q = 0; q < Q; ++q) {
            const u32x4 r = philox4x32_10((uint32_t)i, 0u, wg,
                                          kTagInit | ((uint32_t)c << 8) | (uint32_t)q, k0, k1);
            sp[(((long)w * C + c) * Q + q) * N + slot] = make_uint4(r.v0, r.v1, r.v2, r.v3);
        }
}

// The 4 planes of a quad at site n: one load, or four where the caller's spins
// are not on a 16-byte boundary (csg_obs_records_noalloc takes any).
template <bool ALIGNED>
__device__ __forceinline__ uint4 quad_at(const uint32_t* quad, int n) {
    if constexpr (ALIGNED) return reinterpret_cast<const uint4*>(quad)[n];
    const uint32_t* p = quad + (size_t)4 * n;
    return make_uint4(p[0], p[1], p[2], p[3]);
}

constexpr int kCountThreads = 256;
constexpr int kCountSites = 16;  // sites per thread of the bond counts

// Unsatisfied bonds u[w][c][t][b] and spins up n_up[w][c][t][b], added to what is
// there: blockIdx.x = quad (w, c, q), blockIdx.y = part of the sites (at most
// kCountSites per thread).
template <bool ALIGNED>
static __global__ void __launch_bounds__(kCountThreads) bond_counts_kernel(
    const uint32_t* __restrict__ spins, const uint32_t* __restrict__ bonds, int L, int T, int* u, int* n_up) {
    constexpr int NLU = bit_length(3 * kCountSites), NLM = bit_length(kCountSites);
    const int LH = L / 2, PL = L * LH, NH = L * PL, N = 2 * NH, Q = T / 4;
    const int gq = blockIdx.x, w = gq / (2 * Q), lane = threadIdx.x & 31;
    const uint32_t* const S = spins + (size_t)gq * N * 4;
    const uint32_t* const F = bonds + (size_t)w * 3 * N;
    __shared__ int sum[2][4][32];
    (&sum[0][0][0])[threadIdx.x] = 0;
    static_assert(kCountThreads == 2 * 4 * 32, "one sum per thread");
    __syncthreads();
    uint32_t cu[4][NLU] = {}, cm[4][NLM] = {};
    // the quotients by L L/2 and L/2 from a product with their reciprocals: the
    // halves added keep the result 1/16384 away from an integer, rounding 1/65536
    const float inv_pl = 1.0f / (float)PL, inv_lh = 1.0f / (float)LH;
    for (int n = blockIdx.y * kCountThreads + threadIdx.x; n < N; n += gridDim.y * kCountThreads) {
        const int p = n >= NH, m = n - p * NH;
        const int z = (int)(((float)m + 0.5f) * inv_pl), r = m - z * PL;
        const int y = (int)(((float)r + 0.5f) * inv_lh), h = r - y * LH;
        const int o = (y + z + p) & 1;  // x = 2h + o
        const int no = (1 - p) * NH + m;
        const uint4 s = quad_at<ALIGNED>(S, n);
        const uint4 ax = quad_at<ALIGNED>(S, no + (o ? (h == LH - 1 ? 1 - LH : 1) : 0));
        const uint4 ay = quad_at<ALIGNED>(S, no + (y == L - 1 ? LH - PL : LH));
        const uint4 az = quad_at<ALIGNED>(S, no + (z == L - 1 ? PL - NH : PL));
        const uint32_t fx = F[n], fy = F[N + n], fz = F[2 * N + n];
        const uint32_t sw[4] = {s.x, s.y, s.z, s.w}, xw[4] = {ax.x, ax.y, ax.z, ax.w};
        const uint32_t yw[4] = {ay.x, ay.y, ay.z, ay.w}, zw[4] = {az.x, az.y, az.z, az.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint32_t ux = xor3(sw[k], xw[k], fx), uy = xor3(sw[k], yw[k], fy), uz = xor3(sw[k], zw[k], fz);
            uint32_t c1, c2, carry;
            CSG_FA(cu[k][0], c1, cu[k][0], ux, uy);  // three words of weight 1
            c2 = cu[k][0] & uz;
            cu[k][0] ^= uz;
            CSG_FA(cu[k][1], carry, cu[k][1], c1, c2);
#pragma unroll
            for (int l = 2; l < NLU; ++l) {
                const uint32_t t = cu[k][l] & carry;
                cu[k][l] ^= carry;
                carry = t;
            }
            carry = sw[k];
#pragma unroll
            for (int l = 0; l < NLM; ++l) {
                const uint32_t t = cm[k][l] & carry;
                cm[k][l] ^= carry;
                carry = t;
            }
        }
    }
    int cnt[4];
    packed_column_counts<NLU>(cu, lane, cnt);
#pragma unroll
    for (int k = 0; k < 4; ++k) atomicAdd(&sum[0][k][lane], cnt[k]);
    packed_column_counts<NLM>(cm, lane, cnt);
#pragma unroll
    for (int k = 0; k < 4; ++k) atomicAdd(&sum[1][k][lane], cnt[k]);
    __syncthreads();
    const int what = threadIdx.x >> 7, i = threadIdx.x & 127;  // plane i / 32 of the quad, sample i & 31
    atomicAdd((what ? n_up : u) + (size_t)gq * 128 + i, (&sum[what][0][0])[i]);
}

// Sites where the copies differ in each coordinate plane, diff[w][t][dir][a][b]
// (dir 0, 1, 2 = x, y, z equal to a): a warp per (w, q, dir, a), blockIdx.x = (w,
// q), blockIdx.y = 4 of the 3L planes.  NL: bits of a lane's count, L L / 32 sites.
template <int NL, bool ALIGNED>
static __global__ void __launch_bounds__(128) overlap_planes_kernel(const uint32_t* __restrict__ spins, int L, int T,
                                                                    int* __restrict__ diff) {
    const int LH = L / 2, PL = L * LH, NH = L * PL, N = 2 * NH, Q = T / 4;
    const int w = blockIdx.x / Q, q = blockIdx.x - w * Q, lane = threadIdx.x & 31;
    const int plane = blockIdx.y * 4 + (threadIdx.x >> 5);
    if (plane >= 3 * L) return;
    const int dir = plane / L, a = plane - dir * L;
    const uint32_t* const A = spins + ((size_t)(w * 2) * Q + q) * N * 4;
    const uint32_t* const B = A + (size_t)Q * N * 4;
    uint32_t cd[4][NL] = {};
    const float inv_l = 1.0f / (float)L, inv_lh = 1.0f / (float)LH;
    for (int i = lane; i < L * L; i += 32) {
        int n;  // site i of the plane
        if (dir == 2) {
            n = i < PL ? a * PL + i : NH + a * PL + (i - PL);
        } else if (dir == 1) {  // rows (z, y = a): L/2 sites of each colour
            const int row = (int)(((float)i + 0.5f) * inv_lh), h = i - row * LH;
            n = (row & 1) * NH + ((row >> 1) * L + a) * LH + h;
        } else {  // i = z L + y
            const int z = (int)(((float)i + 0.5f) * inv_l), y = i - z * L;
            n = ((a + y + z) & 1) * NH + i * LH + (a >> 1);
        }
        const uint4 v = quad_at<ALIGNED>(A, n), x = quad_at<ALIGNED>(B, n);
        const uint32_t d[4] = {v.x ^ x.x, v.y ^ x.y, v.z ^ x.z, v.w ^ x.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            uint32_t carry = d[k];
#pragma unroll
            for (int l = 0; l < NL; ++l) {
                const uint32_t t = cd[k][l] & carry;
                cd[k][l] ^= carry;
                carry = t;
            }
        }
    }
    int cnt[4];
    packed_column_counts<NL>(cd, lane, cnt);
#pragma unroll
    for (int k = 0; k < 4; ++k) diff[(((size_t)w * T + 4 * q + k) * 3 * L + plane) * 32 + lane] = cnt[k];
}

// The reference records (obs_s: e[2], m[2], q_0, q_1_r[3], q_1_i[3]) of one
// (sample, temperature) from the counts above, with the float and double
// operations of the host formulas (eamsim.cu:320-325, 477-509) in the same
// order; cosv/sinv hold cos(k a), sin(k a), k = 2 pi / L, computed on the host.
// Built without contraction (-fmad=false), the records equal the host's bit for bit.
static __global__ void records_kernel(const int* __restrict__ u, const int* __restrict__ n_up,
                                      const int* __restrict__ diff, const double* __restrict__ cosv,
                                      const double* __restrict__ sinv, int L, int W, int T, float H,
                                      float* __restrict__ rec) {
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;  // (w, t, b), b fastest
    if (i >= (long)W * 32 * T) return;
    const int b = (int)(i & 31), t = (int)((i >> 5) % T), w = (int)((i >> 5) / T);
    const long long N = (long long)L * L * L;
    float* o = rec + (((size_t)w * 32 + b) * T + t) * 11;
    for (int c = 0; c < 2; ++c) {
        const size_t k = (((size_t)w * 2 + c) * T + t) * 32 + b;
        const int e = 2 * u[k] - 3 * (int)N;  // bond energy
        const float es = (float)(-e);
        const float ms = (float)(2 * n_up[k] - (int)N);
        o[c] = -(es + H * ms) / (float)N;
        o[2 + c] = ms / (float)N;
    }
    const int* d = diff + (size_t)(i >> 5) * 3 * L * 32 + b;
    long long D = 0;
    for (int dir = 0; dir < 3; ++dir) {
        double re = 0.0, im = 0.0;
        for (int a = 0; a < L; ++a) {
            const int n = d[(dir * L + a) * 32];
            if (dir == 0) D += n;
            const long long P = (long long)L * L - 2 * (long long)n;
            re += (double)P * cosv[a];
            im += (double)P * sinv[a];
        }
        o[5 + dir] = (float)(re / (double)N);
        o[8 + dir] = (float)(im / (double)N);
    }
    o[4] = (float)(N - 2 * D) / (float)N;
}

template <bool ALIGNED>
static const void* overlap_planes_for(int L) {
    const int sites = (L * L + 31) / 32;  // of a plane per lane
    return sites <= 3    ? reinterpret_cast<const void*>(overlap_planes_kernel<2, ALIGNED>)
           : sites <= 15 ? reinterpret_cast<const void*>(overlap_planes_kernel<4, ALIGNED>)
           : sites <= 63 ? reinterpret_cast<const void*>(overlap_planes_kernel<6, ALIGNED>)
                         : reinterpret_cast<const void*>(overlap_planes_kernel<10, ALIGNED>);
}

// Queues the records of a state on a stream.  counts: 2 W 2 T 32 ints (unsatisfied
// bonds, then spins up); diff: W T 32 3L ints; all of them written before they are
// read.  Bound: the loads, a pass over the spins and their neighbours and three
// over both copies; 2048 samples at L = 16, 24 temperatures: 102 us
// (47 + 33 + 22; a warp per (word, temperature) walking all sites took 1940)
static inline cudaError_t records_launch(const uint32_t* spins, const uint32_t* bonds, int L, int W, int T, float H,
                                         int* counts, int* diff, const double* cosv, const double* sinv, float* rec,
                                         cudaStream_t st) {
    const size_t n_e = (size_t)W * 2 * T * 32;
    const int Q = T / 4;
    const long N = (long)L * L * L;
    const bool aligned = reinterpret_cast<uintptr_t>(spins) % 16 == 0;
    int* u = counts;
    int* n_up = counts + n_e;
    cudaError_t ce = cudaMemsetAsync(counts, 0, 2 * n_e * sizeof(int), st);
    if (ce != cudaSuccess) return ce;
    {
        const long per_block = (long)kCountThreads * kCountSites;
        void* args[] = {&spins, &bonds, &L, &T, &u, &n_up};
        ce = cudaLaunchKernel(aligned ? reinterpret_cast<const void*>(bond_counts_kernel<true>)
                                      : reinterpret_cast<const void*>(bond_counts_kernel<false>),
                              dim3((unsigned)(W * 2 * Q), (unsigned)((N + per_block - 1) / per_block)),
                              dim3(kCountThreads), args, 0, st);
        if (ce != cudaSuccess) return ce;
    }
    {
        void* args[] = {&spins, &L, &T, &diff};
        ce = cudaLaunchKernel(aligned ? overlap_planes_for<true>(L) : overlap_planes_for<false>(L),
                              dim3((unsigned)(W * Q), (unsigned)((3 * L + 3) / 4)), dim3(128), args, 0, st);
        if (ce != cudaSuccess) return ce;
    }
    const long total = (long)W * 32 * T;
    void* args[] = {&u, &n_up, &diff, &cosv, &sinv, &L, &W, &T, &H, &rec};
    return cudaLaunchKernel(reinterpret_cast<const void*>(records_kernel), dim3((unsigned)((total + 127) / 128)),
                            dim3(128), args, 0, st);
}

}  // namespace csg
