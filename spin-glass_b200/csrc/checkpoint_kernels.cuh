// checkpoint_kernels.cuh — conversion between the engine's state and the
// reference's checkpoint layout (eamsim.cu:655-676) on the device.
//
// A checkpoint holds one uint32 per (sample, copy, site): bits 0..T-1 the
// spins by temperature, bits 26..31 the six bonds -x,+x,-y,+y,-z,+z (1 =
// ferromagnetic).  The engine holds one uint32 per (32 samples, copy,
// temperature, site).  For one (word of samples, copy, site) the two are the
// rows and the columns of a 32x32 bit matrix, so a conversion is a transpose,
// done by one thread in registers: consecutive threads take consecutive sites,
// and each of its 32 checkpoint words is read or written coalesced.  Bound: the
// copies between the host and the device; 1024 samples at L = 16 (34 MB each way)
// took 300 ms for a load and a save when the host converted bit by bit.
#pragma once
#include <cstdint>

namespace csg {

// a[r] bit b <-> a[b] bit r
__device__ __forceinline__ void transpose32(uint32_t (&a)[32]) {
#pragma unroll
    for (int j = 16; j >= 1; j >>= 1) {
        const uint32_t m = j == 16 ? 0x0000FFFFu
                         : j == 8  ? 0x00FF00FFu
                         : j == 4  ? 0x0F0F0F0Fu
                         : j == 2  ? 0x33333333u
                                   : 0x55555555u;
#pragma unroll
        for (int k = 0; k < 32; ++k) {
            if (k & j) continue;
            const uint32_t t = ((a[k] >> j) ^ a[k + j]) & m;
            a[k + j] ^= t;
            a[k] ^= t << j;
        }
    }
}

struct CheckpointDims {
    int L, T;       // lattice side, temperatures (<= 24)
    int w0, words;  // the words a launch converts: w0 .. w0 + words - 1
};

__device__ __forceinline__ long checkpoint_slot(int L, int x, int y, int z) {
    return (long)((x + y + z) & 1) * ((long)L * L * L / 2) + (long)(z * L + y) * (L / 2) + (x >> 1);
}

// State -> checkpoint: thread = (word, copy, site); ref holds the launch's words.
static __global__ void __launch_bounds__(128) checkpoint_save_kernel(const uint32_t* __restrict__ spins,
                                                                     const uint32_t* __restrict__ bonds,
                                                                     CheckpointDims d, uint32_t* __restrict__ ref) {
    const int L = d.L;
    const long N = (long)L * L * L;
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    const int wl = blockIdx.y >> 1, c = blockIdx.y & 1;
    const int w = d.w0 + wl;
    const int x = (int)(i % L), y = (int)(i / L % L), z = (int)(i / ((long)L * L));
    const int xm = x == 0 ? L - 1 : x - 1, ym = y == 0 ? L - 1 : y - 1, zm = z == 0 ? L - 1 : z - 1;
    const long s = checkpoint_slot(L, x, y, z);
    uint32_t a[32];
    const uint4* sp = reinterpret_cast<const uint4*>(spins) + ((long)w * 2 + c) * (d.T / 4) * N + s;
#pragma unroll
    for (int q = 0; q < 6; ++q) {
        const uint4 v = 4 * q < d.T ? sp[q * N] : make_uint4(0, 0, 0, 0);
        a[4 * q] = v.x;
        a[4 * q + 1] = v.y;
        a[4 * q + 2] = v.z;
        a[4 * q + 3] = v.w;
    }
    a[24] = a[25] = 0u;
    const uint32_t* f = bonds + (long)w * 3 * N;
    a[26] = ~f[checkpoint_slot(L, xm, y, z)];
    a[27] = ~f[s];
    a[28] = ~f[N + checkpoint_slot(L, x, ym, z)];
    a[29] = ~f[N + s];
    a[30] = ~f[2 * N + checkpoint_slot(L, x, y, zm)];
    a[31] = ~f[2 * N + s];
    transpose32(a);
    uint32_t* out = ref + ((long)wl * 64 + c) * N + i;
#pragma unroll
    for (int b = 0; b < 32; ++b) out[2 * b * N] = a[b];
}

// Checkpoint -> state: thread = (word, copy, site).
static __global__ void __launch_bounds__(128) checkpoint_load_kernel(const uint32_t* __restrict__ ref,
                                                                     CheckpointDims d, uint32_t* __restrict__ spins,
                                                                     uint32_t* __restrict__ bonds) {
    const int L = d.L;
    const long N = (long)L * L * L;
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    const int wl = blockIdx.y >> 1, c = blockIdx.y & 1;
    const int w = d.w0 + wl;
    const uint32_t* in = ref + ((long)wl * 64 + c) * N + i;
    uint32_t a[32];
#pragma unroll
    for (int b = 0; b < 32; ++b) a[b] = in[2 * b * N];
    transpose32(a);
    const long s = checkpoint_slot(L, (int)(i % L), (int)(i / L % L), (int)(i / ((long)L * L)));
    uint4* sp = reinterpret_cast<uint4*>(spins) + ((long)w * 2 + c) * (d.T / 4) * N + s;
#pragma unroll
    for (int q = 0; q < 6; ++q)
        if (4 * q < d.T) sp[q * N] = make_uint4(a[4 * q], a[4 * q + 1], a[4 * q + 2], a[4 * q + 3]);
    if (c == 0)
#pragma unroll
        for (int k = 0; k < 3; ++k) bonds[((long)w * 3 + k) * N + s] = ~a[27 + 2 * k];
}

// Bond bits of a checkpoint: the copies of a sample must agree, and so must the
// two ends of every bond.  first receives the smallest ((w N + i) 32 + b) 2 +
// kind of a violation (kind 0: copies, 1: ends): the one a walk over words,
// sites and samples meets first.
static __global__ void __launch_bounds__(128) checkpoint_check_kernel(const uint32_t* __restrict__ ref,
                                                                      CheckpointDims d, unsigned long long* first) {
    const int L = d.L;
    const long N = (long)L * L * L;
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    const int wl = blockIdx.y;
    const int x = (int)(i % L), y = (int)(i / L % L), z = (int)(i / ((long)L * L));
    const long nb[3] = {((long)z * L + y) * L + (x + 1 == L ? 0 : x + 1),
                        ((long)z * L + (y + 1 == L ? 0 : y + 1)) * L + x,
                        ((long)(z + 1 == L ? 0 : z + 1) * L + y) * L + x};
    for (int b = 0; b < 32; ++b) {
        const uint32_t* r = ref + ((long)wl * 64 + 2 * b) * N;
        const uint32_t v0 = r[i], v1 = r[N + i];
        const bool copies = (v0 >> 26) != (v1 >> 26);
        bool ends = false;
#pragma unroll
        for (int k = 0; k < 3; ++k) ends |= (((v0 >> (27 + 2 * k)) ^ (r[nb[k]] >> (26 + 2 * k))) & 1u) != 0;
        if (copies || ends) {
            const unsigned long long at = ((unsigned long long)(d.w0 + wl) * N + i) * 32 + b;
            atomicMin(first, at * 2 + (copies ? 0 : 1));
            return;
        }
    }
}

}  // namespace csg
