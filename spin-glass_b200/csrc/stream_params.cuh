// stream_params.cuh — what the streaming engine's kernels (stream_kernels.cuh,
// stream_sweep.cu) and its host code share: launch shapes, the parameter
// block, the measurement accumulators and programmatic dependent launch.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "philox.cuh"
#include "pt_kernel.cuh"

namespace csg {


// Colour launches: blocks of kColourThreads sites of a z-plane's half, walking
// at most kColourMaxZ planes (colour_planes in csg_engine.cu chooses how many).
constexpr int kColourThreads = 128;
constexpr int kColourMaxZ = 16;
constexpr int kStreamNLV = bit_length(6 * kColourMaxZ);  // bits of a per-thread bond count
constexpr int kStreamNLM = bit_length(kColourMaxZ);      // bits of a per-thread site count
// Copies of a temperature quad a colour launch's thread takes: both where it
// only updates (shared bonds, thresholds and addresses); one where it counts,
// since two sets of counters spill (L = 48: 139 against 120 us a launch).
template <bool ACC>
__host__ __device__ constexpr int colour_copies(int copies) { return ACC ? 1 : copies; }
// Blocks per SM the colour kernel is built for, by the registers each variant
// needs without spills that cost (a counting launch at 5 blocks, 96 registers:
// 120 us at L = 48 and 42 at L = 32; at 4, 116 registers: 115 and 37).
template <int FIELD, bool ACC_E, bool ACC_M, int NC>
__host__ __device__ constexpr int colour_blocks() {
    return ACC_E || ACC_M ? 4 : NC == 2 ? (FIELD ? 4 : 5) : (FIELD ? 6 : 7);
}
constexpr int kStreamThreads = 256;  // threads per block of the overlap passes
// Overlap passes (both copies of every quad): blocks of kStreamThreads threads
// over kOverlapSitesPerBlock sites (all N sites of a lattice).
constexpr int kOverlapSPT = 8;
constexpr int kOverlapSitesPerBlock = kStreamThreads * kOverlapSPT;
constexpr int kOverlapNL = bit_length(kOverlapSPT);

// Exchange and overlap pass: sites per thread.  Two leave 64 registers and
// blocks of 512 sites (4 blocks an SM, 512 blocks at L = 32 and 256 samples,
// where blocks of 2048 were 128 for 148 SMs); four: 119 registers, 1 to 5 %
// slower a pass of the engine.
constexpr int kExchangeSites = 2;
constexpr int kExchangeSitesPerBlock = kStreamThreads * kExchangeSites;
constexpr int kExchangeNL = bit_length(kExchangeSites);

struct StreamParams {
    uint32_t* spins;
    const uint32_t* bonds;
    // per-plane totals, added to by the blocks (integer atomics: any order gives
    // the same sums) and cleared by the kernel that consumes them
    int* u_acc;   // [W][C][T][32] unsatisfied bonds after the sweep
    int* up_acc;  // [W][C][T][32] spins up after the sweep
    int* d_acc;   // [W][T][32] sites where the copies differ
    int* energy;  // [W][C][T][32] bond energies after the exchange
    int* magn;    // [W][C][T][32]
    uint32_t* masks;  // [W][C][T] accepted-sample masks of the current round
    int* err;         // set to 1 by a sweep launch whose staging wait gave up
    int L, W, C, T, Q;
    int nblk2;  // blocks per quad of an overlap pass (over all N sites)
    uint32_t k0, k1, word0;
    double H;
    PtTables tab;
};

// The fused sweep launch (stream_sweep.cu): both colours of one sweep in one
// pass over the state, for lattices whose ring of z-planes fits in shared
// memory (stream_sweep_fits).  Energies (acc_e) and magnetisations (acc_m) go
// to the same per-plane totals as the colour launches' counts.
bool stream_sweep_fits(int L);
// Threads per CTA (one CTA per quad) and dynamic shared memory of the fused
// sweep launch for lattice side L (zeros where it does not fit).
void stream_sweep_shape(int L, int* threads, int* smem_bytes);
cudaError_t launch_stream_sweep(const StreamParams& P, long long s, bool gen, bool acc_e, bool acc_m,
                                cudaStream_t st);

// Measurement accumulators (layouts as in PtParams / csg_device_obs).
struct StreamObs {
    long long* e_sum;
    long long* m_sum;
    long long* q_sum;
    long long* q2_sum;
    unsigned long long* q4_sum;
    unsigned int* hist;
    int* e_last;
    int* m_last;
    int* d_last;
};

// Programmatic dependent launch (the sweep's kernels are launched with it): a
// kernel waits here until the previous kernel on the stream has finished and
// its writes are visible, then lets the next kernel's blocks be scheduled as
// soon as all of its own blocks run, so launch latency overlaps the tail.
__device__ __forceinline__ void pdl_enter() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

}  // namespace csg
