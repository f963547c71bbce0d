// analysis_kernels.cu — the result table of a record series on the GPU.
//
// Restates the estimators of the reference's analyze-all.py (lines 38-71) as a
// two-kernel reduction over records already in device memory: per (sample,
// temperature) thermal sums over the measurements, then per temperature the
// disorder mean and variance of every sum (two passes, double precision).  The
// host forms chi_0, xi_L/L, e, m and their errors from those moments with the
// script's formulas.
//
// Bound: the records' bytes.  The thermal sums split the measurements so that
// every SM has work, and bring the 44-byte records in through shared memory
// with consecutive threads on consecutive words.  128 measurements of 2048 samples
// at 24 temperatures (277 MB): the call takes 105 us, 42 of them at
// the measured copy bandwidth; a thread per pair over all measurements, 44 bytes
// apart, took 600 to 770.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <string>
#include <vector>

#include "csg.h"
#include "engine_internal.h"

using csg_detail::fail;  // reported by csg_last_error()

namespace {

constexpr int kRecFloats = 11;  // obs_s: e[2], m[2], q_0, q_1_r[3], q_1_i[3]
constexpr int kSums = 9;        // q_0^2, q_1_r[a]^2 (3), q_1_i[a]^2 (3), e (both copies), m

constexpr int kTile = 256;       // (sample, temperature) pairs per block of the thermal sums
constexpr int kTileBlocks = 4;   // blocks per SM they are built for

// Thermal sums of kTile pairs over a part of the measurements: blockIdx.x =
// tile of pairs, blockIdx.y = part; parts[part][sum][pair].  A measurement's
// records of the tile are one contiguous stretch, copied to shared memory while
// the one before is added.
__global__ void __launch_bounds__(kTile, kTileBlocks)
    thermal_sums_kernel(const float* __restrict__ rec, long long n_meas, int n_pairs, double* __restrict__ parts) {
    __shared__ float buf[2][kTile * kRecFloats];
    const int p0 = blockIdx.x * kTile, tid = threadIdx.x;
    const int n = min(kTile, n_pairs - p0), words = n * kRecFloats;
    const long long m0 = n_meas * blockIdx.y / gridDim.y, m1 = n_meas * (blockIdx.y + 1) / gridDim.y;
    float next[kRecFloats];
    auto fetch = [&](long long m) {
        const float* src = rec + ((size_t)m * n_pairs + p0) * kRecFloats;
#pragma unroll
        for (int k = 0; k < kRecFloats; ++k) {
            const int i = k * kTile + tid;
            next[k] = i < words ? __ldcs(src + i) : 0.f;
        }
    };
    double acc[kSums] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    if (m0 < m1) fetch(m0);
    for (long long m = m0; m < m1; ++m) {
        float* const b = buf[m & 1];  // the other one may still be read
#pragma unroll
        for (int k = 0; k < kRecFloats; ++k) b[k * kTile + tid] = next[k];
        __syncthreads();
        if (m + 1 < m1) fetch(m + 1);
        const float* const v = b + tid * kRecFloats;
        const double q0 = v[4];
        acc[0] += q0 * q0;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const double qr = v[5 + a], qi = v[8 + a];
            acc[1 + a] += qr * qr;
            acc[4 + a] += qi * qi;
        }
        acc[7] += (double)v[0] + (double)v[1];
        acc[8] += (double)v[2] + (double)v[3];
    }
    if (tid < n)
#pragma unroll
        for (int k = 0; k < kSums; ++k)
            parts[((size_t)blockIdx.y * kSums + k) * n_pairs + p0 + tid] = acc[k];
}

// Disorder mean and variance (population, like numpy's var) of each thermal
// mean: blockIdx.x = temperature, blockIdx.y = sum; the parts of a thermal sum
// are added in order.
__global__ void disorder_moments_kernel(const double* __restrict__ parts, int n_parts, int ndis, int nrep,
                                        double n_meas, double* __restrict__ moments) {
    const int r = blockIdx.x, k = blockIdx.y;
    const size_t n_pairs = (size_t)ndis * nrep;
    __shared__ double red[256];
    // the thermal mean of e and m is over measurements and both copies
    auto value = [&](int d) {
        double v = 0.0;
        for (int c = 0; c < n_parts; ++c) v += parts[((size_t)c * kSums + k) * n_pairs + (size_t)d * nrep + r];
        v /= n_meas;
        return k >= 7 ? v / 2.0 : v;
    };
    auto total = [&](double s) {
        __syncthreads();
        red[threadIdx.x] = s;
        __syncthreads();
        for (int h = blockDim.x / 2; h > 0; h >>= 1) {
            if (threadIdx.x < h) red[threadIdx.x] += red[threadIdx.x + h];
            __syncthreads();
        }
        return red[0];
    };
    double s = 0.0;
    for (int d = threadIdx.x; d < ndis; d += blockDim.x) s += value(d);
    const double mean = total(s) / ndis;
    s = 0.0;
    for (int d = threadIdx.x; d < ndis; d += blockDim.x) {
        const double x = value(d) - mean;
        s += x * x;
    }
    const double var = total(s) / ndis;
    if (threadIdx.x == 0) {
        moments[((size_t)r * 2 + 0) * kSums + k] = mean;
        moments[((size_t)r * 2 + 1) * kSums + k] = var;
    }
}

}  // namespace

extern "C" {

int csg_analyze_records(const float* rec, int64_t n_meas, int32_t ndis, int32_t nrep, int32_t L,
                        double* table, void* stream) {
    if (!rec || !table) return fail(CSG_ERR_ARG, "null argument");
    if (n_meas < 1 || ndis < 1 || nrep < 1 || L < 4) return fail(CSG_ERR_ARG, "invalid dimensions");
    cudaStream_t st = (cudaStream_t)stream;
    const int n_pairs = ndis * nrep;
    int device = 0, nsm = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, device);
    if (e != cudaSuccess) return fail(CSG_ERR_CUDA, std::string("analysis: ") + cudaGetErrorString(e));
    // parts of the measurements: as many as one wave of blocks holds
    const int tiles = (n_pairs + kTile - 1) / kTile;
    const int n_parts = (int)std::max<int64_t>(1, std::min<int64_t>({(int64_t)(kTileBlocks * nsm / tiles), n_meas, 512}));
    double* dev = nullptr;
    const size_t n_sums = (size_t)n_parts * n_pairs * kSums, n_mom = (size_t)nrep * 2 * kSums;
    e = csg_detail::scratch_alloc(reinterpret_cast<void**>(&dev), (n_sums + n_mom) * sizeof(double), st);
    if (e != cudaSuccess) return fail(CSG_ERR_NOMEM, std::string("cudaMallocAsync: ") + cudaGetErrorString(e));
    thermal_sums_kernel<<<dim3((unsigned)tiles, (unsigned)n_parts), kTile, 0, st>>>(rec, n_meas, n_pairs, dev);
    disorder_moments_kernel<<<dim3((unsigned)nrep, kSums), 256, 0, st>>>(dev, n_parts, ndis, nrep, (double)n_meas,
                                                                         dev + n_sums);
    std::vector<double> mom(n_mom);
    e = cudaGetLastError();
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(mom.data(), dev + n_sums, n_mom * sizeof(double), cudaMemcpyDeviceToHost, st);
    const cudaError_t e2 = cudaFreeAsync(dev, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return fail(CSG_ERR_CUDA, std::string("analysis: ") + cudaGetErrorString(e));
    if (e2 != cudaSuccess) return fail(CSG_ERR_CUDA, std::string("cudaFreeAsync: ") + cudaGetErrorString(e2));
    // analyze-all.py:52-71, from the disorder moments
    const double pi = 3.14159265358979323846;
    for (int r = 0; r < nrep; ++r) {
        const double* mu = &mom[((size_t)r * 2 + 0) * kSums];
        const double* va = &mom[((size_t)r * 2 + 1) * kSums];
        const double chi0 = mu[0], chi0_v = va[0];
        double chi1 = 0.0, chi1_v = 0.0;
        for (int a = 0; a < 3; ++a) {
            chi1 += mu[1 + a] + mu[4 + a];
            chi1_v += va[1 + a] + va[4 + a];
        }
        chi1 /= 3.0;
        chi1_v /= 3.0;
        const double chif = chi0 / chi1;
        const double chif_v = chif * chif * (chi0_v / (chi0 * chi0) + chi1_v / (chi1 * chi1));
        const double xi = std::sqrt(chif - 1.0) / (2.0 * std::sin(pi / L)) / L;
        const double xi_f = xi / (2.0 * (chif - 1.0));
        const double xi_v = xi_f * xi_f * chif_v;
        double* o = table + (size_t)r * 8;
        o[0] = chi0;
        o[1] = std::sqrt(chi0_v / ndis);
        o[2] = xi;
        o[3] = std::sqrt(xi_v / ndis);
        o[4] = mu[7];
        o[5] = std::sqrt(va[7] / ndis);
        o[6] = mu[8];
        o[7] = std::sqrt(va[8] / ndis);
    }
    return CSG_OK;
}

}  // extern "C"
