// stream_kernels.cuh — parallel tempering for lattices whose temperature quads
// do not fit in shared memory (L > 24), streamed through L2/HBM.
//
// One sweep = one fused launch that updates both colours in a single pass
// over the state (stream_sweep.cu, while its ring of z-planes fits in shared
// memory: L <= 58) or two colour launches (stream_colour_kernel), then, when
// the schedule asks for it, the exchange decisions (stream_decide_kernel), the
// masked exchange and the overlap counts in one pass
// (stream_exchange_overlap_kernel; stream_exchange_kernel or
// stream_overlap_kernel when only one of them is due) and the measurement
// (stream_measure_kernel).  The arithmetic of a site update, of the energies
// and of the exchange rule is the same as the cluster-resident kernel's
// (pt_kernel.cuh), so results are bit-identical to it and to the CPU oracle.
// Blocks add their counts to per-plane totals with integer atomics (any order
// gives the same sums); the kernel that reads a total clears it.  The kernels
// are launched with programmatic dependent launch (pdl_enter).
#pragma once
#include <cstdint>
#include <type_traits>

#include "stream_params.cuh"

namespace csg {

// Address of element off of an array of 4- or 16-byte elements: one multiply-add
// on the multiply pipe.  Left to itself the compiler keeps a 64-bit pointer per
// neighbour and advances each with two adds on the logic/add pipe, which bounds
// the update.
template <typename T>
__device__ __forceinline__ T* elem(T* base, uint32_t off) {
    uint64_t a;
    asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(a) : "r"(off), "n"(sizeof(T)), "l"(base));
    return reinterpret_cast<T*>(a);
}

// The passes over the state go through z forwards and backwards in turn: a
// state larger than L2 (L = 48: 238 MB) then finds what the pass before touched
// last still there (a sweep with exchange and measurement 2 to 3 % faster, with
// exchange alone 4 %).
// Block i of n blocks of slots, the two colours' halves side by side in z.
__device__ __forceinline__ int walk_slots(int i, int n, bool back) {
    const int k = back ? n - 1 - i : i;
    return (k & 1) ? (n + 1) / 2 + k / 2 : k / 2;
}

__device__ __forceinline__ void prefetch_l1(const void* a) {
    asm volatile("prefetch.global.L1 [%0];" ::"l"(a));
}

// One colour of one sweep.  blockIdx.x = (w, q) for NC = 2 copies at once,
// (w, c, q) for NC = 1; blockIdx.y = block of kColourThreads sites of a
// z-plane x chunk of zb z-planes: a thread takes one site (y, h) of the
// plane's half in NC quads and walks zb planes along z, so that its in-plane
// neighbour offsets are fixed for the launch and the other colour's words at
// z - 1 and z are carried from plane to plane (5 instead of 7 loads of 16
// bytes a site).  The two copies of a temperature quad share its bonds,
// thresholds and addresses.  Consecutive blocks take the quads of one word at
// the same sites, so the word's bonds are read once from DRAM and then from L2.
// Bound: logic pipe and issue (56 and 60 % busy) with the latency of the loads
// that miss L1 in between.  256 samples, 2 copies, 32 temperatures, a launch:
// L = 48, 97 -> 75 us (counting: 133 -> 115); L = 32, 29 -> 25 (47 -> 37)
// against a thread per site with 7 loads and index arithmetic for each.
template <int FIELD, bool ACC_E, bool ACC_M, int NC>
__global__ void __launch_bounds__(kColourThreads, colour_blocks<FIELD, ACC_E, ACC_M, NC>())
    stream_colour_kernel(const __grid_constant__ StreamParams P, int p, long long s, int zb, int z_first, int z_step) {
    pdl_enter();
    constexpr int NLV = kStreamNLV, NLM = kStreamNLM;
    const int L = P.L, LH = L / 2, PL = L * LH;
    const int N = L * PL * 2, NH = L * PL;
    // quad gq0 + c * Q, c = 0 .. NC - 1
    const int bx = blockIdx.x, Q = P.Q;
    const int w = NC == 1 ? bx / (P.C * Q) : bx / Q, q = bx % Q;
    const int c0 = NC == 1 ? (bx / Q) % P.C : 0;
    const size_t gq0 = (size_t)(w * P.C + c0) * Q + q;
    const int npb = (PL + kColourThreads - 1) / kColourThreads;
    const int zc = blockIdx.y / npb, pb = blockIdx.y - zc * npb;
    const int z0 = z_first + zc * z_step, z1 = min(L, z0 + zb);
    const int lane = threadIdx.x & 31;
    const int i = pb * kColourThreads + threadIdx.x;  // (y, h) of the plane's half
    const bool active = i < PL;

    BondCounts<NLV> ecnt[NC][4];
    uint32_t mcnt[NC][4][NLM];
#pragma unroll
    for (int c = 0; c < NC; ++c)
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            ecnt[c][k].clear();
#pragma unroll
            for (int l = 0; l < NLM; ++l) mcnt[c][k][l] = 0;
        }
    if (active) {
        const int y = i / LH, h = i - y * LH;
        uint4* const Sq = reinterpret_cast<uint4*>(P.spins) + gq0 * N;
        const size_t copy = (size_t)Q * N;  // from a quad to the other copy's
        const uint32_t* const Fw = P.bonds + (size_t)w * 3 * N;
        uint32_t th0[4], th1[4], th2[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int t = 4 * q + k;
            th0[k] = P.tab.thr[t][0][0];
            th1[k] = P.tab.thr[t][0][1];
            th2[k] = P.tab.thr[t][0][2];
        }
        // the Philox rounds that do not depend on the site, once per launch
        PhiloxFixed pf[NC];
#pragma unroll
        for (int c = 0; c < NC; ++c)
            pf[c] = philox_fix((uint32_t)s, (uint32_t)w + P.word0, kTagSweep | ((uint32_t)(c0 + c) << 8) | (uint32_t)q,
                               P.k0, P.k1);
        // x & 1 of the site in planes z0, z0 + 2, ... is o0, in the others 1 - o0.
        // One x neighbour is the other colour's word at the same h (x + 1 of an
        // even x, x - 1 of an odd one), the other one at h - 1 or h + 1.
        const int o0 = (y + z0 + p) & 1;
        // element offsets from plane z of colour 0; oc, oo: this colour's and
        // the other's half
        const uint32_t oc = (uint32_t)(p * NH + i), oo = (uint32_t)((1 - p) * NH + i);
        const uint32_t iA = h == 0 ? oo + LH - 1 : oo - 1;     // x - 1 of an even x
        const uint32_t iB = h == LH - 1 ? oo - h : oo + 1;     // x + 1 of an odd x
        const uint32_t iE = o0 ? iB : iA, iO = o0 ? iA : iB;
        const uint32_t iYm = y == 0 ? oo + PL - LH : oo - LH;
        const uint32_t iYp = y == L - 1 ? oo - PL + LH : oo + LH;
        // bonds of the x neighbours: at the same h, and at h -+ 1 (the bond to
        // x - 1 belongs to the other colour's site, the one to x + 1 to this)
        const uint32_t fsE = o0 ? oo : oc, fdE = o0 ? oc : iA, fsO = o0 ? oc : oo, fdO = o0 ? iA : oc;
        const uint32_t f2o = (uint32_t)N + iYm, f3o = (uint32_t)N + oc;
        const uint32_t f4o = 2u * N + oo, f5o = 2u * N + oc;
        const uint32_t siteE = (uint32_t)(y * L + 2 * h + o0), siteO = (uint32_t)(y * L + 2 * h + 1 - o0);

        uint4 zm[NC], zcur[NC];
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            zm[c] = *elem(Sq + c * copy + (size_t)(z0 == 0 ? L - 1 : z0 - 1) * PL, oo);
            zcur[c] = *elem(Sq + c * copy + (size_t)z0 * PL, oo);
        }
        auto update_site = [&](const int z, const bool odd) {
            // the lines of the next two planes that no earlier load of this
            // block brought in: on their way while this site is updated
            // (L = 48: 75.0 us a launch instead of 79.5)
            const int zn = z == L - 1 ? 0 : z + 1, zq = z >= L - 2 ? z + 2 - L : z + 2;
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                prefetch_l1(elem(Sq + c * copy + (size_t)zn * PL, oc));
                prefetch_l1(elem(Sq + c * copy + (size_t)zq * PL, oo));
            }
            const uint32_t* const F = Fw + (size_t)z * PL;
            const uint32_t* const Fm = Fw + (size_t)(z == 0 ? L - 1 : z - 1) * PL;
            const uint32_t f0 = __ldg(elem(F, odd ? fsO : fsE)), f1 = __ldg(elem(F, odd ? fdO : fdE));
            const uint32_t f2 = __ldg(elem(F, f2o)), f3 = __ldg(elem(F, f3o));
            const uint32_t f4 = __ldg(elem(Fm, f4o)), f5 = __ldg(elem(F, f5o));
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                uint4* const S = Sq + c * copy + (size_t)z * PL;
                uint4* const Sp = Sq + c * copy + (size_t)zn * PL;
                uint4* const own = elem(S, oc);
                const uint4 cv = *own;
                const uint4 an = *elem(Sp, oo);
                const uint4 ad = *elem(S, odd ? iO : iE);
                const uint4 a2 = *elem(S, iYm), a3 = *elem(S, iYp);
                const u32x4 r = philox_c0((uint32_t)(z * L * L) + (odd ? siteO : siteE), pf[c]);
                const uint32_t rr[4] = {r.v0, r.v1, r.v2, r.v3};
                uint32_t cw[4] = {cv.x, cv.y, cv.z, cv.w};
                const uint32_t n0w[4] = {zcur[c].x, zcur[c].y, zcur[c].z, zcur[c].w};
                const uint32_t n1w[4] = {ad.x, ad.y, ad.z, ad.w};
                const uint32_t n2w[4] = {a2.x, a2.y, a2.z, a2.w}, n3w[4] = {a3.x, a3.y, a3.z, a3.w};
                const uint32_t n4w[4] = {zm[c].x, zm[c].y, zm[c].z, zm[c].w}, n5w[4] = {an.x, an.y, an.z, an.w};
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const uint32_t s0 = cw[k];
                    const uint32_t u0 = xor3(s0, n0w[k], f0), u1 = xor3(s0, n1w[k], f1);
                    const uint32_t u2 = xor3(s0, n2w[k], f2), u3 = xor3(s0, n3w[k], f3);
                    const uint32_t u4 = xor3(s0, n4w[k], f4), u5 = xor3(s0, n5w[k], f5);
                    const uint32_t sa = xor3(u0, u1, u2), ca = maj3(u0, u1, u2);
                    const uint32_t sb = xor3(u3, u4, u5), cb = maj3(u3, u4, u5);
                    uint32_t fl;
                    if constexpr (FIELD == kGeneralField) {
                        uint4 ta, tb;
                        gen_thresholds(P.tab, 4 * q + k, ta, tb);
                        fl = flip_gen(s0, sa, ca, sb, cb, rr[k], ta, tb, P.tab.ucut[4 * q + k][0],
                                      P.tab.ucut[4 * q + k][1]);
                        cw[k] = s0 ^ fl;
                    } else {
                        FlipTerms ft;
                        if constexpr (FIELD == kModerateField) {
                            uint4 ta, tb;
                            gen_thresholds(P.tab, 4 * q + k, ta, tb);
                            ft = flip_field_terms(s0, sa, ca, sb, cb, rr[k], ta, tb);
                        } else {
                            ft = flip_h0_terms(sa, ca, sb, cb, rr[k], th0[k], th1[k], th2[k]);
                        }
                        fl = ft.x | ft.y;
                        cw[k] = flipped(s0, ft);
                    }
                    // post-flip unsatisfied bonds (energy) and spins up, counted at once
                    if constexpr (ACC_E) {
                        if (odd)
                            ecnt[c][k].add_odd(sa, sb, ca, cb, fl);
                        else
                            ecnt[c][k].add_even(sa, sb, ca, cb, fl);
                    }
                    if constexpr (ACC_M) {
                        uint32_t carry = cw[k];
#pragma unroll
                        for (int l = 0; l < NLM; ++l) {
                            const uint32_t m = mcnt[c][k][l];
                            mcnt[c][k][l] = m ^ carry;
                            carry &= m;
                        }
                    }
                }
                *own = make_uint4(cw[0], cw[1], cw[2], cw[3]);
                zm[c] = zcur[c];
                zcur[c] = an;
            }
        };
#pragma unroll 1
        for (int z = z0; z < z1; z += 2) {  // L and zb are even
            update_site(z, false);
            update_site(z + 1, true);
        }
    }
    if constexpr (ACC_E || ACC_M) {
        __shared__ int sred[NC][2][4][32];
        for (int j = threadIdx.x; j < NC * 2 * 4 * 32; j += kColourThreads) (&sred[0][0][0][0])[j] = 0;
        __syncthreads();
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            // all lanes of a block hold counters of its quad: the 4 planes of
            // a warp in one 32x32 transpose per counter level
            int cnt[4];
            if constexpr (ACC_E) {
                uint32_t v[4][NLV];
#pragma unroll
                for (int k = 0; k < 4; ++k)
#pragma unroll
                    for (int l = 0; l < NLV; ++l) v[k][l] = ecnt[c][k].v[l];
                packed_column_counts<NLV>(v, lane, cnt);
#pragma unroll
                for (int k = 0; k < 4; ++k) atomicAdd(&sred[c][0][k][lane], cnt[k]);
            }
            if constexpr (ACC_M) {
                packed_column_counts<NLM>(mcnt[c], lane, cnt);
#pragma unroll
                for (int k = 0; k < 4; ++k) atomicAdd(&sred[c][1][k][lane], cnt[k]);
            }
        }
        __syncthreads();
        const int k = threadIdx.x >> 5;
        static_assert(kColourThreads == 128, "a warp per plane of the quad");
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            const size_t o = (((size_t)w * P.C + c0 + c) * P.T + 4 * q + k) * 32 + lane;
            if constexpr (ACC_E) atomicAdd(&P.u_acc[o], sred[c][0][k][lane]);
            if constexpr (ACC_M) atomicAdd(&P.up_acc[o], sred[c][1][k][lane]);
        }
    }
}

// Exchange decisions of one round: block = (w, c), one warp per pair.  Also
// totals the energies (and magnetisations) of every plane and swaps them for
// the accepted samples.
__global__ void stream_decide_kernel(const __grid_constant__ StreamParams P, long long s, int par,
                                     bool need_M, bool do_swap, unsigned long long* boundary,
                                     unsigned long long* swap_acc, unsigned int* swap_log,
                                     long long log_row, long long log_rows) {
    pdl_enter();
    const int wc = blockIdx.x, w = wc / P.C, c = wc % P.C;
    const int T = P.T, N = P.L * P.L * P.L;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    int* E = P.energy + (size_t)wc * T * 32;
    int* M = P.magn + (size_t)wc * T * 32;
    // totals of every plane of this (word, copy), cleared for the next sweep
    int* ua = P.u_acc + (size_t)wc * T * 32;
    int* pa = P.up_acc + (size_t)wc * T * 32;
    for (int i = threadIdx.x; i < T * 32; i += blockDim.x) {
        const int u = ua[i];
        ua[i] = 0;
        int up = 0;
        if (need_M) {
            up = pa[i];
            pa[i] = 0;
        }
        E[i] = 2 * u - 3 * N;
        M[i] = need_M ? 2 * up - N : 0;
    }
    __syncthreads();
    if (!do_swap) return;
    const uint32_t wg = (uint32_t)w + P.word0;
    for (int t = par + 2 * warp; t + 1 < T; t += 2 * nwarps) {
        const int e0 = E[t * 32 + lane], e1 = E[(t + 1) * 32 + lane];
        const int m0 = M[t * 32 + lane], m1 = M[(t + 1) * 32 + lane];
        const u32x4 r = philox4x32_10((uint32_t)(lane >> 1), (uint32_t)s, wg,
                                      kTagSwap | ((uint32_t)c << 8) | (uint32_t)t, P.k0, P.k1);
        const uint32_t lo = (lane & 1) ? r.v2 : r.v0;
        const uint32_t hi = (lane & 1) ? r.v3 : r.v1;
        const double uu = (double)((((unsigned long long)hi << 32) | lo) >> 11) * 0x1p-53;
        const double dE = __dsub_rn((double)(e0 - e1), __dmul_rn(P.H, (double)(m0 - m1)));
        const double delta = __dmul_rn(__dsub_rn(P.tab.beta[t], P.tab.beta[t + 1]), dE);
        bool acc = true;
        if (delta < 0.0) {
            const double pr = exp(delta);
            if (boundary && fabs(uu - pr) <= pr * 0x1p-40) atomicAdd(boundary, 1ull);
            acc = uu < pr;
        }
        const uint32_t mask = __ballot_sync(0xFFFFFFFFu, acc);
        if (acc) {
            E[t * 32 + lane] = e1;
            E[(t + 1) * 32 + lane] = e0;
            M[t * 32 + lane] = m1;
            M[(t + 1) * 32 + lane] = m0;
        }
        if (lane == 0) {
            P.masks[(size_t)wc * T + t] = mask;
            if (swap_acc) atomicAdd(&swap_acc[(size_t)c * T + t], (unsigned long long)__popc(mask));
            if (swap_log && log_row >= 0 && log_row < log_rows)
                swap_log[(((size_t)log_row * P.W + w) * P.C + c) * T + t] = mask;
        }
    }
    // pairs that do not take part in this round keep a zero mask
    for (int t = threadIdx.x; t < T; t += blockDim.x)
        if (((t - par) & 1) || t + 1 >= T) P.masks[(size_t)wc * T + t] = 0;
}

// Masked exchange: a thread takes one site of one (w, c) and every quad of it,
// so both words of every pair (also across quads) are its own.
__global__ void stream_exchange_kernel(const __grid_constant__ StreamParams P, int par, bool back) {
    pdl_enter();
    const long N = (long)P.L * P.L * P.L;
    const int wc = blockIdx.x;
    const long n = (long)walk_slots(blockIdx.y, gridDim.y, back) * blockDim.x + threadIdx.x;
    if (n >= N) return;
    uint4* base = reinterpret_cast<uint4*>(P.spins) + (size_t)wc * P.Q * N + n;
    const uint32_t* mk = P.masks + (size_t)wc * P.T;
    if (par == 0) {  // pairs (0,1), (2,3) inside every quad
        for (int q = 0; q < P.Q; ++q) {
            uint4 v = base[(size_t)q * N];
            const uint32_t d0 = (v.x ^ v.y) & mk[4 * q], d1 = (v.z ^ v.w) & mk[4 * q + 2];
            v.x ^= d0; v.y ^= d0; v.z ^= d1; v.w ^= d1;
            base[(size_t)q * N] = v;
        }
        return;
    }
    // odd rounds: (1,2) inside a quad, (3 of quad q, 0 of quad q+1) across quads
    uint4 cur = base[0];
    for (int q = 0; q < P.Q; ++q) {
        const uint32_t d = (cur.y ^ cur.z) & mk[4 * q + 1];
        cur.y ^= d;
        cur.z ^= d;
        if (q + 1 < P.Q) {
            uint4 nxt = base[(size_t)(q + 1) * N];
            const uint32_t e = (cur.w ^ nxt.x) & mk[4 * q + 3];
            cur.w ^= e;
            nxt.x ^= e;
            base[(size_t)q * N] = cur;
            cur = nxt;
        } else {
            base[(size_t)q * N] = cur;
        }
    }
}

// Exchange and overlap in one pass (sweeps that both exchange and measure, two
// copies): blockIdx.x = word, blockIdx.y = block of sites.  A thread takes
// kExchangeSites sites of both copies and walks the quads in order; on odd rounds quad q is
// final only after its pair (3 of q, 0 of q+1) is exchanged, so each quad is
// written (and its overlap counted) one step after it is loaded.  Every word
// is read and written by exactly one thread.  The block's overlap counts are
// added to d_acc, as in stream_overlap_kernel.
__global__ void __launch_bounds__(kStreamThreads) stream_exchange_overlap_kernel(
    const __grid_constant__ StreamParams P, int par, bool back) {
    pdl_enter();
    constexpr int kSites = kExchangeSites;
    const int N = P.L * P.L * P.L, T = P.T, Q = P.Q;
    const int w = blockIdx.x, blk = walk_slots(blockIdx.y, gridDim.y, back), lane = threadIdx.x & 31;
    __shared__ int sD[kMaxT][32];
    for (int i = threadIdx.x; i < T * 32; i += kStreamThreads) (&sD[0][0])[i] = 0;
    __syncthreads();
    uint4* base0 = reinterpret_cast<uint4*>(P.spins) + (size_t)(w * 2 + 0) * Q * N;
    uint4* base1 = reinterpret_cast<uint4*>(P.spins) + (size_t)(w * 2 + 1) * Q * N;
    const uint32_t* mk0 = P.masks + (size_t)(w * 2 + 0) * T;
    const uint32_t* mk1 = P.masks + (size_t)(w * 2 + 1) * T;
    int site[kSites];
#pragma unroll
    for (int i = 0; i < kSites; ++i) site[i] = blk * kExchangeSitesPerBlock + i * kStreamThreads + threadIdx.x;
    uint4 prv[2][kSites], cur[2][kSites];
    // store quad qq and add its overlap counts
    auto finish = [&](int qq, uint4 (&v)[2][kSites]) {
        uint32_t cnt[4][kExchangeNL] = {};
#pragma unroll
        for (int i = 0; i < kSites; ++i) {
            if (site[i] < N) {
                base0[(size_t)qq * N + site[i]] = v[0][i];
                base1[(size_t)qq * N + site[i]] = v[1][i];
            }
            const uint32_t x[4] = {v[0][i].x ^ v[1][i].x, v[0][i].y ^ v[1][i].y, v[0][i].z ^ v[1][i].z,
                                   v[0][i].w ^ v[1][i].w};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                uint32_t carry = x[k];
#pragma unroll
                for (int l = 0; l < kExchangeNL; ++l) {
                    const uint32_t t = cnt[k][l] & carry;
                    cnt[k][l] ^= carry;
                    carry = t;
                }
            }
        }
        int n[4];
        packed_column_counts<kExchangeNL>(cnt, lane, n);
#pragma unroll
        for (int k = 0; k < 4; ++k) atomicAdd(&sD[4 * qq + k][lane], n[k]);
    };
    for (int q = 0; q < Q; ++q) {
        const uint32_t a0 = mk0[4 * q], a1 = mk0[4 * q + 1], a2 = mk0[4 * q + 2];
        const uint32_t b0 = mk1[4 * q], b1 = mk1[4 * q + 1], b2 = mk1[4 * q + 2];
#pragma unroll
        for (int i = 0; i < kSites; ++i) {
            const bool ok = site[i] < N;
            uint4 u = ok ? base0[(size_t)q * N + site[i]] : make_uint4(0, 0, 0, 0);
            uint4 v = ok ? base1[(size_t)q * N + site[i]] : make_uint4(0, 0, 0, 0);
            if (par == 0) {  // (0,1) and (2,3) inside the quad
                uint32_t d = (u.x ^ u.y) & a0; u.x ^= d; u.y ^= d;
                d = (u.z ^ u.w) & a2; u.z ^= d; u.w ^= d;
                d = (v.x ^ v.y) & b0; v.x ^= d; v.y ^= d;
                d = (v.z ^ v.w) & b2; v.z ^= d; v.w ^= d;
            } else {  // (1,2) inside; (3 of q-1, 0 of q) across
                uint32_t d = (u.y ^ u.z) & a1; u.y ^= d; u.z ^= d;
                d = (v.y ^ v.z) & b1; v.y ^= d; v.z ^= d;
                if (q > 0) {
                    d = (prv[0][i].w ^ u.x) & mk0[4 * q - 1]; prv[0][i].w ^= d; u.x ^= d;
                    d = (prv[1][i].w ^ v.x) & mk1[4 * q - 1]; prv[1][i].w ^= d; v.x ^= d;
                }
            }
            cur[0][i] = u;
            cur[1][i] = v;
        }
        if (q > 0) finish(q - 1, prv);
#pragma unroll
        for (int i = 0; i < kSites; ++i) {
            prv[0][i] = cur[0][i];
            prv[1][i] = cur[1][i];
        }
    }
    finish(Q - 1, prv);
    __syncthreads();
    for (int i = threadIdx.x; i < T * 32; i += kStreamThreads) {
        const int t = i >> 5, b = i & 31;
        atomicAdd(&P.d_acc[((size_t)w * T + t) * 32 + b], sD[t][b]);
    }
}

// Overlap counts: blockIdx.x = (w, q), blockIdx.y = block of sites; each
// thread kOverlapSPT sites; the block's counts are added to d_acc.
__global__ void __launch_bounds__(kStreamThreads) stream_overlap_kernel(const __grid_constant__ StreamParams P) {
    pdl_enter();
    const long N = (long)P.L * P.L * P.L;
    const int wq = blockIdx.x, w = wq / P.Q, q = wq % P.Q;
    const int lane = threadIdx.x & 31;
    const uint4* A = reinterpret_cast<const uint4*>(P.spins) + ((size_t)(w * P.C + 0) * P.Q + q) * N;
    const uint4* B = reinterpret_cast<const uint4*>(P.spins) + ((size_t)(w * P.C + 1) * P.Q + q) * N;
    constexpr int NL = kOverlapNL;
    uint32_t dc[4][NL];
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int l = 0; l < NL; ++l) dc[k][l] = 0;
    const long n_base = (long)blockIdx.y * kOverlapSitesPerBlock + threadIdx.x;
    for (int m = 0; m < kOverlapSPT; ++m) {
        const long n = n_base + (long)m * kStreamThreads;
        uint4 x = make_uint4(0, 0, 0, 0);
        if (n < N) {
            const uint4 a = __ldg(A + n), b = __ldg(B + n);
            x = make_uint4(a.x ^ b.x, a.y ^ b.y, a.z ^ b.z, a.w ^ b.w);
        }
        const uint32_t xs[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            uint32_t carry = xs[k];
#pragma unroll
            for (int l = 0; l < NL; ++l) {
                const uint32_t t = dc[k][l] & carry;
                dc[k][l] ^= carry;
                carry = t;
            }
        }
    }
    __shared__ int sred[4][32];
    for (int i = threadIdx.x; i < 128; i += kStreamThreads) (&sred[0][0])[i] = 0;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 4; ++k) atomicAdd(&sred[k][lane], column_count<NL>(dc[k], lane));
    __syncthreads();
    if (threadIdx.x < 128) {
        const int k = threadIdx.x >> 5;
        atomicAdd(&P.d_acc[((size_t)w * P.T + 4 * q + k) * 32 + lane], sred[k][lane]);
    }
}

// Measurement accumulators from the energies and the overlap totals:
// blockIdx.x = (word, temperature), thread = (copy, sample); the first 32
// threads also take (and clear) the plane's overlap totals.
__global__ void stream_measure_kernel(const __grid_constant__ StreamParams P, bool need_M,
                                      StreamObs O) {
    pdl_enter();
    const int w = blockIdx.x / P.T, t = blockIdx.x % P.T, T = P.T, N = P.L * P.L * P.L;
    const int c = threadIdx.x >> 5, b = threadIdx.x & 31;
    if (c < P.C) {
        const size_t o = (((size_t)w * P.C + c) * T + t) * 32 + b;
        const int e = P.energy[o], m = P.magn[o];
        if (O.e_sum) atomicAdd(reinterpret_cast<unsigned long long*>(O.e_sum + o), (unsigned long long)(long long)e);
        if (O.e_last) O.e_last[o] = e;
        if (need_M) {
            if (O.m_sum) atomicAdd(reinterpret_cast<unsigned long long*>(O.m_sum + o), (unsigned long long)(long long)m);
            if (O.m_last) O.m_last[o] = m;
        }
    }
    if (P.C != 2 || c != 0) return;
    int* dp = P.d_acc + ((size_t)w * T + t) * 32 + b;
    const int D = *dp;
    *dp = 0;
    const long long Qv = (long long)N - 2LL * D;
    const unsigned long long q2 = (unsigned long long)(Qv * Qv);
    const size_t o = ((size_t)w * T + t) * 32 + b;
    if (O.q_sum) atomicAdd(reinterpret_cast<unsigned long long*>(O.q_sum + o), (unsigned long long)Qv);
    if (O.q2_sum) atomicAdd(reinterpret_cast<unsigned long long*>(O.q2_sum + o), q2);
    if (O.q4_sum) {
        const unsigned long long lo = q2 * q2, hi = __umul64hi(q2, q2);
        atomicAdd(O.q4_sum + 2 * o, lo & 0xFFFFFFFFull);
        atomicAdd(O.q4_sum + 2 * o + 1, (lo >> 32) | (hi << 32));
    }
    if (O.hist) atomicAdd(&O.hist[(size_t)t * (N + 1) + D], 1u);
    if (O.d_last) O.d_last[o] = D;
}

}  // namespace csg
