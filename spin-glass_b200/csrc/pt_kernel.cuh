// pt_kernel.cuh — what the parallel-tempering kernels share: launch
// parameters, acceptance tables, the bit-sliced counting helpers and the flip
// rules, and the thread layout of the cluster-resident kernel
// (pt_resident.cuh, instantiated per lattice side in pt_instances.cu).
//
// Work decomposition of the resident kernel.  A thread-block cluster owns one
// sample word w (32 disorder samples) with all its copies and temperatures.
// The word's C*T/4 temperature quads (4 planes of N uint32 each) are split
// over the K CTAs of the cluster, Qc quads per CTA, and stay in shared memory
// for the whole launch (a section of sweeps).  Nothing but the bonds
// (read-only, through L1) touches global memory between the load at the
// start and the store at the end.
#pragma once
#include <cooperative_groups.h>

#include <cstdint>
#include <type_traits>

#include "philox.cuh"

namespace csg {
namespace cgx = cooperative_groups;

constexpr int kMaxT = 64;
constexpr int kMaxThreads = 512;  // CTA size cap: keeps 128 registers per thread available
// The field kernels whose threads each walk a whole column (one segment) keep
// more state live per site than 128 registers hold; their CTAs are capped at 384
// threads, which leaves 168 registers per thread.  The rule of fields below 2
// then spills nothing at L = 16 (up to 60 bytes of stores and 80 of loads elsewhere,
// L = 20), the general rule 60 to 116 and 96 to 152 (pt_resident.cuh, kSiteGroup).
constexpr int kMaxThreadsGenWalk = 384;
__host__ __device__ constexpr int max_cta_threads(bool gen, int nseg) {
    return gen && nseg == 1 ? kMaxThreadsGenWalk : kMaxThreads;
}

// Which acceptance rule a kernel is built for (csg_engine.cu, build_tables).
enum FieldMode { kNoField = 0, kModerateField = 1, kGeneralField = 2 };

struct PtTables {
    double beta[kMaxT];
    uint32_t thr[kMaxT][2][7];  // acceptance thresholds, valid for U < ucut
    uint8_t ucut[kMaxT][2];     // first U that is always accepted
};

struct PtParams {
    uint32_t* spins;
    const uint32_t* bonds;
    long long* e_sum;
    long long* m_sum;
    long long* q_sum;
    long long* q2_sum;
    unsigned long long* q4_sum;
    unsigned int* hist;
    int* e_last;
    int* m_last;
    int* d_last;
    unsigned long long* swap_acc;
    unsigned int* swap_log;
    long long swap_log_rounds;
    long long swap_round0;
    unsigned long long* boundary;
    double H;
    uint32_t k0, k1;
    uint32_t word0;  // global index of word 0 (Philox counter word 2)
    int W, C, T, Q;
    int K, Qc;
    long long sweep0;
    const long long* sweep_dev;  // if set, added to sweep0 (lets a captured graph advance)
    int n_sweeps;
    int sps, spm;
    long long meas_start;
    int flags;
    PtTables tab;
};

constexpr int kFlagMeasureM = 1;

__host__ __device__ constexpr int bit_length(int v) {
    int b = 0;
    while (v > 0) {
        ++b;
        v >>= 1;
    }
    return b;
}

// Thread layout of the resident kernel for lattice side L: every thread of a
// quad's team owns one column (y, x/2) of a checkerboard colour and a segment
// of ZS = L / NSEG consecutive z; the team has TPQ = L * L/2 * NSEG threads.
// Walking its column along z, a thread finds all six neighbours and bonds of
// each site at offsets fixed for the whole launch (only the first and last
// site of a segment may wrap around in z).
template <int L, int NSEG>
struct Walk {
    static_assert(L % 2 == 0 && L % NSEG == 0, "segments must tile the column");
    static constexpr int LH = L / 2;
    static constexpr int N = L * L * L;
    static constexpr int NH = N / 2;
    static constexpr int PL = L * LH;                          // sites of a colour per z-plane
    static constexpr int NC = PL;                              // columns per colour
    static constexpr int ZS = L / NSEG;                        // sites per thread per colour
    static constexpr int TPQ = NC * NSEG;                      // threads per quad
    static constexpr int NLV = bit_length(6 * ZS);             // energy counter levels
    static constexpr int MPT = (N + 4 * TPQ - 1) / (4 * TPQ);  // 4-site groups per thread
    static constexpr int NLD = bit_length(4 * MPT);            // magnetisation counter levels
    static constexpr int MPH = (NH + 4 * TPQ - 1) / (4 * TPQ); // 4-site groups per half lattice
    static constexpr int NLH = bit_length(4 * MPH);            // overlap counter levels
    static_assert(TPQ >= 32, "a warp spans at most two quads");
};

// Column splits (segments per column) the resident kernel is built with, for
// each L.  The first entry is the default; the first tuned_splits(L) are the
// ones a full GPU may want (and the batch tuner tries), the others are larger
// teams that pay where an SM has few quads (make_plan weighs them all).
__host__ __device__ constexpr int nseg_option(int L, int i) {
    return L == 4 ? (i == 0 ? 4 : 0)
         : L == 6 ? (i == 0 ? 2 : i == 1 ? 6 : 0)
         : L == 8 ? (i == 0 ? 2 : i == 1 ? 1 : i == 2 ? 4 : i == 3 ? 8 : 0)
         : L == 10 ? (i == 0 ? 2 : i == 1 ? 1 : i == 2 ? 5 : 0)
         : L == 12 ? (i == 0 ? 1 : i == 1 ? 2 : i == 2 ? 4 : i == 3 ? 6 : 0)
         : L == 14 ? (i == 0 ? 1 : i == 1 ? 2 : 0)
         : L == 16 ? (i == 0 ? 1 : i == 1 ? 2 : i == 2 ? 4 : 0)
         : L == 18 ? (i == 0 ? 1 : i == 1 ? 3 : 0)
         : L == 20 ? (i == 0 ? 1 : i == 1 ? 2 : 0)
         : (i == 0 ? 1 : 0);
}
__host__ __device__ constexpr int tuned_splits(int L) { return L >= 8 && L <= 16 ? 2 : 1; }
__host__ __device__ constexpr int threads_per_quad(int L, int nseg) { return L * (L / 2) * nseg; }

// One three-input logic instruction with truth table LUT (a = 0xF0, b = 0xCC,
// c = 0xAA).  The update path is bound by the logic pipe (64 lanes per clock
// and SM), so its gates are pinned one by one: left as C expressions, the
// compiler reassociated the XORs across the adders and a site word took 49
// logic instructions beside its Philox share instead of the 23 written (55 to
// 29 with it at L = 16).
template <int LUT>
__device__ __forceinline__ uint32_t lop3(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("lop3.b32 %0, %1, %2, %3, %4;" : "=r"(d) : "r"(a), "r"(b), "r"(c), "n"(LUT));
    return d;
}
__device__ __forceinline__ uint32_t xor3(uint32_t a, uint32_t b, uint32_t c) { return lop3<0x96>(a, b, c); }
__device__ __forceinline__ uint32_t maj3(uint32_t a, uint32_t b, uint32_t c) { return lop3<0xE8>(a, b, c); }

#define CSG_FA(s, cy, a, b, c)                             \
    do {                                                   \
        const uint32_t fa_a = (a), fa_b = (b), fa_c = (c); \
        (s) = xor3(fa_a, fa_b, fa_c);                      \
        (cy) = maj3(fa_a, fa_b, fa_c);                     \
    } while (0)

// Bit-sliced counter update: value += a1 + a2 + 2*(a3 + a4).
template <int NLV>
__device__ __forceinline__ void vc_add_site(uint32_t (&v)[NLV], uint32_t a1, uint32_t a2,
                                            uint32_t a3, uint32_t a4) {
    uint32_t k1, k2a, k2b, k3;
    CSG_FA(v[0], k1, v[0], a1, a2);
    CSG_FA(v[1], k2a, v[1], a3, a4);
    k2b = v[1] & k1;
    v[1] ^= k1;
    if constexpr (NLV > 2) {
        CSG_FA(v[2], k3, v[2], k2a, k2b);
#pragma unroll
        for (int l = 3; l < NLV; ++l) {
            const uint32_t t = v[l] & k3;
            v[l] ^= k3;
            k3 = t;
        }
    }
}

// Two sites at once: value += a1+a2+b1+b2 + 2*(a3+a4+b3+b4).
template <int NLV>
__device__ __forceinline__ void vc_add_2sites(uint32_t (&v)[NLV], uint32_t a1, uint32_t a2,
                                              uint32_t a3, uint32_t a4, uint32_t b1, uint32_t b2,
                                              uint32_t b3, uint32_t b4) {
    uint32_t k1a, k1b, k2a, k2b, k2c, k3a, k3b;
    CSG_FA(v[0], k1a, v[0], a1, a2);
    CSG_FA(v[0], k1b, v[0], b1, b2);
    CSG_FA(v[1], k2a, v[1], a3, a4);
    CSG_FA(v[1], k2b, v[1], b3, b4);
    CSG_FA(v[1], k2c, v[1], k1a, k1b);
    CSG_FA(v[2], k3a, v[2], k2a, k2b);
    k3b = v[2] & k2c;
    v[2] ^= k2c;
    if constexpr (NLV > 3) {
        uint32_t k4;
        CSG_FA(v[3], k4, v[3], k3a, k3b);
#pragma unroll
        for (int l = 4; l < NLV; ++l) {
            const uint32_t t = v[l] & k4;
            v[l] ^= k4;
            k4 = t;
        }
    }
}

// Bit-sliced count of a plane's post-flip unsatisfied bonds, sites taken in
// pairs (even, odd).  A site's adder words sa, sb (weight 1) and ca, cb (weight
// 2) flip with it: with f the flip mask the count is that of sa ^ f, ... .  In a
// full adder of v, a ^ f, b ^ f the flip cancels from the sum, v ^ a ^ b, and
// the carry is v where a and b differ (the sum is not v), else a ^ f: 13
// instructions a site word instead of 14 with the flip applied first (L = 48
// counting launch: 115 -> 112 us).
template <int NLV>
struct BondCounts {
    uint32_t v[NLV];
    uint32_t k1, k2;  // carries of the even site, weight 2 and 4
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int l = 0; l < NLV; ++l) v[l] = 0;
        k1 = k2 = 0;
    }
    static __device__ __forceinline__ uint32_t add_flipped(uint32_t& v, uint32_t a, uint32_t b, uint32_t f) {
        const uint32_t s = xor3(v, a, b), c = lop3<0x8E>(s, v, a ^ f);
        v = s;
        return c;
    }
    __device__ __forceinline__ void add_even(uint32_t sa, uint32_t sb, uint32_t ca, uint32_t cb, uint32_t f) {
        k1 = add_flipped(v[0], sa, sb, f);
        k2 = add_flipped(v[1], ca, cb, f);
    }
    __device__ __forceinline__ void add_odd(uint32_t sa, uint32_t sb, uint32_t ca, uint32_t cb, uint32_t f) {
        const uint32_t j1 = add_flipped(v[0], sa, sb, f), j2 = add_flipped(v[1], ca, cb, f);
        uint32_t k2c, k3a, k3b;
        CSG_FA(v[1], k2c, v[1], k1, j1);
        CSG_FA(v[2], k3a, v[2], k2, j2);
        k3b = v[2] & k2c;
        v[2] ^= k2c;
        if constexpr (NLV > 3) {
            uint32_t k4;
            CSG_FA(v[3], k4, v[3], k3a, k3b);
#pragma unroll
            for (int l = 4; l < NLV; ++l) {
                const uint32_t t = v[l] & k4;
                v[l] ^= k4;
                k4 = t;
            }
        }
    }
    // the last even site of an odd number
    __device__ __forceinline__ void finish_even() {
        const uint32_t k2b = v[1] & k1;
        v[1] ^= k1;
        if constexpr (NLV > 2) {
            uint32_t k3;
            CSG_FA(v[2], k3, v[2], k2, k2b);
#pragma unroll
            for (int l = 3; l < NLV; ++l) {
                const uint32_t t = v[l] & k3;
                v[l] ^= k3;
                k3 = t;
            }
        }
    }
};

// Four single-weight words at once: value += x1 + x2 + x3 + x4.
template <int NLV>
__device__ __forceinline__ void vc_add4(uint32_t (&v)[NLV], uint32_t x1, uint32_t x2, uint32_t x3,
                                        uint32_t x4) {
    uint32_t k1a, k1b, k2;
    CSG_FA(v[0], k1a, v[0], x1, x2);
    CSG_FA(v[0], k1b, v[0], x3, x4);
    CSG_FA(v[1], k2, v[1], k1a, k1b);
#pragma unroll
    for (int l = 2; l < NLV; ++l) {
        const uint32_t t = v[l] & k2;
        v[l] ^= k2;
        k2 = t;
    }
}

// Column popcount of a 32x32 bit matrix held one row per lane: returns, in
// lane j, the number of lanes whose bit j is set.  Five butterfly stages of a
// bit transpose (shuffle, funnel rotate, bit select), then popc.
__device__ __forceinline__ int column_popc(uint32_t v, int lane) {
#pragma unroll
    for (int d = 16; d >= 1; d >>= 1) {
        const uint32_t m = d == 16 ? 0x0000FFFFu
                         : d == 8  ? 0x00FF00FFu
                         : d == 4  ? 0x0F0F0F0Fu
                         : d == 2  ? 0x33333333u
                                   : 0x55555555u;
        const bool upper = (lane & d) != 0;
        const uint32_t t = __shfl_xor_sync(0xFFFFFFFFu, v, d);
        const uint32_t rot = __funnelshift_r(t, t, upper ? d : 32 - d);
        const uint32_t keep = upper ? ~m : m;
        v = (v & keep) | (rot & ~keep);
    }
    return __popc(v);
}

template <int NLV>
__device__ __forceinline__ int column_count(const uint32_t (&v)[NLV], int lane) {
    int s = 0;
#pragma unroll
    for (int l = 0; l < NLV; ++l) s += column_popc(v[l], lane) << l;
    return s;
}

// Column sums of the 4 planes of a warp whose 32 lanes all hold counters of
// one quad: two rounds of lane exchange (lanes i, i^16, then i, i^8) leave
// each lane with one plane, k = lane >> 3, summed over 4 lanes (two more
// counter levels); one 32x32 transpose per level then gives every lane j the
// bits of sample j of all lanes, plane k in bits 8k..8k+7.  Returns, in lane
// j, the totals of sample j for planes 0..3.
template <int NLV>
__device__ __forceinline__ void packed_column_counts(const uint32_t (&v)[4][NLV], int lane,
                                                     int (&cnt)[4]) {
    const bool hi16 = (lane & 16) != 0, hi8 = (lane & 8) != 0;
    uint32_t a[2][NLV + 1];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        uint32_t cy = 0;
#pragma unroll
        for (int l = 0; l < NLV; ++l) {
            const uint32_t mine = hi16 ? v[k + 2][l] : v[k][l];
            const uint32_t other = __shfl_xor_sync(0xFFFFFFFFu, hi16 ? v[k][l] : v[k + 2][l], 16);
            a[k][l] = mine ^ other ^ cy;
            cy = maj3(mine, other, cy);
        }
        a[k][NLV] = cy;
    }
    uint32_t b[NLV + 2];
    uint32_t cy = 0;
#pragma unroll
    for (int l = 0; l <= NLV; ++l) {
        const uint32_t mine = hi8 ? a[1][l] : a[0][l];
        const uint32_t other = __shfl_xor_sync(0xFFFFFFFFu, hi8 ? a[0][l] : a[1][l], 8);
        b[l] = mine ^ other ^ cy;
        cy = maj3(mine, other, cy);
    }
    b[NLV + 1] = cy;
#pragma unroll
    for (int k = 0; k < 4; ++k) cnt[k] = 0;
#pragma unroll
    for (int l = 0; l < NLV + 2; ++l) {
        uint32_t x = b[l];
#pragma unroll
        for (int d = 16; d >= 1; d >>= 1) {  // 32x32 bit transpose (as in column_popc)
            const uint32_t m = d == 16 ? 0x0000FFFFu
                             : d == 8  ? 0x00FF00FFu
                             : d == 4  ? 0x0F0F0F0Fu
                             : d == 2  ? 0x33333333u
                                       : 0x55555555u;
            const bool upper = (lane & d) != 0;
            const uint32_t t = __shfl_xor_sync(0xFFFFFFFFu, x, d);
            const uint32_t rot = __funnelshift_r(t, t, upper ? d : 32 - d);
            const uint32_t keep = upper ? ~m : m;
            x = (x & keep) | (rot & ~keep);
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) cnt[k] += __popc((x >> (8 * k)) & 0xFFu) << l;
    }
}

// All ones where r < t, else zero: the borrow of r - t.  The subtraction runs
// on the logic/add pipe and the borrow's spread on the multiply pipe; a
// compare and a select (of any value) are two instructions of the former.
// (A mask from one 64-bit multiply-add, r * 1 + (2^64 - t), leaves the logic
// pipe out altogether, but its 64-bit addends cost dispatch slots and
// registers: 5 to 9 % slower in the resident kernel at L = 12..20.)
__device__ __forceinline__ uint32_t below(uint32_t r, uint32_t t) {
    uint32_t m;
    asm("{\n .reg .u32 d;\n sub.cc.u32 d, %1, %2;\n subc.u32 %0, 0, 0;\n}" : "=r"(m) : "r"(r), "r"(t));
    return m;
}

// Flip at H = 0: U >= 3 always accepted; U = 2, 1, 0 accepted when the draw is
// below t2, t1, t0 (t0 <= t1 <= t2).  With j the number of those thresholds
// above the draw, a flip is accepted iff U + j >= 3; from the two full adders
// (U = sa + sb + 2(ca + cb)) and the three masks that takes four gates and
// the OR of the two terms, which the caller's own gate absorbs.  (Found by an
// exhaustive search over gate pairs; three compares, five gates and three
// selects did the same in eleven.)
struct FlipTerms {
    uint32_t x, y;  // flip = x | y
};
__device__ __forceinline__ FlipTerms flip_h0_terms(uint32_t sa, uint32_t ca, uint32_t sb, uint32_t cb,
                                                   uint32_t r, uint32_t t0, uint32_t t1, uint32_t t2) {
    const uint32_t m0 = below(r, t0), m1 = below(r, t1), m2 = below(r, t2);
    const uint32_t g = lop3<0x61>(ca, cb, m0);
    const uint32_t h = lop3<0x7E>(sa, m2, g);
    return FlipTerms{lop3<0xE2>(ca, g, h), lop3<0xD4>(sb, m1, h)};
}
// the flip as one word (no kernel takes it: they use flipped below)
__device__ __forceinline__ uint32_t flip_h0(uint32_t sa, uint32_t ca, uint32_t sb, uint32_t cb,
                                            uint32_t r, uint32_t t0, uint32_t t1, uint32_t t2) {
    const FlipTerms f = flip_h0_terms(sa, ca, sb, cb, r, t0, t1, t2);
    return f.x | f.y;
}
// s ^ (x | y): the flipped spin word in one gate
__device__ __forceinline__ uint32_t flipped(uint32_t s, const FlipTerms& f) { return lop3<0x1E>(s, f.x, f.y); }

// A moderate field, 0 < H < 2: always accepted from U = 3 (spin down, s = 0) or
// U = 4 (spin up).  With j thresholds of the spin's own above the draw (three
// or four), j one more for spins down, a flip is accepted iff U + j >= 4.  The
// masks A >= B >= C >= D of j >= 1..4 are selected by the spin; while D is not
// set, j is A ^ B ^ C + 2B.  Thresholds as flip_gen takes them.  31 logic
// instructions a word with the adders and Philox, where flip_gen takes 52.
__device__ __forceinline__ FlipTerms flip_field_terms(uint32_t s0, uint32_t sa, uint32_t ca, uint32_t sb,
                                                      uint32_t cb, uint32_t r, const uint4 ta, const uint4 tb) {
    const uint32_t A = lop3<0xCF>(s0, below(r, tb.z), 0u);            // ~s0 | m
    const uint32_t B = lop3<0xCA>(s0, below(r, tb.y), below(r, ta.z));  // s0 ? up : down
    const uint32_t C = lop3<0xCA>(s0, below(r, tb.x), below(r, ta.y));
    const uint32_t D = lop3<0xCA>(s0, below(r, ta.w), below(r, ta.x));
    const uint32_t c = maj3(sa, sb, xor3(A, B, C));
    const uint32_t o = lop3<0xFE>(ca, cb, B);  // any of the weight-2 terms
    return FlipTerms{lop3<0xF8>(maj3(ca, cb, B), c, o), D};  // two of them, or one and the carry
}

// General field, 0 <= H <= 4.  A flip of centre spin s with U unsatisfied
// bonds is accepted iff U >= ucut_s (dE <= 0) or the draw r < thr[s][U].
// thr[s][U] does not decrease with U and is 0xFFFFFFFF from ucut_s on, and
// ucut_0 <= 3, ucut_1 <= 5, so walking U down from there the accepted set is
// {U >= the smallest U with r < thr[s][U]} - a select chain like the H = 0
// rule.  Only the draw r = 0xFFFFFFFF, below none of the thresholds, needs the
// cut itself.  ta = {thr0[0], thr0[1], thr0[2], thr1[0]},
// tb = {thr1[1], thr1[2], thr1[3], thr1[4]}.
__device__ __forceinline__ uint32_t flip_gen(uint32_t s0, uint32_t sa, uint32_t ca, uint32_t sb,
                                             uint32_t cb, uint32_t r, const uint4 ta, const uint4 tb,
                                             int uc0, int uc1) {
    // U = sa + sb + 2(ca + cb): U >= 4 needs both carries, or one carry and
    // both sum bits; U >= 5 and U >= 6 need both carries.
    const uint32_t v = sa | sb, cx = ca | cb, cc = ca & cb;
    const uint32_t ge1 = cx | v, ge2 = cx | (sa & sb), ge3 = maj3(ca, cb, v);
    const uint32_t ge4 = cc | (cx & sa & sb), ge5 = cc & v;
    uint32_t g0 = ge3;
    g0 = (r < ta.z) ? ge2 : g0;
    g0 = (r < ta.y) ? ge1 : g0;
    g0 = (r < ta.x) ? 0xFFFFFFFFu : g0;
    uint32_t g1 = ge5;
    g1 = (r < tb.w) ? ge4 : g1;
    g1 = (r < tb.z) ? ge3 : g1;
    g1 = (r < tb.y) ? ge2 : g1;
    g1 = (r < tb.x) ? ge1 : g1;
    g1 = (r < ta.w) ? 0xFFFFFFFFu : g1;
    if (r == 0xFFFFFFFFu) {  // accepted: exactly U >= ucut
        const uint32_t ge[8] = {0xFFFFFFFFu, ge1, ge2, ge3, ge4, ge5, cc & sa & sb, 0u};
        g0 = ge[uc0 & 7];
        g1 = ge[uc1 & 7];
    }
    return (s0 & g1) | (~s0 & g0);
}

// The thresholds of plane t in the layout flip_gen takes.
__host__ __device__ inline void gen_thresholds(const PtTables& tab, int t, uint4& ta, uint4& tb) {
    ta = make_uint4(tab.thr[t][0][0], tab.thr[t][0][1], tab.thr[t][0][2], tab.thr[t][1][0]);
    tb = make_uint4(tab.thr[t][1][1], tab.thr[t][1][2], tab.thr[t][1][3], tab.thr[t][1][4]);
}

// Shared-memory layout of one CTA (dynamic):
//   uint32 planes[Qc][4][N] (the 4 temperature planes of each quad as separate
//   arrays, so that every access of one plane by a warp is conflict-free);
//   int sE[Qc*4][32]; int sD[Qc*4][32];
//   int sM[Qc*4][32]                      (only with magnetisations)
//   uint4 sThr[Qc*4][2]; uint8 sUcut[Qc*4][2]   (only for H != 0)
// The exchange masks of a round live in the first 2*Qc words of sD, which is
// cleared again before the overlap counts are added.  At L=16 with 3 quads the
// H=0 layout is 195 KB, under the 196 KB carve-out, so the 48 KB of bonds of
// the word stay in L1.
template <int L>
struct SmemMap {
    static __host__ __device__ size_t bytes(int Qc, bool has_m, bool gen) {
        return (size_t)Qc * L * L * L * 16 + (size_t)Qc * 4 * 32 * 4 * (has_m ? 3 : 2) +
               (gen ? (size_t)Qc * 4 * 32 + (size_t)Qc * 4 * 2 : 0);
    }
};

using ResidentFn = void (*)(PtParams);

// The resident kernel for lattice side L (each defined in its own translation
// unit, pt_instances.cu built with CSG_PT_L = L): for a FieldMode, with nseg
// column segments per thread; nullptr if not built.
#define CSG_DECLARE_RESIDENT(LL) ResidentFn resident_kernel_L##LL(int field, int nseg);
CSG_DECLARE_RESIDENT(4)
CSG_DECLARE_RESIDENT(6)
CSG_DECLARE_RESIDENT(8)
CSG_DECLARE_RESIDENT(10)
CSG_DECLARE_RESIDENT(12)
CSG_DECLARE_RESIDENT(14)
CSG_DECLARE_RESIDENT(16)
CSG_DECLARE_RESIDENT(18)
CSG_DECLARE_RESIDENT(20)
CSG_DECLARE_RESIDENT(22)
CSG_DECLARE_RESIDENT(24)
#undef CSG_DECLARE_RESIDENT

}  // namespace csg
