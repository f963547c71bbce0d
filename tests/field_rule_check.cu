// Checks the flip terms the kernels use (pt_kernel.cuh: flip_h0_terms at H = 0,
// flip_field_terms for a field below 2, and the flipped spin word from them)
// against the acceptance rule, bit for bit: a flip of centre spin s with U
// unsatisfied bonds is accepted iff U >= 3 (at H = 0 and for spins down) or 4
// (spins up in a field), or r < thr[s][U].  Every combination of (s, sa, ca, sb,
// cb) sits in one bit of the words; every draw at an edge (0, each threshold and
// its neighbours, 0xFFFFFFFF) is taken with every table.  Also the counters'
// adders that take the flip inside (BondCounts) against a plain sum.
// Built and run by tests/test_field_rule.py; prints the numbers of mismatches.
#include <cstdint>
#include <cstdio>
#include <vector>

#include "pt_kernel.cuh"

struct Case {
    uint32_t r;
    uint32_t thr[2][4];  // [spin][U], U below the spin's cut
    int field;
};

__global__ void check_kernel(const Case* cases, int n, unsigned* bad) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const Case cs = cases[i];
    // bit b: s0 = b>>4, sa = b&1, ca = (b>>1)&1, sb = (b>>2)&1, cb = (b>>3)&1
    uint32_t s0 = 0, sa = 0, ca = 0, sb = 0, cb = 0, want = 0;
    for (int b = 0; b < 32; ++b) {
        sa |= ((b >> 0) & 1u) << b;
        ca |= ((b >> 1) & 1u) << b;
        sb |= ((b >> 2) & 1u) << b;
        cb |= ((b >> 3) & 1u) << b;
        s0 |= ((b >> 4) & 1u) << b;
        const int s = (b >> 4) & 1;
        const int U = (b & 1) + ((b >> 2) & 1) + 2 * (((b >> 1) & 1) + ((b >> 3) & 1));
        const bool acc = U >= (cs.field ? 3 + s : 3) || cs.r < cs.thr[s][U];
        want |= (acc ? 1u : 0u) << b;
    }
    csg::FlipTerms f;
    if (cs.field)  // the layout of gen_thresholds
        f = csg::flip_field_terms(s0, sa, ca, sb, cb, cs.r,
                                  make_uint4(cs.thr[0][0], cs.thr[0][1], cs.thr[0][2], cs.thr[1][0]),
                                  make_uint4(cs.thr[1][1], cs.thr[1][2], cs.thr[1][3], 0xFFFFFFFFu));
    else
        f = csg::flip_h0_terms(sa, ca, sb, cb, cs.r, cs.thr[0][0], cs.thr[0][1], cs.thr[0][2]);
    if ((f.x | f.y) != want) atomicAdd(bad + cs.field, 1u);
    if (csg::flipped(s0, f) != (s0 ^ want)) atomicAdd(bad + 2, 1u);

    // counters: this word as every one of seven sites, then one more with the
    // flips the other way round
    constexpr int NLV = csg::bit_length(6 * 8);
    csg::BondCounts<NLV> c;
    c.clear();
    for (int k = 0; k < 8; ++k) {
        const uint32_t fl = k == 7 ? ~want : want;
        if (k & 1)
            c.add_odd(sa, sb, ca, cb, fl);
        else
            c.add_even(sa, sb, ca, cb, fl);
    }
    csg::BondCounts<NLV> odd;  // an odd number of sites
    odd.clear();
    odd.add_even(sa, sb, ca, cb, want);
    odd.finish_even();
    bool ok = true;
    for (int b = 0; b < 32; ++b) {
        const int U = (b & 1) + ((b >> 2) & 1) + 2 * (((b >> 1) & 1) + ((b >> 3) & 1));
        const int after = (want >> b) & 1 ? 6 - U : U;  // unsatisfied after the flip
        int got = 0, got1 = 0;
        for (int l = 0; l < NLV; ++l) {
            got += (int)((c.v[l] >> b) & 1u) << l;
            got1 += (int)((odd.v[l] >> b) & 1u) << l;
        }
        ok = ok && got == 7 * after + (6 - after) && got1 == after;
    }
    if (!ok) atomicAdd(bad + 3, 1u);
}

int main() {
    uint64_t z = 0x9E3779B97F4A7C15ull;
    auto rnd = [&]() {
        z += 0x9E3779B97F4A7C15ull;
        uint64_t x = z;
        x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
        x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
        return (uint32_t)(x ^ (x >> 31));
    };
    std::vector<Case> cases;
    for (int k = 0; k < 2000; ++k) {
        Case c{};
        c.field = k & 1;
        // non-decreasing in U, as the tables are; equal, zero and largest ones among
        // them (a spin down has its own thresholds up to U = 2, a spin up to U = 3)
        for (int s = 0; s < 2; ++s) {
            uint32_t prev = k % 5 == 0 ? 0u : rnd() >> (rnd() % 32);
            for (int U = 0; U < 4; ++U) {
                const uint32_t step = k % 7 == 0 ? 0u : rnd() >> (rnd() % 32);
                prev = prev + step < prev ? 0xFFFFFFFFu : prev + step;
                c.thr[s][U] = prev;
            }
        }
        if (!c.field)
            for (int U = 0; U < 4; ++U) c.thr[1][U] = c.thr[0][U];
        std::vector<uint32_t> draws = {0u, 1u, 0xFFFFFFFEu, 0xFFFFFFFFu, rnd(), rnd()};
        for (int s = 0; s < 2; ++s)
            for (int U = 0; U < 4; ++U)
                for (int d = -1; d <= 1; ++d) draws.push_back(c.thr[s][U] + (uint32_t)d);
        for (uint32_t r : draws) {
            c.r = r;
            cases.push_back(c);
        }
    }
    Case* d = nullptr;
    unsigned* bad = nullptr;
    unsigned h[4] = {0, 0, 0, 0};
    if (cudaMalloc(&d, cases.size() * sizeof(Case)) != cudaSuccess) return 2;
    if (cudaMalloc(&bad, sizeof(h)) != cudaSuccess) return 2;
    cudaMemset(bad, 0, sizeof(h));
    cudaMemcpy(d, cases.data(), cases.size() * sizeof(Case), cudaMemcpyHostToDevice);
    const int n = (int)cases.size();
    check_kernel<<<(n + 127) / 128, 128>>>(d, n, bad);
    if (cudaMemcpy(h, bad, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 3;
    std::printf("cases %d zero-field %u field %u flipped %u counters %u\n", n, h[0], h[1], h[2], h[3]);
    cudaFree(d);
    cudaFree(bad);
    return 0;
}
