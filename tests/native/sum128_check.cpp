// Host-side check of Sum128::magnitude (imc_math64.cuh): sums of many addends
// at the ends of the 2^94 units that a tally's accumulators take in one flush.
// Prints one line per property; driven by tests/test_sum128.py.
#define IMC_HD inline
#include "../../mixedprecisionimc.jl_gb300/csrc/imc_math64.cuh"

#include <cstdio>

using namespace imc::m64;

static Sum128 times(double v, int n) {
    Sum128 s;
    s.clear();
    for (int i = 0; i < n; ++i)
        if (!s.add(v, 0)) s.hi = -1;
    return s;
}

int main() {
    uint64_t l, h;
    bool neg;
    // 2^93 twice is the first sum out of range, on either side of zero, and
    // stays out at 2^96 and beyond (where a 32-bit top word would wrap)
    bool refused = true, kept = true;
    for (int n = 2; n <= 1024; ++n)
        refused = refused && !times(0x1p93, n).magnitude(neg, l, h) && !times(-0x1p93, n).magnitude(neg, l, h);
    kept = kept && times(0x1p93, 1).magnitude(neg, l, h) && !neg && l == 0 && h == 1ull << 29;
    kept = kept && times(-0x1p93, 1).magnitude(neg, l, h) && neg && l == 0 && h == 1ull << 29;
    kept = kept && times(-3.0, 5).magnitude(neg, l, h) && neg && l == 15 && h == 0;
    // 2^94 - 1: three sums that meet below it
    Sum128 s = times(0x1p93, 1);
    s.add128(~0ull, (1ull << 29) - 1, false);
    kept = kept && s.magnitude(neg, l, h) && !neg && l == ~0ull && h == (1ull << 30) - 1;
    s.add128(1, 0, false);
    refused = refused && !s.magnitude(neg, l, h);
    // a sum that leaves the range and comes back
    s.clear();
    for (int i = 0; i < 64; ++i) s.add(0x1p93, 0);
    for (int i = 0; i < 64; ++i) s.add(-0x1p93, 0);
    s.add(7.0, 0);
    kept = kept && s.magnitude(neg, l, h) && !neg && l == 7 && h == 0;
    printf("refused %d\nkept %d\n", refused, kept);
    return 0;
}
