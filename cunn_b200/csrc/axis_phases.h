// Residues of a strided input gradient along one axis.
#pragma once

#include <algorithm>
#include <vector>

namespace cunn {
namespace mm {

// One residue of an axis of an input gradient: input positions h0 + i * d (i < n) are reached by taps k0 + t * kstep
// (t < taps) at output positions o0 + i - t * ostep.
struct AxisPhase {
    int h0, n, k0, taps, kstep, o0, ostep;
};

// Residues without taps are listed if `all`; *gaps is set when there are any.
inline std::vector<AxisPhase> axis_phases(int H, int k, int d, int pad, int dil, bool all, bool *gaps)
{
    int g = d, r = dil % d;
    while (r) { const int t = g % r; g = r; r = t; }                       // gcd(d, dil)
    std::vector<AxisPhase> out;
    for (int h0 = 0; h0 < std::min(d, H); ++h0) {
        // the first of its taps is below d / g, the others follow d / g apart
        const int step = d / g;
        int first = dil == 1 ? (h0 + pad) % d : 0;
        while (first < step && first < k && (h0 + pad - first * dil) % d) ++first;
        AxisPhase a{h0, (H - h0 + d - 1) / d, 0, 0, step, 0, dil / g};
        if (first < step && first < k) {
            a.k0 = first;
            a.taps = (k - first - 1) / step + 1;
            a.o0 = (h0 + pad - first * dil) / d;
        }
        if (a.taps || all) out.push_back(a);
        if (!a.taps) *gaps = true;
    }
    return out;
}

}  // namespace mm
}  // namespace cunn
