// Tile shapes of the matrix-free operator's kernels and the lanes of their epilogue (apply_gemm.cu).
#pragma once

#include <algorithm>

namespace tcu {

struct GemmShape {
    int DI, TR, TC, RG, CG, KJ;
};

// The product restricted to the first nsrc source lm and the first ndst destination lm (the
// table then needs degrees p <= order = l_max(src) + l_max(dst)); input vectors hold ldin and
// output vectors ldout complex entries per sphere. The full operator: nsrc = ndst = nlm.
struct SubOp {
    int nsrc, ndst, order, ldin, ldout;
};

// Tile shapes per lmax: G rows DI * tsize <= TR * RG, columns 2 nlm <= TC * CG
inline GemmShape gemm_shape(int L) {
    switch (L) {
        case 2: return {4, 4, 2, 25, 8, 32};   // 100 x 16, 200 threads
        case 3: return {2, 4, 3, 25, 10, 32};  // 98 x 30, 250 threads
        case 4: return {1, 4, 4, 21, 12, 32};  // 81 x 48, 252 threads
        default: return {1, 4, 5, 31, 14, 16}; // lmax 5: 121 x 70, 434 threads
    }
}

// The dipole-source (and dipole-to-dipole) products: G is (DI (order+1)^2) x 6, about 200 rows
inline GemmShape sub_shape(int tsz) {
    const int DI = std::max(1, 200 / tsz);
    return {DI, 4, 2, (DI * tsz + 3) / 4, 3, 16};
}

// threads of a CTA: those of the tile, in whole warps (the term lists' sums cross lanes)
inline int shape_threads(const GemmShape& s) { return (s.RG * s.CG + 31) / 32 * 32; }

// lanes per task of the term lists: what nthr threads allow, at most 16. With nthr a multiple of 32 the tasks x
// lanes, rounded up to whole warps, are one pass over the threads whenever a task has more than one lane, so
// every lane of a warp takes part in the shuffles.
constexpr int epilogue_lanes(int tasks, int nthr, int nsrc) {
    int w = 1;
    while (w < 16 && 2 * w * tasks <= nthr && 2 * w <= nsrc) w *= 2;
    return w;
}

}  // namespace tcu
