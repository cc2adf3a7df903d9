// spec_lut.h -- search tables of the sampled spectra and the observer (host and device).
//
// upper_bound over an ascending table is a chain of up to nine dependent loads in the shading kernels.
// A search table holds, for each of kLutCells equal cells of the table's range, a bracket of the answer
// (low | high << 16), usually one or two entries wide, which the search then starts from: the same
// index, whatever the spacing. The brackets are those of the cell widened by a hundredth of it on both
// sides, far more than the rounding of the cell's number, and the first and last cell are open.
#pragma once
#include <stdint.h>

#include <algorithm>
#include <cmath>
#include <vector>

#ifdef __CUDACC__
#define LUT_HD __host__ __device__ __forceinline__
#else
#define LUT_HD inline
#endif

namespace liar_gpu {

constexpr int kLutCells = 256;

// cells of width 1 / scale from x0; scale 0: no table (too long, not ascending or not finite)
struct SearchLut {
    float x0, scale;
    int32_t at;  // first of its kLutCells words
};

// the first index in [lo, hi) with a[index] > x, hi for none
LUT_HD int upper_bound_in(const float* a, int lo, int hi, float x) {
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (a[mid] > x) hi = mid; else lo = mid + 1;
    }
    return lo;
}

LUT_HD int lut_upper_bound(const uint32_t* luts, SearchLut t, const float* a, int n, float x) {
    if (t.scale == 0.0f) return upper_bound_in(a, 0, n, x);
    const float c = (x - t.x0) * t.scale;
    int cell = kLutCells - 1;  // (also NaN's)
    if (c < (float)(kLutCells - 1)) cell = c > 0.0f ? (int)c : 0;
    const uint32_t b = luts[t.at + cell];
    return upper_bound_in(a, (int)(b & 0xffffu), (int)(b >> 16), x);
}

// appends the search table of a[0 .. n) to luts
inline SearchLut add_lut(std::vector<uint32_t>& luts, const float* a, size_t n) {
    SearchLut t{0.0f, 0.0f, 0};
    if (n < 2 || n > 0xffff) return t;
    for (size_t k = 0; k + 1 < n; ++k)
        if (!(a[k] <= a[k + 1])) return t;
    const float scale = (float)kLutCells / (a[n - 1] - a[0]);
    if (!std::isfinite(a[0]) || !std::isfinite(scale) || !(scale > 0.0f)) return t;
    t.x0 = a[0];
    t.scale = scale;
    t.at = (int32_t)luts.size();
    const auto upper = [&](double x) {
        return (uint32_t)(std::upper_bound(a, a + n, x, [](double v, float e) { return v < (double)e; }) - a);
    };
    for (int c = 0; c < kLutCells; ++c) {
        const uint32_t lo = c == 0 ? 0u : upper((double)a[0] + (c - 0.01) / (double)scale);
        const uint32_t hi = c == kLutCells - 1 ? (uint32_t)n : upper((double)a[0] + (c + 1.01) / (double)scale);
        luts.push_back(lo | (hi << 16));
    }
    return t;
}

}  // namespace liar_gpu
