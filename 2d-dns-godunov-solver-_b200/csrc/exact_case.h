// Whether the straight-line quotients of face_exact.cuh round correctly for a
// case, by its constants and its cells (host).
#pragma once

#include <cstdint>
#include <cstring>

#include "gd2d_internal.h"

namespace gd2d {

// A divisor of the method's range: its exception is a significand of ones
// alone, all 52 bits of them.  (The kernels, which test a row of computed
// divisors at a time, look at the low 32 only: a face in 4e9.  Here that
// would turn the whole case over to the plain formulas, one mesh of 2.09M
// cells in a thousand.)
inline bool exact_divisor(double x) {
    uint64_t b;
    std::memcpy(&b, &x, sizeof b);
    const uint64_t significand = (uint64_t(1) << 52) - 1;
    return x >= 1e-20 && x <= 1e20 && (b & significand) != significand;  // false for NaN
}

// Any case in physical units is in range; one that is not has its cells
// evaluated by the plain formulas.
inline bool exact_rows_case(const DevCase &d, int64_t n_cells, const double *areas, const double *HX) {
    auto in = [](double x, double lo, double hi) { return x >= lo && x <= hi; };  // false for NaN
    if (!exact_divisor(d.face.gm1) || !exact_divisor(d.R) || !in(d.gamma, 1.01, 100.0)) return false;
    if (d.visc_model == VISC_SUTHERLAND && !exact_divisor(d.suth_ref)) return false;
    if (!in(d.venkat_K, 0.0, 1e6) || !in(d.ksi, 0.0, 1e20)) return false;
    for (int64_t i = 0; i < n_cells; ++i)
        if (!exact_divisor(areas[i]) || !exact_divisor(HX[i])) return false;
    return true;
}

}  // namespace gd2d
