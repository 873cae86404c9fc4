// Whether a case takes the straight-line quotients (csrc/exact_case.h), for a
// unit case whose one varied cell or constant is given: one line each, in the
// order of test_exact_case.py.
#include <cmath>
#include <cstdio>
#include <limits>

#include "exact_case.h"

using namespace gd2d;

static double bits(uint64_t b) {
    double x;
    memcpy(&x, &b, sizeof x);
    return x;
}

static void cell(double area, double hx) {
    DevCase d = {};
    d.face.gm1 = 0.4;
    d.R = 287.0;
    d.gamma = 1.4;
    const double A[3] = {1.0, area, 0.5}, H[3] = {1.0, 0.5, hx};
    printf("%d\n", (int)exact_rows_case(d, 3, A, H));
}

int main() {
    const double low = bits(0x3ff00000ffffffffull), low2 = bits(0x3fe12345ffffffffull);  // the low 32 bits set
    const double ones = bits(0x3fffffffffffffffull), ones2 = bits(0x3f2fffffffffffffull);
    const double nearly = bits(0x3ffffffffffffffeull);
    cell(1.0, 1.0);
    cell(low, 1.0);
    cell(1.0, low2);
    cell(nearly, nearly);
    cell(ones, 1.0);
    cell(1.0, ones2);
    cell(1e-21, 1.0);
    cell(1.0, 1e21);
    cell(1.0, std::numeric_limits<double>::quiet_NaN());
    cell(std::numeric_limits<double>::infinity(), 1.0);
    return 0;
}
