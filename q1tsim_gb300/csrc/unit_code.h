// Units of a matrix of 0, +-1 and +-i entries (gate_kernels.cu, gate_run.cu):
// such gates move and re-sign amplitudes without arithmetic.
#pragma once

namespace q1g {

// Unit code of (re, im): 0 -> 1, 1 -> i, 2 -> -1, 3 -> -i; -1 for 0, -2
// otherwise.
inline int unit_code(double re, double im)
{
    if (re == 0.0 && im == 0.0) return -1;
    if (re == 1.0 && im == 0.0) return 0;
    if (re == 0.0 && im == 1.0) return 1;
    if (re == -1.0 && im == 0.0) return 2;
    if (re == 0.0 && im == -1.0) return 3;
    return -2;
}

// A 2x2 matrix with one unit entry per row and column: (swap, u0, u1).
inline bool mono_pair(const double* m, int& swap, int& u0, int& u1)
{
    const int c00 = unit_code(m[0], m[1]), c01 = unit_code(m[2], m[3]);
    const int c10 = unit_code(m[4], m[5]), c11 = unit_code(m[6], m[7]);
    if (c00 >= 0 && c11 >= 0 && c01 == -1 && c10 == -1) {
        swap = 0, u0 = c00, u1 = c11;
        return true;
    }
    if (c01 >= 0 && c10 >= 0 && c00 == -1 && c11 == -1) {
        swap = 1, u0 = c01, u1 = c10;
        return true;
    }
    return false;
}

}  // namespace q1g
