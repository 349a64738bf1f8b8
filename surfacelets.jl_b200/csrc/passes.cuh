// Line geometry shared by the line passes (regpass.cuh, mixpass.cuh).
#pragma once

#include "fft_core.cuh"
#include "plan.h"
#include "prof.h"

namespace sfl {

// Lines of a column-major 3-D array of dims d along axis a (0-based).
inline Lines axis_lines(const int d[3], int a) {
    long long s[3] = {1, d[0], (long long)d[0] * d[1]};
    int o0 = a == 0 ? 1 : 0;
    int o1 = a == 2 ? 1 : 2;
    Lines g;
    g.nlines = d[o0] * d[o1];
    g.B0 = d[o0];
    g.B1 = d[o1];
    g.s0 = s[o0];
    g.s1 = s[o1];
    g.s2 = 0;
    g.si = s[a];
    g.fast_div();
    return g;
}

}  // namespace sfl
