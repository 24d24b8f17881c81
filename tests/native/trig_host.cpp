// Host build of the fixed-point sine and cosine, for the CPU self-test (tests/test_trig.py).
#include <stdint.h>

#include "nd_trig.cuh"

extern "C" void nd_trig_host(const double* x, double* s, double* c, int64_t n) {
    for (int64_t i = 0; i < n; ++i) {
        s[i] = nd::trig::sin(x[i]);
        c[i] = nd::trig::cos(x[i]);
    }
}
