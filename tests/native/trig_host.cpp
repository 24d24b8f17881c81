// Host build of the fixed-point sine and cosine and of the integer division, for the CPU
// self-tests (tests/test_trig.py).
#include <stdint.h>

#include "nd_trig.cuh"

extern "C" void nd_trig_host(const double* x, double* s, double* c, int64_t n) {
    for (int64_t i = 0; i < n; ++i) {
        s[i] = nd::trig::sin(x[i]);
        c[i] = nd::trig::cos(x[i]);
    }
}

extern "C" void nd_trig_times_host(const double* f, const double* x, double* s, double* c, int64_t n) {
    for (int64_t i = 0; i < n; ++i) {
        s[i] = nd::trig::times_sin(f[i], x[i]);
        c[i] = nd::trig::times_cos(f[i], x[i]);
    }
}

extern "C" void nd_exact_div_host(const double* a, const double* b, double* out, int64_t n) {
    for (int64_t i = 0; i < n; ++i) out[i] = nd::exact::div_rn(a[i], b[i]);
}
