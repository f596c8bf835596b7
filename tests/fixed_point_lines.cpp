// The arithmetic of the fixed-point lines (wv_fx.cuh) on the host, as C functions for
// tests/test_fixed_point_lines_cpu.py.  Test infrastructure.
#include "wv_fx.cuh"

#include <cstddef>

using namespace wvgpu::dev;

extern "C" {

// out[i] = the product x[i] as the r2c takes it in
void shift_products(const long long* x, size_t n, int sh, long long* out) {
    for (size_t i = 0; i < n; ++i) out[i] = fx_shift_round(x[i], sh, static_cast<int>(i & 1));
}

// out[i] = (x[i] + fx_half(sh, i & 1)) >> sh: a product aligned to a larger unit
void align_products(const long long* x, size_t n, int sh, long long* out) {
    for (size_t i = 0; i < n; ++i) out[i] = (x[i] + fx_half(sh, static_cast<int>(i & 1))) >> sh;
}

}
