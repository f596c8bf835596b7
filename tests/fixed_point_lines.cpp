// The arithmetic of the fixed-point lines (wv_fx.cuh) on the host, as C functions for
// tests/test_fixed_point_lines_cpu.py.  Test infrastructure.
#include "wv_fx.cuh"
#include "wv_plan.hpp"

#include <cstddef>
#include <utility>
#include <vector>

using namespace wvgpu::dev;

namespace {

std::vector<fxw> words(const std::vector<int32_t>& q) {
    std::vector<fxw> w(q.size() / 4);
    for (size_t i = 0; i < w.size(); ++i) w[i] = {q[4 * i], q[4 * i + 1], q[4 * i + 2], q[4 * i + 3]};
    return w;
}

// One lane-held line; the lanes walked one after the other between barriers.
template <int N, bool INV, int LATE>
void lane_line(std::vector<fxc>& line, int gap) {
    using W = FxW<N>;
    const std::vector<fxw> tw = words(W::R3 > 1 ? wvgpu::fixed_point_stage_twiddles(N, {W::R1, W::R2, W::R3})
                                                : wvgpu::fixed_point_stage_twiddles(N, {W::R1, W::R2}));
    fxc v[W::G][W::E];
    std::vector<fxc> x(W::buffer);
    for (int t = 0; t < W::G; ++t)
        for (int e = 0; e < W::E; ++e) v[t][e] = line[t + W::G * e];
    fx_line_stages<N, INV, LATE>(x.data(), tw.data(), 2, gap, [&](auto step) {
        for (int t = 0; t < W::G; ++t) step(v[t], t);
    });
    for (int t = 0; t < W::G; ++t)
        for (int e = 0; e < W::E; ++e) line[t + W::G * e] = v[t][e];
}

template <bool INV>
void any_line(std::vector<fxc>& line, int gap) {
    const int N = static_cast<int>(line.size());
    const wvgpu::FFTFactors f = wvgpu::factor_fixed_point(N);
    const std::vector<fxw> tw = words(wvgpu::fixed_point_twiddles(N));
    std::vector<fxc> other(N);
    int Ns = 1;
    for (int s = 0; s < f.nstages; ++s) {
        const FxFactors factors{N, f.nstages, f.radix};
        if (s > 0 && fx_any_radix(f.radix[s])) fx_shift_lines(line.data(), N, Ns, 1, N, fx_late_of(factors, s, Ns, nullptr, gap), 0, 1);
        fx_run_stage<INV, true>(line.data(), other.data(), factors, s, Ns, 1, N, tw.data(), nullptr, gap, 0, 1);
        Ns *= f.radix[s];
        std::swap(line, other);
    }
}

struct Form { int lane, radix, late; };  // lane: points per lane where lane-held
#define WV_LENGTHS(X) X(16) X(24) X(32) X(48) X(64) X(96) X(128) X(192) X(256)
Form form_of(int N, bool lanes, bool pair, bool inverse) {
    if (lanes) {
#define X(LEN) if (N == LEN) return {FxW<LEN>::E, FxW<LEN>::R1, inverse ? 0 : pair ? FxW<LEN>::latePair : FxW<LEN>::lateOne};
        WV_LENGTHS(X)
#undef X
    }
    const wvgpu::FFTFactors f = wvgpu::factor_fixed_point(N);
    const int radix = fx_gap_radix(f.nstages, f.radix);
    return {0, radix, N > kFxLateFrom && radix > 0 ? 1 : 0};
}
template <bool INV>
void transform(std::vector<fxc>& line, const Form& form, bool pair, int gap) {
    if (!form.lane) return any_line<INV>(line, gap);
    const int N = static_cast<int>(line.size());
#define X(LEN)                                                                   \
    if (N == LEN) {                                                              \
        if (pair) lane_line<LEN, INV, FxW<LEN>::latePair>(line, gap);            \
        else lane_line<LEN, INV, INV ? 0 : FxW<LEN>::lateOne>(line, gap);        \
    }
    WV_LENGTHS(X)
#undef X
}

unsigned high_word(double v) {
    unsigned hi, lo;
    fx_words(v, hi, lo);
    return hi;
}
// Scale and gap of entries (re, im) with `spare` bits free.
struct Scale { fxscale sc; int gap; };
Scale scale_of(const double* re, const double* im, int n, int spare, const Form& form) {
    float sum = 0.f, most = 0.f;
    for (int i = 0; i < n; ++i) {
        const float m = fx_modulus(fx_mag(high_word(re[i])), im ? fx_mag(high_word(im[i])) : 0.f);
        sum += m;
        most = m > most ? m : most;
    }
    Scale s{fx_scale(sum), form.late ? fx_gap(sum, most, form.radix) : 0};
    s.sc.bit -= spare;
    return s;
}

}  // namespace

extern "C" {

// out[i] = the product x[i] as the r2c takes it in
void shift_products(const long long* x, size_t n, int sh, long long* out) {
    for (size_t i = 0; i < n; ++i) out[i] = fx_shift_round(x[i], sh, static_cast<int>(i & 1));
}

// out[i] = (x[i] + fx_half(sh, i & 1)) >> sh: a product aligned to a larger unit
void align_products(const long long* x, size_t n, int sh, long long* out) {
    for (size_t i = 0; i < n; ++i) out[i] = (x[i] + fx_half(sh, static_cast<int>(i & 1))) >> sh;
}

// r2c of the real rows a and b on one line: spectra (re, im) of k = 0 .. N / 2 of row a.
void real_pair(const double* a, const double* b, int N, int lanes, double* out) {
    const Form form = form_of(N, lanes != 0, true, false);
    const int spare = form.lane ? 2 : 1;
    Scale sa = scale_of(a, nullptr, N, spare, form), sb = scale_of(b, nullptr, N, spare, form);
    const FxUnit o = fx_out(fx_unit(sa.sc) - 1);
    const int gap = sa.gap < sb.gap ? sa.gap : sb.gap;
    sa.sc.bit += gap;
    sb.sc.bit += gap;
    std::vector<fxc> line(N);
    for (int i = 0; i < N; ++i) line[i] = fxc{fx_from_double(a[i], sa.sc), fx_from_double(b[i], sb.sc)};
    transform<false>(line, form, true, gap);
    for (int k = 0; k <= N / 2; ++k) {
        const fxc p = line[k], q = line[(N - k) % N];
        out[2 * k] = fx_to_double(p.x + q.x, o);
        out[2 * k + 1] = fx_to_double(p.y - q.y, o);
    }
}

// A complex line z (re, im pairs).
void complex_line(const double* z, int N, int inverse, int lanes, double* out) {
    const Form form = form_of(N, lanes != 0, false, inverse != 0);
    std::vector<double> re(N), im(N);
    for (int i = 0; i < N; ++i) { re[i] = z[2 * i]; im[i] = z[2 * i + 1]; }
    Scale s = scale_of(re.data(), im.data(), N, form.lane ? 1 : 0, form);
    const FxUnit o = fx_out(fx_unit(s.sc));
    s.sc.bit += s.gap;
    std::vector<fxc> line(N);
    for (int i = 0; i < N; ++i) line[i] = fxc{fx_from_double(re[i], s.sc), fx_from_double(im[i], s.sc)};
    if (inverse) transform<true>(line, form, false, s.gap);
    else transform<false>(line, form, false, s.gap);
    for (int i = 0; i < N; ++i) {
        out[2 * i] = fx_to_double(line[i].x, o);
        out[2 * i + 1] = fx_to_double(line[i].y, o);
    }
}

}
