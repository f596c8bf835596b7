// The y and z passes of FP64 handles on lane-held fixed-point lines (wv_fxwarp.cuh).
#pragma once

#include "wv_fxwarp.cuh"

namespace wvgpu {
namespace dev {

// ---- y ------------------------------------------------------------------------------

constexpr int kFxYWarps = 8;
// Shared memory: stage twiddles and, for each of `cols` columns, a line buffer; the
// tile [y][cols] that makes the global accesses contiguous lies in the same bytes.
template <int N>
inline size_t smem_fxy(int cols) {
    return static_cast<size_t>(FxW<N>::twiddles + cols * FxW<N>::buffer) * 16;
}
// Entry (y, c) of the tile: columns are exclusive-ored with y, so that eight lanes
// of a line (consecutive y, one column) meet eight different banks.
__device__ __forceinline__ int fx_tile(int y, int c, int cols) { return y * cols + (c ^ (y & min(7, cols - 1))); }

// Inverse FFTs along y of output channel blockIdx.z, columns blockIdx.x cols ...,
// plane blockIdx.y: yspec[z][ch][y][kx] from zspec[src][z][pos] (times i l).  A line is
// held by the lanes of one warp; the tile turns the result to rows for the store.
// Bound by integer issue.  256x256x129, 12 channels: 1.71 (FP64 pipe) -> 0.464 ms;
// 192x192x97 0.32 -> 0.27 ms (run-time stages -> lanes).
template <int N>
__global__ void __launch_bounds__(32 * kFxYWarps, FxW<N>::E == 8 ? 3 : 2)
    k_yinv_fx(DescDev d, YInvMap map, const double2* __restrict__ zspec, double2* __restrict__ yspec, unsigned ltop) {
    using W = FxW<N>;
    constexpr int G = W::G, E = W::E;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int P = d.positions, KX = d.kxColumns;
    const int lane = threadIdx.x & 31, t = lane % G, own = (threadIdx.x >> 5) * W::lines + lane / G;
    const int cols = (blockDim.x >> 5) * W::lines;
    const int kx0 = blockIdx.x * cols, z = blockIdx.y, oc = blockIdx.z;
    fxw* tw = reinterpret_cast<fxw*>(smem_raw);
    fxc* x = reinterpret_cast<fxc*>(tw + W::twiddles) + own * W::buffer;
    for (int i = threadIdx.x; i < W::twiddles; i += blockDim.x) tw[i] = d.fxTwY[i];
    const double2* in = zspec + (static_cast<size_t>(map.src[oc]) * d.zTotal + z) * P;
    const int kx = kx0 + own;
    double2 a[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const int pos = kx < KX ? d.ymap[static_cast<size_t>(kx) * N + t + G * e] : -1;
        a[e] = pos >= 0 ? in[pos] : make_double2(0.0, 0.0);
    }
    fxc v[E];
    int unit;
    double w[E];
    auto count = [](int) { return 1.0f; };
    if (map.mulL[oc]) {
        const double* rowL = row_l<double>(d);
#pragma unroll
        for (int e = 0; e < E; ++e) w[e] = rowL[t + G * e];
        fx_quantise_lane<E, G, kFxImag>(a, w, ltop, 0, count, v, unit);
    } else {
        fx_quantise_lane<E, G, kFxPlain>(a, w, 0u, 0, count, v, unit);
    }
    __syncthreads();  // twiddles
    fx_fft_warp<N, true>(v, x, tw, t, fx_silent(unit) ? 0 : fx_two());
    __syncthreads();  // every line buffer read: the tile takes their place
    double2* tile = reinterpret_cast<double2*>(tw + W::twiddles);
    const FxUnit o = fx_out(unit);
#pragma unroll
    for (int e = 0; e < E; ++e)
        tile[fx_tile(t + G * e, own, cols)] = make_double2(fx_to_double(v[e].x, o), fx_to_double(v[e].y, o));
    __syncthreads();
    double2* out = yspec + (static_cast<size_t>(z) * map.nOut + oc) * N * KX + kx0;
    const int g = min(cols, KX - kx0);
    for (int i = threadIdx.x; i < N * cols; i += blockDim.x) {
        const int y = i / cols, c = i - y * cols;
        if (c < g) out[static_cast<size_t>(y) * KX + c] = tile[fx_tile(y, c, cols)];
    }
}

// Forward FFTs along y of channel blockIdx.z, gathered to the active rows:
// fspec[c][z][pos] from pspec[z][c][y][kx].  256x256x129, 4 channels: 0.54 (FP64 pipe)
// -> 0.142 ms.
template <int N>
__global__ void __launch_bounds__(32 * kFxYWarps, FxW<N>::E == 8 ? 3 : 2)
    k_yfwd_fx(DescDev d, const double2* __restrict__ pspec, int nch, double2* __restrict__ fspec) {
    using W = FxW<N>;
    constexpr int G = W::G, E = W::E;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int P = d.positions, KX = d.kxColumns;
    const int lane = threadIdx.x & 31, t = lane % G, own = (threadIdx.x >> 5) * W::lines + lane / G;
    const int cols = (blockDim.x >> 5) * W::lines;
    const int kx0 = blockIdx.x * cols, z = blockIdx.y, ch = blockIdx.z;
    fxw* tw = reinterpret_cast<fxw*>(smem_raw);
    fxc* x = reinterpret_cast<fxc*>(tw + W::twiddles) + own * W::buffer;
    double2* tile = reinterpret_cast<double2*>(tw + W::twiddles);
    for (int i = threadIdx.x; i < W::twiddles; i += blockDim.x) tw[i] = d.fxTwY[i];
    const double2* in = pspec + (static_cast<size_t>(z) * nch + ch) * N * KX + kx0;
    const int g = min(cols, KX - kx0);
    for (int i = threadIdx.x; i < N * cols; i += blockDim.x) {
        const int y = i / cols, c = i - y * cols;
        tile[fx_tile(y, c, cols)] = c < g ? in[static_cast<size_t>(y) * KX + c] : make_double2(0.0, 0.0);
    }
    __syncthreads();
    double2 a[E];
#pragma unroll
    for (int e = 0; e < E; ++e) a[e] = tile[fx_tile(t + G * e, own, cols)];
    __syncthreads();  // the line buffers take the tile's place
    fxc v[E];
    double w[E];
    const FxLine l = fx_line<E, G, kFxPlain, W::lateOne ? W::R1 : 0>(a, w, 0u, 0, [](int) { return 1.0f; });
    fx_fixed<E, kFxPlain>(a, w, l.base - l.gap, v);
    const int unit = l.unit;
    fx_fft_warp<N, false, W::lateOne>(v, x, tw, t, fx_silent(unit) ? 0 : fx_two(), l.gap);
    const int kx = kx0 + own;
    if (kx >= KX) return;
    double2* out = fspec + (static_cast<size_t>(ch) * d.zTotal + z) * P;
    const FxUnit o = fx_out(unit);
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const int pos = d.ymap[static_cast<size_t>(kx) * N + t + G * e];
        if (pos >= 0) out[pos] = make_double2(fx_to_double(v[e].x, o), fx_to_double(v[e].y, o));
    }
}

// Real values of a lane (E a row), for two rows to a line (as fx_line and fx_fixed).
template <int E, int G, int RADIX>
__device__ __forceinline__ FxLine fx_real_line(const double (&a)[E]) {
    float sum = 0.f, most = 0.f;
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const float m = fx_mag(static_cast<unsigned>(__double2hiint(a[e])));
        sum += m;
        if (RADIX) most = fmaxf(most, m);
    }
    sum = fx_group_sum<G>(sum);
    int gap = 0;
    if (RADIX) gap = fx_gap(sum, __uint_as_float(fx_group_max<G>(__float_as_uint(most))), RADIX);
    fxscale sc = fx_scale(sum);
    const bool odd = !fx_plain_sum(sum);
    if (__any_sync(0xffffffffu, odd)) {
        unsigned top = 0;
#pragma unroll
        for (int e = 0; e < E; ++e) top = max(top, static_cast<unsigned>(__double2hiint(a[e])) & 0x7fffffffu);
        top = fx_group_max<G>(top);
        float rel = 0.f, relMost = 0.f;
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const float m = fx_rel(static_cast<unsigned>(__double2hiint(a[e])), top);
            rel += m;
            relMost = fmaxf(relMost, m);
        }
        rel = fx_group_sum<G>(rel);
        if (RADIX) relMost = __uint_as_float(fx_group_max<G>(__float_as_uint(relMost)));
        if (odd) {
            sc = fx_scale(top, rel);
            gap = top == 0 ? kFxAnyGap : RADIX ? fx_gap(rel, relMost, RADIX) : 0;
        }
    }
    sc.bit -= 2;
    return {61 - sc.bit + sc.e0, fx_unit(sc), gap};
}
template <int E>
__device__ __forceinline__ void fx_real_fixed(const double (&a)[E], int base, long long (&out)[E]) {
#pragma unroll
    for (int e = 0; e < E; ++e) {
        int ex;
        const unsigned long long m = fx_mantissa(a[e], ex);
        out[e] = fx_shift_in(m, base - ex, __double2hiint(a[e]));
    }
}
// Two real rows of a lane as the line ra + i rb.
template <int N>
__device__ __forceinline__ void fx_real_pair(const double (&ra)[FxW<N>::E], const double (&rb)[FxW<N>::E], fxc (&v)[FxW<N>::E],
                                             int& ua, int& ub, int& gap) {
    constexpr int E = FxW<N>::E, G = FxW<N>::G, radix = FxW<N>::latePair ? FxW<N>::R1 : 0;
    long long ia[E], ib[E];
    const FxLine la = fx_real_line<E, G, radix>(ra), lb = fx_real_line<E, G, radix>(rb);
    gap = fx_shared_gap(la.gap, lb.gap);
    ua = la.unit;
    ub = lb.unit;
    fx_real_fixed<E>(ra, la.base - gap, ia);
    fx_real_fixed<E>(rb, lb.base - gap, ib);
#pragma unroll
    for (int e = 0; e < E; ++e) v[e] = fxc{ia[e], ib[e]};
}

// ---- field rows along x -----------------------------------------------------------------

constexpr int kFxFieldWarps = 4;
template <int N>
inline size_t smem_fx_field(int warps) { return (FxW<N>::twiddles + warps * FxW<N>::lines * FxW<N>::buffer) * 16; }

// k_xc2r_fields: a warp takes two channels of a line-set of rows as one line.  KX may
// reach N / 2 + 1 (the scalar pipeline's full half spectrum).  Inverse transform at
// 192x192x97: 1.17 ms (FP64 pipe) -> 0.253 ms.
template <int N>
__global__ void __launch_bounds__(32 * kFxFieldWarps, 4)
    k_xc2r_fx(DescDev d, const fxw* __restrict__ twg, const double2* __restrict__ yspec, int nch, double* __restrict__ fields) {
    using W = FxW<N>;
    constexpr int G = W::G, E = W::E, H = W::H;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int Ny = d.Ny, KX = d.kxColumns;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int t = lane % G, line = lane / G;
    fxw* tw = reinterpret_cast<fxw*>(smem_raw);
    fxc* x = reinterpret_cast<fxc*>(tw + W::twiddles) + static_cast<size_t>(warp * W::lines + line) * W::buffer;
    for (int i = threadIdx.x; i < W::twiddles; i += blockDim.x) tw[i] = twg[i];
    const int rows = Ny * d.zTotal, pairs = (nch + 1) / 2;
    const int unitOfWork = blockIdx.x * (blockDim.x >> 5) + warp;
    const int p = unitOfWork % pairs, first = unitOfWork / pairs * W::lines;
    const bool live = first + line < rows;
    const int row = min(first + line, rows - 1);
    const int z = row / Ny, y = row - z * Ny;
    const double* rowK = row_k<double>(d);
    const unsigned wtop = fx_row_k_top(rowK, KX);
    // entries k = t + G i of both channels, and k = N / 2 on lane 0
    fxc AB[2][H + 1];
    int unit[2] = {kFxZero, kFxZero};
    auto count = [&](int i) { return (i == 0 && t == 0) || i == H ? 1.0f : 2.0f; };
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const int c = 2 * p + q;
        const double2* h = yspec + ((static_cast<size_t>(z) * nch + min(c, nch - 1)) * Ny + y) * KX;
        double2 a[H + 1];
        double w[H + 1];
        const bool useK = ((d.c2rUseK >> c) & 1) != 0;
#pragma unroll
        for (int i = 0; i < H + 1; ++i) {
            const int k = t + G * i;
            const bool has = c < nch && k < KX && (i < H || t == 0);
            a[i] = has ? h[k] : make_double2(0.0, 0.0);
            w[i] = useK && has ? rowK[k] : 0.0;
            if (k == 0 || i == H) a[i].y = 0.0;  // c2r semantics
        }
        if (useK) {
            fx_quantise_lane<H + 1, G, kFxImag>(a, w, wtop, 1, count, AB[q], unit[q]);
            AB[q][H].y = 0;
        } else {
            fx_quantise_lane<H + 1, G, kFxPlain>(a, w, 0u, 1, count, AB[q], unit[q]);
        }
    }
    __syncthreads();  // twiddles
    fxc v[E];
#pragma unroll
    for (int i = 0; i < H; ++i) {
        const fxc a = AB[0][i], b = AB[1][i];
        const int k = t + G * i;
        v[i] = fxc{a.x - b.y, a.y + b.x};
        x[fx_pad(k == 0 ? N / 2 : N - k)] = k == 0 ? fxc{AB[0][H].x, AB[1][H].x} : fxc{a.x + b.y, b.x - a.y};
    }
    __syncwarp();
#pragma unroll
    for (int e = H; e < E; ++e) v[e] = x[fx_pad(t + G * e)];
    __syncwarp();
    fx_fft_warp<N, true>(v, x, tw, t, fx_silent(max(unit[0], unit[1])) ? 0 : fx_two());
    if (!live) return;
    const FxUnit oa = fx_out(unit[0]), ob = fx_out(unit[1]);
    const size_t R = static_cast<size_t>(N) * Ny * d.Nz;
    double* o = fields + static_cast<size_t>(2 * p) * R + (static_cast<size_t>(z) * Ny + y) * N;
#pragma unroll
    for (int e = 0; e < E; ++e) {
        o[t + G * e] = fx_to_double(v[e].x, oa);
        if (2 * p + 1 < nch) o[R + t + G * e] = fx_to_double(v[e].y, ob);
    }
}

// k_xr2c_fields: a warp takes two channels of a line-set of rows as one line.  Forward
// transform at 256x256x65, hydrostatic: 0.305 ms with run-time lines (0.893 on the FP64
// pipe), 0.220 with these, 0.234 with the finer start of lines of samples.
template <int N>
__global__ void __launch_bounds__(32 * kFxFieldWarps, 4)
    k_xr2c_fx(DescDev d, const fxw* __restrict__ twg, const double* __restrict__ fields, int nch, double2* __restrict__ pspec) {
    using W = FxW<N>;
    constexpr int G = W::G, E = W::E, H = W::H;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int Ny = d.Ny, KX = d.kxColumns;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int t = lane % G, line = lane / G;
    fxw* tw = reinterpret_cast<fxw*>(smem_raw);
    fxc* x = reinterpret_cast<fxc*>(tw + W::twiddles) + static_cast<size_t>(warp * W::lines + line) * W::buffer;
    for (int i = threadIdx.x; i < W::twiddles; i += blockDim.x) tw[i] = twg[i];
    const int rows = Ny * d.zTotal, pairs = (nch + 1) / 2;
    const int unitOfWork = blockIdx.x * (blockDim.x >> 5) + warp;
    const int p = unitOfWork % pairs, first = unitOfWork / pairs * W::lines;
    const bool live = first + line < rows, both = 2 * p + 1 < nch;
    const int row = min(first + line, rows - 1);
    const int z = row / Ny, y = row - z * Ny;
    const size_t R = static_cast<size_t>(N) * Ny * d.Nz;
    const double* in = fields + static_cast<size_t>(2 * p) * R + (static_cast<size_t>(z) * Ny + y) * N;
    double ra[E], rb[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
        ra[e] = in[t + G * e];
        rb[e] = both ? in[R + t + G * e] : 0.0;
    }
    fxc v[E];
    int ua, ub, gap;
    fx_real_pair<N>(ra, rb, v, ua, ub, gap);
    __syncthreads();  // twiddles
    fx_fft_warp<N, false, W::latePair>(v, x, tw, t, fx_silent(max(ua, ub)) ? 0 : fx_two(), gap);
#pragma unroll
    for (int e = H; e < E; ++e) x[fx_pad(t + G * e)] = v[e];
    __syncwarp();
    if (!live) return;
    const FxUnit oa = fx_out(ua - 1), ob = fx_out(ub - 1);  // the halves of the split
    double2* out = pspec + ((static_cast<size_t>(z) * nch + 2 * p) * Ny + y) * KX;
    const size_t cstride = static_cast<size_t>(Ny) * KX;
    auto store = [&](int k, fxc a, fxc b) {
        out[k] = make_double2(fx_to_double(a.x + b.x, oa), fx_to_double(a.y - b.y, oa));
        if (both) out[cstride + k] = make_double2(fx_to_double(a.y + b.y, ob), fx_to_double(b.x - a.x, ob));
    };
#pragma unroll
    for (int i = 0; i < H; ++i) {
        const int k = t + G * i;
        if (k < KX) store(k, v[i], k == 0 ? v[0] : x[fx_pad(N - k)]);
    }
    if (t == 0 && N / 2 < KX) store(N / 2, v[H], v[H]);
}

// ---- phases ----------------------------------------------------------------------------

// exp(i angle) rounded from fixed point: the angle in turns is the exact product of
// its 53 bits with 1 / (2 pi) to 128 bits, the nearest of 256 table entries is
// turned by the remainder |r| <= pi / 256 with Taylor sums (sine to r^7, cosine to
// r^6; the next terms are below 2^-62).  Angles below 2^-6 rad take the Taylor sums in
// FP64 (to a^7 and a^6), so that a small sine keeps its digits.  About 170 integer instructions; the FP64
// sincos it replaces takes some 50 operations of a pipe that retires 1.7 per clock
// and SM (30 clocks against 1.3 a value).
__device__ __forceinline__ void fx_phase(double angle, const fxw* __restrict__ table, double& cs, double& sn) {
    const unsigned hi = static_cast<unsigned>(__double2hiint(angle));
    const int e = static_cast<int>((hi >> 20) & 0x7ffu);
    if (e >= 1023 + 31) {  // beyond 2^31 rad (and inf, NaN): the library's reduction
        sincos(angle, &sn, &cs);
        return;
    }
    if (e < 1023 - 6) {  // below 2^-6 rad the fixed point's 2^-62 is no longer small against the sine
        const double q = angle * angle;
        sn = fma(angle * q, fma(q, fma(q, -1.0 / 5040.0, 1.0 / 120.0), -1.0 / 6.0), angle);
        cs = fma(q, fma(q, fma(q, -1.0 / 720.0, 1.0 / 24.0), -0.5), 1.0);
        return;
    }
    const unsigned long long m = static_cast<unsigned long long>((hi & 0xfffffu) | 0x100000u) << 32 |
                                 static_cast<unsigned>(__double2loint(angle));
    constexpr unsigned long long c1 = 0x28be60db9391054aull, c0 = 0x7f09d5f47d4d3770ull;  // 2^128 / (2 pi)
    const unsigned long long lo = m * c1, add = __umul64hi(m, c0);
    unsigned long long q1 = __umul64hi(m, c1), q0 = lo + add;
    q1 += q0 < lo ? 1ull : 0ull;
    const int s = 1075 - e;  // turns = (q1:q0) 2^-(64 + s); s > 21
    unsigned long long f;
    if (s < 64) f = (q0 >> s) | (q1 << (64 - s));
    else f = s < 128 ? q1 >> (s - 64) : 0ull;
    if (static_cast<int>(hi) < 0) f = 0ull - f;
    const unsigned idx = static_cast<unsigned>((f + (1ull << 55)) >> 56) & 255u;
    const long long r = static_cast<long long>(f - (static_cast<unsigned long long>(idx) << 56));  // turns, Q64
    constexpr long long qpi = 3622009729038561421ll;  // pi / 4
    const long long th = fx_rmul(r, fx_qh(qpi), fx_ql(qpi)) * 2;                // 2 pi r in Q62
    const long long s2 = fx_prod(th, th);
    constexpr long long k6 = 768614336404564651ll, k120 = 38430716820228233ll, k5040 = 915017067148291ll;
    constexpr long long k24 = 192153584101141163ll, k720 = 6405119470038039ll, k2 = 2305843009213693952ll;
    const long long ps = k6 - fx_prod(k120 - fx_rmul(s2, fx_qh(k5040), fx_ql(k5040)), s2);
    const long long pc = k2 - fx_prod(k24 - fx_rmul(s2, fx_qh(k720), fx_ql(k720)), s2);
    const fxc small = {-fx_prod(pc, s2), th - fx_prod(fx_prod(ps, s2), th)};  // cos r - 1, sin r
    const fxw w = table[idx];
    const fxc turned = fx_cmul<false>(small, w);
    const long long tc = static_cast<long long>(w.ch) * 4294967296ll + w.cl, ts = static_cast<long long>(w.sh) * 4294967296ll + w.sl;
    cs = fx_to_double(tc + turned.x, 1023 - 62);
    sn = fx_to_double(ts + turned.y, 1023 - 62);
}

// ---- z ------------------------------------------------------------------------------

// Field spectra u, v, w, eta of one (mode, j) (vinv_field_spectra's formulas with
// the structure of the factors used: W's and the geostrophic u, v factors are
// imaginary, and UAp Ap + conj(UAp) Am = Re(UAp) (Ap + Am) + i Im(UAp) (Ap - Am)).
__device__ __forceinline__ void fx_field_spectra(const DescDev& d, const double* __restrict__ Ap, const double* __restrict__ Am,
                                                 const double* __restrict__ A0, double elapsed, int w, unsigned char flags, int j,
                                                 double2 (&f)[4]) {
    const int idx = j + d.Nj * w;
    double c, s;
    fx_phase(d.omega[idx] * elapsed, d.fxPhase, c, s);
    const zd p0 = zload(Ap + 2 * idx), m0 = zload(Am + 2 * idx), a = zload(A0 + 2 * idx);
    const zd p = {p0.re * c - p0.im * s, p0.re * s + p0.im * c};
    const zd m = {m0.re * c + m0.im * s, m0.im * c - m0.re * s};
    const zd sum = {p.re + m.re, p.im + m.im}, dif = {p.re - m.re, p.im - m.im};
    const zd uap = zload(d.UAp + 2 * idx), vap = zload(d.VAp + 2 * idx);
    const double wi = d.WAp[2 * idx + 1], u0 = d.UA0[2 * idx + 1], v0 = d.VA0[2 * idx + 1];
    const double nap = d.NAp[idx], na0 = d.NA0[idx];
    f[0] = make_double2(uap.re * sum.re - uap.im * dif.im - u0 * a.im, uap.re * sum.im + uap.im * dif.re + u0 * a.re);
    f[1] = make_double2(vap.re * sum.re - vap.im * dif.im - v0 * a.im, vap.re * sum.im + vap.im * dif.re + v0 * a.re);
    f[2] = make_double2(-wi * sum.im, wi * sum.re);
    f[3] = make_double2(nap * dif.re + na0 * a.re, nap * dif.im + na0 * a.im);
    if (flags & 1) {
#pragma unroll
        for (int q = 0; q < 4; ++q) f[q].y = -f[q].y;
    }
    if (flags & 2) {
#pragma unroll
        for (int q = 0; q < 4; ++q) f[q].y = 0.0;
    }
}

// Projection of one (mode, j) of the forward transforms: U, V, W, E are the unscaled
// channel values, sc their normalisation.  One linear map for the flux and the
// forward transform (projectFluxTargetMode, projectNonhydrostaticMode,
// projectHydrostaticMode, kernel.cpp:299-431): with the real factors Cu, Cv, Cw
//   wave = Cu U + Cv V + i Cw W,  a0 = i (k V - l U) vort + E buoy,
//   b = (E - NA0 a0) ApmN,  cp = wave + b,  cm = wave - b.
template <bool FLUX>
__device__ __forceinline__ void fx_project(const DescDev& d, int w, int j, double2 U, double2 V, double2 W, double2 E, double sc,
                                           double elapsed, double maxSpeed, int applyDamping, const double* __restrict__ Ap,
                                           const double* __restrict__ Am, const double* __restrict__ A0,
                                           double* __restrict__ Fp, double* __restrict__ Fm, double* __restrict__ F0) {
    const int idx = j + d.Nj * w;
    const double k = d.k[w], l = d.l[w];
    const double vort = d.A0FromVorticity[idx], buoy = d.A0FromBuoyancy[idx], na0 = d.NA0[idx], apmn = d.ApmN[idx];
    const double a0r = (l * U.y - k * V.y) * vort + E.x * buoy, a0i = (k * V.x - l * U.x) * vort + E.y * buoy;
    double cpr, cpi, cmr, cmi;
    if (w == 0) {
        const double is = d.inertialScale[j];
        cpr = is * (U.x + V.y); cpi = is * (U.y - V.x);
        cmr = cpr; cmi = -cpi;
    } else {
        double wr, wi;
        if (d.hydrostatic) {
            const double g = -d.ApmD[2 * idx + 1];
            wr = g * (k * U.x + l * V.x); wi = g * (k * U.y + l * V.y);
        } else {
            const double g = d.ApmDScaled[idx], h = (d.Kh[w] / 2.0) * d.apmWPrefactor[j];
            wr = (d.cosAlpha[w] * U.x + d.sinAlpha[w] * V.x) * g - h * W.y;
            wi = (d.cosAlpha[w] * U.y + d.sinAlpha[w] * V.y) * g + h * W.x;
        }
        const double br = (E.x - na0 * a0r) * apmn, bi = (E.y - na0 * a0i) * apmn;
        cpr = wr + br; cpi = wi + bi; cmr = wr - br; cmi = wi - bi;
    }
    double c, s;
    fx_phase(d.omega[idx] * elapsed, d.fxPhase, c, s);
    c *= sc; s *= sc;
    zd fp{cpr * c + cpi * s, cpi * c - cpr * s};  // cp conj(p)
    zd fm{cmr * c - cmi * s, cmr * s + cmi * c};  // cm p
    zd f0{a0r * sc, a0i * sc};
    if (FLUX && applyDamping) {
        const double sd = __dmul_rn(maxSpeed, d.damping[idx]);
        fp = zadd(fp, zscale(zload(Ap + 2 * idx), sd));
        fm = zadd(fm, zscale(zload(Am + 2 * idx), sd));
        f0 = zadd(f0, zscale(zload(A0 + 2 * idx), sd));
    }
    zstore(Fp + 2 * idx, fp);
    zstore(Fm + 2 * idx, fm);
    zstore(F0 + 2 * idx, f0);
}

constexpr int kFxZWarps = 8;
// Lines of one retained column: 4 (flux) or 2 in the inverse, 2 forward; each is a
// warp's, so a column's lines run side by side (a small grid has few columns, and a
// warp that walked them in turn took 24 us at 16x16x9).
// A block holds 8 / lines sets of FxW<N>::lines columns.
template <int N>
inline size_t smem_fx_z(int lines, int sets) {
    const size_t columns = static_cast<size_t>(sets) * FxW<N>::lines;
    return (FxW<N>::twiddles + columns * (lines * FxW<N>::buffer + 2 * N)) * 16;
}

// k_vinv_fft (wv_vfft.cuh) in fixed point: the pairs (u | w), (v | eta) and, for the
// flux, (m w | -m u), (m eta | -m v).  The two channels of a pair keep their own
// scales (the even and the odd part separate them again), so neither rounds at the
// other's magnitude.  Bound by integer issue and, in the field spectra, by FP64.
// 256x256x129: 0.99 (FP64 pipe) -> 0.222 ms; 16x16x9 24 -> 14 us with a line per warp.
template <int N, bool FLUX>
__global__ void __launch_bounds__(32 * kFxZWarps, FxW<N>::E == 8 ? 3 : 2)
    k_vinv_fx(DescDev d, const double* __restrict__ Ap, const double* __restrict__ Am, const double* __restrict__ A0,
              double elapsed, double2* __restrict__ zspec, unsigned long long* __restrict__ maxSpeedBits) {
    using W = FxW<N>;
    constexpr int G = W::G, E = W::E, H = W::H, kLines = FLUX ? 4 : 2;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int Nj = d.Nj, P = d.positions;
    const int lane = threadIdx.x & 31, t = lane % G, warp = threadIdx.x >> 5;
    const int set = warp / kLines, l = warp - set * kLines;
    const int sets = (blockDim.x >> 5) / kLines;
    const int member = blockIdx.y;
    if (member > 0) {
        const long long o = member * d.memberStride;
        Ap += o; Am += o; A0 += o;
        zspec += static_cast<size_t>(member) * d.Nz * P;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0 && maxSpeedBits) maxSpeedBits[member] = 0ull;
    fxw* tw = reinterpret_cast<fxw*>(smem_raw);
    const int column = set * W::lines + lane / G;
    fxc* x = reinterpret_cast<fxc*>(tw + W::twiddles) + static_cast<size_t>(column * kLines + l) * W::buffer;
    double2* fld = reinterpret_cast<double2*>(reinterpret_cast<fxc*>(tw + W::twiddles) +
                                              static_cast<size_t>(sets) * W::lines * kLines * W::buffer) +
                   static_cast<size_t>(column) * 2 * N;  // field spectra [4][N/2]
    for (int i = threadIdx.x; i < W::twiddles; i += blockDim.x) tw[i] = d.fxTwZ[i];
    const int want = blockIdx.x * sets * W::lines + column;
    const bool live = want < d.Nkl;
    const int mode = min(want, d.Nkl - 1);
    const double* mz = static_cast<const double*>(d.tMz);
    const unsigned mtop = static_cast<unsigned>(__double2hiint(mz[Nj - 1]));
    {
        const int w = d.modeWV[mode];
        const unsigned char flags = d.modeFlags[mode];
#pragma unroll 1
        for (int i = l; i < H; i += kLines) {  // the column's warps share its coefficients
            const int j = t + G * i;
            double2 f[4];
            if (j < Nj) fx_field_spectra(d, Ap, Am, A0, elapsed, w, flags, j, f);
#pragma unroll
            for (int q = 0; q < 4; ++q) fld[q * (N / 2) + j] = j < Nj ? f[q] : make_double2(0.0, 0.0);
        }
    }
    __syncthreads();
    int derivC = -1, derivS = -1;  // channels of the z derivatives of targets l and l - 2
    if constexpr (FLUX)
        for (int q = 0; q < d.nt; ++q) {
            if (d.tq[q] == l) derivC = 4 + q;
            if (d.tq[q] == l - 2) derivS = 4 + q;
        }
    const int pos = d.modePos[mode], cpos = d.modeCompPos[mode];
    auto count = [&](int i) { return i == 0 && t == 0 ? 1.0f : 2.0f; };
    // fld slots of the cosine and sine channels: (0|2) (1|3) (2|0) (3|1)
    const int qs = l < 2 ? l + 2 : l - 2;
    const int chC = l < 2 ? l : derivC, chS = l < 2 ? l + 2 : derivS;
    double2 a[H];
    double wgt[H];
    fxc C[H], D[H];
    int uC, uD;
    if (l < 2) {
#pragma unroll
        for (int i = 0; i < H; ++i) a[i] = fld[l * (N / 2) + t + G * i];
        fx_quantise_lane<H, G, kFxPlain>(a, wgt, 0u, 1, count, C, uC);
#pragma unroll
        for (int i = 0; i < H; ++i) a[i] = fld[qs * (N / 2) + t + G * i];
        fx_quantise_lane<H, G, kFxPlain>(a, wgt, 0u, 1, count, D, uD);
    } else {
#pragma unroll
        for (int i = 0; i < H; ++i) {
            a[i] = fld[l * (N / 2) + t + G * i];
            wgt[i] = t + G * i < Nj ? mz[t + G * i] : 0.0;
        }
        fx_quantise_lane<H, G, kFxReal>(a, wgt, mtop, 1, count, C, uC);
#pragma unroll
        for (int i = 0; i < H; ++i) {
            a[i] = fld[qs * (N / 2) + t + G * i];
            wgt[i] = -wgt[i];
        }
        fx_quantise_lane<H, G, kFxReal>(a, wgt, mtop, 1, count, D, uD);
    }
    // 2 y[j] = C_j + i D_j, 2 y[N-j] = C_j - i D_j, 2 y[0] = C_0
    fxc v[E];
#pragma unroll
    for (int i = 0; i < H; ++i) {
        const int j = t + G * i;
        if (j == 0) D[i] = fxc{0, 0};
        v[i] = fxc{C[i].x - D[i].y, C[i].y + D[i].x};
        x[fx_pad(j == 0 ? N / 2 : N - j)] = j == 0 ? fxc{0, 0} : fxc{C[i].x + D[i].y, C[i].y - D[i].x};
    }
    __syncwarp();
#pragma unroll
    for (int e = H; e < E; ++e) v[e] = x[fx_pad(t + G * e)];
    __syncwarp();
    fx_fft_warp<N, false>(v, x, tw, t, fx_silent(max(uC, uD)) ? 0 : fx_two());
#pragma unroll
    for (int e = H; e < E; ++e) x[fx_pad(t + G * e)] = v[e];
    __syncwarp();
    if (!live) return;
    // even part -> cosine channel, odd part -> sine channel, n = 0 .. N / 2
    const FxUnit oC = fx_out(uC - 2), oD = fx_out(uD - 2);
    double2* baseC = zspec + static_cast<size_t>(chC) * d.zTotal * P;
    double2* baseS = zspec + static_cast<size_t>(chS) * d.zTotal * P;
    auto put = [&](int n, fxc a1, fxc b1) {
        const size_t o = static_cast<size_t>(n) * P;
        if (chC >= 0) {
            const double2 ev = make_double2(fx_to_double(a1.x + b1.x, oC), fx_to_double(a1.y + b1.y, oC));
            baseC[o + pos] = ev;
            if (cpos >= 0) baseC[o + cpos] = make_double2(ev.x, -ev.y);
        }
        if (chS >= 0) {
            const double2 od = make_double2(fx_to_double(a1.x - b1.x, oD), fx_to_double(a1.y - b1.y, oD));
            baseS[o + pos] = od;
            if (cpos >= 0) baseS[o + cpos] = make_double2(od.x, -od.y);
        }
    };
#pragma unroll
    for (int i = 0; i < H; ++i) {
        const int n = t + G * i;
        put(n, v[i], n == 0 ? v[0] : x[fx_pad(N - n)]);
    }
    if (t == 0) put(N / 2, v[H], v[H]);
}

// k_vfwd_fft in fixed point: lines (u | w) and (v | eta) of a column by two warps,
// which then share its coefficients' projection (FP64; its chain of dependent
// operations is what small grids wait for).  256x256x129: 0.81 (FP64 pipe) -> 0.180 ms.
template <int N, bool FLUX>
__global__ void __launch_bounds__(32 * kFxZWarps, FxW<N>::E == 8 ? 3 : 2)
    k_vfwd_fx(DescDev d, const double2* __restrict__ fspec, int nch, double elapsed, const double* __restrict__ Ap,
              const double* __restrict__ Am, const double* __restrict__ A0, const unsigned long long* __restrict__ maxSpeedBits,
              int applyDamping, double* __restrict__ Fp, double* __restrict__ Fm, double* __restrict__ F0) {
    using W = FxW<N>;
    constexpr int G = W::G, E = W::E, H = W::H, L = N / 2;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int Nj = d.Nj, P = d.positions;
    const int lane = threadIdx.x & 31, t = lane % G, warp = threadIdx.x >> 5;
    const int set = warp >> 1, l = warp & 1, sets = blockDim.x >> 6;
    const int member = blockIdx.y;
    if (member > 0) {
        const long long o = member * d.memberStride;
        if (Ap) { Ap += o; Am += o; A0 += o; }
        Fp += o; Fm += o; F0 += o;
        fspec += static_cast<size_t>(member) * d.Nz * P;
        if (maxSpeedBits) maxSpeedBits += member;
    }
    fxw* tw = reinterpret_cast<fxw*>(smem_raw);
    const int column = set * W::lines + lane / G;
    fxc* x = reinterpret_cast<fxc*>(tw + W::twiddles) + static_cast<size_t>(column * 2 + l) * W::buffer;
    double2* X = reinterpret_cast<double2*>(reinterpret_cast<fxc*>(tw + W::twiddles) +
                                            static_cast<size_t>(sets) * W::lines * 2 * W::buffer) +
                 static_cast<size_t>(column) * 2 * N;  // transformed slots [4][N/2]: 0 u, 1 v (cosine), 2 w, 3 eta (sine)
    for (int i = threadIdx.x; i < W::twiddles; i += blockDim.x) tw[i] = d.fxTwZ[i];
    const int want = blockIdx.x * sets * W::lines + column;
    const bool live = want < d.Nkl;
    const int mode = min(want, d.Nkl - 1);
    int cc = -1, cs = -1;  // channels of slots l and 2 + l
    for (int c = 0; c < nch; ++c) {
        const int q = FLUX ? d.tq[c] : ((d.hydrostatic && c == 2) ? 3 : c);
        if (q == l) cc = c;
        if (q == 2 + l) cs = c;
    }
    {
        const int pos = d.modePos[mode];
        const double2* hc = fspec + static_cast<size_t>(max(cc, 0)) * d.zTotal * P + pos;
        const double2* hs = fspec + static_cast<size_t>(max(cs, 0)) * d.zTotal * P + pos;
        double2 a[H + 1], b[H];
        double none5[H + 1], none4[H];
#pragma unroll
        for (int i = 0; i < H + 1; ++i) {
            const int zz = t + G * i;
            a[i] = cc >= 0 && (i < H || t == 0) ? hc[static_cast<size_t>(zz) * P] : make_double2(0.0, 0.0);
            if (i < H) b[i] = cs >= 0 && zz != 0 ? hs[static_cast<size_t>(zz) * P] : make_double2(0.0, 0.0);
        }
        fxc C[H + 1], S[H];
        constexpr int radix = W::latePair ? W::R1 : 0;
        const FxLine lC = fx_line<H + 1, G, kFxPlain, radix>(a, none5, 0u, 1, [&](int i) { return (i == 0 && t == 0) || i == H ? 1.0f : 2.0f; });
        const FxLine lS = fx_line<H, G, kFxPlain, radix>(b, none4, 0u, 1, [&](int) { return 2.0f; });
        const int gap = fx_shared_gap(lC.gap, lS.gap), uC = lC.unit, uS = lS.unit;
        fx_fixed<H + 1, kFxPlain>(a, none5, lC.base - gap, C);
        fx_fixed<H, kFxPlain>(b, none4, lS.base - gap, S);
        __syncthreads();  // twiddles
        // y[0] = c_0, y[L] = c_L, y[z] = c_z + s_z, y[N-z] = c_z - s_z
        fxc v[E];
#pragma unroll
        for (int i = 0; i < H; ++i) {
            const int zz = t + G * i;
            v[i] = fx_add(C[i], S[i]);
            x[fx_pad(zz == 0 ? L : N - zz)] = zz == 0 ? C[H] : fx_sub(C[i], S[i]);
        }
        __syncwarp();
#pragma unroll
        for (int e = H; e < E; ++e) v[e] = x[fx_pad(t + G * e)];
        __syncwarp();
        fx_fft_warp<N, false, W::latePair>(v, x, tw, t, fx_silent(max(uC, uS)) ? 0 : fx_two(), gap);
        const FxUnit oC = fx_out(uC - 1), oS = fx_out(uS - 1);
#pragma unroll
        for (int e = H; e < E; ++e) x[fx_pad(t + G * e)] = v[e];
        __syncwarp();
#pragma unroll
        for (int i = 0; i < H; ++i) {
            const int j = t + G * i;
            if (j >= Nj) continue;
            const fxc p = v[i], q = j == 0 ? v[0] : x[fx_pad(N - j)];
            X[l * L + j] = make_double2(fx_to_double(p.x + q.x, oC), fx_to_double(p.y + q.y, oC));
            // i times the odd part
            X[(2 + l) * L + j] = make_double2(-fx_to_double(p.y - q.y, oS), fx_to_double(p.x - q.x, oS));
        }
    }
    __syncthreads();
    if (!live) return;
    const int w = d.modeWV[mode];
    const bool conj = d.modeFlags[mode] & 1;
    const double sc = 1.0 / (static_cast<double>(L) * static_cast<double>(d.Nx) * static_cast<double>(d.Ny));
    double maxSpeed = 0.0;
    if (FLUX && applyDamping) maxSpeed = __longlong_as_double((long long)*maxSpeedBits);
#pragma unroll 1
    for (int i = l; i < H; i += 2) {
        const int j = t + G * i;
        if (j >= Nj) continue;
        double2 U = X[j], V = X[L + j], Wv = X[2 * L + j], E = X[3 * L + j];
        if (conj) { U.y = -U.y; V.y = -V.y; Wv.y = -Wv.y; E.y = -E.y; }
        fx_project<FLUX>(d, w, j, U, V, Wv, E, sc, elapsed, maxSpeed, applyDamping, Ap, Am, A0, Fp, Fm, F0);
    }
}

}  // namespace dev
}  // namespace wvgpu
