// Fixed-point FFT lines (wv_fx.cuh) of 16 to 256 points held by lanes: a line of N
// = E G points (E = 8, or 12 for three times a power of two) belongs to G lanes of
// one warp, lane t holding points t + G e, e < E, before and after the transform; 32 / G
// lines ride in a warp.  The stages (8 x 2, 8 x 4, 8 x 8, 8 x 4 x 4, 8 x 8 x 4; 2 x 12,
// 4 x 12, 4 x 2 x 12, 4 x 4 x 12) work on registers, with one exchange through shared
// memory between two of them (warp barriers only).
//
// What bounds these lines is the number of instructions issued: against the
// run-time Stockham stages of wv_fx.cuh every index is a constant here, the first
// and last stage work on registers, stage twiddles are stored in the order the
// lanes read them, and the line buffers are padded by one entry in eight (no bank
// conflicts on 16-byte accesses).
#pragma once

#include "wv_kernels.cuh"

namespace wvgpu {
namespace dev {

// A line by its lanes (fx_line_stages).
template <int N, bool INV, int LATE = 0>
__device__ __forceinline__ void fx_fft_warp(fxc (&v)[FxW<N>::E], fxc* __restrict__ x, const fxw* __restrict__ tw, int t, int two,
                                            int gap = 0) {
    fx_line_stages<N, INV, LATE>(x, tw, two, gap, [&](auto step) {
        step(v, t);
        __syncwarp();
    });
}

// maxima and sums over the lanes of a line
template <int G>
__device__ __forceinline__ unsigned fx_group_max(unsigned v) {
    if constexpr (G == 32) return __reduce_max_sync(0xffffffffu, v);
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
template <int G>
__device__ __forceinline__ unsigned fx_group_add(unsigned v) {
    if constexpr (G == 32) return __reduce_add_sync(0xffffffffu, v);
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
template <int G>
__device__ __forceinline__ float fx_group_sum(float v) {
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// mantissa (2^e at bit 62) and exponent of a double
__device__ __forceinline__ unsigned long long fx_mantissa(double v, int& e) {
    const unsigned hi = static_cast<unsigned>(__double2hiint(v)), lo = static_cast<unsigned>(__double2loint(v));
    e = static_cast<int>((hi >> 20) & 0x7ffu);
    return (static_cast<unsigned long long>((hi & 0xfffffu) | 0x100000u) << 32 | lo) << 10;
}

// What a line's entries are multiplied by: nothing, real weights w, or i w.
enum FxWeight { kFxPlain, kFxReal, kFxImag };

// High word of the largest k (a full half spectrum ends with a zero weight).
__device__ __forceinline__ unsigned fx_row_k_top(const double* __restrict__ rowK, int KX) {
    return static_cast<unsigned>(max(__double2hiint(rowK[KX - 1]), __double2hiint(rowK[max(KX - 2, 0)])));
}

// How a line's entries become fixed point: shift base less the entry's exponents (less
// `gap` where the line starts finer), and the unit they end with.
struct FxLine { int base, unit, gap; };

// Of the line whose C entries a lane holds, weighted.  count(c): how often entry c enters
// the sum of moduli; spare: bits kept free (1 when two rows share the line); wtop: high
// word of the largest |w|; RADIX: that of the first stage where the line may start finer.
template <int C, int G, FxWeight MODE, int RADIX = 0, int FRAME = 1, typename Count>
__device__ __forceinline__ FxLine fx_line(const double2 (&v)[C], const double (&w)[C], unsigned wtop, int spare, Count count) {
    float sum = 0.f, most = 0.f;
#pragma unroll
    for (int c = 0; c < C; ++c) {
        float m = fx_modulus(fx_mag(static_cast<unsigned>(__double2hiint(v[c].x))),
                             fx_mag(static_cast<unsigned>(__double2hiint(v[c].y))));
        if (MODE != kFxPlain) m *= fx_mag(static_cast<unsigned>(__double2hiint(w[c])));
        sum += count(c) * m;
        if (RADIX) most = fmaxf(most, m);
    }
    sum = fx_group_sum<G>(sum);
    int gap = 0;
    if (RADIX) gap = fx_gap(sum, __uint_as_float(fx_group_max<G>(__float_as_uint(most))), RADIX);
    fxscale sc = fx_scale(sum);
    int wexp = 0;
    bool zero = false;
    const bool odd = !fx_plain_sum(sum);
    if (__any_sync(0xffffffffu, odd)) {
        unsigned top = 0;
#pragma unroll
        for (int c = 0; c < C; ++c)
            top = max(top, max(static_cast<unsigned>(__double2hiint(v[c].x)) & 0x7fffffffu,
                               static_cast<unsigned>(__double2hiint(v[c].y)) & 0x7fffffffu));
        top = fx_group_max<G>(top);
        float rel = 0.f, relMost = 0.f;
#pragma unroll
        for (int c = 0; c < C; ++c) {
            float m = fx_modulus(fx_rel(static_cast<unsigned>(__double2hiint(v[c].x)), top),
                                 fx_rel(static_cast<unsigned>(__double2hiint(v[c].y)), top));
            if (MODE != kFxPlain) m *= fx_rel(static_cast<unsigned>(__double2hiint(w[c])), wtop) * 1.00001f;
            rel += count(c) * m;
            if (RADIX) relMost = fmaxf(relMost, m);
        }
        rel = fx_group_sum<G>(rel);
        if (RADIX) relMost = __uint_as_float(fx_group_max<G>(__float_as_uint(relMost)));
        if (odd) {
            sc = fx_scale(top, rel);
            zero = top == 0 || (MODE != kFxPlain && wtop == 0 && sc.e0 < 0x7ff);
            gap = zero ? kFxAnyGap : RADIX ? fx_gap(rel, relMost, RADIX) : 0;
            if (MODE != kFxPlain) wexp = static_cast<int>((wtop >> 20) & 0x7ffu) - 1023;
        }
    }
    sc.bit -= spare + FRAME;
    return {61 - sc.bit + sc.e0 + (MODE != kFxPlain ? wexp + 1022 : 0),
            zero ? kFxZero : sc.e0 >= 0x7ff ? kFxBad : sc.e0 + wexp - sc.bit, gap};
}
template <int C, FxWeight MODE>
__device__ __forceinline__ void fx_fixed(const double2 (&v)[C], const double (&w)[C], int base, fxc (&out)[C]) {
#pragma unroll
    for (int c = 0; c < C; ++c) {
        int ex, ey;
        unsigned long long mx = fx_mantissa(v[c].x, ex), my = fx_mantissa(v[c].y, ey);
        const int sx = __double2hiint(v[c].x), sy = __double2hiint(v[c].y);
        if constexpr (MODE != kFxPlain) {
            int ew;
            const unsigned long long mw = fx_mantissa(w[c], ew) << 1;
            const int sw = __double2hiint(w[c]);
            mx = __umul64hi(mx, mw);  // 2^(e + ew - 1022) at bit 62
            my = __umul64hi(my, mw);
            const long long wx = fx_shift_in(mx, base - ew - ex, sx ^ sw), wy = fx_shift_in(my, base - ew - ey, sy ^ sw);
            out[c] = MODE == kFxImag ? fxc{-wy, wx} : fxc{wx, wy};
        } else {
            out[c].x = fx_shift_in(mx, base - ex, sx);
            out[c].y = fx_shift_in(my, base - ey, sy);
        }
    }
}
// Both for a line that doesn't start finer.
template <int C, int G, FxWeight MODE, typename Count>
__device__ __forceinline__ void fx_quantise_lane(const double2 (&v)[C], const double (&w)[C], unsigned wtop, int spare, Count count,
                                                 fxc (&out)[C], int& unit) {
    const FxLine l = fx_line<C, G, MODE>(v, w, wtop, spare, count);
    fx_fixed<C, MODE>(v, w, l.base, out);
    unit = l.unit;
}
// Two rows or channels of a line: both start finer by the smaller gap.
__device__ __forceinline__ int fx_shared_gap(int a, int b) { return min(a, b); }

// ---------------------------------------------------------------------------
// x pass of the FP64 flux: c2r of the velocities and of every derivative, the
// quadratic products and their r2c.  Two real rows share one complex line (Z = A + i B
// for the c2r, S_a + i S_b for the r2c); each row keeps its own scale, so its rounding stays
// relative to its own magnitude whatever its partner holds.  Products are formed as
// (a b) >> 62 on velocities normalised to 62 bits and added at the largest unit of
// a target's three.

// (a b) >> 62 rounded, |a| < 2^62, |b| < 2^61
__device__ __forceinline__ long long fx_prod(long long a, long long b) {
    const int ah = fx_hi(a), bh = fx_hi(b);
    const long long m = fx_mad(fx_lo(a), bh, fx_mad(ah, fx_lo(b), kFxHalf)) >> 30;
    return fx_mad(ah, bh * 4, m);
}
// A velocity normalised to 62 bits (leading bit of the row's largest: 61), cut to
// the 53 a double holds: the fields that nonlinearFluxWithAdvectionFields returns
// are then exactly those the flux used, and a flux given them forms the same
// products bit for bit.  (Rounding up past the leading bit would change the
// normalisation: the last step is dropped there.)
__device__ __forceinline__ long long fx_round53(long long v) {
    const long long most = (1ll << 62) - 512;
    const long long r = (v + 256) & ~511ll;
    return r > most ? most : r < -most ? -most : r;
}
__device__ __forceinline__ unsigned fx_abs_hi(long long v) {
    return static_cast<unsigned>(static_cast<unsigned long long>(v < 0 ? -v : v) >> 32);
}
__device__ __forceinline__ int fx_pick(const int (&a)[3], int i) { return i == 0 ? a[0] : i == 1 ? a[1] : a[2]; }

// Rows 2p and 2p + 1 of the x pass (0 u, 1 v, 2 w, then 3 + 3 t + (x, y, z derivative
// of target t)) as the lane's entries of the line Z = A + i B.
template <int N, int EK>
__device__ __forceinline__ void fx_load_pair(const DescDev& d, const double2* __restrict__ yrow, size_t cstride,
                                             const double* __restrict__ rowK, unsigned wtop, int p, int nReal, fxc* __restrict__ x,
                                             int t, fxc (&v)[FxW<N>::E], int (&unit)[2]) {
    constexpr int G = FxW<N>::G, E = FxW<N>::E;
    const int KX = d.kxColumns, nt = d.nt;
    // rows 2p and 2p + 1: spectrum entries k = t + G i, both rows' loads in flight
    double2 raw[2][EK];
    int weighted = 0;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const int r = 2 * p + q;
        int ch = r;
        if (r >= 3) {
            const int tt = (r - 3) / 3, kind = (r - 3) - 3 * tt;
            if (kind == 0) weighted |= 1 << q;
            ch = kind == 0 ? d.tq[tt & 3] : kind == 1 ? 4 + tt : 4 + nt + tt;
        }
        const double2* h = yrow + ch * cstride;
#pragma unroll
        for (int i = 0; i < EK; ++i) {
            const int k = t + G * i;
            raw[q][i] = k < KX && r < nReal ? h[k] : make_double2(0.0, 0.0);
        }
        if (t == 0) raw[q][0].y = 0.0;  // c2r semantics
    }
    fxc A[EK], B[EK];
    auto count = [&](int i) { return i == 0 && t == 0 ? 1.0f : 2.0f; };
#pragma unroll 1
    for (int q = 0; q < 2; ++q) {  // one copy of the code: it must stay in the instruction cache
        double2 a[EK];
        double w[EK];
#pragma unroll
        for (int i = 0; i < EK; ++i) {
            a[i] = q ? raw[1][i] : raw[0][i];
            A[i] = B[i];
        }
        int u;
        if ((weighted >> q) & 1) {
#pragma unroll
            for (int i = 0; i < EK; ++i) w[i] = t + G * i < KX ? rowK[t + G * i] : 0.0;
            fx_quantise_lane<EK, G, kFxImag>(a, w, wtop, 1, count, B, u);
        } else {
            fx_quantise_lane<EK, G, kFxPlain>(a, w, 0u, 1, count, B, u);
        }
        unit[0] = unit[1];
        unit[1] = u;
    }
    // Z = A + i B at k and its mirror at N - k; nothing between
#pragma unroll
    for (int i = 0; i < EK; ++i) {
        const fxc a = A[i], b = B[i];
        v[i] = fxc{a.x - b.y, a.y + b.x};
        const int k = t + G * i;
        const fxc m = {a.x + b.y, b.x - a.y};
        x[fx_pad(k == 0 ? N - G * EK : N - k)] = k == 0 ? fxc{0, 0} : m;
    }
#pragma unroll
    for (int e = EK; e < E - EK; ++e) v[e] = fxc{0, 0};
    __syncwarp();
#pragma unroll
    for (int e = E - EK; e < E; ++e) v[e] = x[fx_pad(t + G * e)];
    __syncwarp();
}

// Scale of a caller's velocity row, largest high word `top`: its leading bit at 61.
__device__ __forceinline__ fxscale fx_velocity_scale(unsigned top) { return {max(static_cast<int>(top >> 20), kFxLowest), 61, top == 0}; }

// Samples of an advecting velocity row (or the caller's doubles), normalised to 62
// bits, into phys; returns the unit.
template <int N>
__device__ __forceinline__ int fx_velocity(const long long (&smp)[FxW<N>::E], int unit, int t, long long* __restrict__ phys,
                                           const double* __restrict__ advIn, double* __restrict__ advOut,
                                           double* __restrict__ keep) {
    constexpr int G = FxW<N>::G, E = FxW<N>::E;
    unsigned top = 0;
    if (advIn) {
        double a[E];
#pragma unroll
        for (int e = 0; e < E; ++e) {
            a[e] = advIn[t + G * e];
            top = max(top, static_cast<unsigned>(__double2hiint(a[e])) & 0x7fffffffu);
        }
        top = fx_group_max<G>(top);
        const fxscale sc = fx_velocity_scale(top);
#pragma unroll
        for (int e = 0; e < E; ++e) {
            phys[t + G * e] = fx_from_double(a[e], sc);
            if (keep) keep[t + G * e] = a[e];
        }
        return fx_unit(sc);
    }
#pragma unroll
    for (int e = 0; e < E; ++e) top = max(top, fx_abs_hi(smp[e]));
    top = fx_group_max<G>(top);
    const int sh = max(0, __clz(static_cast<int>(top)) - 2);
    const FxUnit o = fx_out(unit - sh);
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const long long s = fx_round53(smp[e] << sh);
        phys[t + G * e] = s;
        if (advOut) advOut[t + G * e] = fx_to_double(s, o);
        if (keep) keep[t + G * e] = fx_to_double(s, o);
    }
    return unit - sh;
}

// r2c of the products Sa, Sb (Sb null: none) of a row as one line; out[k], k < KX, and
// out[cstride + k].
template <int N>
__device__ __forceinline__ void fx_forward_pair(const long long* __restrict__ Sa, const long long* __restrict__ Sb, int unitA,
                                                int unitB, fxc* __restrict__ x, const fxw* __restrict__ tw, int t, int two,
                                                int KX, double2* __restrict__ out, size_t cstride) {
    constexpr int G = FxW<N>::G, E = FxW<N>::E, H = E / 2;
    using W = FxW<N>;
    const bool both = Sb != nullptr;
    fxc v[E];
    int sh[2], u[2], gap = kFxAnyGap;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        unsigned sum = 0, most = 0;
        if (q == 0 || both)
#pragma unroll
            for (int e = 0; e < E; ++e) {
                const unsigned m = (fx_abs_hi((q ? Sb : Sa)[t + G * e]) >> 9) + 1u;
                sum += m;
                if (W::latePair) most = max(most, m);
            }
        sum = fx_group_add<G>(sum);
        const int bits = 32 - __clz(static_cast<int>(sum));
        sh[q] = 41 + bits - 59;                  // sum |S| < 2^59 after the shift
        u[q] = (q ? unitB : unitA) + sh[q] - 1;  // the halves of the split below
        if (W::latePair && (q == 0 || both))
            gap = fx_shared_gap(gap, max(0, bits - (32 - __clz(static_cast<int>(fx_group_max<G>(most) * W::R1)))));
    }
    if (!W::latePair) gap = 0;
    sh[0] -= gap;
    sh[1] -= gap;
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const long long a = Sa[t + G * e], b = both ? Sb[t + G * e] : 0;
        v[e].x = fx_shift_round(a, sh[0], t & 1);
        v[e].y = fx_shift_round(b, sh[1], t & 1);
    }
    fx_fft_warp<N, false, W::latePair>(v, x, tw, t, fx_silent(max(unitA, both ? unitB : unitA)) ? 0 : two, gap);
    __syncwarp();
#pragma unroll
    for (int e = H; e < E; ++e) x[fx_pad(t + G * e)] = v[e];
    __syncwarp();
    const FxUnit o0 = fx_out(u[0]), o1 = fx_out(u[1]);
#pragma unroll
    for (int i = 0; i < H; ++i) {
        const int k = t + G * i;
        const fxc a = v[i], b = k == 0 ? v[0] : x[fx_pad(N - k)];
        if (k < KX) {
            out[k] = make_double2(fx_to_double(a.x + b.x, o0), fx_to_double(a.y - b.y, o0));
            if (both) out[cstride + k] = make_double2(fx_to_double(a.y + b.y, o1), fx_to_double(b.x - a.x, o1));
        }
    }
}

// The x pass: a block takes one line-set of rows, a warp a pair of their c2r, all threads
// a sample's products, a warp a pair of the r2c.  A warp holds one pair of rows at a
// time, so three blocks fit an SM.  (A warp per row with all its transforms in registers
// gained 2 to 4 % on 12 to 40 line-sets an SM of 16 or 128 points and lost 4 to 7 % on
// more, 10 to 30 % on fewer: flux 128x128x65 290 against 295 us, 128x256x129 1137 against
// 1064, 128x64x33 133 against 109.)  256x256x129: 5.92 (FP64 pipe) -> 1.07 ms, 53 % of
// the issue slots; 192x192x97 1.00 -> 0.55 ms (run-time stages -> lanes).
// physOut / advOut / advIn / maxSpeedBits as k_xflux.
// EK: spectrum entries of a lane (kx < EK G; E / 2 at most, fewer under the 2/3 rule).
// How a product comes to its target's unit: (p + half) >> shift (fx_half).
struct alignas(16) FxAlign { long long half; int shift; };
constexpr int kFxCoWarps = 8;  // (3 + 3 nt + 1) / 2 <= 8 pairs
template <int N>
inline size_t smem_xflux_co() { return (FxW<N>::twiddles + kFxCoWarps * FxW<N>::lines * FxW<N>::buffer) * 16 + (3 + 4) * FxW<N>::samples * 8; }

template <int N, int EK>
__global__ void __launch_bounds__(32 * kFxCoWarps, FxW<N>::E == 8 ? 3 : 2)
    k_xflux_fxco(DescDev d, const fxw* __restrict__ twg, const double2* __restrict__ yspec, double2* __restrict__ pspec,
                 unsigned long long* __restrict__ maxSpeedBits, double* __restrict__ physOut, double* __restrict__ advOut,
                 const double* __restrict__ advIn) {
    using W = FxW<N>;
    constexpr int G = W::G, E = W::E;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int rowUnit[16][W::lines], sUnit[4][W::lines];
    __shared__ FxAlign align[2][12][W::lines];  // [odd sample][target, kind][line]
    const int Ny = d.Ny, KX = d.kxColumns, nt = d.nt;
    const int nIn = 4 + 2 * nt, nReal = 3 + 3 * nt;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int t = lane % G, line = lane / G;
    fxw* tw = reinterpret_cast<fxw*>(smem_raw);
    fxc* buffers = reinterpret_cast<fxc*>(tw + W::twiddles);  // [pair][line][buffer]
    fxc* x = buffers + static_cast<size_t>(warp * W::lines + line) * W::buffer;
    long long* phys = reinterpret_cast<long long*>(buffers + kFxCoWarps * W::lines * W::buffer);  // [3][line][N]
    long long* S = phys + 3 * W::samples;                                                               // [nt][line][N]
    const int two = fx_two();
    for (int i = threadIdx.x; i < W::twiddles; i += blockDim.x) tw[i] = twg[i];
    const double* rowK = row_k<double>(d);
    const size_t cstride = static_cast<size_t>(Ny) * KX;
    const size_t R3 = static_cast<size_t>(N) * Ny * d.Nz;
    const int rows = Ny * d.zTotal;
    const unsigned wtop = fx_row_k_top(rowK, KX);
    const int first = blockIdx.x * W::lines;
    const bool live = first + line < rows;
    const int row = min(first + line, rows - 1);
    const int z = row / Ny, y = row - z * Ny;
    const int p = warp;
    __syncthreads();
    if (2 * p < nReal) {
        fxc v[E];
        int unit[2] = {kFxZero, kFxZero};
        fx_load_pair<N, EK>(d, yspec + (static_cast<size_t>(z) * nIn * Ny + y) * KX, cstride, rowK, wtop, p, nReal, x, t, v, unit);
        fx_fft_warp<N, true>(v, x, tw, t, fx_silent(max(unit[0], unit[1])) ? 0 : two);
#pragma unroll
        for (int e = 0; e < E; ++e) x[t + G * e] = v[e];
#pragma unroll 1
        for (int q = 0; q < 2; ++q) {
            const int r = 2 * p + q;
            if (r >= nReal) break;
            int uq = q ? unit[1] : unit[0];
            double* keep = physOut && live ? physOut + ((static_cast<size_t>(z) * nReal + r) * Ny + y) * N : nullptr;
            long long smp[E];
#pragma unroll
            for (int e = 0; e < E; ++e) smp[e] = q ? v[e].y : v[e].x;
            if (r < 3) {
                const size_t g = static_cast<size_t>(r) * R3 + (static_cast<size_t>(z) * Ny + y) * N;
                uq = fx_velocity<N>(smp, uq, t, phys + (r * W::lines + line) * N, advIn ? advIn + g : nullptr,
                                    advOut && live ? advOut + g : nullptr, keep);
            } else if (keep) {
                const FxUnit o = fx_out(uq);
#pragma unroll
                for (int e = 0; e < E; ++e) keep[t + G * e] = fx_to_double(smp[e], o);
            }
            if (t == 0) rowUnit[r][line] = uq;
        }
    }
    __syncthreads();
    // a target's products are added at the largest unit of its three
    for (int i = threadIdx.x; i < 2 * nt * W::lines; i += 32 * kFxCoWarps) {
        const int ln = i % W::lines, odd = (i / W::lines) & 1, tt = i / (2 * W::lines);
        int un[3];
#pragma unroll
        for (int kind = 0; kind < 3; ++kind) un[kind] = rowUnit[kind][ln] + rowUnit[3 + 3 * tt + kind][ln] - 1023 + 62;
        const int most = max(un[0], max(un[1], un[2]));
#pragma unroll
        for (int kind = 0; kind < 3; ++kind) {
            const int sh = min(63, most - un[kind]);
            align[odd][3 * tt + kind][ln] = FxAlign{fx_half(sh, odd), sh};
        }
        if (odd == 0) sUnit[tt][ln] = most;
    }
    __syncthreads();
    // a sample a thread
    for (int s = threadIdx.x; s < W::samples; s += 32 * kFxCoWarps) {
        const int ln = s / N, xx = s - ln * N;
        for (int tt = 0; tt < nt; ++tt) {
            long long acc = 0;
#pragma unroll
            for (int kind = 0; kind < 3; ++kind) {
                const int r = 3 + 3 * tt + kind;
                const fxc* b = buffers + static_cast<size_t>((r >> 1) * W::lines + ln) * W::buffer;
                const long long q = (r & 1) ? b[xx].y : b[xx].x;
                const FxAlign a = align[s & 1][r - 3][ln];
                acc -= (fx_prod(phys[kind * W::samples + s], q) + a.half) >> a.shift;
            }
            S[tt * W::samples + s] = acc;
        }
        if (maxSpeedBits) {
            const double U = fx_to_double(phys[s], rowUnit[0][ln]), V = fx_to_double(phys[W::samples + s], rowUnit[1][ln]);
            double m = U * U + V * V;
            // samples of one row among a warp's 32: the power of two that divides N
            constexpr int kSpan = (N & -N) < 32 ? (N & -N) : 32;
#pragma unroll
            for (int o = kSpan / 2; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
            m = fmax(m, 0.0);
            const int zz = min(first + ln, rows - 1) / Ny;
            if (lane % kSpan == 0) atomicMax(maxSpeedBits + zz / d.Nz, (unsigned long long)__double_as_longlong(sqrt(m)));
        }
    }
    __syncthreads();
    if (2 * p < nt) {
        const bool both = 2 * p + 1 < nt;
        const long long* Sa = S + 2 * p * W::samples + line * N;
        fx_forward_pair<N>(Sa, both ? Sa + W::samples : nullptr, sUnit[2 * p][line], both ? sUnit[2 * p + 1][line] : 0, x, tw, t, two,
                           live ? KX : 0, pspec + ((static_cast<size_t>(z) * nt + 2 * p) * Ny + y) * KX, cstride);
    }
}

}  // namespace dev
}  // namespace wvgpu
