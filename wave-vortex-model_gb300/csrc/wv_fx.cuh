// FFTs of FP64 data in 64-bit block fixed point on the integer pipes.
//
// The FP64 pipe of this GPU retires about 1.7 operations per SM and clock
// (measured; 1/64 of the FP32 rate), which bounded every FP64 transform.  The
// integer pipes add 63 64-bit values per SM and clock and run 32 32 x 32 -> 64-bit
// multiplies, so a butterfly costs about 10 times less there.  A line of doubles is
// scaled by one power of two to 64-bit integers, transformed exactly in its sums and
// to one unit in its products, and scaled back.  Flux at 256x256x129: 9.6 -> 2.06 ms.
//
// Range: with B = sum |x_k| over the line (every partial sum of a DFT is at most
// B in magnitude, twiddles having modulus 1), the scale puts B into (2^60, 2^61), a bit
// lower for two rows to a line and another for lane-held products: no sum overflows 63
// bits and no product its accumulator.
// Precision: the unit is 2^-58 to 2^-61 of B; quantisation contributes 0.29 units
// per entry and each twiddle product at most about one.  B / rms and the early
// stages' noise both grow with sqrt(N) on flat lines, so long lines start finer: an
// output of the first s stages is a sum of P_s = R_1 ... R_s entries, at most P_s max|x|,
// and while that is below B the line is held on a scale finer by the difference
// (fx_gap) and shifted down stage by stage: run-time lines past 192 points, and lane-held
// ones of 128 and more whose input is samples (spectra fall off; flat ones of 85 of 256
// entries stay at 1.7e-16).  Errors then stay at 0.5 to 1.6e-16 of the line at every
// length, those of mixed-radix FFTs in doubles at 1.4 to 2.5e-16 (without it 3.3e-16 at 1024).
#pragma once

#include <cstdint>
#ifdef __CUDACC__
#include <cuda_runtime.h>
#endif

#ifdef __CUDACC__
#define WV_HD __host__ __device__ __forceinline__
#define WV_DEV __device__ __forceinline__
#else
#define WV_HD inline
#define WV_DEV inline
#endif

namespace wvgpu {
namespace dev {

struct alignas(16) fxc { long long x, y; };
// Twiddle in Q62, each part as a signed high word and a signed low word
// (value = h 2^32 + l): re_h, re_l, im_h, im_l.
struct alignas(16) fxw { int ch, cl, sh, sl; };

WV_HD fxc fx_add(fxc a, fxc b) { return {a.x + b.x, a.y + b.y}; }
WV_HD fxc fx_sub(fxc a, fxc b) { return {a.x - b.x, a.y - b.y}; }
template <bool INV> WV_HD fxc fx_mul_mi(fxc a) { return INV ? fxc{-a.y, a.x} : fxc{a.y, -a.x}; }

// signed high and low words of x: x = h 2^32 + l, |l| <= 2^31
WV_HD int fx_lo(long long x) { return static_cast<int>(static_cast<unsigned>(x)); }
WV_HD int fx_hi(long long x) {
    return static_cast<int>(x >> 32) + static_cast<int>(static_cast<unsigned>(x) >> 31);
}
// a b + c in one instruction (written out: the compiler otherwise splits most of the
// sums below into products and 64-bit additions, 55 instructions for a complex
// product instead of 26)
WV_HD long long fx_mad(int a, int b, long long c) {
#ifdef __CUDA_ARCH__
    long long r;
    asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
    return r;
#else
    return c + static_cast<long long>(a) * b;
#endif
}
constexpr long long kFxHalf = 1ll << 29;

// x w (INV: x conj w), |x| < 2^61 (1 - 2^-9).  Twelve 32 x 32 -> 64 products: the
// low x low terms (at most one unit) are dropped, the middle ones are rounded to
// the unit and enter the high sum, whose operand carries the factor 4 of Q62.
template <bool INV>
WV_HD fxc fx_cmul(fxc a, fxw w) {
    const int xh = fx_hi(a.x), xl = fx_lo(a.x), yh = fx_hi(a.y), yl = fx_lo(a.y);
    const int nh = -w.sh, nl = -w.sl;
    const int sh = INV ? nh : w.sh, sl = INV ? nl : w.sl, mh = INV ? w.sh : nh, ml = INV ? w.sl : nl;
    long long r = fx_mad(xh, w.cl, kFxHalf), i = fx_mad(xh, sl, kFxHalf);
    r = fx_mad(xl, w.ch, r); i = fx_mad(xl, sh, i);
    r = fx_mad(yh, ml, r);   i = fx_mad(yh, w.cl, i);
    r = fx_mad(yl, mh, r);   i = fx_mad(yl, w.ch, i);
    r >>= 30; i >>= 30;
    const int xh4 = xh * 4, yh4 = yh * 4;
    r = fx_mad(xh4, w.ch, r); i = fx_mad(xh4, sh, i);
    r = fx_mad(yh4, mh, r);   i = fx_mad(yh4, w.ch, i);
    return fxc{r, i};
}
// x w for |x| < 2^60 (1 - 2^-9): the middle terms as four high halves (32-bit sums;
// each cuts half a unit on average, `two` gives it back), 27 instructions against 37.
// two: the value 2 in a register the compiler cannot rebuild (fx_two); 0 on all-zero
// lines, which stay exactly zero.  Twiddles +-1 and +-i (no low words) cut nothing.
template <bool INV>
WV_HD fxc fx_cmul60(fxc a, fxw w, int two) {
    const long long x4 = a.x << 2, y4 = a.y << 2;
    const int xl = fx_lo(x4), yl = fx_lo(y4), xh = fx_hi(x4), yh = fx_hi(y4);
    const int nh = -w.sh, nl = -w.sl;
    const int sih = INV ? nh : w.sh, sil = INV ? nl : w.sl, mh = INV ? w.sh : nh, ml = INV ? w.sl : nl;
#ifdef __CUDA_ARCH__
    auto mad = [](int p, int q, int c) { int r; asm("mad.hi.s32 %0, %1, %2, %3;" : "=r"(r) : "r"(p), "r"(q), "r"(c)); return r; };
    auto mul = [](int p, int q) { long long r; asm("mul.wide.s32 %0, %1, %2;" : "=l"(r) : "r"(p), "r"(q)); return r; };
#else
    auto mad = [](int p, int q, int c) { return static_cast<int>((static_cast<long long>(p) * q) >> 32) + c; };
    auto mul = [](int p, int q) { return static_cast<long long>(p) * q; };
#endif
    const unsigned low = static_cast<unsigned>(w.cl | w.sl);
    const int mean = static_cast<int>(low < static_cast<unsigned>(two) ? low : static_cast<unsigned>(two));
    const int m = mad(xh, w.cl, mad(xl, w.ch, mad(yh, ml, mad(yl, mh, mean))));
    const int n = mad(xh, sil, mad(xl, sih, mad(yh, w.cl, mad(yl, w.ch, mean))));
    return fxc{mul(xh, w.ch) + mul(yh, mh) + static_cast<long long>(m), mul(xh, sih) + mul(yh, w.ch) + static_cast<long long>(n)};
}
#ifdef __CUDACC__
__device__ __forceinline__ int fx_two() {
    int r;
    asm volatile("mov.u32 %0, 2;" : "=r"(r));
    return r;
}
#endif
// x c for a real Q62 constant (h, l)
WV_HD long long fx_rmul(long long x, int ch, int cl) {
    const int xh = fx_hi(x);
    const long long m = fx_mad(fx_lo(x), ch, fx_mad(xh, cl, kFxHalf)) >> 30;
    return fx_mad(xh * 4, ch, m);
}
// high and low words of a Q62 constant
WV_HD constexpr int fx_qh(long long q) { return static_cast<int>((q + 0x80000000ll) >> 32); }
WV_HD constexpr int fx_ql(long long q) { return static_cast<int>(static_cast<unsigned>(q)); }

// R-point DFTs of registers (forward: exp(-2 pi i k n / R); INV: conjugate).
template <bool INV>
WV_HD void fx_dft2(fxc& a, fxc& b) { const fxc t = fx_sub(a, b); a = fx_add(a, b); b = t; }
template <bool INV>
WV_HD void fx_dft4(fxc& v0, fxc& v1, fxc& v2, fxc& v3) {
    const fxc a = fx_add(v0, v2), b = fx_sub(v0, v2), c = fx_add(v1, v3), d = fx_mul_mi<INV>(fx_sub(v1, v3));
    v0 = fx_add(a, c); v1 = fx_add(b, d); v2 = fx_sub(a, c); v3 = fx_sub(b, d);
}
template <bool INV>
WV_HD void fx_dft3(fxc& v0, fxc& v1, fxc& v2) {
    constexpr long long q = 3993837246235628775ll;
    const fxc t = fx_add(v1, v2), e = fx_sub(v1, v2);
    // (the last bit of v0 decides halves: their mean is zero)
    const fxc m = {v0.x - ((t.x + (v0.x & 1)) >> 1), v0.y - ((t.y + (v0.y & 1)) >> 1)};
    const fxc s = {fx_rmul(e.x, fx_qh(q), fx_ql(q)), fx_rmul(e.y, fx_qh(q), fx_ql(q))};
    const fxc i = INV ? fxc{-s.y, s.x} : fxc{s.y, -s.x};  // -/+ i sin(60) (v1 - v2)
    v0 = fx_add(v0, t); v1 = fx_add(m, i); v2 = fx_sub(m, i);
}
template <bool INV>
WV_HD void fx_dft5(fxc& v0, fxc& v1, fxc& v2, fxc& v3, fxc& v4) {
    // cos(72) = (sqrt5 - 1)/4, cos(144) = -(sqrt5 + 1)/4: sums of -1/4 and sqrt5/4
    constexpr long long qd = 2578010857022246787ll;  // sqrt(5)/4
    constexpr long long q1 = 4385974038932618941ll;  // sin 72
    constexpr long long q2 = 2710681029835013083ll;  // sin 144
    const fxc a = fx_add(v1, v4), b = fx_add(v2, v3), c = fx_sub(v1, v4), d = fx_sub(v2, v3);
    const fxc t = fx_add(a, b), u = fx_sub(a, b);
    const fxc du = {fx_rmul(u.x, fx_qh(qd), fx_ql(qd)), fx_rmul(u.y, fx_qh(qd), fx_ql(qd))};
    const fxc m = {v0.x - ((t.x + (v0.x & 3)) >> 2), v0.y - ((t.y + (v0.y & 3)) >> 2)};
    const fxc m1 = fx_add(m, du), m2 = fx_sub(m, du);
    const fxc s1 = {fx_rmul(c.x, fx_qh(q1), fx_ql(q1)) + fx_rmul(d.x, fx_qh(q2), fx_ql(q2)),
                    fx_rmul(c.y, fx_qh(q1), fx_ql(q1)) + fx_rmul(d.y, fx_qh(q2), fx_ql(q2))};
    const fxc s2 = {fx_rmul(c.x, fx_qh(q2), fx_ql(q2)) - fx_rmul(d.x, fx_qh(q1), fx_ql(q1)),
                    fx_rmul(c.y, fx_qh(q2), fx_ql(q2)) - fx_rmul(d.y, fx_qh(q1), fx_ql(q1))};
    const fxc i1 = fx_mul_mi<INV>(s1), i2 = fx_mul_mi<INV>(s2);
    v0 = fx_add(v0, t);
    v1 = fx_add(m1, i1); v4 = fx_sub(m1, i1);
    v2 = fx_add(m2, i2); v3 = fx_sub(m2, i2);
}
template <bool INV>
WV_HD fxc fx_rot8(fxc a) {  // a exp(-/+ i pi/4)
    constexpr long long q = 3260954456333195553ll;
    const long long p = fx_rmul(a.x, fx_qh(q), fx_ql(q)), s = fx_rmul(a.y, fx_qh(q), fx_ql(q));
    return INV ? fxc{p - s, p + s} : fxc{p + s, s - p};
}
template <bool INV>
WV_HD void fx_dft8(fxc (&v)[8]) {
    fx_dft4<INV>(v[0], v[2], v[4], v[6]);
    fx_dft4<INV>(v[1], v[3], v[5], v[7]);
    const fxc o0 = v[1], o1 = fx_rot8<INV>(v[3]), o2 = fx_mul_mi<INV>(v[5]), o3 = fx_mul_mi<INV>(fx_rot8<INV>(v[7]));
    const fxc e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6];
    v[0] = fx_add(e0, o0); v[4] = fx_sub(e0, o0);
    v[1] = fx_add(e1, o1); v[5] = fx_sub(e1, o1);
    v[2] = fx_add(e2, o2); v[6] = fx_sub(e2, o2);
    v[3] = fx_add(e3, o3); v[7] = fx_sub(e3, o3);
}
// 12 = 4 x 3 by coprime index maps (no twiddles): n = 4 n1 + 3 n2, k = 4 k1 + 9 k2 mod 12
template <bool INV>
WV_HD void fx_dft12(fxc (&v)[12]) {
    fx_dft4<INV>(v[0], v[3], v[6], v[9]);
    fx_dft4<INV>(v[4], v[7], v[10], v[1]);
    fx_dft4<INV>(v[8], v[11], v[2], v[5]);
    fx_dft3<INV>(v[0], v[4], v[8]);
    fx_dft3<INV>(v[3], v[7], v[11]);
    fx_dft3<INV>(v[6], v[10], v[2]);
    fx_dft3<INV>(v[9], v[1], v[5]);
    // v[4 n1 + 3 n2] now holds (k1, k2) = (n1, n2), output 4 k1 + 9 k2
    const fxc t3 = v[3], t1 = v[1], t6 = v[6], t7 = v[7], t9 = v[9], t11 = v[11], t5 = v[5], t2 = v[2], t10 = v[10];
    v[9] = t3;              // (0, 1)
    v[6] = t6;              // (0, 2)
    v[3] = t9;              // (0, 3): 27 mod 12
    v[1] = t7;              // (1, 1): 13 mod 12
    v[10] = t10;            // (1, 2): 22 mod 12
    v[7] = t1;              // (1, 3): 31 mod 12
    v[5] = t11;             // (2, 1): 17 mod 12
    v[2] = t2;              // (2, 2): 26 mod 12
    v[11] = t5;             // (2, 3): 35 mod 12
}
template <int R, bool INV>
WV_HD void fx_dft(fxc (&v)[R]) {
    if constexpr (R == 2) fx_dft2<INV>(v[0], v[1]);
    else if constexpr (R == 3) fx_dft3<INV>(v[0], v[1], v[2]);
    else if constexpr (R == 4) fx_dft4<INV>(v[0], v[1], v[2], v[3]);
    else if constexpr (R == 5) fx_dft5<INV>(v[0], v[1], v[2], v[3], v[4]);
    else if constexpr (R == 8) fx_dft8<INV>(v);
    else fx_dft12<INV>(v);
}

// ---- doubles to and from the line's fixed point -----------------------------------

// Words of a double's bits.
WV_HD void fx_words(double v, unsigned& hi, unsigned& lo) {
#ifdef __CUDA_ARCH__
    hi = static_cast<unsigned>(__double2hiint(v));
    lo = static_cast<unsigned>(__double2loint(v));
#else
    uint64_t u;
    __builtin_memcpy(&u, &v, 8);
    hi = static_cast<unsigned>(u >> 32);
    lo = static_cast<unsigned>(u);
#endif
}
WV_HD double fx_double(unsigned long long bits) {
#ifdef __CUDA_ARCH__
    return __longlong_as_double(static_cast<long long>(bits));
#else
    double v;
    __builtin_memcpy(&v, &bits, 8);
    return v;
#endif
}
WV_HD float fx_float(unsigned bits) {
#ifdef __CUDA_ARCH__
    return __uint_as_float(bits);
#else
    float v;
    __builtin_memcpy(&v, &bits, 4);
    return v;
#endif
}
WV_HD unsigned fx_float_bits(float v) {
#ifdef __CUDA_ARCH__
    return __float_as_uint(v);
#else
    unsigned b;
    __builtin_memcpy(&b, &v, 4);
    return b;
#endif
}
// |v| / 2^(e0) as a float from the high word of v (e0: the biased exponent of the
// line's largest high word `top`, so the largest value lies in [1, 2))
WV_HD float fx_rel(unsigned hi, unsigned top) {
    const int r = static_cast<int>(hi & 0x7fffffffu) - static_cast<int>(top & 0x7ff00000u) + (127 << 20);
    return fx_float(static_cast<unsigned>(r > 0 ? r : 0) << 3);
}
// bound of |re + i im|: max + (sqrt2 - 1) min >= the modulus
WV_HD float fx_modulus(float a, float b) { return (a > b ? a : b) + 0.41422f * (a > b ? b : a); }

// |v| as a float from the high word of v: 0 below 2^-126, inf from 2^128 on
WV_HD float fx_mag(unsigned hi) {
    unsigned a = hi & 0x7fffffffu;
    a = a < (896u << 20) ? (896u << 20) : a;
    a = a > (1151u << 20) ? (1151u << 20) : a;
    return fx_float(a * 8u - (896u << 23));
}
// Whether a sum of fx_mag moduli gives a line's scale by itself; lines outside (all
// zero, tiny, huge or non-finite) take their scale from their largest entry.
WV_HD bool fx_plain_sum(float l1) { return l1 > 1e-30f && l1 < 1e30f; }

// Lowest exponent of a scale (2^-919): zeros carry an implied leading bit that has to leave
// through the shift, 61 - bit + e0 >= 63 with bit <= 101.  Lines below lose digits.
constexpr int kFxLowest = 104;
// Scale of a line: the bit position of 2^e0.  l1: the sum of fx_modulus over the
// line (its words were cut after 20 bits, hence the factor).
struct fxscale {
    int e0;   // biased exponent at bit `bit`
    int bit;
    bool zero = false;  // no entry but zeros
    int gap = 0;        // bits by which the line may start finer (fx_gap)
};
WV_HD fxscale fx_scale(unsigned top, float l1) {
    const float s = l1 * 1.0025f;
    int el = static_cast<int>(fx_float_bits(s) >> 23) - 126;  // s < 2^el
    if (el < -40) el = -40;                                   // (weighted rows of one dominant, weightless entry)
    const int e0 = static_cast<int>(top >> 20);
    return {e0 < kFxLowest ? kFxLowest : e0, 61 - el, top == 0};
}
// the same from a sum of fx_mag moduli
WV_HD fxscale fx_scale(float l1) {
    const int el = static_cast<int>(fx_float_bits(l1 * 1.0025f) >> 23) - 126;
    return {1023, 61 - el};
}
// Bits between a line's sum of moduli and `radix` times its largest modulus.
WV_HD int fx_gap(float l1, float most, int radix) {
    const int g = static_cast<int>(fx_float_bits(l1 * 1.0025f) >> 23) - static_cast<int>(fx_float_bits(most * radix * 1.0025f) >> 23);
    return g > 0 ? g : 0;
}
constexpr int kFxAnyGap = 31;  // of an all-zero line, which limits no partner
// m (2^e at bit 62) shifted right by rs + 1 and rounded to nearest, negated if asked.
// Roundings here have mean zero on both signs: a mean of a fraction of a unit, the same
// in every line, would add up in the lowest modes of the passes that follow (0.25 units
// here put 2e-12 instead of 2e-13 on the flux VJP's largest scales at 96x64x49).
WV_HD long long fx_shift_in(unsigned long long m, int rs, int sign) {
    const long long s = sign >> 31;  // 0 or -1; one's complement + 1 is the negative
    return ((static_cast<long long>(m >> (rs > 63 ? 63 : rs)) ^ s) + 1) >> 1;
}
// Half of 2^sh, less one on odd places: (x + fx_half(sh, odd)) >> sh rounds to nearest and
// decides ties up and down in turn.  (A plain shift cuts half a unit, the same in every
// sample of a row, which adds up in the row's mean.)  sh <= 63, |x| < 2^62; 63 gives 0.
WV_HD long long fx_half(int sh, int odd) {
    return static_cast<long long>(((1ull << sh) - static_cast<unsigned long long>(odd)) >> 1);
}
// x 2^-sh at an odd or even place, rounded
WV_HD long long fx_shift_round(long long x, int sh, int odd) { return sh > 0 ? (x + fx_half(sh, odd)) >> sh : x << -sh; }
// v in the line's fixed point (zeros and denormals leave through the shift)
WV_HD long long fx_from_double(double v, fxscale sc) {
    unsigned hi, lo;
    fx_words(v, hi, lo);
    const int e = static_cast<int>((hi >> 20) & 0x7ffu);
    const unsigned long long m = (static_cast<unsigned long long>((hi & 0xfffffu) | 0x100000u) << 32 | lo) << 10;  // 2^e at bit 62
    return fx_shift_in(m, 61 - sc.bit + sc.e0 - e, static_cast<int>(hi));
}
// Exponent of the unit (biased): real value = integer * 2^(unit - 1023).
// kFxBad marks a line that held a non-finite value.
constexpr int kFxBad = 1 << 28;
// unit of an all-zero line (fx_silent); units derived from it stay below half of it
constexpr int kFxZero = -(1 << 24);
WV_HD bool fx_silent(int unit) { return unit < kFxZero / 2; }
WV_HD int fx_unit(fxscale sc) { return sc.zero ? kFxZero : sc.e0 >= 0x7ff ? kFxBad : sc.e0 - sc.bit; }
WV_HD int fx_clz(unsigned v) {
#ifdef __CUDA_ARCH__
    return __clz(static_cast<int>(v));
#else
    return v ? __builtin_clz(v) : 32;
#endif
}
// integer * 2^(unit - 1023) rounded to the nearest double, for a line's unit taken apart
// once.  Units 1 to 1983 (bounds of the line's sum of moduli from 2^-961 to 2^1021) make
// every value a normal double; a line below comes out as zeros, one above as NaN.
struct FxUnit {
    int unit;
    unsigned keep, set;  // masks of the high word: 0 flushes the line, set makes it NaN
};
WV_HD FxUnit fx_out(int unit) {
    const bool huge = unit > 1983, tiny = unit < 1;
    return FxUnit{huge || tiny ? 1000 : unit, tiny ? 0u : 0xffffffffu, huge ? 0x7ff80000u : 0u};
}
WV_HD double fx_to_double(long long x, FxUnit o) {
    unsigned lo = static_cast<unsigned>(x), hi = static_cast<unsigned>(static_cast<unsigned long long>(x) >> 32);
    const unsigned s = static_cast<unsigned>(static_cast<int>(hi) >> 31);
    const unsigned long long a = (static_cast<unsigned long long>(hi ^ s) << 32 | (lo ^ s)) + (s & 1u);
    lo = static_cast<unsigned>(a);
    hi = static_cast<unsigned>(a >> 32);
    int base = o.unit + 62;
    if (hi == 0) { hi = lo; lo = 0; base -= 32; }
    const int lz = fx_clz(hi);
    // leading bit to bit 62, half a unit of the 53 bits added, cut; the hidden bit and a
    // carry past it add to the exponent field
#ifdef __CUDA_ARCH__
    const unsigned long long top = static_cast<unsigned long long>(__funnelshift_l(lo, hi, lz)) << 32 | lo << (lz & 31);
#else
    const unsigned long long top = (static_cast<unsigned long long>(hi) << 32 | lo) << (lz & 31);
#endif
    const unsigned long long m = ((top >> 1) + 512) >> 10;
    unsigned h = static_cast<unsigned>(m >> 32) + (static_cast<unsigned>(base - lz) << 20);
    if (hi == 0) h = 0;
    h = ((h & o.keep) | (s & 0x80000000u)) | o.set;
#ifdef __CUDA_ARCH__
    return __hiloint2double(static_cast<int>(h), static_cast<int>(m));
#else
    return fx_double(static_cast<unsigned long long>(h) << 32 | static_cast<unsigned>(m));
#endif
}
WV_HD double fx_to_double(long long x, int unit) { return fx_to_double(x, fx_out(unit)); }

// ---- lines of 16 to 256 points held by lanes (wv_fxwarp.cuh) ------------------------------

template <int N> struct FxW {
    static constexpr int E = N % 3 == 0 ? 12 : 8;  // points of a lane
    static constexpr int H = E / 2;
    static constexpr int G = N / E;                // lanes of a line
    static constexpr int lines = 32 / G;           // lines of a warp
    static constexpr int samples = lines * N;      // points of a warp: 32 E
    static constexpr int buffer = N + N / 8;       // padded line buffer
    // radices of the stages (their products end with N; R3 = 1: two stages)
    static constexpr int R1 = E == 8 ? 8 : N == 24 ? 2 : 4;
    static constexpr int R2 = E == 8 ? (N == 16 ? 2 : (N == 32 || N == 128) ? 4 : 8) : N == 96 ? 2 : N == 192 ? 4 : 12;
    static constexpr int R3 = N / (R1 * R2);
    static constexpr int twiddles = (R2 - 1) * R1 + (R3 - 1) * R1 * R2;
    // stages before which a line of samples is shifted down (fx_gap), for two rows or
    // channels to a line and for one: as many as keep the error below a double FFT's
    static constexpr int latePair = N == 256 ? 2 : N >= 128 ? 1 : 0;
    static constexpr int lateOne = N == 256 ? 1 : 0;
};
WV_HD int fx_pad(int i) { return i + (i >> 3); }

// Stage of radix R behind Ns points already combined; tw[(r - 1) Ns + k].  SHIFT: the
// inputs come down by sh bits, rounded by the half unit that the stage before added to
// all outputs of a butterfly (on its first input; NEXT: by nextSh bits).  Ties go up and
// down in turn over the butterflies of one k, which the following stages sum.
template <int N, int R, int Ns, bool INV, bool SHIFT, bool NEXT>
WV_HD void fx_wstage(fxc (&v)[FxW<N>::E], const fxw* tw, int t, int two, int sh, int nextSh) {
    constexpr int G = FxW<N>::G, B = FxW<N>::E / R;
#pragma unroll
    for (int b = 0; b < B; ++b) {
        const int j = t + G * b, k = j & (Ns - 1);  // (Ns is a power of two)
        fxc u[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            u[r] = v[b + B * r];
            if (SHIFT) u[r] = fxc{u[r].x >> sh, u[r].y >> sh};
            if (r > 0 && Ns > 1) u[r] = fx_cmul60<INV>(u[r], tw[(r - 1) * Ns + k], two);
        }
        if (NEXT) {
            const long long half = fx_half(nextSh, (j / Ns) & 1);
            u[0] = fxc{u[0].x + half, u[0].y + half};
        }
        fx_dft<R, INV>(u);
#pragma unroll
        for (int r = 0; r < R; ++r) v[b + B * r] = u[r];
    }
}
// v[b + B r], the outputs of a stage of radix R, to their places, and back in lane order
template <int N, int R, int Ns>
WV_HD void fx_wscatter(const fxc (&v)[FxW<N>::E], fxc* x, int t) {
    constexpr int G = FxW<N>::G, B = FxW<N>::E / R;
#pragma unroll
    for (int b = 0; b < B; ++b) {
        const int j = t + G * b, k = j & (Ns - 1), jq = j / Ns;
#pragma unroll
        for (int r = 0; r < R; ++r) x[fx_pad(jq * Ns * R + k + r * Ns)] = v[b + B * r];
    }
}
template <int N>
WV_HD void fx_wgather(fxc (&v)[FxW<N>::E], const fxc* x, int t) {
#pragma unroll
    for (int e = 0; e < FxW<N>::E; ++e) v[e] = x[fx_pad(t + FxW<N>::G * e)];
}
// The whole line (sum of moduli below 2^60, 2^gap times that in the first stage); x: this
// line's buffer, tw: the stage twiddles; LATE: FxW's latePair or lateOne, `gap` its bits.
// each(f): f(v, t) for every lane of the line, a barrier after it (fx_fft_warp; a host
// test walks the lanes).
template <int N, bool INV, int LATE, typename Each>
WV_DEV void fx_line_stages(fxc* x, const fxw* tw, int two, int gap, Each each) {
    using W = FxW<N>;
    constexpr bool three = W::R3 > 1, second = LATE >= 1, third = LATE >= 2 && three;
    constexpr int most2 = W::R2 == 8 ? 3 : W::R2 == 4 ? 2 : W::R2 == 2 ? 1 : 4;  // ceil log2 R2
    const int sh2 = third && gap > most2 ? most2 : gap, sh3 = gap - sh2;
    each([=](fxc (&v)[W::E], int t) {
        fx_wstage<N, W::R1, 1, INV, false, second>(v, tw, t, two, 0, sh2);
        fx_wscatter<N, W::R1, 1>(v, x, t);
    });
    each([=](fxc (&v)[W::E], int t) { fx_wgather<N>(v, x, t); });
    each([=](fxc (&v)[W::E], int t) {
        fx_wstage<N, W::R2, W::R1, INV, second, third>(v, tw, t, two, sh2, sh3);
        if constexpr (three) fx_wscatter<N, W::R2, W::R1>(v, x, t);
    });
    if constexpr (three) {
        each([=](fxc (&v)[W::E], int t) { fx_wgather<N>(v, x, t); });
        each([=](fxc (&v)[W::E], int t) {
            fx_wstage<N, W::R3, W::R1 * W::R2, INV, third, false>(v, tw + (W::R2 - 1) * W::R1, t, two, sh3, 0);
        });
    }
}

// ---- lines of any length, run-time stages -----------------------------------------------

// How far a line is shifted down before a stage: its gap (one for all lines, or one each)
// as far as the stage's span needs it, `before` bits of which went with earlier stages.
struct FxLate {
    const int* gaps;
    int gap, before, after;
    WV_HD int operator()(int line) const {
        const int g = gaps ? gaps[line] : gap;
        return (g < after ? g : after) - (g < before ? g : before);
    }
};
constexpr int kFxLateFrom = 192;       // longer run-time lines of a warp start finer
constexpr int kFxBlockLateFrom = 512;  // of a block: one complex line each, with a bit or two more
WV_HD int fx_ceil_log2(int n) { return n <= 1 ? 0 : 32 - fx_clz(static_cast<unsigned>(n - 1)); }
// One stage over `lines` lines (as fft_stage): radix R from src to dst.  What comes down is
// rounded with ties in turn over the blocks of Ns points, which the stages sum for one k.
template <int R, bool INV, bool LATE>
WV_HD void fx_stage(const fxc* __restrict__ src, fxc* __restrict__ dst, int N, int Ns, int lines, int ld,
                    const fxw* __restrict__ tw, FxLate late, int tid, int nt) {
    const int nb = N / R;
    const int tstride = N / (Ns * R);
    const bool p2 = (N & (N - 1)) == 0;
    const int nbShift = 31 - fx_clz(static_cast<unsigned>(nb)), nsShift = 31 - fx_clz(static_cast<unsigned>(Ns));
    for (int it = tid; it < lines * nb; it += nt) {
        int line, j, k, jq;
        if (p2) {
            line = it >> nbShift; j = it & (nb - 1); k = j & (Ns - 1); jq = j >> nsShift;
        } else {
            line = it / nb; j = it - line * nb; jq = j / Ns; k = j - jq * Ns;
        }
        const fxc* in = src + line * ld + j;
        const int sh = LATE ? late(line) : 0, blocks = LATE ? nb / Ns : 0;
        fxc v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = in[r * nb];
        if (LATE && sh > 0) {
            const long long h[2] = {fx_half(sh, jq & 1), fx_half(sh, (jq + blocks) & 1)};
#pragma unroll
            for (int r = 0; r < R; ++r) v[r] = fxc{(v[r].x + h[r & 1]) >> sh, (v[r].y + h[r & 1]) >> sh};
        }
        if (Ns > 1) {
            const int ts = k * tstride;
#pragma unroll
            for (int r = 1; r < R; ++r) v[r] = fx_cmul<INV>(v[r], tw[r * ts]);
        }
        fx_dft<R, INV>(v);
        fxc* out = dst + line * ld + jq * Ns * R + k;
#pragma unroll
        for (int r = 0; r < R; ++r) out[r * Ns] = v[r];
    }
}
// Any other radix: one output per work item, an O(R) sum.  (fx_shift_lines before it: R
// items read each entry.)
template <bool INV>
WV_HD void fx_stage_any(const fxc* __restrict__ src, fxc* __restrict__ dst, int N, int R, int Ns, int lines, int ld,
                        const fxw* __restrict__ tw, int tid, int nt) {
    const int nb = N / R;
    const int tstride = N / (Ns * R);
    for (int it = tid; it < lines * N; it += nt) {
        const int line = it / N, rem = it - line * N;
        const int j = rem % nb, r = rem / nb;
        const fxc* in = src + line * ld;
        const int k = j % Ns;
        const int step = (k * tstride + r * nb) % N;
        fxc acc = in[j];
        int e = step;
        for (int m = 1; m < R; ++m) {
            acc = fx_add(acc, fx_cmul<INV>(in[j + m * nb], tw[e]));
            e += step;
            if (e >= N) e -= N;
        }
        dst[line * ld + (j / Ns) * Ns * R + k + r * Ns] = acc;
    }
}

struct FxFactors { int N, nstages; const int* radix; };
// Radix of fx_gap; 0: one stage has nothing to come down before.
WV_HD int fx_gap_radix(int nstages, const int* radix) { return nstages > 1 ? radix[0] : 0; }
WV_HD void fx_shift_lines(fxc* lines_, int N, int Ns, int lines, int ld, FxLate late, int tid, int nt) {
    for (int it = tid; it < lines * N; it += nt) {
        const int line = it / N, i = it - line * N;
        const int sh = late(line);
        const long long h = fx_half(sh, (i / Ns) & 1);
        const fxc a = lines_[line * ld + i];
        lines_[line * ld + i] = fxc{(a.x + h) >> sh, (a.y + h) >> sh};
    }
}
WV_HD bool fx_any_radix(int R) { return R != 2 && R != 3 && R != 4 && R != 5 && R != 8; }
// What the lines are shifted down by before stage s > 0, which follows Ns points combined:
// all that is left before the last one (the float sums behind a gap may round it up).
WV_HD FxLate fx_late_of(const FxFactors& f, int s, int Ns, const int* gaps, int gap) {
    return {gaps, gap, fx_ceil_log2(Ns / f.radix[0]), Ns * f.radix[s] == f.N ? kFxAnyGap : fx_ceil_log2(Ns * f.radix[s] / f.radix[0])};
}
// Stage s of the lines, work items tid, tid + nt ...  LATE: lines past kFxLateFrom.
template <bool INV, bool LATE>
WV_HD void fx_run_stage(const fxc* a, fxc* b, const FxFactors& f, int s, int Ns, int lines, int ld, const fxw* tw, const int* gaps,
                        int gap, int tid, int nt) {
    const int R = f.radix[s];
    const FxLate late = LATE && s > 0 ? fx_late_of(f, s, Ns, gaps, gap) : FxLate{nullptr, 0, 0, 0};
    if (R == 8) fx_stage<8, INV, LATE>(a, b, f.N, Ns, lines, ld, tw, late, tid, nt);
    else if (R == 4) fx_stage<4, INV, LATE>(a, b, f.N, Ns, lines, ld, tw, late, tid, nt);
    else if (R == 2) fx_stage<2, INV, LATE>(a, b, f.N, Ns, lines, ld, tw, late, tid, nt);
    else if (R == 3) fx_stage<3, INV, LATE>(a, b, f.N, Ns, lines, ld, tw, late, tid, nt);
    else if (R == 5) fx_stage<5, INV, LATE>(a, b, f.N, Ns, lines, ld, tw, late, tid, nt);
    else fx_stage_any<INV>(a, b, f.N, R, Ns, lines, ld, tw, tid, nt);
}

#ifdef __CUDACC__
// Lines of doubles (re, im) in place to fixed point: one group of warps per line
// sums the moduli, then every entry is scaled.  unit[line] receives fx_unit, gaps[line]
// the bits by which the lines start finer (radix: fx_gap_radix, 0 up to kFxBlockLateFrom).
// Called by all threads of the block.
__device__ inline void fx_quantise(double2* lines_, int N, int lines, int ld, int radix, int* unit, int* gaps) {
    __shared__ unsigned redTop[32];
    __shared__ float redSum[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const int per = lines < warps ? warps / lines : 1;  // warps of one line
    const int groups = warps / per;
    fxc* out = reinterpret_cast<fxc*>(lines_);
    for (int l0 = 0; l0 < lines; l0 += groups) {
        const int g = warp / per, line = l0 + g;
        const bool has = g < groups && line < lines;
        const int t = (warp - g * per) * 32 + lane, step = per * 32;
        const double2* row = lines_ + line * ld;
        auto total = [&](float sum) {  // over the warps of the line
            for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            if (per > 1) {
                if (lane == 0) redSum[warp] = sum;
                __syncthreads();
                if (has) {
                    sum = 0.f;
                    for (int w = 0; w < per; ++w) sum += redSum[g * per + w];
                }
            }
            return sum;
        };
        float sum = 0.f;
        if (has)
            for (int i = t; i < N; i += step) {
                const double2 v = row[i];
                sum += fx_modulus(fx_mag(static_cast<unsigned>(__double2hiint(v.x))),
                                  fx_mag(static_cast<unsigned>(__double2hiint(v.y))));
            }
        sum = total(sum);
        fxscale sc = fx_scale(sum);
        unsigned top = 0;  // of an odd line
        const bool odd = has && !fx_plain_sum(sum);
        if (per > 1 ? __syncthreads_or(odd) : __any_sync(0xffffffffu, odd)) {
            if (has)
                for (int i = t; i < N; i += step) {
                    const double2 v = row[i];
                    top = max(top, max(static_cast<unsigned>(__double2hiint(v.x)) & 0x7fffffffu,
                                       static_cast<unsigned>(__double2hiint(v.y)) & 0x7fffffffu));
                }
            top = __reduce_max_sync(0xffffffffu, top);
            if (per > 1) {
                if (lane == 0) redTop[warp] = top;
                __syncthreads();
                if (has)
                    for (int w = 0; w < per; ++w) top = max(top, redTop[g * per + w]);
            }
            float rel = 0.f;
            if (has)
                for (int i = t; i < N; i += step) {
                    const double2 v = row[i];
                    rel += fx_modulus(fx_rel(static_cast<unsigned>(__double2hiint(v.x)), top),
                                      fx_rel(static_cast<unsigned>(__double2hiint(v.y)), top));
                }
            rel = total(rel);
            if (odd) {
                sc = fx_scale(top, rel);
                sum = rel;
            }
        }
        int gap = 0;
        if (radix > 0) {  // the largest modulus of a long line
            float most = 0.f;
            if (has)
                for (int i = t; i < N; i += step) {
                    const unsigned x = static_cast<unsigned>(__double2hiint(row[i].x)), y = static_cast<unsigned>(__double2hiint(row[i].y));
                    most = fmaxf(most, odd ? fx_modulus(fx_rel(x, top), fx_rel(y, top)) : fx_modulus(fx_mag(x), fx_mag(y)));
                }
            unsigned bits = __reduce_max_sync(0xffffffffu, fx_float_bits(most));
            if (per > 1) {
                __syncthreads();  // (redTop may still be read)
                if (lane == 0) redTop[warp] = bits;
                __syncthreads();
                if (has)
                    for (int w = 0; w < per; ++w) bits = max(bits, redTop[g * per + w]);
                __syncthreads();
            }
            gap = fx_gap(sum, fx_float(bits), radix);
        }
        if (has) {
            if (t == 0) { unit[line] = fx_unit(sc); gaps[line] = gap; }
            sc.bit += gap;
            for (int i = t; i < N; i += step) {
                const double2 v = row[i];
                out[line * ld + i] = fxc{fx_from_double(v.x, sc), fx_from_double(v.y, sc)};
            }
        }
        if (per > 1 && l0 + groups < lines) __syncthreads();  // the partial results are reused
    }
    __syncthreads();
}

// All stages over fixed-point lines; returns the buffer holding the result.  gaps: bits by
// which each line starts finer (null: `gap` for every line); LATE lines of a warp come down
// in the stages, the block's (gaps given) after the first one, at once: its kernels hold
// the stages a single time (twice cost k_xadj a block of an SM: flux VJP 60x50x31 285 ->
// 339 us), and 1024 points end at 1.8e-16.
// WARP: the lines belong to one warp (no block barrier), else to the block.
template <bool INV, bool WARP, bool LATE>
__device__ inline fxc* fx_all_stages(fxc* a, fxc* b, const FxFactors f, int lines, int ld, const fxw* tw, const int* gaps, int gap) {
    const int tid = WARP ? (threadIdx.x & 31) : threadIdx.x, nt = WARP ? 32 : blockDim.x;
    int Ns = 1;
    for (int s = 0; s < f.nstages; ++s) {
        if (WARP && LATE && s > 0 && fx_any_radix(f.radix[s])) {
            fx_shift_lines(a, f.N, Ns, lines, ld, fx_late_of(f, s, Ns, gaps, gap), tid, nt);
            __syncwarp();
        }
        if (!WARP && s == 1 && gaps) {
            fx_shift_lines(a, f.N, Ns, lines, ld, FxLate{gaps, 0, 0, kFxAnyGap}, tid, nt);
            __syncthreads();
        }
        fx_run_stage<INV, LATE>(a, b, f, s, Ns, lines, ld, tw, gaps, gap, tid, nt);
        if (WARP) __syncwarp(); else __syncthreads();
        Ns *= f.radix[s];
        fxc* t = a; a = b; b = t;
    }
    return a;
}
// fft_lines of FP64 lines: scaled, transformed and scaled back in place.
template <bool INV>
__device__ inline double2* fx_fft_lines(double2* a, double2* b, const FxFactors f, int lines, int ld, const fxw* tw) {
    __shared__ int unit[16], gaps[16];
    fx_quantise(a, f.N, lines, ld, f.N > kFxBlockLateFrom ? fx_gap_radix(f.nstages, f.radix) : 0, unit, gaps);
    fxc *fa = reinterpret_cast<fxc*>(a), *fb = reinterpret_cast<fxc*>(b);
    fxc* r = fx_all_stages<INV, false, false>(fa, fb, f, lines, ld, tw, f.N > kFxBlockLateFrom ? gaps : nullptr, 0);
    double2* out = reinterpret_cast<double2*>(r);
    for (int i = threadIdx.x; i < lines * f.N; i += blockDim.x) {
        const int line = i / f.N, k = i - line * f.N, u = unit[line];
        const fxc v = r[line * ld + k];
        out[line * ld + k] = make_double2(fx_to_double(v.x, u), fx_to_double(v.y, u));
    }
    __syncthreads();
    return out;
}
#endif

}  // namespace dev
}  // namespace wvgpu
