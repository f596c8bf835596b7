// The flux VJP of FP64 handles on lane-held fixed-point lines (wv_fxwarp.cuh): the
// transposed passes of wv_adjoint.cuh and wv_vfft.cuh for lengths of 16 to 256.
#pragma once

#include "wv_fxyz.cuh"

namespace wvgpu {
namespace dev {

// Cotangents of the transformed channels u, v, w, eta of one (mode, j)
// (vfwd_adj_values' formulas: the map of fx_project transposed).
__device__ __forceinline__ void fx_vfwd_adj_values(const DescDev& d, const double* __restrict__ Fpb,
                                                   const double* __restrict__ Fmb, const double* __restrict__ F0b,
                                                   double elapsed, int w, int j, double2 (&f)[4]) {
    const int idx = j + d.Nj * w;
    double c, s;
    fx_phase(d.omega[idx] * elapsed, d.fxPhase, c, s);
    const zd fp = zload(Fpb + 2 * idx), fm = zload(Fmb + 2 * idx), a0 = zload(F0b + 2 * idx);
    const zd cp{fp.re * c - fp.im * s, fp.re * s + fp.im * c};  // Fp_bar p
    const zd cm{fm.re * c + fm.im * s, fm.im * c - fm.re * s};  // Fm_bar conj(p)
    const double buoy = d.A0FromBuoyancy[idx];
    if (w == 0) {
        const double is = d.inertialScale[j];
        const double tr = cp.re + cm.re, ti = cp.im - cm.im;
        f[0] = make_double2(is * tr, is * ti);
        f[1] = make_double2(-is * ti, is * tr);
        f[2] = make_double2(0.0, 0.0);
        f[3] = make_double2(buoy * a0.re, buoy * a0.im);
        return;
    }
    const double apmn = d.ApmN[idx], na0 = d.NA0[idx];
    const double wr = cp.re + cm.re, wi = cp.im + cm.im;
    const double br = (cp.re - cm.re) * apmn, bi = (cp.im - cm.im) * apmn;
    const double ar = a0.re - na0 * br, ai = a0.im - na0 * bi;
    const double vort = d.A0FromVorticity[idx];
    const double lv = d.l[w] * vort, kv = d.k[w] * vort;
    double cu, cv, h;
    if (d.hydrostatic) {
        const double g = -d.ApmD[2 * idx + 1];
        cu = d.k[w] * g; cv = d.l[w] * g; h = 0.0;
    } else {
        const double g = d.ApmDScaled[idx];
        cu = d.cosAlpha[w] * g; cv = d.sinAlpha[w] * g; h = (d.Kh[w] / 2.0) * d.apmWPrefactor[j];
    }
    f[0] = make_double2(cu * wr - lv * ai, cu * wi + lv * ar);
    f[1] = make_double2(cv * wr + kv * ai, cv * wi - kv * ar);
    f[2] = make_double2(h * wi, -h * wr);
    f[3] = make_double2(br + buoy * ar, bi + buoy * ai);
}

// vinv_adj_store with the factors' structure used (fx_field_spectra transposed).
__device__ __forceinline__ void fx_vinv_adj_store(const DescDev& d, int idx, double elapsed, double2 ub, double2 vb, double2 wb,
                                                  double2 nb, double* __restrict__ Apb, double* __restrict__ Amb,
                                                  double* __restrict__ A0b) {
    const zd uap = zload(d.UAp + 2 * idx), vap = zload(d.VAp + 2 * idx);
    const double wi = d.WAp[2 * idx + 1], u0 = d.UA0[2 * idx + 1], v0 = d.VA0[2 * idx + 1];
    const double nap = d.NAp[idx], na0 = d.NA0[idx];
    const double pr = uap.re * ub.x + vap.re * vb.x, pi = uap.re * ub.y + vap.re * vb.y;
    const double qr = uap.im * ub.x + vap.im * vb.x, qi = uap.im * ub.y + vap.im * vb.y;
    const double wr = wi * wb.y, wim = -wi * wb.x;
    const zd ape{pr + qi + wr + nap * nb.x, pi - qr + wim + nap * nb.y};
    const zd ame{pr - qi + wr - nap * nb.x, pi + qr + wim - nap * nb.y};
    double c, s;
    fx_phase(d.omega[idx] * elapsed, d.fxPhase, c, s);
    zstore(Apb + 2 * idx, zd{ape.re * c + ape.im * s, ape.im * c - ape.re * s});  // ape conj(p)
    zstore(Amb + 2 * idx, zd{ame.re * c - ame.im * s, ame.re * s + ame.im * c});  // ame p
    zstore(A0b + 2 * idx, zd{u0 * ub.y + v0 * vb.y + na0 * nb.x, -u0 * ub.x - v0 * vb.x + na0 * nb.y});
}

// The VJP's four kernels, 128x128x65: 2.06 ms on the FP64 pipe (forward fields
// included) -> 0.66 ms; all bound by integer issue.
//
// k_vfwd_adj_fft: lines (u | w), (v | eta) of a column by two warps;
// y[0] = X_0, y[j] = (X_j + i Y_j) / 2, y[N-j] = (X_j - i Y_j) / 2.
template <int N>
__global__ void __launch_bounds__(32 * kFxZWarps, FxW<N>::E == 8 ? 3 : 2)
    k_vfwd_adj_fx(DescDev d, const double* __restrict__ Fpb, const double* __restrict__ Fmb, const double* __restrict__ F0b,
                  double elapsed, double2* __restrict__ zadj) {
    using W = FxW<N>;
    constexpr int G = W::G, E = W::E, H = W::H, L = N / 2;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int Nj = d.Nj, P = d.positions;
    const int lane = threadIdx.x & 31, t = lane % G, warp = threadIdx.x >> 5;
    const int set = warp >> 1, l = warp & 1, sets = blockDim.x >> 6;
    fxw* tw = reinterpret_cast<fxw*>(smem_raw);
    const int column = set * W::lines + lane / G;
    fxc* x = reinterpret_cast<fxc*>(tw + W::twiddles) + static_cast<size_t>(column * 2 + l) * W::buffer;
    double2* fld = reinterpret_cast<double2*>(reinterpret_cast<fxc*>(tw + W::twiddles) +
                                              static_cast<size_t>(sets) * W::lines * 2 * W::buffer) +
                   static_cast<size_t>(column) * 2 * N;  // [4][N/2]
    for (int i = threadIdx.x; i < W::twiddles; i += blockDim.x) tw[i] = d.fxTwZ[i];
    const int want = blockIdx.x * sets * W::lines + column;
    const bool live = want < d.Nkl;
    const int mode = min(want, d.Nkl - 1);
#pragma unroll 1
    for (int i = l; i < H; i += 2) {
        const int j = t + G * i;
        double2 f[4];
        if (j < Nj) fx_vfwd_adj_values(d, Fpb, Fmb, F0b, elapsed, d.modeWV[mode], j, f);
#pragma unroll
        for (int q = 0; q < 4; ++q) fld[q * L + j] = j < Nj ? f[q] : make_double2(0.0, 0.0);
    }
    __syncthreads();
    int tc = -1, ts = -1;  // targets of the cosine slot l and the sine slot 2 + l
    for (int q = 0; q < d.nt; ++q) {
        if (d.tq[q] == l) tc = q;
        if (d.tq[q] == 2 + l) ts = q;
    }
    double2 a[H];
    double none[H];
    fxc C[H], D[H];
    int uC, uD;
#pragma unroll
    for (int i = 0; i < H; ++i) a[i] = tc >= 0 ? fld[l * L + t + G * i] : make_double2(0.0, 0.0);
    fx_quantise_lane<H, G, kFxPlain>(a, none, 0u, 1, [](int) { return 2.0f; }, C, uC);
#pragma unroll
    for (int i = 0; i < H; ++i) a[i] = ts >= 0 ? fld[(2 + l) * L + t + G * i] : make_double2(0.0, 0.0);
    fx_quantise_lane<H, G, kFxPlain>(a, none, 0u, 1, [](int) { return 2.0f; }, D, uD);
    fxc v[E];
#pragma unroll
    for (int i = 0; i < H; ++i) {  // 2 y
        const int j = t + G * i;
        if (j == 0) {
            v[i] = fxc{2 * C[i].x, 2 * C[i].y};
            x[fx_pad(L)] = fxc{0, 0};
        } else {
            v[i] = fxc{C[i].x - D[i].y, C[i].y + D[i].x};
            x[fx_pad(N - j)] = fxc{C[i].x + D[i].y, C[i].y - D[i].x};
        }
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
    const double sc = 1.0 / (static_cast<double>(L) * static_cast<double>(d.Nx) * static_cast<double>(d.Ny));
    const int pos = d.modePos[mode], cpos = d.modeCompPos[mode];
    const double sign = (d.modeFlags[mode] & 1) ? -sc : sc;
    const FxUnit oC = fx_out(uC - 1), oC0 = fx_out(uC - 2), oD = fx_out(uD - 1);
    auto put = [&](int n, fxc a1, fxc b1, const FxUnit& o) {
        if (tc >= 0) {
            double2* base = zadj + (static_cast<size_t>(tc) * d.Nz + n) * P;
            base[pos] = make_double2(fx_to_double(a1.x + b1.x, o) * sc, fx_to_double(a1.y + b1.y, o) * sign);
            if (cpos >= 0) base[cpos] = make_double2(0.0, 0.0);
        }
        if (ts >= 0) {
            double2* base = zadj + (static_cast<size_t>(ts) * d.Nz + n) * P;
            base[pos] = make_double2(fx_to_double(a1.x - b1.x, oD) * sc, fx_to_double(a1.y - b1.y, oD) * sign);
            if (cpos >= 0) base[cpos] = make_double2(0.0, 0.0);
        }
    };
#pragma unroll
    for (int i = 0; i < H; ++i) {
        const int n = t + G * i;
        put(n, v[i], n == 0 ? v[0] : x[fx_pad(N - n)], n == 0 ? oC0 : oC);  // w_z = 1 at the ends, 2 inside
    }
    if (t == 0) put(L, v[H], v[H], oC0);
}

// Shared memory of k_vinv_adj_fx: line buffers and the parts [8][N/2] of each column.
template <int N>
inline size_t smem_fx_vinv_adj(int sets) {
    const size_t columns = static_cast<size_t>(sets) * FxW<N>::lines;
    return (FxW<N>::twiddles + columns * (4 * FxW<N>::buffer + 4 * N)) * 16;
}
// k_vinv_adj_fft: the four lines of a column by four warps, which then share its
// coefficients; y[0] = o_0, y[L] = o_L, y[z] = (o_z + i s_z) / 2, y[N-z] = (o_z - i s_z) / 2.
template <int N>
__global__ void __launch_bounds__(32 * kFxZWarps, 2)
    k_vinv_adj_fx(DescDev d, const double2* __restrict__ fadj, double elapsed, double* __restrict__ Apb,
                  double* __restrict__ Amb, double* __restrict__ A0b) {
    using W = FxW<N>;
    constexpr int G = W::G, E = W::E, H = W::H, L = N / 2;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int Nj = d.Nj, Nz = d.Nz, P = d.positions;
    const int lane = threadIdx.x & 31, t = lane % G, warp = threadIdx.x >> 5;
    const int set = warp >> 2, l = warp & 3, sets = blockDim.x >> 7;
    fxw* tw = reinterpret_cast<fxw*>(smem_raw);
    const int column = set * W::lines + lane / G;
    fxc* x = reinterpret_cast<fxc*>(tw + W::twiddles) + static_cast<size_t>(column * 4 + l) * W::buffer;
    double2* X = reinterpret_cast<double2*>(reinterpret_cast<fxc*>(tw + W::twiddles) +
                                            static_cast<size_t>(sets) * W::lines * 4 * W::buffer) +
                 static_cast<size_t>(column) * 4 * N;  // [line][even | odd][N/2]
    for (int i = threadIdx.x; i < W::twiddles; i += blockDim.x) tw[i] = d.fxTwZ[i];
    const int want = blockIdx.x * sets * W::lines + column;
    const bool live = want < d.Nkl;
    const int mode = min(want, d.Nkl - 1);
    int derivC = -1, derivS = -1;
    for (int q = 0; q < d.nt; ++q) {
        if (d.tq[q] == l) derivC = 4 + q;
        if (d.tq[q] == l - 2) derivS = 4 + q;
    }
    const int chC = l < 2 ? l : derivC, chS = l < 2 ? l + 2 : derivS;
    {
        const int pos = d.modePos[mode], cpos = d.modeCompPos[mode];
        const unsigned char flags = d.modeFlags[mode];
        // stored row + conjugated completion row, in the frame of k_vinv
        auto colval = [&](int ch, int z) {
            const double2* r = fadj + (static_cast<size_t>(ch) * Nz + z) * P;
            double2 v = r[pos];
            if (cpos >= 0) { const double2 c = r[cpos]; v = make_double2(v.x + c.x, v.y - c.y); }
            if (flags & 2) v.y = 0.0;
            if (flags & 1) v.y = -v.y;
            return v;
        };
        double2 a[H + 1], b[H];
        double none5[H + 1], none4[H];
#pragma unroll
        for (int i = 0; i < H + 1; ++i) {
            const int z = t + G * i;
            a[i] = chC >= 0 && (i < H || t == 0) ? colval(chC, z) : make_double2(0.0, 0.0);
            if (i < H) b[i] = chS >= 0 && z != 0 ? colval(chS, z) : make_double2(0.0, 0.0);
        }
        fxc C[H + 1], S[H];
        constexpr int radix = W::latePair ? W::R1 : 0;
        auto twice = [](int) { return 2.0f; };
        const FxLine lC = fx_line<H + 1, G, kFxPlain, radix>(a, none5, 0u, 1, twice), lS = fx_line<H, G, kFxPlain, radix>(b, none4, 0u, 1, twice);
        const int gap = fx_shared_gap(lC.gap, lS.gap), uC = lC.unit, uS = lS.unit;
        fx_fixed<H + 1, kFxPlain>(a, none5, lC.base - gap, C);
        fx_fixed<H, kFxPlain>(b, none4, lS.base - gap, S);
        __syncthreads();  // twiddles
        fxc v[E];
#pragma unroll
        for (int i = 0; i < H; ++i) {  // 2 y
            const int z = t + G * i;
            if (z == 0) {
                v[i] = fxc{2 * C[i].x, 2 * C[i].y};
                x[fx_pad(L)] = fxc{2 * C[H].x, 2 * C[H].y};
            } else {
                v[i] = fxc{C[i].x - S[i].y, C[i].y + S[i].x};
                x[fx_pad(N - z)] = fxc{C[i].x + S[i].y, C[i].y - S[i].x};
            }
        }
        __syncwarp();
#pragma unroll
        for (int e = H; e < E; ++e) v[e] = x[fx_pad(t + G * e)];
        __syncwarp();
        fx_fft_warp<N, false, W::latePair>(v, x, tw, t, fx_silent(max(uC, uS)) ? 0 : fx_two(), gap);
#pragma unroll
        for (int e = H; e < E; ++e) x[fx_pad(t + G * e)] = v[e];
        __syncwarp();
        const FxUnit oC = fx_out(uC - 2), oC0 = fx_out(uC - 3), oS = fx_out(uS - 2);
#pragma unroll
        for (int i = 0; i < H; ++i) {
            const int j = t + G * i;
            if (j >= Nj) continue;
            const fxc p = v[i], q = j == 0 ? v[0] : x[fx_pad(N - j)];
            const FxUnit& o = j == 0 ? oC0 : oC;  // Ccos's 1/2 at j = 0
            X[2 * l * L + j] = make_double2(fx_to_double(p.x + q.x, o), fx_to_double(p.y + q.y, o));
            X[(2 * l + 1) * L + j] = make_double2(fx_to_double(p.x - q.x, oS), fx_to_double(p.y - q.y, oS));
        }
    }
    __syncthreads();
    if (!live) return;
#pragma unroll 1
    for (int i = l; i < H; i += 4) {
        const int j = t + G * i;
        if (j >= Nj) continue;
        const double m = static_cast<const double*>(d.tMz)[j];
        // u_bar = Ccos^T U + (-m) Csin^T u_z;  w_bar = Csin^T W + m Ccos^T w_z; likewise v, eta
        const double2 e0 = X[j], o0 = X[L + j], e1 = X[2 * L + j], o1 = X[3 * L + j];
        const double2 e2 = X[4 * L + j], o2 = X[5 * L + j], e3 = X[6 * L + j], o3 = X[7 * L + j];
        fx_vinv_adj_store(d, j + Nj * d.modeWV[mode], elapsed, make_double2(e0.x - m * o2.x, e0.y - m * o2.y),
                          make_double2(e1.x - m * o3.x, e1.y - m * o3.y), make_double2(o0.x + m * e2.x, o0.y + m * e2.y),
                          make_double2(o1.x + m * e3.x, o1.y + m * e3.y), Apb, Amb, A0b);
    }
}

// k_yfwd_pair: FFT_y(srcA) + (-i l) FFT_y(srcB), gathered to the active rows.
template <int N>
__global__ void __launch_bounds__(32 * kFxYWarps, 2)
    k_yfwd_pair_fx(DescDev d, YFwdPairMap map, const double2* __restrict__ yin, int nIn, double2* __restrict__ fout) {
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
    const int g = min(cols, KX - kx0);
    const double* rowL = row_l<double>(d);
    double2 sum[E];
#pragma unroll
    for (int e = 0; e < E; ++e) sum[e] = make_double2(0.0, 0.0);
#pragma unroll 1
    for (int part = 0; part < 2; ++part) {
        const int src = part == 0 ? map.srcA[ch] : map.srcB[ch];
        if (src < 0) break;  // (the block's: every thread leaves)
        const double2* in = yin + (static_cast<size_t>(z) * nIn + src) * N * KX + kx0;
        for (int i = threadIdx.x; i < N * cols; i += blockDim.x) {
            const int y = i / cols, c = i - y * cols;
            tile[fx_tile(y, c, cols)] = c < g ? in[static_cast<size_t>(y) * KX + c] : make_double2(0.0, 0.0);
        }
        __syncthreads();
        double2 a[E];
#pragma unroll
        for (int e = 0; e < E; ++e) a[e] = tile[fx_tile(t + G * e, own, cols)];
        __syncthreads();
        fxc v[E];
        double none[E];
        const FxLine l = fx_line<E, G, kFxPlain, W::lateOne ? W::R1 : 0>(a, none, 0u, 0, [](int) { return 1.0f; });
        fx_fixed<E, kFxPlain>(a, none, l.base - l.gap, v);
        fx_fft_warp<N, false, W::lateOne>(v, x, tw, t, fx_silent(l.unit) ? 0 : fx_two(), l.gap);
        const FxUnit o = fx_out(l.unit);
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const double re = fx_to_double(v[e].x, o), im = fx_to_double(v[e].y, o);
            if (part == 0) {
                sum[e] = make_double2(re, im);
            } else {
                const double lv = rowL[t + G * e];
                sum[e] = make_double2(sum[e].x + lv * im, sum[e].y - lv * re);
            }
        }
        __syncthreads();  // every line buffer done with: the next tile
    }
    const int kx = kx0 + own;
    if (kx >= KX) return;
    double2* out = fout + (static_cast<size_t>(ch) * d.zTotal + z) * P;
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const int pos = d.ymap[static_cast<size_t>(kx) * N + t + G * e];
        if (pos >= 0) out[pos] = sum[e];
    }
}

// k_xadj on kept rows: a block takes one line-set of rows, as k_xflux_fxco.  Two warps
// transform the adjoint spectra, every thread forms a sample's gradients in FP64
// (24 operations), a warp each transforms two of the 3 + 3 nt gradient rows.
template <int N>
inline size_t smem_xadj_fx() {
    return (FxW<N>::twiddles + kFxCoWarps * FxW<N>::lines * FxW<N>::buffer) * 16 + 4 * FxW<N>::samples * 8 + 7 * (FxW<N>::samples / 2) * 16;
}
template <int N>
__global__ void __launch_bounds__(32 * kFxCoWarps, 2)
    k_xadj_fx(DescDev d, const fxw* __restrict__ twg, const double2* __restrict__ yadj, double2* __restrict__ yout,
              const double* __restrict__ physIn) {
    using W = FxW<N>;
    constexpr int G = W::G, E = W::E, H = W::H;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int Ny = d.Ny, KX = d.kxColumns, nt = d.nt;
    const int nIn = 4 + 2 * nt, nReal = 3 + 3 * nt;
    const int lane = threadIdx.x & 31, p = threadIdx.x >> 5;
    const int t = lane % G, line = lane / G;
    fxw* tw = reinterpret_cast<fxw*>(smem_raw);
    fxc* buffers = reinterpret_cast<fxc*>(tw + W::twiddles);  // [pair][line][buffer]
    fxc* x = buffers + static_cast<size_t>(p * W::lines + line) * W::buffer;
    double* Sb = reinterpret_cast<double*>(buffers + kFxCoWarps * W::lines * W::buffer);  // adjoint rows [nt][line][N]
    double2* specV = reinterpret_cast<double2*>(Sb + 4 * W::samples);                             // U, V, W [3][line][N/2]
    double2* specX = specV + 3 * (W::samples / 2);                                                      // x derivatives [nt][line][N/2]
    const int two = fx_two();
    for (int i = threadIdx.x; i < W::twiddles; i += blockDim.x) tw[i] = twg[i];
    const size_t cstride = static_cast<size_t>(Ny) * KX;
    const int rows = Ny * d.zTotal;
    const int first = blockIdx.x * W::lines;
    const bool live = first + line < rows;
    const int row = min(first + line, rows - 1);
    const int z = row / Ny, y = row - z * Ny;
    __syncthreads();
    if (2 * p < nt) {
        // c2r of the adjoint spectra, interior kx at weight 1/2 (adjoint of r2c)
        fxc AB[2][H], v[E];
        int unit[2] = {kFxZero, kFxZero};
        auto count = [&](int i) { return i == 0 && t == 0 ? 1.0f : 2.0f; };
        double none[H];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const bool has = 2 * p + q < nt;
            const double2* h = yadj + ((static_cast<size_t>(z) * nt + 2 * p + (has ? q : 0)) * Ny + y) * KX;
            double2 a[H];
#pragma unroll
            for (int i = 0; i < H; ++i) {
                const int k = t + G * i;
                const double2 s = has && k < KX ? h[k] : make_double2(0.0, 0.0);
                a[i] = k == 0 ? make_double2(s.x, 0.0) : make_double2(0.5 * s.x, 0.5 * s.y);
            }
            fx_quantise_lane<H, G, kFxPlain>(a, none, 0u, 1, count, AB[q], unit[q]);
        }
#pragma unroll
        for (int i = 0; i < H; ++i) {
            const fxc a = AB[0][i], b = AB[1][i];
            const int k = t + G * i;
            v[i] = fxc{a.x - b.y, a.y + b.x};
            x[fx_pad(k == 0 ? N / 2 : N - k)] = k == 0 ? fxc{0, 0} : fxc{a.x + b.y, b.x - a.y};
        }
        __syncwarp();
#pragma unroll
        for (int e = H; e < E; ++e) v[e] = x[fx_pad(t + G * e)];
        __syncwarp();
        fx_fft_warp<N, true>(v, x, tw, t, fx_silent(max(unit[0], unit[1])) ? 0 : two);
        const FxUnit oa = fx_out(unit[0]), ob = fx_out(unit[1]);
#pragma unroll
        for (int e = 0; e < E; ++e) {
            Sb[2 * p * W::samples + line * N + t + G * e] = fx_to_double(v[e].x, oa);
            if (2 * p + 1 < nt) Sb[(2 * p + 1) * W::samples + line * N + t + G * e] = fx_to_double(v[e].y, ob);
        }
    }
    __syncthreads();
    for (int s = threadIdx.x; s < W::samples; s += 32 * kFxCoWarps) {
        // a sample a thread: g_U = -sum S q_x ..., and -S (U, V, W) for the derivative rows
        const int ln = s / N, xx = s - ln * N;
        const int rr = min(first + ln, rows - 1), zz = rr / Ny, yy = rr - zz * Ny;
        const double* ph = physIn + (static_cast<size_t>(zz) * nReal * Ny + yy) * N + xx;
        const size_t rs = static_cast<size_t>(Ny) * N;
        const double vel[3] = {ph[0], ph[rs], ph[2 * rs]};
        double g[3] = {0.0, 0.0, 0.0};
        auto slot = [&](int r) {  // row r of the gradients: half of an entry of line r / 2
            return reinterpret_cast<double*>(buffers + static_cast<size_t>((r >> 1) * W::lines + ln) * W::buffer + xx) + (r & 1);
        };
        for (int tt = 0; tt < nt; ++tt) {
            const double sb = Sb[tt * W::samples + s];
#pragma unroll
            for (int kind = 0; kind < 3; ++kind) {
                const int r = 3 + 3 * tt + kind;
                g[kind] -= sb * ph[r * rs];
                *slot(r) = -sb * vel[kind];
            }
        }
#pragma unroll
        for (int kind = 0; kind < 3; ++kind) *slot(kind) = g[kind];
        if (nReal & 1) *slot(nReal) = 0.0;
    }
    __syncthreads();
    if (2 * p < nReal) {
        double ra[E], rb[E];
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const double2 s = reinterpret_cast<const double2*>(x)[t + G * e];
            ra[e] = s.x;
            rb[e] = s.y;
        }
        __syncwarp();
        fxc v[E];
        int ua, ub, gap;
        fx_real_pair<N>(ra, rb, v, ua, ub, gap);
        fx_fft_warp<N, false, W::latePair>(v, x, tw, t, fx_silent(max(ua, ub)) ? 0 : two, gap);
#pragma unroll
        for (int e = H; e < E; ++e) x[fx_pad(t + G * e)] = v[e];
        __syncwarp();
        const double* rowK = row_k<double>(d);
        // interior kx doubled (adjoint of c2r); the split's halves cancel it there
        const FxUnit oa = fx_out(ua), ob = fx_out(ub), oa0 = fx_out(ua - 1), ob0 = fx_out(ub - 1);
        auto store = [&](int r, int k, double2 val) {
            if (r < 3) { specV[(r * W::lines + line) * (N / 2) + k] = val; return; }
            const int tt = (r - 3) / 3, kind = (r - 3) - 3 * tt;
            if (kind == 0) {  // (i k)^* = -i k
                const double kk = rowK[k];
                specX[(tt * W::lines + line) * (N / 2) + k] = make_double2(kk * val.y, -kk * val.x);
                return;
            }
            const int c = kind == 1 ? 4 + tt : 4 + nt + tt;
            if (live) yout[(static_cast<size_t>(z) * nIn + c) * cstride + static_cast<size_t>(y) * KX + k] = val;
        };
#pragma unroll
        for (int i = 0; i < H; ++i) {
            const int k = t + G * i;
            if (k >= KX) continue;
            const fxc a = v[i], b = k == 0 ? v[0] : x[fx_pad(N - k)];
            const FxUnit& pa = k == 0 ? oa0 : oa;
            const FxUnit& pb = k == 0 ? ob0 : ob;
            store(2 * p, k, make_double2(fx_to_double(a.x + b.x, pa), fx_to_double(a.y - b.y, pa)));
            if (2 * p + 1 < nReal) store(2 * p + 1, k, make_double2(fx_to_double(a.y + b.y, pb), fx_to_double(b.x - a.x, pb)));
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 4 * W::lines * KX; i += blockDim.x) {
        const int k = i % KX, rest = i / KX;
        const int ln = rest % W::lines, c = rest / W::lines;
        if (first + ln >= rows) continue;
        double2 o = c < 3 ? specV[(c * W::lines + ln) * (N / 2) + k] : make_double2(0.0, 0.0);
        for (int tt = 0; tt < nt; ++tt)
            if (d.tq[tt] == c) {
                const double2 e = specX[(tt * W::lines + ln) * (N / 2) + k];
                o = make_double2(o.x + e.x, o.y + e.y);
            }
        const int rr = first + ln, zz = rr / Ny, yy = rr - zz * Ny;
        yout[(static_cast<size_t>(zz) * nIn + c) * cstride + static_cast<size_t>(yy) * KX + k] = o;
    }
}

}  // namespace dev
}  // namespace wvgpu
