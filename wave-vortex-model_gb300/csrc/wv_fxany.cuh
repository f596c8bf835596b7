// The y, z and field x passes of FP64 handles in fixed point for every length: the
// run-time stages of wv_fx.cuh over lines in shared memory, each line owned by one
// warp from its scaling to its result (no block barrier inside the transforms).
// Lengths with lane-held lines take wv_fxyz.cuh where it has the pass.
#pragma once

#include "wv_fxflux.cuh"
#include "wv_fxyz.cuh"

namespace wvgpu {
namespace dev {

// Lines are odd numbers of 16-byte entries apart: a column of the [line][entry]
// buffer then meets all banks.
__host__ __device__ inline int fx_any_ld(int N) { return N | 1; }

// Scale of a line whose entry i (0 <= i < n) is at(i), counted count(i) times in the
// sum of moduli; the warp's lanes share the entries.  radix > 0: with the bits by which
// the line may start finer.
template <typename At, typename Count>
__device__ __forceinline__ fxscale fx_warp_scale(int n, int lane, int radix, At at, Count count) {
    float sum = 0.f, most = 0.f;
    for (int i = lane; i < n; i += 32) {
        const double2 v = at(i);
        const float m = fx_modulus(fx_mag(static_cast<unsigned>(__double2hiint(v.x))), fx_mag(static_cast<unsigned>(__double2hiint(v.y))));
        sum += count(i) * m;
        most = fmaxf(most, m);
    }
    sum = fx_group_sum<32>(sum);
    if (fx_plain_sum(sum)) {
        fxscale sc = fx_scale(sum);
        if (radix > 0) sc.gap = fx_gap(sum, __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(most))), radix);
        return sc;
    }
    unsigned top = 0;
    for (int i = lane; i < n; i += 32) {
        const double2 v = at(i);
        top = max(top, max(static_cast<unsigned>(__double2hiint(v.x)) & 0x7fffffffu,
                           static_cast<unsigned>(__double2hiint(v.y)) & 0x7fffffffu));
    }
    top = __reduce_max_sync(0xffffffffu, top);
    float rel = 0.f;
    most = 0.f;
    for (int i = lane; i < n; i += 32) {
        const double2 v = at(i);
        const float m = fx_modulus(fx_rel(static_cast<unsigned>(__double2hiint(v.x)), top),
                                   fx_rel(static_cast<unsigned>(__double2hiint(v.y)), top));
        rel += count(i) * m;
        most = fmaxf(most, m);
    }
    rel = fx_group_sum<32>(rel);
    most = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(most)));
    fxscale sc = fx_scale(top, rel);
    if (radix > 0) sc.gap = sc.zero ? kFxAnyGap : fx_gap(rel, most, radix);
    return sc;
}
// LATE in the kernels below: the lines are longer than kFxLateFrom and may start finer.
// ---- y ------------------------------------------------------------------------------

constexpr int kFxAnyWarps = 8;
// Columns of a block of `planes` (z, channel) planes: about 2048 entries, but down to a
// line per warp while the blocks don't reach every SM twice.
inline int fx_any_cols(int Ny, int kxColumns, size_t planes, size_t sms) {
    int c = 2048 / Ny;
    if (c > 32 * kFxAnyWarps) c = 32 * kFxAnyWarps;  // (a lane keeps one line's unit)
    if (c > kxColumns) c = kxColumns;
    while (c > kFxAnyWarps && (kxColumns + c - 1) / c * planes < 2 * sms) c = (c + 1) / 2;
    return c < 1 ? 1 : c;
}
inline size_t smem_fx_any_y(int Ny, int cols) {
    return (static_cast<size_t>(Ny) + 2 * static_cast<size_t>(cols) * fx_any_ld(Ny)) * 16;
}

__device__ __forceinline__ void fx_any_twiddles(fxw* tw, const fxw* __restrict__ twg, int N) {
    for (int i = threadIdx.x; i < N; i += blockDim.x) tw[i] = twg[i];
    __syncthreads();
}
// k_yinv, channel blockIdx.z.  Bound by shared memory: a stage reads and writes every
// entry.  60x50x31 hydrostatic, all five passes: 268 (FP64 pipe) -> 111 us.
template <bool LATE>
__global__ void __launch_bounds__(32 * kFxAnyWarps)
    k_yinv_fxany(DescDev d, YInvMap map, const double2* __restrict__ zspec, double2* __restrict__ yspec, int cols) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int Ny = d.Ny, P = d.positions, KX = d.kxColumns, ld = fx_any_ld(Ny);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const int kx0 = blockIdx.x * cols, z = blockIdx.y, oc = blockIdx.z;
    const int g = min(cols, KX - kx0);
    fxw* tw = reinterpret_cast<fxw*>(smem_raw);
    double2* bufA = reinterpret_cast<double2*>(tw + Ny);
    double2* bufB = bufA + static_cast<size_t>(cols) * ld;
    fx_any_twiddles(tw, static_cast<const fxw*>(d.twy), Ny);
    const double2* in = zspec + (static_cast<size_t>(map.src[oc]) * d.zTotal + z) * P;
    const double* rowL = row_l<double>(d);
    const bool mulL = map.mulL[oc] != 0;
    const int each = (cols + warps - 1) / warps;  // lines of a warp
    const int c0 = warp * each, nl = min(each, g - c0);
    __shared__ int gaps[kFxAnyWarps][LATE ? 32 : 1];  // of the warp's lines
    int units = 0;  // lane l keeps the unit of line c0 + l (each <= 32)
    for (int l = 0; l < nl; ++l) {
        double2* row = bufA + (c0 + l) * ld;
        const int* ym = d.ymap + static_cast<size_t>(kx0 + c0 + l) * Ny;
        for (int i = lane; i < Ny; i += 32) {
            const int pos = ym[i];
            double2 v = pos >= 0 ? in[pos] : make_double2(0.0, 0.0);
            if (mulL) v = make_double2(-rowL[i] * v.y, rowL[i] * v.x);
            row[i] = v;
        }
        fxscale sc = fx_warp_scale(Ny, lane, LATE ? fx_gap_radix(d.fy.nstages, d.fy.radix) : 0, [&](int i) { return row[i]; }, [](int) { return 1.0f; });
        if (lane == l) units = fx_unit(sc);
        if (LATE && lane == 0) gaps[warp][l] = sc.gap;
        sc.bit += sc.gap;
        fxc* q = reinterpret_cast<fxc*>(row);
        for (int i = lane; i < Ny; i += 32) {
            const double2 v = row[i];
            q[i] = fxc{fx_from_double(v.x, sc), fx_from_double(v.y, sc)};
        }
    }
    __syncwarp();
    double2* res = bufA;
    if (nl > 0) {
        fxc* r = fx_all_stages<true, true, LATE>(reinterpret_cast<fxc*>(bufA + c0 * ld), reinterpret_cast<fxc*>(bufB + c0 * ld),
                                                 FxFactors{d.fy.N, d.fy.nstages, d.fy.radix}, nl, ld, tw, gaps[warp], 0);
        for (int l = 0; l < nl; ++l) {
            const int u = __shfl_sync(0xffffffffu, units, l);
            double2* o = reinterpret_cast<double2*>(r + l * ld);
            for (int i = lane; i < Ny; i += 32) {
                const fxc v = r[l * ld + i];
                o[i] = make_double2(fx_to_double(v.x, fx_out(u)), fx_to_double(v.y, fx_out(u)));
            }
        }
    }
    if (d.fy.nstages & 1) res = bufB;
    __syncthreads();
    double2* out = yspec + (static_cast<size_t>(z) * map.nOut + oc) * Ny * KX + kx0;
    for (int i = threadIdx.x; i < g * Ny; i += blockDim.x) {
        const int y = i / g, c = i - y * g;
        out[static_cast<size_t>(y) * KX + c] = res[c * ld + y];
    }
}

// k_yfwd, channel blockIdx.z.
template <bool LATE>
__global__ void __launch_bounds__(32 * kFxAnyWarps)
    k_yfwd_fxany(DescDev d, const double2* __restrict__ pspec, int nch, double2* __restrict__ fspec, int cols) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int Ny = d.Ny, P = d.positions, KX = d.kxColumns, ld = fx_any_ld(Ny);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const int kx0 = blockIdx.x * cols, z = blockIdx.y, ch = blockIdx.z;
    const int g = min(cols, KX - kx0);
    fxw* tw = reinterpret_cast<fxw*>(smem_raw);
    double2* bufA = reinterpret_cast<double2*>(tw + Ny);
    double2* bufB = bufA + static_cast<size_t>(cols) * ld;
    const double2* in = pspec + (static_cast<size_t>(z) * nch + ch) * Ny * KX + kx0;
    for (int i = threadIdx.x; i < g * Ny; i += blockDim.x) {
        const int y = i / g, c = i - y * g;
        bufA[c * ld + y] = in[static_cast<size_t>(y) * KX + c];
    }
    fx_any_twiddles(tw, static_cast<const fxw*>(d.twy), Ny);  // (ends with a block barrier)
    const int each = (cols + warps - 1) / warps;
    const int c0 = warp * each, nl = min(each, g - c0);
    if (nl <= 0) return;
    __shared__ int gaps[kFxAnyWarps][LATE ? 32 : 1];
    int units = 0;
    for (int l = 0; l < nl; ++l) {
        double2* row = bufA + (c0 + l) * ld;
        fxscale sc = fx_warp_scale(Ny, lane, LATE ? fx_gap_radix(d.fy.nstages, d.fy.radix) : 0, [&](int i) { return row[i]; }, [](int) { return 1.0f; });
        if (lane == l) units = fx_unit(sc);
        if (LATE && lane == 0) gaps[warp][l] = sc.gap;
        sc.bit += sc.gap;
        fxc* q = reinterpret_cast<fxc*>(row);
        for (int i = lane; i < Ny; i += 32) {
            const double2 v = row[i];
            q[i] = fxc{fx_from_double(v.x, sc), fx_from_double(v.y, sc)};
        }
    }
    __syncwarp();
    const fxc* r = fx_all_stages<false, true, LATE>(reinterpret_cast<fxc*>(bufA + c0 * ld), reinterpret_cast<fxc*>(bufB + c0 * ld),
                                                    FxFactors{d.fy.N, d.fy.nstages, d.fy.radix}, nl, ld, tw, gaps[warp], 0);
    double2* out = fspec + (static_cast<size_t>(ch) * d.zTotal + z) * P;
    for (int l = 0; l < nl; ++l) {
        const int u = __shfl_sync(0xffffffffu, units, l);
        const int* ym = d.ymap + static_cast<size_t>(kx0 + c0 + l) * Ny;
        for (int i = lane; i < Ny; i += 32) {
            const int pos = ym[i];
            const fxc v = r[l * ld + i];
            if (pos >= 0) out[pos] = make_double2(fx_to_double(v.x, fx_out(u)), fx_to_double(v.y, fx_out(u)));
        }
    }
}

// ---- field rows along x -----------------------------------------------------------------

// Shared memory of the field kernels: twiddles [Nx], per warp two buffers of one line.
inline size_t smem_fx_any_x(int Nx, int warps) { return (static_cast<size_t>(Nx) + static_cast<size_t>(warps) * 2 * Nx) * 16; }

// k_xc2r_fields: a warp takes two channels of a (y, z) row as one line.  A warp per
// row with all its channels leaves small grids to a few long-running warps.
template <int EK>
__global__ void __launch_bounds__(32 * kFxAnyWarps, 2)
    k_xc2r_fxany(DescDev d, FFTDev f, const fxw* __restrict__ twg, const double2* __restrict__ yspec, int nch,
                 double* __restrict__ fields) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int Nx = d.Nx, Ny = d.Ny, KX = d.kxColumns;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    fxw* tw = reinterpret_cast<fxw*>(smem_raw);
    fxc* bufA = reinterpret_cast<fxc*>(tw + Nx) + static_cast<size_t>(warp) * 2 * Nx;
    fxc* bufB = bufA + Nx;
    fx_any_twiddles(tw, twg, Nx);
    const size_t R = static_cast<size_t>(Nx) * Ny * d.Nz;
    const int pairs = (nch + 1) / 2, units = Ny * d.zTotal * pairs;
    for (int unit = blockIdx.x * warps + warp; unit < units; unit += gridDim.x * warps) {
        const int row = unit / pairs, ca = 2 * (unit - row * pairs), cb = ca + 1;
        const int z = row / Ny, y = row - z * Ny;
        const double2* h = yspec + ((static_cast<size_t>(z) * nch + ca) * Ny + y) * KX;
        fxc A[EK], B[EK];
        int uA, uB, gap;
        fx_load_rows<EK>(h, cb < nch ? h + static_cast<size_t>(Ny) * KX : nullptr, ((d.c2rUseK >> ca) & 1) != 0,
                         cb < nch && ((d.c2rUseK >> cb) & 1) != 0, KX, Nx, fx_gap_radix(f.nstages, f.radix), lane, row_k<double>(d), A, B, uA, uB, gap);
        fx_pack_rows<EK>(A, B, bufA, KX, Nx, lane);
        __syncwarp();
        const fxc* r = fx_row_stages<EK, true>(bufA, bufB, FxFactors{f.N, f.nstages, f.radix}, 1, tw, gap);
        double* o = fields + static_cast<size_t>(ca) * R + (static_cast<size_t>(z) * Ny + y) * Nx;
        for (int x = lane; x < Nx; x += 32) {
            o[x] = fx_to_double(r[x].x, fx_out(uA));
            if (cb < nch) o[R + x] = fx_to_double(r[x].y, fx_out(uB));
        }
        __syncwarp();
    }
}

// k_xr2c_fields: a warp takes two channels of a (y, z) row as one line.
template <bool LATE>
__global__ void __launch_bounds__(32 * kFxAnyWarps, 2)
    k_xr2c_fxany(DescDev d, FFTDev f, const fxw* __restrict__ twg, const double* __restrict__ fields, int nch,
                 double2* __restrict__ pspec) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int Nx = d.Nx, Ny = d.Ny, KX = d.kxColumns;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    fxw* tw = reinterpret_cast<fxw*>(smem_raw);
    fxc* bufA = reinterpret_cast<fxc*>(tw + Nx) + static_cast<size_t>(warp) * 2 * Nx;
    fxc* bufB = bufA + Nx;
    fx_any_twiddles(tw, twg, Nx);
    const size_t R = static_cast<size_t>(Nx) * Ny * d.Nz;
    const int pairs = (nch + 1) / 2, units = Ny * d.zTotal * pairs;
    for (int unit = blockIdx.x * warps + warp; unit < units; unit += gridDim.x * warps) {
        const int row = unit / pairs, c = 2 * (unit - row * pairs);
        const int z = row / Ny, y = row - z * Ny;
        const bool both = c + 1 < nch;
        double2* raw = reinterpret_cast<double2*>(bufB);  // the samples, in their fixed-point slots
        const double* s = fields + static_cast<size_t>(c) * R + (static_cast<size_t>(z) * Ny + y) * Nx;
        for (int x = lane; x < Nx; x += 32) raw[x] = make_double2(s[x], both ? s[R + x] : 0.0);
        auto one = [](int) { return 1.0f; };
        const int radix = LATE ? fx_gap_radix(f.nstages, f.radix) : 0;
        fxscale sa = fx_warp_scale(Nx, lane, radix, [&](int x) { return make_double2(raw[x].x, 0.0); }, one);
        fxscale sb = fx_warp_scale(Nx, lane, radix, [&](int x) { return make_double2(raw[x].y, 0.0); }, one);
        sa.bit -= 1;
        sb.bit -= 1;
        const int ua = fx_unit(sa) - 1, ub = fx_unit(sb) - 1;  // the halves of the split below
        const int gap = fx_shared_gap(sa.gap, sb.gap);
        sa.bit += gap;
        sb.bit += gap;
        for (int x = lane; x < Nx; x += 32) bufA[x] = fxc{fx_from_double(raw[x].x, sa), fx_from_double(raw[x].y, sb)};
        __syncwarp();
        const fxc* r = fx_all_stages<false, true, LATE>(bufA, bufB, FxFactors{f.N, f.nstages, f.radix}, 1, Nx, tw, nullptr, gap);
        double2* o = pspec + ((static_cast<size_t>(z) * nch + c) * Ny + y) * KX;
        for (int k = lane; k < KX; k += 32) {
            const fxc a = r[k], b = r[k == 0 ? 0 : Nx - k];
            o[k] = make_double2(fx_to_double(a.x + b.x, fx_out(ua)), fx_to_double(a.y - b.y, fx_out(ua)));
            if (both)
                o[static_cast<size_t>(Ny) * KX + k] = make_double2(fx_to_double(a.y + b.y, fx_out(ub)), fx_to_double(b.x - a.x, fx_out(ub)));
        }
        __syncwarp();
    }
}

// ---- z ------------------------------------------------------------------------------

// Shared memory of the z kernels: twiddles [N], per warp two buffers of `lines` lines.
inline size_t smem_fx_any_z(int N, int lines, int warps) {
    return (static_cast<size_t>(N) + static_cast<size_t>(warps) * 2 * lines * N) * 16;
}

// k_vinv_fx for any length, one retained column per warp.
template <bool FLUX, bool LATE>
__global__ void __launch_bounds__(32 * kFxAnyWarps)
    k_vinv_fxany(DescDev d, const double* __restrict__ Ap, const double* __restrict__ Am, const double* __restrict__ A0,
                 double elapsed, double2* __restrict__ zspec, unsigned long long* __restrict__ maxSpeedBits) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int kLines = FLUX ? 4 : 2;
    const int N = d.fz.N, L = N / 2, Nj = d.Nj, P = d.positions;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const int member = blockIdx.y;
    if (member > 0) {
        const long long o = member * d.memberStride;
        Ap += o; Am += o; A0 += o;
        zspec += static_cast<size_t>(member) * d.Nz * P;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0 && maxSpeedBits) maxSpeedBits[member] = 0ull;
    fxw* tw = reinterpret_cast<fxw*>(smem_raw);
    fxc* bufA = reinterpret_cast<fxc*>(tw + N) + static_cast<size_t>(warp) * 2 * kLines * N;
    fxc* bufB = bufA + kLines * N;
    double2* fld = reinterpret_cast<double2*>(bufB);  // [4][Nj] until the lines are built (Nj <= N / 2)
    fx_any_twiddles(tw, static_cast<const fxw*>(d.twz), N);
    const int mode = blockIdx.x * warps + warp;
    if (mode >= d.Nkl) return;
    const int w = d.modeWV[mode];
    const unsigned char flags = d.modeFlags[mode];
    const double* mz = static_cast<const double*>(d.tMz);
    for (int j = lane; j < Nj; j += 32) {
        double2 f[4];
        fx_field_spectra(d, Ap, Am, A0, elapsed, w, flags, j, f);
#pragma unroll
        for (int q = 0; q < 4; ++q) fld[q * Nj + j] = f[q];
    }
    int derivChan[4] = {-1, -1, -1, -1};
    if constexpr (FLUX)
        for (int q = 0; q < d.nt; ++q) derivChan[d.tq[q]] = 4 + q;
    auto count = [](int j) { return j == 0 ? 1.0f : 2.0f; };
    __shared__ int gaps[kFxAnyWarps][kLines];
    int uC[kLines], uD[kLines];
#pragma unroll
    for (int l = 0; l < kLines; ++l) {
        const int qc = l, qs = l < 2 ? l + 2 : l - 2;
        auto atC = [&](int j) { const double2 v = fld[qc * Nj + j]; const double m = l < 2 ? 1.0 : mz[j]; return make_double2(m * v.x, m * v.y); };
        auto atD = [&](int j) { const double2 v = fld[qs * Nj + j]; const double m = l < 2 ? 1.0 : -mz[j]; return make_double2(m * v.x, m * v.y); };
        const int radix = LATE ? fx_gap_radix(d.fz.nstages, d.fz.radix) : 0;
        fxscale sC = fx_warp_scale(Nj, lane, radix, atC, count), sD = fx_warp_scale(Nj, lane, radix, atD, count);
        sC.bit -= 1; sD.bit -= 1;
        uC[l] = fx_unit(sC); uD[l] = fx_unit(sD);
        const int gap = fx_shared_gap(sC.gap, sD.gap);
        if (LATE && lane == 0) gaps[warp][l] = gap;
        sC.bit += gap; sD.bit += gap;
        // 2 y[j] = C_j + i D_j, 2 y[N-j] = C_j - i D_j, 2 y[0] = C_0; nothing between
        fxc* y = bufA + l * N;
        for (int j = lane; j < Nj; j += 32) {
            const double2 cv = atC(j), dv = atD(j);
            const fxc C = {fx_from_double(cv.x, sC), fx_from_double(cv.y, sC)};
            const fxc D = {fx_from_double(dv.x, sD), fx_from_double(dv.y, sD)};
            if (j == 0) { y[0] = C; continue; }
            y[j] = fxc{C.x - D.y, C.y + D.x};
            y[N - j] = fxc{C.x + D.y, C.y - D.x};
        }
        for (int k = Nj + lane; k <= N - Nj; k += 32) y[k] = fxc{0, 0};
    }
    __syncwarp();
    const fxc* F = fx_all_stages<false, true, LATE>(bufA, bufB, FxFactors{d.fz.N, d.fz.nstages, d.fz.radix}, kLines, N, tw, gaps[warp], 0);
    const int pos = d.modePos[mode], cpos = d.modeCompPos[mode];
#pragma unroll
    for (int l = 0; l < kLines; ++l) {
        const int chC = l < 2 ? l : derivChan[l], chS = l < 2 ? l + 2 : derivChan[l - 2];
        const fxc* row = F + l * N;
        for (int n = lane; n <= L; n += 32) {
            const fxc a = row[n], b = row[n == 0 ? 0 : N - n];
            if (chC >= 0) {
                const double2 ev = make_double2(fx_to_double(a.x + b.x, fx_out(uC[l] - 2)), fx_to_double(a.y + b.y, fx_out(uC[l] - 2)));
                double2* base = zspec + (static_cast<size_t>(chC) * d.zTotal + n) * P;
                base[pos] = ev;
                if (cpos >= 0) base[cpos] = make_double2(ev.x, -ev.y);
            }
            if (chS >= 0) {
                const double2 od = make_double2(fx_to_double(a.x - b.x, fx_out(uD[l] - 2)), fx_to_double(a.y - b.y, fx_out(uD[l] - 2)));
                double2* base = zspec + (static_cast<size_t>(chS) * d.zTotal + n) * P;
                base[pos] = od;
                if (cpos >= 0) base[cpos] = make_double2(od.x, -od.y);
            }
        }
    }
}

// k_vfwd_fx for any length, one retained column per warp.
template <bool FLUX, bool LATE>
__global__ void __launch_bounds__(32 * kFxAnyWarps)
    k_vfwd_fxany(DescDev d, const double2* __restrict__ fspec, int nch, double elapsed, const double* __restrict__ Ap,
                 const double* __restrict__ Am, const double* __restrict__ A0, const unsigned long long* __restrict__ maxSpeedBits,
                 int applyDamping, double* __restrict__ Fp, double* __restrict__ Fm, double* __restrict__ F0) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int N = d.fz.N, L = N / 2, Nj = d.Nj, P = d.positions;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const int member = blockIdx.y;
    if (member > 0) {
        const long long o = member * d.memberStride;
        if (Ap) { Ap += o; Am += o; A0 += o; }
        Fp += o; Fm += o; F0 += o;
        fspec += static_cast<size_t>(member) * d.Nz * P;
        if (maxSpeedBits) maxSpeedBits += member;
    }
    fxw* tw = reinterpret_cast<fxw*>(smem_raw);
    fxc* bufA = reinterpret_cast<fxc*>(tw + N) + static_cast<size_t>(warp) * 4 * N;
    fxc* bufB = bufA + 2 * N;
    fx_any_twiddles(tw, static_cast<const fxw*>(d.twz), N);
    const int mode = blockIdx.x * warps + warp;
    if (mode >= d.Nkl) return;
    const int w = d.modeWV[mode];
    const bool conj = d.modeFlags[mode] & 1;
    const int pos = d.modePos[mode];
    int chanOfQ[4] = {-1, -1, -1, -1};
    for (int c = 0; c < nch; ++c) chanOfQ[FLUX ? d.tq[c] : ((d.hydrostatic && c == 2) ? 3 : c)] = c;
    auto count = [L](int z) { return z == 0 || z == L ? 1.0f : 2.0f; };
    __shared__ int gaps[kFxAnyWarps][2];
    int uC[2], uS[2];
#pragma unroll
    for (int l = 0; l < 2; ++l) {
        const int cc = chanOfQ[l], cs = chanOfQ[2 + l];
        double2* rc = reinterpret_cast<double2*>(bufB + l * N);  // [L + 1] cosine, then [L - 1] sine samples
        double2* rs = rc + L;                                     // entry z of the sine channel, 1 <= z < L
        for (int z = lane; z <= L; z += 32)
            rc[z] = cc >= 0 ? fspec[(static_cast<size_t>(cc) * d.zTotal + z) * P + pos] : make_double2(0.0, 0.0);
        for (int z = 1 + lane; z < L; z += 32)
            rs[z] = cs >= 0 ? fspec[(static_cast<size_t>(cs) * d.zTotal + z) * P + pos] : make_double2(0.0, 0.0);
        __syncwarp();
        const int radix = LATE ? fx_gap_radix(d.fz.nstages, d.fz.radix) : 0;
        fxscale sC = fx_warp_scale(L + 1, lane, radix, [&](int z) { return rc[z]; }, count);
        fxscale sS = fx_warp_scale(L, lane, radix, [&](int z) { return z == 0 ? make_double2(0.0, 0.0) : rs[z]; }, count);
        sC.bit -= 1; sS.bit -= 1;
        uC[l] = fx_unit(sC); uS[l] = fx_unit(sS);
        const int gap = fx_shared_gap(sC.gap, sS.gap);
        if (LATE && lane == 0) gaps[warp][l] = gap;
        sC.bit += gap; sS.bit += gap;
        fxc* y = bufA + l * N;
        for (int z = lane; z <= L; z += 32) {
            const double2 cv = rc[z];
            const fxc C = {fx_from_double(cv.x, sC), fx_from_double(cv.y, sC)};
            if (z == 0 || z == L) { y[z] = C; continue; }
            const double2 sv = rs[z];
            const fxc S = {fx_from_double(sv.x, sS), fx_from_double(sv.y, sS)};
            y[z] = fx_add(C, S);
            y[N - z] = fx_sub(C, S);
        }
    }
    __syncwarp();
    const fxc* F = fx_all_stages<false, true, LATE>(bufA, bufB, FxFactors{d.fz.N, d.fz.nstages, d.fz.radix}, 2, N, tw, gaps[warp], 0);
    double maxSpeed = 0.0;
    if (FLUX && applyDamping) maxSpeed = __longlong_as_double((long long)*maxSpeedBits);
    const double sc = 1.0 / (static_cast<double>(L) * static_cast<double>(d.Nx) * static_cast<double>(d.Ny));
    for (int j = lane; j < Nj; j += 32) {
        double2 X[4];
#pragma unroll
        for (int l = 0; l < 2; ++l) {
            const fxc p = F[l * N + j], q = F[l * N + (j == 0 ? 0 : N - j)];
            X[l] = make_double2(fx_to_double(p.x + q.x, fx_out(uC[l] - 1)), fx_to_double(p.y + q.y, fx_out(uC[l] - 1)));
            X[2 + l] = make_double2(-fx_to_double(p.y - q.y, fx_out(uS[l] - 1)), fx_to_double(p.x - q.x, fx_out(uS[l] - 1)));
        }
        if (conj) {
#pragma unroll
            for (int q = 0; q < 4; ++q) X[q].y = -X[q].y;
        }
        fx_project<FLUX>(d, w, j, X[0], X[1], X[2], X[3], sc, elapsed, maxSpeed, applyDamping, Ap, Am, A0, Fp, Fm, F0);
    }
}

}  // namespace dev
}  // namespace wvgpu
