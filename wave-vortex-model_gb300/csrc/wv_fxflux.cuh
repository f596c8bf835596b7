// The x pass of the FP64 flux in fixed point for row lengths without a lane-held
// line (wv_fxwarp.cuh): the same arithmetic with run-time stages (fx_all_stages) over
// one warp's lines in shared memory, one warp per (y, z) row.
#pragma once

#include "wv_fxwarp.cuh"

namespace wvgpu {
namespace dev {

// Pairs of one batch: enough lines to give every lane a radix-8 butterfly.
inline int fx_xany_pairs(int Nx, int nt) {
    const int all = (3 + 3 * nt + 1) / 2;
    const int p = 256 / Nx;
    return p < 1 ? 1 : p < all ? p : all;
}
// Shared memory of a warp: two line buffers, u, v, w and the products; rounded up
// to the 16 bytes that the next warp's lines are aligned to (odd Nx).
__host__ __device__ inline size_t fx_xany_warp_bytes(int Nx, int nt, int pairs) {
    return (static_cast<size_t>(Nx) * (32 * pairs + 24 + 8 * nt) + 15) / 16 * 16;
}

// Two spectrum rows in fixed point, held by a warp: entries k = lane + 32 i (0 from KX
// on; a null row: zeros), units as fx_unit, `gap` the bits by which their line starts finer.
template <int EK>
__device__ __forceinline__ void fx_load_rows(const double2* __restrict__ hA, const double2* __restrict__ hB, bool kA, bool kB,
                                             int KX, int Nx, int radix, int lane, const double* __restrict__ rowK, fxc (&A)[EK],
                                             fxc (&B)[EK], int& unitA, int& unitB, int& gap) {
    constexpr int radix1 = EK > 2 ? 1 : 0;  // (64 columns and fewer: no rows past kFxLateFrom)
    double2 v[2][EK];
    double w[EK];
    FxLine l[2];
    auto count = [&](int i) { const int k = lane + 32 * i; return k == 0 || 2 * k == Nx ? 1.0f : 2.0f; };
    auto weights = [&]() {
#pragma unroll
        for (int i = 0; i < EK; ++i) w[i] = lane + 32 * i < KX ? rowK[lane + 32 * i] : 0.0;
    };
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const double2* h = q ? hB : hA;
#pragma unroll
        for (int i = 0; i < EK; ++i) {
            const int k = lane + 32 * i;
            v[q][i] = h && k < KX ? h[k] : make_double2(0.0, 0.0);
            if (k == 0 || 2 * k == Nx) v[q][i].y = 0.0;  // c2r semantics
        }
    }
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        if (q ? kB : kA) {
            weights();
            l[q] = fx_line<EK, 32, kFxImag, radix1, 0>(v[q], w, fx_row_k_top(rowK, KX), 1, count);
        } else {
            l[q] = fx_line<EK, 32, kFxPlain, radix1, 0>(v[q], w, 0u, 1, count);
        }
    }
    // (fx_line's gap is against one entry; the first stage adds `radix` of them)
    gap = radix1 && radix > 0 && Nx > kFxLateFrom ? max(0, fx_shared_gap(l[0].gap, l[1].gap) - fx_ceil_log2(radix)) : 0;
    if (gap < 2) gap = 0;  // not worth the shifts
    unitA = l[0].unit;
    unitB = l[1].unit;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        fxc(&row)[EK] = q ? B : A;
        if (q ? kB : kA) {
            weights();
            fx_fixed<EK, kFxImag>(v[q], w, l[q].base - gap, row);
#pragma unroll
            for (int i = 0; i < EK; ++i)
                if (2 * (lane + 32 * i) == Nx) row[i].y = 0;
        } else {
            fx_fixed<EK, kFxPlain>(v[q], w, l[q].base - gap, row);
        }
    }
}

// Rows of x past kFxLateFrom points have more than 64 columns (EK > 2) or keep no gap; most
// spectra of a flow fall off and have none to speak of (fx_load_rows).
template <int EK, bool INV>
__device__ inline fxc* fx_row_stages(fxc* a, fxc* b, const FxFactors f, int lines, const fxw* tw, int gap) {
    if (EK > 2 && gap > 0) return fx_all_stages<INV, true, (EK > 2)>(a, b, f, lines, f.N, tw, nullptr, gap);
    return fx_all_stages<INV, true, false>(a, b, f, lines, f.N, tw, nullptr, 0);
}
// Z = A + i B and its mirror into the line (every entry of it written).
template <int EK>
__device__ __forceinline__ void fx_pack_rows(const fxc (&A)[EK], const fxc (&B)[EK], fxc* __restrict__ line, int KX, int Nx,
                                             int lane) {
    for (int i = KX + lane; i <= Nx - KX; i += 32) line[i] = fxc{0, 0};
#pragma unroll
    for (int i = 0; i < EK; ++i) {
        const int k = lane + 32 * i;
        if (k < KX) {
            line[k] = fxc{A[i].x - B[i].y, A[i].y + B[i].x};
            if (k > 0 && 2 * k != Nx) line[Nx - k] = fxc{A[i].x + B[i].y, B[i].x - A[i].y};
        }
    }
}

__device__ __forceinline__ long long fx_abs(long long v) { return v < 0 ? -v : v; }

// The row order of the x pass: 0 u, 1 v, 2 w, then 3 + 3 t + (x, y, z derivative of
// target t).  physOut / advOut / advIn / maxSpeedBits as k_xflux.
template <int EK>
__global__ void __launch_bounds__(512, 1) k_xflux_fxany(DescDev d, FFTDev f, const fxw* __restrict__ twg,
                                                    const double2* __restrict__ yspec, double2* __restrict__ pspec,
                                                    unsigned long long* __restrict__ maxSpeedBits, double* __restrict__ physOut,
                                                    double* __restrict__ advOut, const double* __restrict__ advIn, int pairs) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int Nx = d.Nx, Ny = d.Ny, KX = d.kxColumns, nt = d.nt;
    const int nIn = 4 + 2 * nt, nReal = 3 + 3 * nt;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    fxw* tw = reinterpret_cast<fxw*>(smem_raw);  // [Nx]
    for (int i = threadIdx.x; i < Nx; i += blockDim.x) tw[i] = twg[i];
    __syncthreads();
    unsigned char* mine = smem_raw + static_cast<size_t>(Nx) * 16 +
                          warp * fx_xany_warp_bytes(Nx, nt, pairs);
    fxc* bufA = reinterpret_cast<fxc*>(mine);  // [pairs][Nx]
    fxc* bufB = bufA + pairs * Nx;
    long long* phys = reinterpret_cast<long long*>(bufB + pairs * Nx);  // u, v, w [3][Nx]
    long long* S = phys + 3 * Nx;                                       // [nt][Nx]
    const FxFactors fac{f.N, f.nstages, f.radix};
    const double* rowK = row_k<double>(d);
    const size_t cstride = static_cast<size_t>(Ny) * KX;
    const size_t R3 = static_cast<size_t>(Nx) * Ny * d.Nz;
    const int rows = Ny * d.zTotal;
    double vmax2 = 0.0;
    int speedMember = -1;
    for (int row = blockIdx.x * warps + warp; row < rows; row += gridDim.x * warps) {
        const int z = row / Ny, y = row - z * Ny;
        const double2* yrow = yspec + (static_cast<size_t>(z) * nIn * Ny + y) * KX;
        int physUnit[3] = {0, 0, 0}, sUnit[4] = {0, 0, 0, 0};
        for (int p0 = 0; 2 * p0 < nReal; p0 += pairs) {
            const int np = min(pairs, (nReal + 1) / 2 - p0);
            int units = 0;  // lane 2 i (2 i + 1) keeps the unit of row A (B) of pair i
            int gap = 0;    // (rows past kFxLateFrom: one pair a batch)
            for (int i = 0; i < np; ++i) {
                fxc A[EK], B[EK];
                int uA, uB;
                bool useK[2] = {false, false};
                auto spectrum = [&](int q) -> const double2* {
                    const int r = 2 * (p0 + i) + q;
                    if (r >= nReal) return nullptr;
                    int ch = r;
                    if (r >= 3) {
                        const int t = (r - 3) / 3, kind = (r - 3) - 3 * t;
                        useK[q] = kind == 0;
                        ch = kind == 0 ? d.tq[t] : kind == 1 ? 4 + t : 4 + nt + t;
                    }
                    return yrow + ch * cstride;
                };
                const double2 *hA = spectrum(0), *hB = spectrum(1);
                fx_load_rows<EK>(hA, hB, useK[0], useK[1], KX, Nx, fx_gap_radix(f.nstages, f.radix), lane, rowK, A, B, uA, uB, gap);
                if (lane == 2 * i) units = uA;
                if (lane == 2 * i + 1) units = uB;
                fx_pack_rows<EK>(A, B, bufA + i * Nx, KX, Nx, lane);
            }
            __syncwarp();
            const fxc* res = fx_row_stages<EK, true>(bufA, bufB, fac, np, tw, gap);
            const long long* real = reinterpret_cast<const long long*>(res);
            for (int i = 0; i < 2 * np; ++i) {
                const int r = 2 * p0 + i;
                if (r >= nReal) break;
                const int unit = __shfl_sync(0xffffffffu, units, i);
                const long long* a = real + static_cast<size_t>(i >> 1) * 2 * Nx + (i & 1);  // stride 2
                double* keep = physOut ? physOut + ((static_cast<size_t>(z) * nReal + r) * Ny + y) * Nx : nullptr;
                if (r < 3) {
                    // the advecting velocity, normalised to 62 bits
                    const size_t g = static_cast<size_t>(r) * R3 + (static_cast<size_t>(z) * Ny + y) * Nx;
                    unsigned top = 0;
                    if (advIn) {
                        for (int x = lane; x < Nx; x += 32)
                            top = max(top, static_cast<unsigned>(__double2hiint(advIn[g + x])) & 0x7fffffffu);
                        top = __reduce_max_sync(0xffffffffu, top);
                        const fxscale sc = fx_velocity_scale(top);
                        for (int x = lane; x < Nx; x += 32) {
                            const double v = advIn[g + x];
                            phys[r * Nx + x] = fx_from_double(v, sc);
                            if (keep) keep[x] = v;
                        }
                        const int un = fx_unit(sc);
                        if (r == 0) physUnit[0] = un; else if (r == 1) physUnit[1] = un; else physUnit[2] = un;
                    } else {
                        for (int x = lane; x < Nx; x += 32)
                            top = max(top, static_cast<unsigned>(static_cast<unsigned long long>(fx_abs(a[2 * x])) >> 32));
                        top = __reduce_max_sync(0xffffffffu, top);
                        const int sh = max(0, __clz(static_cast<int>(top)) - 2);
                        const FxUnit o = fx_out(unit - sh);
                        for (int x = lane; x < Nx; x += 32) {
                            const long long v = fx_round53(a[2 * x] << sh);
                            phys[r * Nx + x] = v;
                            if (advOut) advOut[g + x] = fx_to_double(v, o);
                            if (keep) keep[x] = fx_to_double(v, o);
                        }
                        const int un = unit - sh;
                        if (r == 0) physUnit[0] = un; else if (r == 1) physUnit[1] = un; else physUnit[2] = un;
                    }
                    continue;
                }
                const int t = (r - 3) / 3, kind = (r - 3) - 3 * t;
                const int pu = kind == 0 ? physUnit[0] : kind == 1 ? physUnit[1] : physUnit[2];
                const int un = pu + unit - 1023 + 62;
                const long long* vel = phys + kind * Nx;
                long long* s = S + t * Nx;
                const int before = t == 0 ? sUnit[0] : t == 1 ? sUnit[1] : t == 2 ? sUnit[2] : sUnit[3];
                const int now = kind == 0 ? un : max(before, un);
                const int shS = kind == 0 ? 0 : min(63, now - before), shP = min(63, now - un);
                const FxUnit o = fx_out(unit);
                const long long hS = fx_half(shS, lane & 1), hP = fx_half(shP, lane & 1);
                for (int x = lane; x < Nx; x += 32) {
                    const long long v = a[2 * x];
                    const long long pr = (fx_prod(vel[x], v) + hP) >> shP;
                    s[x] = kind == 0 ? -pr : ((s[x] + hS) >> shS) - pr;
                    if (keep) keep[x] = fx_to_double(v, o);
                }
                if (t == 0) sUnit[0] = now; else if (t == 1) sUnit[1] = now; else if (t == 2) sUnit[2] = now; else sUnit[3] = now;
            }
            __syncwarp();
        }
        // max |u_h| (only when adaptive damping consumes it)
        if (maxSpeedBits) {
            const int member = z / d.Nz;
            if (member != speedMember) {
                if (speedMember >= 0) {
                    for (int o = 16; o > 0; o >>= 1) vmax2 = fmax(vmax2, __shfl_xor_sync(0xffffffffu, vmax2, o));
                    if (lane == 0) atomicMax(maxSpeedBits + speedMember, (unsigned long long)__double_as_longlong(sqrt(vmax2)));
                }
                speedMember = member;
                vmax2 = 0.0;
            }
            const FxUnit oU = fx_out(physUnit[0]), oV = fx_out(physUnit[1]);
            for (int x = lane; x < Nx; x += 32) {
                const double U = fx_to_double(phys[x], oU), V = fx_to_double(phys[Nx + x], oV);
                vmax2 = fmax(vmax2, U * U + V * V);
            }
        }
        // r2c of the products, two targets to a line
        for (int t0 = 0; t0 < nt; t0 += 2 * pairs) {
            const int nl = min(pairs, (nt - t0 + 1) / 2);
            int units = 0, gap = 0;
            for (int i = 0; i < nl; ++i) {
                int sh[2] = {0, 0};
                gap = EK > 2 && Nx > kFxLateFrom && f.nstages > 1 ? kFxAnyGap : 0;
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const int t = t0 + 2 * i + q;
                    if (t >= nt) continue;
                    unsigned sum = 0, most = 0;
                    for (int x = lane; x < Nx; x += 32) {
                        const unsigned m = static_cast<unsigned>(static_cast<unsigned long long>(fx_abs(S[t * Nx + x])) >> 41) + 1u;
                        sum += m;
                        most = max(most, m);
                    }
                    sum = __reduce_add_sync(0xffffffffu, sum);
                    most = __reduce_max_sync(0xffffffffu, most);
                    const int bits = 32 - __clz(static_cast<int>(sum));
                    sh[q] = 41 + bits - 60;  // sum |S| < 2^60 after the shift
                    gap = min(gap, max(0, bits - (32 - __clz(static_cast<int>(most))) - fx_ceil_log2(f.radix[0])));
                    const int u = (t == 0 ? sUnit[0] : t == 1 ? sUnit[1] : t == 2 ? sUnit[2] : sUnit[3]) + sh[q] - 1;
                    if (lane == 2 * i + q) units = u;
                }
                sh[0] -= gap;
                sh[1] -= gap;
                const long long* a = S + (t0 + 2 * i) * Nx;
                const bool both = t0 + 2 * i + 1 < nt;
                for (int x = lane; x < Nx; x += 32) {
                    fxc v;
                    v.x = fx_shift_round(a[x], sh[0], lane & 1);
                    v.y = both ? fx_shift_round(a[Nx + x], sh[1], lane & 1) : 0;
                    bufA[i * Nx + x] = v;
                }
            }
            __syncwarp();
            const fxc* res = fx_row_stages<EK, false>(bufA, bufB, fac, nl, tw, gap);
            for (int i = 0; i < nl; ++i) {
                const int t = t0 + 2 * i;
                const int ua = __shfl_sync(0xffffffffu, units, 2 * i), ub = __shfl_sync(0xffffffffu, units, 2 * i + 1);
                double2* out = pspec + ((static_cast<size_t>(z) * nt + t) * Ny + y) * KX;
                const FxUnit oa = fx_out(ua), ob = fx_out(ub);
                for (int k = lane; k < KX; k += 32) {
                    const fxc a = res[i * Nx + k], b = res[i * Nx + (k == 0 ? 0 : Nx - k)];
                    out[k] = make_double2(fx_to_double(a.x + b.x, oa), fx_to_double(a.y - b.y, oa));
                    if (t + 1 < nt)
                        out[cstride + k] = make_double2(fx_to_double(a.y + b.y, ob), fx_to_double(b.x - a.x, ob));
                }
            }
            __syncwarp();
        }
    }
    if (maxSpeedBits && speedMember >= 0) {
        for (int o = 16; o > 0; o >>= 1) vmax2 = fmax(vmax2, __shfl_xor_sync(0xffffffffu, vmax2, o));
        if (lane == 0) atomicMax(maxSpeedBits + speedMember, (unsigned long long)__double_as_longlong(sqrt(vmax2)));
    }
}

}  // namespace dev
}  // namespace wvgpu
