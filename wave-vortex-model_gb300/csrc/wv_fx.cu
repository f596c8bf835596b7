// Host side of the FP64 kernels on fixed-point lines.  See wv_fx_launch.hpp.
#include "wv_fx_launch.hpp"
#include "wv_fxflux.cuh"
#include "wv_fxyz.cuh"
#include "wv_fxany.cuh"
#include "wv_fxadj.cuh"
#include "wv_internal.hpp"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>

namespace wvgpu {
namespace {

unsigned cdiv(size_t a, size_t b) { return static_cast<unsigned>((a + b - 1) / b); }

// Line lengths held by the lanes of a warp (wv_fxwarp.cuh); NN: the length.
#define WV_FXW_CASE(LEN, ...) case LEN: { constexpr int NN = LEN; __VA_ARGS__; } break
#define WV_FXW_SWITCH(N, ...)          \
    switch (N) {                       \
        WV_FXW_CASE(16, __VA_ARGS__);  \
        WV_FXW_CASE(24, __VA_ARGS__);  \
        WV_FXW_CASE(32, __VA_ARGS__);  \
        WV_FXW_CASE(48, __VA_ARGS__);  \
        WV_FXW_CASE(64, __VA_ARGS__);  \
        WV_FXW_CASE(96, __VA_ARGS__);  \
        WV_FXW_CASE(128, __VA_ARGS__); \
        WV_FXW_CASE(192, __VA_ARGS__); \
        WV_FXW_CASE(256, __VA_ARGS__); \
        default: break;                \
    }
// Lines of a warp; 0: no lane-held line of this length.
inline size_t fx_lane_lines(size_t N) {
    WV_FXW_SWITCH(N, return dev::FxW<NN>::lines);
    return 0;
}
inline bool fx_lane_length(size_t N) { return fx_lane_lines(N) != 0; }
template <int N>
std::vector<int32_t> lane_table() {
    using W = dev::FxW<N>;
    if (W::R3 > 1) return fixed_point_stage_twiddles(N, {W::R1, W::R2, W::R3});
    return fixed_point_stage_twiddles(N, {W::R1, W::R2});
}

// The x pass: lane-held rows where the length allows (kx < Nx / 2 always holds on
// the transform's own rows); else rows of up to 512 samples and 256 kx columns on
// run-time stages; longer rows keep the block kernel.
inline bool fx_x_lane(const Plan& p) { return fx_lane_length(p.Nx) && 2 * p.kxColumns <= p.Nx; }
inline bool fx_x_any(const Plan& p) { return p.Nx <= 512 && p.kxColumns <= 256; }
// Spectrum entries of a lane in the x pass under the 2/3 rule, and at most.
template <int N>
struct XKernels {
    static constexpr int few = dev::FxW<N>::E == 8 ? 3 : 5, all = dev::FxW<N>::H;
};
// Warps of a y or z block: 8, fewer where the columns of a plane (the retained
// columns) do not fill them; powers of two in y, as the tile's swizzle needs.
inline int fx_y_warps(size_t Ny, size_t kxColumns) {
    const size_t lines = fx_lane_lines(Ny);
    int warps = 1;
    while (warps < dev::kFxYWarps && warps * lines < kxColumns) warps *= 2;
    return warps;
}
// Column sets of a z block (its warps: sets x lines of a column): enough blocks for
// every SM before the blocks grow to 8 warps.
inline int fx_z_sets(const Plan& p, int lines) {
    const size_t columns = fx_lane_lines(p.fz.N), units = (p.Nkl + columns - 1) / columns, sms = grid_cap(1);
    return static_cast<int>(std::min<size_t>(dev::kFxZWarps / lines, std::max<size_t>(1, units / sms)));
}
// Lines of any length along z: warps of a block, as shared memory allows.
inline int fx_z_any_warps(const Plan& p, int lines) {
    const size_t each = 2 * static_cast<size_t>(lines) * p.fz.N * 16, sms = grid_cap(1);
    const size_t room = std::max<size_t>(1, (100 * 1024) / each);
    return static_cast<int>(std::min<size_t>({room, dev::kFxAnyWarps, std::max<size_t>(1, (p.Nkl + sms - 1) / sms)}));
}
// The run-time field kernels along x: a warp per row and channel pair.
struct FxFieldLaunch { int warps, grid; size_t smem; };
inline FxFieldLaunch fx_field_launch(size_t Nx, size_t rows, int nch) {
    FxFieldLaunch l{};
    const size_t units = rows * ((nch + 1) / 2), each = 2 * Nx * 16;
    l.warps = static_cast<int>(std::min<size_t>(dev::kFxAnyWarps, std::max<size_t>(1, (104 * 1024 - Nx * 16) / each)));
    while (l.warps > 1 && units < l.warps * static_cast<size_t>(grid_cap(1))) l.warps /= 2;
    l.smem = dev::smem_fx_any_x(static_cast<int>(Nx), l.warps);
    l.grid = static_cast<int>(std::min<size_t>((units + l.warps - 1) / l.warps, grid_cap(2)));
    return l;
}
// Grid and warps of the lane-held field kernels (a warp per line-set and channel pair;
// single warps while they don't fill every SM).
struct FxLaneField { unsigned grid; int warps; };
FxLaneField fx_lane_field(const Plan& p, const dev::DescDev& d, int nch) {
    const size_t sets = (p.Ny * d.zTotal + fx_lane_lines(p.Nx) - 1) / fx_lane_lines(p.Nx), units = sets * ((nch + 1) / 2);
    const int warps = units < dev::kFxFieldWarps * static_cast<size_t>(grid_cap(1)) ? 1 : dev::kFxFieldWarps;
    return {cdiv(units, warps), warps};
}
struct FxXLaunch { int warps, grid, pairs; size_t smem; };
inline FxXLaunch fx_x_launch(const Plan& p, int members) {
    FxXLaunch l{};
    const int nt = p.targets.count, Nx = static_cast<int>(p.Nx);
    l.pairs = dev::fx_xany_pairs(Nx, nt);
    const size_t warp = dev::fx_xany_warp_bytes(Nx, nt, l.pairs), table = p.Nx * sizeof(dev::fxw);
    const size_t most = 226 * 1024;
    // 16 warps per SM (128 registers a thread) as two blocks where they fit
    // beside each other, else one block of as many warps as shared memory holds
    if (2 * (8 * warp + table) <= most) l.warps = 8;
    else l.warps = static_cast<int>(std::min<size_t>(16, (most - table) / warp));
    const size_t rows = p.Ny * p.Nz * members;
    l.smem = table + l.warps * warp;
    l.grid = static_cast<int>(std::min<size_t>((rows + l.warps - 1) / l.warps, grid_cap(l.warps == 8 ? 2 : 1)));
    return l;
}
#define WV_FXX_SWITCH(KX, ...)                           \
    if ((KX) <= 64) { constexpr int EK = 2; __VA_ARGS__; }      \
    else if ((KX) <= 128) { constexpr int EK = 4; __VA_ARGS__; } \
    else { constexpr int EK = 8; __VA_ARGS__; }

}  // namespace

std::vector<int32_t> fx_lane_table(size_t N) {
    WV_FXW_SWITCH(N, return lane_table<NN>());
    return {};
}

cudaError_t fx_set_limits(const Plan& p) {
    cudaError_t e = cudaSuccess;
    auto set = [&](auto* kernel, size_t bytes) {
        if (e == cudaSuccess) e = raise_smem_limit(reinterpret_cast<const void*>(kernel), static_cast<int>(bytes));
    };
    WV_FXW_SWITCH(p.Ny, {
        set(dev::k_yinv_fx<NN>, dev::smem_fxy<NN>(dev::kFxYWarps * dev::FxW<NN>::lines));
        set(dev::k_yfwd_fx<NN>, dev::smem_fxy<NN>(dev::kFxYWarps * dev::FxW<NN>::lines));
    });
    if (!fx_lane_length(p.Ny)) {
        // (the scalar pipeline has the most columns)
        const size_t sm = dev::smem_fx_any_y(static_cast<int>(p.Ny), dev::fx_any_cols(static_cast<int>(p.Ny), 1 << 20, 1, 1));
        const bool late = p.Ny > dev::kFxLateFrom;
        set(late ? dev::k_yinv_fxany<true> : dev::k_yinv_fxany<false>, sm);
        set(late ? dev::k_yfwd_fxany<true> : dev::k_yfwd_fxany<false>, sm);
    }
    WV_FXW_SWITCH(p.Nx, {
        set(dev::k_xc2r_fx<NN>, dev::smem_fx_field<NN>(dev::kFxFieldWarps));
        set(dev::k_xr2c_fx<NN>, dev::smem_fx_field<NN>(dev::kFxFieldWarps));
    });
    if (fx_x_any(p) && !fx_lane_length(p.Nx)) {
        const FxFieldLaunch l = fx_field_launch(p.Nx, SIZE_MAX / 4, 1);
        set(dev::k_xc2r_fxany<2>, l.smem); set(dev::k_xc2r_fxany<4>, l.smem); set(dev::k_xc2r_fxany<8>, l.smem);
        set(p.Nx > dev::kFxLateFrom ? dev::k_xr2c_fxany<true> : dev::k_xr2c_fxany<false>, l.smem);
    }
    if (p.fz.N > 0 && !fx_lane_length(p.fz.N)) {
        const size_t inv = dev::smem_fx_any_z(p.fz.N, 4, fx_z_any_warps(p, 4)), two = dev::smem_fx_any_z(p.fz.N, 2, fx_z_any_warps(p, 2));
        if (p.fz.N > dev::kFxLateFrom) {
            set(dev::k_vinv_fxany<true, true>, inv); set(dev::k_vinv_fxany<false, true>, two);
            set(dev::k_vfwd_fxany<true, true>, two); set(dev::k_vfwd_fxany<false, true>, two);
        } else {
            set(dev::k_vinv_fxany<true, false>, inv); set(dev::k_vinv_fxany<false, false>, two);
            set(dev::k_vfwd_fxany<true, false>, two); set(dev::k_vfwd_fxany<false, false>, two);
        }
    }
    WV_FXW_SWITCH(p.fz.N, {
        set(dev::k_vinv_fx<NN, true>, dev::smem_fx_z<NN>(4, 2));
        set(dev::k_vinv_fx<NN, false>, dev::smem_fx_z<NN>(2, 4));
        set(dev::k_vfwd_fx<NN, true>, dev::smem_fx_z<NN>(2, 4));
        set(dev::k_vfwd_fx<NN, false>, dev::smem_fx_z<NN>(2, 4));
    });
    if (fx_x_lane(p)) {
        WV_FXW_SWITCH(p.Nx, {
            using X = XKernels<NN>;
            set(dev::k_xflux_fxco<NN, X::few>, dev::smem_xflux_co<NN>());
            set(dev::k_xflux_fxco<NN, X::all>, dev::smem_xflux_co<NN>());
        });
    }
    else if (fx_x_any(p)) { WV_FXX_SWITCH(p.kxColumns, set(dev::k_xflux_fxany<EK>, fx_x_launch(p, 1).smem)); }
    return e;
}

cudaError_t fx_set_limits_adj(const Plan& p) {
    cudaError_t e = cudaSuccess;
    auto set = [&](auto* kernel, size_t bytes) {
        if (e == cudaSuccess) e = raise_smem_limit(reinterpret_cast<const void*>(kernel), static_cast<int>(bytes));
    };
    WV_FXW_SWITCH(p.fz.N, {
        set(dev::k_vfwd_adj_fx<NN>, dev::smem_fx_z<NN>(2, 4));
        set(dev::k_vinv_adj_fx<NN>, dev::smem_fx_vinv_adj<NN>(2));
    });
    WV_FXW_SWITCH(p.Ny, set(dev::k_yfwd_pair_fx<NN>, dev::smem_fxy<NN>(dev::kFxYWarps * dev::FxW<NN>::lines)));
    if (fx_x_lane(p)) { WV_FXW_SWITCH(p.Nx, set(dev::k_xadj_fx<NN>, dev::smem_xadj_fx<NN>())); }
    return e;
}

bool fx_vfwd_adj(const Plan& p, const dev::DescDev& d, const double* Fpb, const double* Fmb, const double* F0b, double elapsed,
                 double2* zadj, cudaStream_t s) {
    if (!fx_lane_length(p.fz.N)) return false;
    const int sets = fx_z_sets(p, 2);
    WV_FXW_SWITCH(p.fz.N, (dev::k_vfwd_adj_fx<NN><<<cdiv(p.Nkl, sets * dev::FxW<NN>::lines), 64 * sets, dev::smem_fx_z<NN>(2, sets), s>>>(
                              d, Fpb, Fmb, F0b, elapsed, zadj)));
    return true;
}

bool fx_vinv_adj(const Plan& p, const dev::DescDev& d, const double2* fadj, double elapsed, double* Apb, double* Amb,
                 double* A0b, cudaStream_t s) {
    if (!fx_lane_length(p.fz.N)) return false;
    const int sets = fx_z_sets(p, 4);
    WV_FXW_SWITCH(p.fz.N, (dev::k_vinv_adj_fx<NN><<<cdiv(p.Nkl, sets * dev::FxW<NN>::lines), 128 * sets, dev::smem_fx_vinv_adj<NN>(sets), s>>>(
                              d, fadj, elapsed, Apb, Amb, A0b)));
    return true;
}

bool fx_yfwd_pair(const Plan& p, const dev::DescDev& d, const dev::YFwdPairMap& map, const double2* y, int nIn, double2* f,
                  cudaStream_t s) {
    if (!fx_lane_length(p.Ny)) return false;
    const int warps = fx_y_warps(p.Ny, d.kxColumns), cols = warps * static_cast<int>(fx_lane_lines(p.Ny));
    const dim3 grid(cdiv(d.kxColumns, cols), d.zTotal, map.nOut);
    WV_FXW_SWITCH(p.Ny, (dev::k_yfwd_pair_fx<NN><<<grid, 32 * warps, dev::smem_fxy<NN>(cols), s>>>(d, map, y, nIn, f)));
    return true;
}

bool fx_xadj(const Plan& p, const dev::DescDev& d, const FxRows& r, const double2* yadj, double2* yout, const double* rowsIn,
             cudaStream_t s) {
    if (!fx_x_lane(p) || !rowsIn) return false;
    const size_t rows = p.Ny * static_cast<size_t>(d.zTotal), lines = fx_lane_lines(p.Nx);
    WV_FXW_SWITCH(p.Nx, (dev::k_xadj_fx<NN><<<cdiv(rows, lines), 32 * dev::kFxCoWarps, dev::smem_xadj_fx<NN>(), s>>>(
                            d, r.twXLane, yadj, yout, rowsIn)));
    return true;
}

// Against the paired-FP32 kernels, flux in us, paired / fixed point (nonhydrostatic):
// every axis with lane-held lines 16x16x9 64 / 47, 48x48x25 99 / 66, 64x64x33 73 / 73,
// 96x96x49 216 / 187, 128x128x65 328 / 297, 256x256x129 2279 / 2072; run-time stages lose
// (0.6 to 0.8 times as fast).  On small grids whose y and z lines the paired form holds in
// warp registers it wins below 65536 points (32x32x17 42 / 49, 64x32x17 52 / 51,
// 32x32x33 57 / 49), hydrostatic up to twice that (64x64x17 52 / 56, 64x64x33 66 / 68:
// within 8 %, and 1e-16 instead of 1e-12 of error).  Rows of 192 points are 12 a lane at
// two blocks an SM and lose on wide grids (192x96x49 301 / 330, 192x192x97 1024 / 1087);
// y lines of 192 beside other rows would win (96x192x49 409 / 326, 32x192x33 148 / 91).
bool fx_beats_paired(const Plan& p) {
    const bool small = p.Ny % 32 == 0 && p.fz.N % 32 == 0 && p.Nx * p.Ny * p.Nz < 65536;
    return fx_x_lane(p) && fx_lane_length(p.Ny) && fx_lane_length(p.fz.N) && p.Nx != 192 && p.Ny != 192 && !small;
}

bool fx_has_rows(const Plan& p) { return fx_x_lane(p) || fx_x_any(p); }

bool fx_xflux(const Plan& p, const dev::DescDev& d, const FxRows& r, const double2* y, double2* ps,
              unsigned long long* speed, double* physOut, double* advOut, const double* advIn, cudaStream_t s) {
    if (fx_x_lane(p)) {
        const size_t rows = p.Ny * p.Nz * d.members, perWarp = fx_lane_lines(p.Nx);
        const size_t units = (rows + perWarp - 1) / perWarp;
        WV_FXW_SWITCH(p.Nx, {
            using X = XKernels<NN>;
            const bool few = p.kxColumns <= static_cast<size_t>(X::few) * dev::FxW<NN>::G;
            auto* kernel = few ? dev::k_xflux_fxco<NN, X::few> : dev::k_xflux_fxco<NN, X::all>;
            kernel<<<static_cast<unsigned>(units), 32 * dev::kFxCoWarps, dev::smem_xflux_co<NN>(), s>>>(
                d, r.twXLane, y, ps, speed, physOut, advOut, advIn);
        });
        return true;
    }
    if (!fx_x_any(p)) return false;
    const FxXLaunch l = fx_x_launch(p, d.members);
    WV_FXX_SWITCH(p.kxColumns, (dev::k_xflux_fxany<EK><<<l.grid, 32 * l.warps, l.smem, s>>>(
                                   d, r.x, r.twX, y, ps, speed, physOut, advOut, advIn, l.pairs)));
    return true;
}

void fx_yinv(const Plan& p, const dev::DescDev& d, const dev::YInvMap& map, const double2* z, double2* y, cudaStream_t s) {
    const int Ny = static_cast<int>(p.Ny);
    if (!fx_lane_length(p.Ny)) {
        const int cols = dev::fx_any_cols(Ny, d.kxColumns, static_cast<size_t>(d.zTotal) * map.nOut, grid_cap(1));
        auto* kernel = Ny > dev::kFxLateFrom ? dev::k_yinv_fxany<true> : dev::k_yinv_fxany<false>;
        kernel<<<dim3(cdiv(d.kxColumns, cols), d.zTotal, map.nOut), 32 * dev::kFxAnyWarps, dev::smem_fx_any_y(Ny, cols), s>>>(
            d, map, z, y, cols);
        return;
    }
    const int warps = fx_y_warps(p.Ny, d.kxColumns), cols = warps * static_cast<int>(fx_lane_lines(p.Ny));
    const dim3 grid(cdiv(d.kxColumns, cols), d.zTotal, map.nOut);
    double ltop = 0.0;
    for (double l : p.rowL) ltop = std::max(ltop, std::fabs(l));
    uint64_t bits;
    std::memcpy(&bits, &ltop, 8);
    WV_FXW_SWITCH(p.Ny, (dev::k_yinv_fx<NN><<<grid, 32 * warps, dev::smem_fxy<NN>(cols), s>>>(
                            d, map, z, y, static_cast<unsigned>(bits >> 32))));
}

void fx_yfwd(const Plan& p, const dev::DescDev& d, const double2* ps, int nch, double2* f, cudaStream_t s) {
    const int Ny = static_cast<int>(p.Ny);
    if (!fx_lane_length(p.Ny)) {
        const int cols = dev::fx_any_cols(Ny, d.kxColumns, static_cast<size_t>(d.zTotal) * nch, grid_cap(1));
        auto* kernel = Ny > dev::kFxLateFrom ? dev::k_yfwd_fxany<true> : dev::k_yfwd_fxany<false>;
        kernel<<<dim3(cdiv(d.kxColumns, cols), d.zTotal, nch), 32 * dev::kFxAnyWarps, dev::smem_fx_any_y(Ny, cols), s>>>(
            d, ps, nch, f, cols);
        return;
    }
    const int warps = fx_y_warps(p.Ny, d.kxColumns), cols = warps * static_cast<int>(fx_lane_lines(p.Ny));
    const dim3 grid(cdiv(d.kxColumns, cols), d.zTotal, nch);
    WV_FXW_SWITCH(p.Ny, (dev::k_yfwd_fx<NN><<<grid, 32 * warps, dev::smem_fxy<NN>(cols), s>>>(d, ps, nch, f)));
}

bool fx_xc2r(const Plan& p, const dev::DescDev& d, const FxRows& r, const double2* y, int nch, double* fields, cudaStream_t s) {
    if (fx_lane_length(p.Nx)) {
        const FxLaneField l = fx_lane_field(p, d, nch);
        WV_FXW_SWITCH(p.Nx, (dev::k_xc2r_fx<NN><<<l.grid, 32 * l.warps, dev::smem_fx_field<NN>(l.warps), s>>>(
                                d, r.twXLane, y, nch, fields)));
        return true;
    }
    if (p.Nx > 512 || d.kxColumns > 256) return false;
    const FxFieldLaunch l = fx_field_launch(p.Nx, p.Ny * d.zTotal, nch);
    WV_FXX_SWITCH(d.kxColumns, (dev::k_xc2r_fxany<EK><<<l.grid, 32 * l.warps, l.smem, s>>>(d, r.x, r.twX, y, nch, fields)));
    return true;
}

bool fx_xr2c(const Plan& p, const dev::DescDev& d, const FxRows& r, const double* fields, int nch, double2* ps, cudaStream_t s) {
    if (fx_lane_length(p.Nx)) {
        const FxLaneField l = fx_lane_field(p, d, nch);
        WV_FXW_SWITCH(p.Nx, (dev::k_xr2c_fx<NN><<<l.grid, 32 * l.warps, dev::smem_fx_field<NN>(l.warps), s>>>(
                                d, r.twXLane, fields, nch, ps)));
        return true;
    }
    if (p.Nx > 512 || d.kxColumns > 256) return false;
    const FxFieldLaunch l = fx_field_launch(p.Nx, p.Ny * d.zTotal, nch);
    auto* kernel = p.Nx > dev::kFxLateFrom ? dev::k_xr2c_fxany<true> : dev::k_xr2c_fxany<false>;
    kernel<<<l.grid, 32 * l.warps, l.smem, s>>>(d, r.x, r.twX, fields, nch, ps);
    return true;
}

bool fx_vinv(const Plan& p, const dev::DescDev& d, bool flux, double elapsed, const double* Ap, const double* Am,
             const double* A0, double2* z, unsigned long long* speed, cudaStream_t s) {
    if (p.fz.N == 0) return false;
    if (!fx_lane_length(p.fz.N)) {
        const int lines = flux ? 4 : 2, warps = fx_z_any_warps(p, lines);
        const dim3 grid(cdiv(p.Nkl, warps), d.members);
        const size_t sm = dev::smem_fx_any_z(p.fz.N, lines, warps);
        const bool late = p.fz.N > dev::kFxLateFrom;
        auto* kernel = flux ? (late ? dev::k_vinv_fxany<true, true> : dev::k_vinv_fxany<true, false>)
                            : (late ? dev::k_vinv_fxany<false, true> : dev::k_vinv_fxany<false, false>);
        kernel<<<grid, 32 * warps, sm, s>>>(d, Ap, Am, A0, elapsed, z, speed);
        return true;
    }
    const int lines = flux ? 4 : 2, sets = fx_z_sets(p, lines), warps = sets * lines;
    const dim3 grid(cdiv(p.Nkl, sets * fx_lane_lines(p.fz.N)), d.members);
    WV_FXW_SWITCH(p.fz.N, {
        const size_t sm = dev::smem_fx_z<NN>(lines, sets);
        if (flux) dev::k_vinv_fx<NN, true><<<grid, 32 * warps, sm, s>>>(d, Ap, Am, A0, elapsed, z, speed);
        else dev::k_vinv_fx<NN, false><<<grid, 32 * warps, sm, s>>>(d, Ap, Am, A0, elapsed, z, speed);
    });
    return true;
}

bool fx_vfwd(const Plan& p, const dev::DescDev& d, bool flux, const double2* f, int nch, double elapsed, const double* Ap,
             const double* Am, const double* A0, const unsigned long long* speed, int damping, double* Fp, double* Fm,
             double* F0, cudaStream_t s) {
    if (p.fz.N == 0) return false;
    if (!fx_lane_length(p.fz.N)) {
        const int warps = fx_z_any_warps(p, 2);
        const dim3 grid(cdiv(p.Nkl, warps), d.members);
        const size_t sm = dev::smem_fx_any_z(p.fz.N, 2, warps);
        const bool late = p.fz.N > dev::kFxLateFrom;
        auto* kernel = flux ? (late ? dev::k_vfwd_fxany<true, true> : dev::k_vfwd_fxany<true, false>)
                            : (late ? dev::k_vfwd_fxany<false, true> : dev::k_vfwd_fxany<false, false>);
        kernel<<<grid, 32 * warps, sm, s>>>(d, f, nch, elapsed, Ap, Am, A0, speed, damping, Fp, Fm, F0);
        return true;
    }
    const int sets = fx_z_sets(p, 2), warps = 2 * sets;
    const dim3 grid(cdiv(p.Nkl, sets * fx_lane_lines(p.fz.N)), d.members);
    WV_FXW_SWITCH(p.fz.N, {
        const size_t sm = dev::smem_fx_z<NN>(2, sets);
        if (flux)
            dev::k_vfwd_fx<NN, true><<<grid, 32 * warps, sm, s>>>(d, f, nch, elapsed, Ap, Am, A0, speed, damping, Fp, Fm, F0);
        else
            dev::k_vfwd_fx<NN, false><<<grid, 32 * warps, sm, s>>>(d, f, nch, elapsed, Ap, Am, A0, speed, damping, Fp, Fm, F0);
    });
    return true;
}

}  // namespace wvgpu

namespace wvgpu {

// The dynamic shared-memory cap is a process-wide attribute of each kernel, not of
// a handle: only ever raise it, so a handle created for a smaller grid cannot shrink
// the cap below what a live handle for a larger grid launches with.
cudaError_t raise_smem_limit(const void* kernel, int bytes) {
    static std::mutex mutex;
    std::lock_guard<std::mutex> lock(mutex);
    cudaFuncAttributes a{};
    cudaError_t e = cudaFuncGetAttributes(&a, kernel);
    if (e != cudaSuccess) return e;
    if (a.maxDynamicSharedSizeBytes >= bytes) return cudaSuccess;
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}

}  // namespace wvgpu
