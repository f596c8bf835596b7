// Launchers of the FP64 kernels on fixed-point lines (wv_fx.cu).  The bool ones
// return false, launching nothing, where the plan's length has no such kernel.
#pragma once

#include "wv_kernels.cuh"
#include "wv_plan.hpp"

#include <cuda_runtime.h>
#include <vector>

namespace wvgpu {

// Tables of the x pass: run-time stages (any length) and stage order (lane-held).
struct FxRows {
    dev::FFTDev x;
    const dev::fxw* twX;
    const dev::fxw* twXLane;
};

// Stage twiddles of a lane-held line of N points; empty where there is none.
std::vector<int32_t> fx_lane_table(size_t N);
// Shared-memory limits of every kernel a handle of this plan launches.
cudaError_t fx_set_limits(const Plan& p);

// Whether the fixed-point kernels beat the paired-FP32 ones of FP32X2 handles.
bool fx_beats_paired(const Plan& p);
// Whether fx_xflux serves the plan's rows.
bool fx_has_rows(const Plan& p);
bool fx_xflux(const Plan& p, const dev::DescDev& d, const FxRows& rows, const double2* y, double2* ps,
              unsigned long long* speed, double* physOut, double* advOut, const double* advIn, cudaStream_t s);
bool fx_xc2r(const Plan& p, const dev::DescDev& d, const FxRows& rows, const double2* y, int nch, double* fields,
             cudaStream_t s);
bool fx_xr2c(const Plan& p, const dev::DescDev& d, const FxRows& rows, const double* fields, int nch, double2* ps,
             cudaStream_t s);
void fx_yinv(const Plan& p, const dev::DescDev& d, const dev::YInvMap& map, const double2* z, double2* y, cudaStream_t s);
void fx_yfwd(const Plan& p, const dev::DescDev& d, const double2* ps, int nch, double2* f, cudaStream_t s);
bool fx_vinv(const Plan& p, const dev::DescDev& d, bool flux, double elapsed, const double* Ap, const double* Am,
             const double* A0, double2* z, unsigned long long* speed, cudaStream_t s);
bool fx_vfwd(const Plan& p, const dev::DescDev& d, bool flux, const double2* f, int nch, double elapsed, const double* Ap,
             const double* Am, const double* A0, const unsigned long long* speed, int damping, double* Fp, double* Fm,
             double* F0, cudaStream_t s);

// The flux VJP's passes (fx_xadj: on kept rows of the x pass).
cudaError_t fx_set_limits_adj(const Plan& p);
bool fx_vfwd_adj(const Plan& p, const dev::DescDev& d, const double* Fpb, const double* Fmb, const double* F0b, double elapsed,
                 double2* zadj, cudaStream_t s);
bool fx_xadj(const Plan& p, const dev::DescDev& d, const FxRows& rows, const double2* yadj, double2* yout,
             const double* rowsIn, cudaStream_t s);
bool fx_yfwd_pair(const Plan& p, const dev::DescDev& d, const dev::YFwdPairMap& map, const double2* y, int nIn, double2* f,
                  cudaStream_t s);
bool fx_vinv_adj(const Plan& p, const dev::DescDev& d, const double2* fadj, double elapsed, double* Apb, double* Amb,
                 double* A0b, cudaStream_t s);

}  // namespace wvgpu
