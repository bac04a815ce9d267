// Matrix-free chi2 gradient and Gauss-Newton products (ps_adjoint.cu).
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>

#include "ps_device.hpp"

namespace psb {

constexpr int kAdjMaxMa = 96;  // parameters at most (88 shape coefficients + 8)
constexpr int kAdjDirs = 8;    // directions of one batched product

// What a call brings along, passed to the first kernel by value.
struct AdjArgs {
    double a[kAdjMaxMa];  // parameters
    double v[kAdjMaxMa];  // one direction over all parameters (zero on fixed ones)
    int unit[kAdjDirs];   // batched: direction d is this parameter's unit vector (-1: zero)
};

enum AdjMode {
    kAdjGradient,  // beta = J^T W (y_obs - y)
    kAdjProduct,   // J^T W (J v)
    kAdjUnits      // J^T W (J e) for kAdjDirs unit vectors e
};

// Doubles of work memory of a gradient or product; batched: of those and a batch
// of kAdjDirs products, about twice as many.
size_t adjoint_work_doubles(const DevProblem& P, bool batched);
// Scalars of the last evaluation at work: the convexity residuals chck (3) at
// kAdjMiscChk, the facet-area sum after them.
constexpr int kAdjMiscChk = 33;
constexpr int kAdjMiscSarea = 36;
// Kernel launches of one launch_adjoint call.
inline int adjoint_launches(const DevProblem& P) { return P.n_ablocks > 0 ? 7 : 6; }
// chi2 into d_chi2; the result over the free parameters into d_out (mfit
// values, kAdjDirs times mfit for kAdjUnits).
cudaError_t launch_adjoint(const DevProblem& P, const DevProblem* dP, double* work, const AdjArgs& args, AdjMode mode,
                           double* d_out, double* d_chi2, cudaStream_t s);

}  // namespace psb
