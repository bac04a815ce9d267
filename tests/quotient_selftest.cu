// Device entry point of tests/test_quotients.py: the branch-free reciprocal and
// quotients of the fit kernels beside the division operator.
#include "../periodsearch_b200/csrc/ps_fit_common.cuh"

namespace {

__global__ void quotients(const double* a, const double* d, int n, double* out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const psb::fitcommon::QuotientsBy by(d[i]);
    out[i] = psb::fitcommon::plain_numerator(a[i]) ? by.of(a[i]) : by.of_any(a[i]);
    out[n + i] = a[i] / d[i];
    out[2 * n + i] = by.y;
    out[3 * n + i] = 1.0 / d[i];
    out[4 * n + i] = psb::fitcommon::rcp_newton(d[i]);
}

}  // namespace

// out: quotient, a / d, reciprocal, 1 / d, Newton reciprocal, n values each
extern "C" int quotient_selftest(const double* a, const double* d, int n, double* out) {
    double* buf = nullptr;
    if (n <= 0 || cudaMalloc(&buf, sizeof(double) * 7 * (size_t)n) != cudaSuccess) return -1;
    cudaMemcpy(buf, a, sizeof(double) * n, cudaMemcpyHostToDevice);
    cudaMemcpy(buf + n, d, sizeof(double) * n, cudaMemcpyHostToDevice);
    quotients<<<(n + 255) / 256, 256>>>(buf, buf + n, n, buf + 2 * (size_t)n);
    const cudaError_t e = cudaMemcpy(out, buf + 2 * (size_t)n, sizeof(double) * 5 * (size_t)n, cudaMemcpyDeviceToHost);
    cudaFree(buf);
    return e == cudaSuccess ? 0 : -2;
}
