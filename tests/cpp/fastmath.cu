// Evaluates the table-driven functions of device/rrea_fastmath.cuh and the
// quotient of device/rrea_exact_quot.cuh on arrays, beside CUDA's, for
// tests/test_gpu_fastmath.py.
#include "../../rrea_feedback_warpx_amrex_geant4_gb300/csrc/device/rrea_exact_quot.cuh"
#include "../../rrea_feedback_warpx_amrex_geant4_gb300/csrc/device/rrea_fastmath.cuh"

using namespace rrea_dev;

namespace {

__global__ void eval(int which, const double* arena, const double* x, const double* y, int n, double* out, double* out2)
{
    int const i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double a = 0.0, b = 0.0;
    switch (which) {
    case 0: a = frsqrt(x[i]); b = rsqrt(x[i]); break;
    case 1: a = rrea_dev::fsqrt(x[i]); b = sqrt(x[i]); break;
    case 2: fsincos(arena, x[i], a, b); break;
    case 3: sincos(x[i], &a, &b); break;
    case 4: sincos_turn(arena, x[i], a, b); break;
    case 5: a = fatan2(arena, y[i], x[i]); b = atan2(y[i], x[i]); break;
    case 6: a = exact_quot(x[i], exact_divisor(y[i])); b = x[i] / y[i]; break;
    default: break;
    }
    out[i] = a;
    out2[i] = b;
}

}  // namespace

// x, y, out and out2 are host arrays of n; arena is the loaded arena's first
// doubles (the constant tables).  Returns 0, or a CUDA error.
extern "C" int fastmath_eval(int which, const double* arena, int arena_n, const double* x, const double* y, int n,
                             double* out, double* out2)
{
    double* d = nullptr;
    size_t const total = static_cast<size_t>(arena_n) + 4 * static_cast<size_t>(n);
    cudaError_t e = cudaMalloc(reinterpret_cast<void**>(&d), total * sizeof(double));
    if (e != cudaSuccess) return static_cast<int>(e);
    double* const dx = d + arena_n;
    size_t const bytes = static_cast<size_t>(n) * sizeof(double);
    e = cudaMemcpy(d, arena, static_cast<size_t>(arena_n) * sizeof(double), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(dx, x, bytes, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(dx + n, y, bytes, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        eval<<<(n + 127) / 128, 128>>>(which, d, dx, dx + n, n, dx + 2 * static_cast<size_t>(n),
                                       dx + 3 * static_cast<size_t>(n));
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(out, dx + 2 * static_cast<size_t>(n), bytes, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(out2, dx + 3 * static_cast<size_t>(n), bytes, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return static_cast<int>(e);
}
