// Maxwell TM-RZ field update on the device (I/RreaMaxwellTMRZ.H:147-228),
// composed as the Maxwell part of RreaAmrexAdvance::AdvanceOneStep
// (S/RreaAmrexAdvance.cpp:690-780): restagger B by (dt - dt_sub)/2, then per
// material substep B, Silver-Mueller, E with the face current, then restagger
// back and Silver-Mueller.
//
// The grids stay in L2 (84 MB of vectors on the largest, 512 x 4096), so what
// bounds these kernels is the FP64 pipe (2 multiply-adds per clock per SM),
// and on it a division costs ten multiply-adds.  Hence every quotient is a
// product with a reciprocal and one residual correction (`exact_quot`, three
// operations, the rounding of the division itself), the constants come from
// the host, and a thread owns one column index i over several rows: the
// reciprocal of (i + 1/2) dr is formed once, and the row below is already in
// registers.  B, its restagger and the open faces are one launch: the two B
// updates read the same E, and the faces only E.
// Measured on 512 x 4096: ten updates of two substeps with the upload and
// download of the vectors and the particle diagnostics 16.0 -> 6.6 ms.
#include "rrea_kernels.h"
#include "device/rrea_exact_quot.cuh"

#include <cuda_runtime.h>

namespace rrea_dev {
namespace {

constexpr double kEps0 = 8.8541878128e-12;
constexpr double kMu0 = 1.25663706212e-6;
constexpr double kCLight = 299792458.0;

__device__ __forceinline__ size_t er_at(int nr, int i, int j)
{
    return static_cast<size_t>(i) + static_cast<size_t>(nr + 1) * j;
}
__device__ __forceinline__ size_t ez_at(int nr, int i, int j)
{
    return static_cast<size_t>(i) + static_cast<size_t>(nr) * j;
}

// dBtheta/dt = dEz/dr - dEr/dz at the interior corners, over dt_a and (when
// twice) again over dt_b, and with open_faces the Silver-Mueller boundary
// corners; where the reference's passes overlap the later pass wins: axis,
// then the z rows, then the outer column.
__global__ void __launch_bounds__(256) advance_b_kernel(int nr, int nz, ExactDivisor dr, ExactDivisor dz, double dt_a,
                                                        double dt_b, bool twice, bool open_faces, int rows,
                                                        const double* __restrict__ er, const double* __restrict__ ez,
                                                        double* __restrict__ bt)
{
    int const i = blockIdx.x * 32 + threadIdx.x;
    if (i > nr) return;
    int const j0 = (blockIdx.y * 8 + threadIdx.y) * rows;
    int const j1 = min(j0 + rows, nz + 1);
    bool const inner = i > 0 && i < nr;
    double below = inner && j0 > 0 && j0 < nz ? er[er_at(nr, i, j0 - 1)] : 0.0;
    for (int j = j0; j < j1; ++j) {
        size_t const c = er_at(nr, i, j);
        if (inner && j > 0 && j < nz) {
            double const here = er[c];
            double const curl = exact_quot(ez[ez_at(nr, i, j)] - ez[ez_at(nr, i - 1, j)], dr)
                - exact_quot(here - below, dz);
            below = here;
            double b = bt[c] + dt_a * curl;
            if (twice) b += dt_b * curl;
            bt[c] = b;
            continue;
        }
        if (inner && j == 0) below = er[c];
        if (!open_faces) continue;
        if (i == 0) bt[c] = 0.0;
        else if (j == 0) bt[c] = -er[er_at(nr, i, 0)] / kCLight;
        else if (j == nz) bt[c] = er[er_at(nr, i, nz - 1)] / kCLight;
        else bt[c] = -ez[ez_at(nr, nr - 1, j)] / kCLight;
    }
}

// Ampere with the face current, no conductivity: Er on radial faces (axis
// face pinned to 0), Ez on axial faces.  c2dt = dt / (eps0 mu0), dte = dt /
// eps0.
__global__ void __launch_bounds__(256) advance_e_kernel(int nr, int nz, double dr, ExactDivisor dz, double c2dt,
                                                        double dte, int rows, const double* __restrict__ bt,
                                                        const double* __restrict__ jr, const double* __restrict__ jz,
                                                        double* __restrict__ er, double* __restrict__ ez)
{
    int const i = blockIdx.x * 32 + threadIdx.x;
    if (i > nr) return;
    int const j0 = (blockIdx.y * 8 + threadIdx.y) * rows;
    int const j1 = min(j0 + rows, nz + 1);
    if (j0 >= j1) return;
    double const fi = i, fi1 = i + 1;
    double const radius = (fi + 0.5) * dr;
    ExactDivisor const rad = exact_divisor(radius);
    double here = bt[er_at(nr, i, j0)];
    for (int j = j0; j < j1; ++j) {
        double const above = j < nz ? bt[er_at(nr, i, j + 1)] : 0.0;
        if (j < nz) {
            size_t const face = er_at(nr, i, j);
            double drive = exact_quot(-c2dt * (above - here), dz);
            drive -= dte * jr[face];
            er[face] = i == 0 ? 0.0 : er[face] + drive;
        }
        if (i < nr) {
            size_t const face = ez_at(nr, i, j);
            double drive = exact_quot(c2dt * (fi1 * bt[er_at(nr, i + 1, j)] - fi * here), rad);
            drive -= dte * jz[face];
            ez[face] += drive;
        }
        here = above;
    }
}

// Rows per thread: up to eight, while the grid still gives every SM its
// resident threads (below that the rows' serial chain costs more than the
// reciprocal it saves), and as many as a launch's second dimension needs to
// reach the last row (65,535 blocks of 8 threads).
int rows_for(int nr, int nz, int num_threads)
{
    int64_t const rows = static_cast<int64_t>(nr + 1) * (nz + 1) / num_threads;
    int64_t const least = (static_cast<int64_t>(nz) + 65535 * 8) / (65535 * 8);
    int64_t const good = rows < 1 ? 1 : (rows > 8 ? 8 : rows);
    return static_cast<int>(good > least ? good : least);
}

dim3 grid_for(int nr, int nz, int rows)
{
    return dim3(static_cast<unsigned>(nr / 32 + 1), static_cast<unsigned>((nz + 1 + 8 * rows - 1) / (8 * rows)));
}

constexpr int kFieldThreads = 152 * 1024;   // a GB300's SMs by half of an SM's threads

}  // namespace
}  // namespace rrea_dev

namespace rrea_launch {

cudaError_t maxwell_advance_b(int nr, int nz, double dr, double dz, double dt_a, double dt_b, bool twice,
                              bool open_faces, const double* er, const double* ez, double* bt, cudaStream_t stream)
{
    using namespace rrea_dev;
    note_launch();
    int const rows = rows_for(nr, nz, kFieldThreads);
    advance_b_kernel<<<grid_for(nr, nz, rows), dim3(32, 8), 0, stream>>>(nr, nz, exact_divisor(dr),
                                                                         exact_divisor(dz), dt_a, dt_b, twice,
                                                                         open_faces, rows, er, ez, bt);
    return cudaGetLastError();
}

cudaError_t maxwell_advance_e(int nr, int nz, double dr, double dz, double dt, const double* bt, const double* jr,
                              const double* jz, double* er, double* ez, cudaStream_t stream)
{
    using namespace rrea_dev;
    note_launch();
    int const rows = rows_for(nr, nz, kFieldThreads);
    advance_e_kernel<<<grid_for(nr, nz, rows), dim3(32, 8), 0, stream>>>(nr, nz, dr, exact_divisor(dz),
                                                                         dt / (kEps0 * kMu0), dt / kEps0, rows, bt, jr,
                                                                         jz, er, ez);
    return cudaGetLastError();
}

cudaError_t maxwell_step(int nr, int nz, double dr, double dz, double dt, int substeps, double* er, double* ez,
                         double* bt, const double* jr, const double* jz, cudaStream_t stream)
{
    double const dts = dt / static_cast<double>(substeps);
    double const restagger = 0.5 * (dt - dts);
    cudaError_t e = cudaSuccess;
    for (int k = 0; k < substeps && e == cudaSuccess; ++k) {
        // the first substep's B carries the restagger: both read this E
        e = k == 0 ? maxwell_advance_b(nr, nz, dr, dz, restagger, dts, true, true, er, ez, bt, stream)
                   : maxwell_advance_b(nr, nz, dr, dz, dts, 0.0, false, true, er, ez, bt, stream);
        if (e == cudaSuccess) e = maxwell_advance_e(nr, nz, dr, dz, dts, bt, jr, jz, er, ez, stream);
    }
    if (e != cudaSuccess) return e;
    return maxwell_advance_b(nr, nz, dr, dz, -restagger, 0.0, false, true, er, ez, bt, stream);
}

}  // namespace rrea_launch
