// gs_fft.h -- FP64 convolution of a real periodic mesh (k_fft.cu).
#pragma once

#include "gs_internal.h"

namespace gs {

// Mesh sizes that convolve_mesh takes.
bool convolve_supports(int g);

// Twiddle factors exp(-2 pi i k / g), k < g, for convolve_mesh.
ErrorStatus convolve_table(int g, double2 *tw, cudaStream_t s);

// The factor of a deposited mesh that makes it a density in units of the mean:
// *device where that is set, else value.
struct MeshScale {
    const double *device;
    double value;
};

#ifdef __CUDACC__
// Density contrast of a cell: density times scale, less one, rounded once.
__device__ __forceinline__ double contrast(double density, double scale)
{
    return fma(density, scale, -1.0);
}
#endif

// mesh [g^3] <- g^3 times the convolution of its contrast() with the kernel whose
// transform is the real table[kx^2 + ky^2 + kz^2] (|k| at most g / 2 on each axis),
// in place.
ErrorStatus convolve_mesh(double *mesh, int g, const MeshScale &scale, const double *table,
                          const double2 *tw, cudaStream_t s);

constexpr int kConvolveLaunches = 5;

}  // namespace gs
