// FP64 Hartley passes of the topology correction's Poisson solve -- see hartley.cu.
#pragma once

#include "common.cuh"

namespace binder {

// The cosine and sine halves of an n-point Hartley transform on the device, rows k = 0 .. n/2 and
// columns j = 0 .. n/2, padded with zeros to multiples of 8 and 4: cos at dev, sin after it.
struct HartleyMatrix {
    int n = 0, rows = 0, cols = 0;  // padded rows and columns
    double *dev = nullptr;
    void init(int n, cudaStream_t s);  // from the stream-ordered pool; synchronises
    void release(cudaStream_t s);
};

enum HartleyMode : int {
    kHartleyPlain = 0,    // y = H x
    kHartleyScaled = 1,   // y = (H x) * out_scale + sums / count, per component
    kHartleyPoisson = 2,  // y = H (-(H x) / (lambda V)) along the outermost axis (outer == 1)
};

struct HartleyArgs {
    const double *in;
    double *out;
    long V;            // elements between components
    long outer, s;     // element (o, j, t) of the axis at o * n * s + j * s + t
    int nz;            // kHartleyPoisson: t = ky * nz + kz
    const double *cos_x, *cos_y, *cos_z;  // cos(2 pi k / n) per axis
    double out_scale[3];
    const double *sums;  // on the device: the offset is a mean that no host needs to know
    double count;
};

// One pass over `ncomp` components along the axis of H (at most 256 long).
void launch_hartley(const HartleyArgs &a, const HartleyMatrix &H, HartleyMode mode, int ncomp,
                    cudaStream_t s);

}  // namespace binder
