// Two DCT passes per launch on the tensor cores -- see pair_transform.cu.
#pragma once

#include "umma_transform.cuh"

namespace binder {

// Two consecutive passes of the DCT-prior M-step with the field between them kept on chip.
enum PairKind : int {
    kPairForward = 0,   // forward along z, then y, of one (y, z) plane
    kPairSpectral = 1,  // forward along x, prior scaling (+ noise, costs), inverse along x
    kPairInverse = 2,   // inverse along y, then z, of one (y, z) plane; voxel positions added
};

// Whether the pair kernels take an nx x ny x nz volume (nz == 1: an image, kPairSpectral only):
// BF16 operands, every axis at most 256 long (the MMA's N) and the tiles within shared memory.  With
// the split that leaves out planes of about 241 x 81 and more, and 209 x 128 to 241 x 96 either way
// round; their volumes take the per-axis passes.
bool pair_supported(int nx, int ny, int nz, int planes);

// One pair over `ncomp` components of a volume; `a` as for launch_axis_pass_tc (in, out, D, st,
// sigma2, sample, noise, ..., xpos, skip, chain_comps; a.out may be a.in for kPairSpectral).
// M1, M2: the first and the second pass's matrices.  planes 2: BF16 hi / lo split, three products
// per element in the order of the per-axis passes (the results are theirs bit for bit); planes 1:
// one BF16 product.
void launch_pair_pass(const AxisArgs<float> &a, PairKind kind, int nx, int ny, int nz,
                      const UmmaMatrix &M1, const UmmaMatrix &M2, int ncomp, int planes,
                      cudaStream_t s);

}  // namespace binder
