// Explicit instantiations of the half-length Coulomb passes for a group of lengths
// (split across files so that nvcc compiles them in parallel).
#include "coulomb_half.cuh"
namespace sincgpu {
SINCGPU_HALF_INSTANTIATE(7, 9)
SINCGPU_HALF_INSTANTIATE(8, 8)
}  // namespace sincgpu
