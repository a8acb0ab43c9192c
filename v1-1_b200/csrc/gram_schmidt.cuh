// Coefficients of a modified Gram-Schmidt step from one pass of dots, shared by the A-vector's
// and the orbitals' Krylov kernels.
#pragma once

namespace sincgpu {

// With r_i = <v_i, p> and L_ik = <v_i, v_k> (k < i), the coefficients h of the sequential
// projections solve (I + L) h = r.  L, the vectors' loss of orthogonality, is not small in
// general: modified Gram-Schmidt loses it as the Krylov space comes to hold the solution of
// A x = v_0, and in a chain of thirty A-vectors (mean energy ten times its spread) |L| grows
// from rounding to 1e-3 .. 0.9.  So nothing is cut after a power of L: T = (I + L)^-1 is kept
// row by row (its part below the diagonal), as in the inverse compact WY form of Swirydowicz
// et al., and h = T r.  Rows i < j are ready, row j of h is r_j - L_j h (gs_solve), and row j of
// T, -L_j T, is formed for the later steps (gs_extend), which the rest of this one need not
// wait for (A-vector step of 3136 determinants 522 us; 529 with it in front of the projections).

// r(i), l(k): <v_i, p> and <v_j, v_k>; t(i, k): row i < j of T.  h, part: shared memory, j <
// 128, one value per warp (nothing else writes it before the CTA's next barrier).  Called by a
// whole CTA of NW warps; h[0 .. j - 1] are there after it and every thread gets h_j.
template <int NW, class R, class L, class T>
__device__ __forceinline__ double gs_solve(int j, double* h, double* part, R r, L l, T t) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double s = 0.0;  // this warp's part of L_j h
  for (int i = warp; i < j; i += NW) {
    double a = 0.0;
    for (int k = lane; k < i; k += 32) a = fma(t(i, k), r(k), a);
    for (int o = 16; o > 0; o >>= 1) a += __shfl_down_sync(0xffffffffu, a, o);
    if (lane == 0) {
      a += r(i);
      h[i] = a;
      s = fma(l(i), a, s);
    }
  }
  if (lane == 0) part[warp] = s;
  __syncthreads();
  double b[4] = {r(j), 0.0, 0.0, 0.0};
#pragma unroll
  for (int w = 0; w < NW; ++w) b[w & 3] -= part[w];
  return (b[0] + b[1]) + (b[2] + b[3]);
}

// put(k, v): element k of row j of T, for k = k0, k0 + kstep, ... < j (the CTAs share them)
template <class L, class T, class PUT>
__device__ __forceinline__ void gs_extend(int j, L l, T t, int k0, int kstep, PUT put) {
  const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  for (int k = k0 + (int)(threadIdx.x >> 5) * kstep; k < j; k += nw * kstep) {
    double a = 0.0;
    for (int m = k + 1 + lane; m < j; m += 32) a = fma(l(m), t(m, k), a);
    for (int o = 16; o > 0; o >>= 1) a += __shfl_down_sync(0xffffffffu, a, o);
    if (lane == 0) put(k, -(l(k) + a));
  }
}

}  // namespace sincgpu
