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
// et al., and h = T r.  Rows i < j are ready, row j of h is r_j - L_j h, and row j of T,
// -L_j T, is formed beside them for the later steps.
//
// r(i), l(k): <v_i, p> and <v_j, v_k>; t(i, k): row i < j of T; put(k, v): element k of its
// row j, for k = k0, k0 + kstep, ... < j (the CTAs share them).  h: shared memory, j < 128.
// Called by a whole CTA; h[0 .. j - 1] are there after it and every thread gets h_j.
template <class R, class L, class T, class PUT>
__device__ __forceinline__ double gs_coefficients(int j, double* h, R r, L l, T t, int k0, int kstep, PUT put) {
  const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const int nk = k0 < j ? (j - k0 + kstep - 1) / kstep : 0;
  for (int w = threadIdx.x >> 5; w < j + nk; w += nw) {
    double a = 0.0;
    const int k1 = w < j ? 0 : k0 + (w - j) * kstep;
    if (w < j)
      for (int k = lane; k < w; k += 32) a = fma(t(w, k), r(k), a);
    else
      for (int m = k1 + 1 + lane; m < j; m += 32) a = fma(l(m), t(m, k1), a);
    for (int o = 16; o > 0; o >>= 1) a += __shfl_down_sync(0xffffffffu, a, o);
    if (lane == 0) {
      if (w < j) h[w] = r(w) + a;
      else put(k1, -(l(k1) + a));
    }
  }
  __syncthreads();
  double a = 0.0;  // every warp for itself
  for (int k = lane; k < j; k += 32) a = fma(l(k), h[k], a);
  for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
  return r(j) - a;
}

}  // namespace sincgpu
