// Orbital right-hand side (MCTDH.SRC/derivs.f90:629-852, actreduced00) for the sinc
// project (numr=1, bondpoints=1, nonuc_checkflag=1, no frozen core):
//   Y      = phi x denmat                                   (lines 674-676)
//   S      = KE(Y) + pot*Y + E_z(t) z*Y                     (lines 712-752)
//   S     += sum_k reducedpot(:,k,i) phi_k                  (line 763, mult_reducedpot)
//   S      = timefac * S x invdenmat        (dentimeflag)   (lines 788-790)
//   out    = S - proj x <proj|S>            (projflag)      (lines 806-807, project00)
// Kernels: mix and projector subtraction (lin_kernel, FP64 tensor cores), KE (ke.cu,
// fused pot/pulse), reducedpot apply + invdenmat mix (one pass over reducedpot, the
// dominant HBM stream), projector dots (FP64 tensor cores, split-K, deterministic).
//
// The other per-point kernels work on tiles of 32 consecutive grid points (one per
// lane) by all orbitals: each warp handles a subset of output orbitals, reads
// every (orbital, tile) row as one coalesced 512-byte segment, and the small
// per-point vectors (phi, the partial sums) and n x n matrices sit in shared
// memory, so no thread keeps an n-vector in registers.
#include <algorithm>
#include "context.hpp"
#include "dmma.cuh"

namespace sincgpu {

constexpr int TXO = 32;          // grid points per tile (lanes)
constexpr int kMaxOrbRhs = 32;   // largest orbital count of these kernels
constexpr int kRhsSmemMax = 64 * 1024;

// out(x,i) = [base(x,i)] + sgn sum_s sum_j src_s(x,j) mat_s(j,i), s < NS (column-major n x n
// complex matrices): the mix with denmat or an overlap's root, the projection and the
// Jacobian's combination, as products of a G x 2n by a 2n x 2n real matrix on the FP64
// tensor cores (complex entries as 2 x 2 real blocks).  A warp owns LMT x 8 points and all
// 2n columns (NT fragments of 8 = 4 orbitals).  Fragments of src come straight from
// global memory (lanes = 8 points x (2 orbitals, re/im): whole lines), all of a source
// in flight together; the matrices sit in shared memory in fragment order, read once
// per warp.  Bound by HBM: 16 G n (NS + 1 or 2) bytes, 3.4 to 7 us at 41^3 / 10 orbitals.
// The per-point form (one lane per point, matrix and tile read from shared memory for
// every product) was bound by shared-memory reads: mix 11.3 -> 8.5, projection 12.6 ->
// 8.5, Jacobian's combination 18.3 -> 14.2 us there (cold caches).
constexpr int LMT = 2;            // fragments of 8 points per warp
constexpr int kLinWarps = 8;
template <int NS, int NT>
__global__ void __launch_bounds__(32 * kLinWarps) lin_kernel(const double2* base,
                                                             const double2* src0,
                                                             const double2* mat0,
                                                             const double2* src1,
                                                             const double2* mat1, double sgn, int n,
                                                             long long G, double2* out) {
  constexpr int KS = 2 * NT;  // K steps of 4 = 2 orbitals
  extern __shared__ double lsm[];  // [NS][KS][NT][32]
  grid_dependency_wait();
  grid_dependents_launch();
  const int tid = threadIdx.x, lane = tid & 31, g = lane >> 2, t = lane & 3;
  for (int e = tid; e < NS * KS * NT * 32; e += blockDim.x) {
    const int l = e & 31, nt = (e >> 5) % NT, ks = (e >> 5) / NT % KS, s = (e >> 5) / (NT * KS);
    const int j = 2 * ks + ((l & 3) >> 1), i = 4 * nt + (l >> 3), cj = l & 1, ci = (l >> 2) & 1;
    double v = 0.0;
    if (j < n && i < n) {
      const double2 m = (s ? mat1 : mat0)[j + n * i];
      v = cj == ci ? m.x : (cj ? -m.y : m.y);
    }
    lsm[e] = sgn * v;
  }
  const long long x0 = (blockIdx.x * (long long)kLinWarps + (tid >> 5)) * (8 * LMT) + g;
  double acc[LMT][NT][2];
#pragma unroll
  for (int m = 0; m < LMT; ++m)
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      const long long x = x0 + 8 * m;
      const int i = 4 * nt + t;
      const double2 b = base && x < G && i < n ? base[(long long)i * G + x] : make_double2(0.0, 0.0);
      acc[m][nt][0] = b.x;
      acc[m][nt][1] = b.y;
    }
  double a[KS][LMT];
#pragma unroll
  for (int s = 0; s < NS; ++s) {
    const double* src = reinterpret_cast<const double*>(s ? src1 : src0) + (t & 1);
#pragma unroll
    for (int ks = 0; ks < KS; ++ks)
#pragma unroll
      for (int m = 0; m < LMT; ++m) {
        const long long x = x0 + 8 * m;
        const int j = 2 * ks + (t >> 1);
        a[ks][m] = j < n && x < G ? src[2 * ((long long)j * G + x)] : 0.0;
      }
    if (s == 0) __syncthreads();  // the matrices
#pragma unroll
    for (int ks = 0; ks < KS; ++ks) {
      if (2 * ks >= n) break;
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        const double b = lsm[((s * KS + ks) * NT + nt) * 32 + lane];
#pragma unroll
        for (int m = 0; m < LMT; ++m) dmma_884(acc[m][nt], a[ks][m], b);
      }
    }
  }
#pragma unroll
  for (int m = 0; m < LMT; ++m)
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      const long long x = x0 + 8 * m;
      const int i = 4 * nt + t;
      if (x < G && i < n) out[(long long)i * G + x] = make_double2(acc[m][nt][0], acc[m][nt][1]);
    }
}

// s_i = acc(x,i) + sum_k V(x,k,i) phi_k(x) over i in [i0, i0+ni); then, when
// `dentime`, t_i = timefac * sum_j s_j inv(j,i) (all n orbitals present).
__global__ void __launch_bounds__(TXO * kMaxOrbRhs) redpot_kernel(const double2* phi,
                                                           const double2* V,
                                                           const double2* acc_in,
                                                           const double2* inv, double2 timefac,
                                                           int n, int i0, int ni, int dentime, long long G,
                                                           double2* out) {
  extern __shared__ double2 rsm[];
  grid_dependency_wait();
  grid_dependents_launch();
  double2* sinv = rsm;                 // n*n (dentime)
  double2* sph = rsm + n * n;          // n x TXO
  double2* ss = sph + n * TXO;         // n x TXO (dentime)
  const int lx = threadIdx.x, ty = threadIdx.y, tid = ty * TXO + lx;
  if (dentime)
    for (int e = tid; e < n * n; e += TXO * blockDim.y) sinv[e] = inv[e];
  const long long x = blockIdx.x * (long long)TXO + lx;
  const bool ok = x < G;
  for (int k = ty; k < n; k += blockDim.y) sph[k * TXO + lx] = ok ? phi[(long long)k * G + x] : make_double2(0.0, 0.0);
  __syncthreads();
  if (ok) {
    for (int ii = ty; ii < ni; ii += blockDim.y) {
      double2 a = acc_in ? acc_in[(long long)ii * G + x] : make_double2(0.0, 0.0);
      const double2* Vi = V + (long long)n * ii * G + x;  // V(x,k,i): column k + n*ii
#pragma unroll 4
      for (int k = 0; k < n; ++k) cfma(a, Vi[(long long)k * G], sph[k * TXO + lx]);
      if (dentime) ss[ii * TXO + lx] = a;
      else out[(long long)ii * G + x] = a;
    }
    (void)i0;
  }
  if (!dentime) return;
  __syncthreads();
  if (!ok) return;
  for (int i = ty; i < n; i += blockDim.y) {
    double2 a = make_double2(0.0, 0.0);
    for (int j = 0; j < n; ++j) cfma(a, ss[j * TXO + lx], sinv[j + n * i]);
    out[(long long)i * G + x] = cmul(timefac, a);
  }
}

// actreduced blended over two mean-field slots without projection (the orbital
// Jacobian): out = f0 A_0 + f1 A_1 with A_s = timefac ((Y D_s + V_s . x) I_s) and
// Y = KE(x) (+ potential and field), per point in one pass: the mix,
// redpot_kernel (dentime) and axpby_kernel in one, without the
// per-slot temporaries.
__global__ void __launch_bounds__(TXO * kMaxOrbRhs) blend2_kernel(
    const double2* __restrict__ xin, const double2* __restrict__ Y, const double2* __restrict__ V0,
    const double2* __restrict__ V1, const double2* __restrict__ D0, const double2* __restrict__ D1,
    const double2* __restrict__ I0, const double2* __restrict__ I1, double2 timefac, double f0, double f1, int n,
    long long G, double2* __restrict__ out) {
  extern __shared__ double2 rsm[];
  double2* sD = rsm;            // [2][n*n]
  double2* sI = sD + 2 * n * n;  // [2][n*n]
  double2* sx = sI + 2 * n * n;  // n x TXO
  double2* sy = sx + n * TXO;    // n x TXO
  double2* ss = sy + n * TXO;    // n x TXO
  const int lx = threadIdx.x, ty = threadIdx.y, tid = ty * TXO + lx;
  for (int e = tid; e < n * n; e += TXO * blockDim.y) {
    sD[e] = D0[e];
    sD[n * n + e] = D1[e];
    sI[e] = I0[e];
    sI[n * n + e] = I1[e];
  }
  const long long x = blockIdx.x * (long long)TXO + lx;
  const bool ok = x < G;
  for (int j = ty; j < n; j += blockDim.y) {
    sx[j * TXO + lx] = ok ? xin[(long long)j * G + x] : make_double2(0.0, 0.0);
    sy[j * TXO + lx] = ok ? Y[(long long)j * G + x] : make_double2(0.0, 0.0);
  }
  const int ii = ty;  // one warp per orbital
  double2 res = make_double2(0.0, 0.0);
  for (int s = 0; s < 2; ++s) {
    __syncthreads();  // tiles loaded (s = 0); the previous slot's ss reads done (s = 1)
    if (ok) {
      const double2* Ds = sD + s * n * n;
      double2 a = make_double2(0.0, 0.0);
      for (int j = 0; j < n; ++j) cfma(a, sy[j * TXO + lx], Ds[j + n * ii]);
      const double2* Vi = (s ? V1 : V0) + (long long)n * ii * G + x;
#pragma unroll 4
      for (int k = 0; k < n; ++k) cfma(a, Vi[(long long)k * G], sx[k * TXO + lx]);
      ss[ii * TXO + lx] = a;
    }
    __syncthreads();
    if (ok) {
      const double2* Is = sI + s * n * n;
      double2 t = make_double2(0.0, 0.0);
      for (int j = 0; j < n; ++j) cfma(t, ss[j * TXO + lx], Is[j + n * ii]);
      t = cmul(timefac, t);
      res = s == 0 ? make_double2(f0 * t.x, f0 * t.y) : make_double2(fma(f1, t.x, 1.0 * res.x), fma(f1, t.y, 1.0 * res.y));
    }
  }
  if (ok) out[(long long)ii * G + x] = res;
}

// M(j,i) = sum_s f_s sum_l D_s(j,l) I_s(l,i): one thread per element (n*n <= 1024)
__global__ void blendq_m_kernel(const double2* __restrict__ D0, const double2* __restrict__ D1,
                                const double2* __restrict__ I0, const double2* __restrict__ I1, double f0, double f1,
                                int n, double2* __restrict__ M) {
  const int e = threadIdx.x;
  if (e >= n * n) return;
  const int j = e % n, i = e / n;
  double2 a0 = make_double2(0.0, 0.0), a1 = make_double2(0.0, 0.0);
  for (int l = 0; l < n; ++l) {
    cfma(a0, D0[j + n * l], I0[l + n * i]);
    cfma(a1, D1[j + n * l], I1[l + n * i]);
  }
  M[e] = make_double2(fma(f1, a1.x, f0 * a0.x), fma(f1, a1.y, f0 * a0.y));
}

// Q(x,k,i) = sum_s sum_j V_s(x,k,j) (f_s I_s(j,i)), reducedpot layout (x fastest,
// then k, then i): per tile of TXO points the rows V_s(., k, j) of one k are staged
// (warp j loads row j of both slots), then warp i forms Q(., k, i)
__global__ void __launch_bounds__(TXO * kMaxOrbRhs) blendq_build_kernel(
    const double2* __restrict__ V0, const double2* __restrict__ V1, const double2* __restrict__ I0,
    const double2* __restrict__ I1, double f0, double f1, int n, long long G, double2* __restrict__ Q) {
  extern __shared__ double2 rsm[];
  double2* sJ = rsm;             // [2][n*n]
  double2* sV = sJ + 2 * n * n;  // [2][n][TXO]
  const int lx = threadIdx.x, ty = threadIdx.y, tid = ty * TXO + lx;
  for (int e = tid; e < n * n; e += TXO * blockDim.y) {
    const double2 a = I0[e], b = I1[e];
    sJ[e] = make_double2(f0 * a.x, f0 * a.y);
    sJ[n * n + e] = make_double2(f1 * b.x, f1 * b.y);
  }
  const long long x = blockIdx.x * (long long)TXO + lx;
  const bool ok = x < G;
  for (int k = 0; k < n; ++k) {
    __syncthreads();  // the previous k's rows are used (and sJ is staged)
    for (int j = ty; j < n; j += blockDim.y) {
      const long long o = (long long)(k + n * j) * G + x;
      sV[j * TXO + lx] = ok ? V0[o] : make_double2(0.0, 0.0);
      sV[(n + j) * TXO + lx] = ok ? V1[o] : make_double2(0.0, 0.0);
    }
    __syncthreads();
    if (ok) {
      for (int i = ty; i < n; i += blockDim.y) {
        double2 a = make_double2(0.0, 0.0);
        for (int j = 0; j < n; ++j) cfma(a, sV[j * TXO + lx], sJ[j + n * i]);
        for (int j = 0; j < n; ++j) cfma(a, sV[(n + j) * TXO + lx], sJ[n * n + j + n * i]);
        Q[(long long)(k + n * i) * G + x] = a;
      }
    }
  }
}

// out(x,i) = timefac (sum_j Y(x,j) M(j,i) + sum_k Q(x,k,i) xin(x,k))
__global__ void __launch_bounds__(TXO * kMaxOrbRhs) blendq_apply_kernel(
    const double2* xin, const double2* Y, const double2* Q,
    const double2* M, double2 timefac, int n, long long G, double2* out) {
  extern __shared__ double2 rsm[];
  grid_dependency_wait();
  grid_dependents_launch();
  double2* sM = rsm;            // n*n
  double2* sx = sM + n * n;     // n x TXO
  double2* sy = sx + n * TXO;   // n x TXO
  const int lx = threadIdx.x, ty = threadIdx.y, tid = ty * TXO + lx;
  for (int e = tid; e < n * n; e += TXO * blockDim.y) sM[e] = M[e];
  const long long x = blockIdx.x * (long long)TXO + lx;
  const bool ok = x < G;
  for (int j = ty; j < n; j += blockDim.y) {
    sx[j * TXO + lx] = ok ? xin[(long long)j * G + x] : make_double2(0.0, 0.0);
    sy[j * TXO + lx] = ok ? Y[(long long)j * G + x] : make_double2(0.0, 0.0);
  }
  __syncthreads();
  if (!ok) return;
  for (int i = ty; i < n; i += blockDim.y) {
    double2 a = make_double2(0.0, 0.0);
    for (int j = 0; j < n; ++j) cfma(a, sy[j * TXO + lx], sM[j + n * i]);
    const double2* Qi = Q + (long long)n * i * G + x;
#pragma unroll 4
    for (int k = 0; k < n; ++k) cfma(a, Qi[(long long)k * G], sx[k * TXO + lx]);
    out[(long long)i * G + x] = cmul(timefac, a);
  }
}

// partial[blk][j + n*i] = sum_{x in blk} conj(P_j(x)) T_i(x); block blk covers
// DCH consecutive points, warp w the rows j = w, w + (warps per block), ...
// (beyond 16 orbitals).  BL points per block: 256 (eight terms per lane before the shuffle
// tree, a quarter of the partials to reduce) where they fit shared memory, else 64
constexpr int DCH = 64;
template <int BL>
__global__ void __launch_bounds__(TXO * kMaxOrbRhs) dots_kernel(const double2* __restrict__ Pm,
                                                         const double2* __restrict__ Tm, int n, long long G,
                                                         double2* __restrict__ partial) {
  extern __shared__ double2 rsm[];
  double2* tt = rsm;  // n x BL
  const int lx = threadIdx.x, ty = threadIdx.y, tid = ty * TXO + lx;
  const long long x0 = blockIdx.x * (long long)BL;
  const int nth = TXO * blockDim.y;
  // staged in batches of 8 elements per thread: the 8 loads are in flight together
  for (int e0 = tid; e0 < n * BL; e0 += 8 * nth) {
    double2 v[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const int e = e0 + r * nth;
      const int i = e / BL, k = e % BL;
      const long long x = x0 + k;
      v[r] = (e < n * BL && x < G) ? Tm[(long long)i * G + x] : make_double2(0.0, 0.0);
    }
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const int e = e0 + r * nth;
      if (e < n * BL) tt[e] = v[r];
    }
  }
  __syncthreads();
  const int nn = n * n;
  for (int j = ty; j < n; j += blockDim.y) {
    double2 pv[BL / TXO];
#pragma unroll
    for (int r = 0; r < BL / TXO; ++r) {
      const long long x = x0 + r * TXO + lx;
      pv[r] = x < G ? Pm[(long long)j * G + x] : make_double2(0.0, 0.0);
    }
    for (int i = 0; i < n; ++i) {
      double2 a = make_double2(0.0, 0.0);
#pragma unroll
      for (int r = 0; r < BL / TXO; ++r) {  // conj(p) t
        const double2 p = pv[r], t = tt[i * BL + r * TXO + lx];
        a.x = fma(p.x, t.x, fma(p.y, t.y, a.x));
        a.y = fma(p.x, t.y, fma(-p.y, t.x, a.y));
      }
      for (int o = 16; o > 0; o >>= 1) {
        a.x += __shfl_down_sync(0xffffffffu, a.x, o);
        a.y += __shfl_down_sync(0xffffffffu, a.y, o);
      }
      if (lx == 0) partial[(long long)blockIdx.x * nn + j + n * i] = a;
    }
  }
}

// one CTA per element: strided partial sums then a fixed-shape tree (deterministic)
__global__ void __launch_bounds__(128) dots_reduce_kernel(const double2* __restrict__ partial,
                                                          int nblk, int nn, double2* __restrict__ D) {
  __shared__ double2 red[128];
  const int e = blockIdx.x;
  double2 s = make_double2(0.0, 0.0);
  for (int b = threadIdx.x; b < nblk; b += 128) s = cadd(s, partial[(long long)b * nn + e]);
  red[threadIdx.x] = s;
  __syncthreads();
  for (int w = 64; w > 0; w >>= 1) {
    if (threadIdx.x < w) red[threadIdx.x] = cadd(red[threadIdx.x], red[threadIdx.x + w]);
    __syncthreads();
  }
  if (threadIdx.x == 0) D[e] = red[0];
}

// D(j,i) = sum_x conj(P_j(x)) T_i(x) [+ conj(X_j(x)) O_i(x)] on the FP64 tensor cores: the
// 2n x 2n real products of the rows (orbital, re/im), K = the points.  A warp sums a
// run of points into all NT x NT fragments (n <= 4 NT orbitals), fragments straight from
// global memory (lanes = 4 points x (4 orbitals, re/im)); the CTA adds its warps' sums in
// order, and the last CTA to finish adds the CTAs' partials in a fixed order
// (deterministic).  Bound by HBM: 32 G n bytes a pair, 3.4 us at 41^3 / 10 orbitals, and
// by the latency of the two sums at its end.  dots_kernel below spends ten shuffles on
// each of its n^2 sums per 64 or 256 points: with its reduction 24.5 -> 13.5 us there, the
// Jacobian's two products of one launch instead of four 34 -> 17.8 us (cold caches).
constexpr int kDotWarps = 16, kDotBlocks = 148;
constexpr int dot_points(int nt) { return nt <= 3 ? 16 : 8; }  // points per step of a warp (by registers)
template <int NT>
__global__ void __launch_bounds__(32 * kDotWarps) dots_mma_kernel(const double2* P,
                                                                  const double2* T,
                                                                  const double2* X,
                                                                  const double2* O, int n, long long G,
                                                                  double2* part, double2* D,
                                                                  unsigned* count) {
  extern __shared__ double dsm[];  // [kDotWarps][NT * NT * 64]
  __shared__ unsigned last;
  grid_dependency_wait();
  grid_dependents_launch();
  constexpr int NE = NT * NT * 64, kDotPts = dot_points(NT);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const long long W = (long long)gridDim.x * kDotWarps, w = (long long)warp * gridDim.x + blockIdx.x;
  double acc[NT][NT][2];
#pragma unroll
  for (int a = 0; a < NT; ++a)
#pragma unroll
    for (int b = 0; b < NT; ++b) acc[a][b][0] = acc[a][b][1] = 0.0;
  for (int s = 0; s < (X ? 2 : 1); ++s) {
    const double* L = reinterpret_cast<const double*>(s ? X : P) + (g & 1);
    const double* R = reinterpret_cast<const double*>(s ? O : T) + (g & 1);
    for (long long x0 = w * kDotPts; x0 < G; x0 += W * kDotPts) {
      double l[NT][kDotPts / 4], r[NT][kDotPts / 4];
#pragma unroll
      for (int q = 0; q < kDotPts / 4; ++q)
#pragma unroll
        for (int a = 0; a < NT; ++a) {
          const int j = 4 * a + (g >> 1);
          const long long x = x0 + 4 * q + t;
          const bool ok = j < n && x < G;
          l[a][q] = ok ? L[2 * ((long long)j * G + x)] : 0.0;
          r[a][q] = ok ? R[2 * ((long long)j * G + x)] : 0.0;
        }
#pragma unroll
      for (int q = 0; q < kDotPts / 4; ++q)
#pragma unroll
        for (int a = 0; a < NT; ++a)
#pragma unroll
          for (int b = 0; b < NT; ++b) dmma_884(acc[a][b], l[a][q], r[b][q]);
    }
  }
#pragma unroll
  for (int a = 0; a < NT; ++a)
#pragma unroll
    for (int b = 0; b < NT; ++b) {  // row 8 a + g, columns 8 b + 2 t, + 1
      double* o = dsm + warp * NE + (8 * a + g) * (8 * NT) + 8 * b + 2 * t;
      o[0] = acc[a][b][0];
      o[1] = acc[a][b][1];
    }
  __syncthreads();
  for (int e = tid; e < NE; e += blockDim.x) {
    double v = 0.0;
#pragma unroll
    for (int q = 0; q < kDotWarps; ++q) v += dsm[q * NE + e];
    dsm[e] = v;  // element e of warp 0's block is read by this thread alone
  }
  __syncthreads();
  const int nn = n * n;
  for (int e = tid; e < nn; e += blockDim.x) {
    const int j = e % n, i = e / n;
    const double* c0 = dsm + (2 * j) * (8 * NT) + 2 * i;  // (re, .) row
    const double* c1 = c0 + 8 * NT;                       // (im, .) row
    part[(long long)blockIdx.x * nn + e] = make_double2(c0[0] + c1[1], c0[1] - c1[0]);
  }
  __threadfence();
  __syncthreads();
  if (tid == 0) last = atomicAdd(count, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  // thread (c, e) sums the c-th share of the CTAs for element e (consecutive threads,
  // consecutive elements; eight loads in flight), then the shares are added in order
  // (eight a share at least: the shares of few elements are added one after another, 512 of
  // one orbital's single element took 8 us)
  const int nc = max(1, min((int)blockDim.x / nn, (int)gridDim.x / 8)), per = ((int)gridDim.x + nc - 1) / nc;
  double2* sh = reinterpret_cast<double2*>(dsm);  // [nc][nn]
  for (int q = tid; q < nc * nn; q += blockDim.x) {
    const int cc = q / nn, e = q - cc * nn, b1 = min((int)gridDim.x, (cc + 1) * per);
    double2 v = make_double2(0.0, 0.0);
    for (int b = cc * per; b < b1; b += 8) {
      double2 w[8];
#pragma unroll
      for (int u = 0; u < 8; ++u)
        w[u] = b + u < b1 ? __ldcg(part + (long long)(b + u) * nn + e) : make_double2(0.0, 0.0);
#pragma unroll
      for (int u = 0; u < 8; ++u) v = cadd(v, w[u]);
    }
    sh[q] = v;
  }
  __syncthreads();
  for (int e = tid; e < nn; e += blockDim.x) {
    double2 v = sh[e];
    for (int cc = 1; cc < nc; ++cc) v = cadd(v, sh[cc * nn + e]);
    D[e] = v;
  }
  if (tid == 0) *count = 0;  // for the next launch on this stream
}

// a += b (n^2 elements)
__global__ void mat_add_kernel(double2* __restrict__ a, const double2* __restrict__ b, int nn) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e < nn) a[e] = cadd(a[e], b[e]);
}

// acc = a * acc + b * in  (or acc = b * in when `first`)
__global__ void axpby_kernel(double2* __restrict__ acc, const double2* __restrict__ in, double a, double b,
                             long long len, int first) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < len;
       i += (long long)gridDim.x * blockDim.x) {
    const double2 v = in[i];
    if (first) {
      acc[i] = make_double2(b * v.x, b * v.y);
    } else {
      const double2 w = acc[i];
      acc[i] = make_double2(fma(b, v.x, a * w.x), fma(b, v.y, a * w.y));
    }
  }
}

namespace {

// the kernels' shared-memory limit: one fixed value (race-free across threads)
int rhs_attrs() {
  static const cudaError_t attr = [] {
    for (const void* k : {(const void*)redpot_kernel, (const void*)dots_kernel<DCH>, (const void*)dots_kernel<4 * DCH>,
                          (const void*)blend2_kernel, (const void*)blendq_build_kernel,
                          (const void*)blendq_apply_kernel}) {
      const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kRhsSmemMax);
      if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
  }();
  SG_CUDA(attr);
  return SINCGPU_OK;
}

template <int NS, int NT>
int launch_lin_t(Ctx& c, const double2* base, const double2* s0, const double2* m0, const double2* s1,
                 const double2* m1, double sgn, double2* out) {
  constexpr size_t sm = sizeof(double) * NS * 2 * NT * NT * 32;
  static const cudaError_t attr =
      cudaFuncSetAttribute(lin_kernel<NS, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  SG_CUDA(attr);
  return launch_early(c.stream, lin_kernel<NS, NT>, dim3(ceil_div(c.G, 8 * LMT * kLinWarps)), dim3(32 * kLinWarps), sm,
                      base, s0, m0, s1, m1, sgn, c.nspf, c.G, out);
}

// out = [base] + sgn (s0 m0 [+ s1 m1]) over the orbitals (lin_kernel)
int launch_lin(Ctx& c, const double2* base, const double2* s0, const double2* m0, const double2* s1,
               const double2* m1, double sgn, double2* out) {
#define SG_LIN(NT)                                                                                \
  case NT:                                                                                        \
    return s1 ? launch_lin_t<2, NT>(c, base, s0, m0, s1, m1, sgn, out)                            \
              : launch_lin_t<1, NT>(c, base, s0, m0, nullptr, nullptr, sgn, out);
  switch ((c.nspf + 3) / 4) {
    SG_LIN(1)
    SG_LIN(2)
    SG_LIN(3)
    SG_LIN(4)
    SG_LIN(5)
    SG_LIN(6)
    SG_LIN(7)
    default:
      SG_LIN(8)
  }
#undef SG_LIN
}

template <int NT>
int launch_dots_mma(Ctx& c, const double2* P, const double2* T, const double2* X, const double2* O, double2* D,
                    double2* part) {
  constexpr size_t sm = sizeof(double) * kDotWarps * NT * NT * 64;
  static const cudaError_t attr =
      cudaFuncSetAttribute(dots_mma_kernel<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  SG_CUDA(attr);
  const int nb = (int)std::min<long long>(kDotBlocks, ceil_div(c.G, dot_points(NT)));
  return launch_early(c.stream, dots_mma_kernel<NT>, dim3(nb), dim3(32 * kDotWarps), sm, P, T, X, O, c.nspf, c.G, part, D,
                      c.d_count);
}

// one warp per orbital (n <= 32): every warp of a block has the same share of
// the per-orbital loops
dim3 tile_for(int n) { return dim3(TXO, (unsigned)std::max(1, std::min(n, kMaxOrbRhs))); }

size_t smem_redpot(int n) { return sizeof(double2) * ((size_t)n * n + 2 * (size_t)n * TXO); }
size_t smem_dots(int n, int bl = DCH) { return sizeof(double2) * (size_t)n * bl; }

// D = <P|T> [+ <X|O>]: the tensor-core form up to 16 orbitals (its accumulators: 128
// registers a thread at 16), beyond that one pass of dots_kernel per pair
int launch_dots(Ctx& c, const double2* P, const double2* T, const double2* X, const double2* O, double2* D,
                double2* part) {
  const int n = c.nspf;
  switch ((n + 3) / 4) {
    case 1: return launch_dots_mma<1>(c, P, T, X, O, D, part);
    case 2: return launch_dots_mma<2>(c, P, T, X, O, D, part);
    case 3: return launch_dots_mma<3>(c, P, T, X, O, D, part);
    case 4: return launch_dots_mma<4>(c, P, T, X, O, D, part);
    default: break;
  }
  const bool wide = smem_dots(n, 4 * DCH) <= (size_t)kRhsSmemMax;
  const int nb = ceil_div(c.G, wide ? 4 * DCH : DCH);
  double2* second = part + (size_t)orbital_dots_scratch(c) * n * n - (size_t)n * n;  // the scratch's last n^2
  for (int s = 0; s < (X ? 2 : 1); ++s) {
    if (wide)
      dots_kernel<4 * DCH><<<nb, tile_for(n), smem_dots(n, 4 * DCH), c.stream>>>(s ? X : P, s ? O : T, n, c.G, part);
    else
      dots_kernel<DCH><<<nb, tile_for(n), smem_dots(n), c.stream>>>(s ? X : P, s ? O : T, n, c.G, part);
    SG_LAUNCHED();
    dots_reduce_kernel<<<n * n, 128, 0, c.stream>>>(part, nb, n * n, s ? second : D);
    SG_LAUNCHED();
  }
  if (X) {
    mat_add_kernel<<<ceil_div(n * n, 256), 256, 0, c.stream>>>(D, second, n * n);
    SG_LAUNCHED();
  }
  return SINCGPU_OK;
}

}  // namespace

int orbital_dots_scratch(const Ctx& c) { return std::max(ceil_div(c.G, DCH), kDotBlocks) + 1; }

int orbital_dots(Ctx& c, const double2* P, const double2* T, double2* D, double2* part, const double2* X,
                 const double2* O) {
  SG_CHECK(c.nspf <= kMaxOrbRhs, SINCGPU_ERANGE, "at most %d orbitals", kMaxOrbRhs);
  SG_TRY(rhs_attrs());
  return launch_dots(c, P, T, X, O, D, part);
}

int orbital_mix(Ctx& c, const double2* in, const double2* mat, double2* out) {
  SG_CHECK(c.nspf <= kMaxOrbRhs, SINCGPU_ERANGE, "at most %d orbitals", kMaxOrbRhs);
  return launch_lin(c, nullptr, in, mat, nullptr, nullptr, 1.0, out);
}

int jac_combine(Ctx& c, const double2* T, const double2* P, const double2* M, const double2* X, const double2* D2,
                double2* out) {
  SG_CHECK(c.nspf <= kMaxOrbRhs, SINCGPU_ERANGE, "at most %d orbitals", kMaxOrbRhs);
  return launch_lin(c, T, P, M, X, D2, -1.0, out);
}

int axpby(Ctx& c, double2* acc, const double2* in, double a, double b, long long len, bool first) {
  axpby_kernel<<<std::min<long long>(ceil_div(len, 256), 148 * 8), 256, 0, c.stream>>>(acc, in, a, b, len,
                                                                                        first ? 1 : 0);
  SG_LAUNCHED();
  return SINCGPU_OK;
}

int mult_reducedpot_range(Ctx& c, const double2* phi, const double2* redpot, int i0, int ni,
                          double2* out) {
  const int n = c.nspf;
  SG_CHECK(n <= kMaxOrbRhs, SINCGPU_ERANGE, "at most %d orbitals", kMaxOrbRhs);
  SG_TRY(rhs_attrs());
  ProfScope ps(c, ST_RHS_REDPOT);
  return launch_early(c.stream, redpot_kernel, dim3(ceil_div(c.G, TXO)), tile_for(n), smem_redpot(n), phi, redpot, nullptr,
                      nullptr, make_double2(1, 0), n, i0, ni, 0, c.G, out);
}

int mult_reducedpot(Ctx& c, const double2* phi, const double2* redpot, double2* out) {
  return mult_reducedpot_range(c, phi, redpot, 0, c.nspf, out);
}

namespace {
// actreduced temporaries in ws_rhs: Y = phi denmat, S = KE(Y), T, split-K partials, D
struct RhsTemps {
  double2 *Y, *S, *T, *part, *D;
};
int rhs_temps(Ctx& c, RhsTemps& t) {
  const int n = c.nspf;
  SG_CHECK(n <= kMaxOrbRhs, SINCGPU_ERANGE, "at most %d orbitals", kMaxOrbRhs);
  SG_TRY(rhs_attrs());
  const long long G = c.G;
  const int nb = orbital_dots_scratch(c);
  const size_t need = sizeof(double2) * (3 * (size_t)n * G + (size_t)nb * n * n + (size_t)n * n);
  SG_TRY(c.ws_rhs.ensure(need));
  t.Y = (double2*)c.ws_rhs.ptr;
  t.S = t.Y + (size_t)n * G;
  t.T = t.S + (size_t)n * G;
  t.part = t.T + (size_t)n * G;
  t.D = t.part + (size_t)nb * n * n;
  return SINCGPU_OK;
}
}  // namespace

int actreduced(Ctx& c, const double2* phi, const double2* proj, const double2* denmat,
               const double2* invdenmat, const double2* redpot, double2 timefac, int dentimeflag,
               int projflag, double zfield, double2* out) {
  SG_TRY(actreduced_pre(c, phi, denmat, zfield));
  return actreduced_post(c, phi, proj, invdenmat, redpot, timefac, dentimeflag, projflag, out);
}

int actreduced_pre(Ctx& c, const double2* phi, const double2* denmat, double zfield) {
  RhsTemps t;
  SG_TRY(rhs_temps(c, t));
  const int n = c.nspf;
  {
    ProfScope ps(c, ST_RHS_MIX);
    SG_TRY(orbital_mix(c, phi, denmat, t.Y));
  }
  return mult_ke(c, t.Y, t.S, n, true, zfield);
}

int actreduced_ke(Ctx& c, const double2* phi, double zfield) {
  RhsTemps t;
  SG_TRY(rhs_temps(c, t));
  return mult_ke(c, phi, t.Y, c.nspf, true, zfield);
}

int actreduced_mix_ke(Ctx& c, const double2* denmat) {
  RhsTemps t;
  SG_TRY(rhs_temps(c, t));
  ProfScope ps(c, ST_RHS_MIX);
  return orbital_mix(c, t.Y, denmat, t.S);
}

bool actreduced_blend2_fits(int n) {
  return n <= kMaxOrbRhs && sizeof(double2) * (4 * (size_t)n * n + 3 * (size_t)n * TXO) <= (size_t)kRhsSmemMax;
}

int actreduced_blend2(Ctx& c, const double2* x, const double2* const* denmat, const double2* const* invdenmat,
                      const double2* const* redpot, const double* facs, double2 timefac, double zfield,
                      double2* out) {
  RhsTemps t;
  SG_TRY(rhs_temps(c, t));
  const int n = c.nspf;
  SG_TRY(mult_ke(c, x, t.Y, n, true, zfield));
  ProfScope ps(c, ST_RHS_REDPOT);
  const size_t sm = sizeof(double2) * (4 * (size_t)n * n + 3 * (size_t)n * TXO);
  blend2_kernel<<<ceil_div(c.G, TXO), tile_for(n), sm, c.stream>>>(x, t.Y, redpot[0], redpot[1], denmat[0],
                                                                    denmat[1], invdenmat[0], invdenmat[1], timefac,
                                                                    facs[0], facs[1], n, c.G, out);
  SG_LAUNCHED();
  return SINCGPU_OK;
}

size_t smem_bq_build(int n) { return sizeof(double2) * (2 * (size_t)n * n + 2 * (size_t)n * TXO); }
size_t smem_bq_apply(int n) { return sizeof(double2) * ((size_t)n * n + 2 * (size_t)n * TXO); }

bool actreduced_blendq_fits(int n) {
  return n <= kMaxOrbRhs && smem_bq_build(n) <= (size_t)kRhsSmemMax && smem_bq_apply(n) <= (size_t)kRhsSmemMax;
}

int blendq_prepare(Ctx& c, const double2* const* denmat, const double2* const* invdenmat,
                   const double2* const* redpot, const double* facs) {
  const int n = c.nspf;
  SG_CHECK(actreduced_blendq_fits(n), SINCGPU_ERANGE, "blended reduced potential: at most %d orbitals", kMaxOrbRhs);
  SG_TRY(rhs_attrs());
  const size_t nq = (size_t)c.G * n * n;
  SG_TRY(c.ws_bq.ensure(sizeof(double2) * (nq + (size_t)n * n)));
  double2* Q = (double2*)c.ws_bq.ptr;
  ProfScope ps(c, ST_RHS_REDPOT);
  blendq_m_kernel<<<1, 1024, 0, c.stream>>>(denmat[0], denmat[1], invdenmat[0], invdenmat[1], facs[0], facs[1], n,
                                            Q + nq);
  SG_LAUNCHED();
  blendq_build_kernel<<<ceil_div(c.G, TXO), tile_for(n), smem_bq_build(n), c.stream>>>(
      redpot[0], redpot[1], invdenmat[0], invdenmat[1], facs[0], facs[1], n, c.G, Q);
  SG_LAUNCHED();
  return SINCGPU_OK;
}

int actreduced_blendq(Ctx& c, const double2* x, double2 timefac, double zfield, double2* out) {
  RhsTemps t;
  SG_TRY(rhs_temps(c, t));
  const int n = c.nspf;
  const double2* Q = (const double2*)c.ws_bq.ptr;
  SG_CHECK(Q, SINCGPU_ESTATE, "blended reduced potential not prepared");
  SG_TRY(mult_ke(c, x, t.Y, n, true, zfield));
  ProfScope ps(c, ST_RHS_REDPOT);
  return launch_early(c.stream, blendq_apply_kernel, dim3(ceil_div(c.G, TXO)), tile_for(n), smem_bq_apply(n), x, t.Y, Q,
                      Q + (size_t)c.G * n * n, timefac, n, c.G, out);
}

int actreduced_temps(Ctx& c, double2** S, double2** T) {
  RhsTemps t;
  SG_TRY(rhs_temps(c, t));
  *S = t.S;
  *T = t.T;
  return SINCGPU_OK;
}

int actreduced_post(Ctx& c, const double2* phi, const double2* proj, const double2* invdenmat,
                    const double2* redpot, double2 timefac, int dentimeflag, int projflag, double2* out,
                    bool t_ready) {
  RhsTemps t;
  SG_TRY(rhs_temps(c, t));
  const int n = c.nspf;
  const long long G = c.G;
  const int bt = ceil_div(G, TXO);
  double2 *S = t.S, *T = t.T, *part = t.part, *D = t.D;
  double2* dst = projflag == 1 ? T : out;
  if (!t_ready) {
    ProfScope ps(c, ST_RHS_REDPOT);
    SG_TRY(launch_early(c.stream, redpot_kernel, dim3(bt), tile_for(n), smem_redpot(n), phi, redpot, S, invdenmat, timefac,
                        n, 0, n, dentimeflag ? 1 : 0, G, dst));
  }
  if (projflag == 1) {
    ProfScope ps(c, ST_RHS_PROJ);
    SG_TRY(launch_dots(c, proj, T, nullptr, nullptr, D, part));
    SG_TRY(launch_lin(c, T, proj, D, nullptr, nullptr, -1.0, out));
  }
  return SINCGPU_OK;
}

}  // namespace sincgpu
