// Krylov exponential propagator of the A-vector on the device.
//
// Restates Sidje's Expokit DGEXPV as the reference's variant DGEXPVxxx20
// (MCTDH.SRC/expokit.f90:2222-2660) that expoavecprop calls
// (MCTDH.SRC/expo_driver.f90:827-1055): w = exp(t A) v for the real-ified
// A-vector (complex nc-vector viewed as 2*nc reals), A = timefac * H with H the
// CI sigma operator (sparsesparsemult_byproc, ci.cu).  Full (modified
// Gram-Schmidt) Arnoldi, happy-breakdown test, (6,6) Pade with scaling and
// squaring of the small Hessenberg (DGPADM, expokit.f90:526-713), local error
// estimate and step-size control with the reference's modification that the next
// step is never shorter than the accepted one, and the returned step guess.
// All vector and matrix arithmetic runs on the GPU in FP64; the host only reads
// the few scalars that decide step acceptance.
#include <algorithm>
#include <cmath>
#include <vector>
#include <cooperative_groups.h>
#include "context.hpp"
#include "dmma.cuh"
#include "gram_schmidt.cuh"

namespace sincgpu {

constexpr int kKryThreads = 1024;
constexpr int kMaxKry = 124;  // Krylov dimension limit (Pade order m + 2 <= 126)

// block reduction (fixed shape -> deterministic)
__device__ double block_sum(double v, double* red) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  double s = 0.0;
  if (threadIdx.x < 32) {
    s = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.0;
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (threadIdx.x == 0) red[32] = s;
  }
  __syncthreads();
  return red[32];
}

struct KryState {  // device scalars
  double beta;     // |w|
  double avnorm;   // |A v_{m+1}|
  int mbrk;        // 0 = no breakdown, else breakdown dimension
};

// V[0] = w / beta (beta computed here and stored)
__global__ void __launch_bounds__(kKryThreads) kry_start_kernel(const double* __restrict__ w, long long n,
                                                                double* __restrict__ V, KryState* st,
                                                                int compute_beta) {
  __shared__ double red[33];
  double s = 0.0;
  if (compute_beta) {
    for (long long i = threadIdx.x; i < n; i += blockDim.x) s += w[i] * w[i];
    s = block_sum(s, red);
    if (threadIdx.x == 0) st->beta = sqrt(s);
  }
  __syncthreads();
  const double b = compute_beta ? sqrt(s) : st->beta;
  const double inv = 1.0 / b;
  for (long long i = threadIdx.x; i < n; i += blockDim.x) V[i] = inv * w[i];
  if (threadIdx.x == 0) st->mbrk = 0;
}

// modified Gram-Schmidt of p = V[j+1] (the matvec of V[j]) against V[0..j],
// Hessenberg column j, breakdown test, normalisation (expokit.f90:2327-2346).
__global__ void __launch_bounds__(kKryThreads) kry_mgs_kernel(double* __restrict__ V, long long n, int j,
                                                              double* __restrict__ Hm, int mh,
                                                              double break_tol, KryState* st) {
  __shared__ double red[33];
  if (st->mbrk) return;
  double* p = V + (long long)(j + 1) * n;
  for (int i = 0; i <= j; ++i) {
    const double* vi = V + (long long)i * n;
    double s = 0.0;
    for (long long k = threadIdx.x; k < n; k += blockDim.x) s += vi[k] * p[k];
    const double hij = block_sum(s, red);
    for (long long k = threadIdx.x; k < n; k += blockDim.x) p[k] -= hij * vi[k];
    if (threadIdx.x == 0) Hm[(long long)j * mh + i] = hij;
    __syncthreads();
  }
  double s = 0.0;
  for (long long k = threadIdx.x; k < n; k += blockDim.x) s += p[k] * p[k];
  const double h = sqrt(block_sum(s, red));
  if (h <= break_tol) {
    if (threadIdx.x == 0) st->mbrk = j + 1;
    return;
  }
  if (threadIdx.x == 0) Hm[(long long)j * mh + j + 1] = h;
  const double inv = 1.0 / h;
  for (long long k = threadIdx.x; k < n; k += blockDim.x) p[k] *= inv;
}

// One Arnoldi step's orthogonalisation on a thread-block cluster: the modified
// Gram-Schmidt coefficients from one pass of dots (gs_solve) instead of
// kry_mgs_kernel's j + 1 dependent sums.  Row j of L is formed in the same pass over V (v_j
// is a row already).
//
// CTA q of the cluster owns the slice [q S, q S + S) of the vectors, S = ceil(n /
// kGsCluster) rounded up to even; p, v_j and the first `cap` rows of the slice sit in
// shared memory (all of them for 30 vectors up to some 5,800 determinants), further rows
// come from L2.  A warp sums up to four rows over half the slice; the CTAs' partials are added
// in a fixed order through distributed shared memory, so every CTA gets the same value.
// What bounds it: the latency of its dependent stages (load of p, dots, update, norm) and
// two cluster barriers.  The rows' way into shared memory comes before the wait for the
// sigma product that writes p: that product and the step before may still run (512
// threads, so that all fit an SM).  After the wait, at 25 rows of 3136 determinants: loads
// 0.8 us, dots 2.2, barrier 0.7, coefficients 1.3, update 0.9, norm 1.2.  One A-vector step
// of 30 vectors at 3136 determinants, launches included: 810 -> 522 us, of which clusters of
// 8 whose rows came from L2 after the sigma product had ended took 14 us a vector.  One CTA
// with sequential projections is slower at every size: 25 determinants 0.87 ms a step of up
// to 30 vectors, 0.35 on the cluster; 450 0.95 and 0.38; 3136 1.57 and 0.53.
constexpr int kGsCluster = 16;
constexpr int kGsThreads = 32 * kGsCluster;
constexpr long long kGsSlice = 8100;    // most values of a slice
constexpr long long kGsValues = 23900;  // of dynamic shared memory: p, v_j, rows of T, rows of V
static_assert(2 * kGsSlice + kMaxKry * (kMaxKry - 1) / 2 <= kGsValues, "p, v_j and T must fit");

__device__ __forceinline__ void cp_async16(double* smem, const double* gmem) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem));
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// out[half][i] = (<v, x>, <v, y>) with v = row(i) over the warp's half of the slice, for the NR
// rows i0, i0 + 8, .. (the last row for those past it); the lanes' sums change places as
// they are halved, so that 2 NR values take 2 NR + 1 or so exchanges instead of 10 NR
template <int NR, class Row>
__device__ __forceinline__ void gs_dots(int i0, int last, int half, int len, const double* x, const double* y, Row row,
                                        double2 (*out)[128]) {
  const int lane = threadIdx.x & 31;
  const double* v[NR];
  double a[2 * NR];
#pragma unroll
  for (int u = 0; u < NR; ++u) {
    v[u] = row(min(i0 + 8 * u, last));
    a[2 * u] = a[2 * u + 1] = 0.0;
  }
#pragma unroll 4
  for (int k = 32 * half + lane; k < len; k += 64) {
    const double xk = x[k], yk = y[k];
#pragma unroll
    for (int u = 0; u < NR; ++u) {
      const double vk = v[u][k];
      a[2 * u] = fma(vk, xk, a[2 * u]);
      a[2 * u + 1] = fma(vk, yk, a[2 * u + 1]);
    }
  }
  int which = 0;
#pragma unroll
  for (int o = 16, c = NR; o > 0; o >>= 1, c >>= 1) {
    if (c > 0) {  // keep c of the 2 c values left
      const bool up = lane & o;
#pragma unroll
      for (int u = 0; u < c; ++u) {
        const double give = up ? a[u] : a[u + c], keep = up ? a[u + c] : a[u];
        a[u] = keep + __shfl_xor_sync(0xffffffffu, give, o);
      }
      if (up) which += c;
    } else {
      a[0] += __shfl_xor_sync(0xffffffffu, a[0], o);
    }
  }
  const int i = i0 + 8 * (which >> 1);
  if (lane % (16 / NR) == 0 && i <= last) (which & 1 ? out[half][i].y : out[half][i].x) = a[0];
}

// ALL: cap = j, every row in shared memory
template <bool ALL>
__global__ void __launch_bounds__(kGsThreads) kry_gs_kernel(double* V, long long n, int S, int cap, int j,
                                                            double* Hm, int mh, double* Tm, double break_tol,
                                                            KryState* st) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  extern __shared__ __align__(16) double gsm[];  // p, v_j, rows 0 .. cap - 1 of the slice, rows of T
  __shared__ double2 part[kGsCluster][128];  // every CTA's partial dots <v_i, p>, <v_i, v_j>
  __shared__ double2 dots[2][128];           // this CTA's, by halves of its slice
  __shared__ double npart[kGsCluster], red[kGsThreads / 32], lpart[kGsThreads / 32], r[128], lrow[128], h[128];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rank = cl.block_rank();
  const long long lo = (long long)rank * S;
  const int len = (int)max(0LL, min((long long)S, n - lo));
  double* ps = gsm;
  double* Ts = gsm + (long long)(2 + cap) * S;  // row i from i (i - 1) / 2
  double* pg = V + (long long)(j + 1) * n + lo;
  auto row = [&](int i) -> const double* {
    if (ALL) return gsm + (i == j ? 1 : 2 + i) * S;
    return i == j ? gsm + S : i < cap ? gsm + (long long)(2 + i) * S : V + (long long)i * n + lo;
  };
  // Before the wait: rows 0 .. j - 1 of V and 0 .. j - 2 of T, all of steps that have ended
  // (the step in front waits for its own predecessor before it lets this one start).
  // Rows as pairs: n, S and so every len are even.
  for (int i = warp; i < cap; i += kGsThreads / 32)
    for (int k = 2 * lane; k < len; k += 64)
      cp_async16(gsm + (long long)(2 + i) * S + k, V + (long long)i * n + lo + k);
  for (int i = warp; i < j - 1; i += kGsThreads / 32)
    for (int k = lane; k < i; k += 32) Ts[i * (i - 1) / 2 + k] = __ldcg(Tm + (long long)i * mh + k);
  cp_async_wait_all();
  cl.sync();  // the CTAs whose shared memory is written are there
  grid_dependency_wait();
  grid_dependents_launch();
  const int brk_before = *(volatile int*)&st->mbrk;  // the same value in every CTA
  const double* vj = V + (long long)j * n + lo;
  for (int k = tid; k < len; k += kGsThreads) {
    ps[k] = __ldcg(pg + k);
    gsm[S + k] = __ldcg(vj + k);
  }
  if (tid < j - 1) Ts[(j - 1) * (j - 2) / 2 + tid] = __ldcg(Tm + (long long)(j - 1) * mh + tid);
  __syncthreads();
  if (brk_before) return;
  for (int base = 0; base <= j; base += 32) {
    const int i0 = base + (warp & 7), left = j + 1 - base;
    if (left > 16) gs_dots<4>(i0, j, warp >> 3, len, ps, gsm + S, row, dots);
    else if (left > 8) gs_dots<2>(i0, j, warp >> 3, len, ps, gsm + S, row, dots);
    else gs_dots<1>(i0, j, warp >> 3, len, ps, gsm + S, row, dots);
  }
  __syncthreads();
  static_assert(kGsThreads / 32 == kGsCluster, "a warp per CTA of the cluster");
  for (int i = lane; i <= j; i += 32) *cl.map_shared_rank(&part[rank][i], warp) = cadd(dots[0][i], dots[1][i]);
  cl.sync();
  if (tid <= j) {
    double2 a[2] = {make_double2(0.0, 0.0), make_double2(0.0, 0.0)};
#pragma unroll
    for (int q = 0; q < kGsCluster; ++q) a[q & 1] = cadd(a[q & 1], part[q][tid]);
    const double2 sum = cadd(a[0], a[1]);
    r[tid] = sum.x;
    lrow[tid] = sum.y;  // row j of L (its diagonal is not used)
  }
  __syncthreads();
  // the same in every CTA
  auto trow = [&](int i, int k) { return Ts[i * (i - 1) / 2 + k]; };
  auto ldot = [&](int k) { return lrow[k]; };
  const double hj = gs_solve<kGsThreads / 32>(j, h, lpart, [&](int i) { return r[i]; }, ldot, trow);
  if (rank == 0 && tid <= j) Hm[(long long)j * mh + tid] = tid < j ? h[tid] : hj;
  double s = 0.0;
  const int staged = ALL ? j : cap;
  for (int k = tid; k < len; k += kGsThreads) {
    double x[4] = {fma(-hj, gsm[S + k], ps[k]), 0.0, 0.0, 0.0};
    int i = 0;
#pragma unroll 2
    for (; i + 4 <= staged; i += 4)
#pragma unroll
      for (int u = 0; u < 4; ++u) x[u] = fma(-h[i + u], gsm[(2 + i + u) * S + k], x[u]);
    for (; i < staged; ++i) x[0] = fma(-h[i], gsm[(2 + i) * S + k], x[0]);
    for (; !ALL && i + 4 <= j; i += 4)
#pragma unroll
      for (int u = 0; u < 4; ++u) x[u] = fma(-h[i + u], V[(long long)(i + u) * n + lo + k], x[u]);
    for (; !ALL && i < j; ++i) x[0] = fma(-h[i], V[(long long)i * n + lo + k], x[0]);
    x[0] += x[1] + (x[2] + x[3]);
    ps[k] = x[0];
    s = fma(x[0], x[0], s);
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) red[warp] = s;
  __syncthreads();
  if (warp == 0) {
    s = lane < kGsThreads / 32 ? red[lane] : 0.0;
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane < kGsCluster) *cl.map_shared_rank(&npart[rank], lane) = s;
  }
  auto arrived = cl.barrier_arrive();
  gs_extend(j, ldot, trow, rank, kGsCluster, [&](int k, double v) { Tm[(long long)j * mh + k] = v; });
  cl.barrier_wait(std::move(arrived));
  double t = 0.0;
#pragma unroll
  for (int q = 0; q < kGsCluster; ++q) t += npart[q];
  const double hn = sqrt(t);
  const bool brk = hn <= break_tol;
  if (rank == 0 && tid == 0) {
    if (brk) st->mbrk = j + 1;
    else Hm[(long long)j * mh + j + 1] = hn;
  }
  const double inv = 1.0 / hn;
  for (int k = tid; k < len; k += kGsThreads) pg[k] = brk ? ps[k] : ps[k] * inv;
}

// w = beta * V[0:mx]^T exph[0:mx]; beta <- |w|, over the same cluster and slices
__global__ void __launch_bounds__(kKryThreads) kry_update_cluster_kernel(const double* __restrict__ V, long long n,
                                                                         int S, int mx,
                                                                         const double* __restrict__ exph,
                                                                         double* __restrict__ w, KryState* st) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  __shared__ double red[33], ex[128];
  __shared__ double npart;
  const int tid = threadIdx.x;
  const double beta = st->beta;
  const long long lo = (long long)cl.block_rank() * S;
  const int len = (int)max(0LL, min((long long)S, n - lo));
  for (int i = tid; i < mx; i += kKryThreads) ex[i] = exph[i];
  cl.sync();  // every CTA has read beta
  double s = 0.0;
  for (int k = tid; k < len; k += kKryThreads) {
    const double* vk = V + lo + k;
    double acc = 0.0;
#pragma unroll 8
    for (int i = 0; i < mx; ++i) acc += vk[(long long)i * n] * ex[i];
    const double v = beta * acc;
    w[lo + k] = v;
    s += v * v;
  }
  s = block_sum(s, red);
  if (tid == 0) npart = s;
  cl.sync();
  if (cl.block_rank() == 0 && tid == 0) {
    double t = 0.0;
    for (int q = 0; q < kGsCluster; ++q) t += *cl.map_shared_rank(&npart, q);
    st->beta = sqrt(t);
  }
  cl.sync();  // no CTA leaves while its partial is read
}

// a launch on one cluster of kGsCluster CTAs; `early`: before the kernel in front of it has ended
struct GsLaunch {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[2];
  GsLaunch(int threads, size_t smem, cudaStream_t stream, bool early) {
    cfg.gridDim = dim3(kGsCluster, 1, 1);
    cfg.blockDim = dim3(threads, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = kGsCluster;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = early ? 2 : 1;
  }
};
template <class... KA, class... A>
static int launch_gs_cluster(Ctx& c, void (*kernel)(KA...), int threads, size_t smem, bool early, A... args) {
  GsLaunch l(threads, smem, c.stream, early);
  SG_CUDA(cudaLaunchKernelEx(&l.cfg, kernel, (KA)args...));
  count_launch();
  return SINCGPU_OK;
}

// Whether the device places the cluster kernels, with the most shared memory that they take:
// 16 CTAs are more than every device has to place (8), and a part of one may hold fewer.
// Sets the kernels' attributes; once per process.
static bool gs_cluster_fits() {
  static const bool fits = [] {
    constexpr size_t smem = sizeof(double) * kGsValues;
    for (auto k : {kry_gs_kernel<true>, kry_gs_kernel<false>}) {
      int n = 0;
      GsLaunch l(kGsThreads, smem, nullptr, false);
      if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
          cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
          cudaOccupancyMaxActiveClusters(&n, k, &l.cfg) != cudaSuccess || n < 1)
        return false;
    }
    int n = 0;
    GsLaunch l(kKryThreads, 0, nullptr, false);
    return cudaFuncSetAttribute(kry_update_cluster_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) ==
               cudaSuccess &&
           cudaOccupancyMaxActiveClusters(&n, kry_update_cluster_kernel, &l.cfg) == cudaSuccess && n >= 1;
  }();
  if (!fits) (void)cudaGetLastError();
  return fits;
}

__global__ void __launch_bounds__(kKryThreads) kry_avnorm_kernel(const double* __restrict__ p, long long n,
                                                                 KryState* st) {
  __shared__ double red[33];
  if (st->mbrk) return;
  double s = 0.0;
  for (long long k = threadIdx.x; k < n; k += blockDim.x) s += p[k] * p[k];
  s = block_sum(s, red);
  if (threadIdx.x == 0) st->avnorm = sqrt(s);
}

// (6,6) Pade exp(t H) with scaling and squaring (DGPADM), H = Hm[0:mx,0:mx]
// (column-major, leading dimension mh); writes column `col` of exp(t H) to exph
// and, when Efull is given, the whole matrix (column-major, leading dimension mx).
// One CTA; mx <= kMaxPade.  The five work matrices live in dynamic shared memory with the
// leading dimension ld = 4 mod 8 (fragment loads without bank conflicts), or in `gscratch`
// (global, 5 mx^2 doubles, ld = mx) when it is given.
// Bound by latency: some 20 products and mx elimination steps, one after another.  The
// products run on the FP64 tensor cores, a warp per 8 x 8 tile.  The scaling leaves
// |H| < 1/2, so the denominator D of the approximant has |D - I| <= exp(1/4) - 1 < 0.3 in
// the infinity norm: its rows stay dominated by their diagonal and the elimination needs
// no pivoting (no element grows by more than 2).  It takes column k from all other rows,
// a division and a barrier a step, and no back substitution follows.  Order 32:
// 49 us; 138 with one thread per element, pivoting and a triangular solve (order ~13: 20, was 27).
constexpr int kMaxPade = 128;
constexpr int kPadeDeg = 6;
constexpr int kPadeThreads = 512;
inline int pade_ld(int m) { return (m + 3) / 8 * 8 + 4; }
struct PadeCoef {
  double c[kPadeDeg + 1];
  constexpr PadeCoef() : c{} {
    c[0] = 1.0;
    for (int k = 1; k <= kPadeDeg; ++k)
      c[k] = (c[k - 1] * (double)(kPadeDeg + 1 - k)) / (double)(k * (2 * kPadeDeg + 1 - k));
  }
};
// out(:,j) = f(sum_k X(:,k) Y(k,j), i, j), all m x m; ends with a barrier
template <class F>
__device__ __forceinline__ void pade_product(double* out, const double* X, const double* Y, int m, int ld, F f) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const int nt = (m + 7) >> 3, g = lane >> 2, q = lane & 3;
  for (int t = warp; t < nt * nt; t += nw) {
    const int i = t % nt * 8 + g, j0 = t / nt * 8;
    const bool iok = i < m, jok = j0 + g < m;
    const double* x = X + i;
    const double* y = Y + ld * (j0 + g);
    double d[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
#pragma unroll 4
    for (int k = q; k - q < m; k += 8) {
      const double a0 = iok && k < m ? x[ld * k] : 0.0, b0 = jok && k < m ? y[k] : 0.0;
      const double a1 = iok && k + 4 < m ? x[ld * (k + 4)] : 0.0, b1 = jok && k + 4 < m ? y[k + 4] : 0.0;
      dmma_884(d[0], a0, b0);
      dmma_884(d[1], a1, b1);
    }
#pragma unroll
    for (int u = 0; u < 2; ++u)
      if (iok && j0 + 2 * q + u < m) out[i + ld * (j0 + 2 * q + u)] = f(d[0][u] + d[1][u], i, j0 + 2 * q + u);
  }
  __syncthreads();
}
__global__ void __launch_bounds__(kPadeThreads) kry_padm_kernel(const double* __restrict__ Hm, int mh, int mx,
                                                                double t, double* __restrict__ exph,
                                                                int* __restrict__ ns_out, int col,
                                                                double* __restrict__ Efull,
                                                                double* __restrict__ gscratch, int ld) {
  constexpr int R = kMaxPade / 32;
  constexpr PadeCoef coef;
  static_assert(kPadeDeg == 6, "the steps below are those of degree 6");
  extern __shared__ double psm[];  // H, A, P, Q, T: m x m each, leading dimension ld
  __shared__ double rows[kMaxPade];
  const int m = mx, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nw = blockDim.x >> 5;
  double* H = gscratch ? gscratch : psm;
  double* A = H + ld * m;
  double* P = A + ld * m;
  double* Q = P + ld * m;
  double* T = Q + ld * m;
  for (int j = warp; j < m; j += nw)
    for (int i = lane; i < m; i += 32) {
      H[i + ld * j] = Hm[(long long)j * mh + i];
      P[i + ld * j] = i == j ? coef.c[5] : 0.0;
      Q[i + ld * j] = i == j ? coef.c[6] : 0.0;
    }
  __syncthreads();
  // infinity norm: max row sum of |H|
  for (int r = warp; r < m; r += nw) {
    double s = 0.0;
    for (int j = lane; j < m; j += 32) s += fabs(H[r + ld * j]);
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) rows[r] = s;
  }
  __syncthreads();
  double hn = 0.0;  // every warp for itself
  for (int i = lane; i < m; i += 32) hn = fmax(hn, rows[i]);
  for (int o = 16; o > 0; o >>= 1) hn = fmax(hn, __shfl_xor_sync(0xffffffffu, hn, o));
  const double hnorm = fabs(t * hn);
  if (hnorm == 0.0) {
    for (int i = tid; i < m; i += blockDim.x) exph[i] = i == col ? 1.0 : 0.0;
    if (Efull)
      for (int e = tid; e < m * m; e += blockDim.x) Efull[e] = (e % m) == (e / m) ? 1.0 : 0.0;
    if (tid == 0) *ns_out = 0;
    return;
  }
  const int ns = max(0, (int)(log(hnorm) / log(2.0)) + 2);
  const double scale = t / (double)(1LL << ns);
  const double scale2 = scale * scale;
  auto swap_with_T = [&](double*& X) {
    double* const old = X;
    X = T;
    T = old;
  };
  pade_product(A, H, H, m, ld, [&](double s, int, int) { return scale2 * s; });
  // even part Q and odd part P of the numerator, by Horner's rule in turns
#pragma unroll 1
  for (int k = 4; k >= 0; --k) {
    const double ck = coef.c[k];
    double*& X = k & 1 ? P : Q;
    pade_product(T, X, A, m, ld, [&](double s, int i, int j) { return s + (i == j ? ck : 0.0); });
    swap_with_T(X);
  }
  pade_product(T, P, H, m, ld, [&](double s, int i, int j) {
    Q[i + ld * j] -= scale * s;  // the denominator
    return scale * s;
  });
  swap_with_T(P);
  // X of D X = P: elimination of column k from every row but its own
  for (int k = 0; k < m; ++k) {
    const double pv = Q[k + ld * k];
    double l[R];
#pragma unroll
    for (int u = 0; u < R; ++u) {
      const int i = lane + 32 * u;
      l[u] = i < m && i != k ? Q[i + ld * k] / pv : 0.0;
    }
    const int nq = m - (k + 1);  // columns k + 1 .. of D, then all of P
#pragma unroll 4
    for (int j = warp; j < nq + m; j += nw) {
      double* M = j < nq ? Q + ld * (k + 1 + j) : P + ld * (j - nq);
      const double mk = M[k];
#pragma unroll
      for (int u = 0; u < R; ++u)
        if (lane + 32 * u < m) M[lane + 32 * u] -= l[u] * mk;
    }
    __syncthreads();
  }
  // exp(scale H) = 2 X + I
  for (int j = warp; j < m; j += nw)
    for (int i = lane; i < m; i += 32)
      P[i + ld * j] = 2.0 * (P[i + ld * j] / Q[i + ld * i]) + (i == j ? 1.0 : 0.0);
  __syncthreads();
  for (int s = 0; s < ns; ++s) {
    pade_product(T, P, P, m, ld, [&](double v, int, int) { return v; });
    swap_with_T(P);
  }
  for (int i = tid; i < m; i += blockDim.x) exph[i] = P[i + ld * col];
  if (Efull)
    for (int j = warp; j < m; j += nw)
      for (int i = lane; i < m; i += 32) Efull[i + m * j] = P[i + ld * j];
  if (tid == 0) *ns_out = ns;
}

// w = beta * V[0:mx]^T exph[0:mx]; beta <- |w|
__global__ void __launch_bounds__(kKryThreads) kry_update_kernel(const double* __restrict__ V, long long n,
                                                                 int mx, const double* __restrict__ exph,
                                                                 double* __restrict__ w, KryState* st) {
  __shared__ double red[33];
  const double beta = st->beta;
  double s = 0.0;
  for (long long k = threadIdx.x; k < n; k += blockDim.x) {
    double acc = 0.0;
    for (int i = 0; i < mx; ++i) acc += V[(long long)i * n + k] * exph[i];
    const double v = beta * acc;
    w[k] = v;
    s += v * v;
  }
  s = block_sum(s, red);
  if (threadIdx.x == 0) st->beta = sqrt(s);
}

int pade_expm(Ctx& c, const double* Hm, int mh, int mx, double t, int col, double* exph, double* Efull,
              double* gscratch, int* d_ns) {
  SG_CHECK(mx >= 1 && mx <= kMaxPade, SINCGPU_ERANGE, "Pade order %d outside [1,%d]", mx, kMaxPade);
  // process-wide attribute, one fixed value, set once (thread-safe static init)
  static const cudaError_t attr = cudaFuncSetAttribute(
      kry_padm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(sizeof(double) * 5 * 64 * pade_ld(64)));
  SG_CUDA(attr);
  const bool smem = mx <= 64;
  SG_CHECK(smem || gscratch, SINCGPU_EINVAL, "Pade order %d needs global scratch", mx);
  const int ld = smem ? pade_ld(mx) : mx;
  const size_t psmem = smem ? sizeof(double) * 5 * (size_t)mx * ld : 0;
  kry_padm_kernel<<<1, kPadeThreads, psmem, c.stream>>>(Hm, mh, mx, t, exph, d_ns, col, Efull,
                                                        smem ? nullptr : gscratch, ld);
  SG_LAUNCHED();
  return SINCGPU_OK;
}

static double fortran_nint(double x) { return x >= 0 ? std::floor(x + 0.5) : -std::floor(-x + 0.5); }

int expv_avector(Ctx& c, const double2* v, double2* w, double t, double2 timefac, int m, double tol,
                 double anorm, double* stepguess, int* nstep_out, double ez, double nucdipz, int maxdim_in,
                 int* nmult_out) {
  CIState& s = c.ci;
  SG_CHECK(s.attached && s.assembled, SINCGPU_ESTATE, "sparse CI matrices not assembled");
  const int nc = s.nc;
  const long long n = 2LL * nc;
  // the reference checks m < maxdim (DGEXPVxxx2's maxdim argument; n by default)
  const long long maxdim = maxdim_in > 0 ? maxdim_in : n;
  SG_CHECK(m > 0 && m < maxdim && m <= kMaxKry, SINCGPU_ERANGE, "Krylov dimension %d outside [1,%lld)", m,
           std::min<long long>(maxdim, kMaxKry + 1));
  const int mh = m + 2;
  const size_t need = sizeof(double) * ((size_t)(m + 2) * n + (size_t)mh * mh + 128 + 6 * (size_t)mh * mh) +
                      sizeof(KryState) + 64;
  SG_TRY(c.ws_kry.ensure(need));
  double* V = (double*)c.ws_kry.ptr;
  double* Hm = V + (size_t)(m + 2) * n;
  double* exph = Hm + (size_t)mh * mh;
  double* pscr = exph + 128;
  double* Tm = pscr + 5 * (size_t)mh * mh;  // kry_gs_kernel's T
  KryState* dst = (KryState*)(Tm + (size_t)mh * mh);
  int* d_ns = (int*)(dst + 1);
  int nmult = 0;
  const double delta = 1.2, gamma = 0.9, break_tol = 1.0e-7;
  double eps = std::fabs((4.0 / 3.0 - 1.0) * 3.0 - 1.0);
  if (tol <= eps) tol = std::sqrt(eps);
  const double rndoff = eps * anorm;
  (void)rndoff;
  const double sgn = t >= 0 ? 1.0 : -1.0;
  const double t_out = std::fabs(t);
  const double sqr1 = std::sqrt(0.1);
  double t_now = 0.0, t_step = 0.0, t_last = 0.0, t_new = *stepguess;
  double xm = 1.0 / m;
  int nstep = 0;
  // w = v; beta = |w|
  SG_CUDA(cudaMemcpyAsync(w, v, sizeof(double2) * nc, cudaMemcpyDeviceToDevice, c.stream));
  KryState hst{};
  bool have_beta = false;
  ProfScope ps(c, ST_CI);
  // the cluster kernels where a slice of p and v_j fits shared memory and the device places
  // them, else one CTA
  const long long S = ((n + kGsCluster - 1) / kGsCluster + 1) / 2 * 2;
  const bool cluster = c.kry_cluster && S <= kGsSlice && gs_cluster_fits();
  while (t_now < t_out) {
    ++nstep;
    t_last = t_step;
    t_step = std::min(t_out - t_now, t_new);
    SG_CUDA(cudaMemsetAsync(Hm, 0, sizeof(double) * mh * mh, c.stream));
    kry_start_kernel<<<1, kKryThreads, 0, c.stream>>>((const double*)w, n, V, dst, have_beta ? 0 : 1);
    SG_LAUNCHED();
    for (int j = 0; j < m; ++j) {
      ++nmult;
      SG_TRY(ci_sigma(c, (const double2*)(V + (size_t)j * n), (double2*)(V + (size_t)(j + 1) * n), c.nucrepulsion, ez,
                      nucdipz, timefac, &dst->mbrk));
      if (cluster) {
        const long long tri = j * (j - 1) / 2;
        const int cap = (int)std::min<long long>(j, (kGsValues - tri) / S - 2);
        SG_TRY(launch_gs_cluster(c, cap == j ? kry_gs_kernel<true> : kry_gs_kernel<false>, kGsThreads, sizeof(double) * ((2 + cap) * (size_t)S + tri), true, V,
                                 n, (int)S, cap, j, Hm, mh, Tm, break_tol, dst));
      } else {
        kry_mgs_kernel<<<1, kKryThreads, 0, c.stream>>>(V, n, j, Hm, mh, break_tol, dst);
        SG_LAUNCHED();
      }
    }
    ++nmult;
    SG_TRY(ci_sigma(c, (const double2*)(V + (size_t)m * n), (double2*)(V + (size_t)(m + 1) * n), c.nucrepulsion, ez,
                    nucdipz, timefac, &dst->mbrk));
    kry_avnorm_kernel<<<1, kKryThreads, 0, c.stream>>>(V + (size_t)(m + 1) * n, n, dst);
    SG_LAUNCHED();
    SG_CUDA(cudaMemcpyAsync(&hst, dst, sizeof(KryState), cudaMemcpyDeviceToHost, c.stream));
    SG_CUDA(cudaStreamSynchronize(c.stream));
    have_beta = true;
    int k1 = 2, mbrkdwn = m;
    if (hst.mbrk) {
      k1 = 0;
      mbrkdwn = hst.mbrk;
      t_step = t_out - t_now;
    }
    {  // Hm(m+2, m+1) = 1  (expokit.f90:2356)
      const double one = 1.0;
      SG_CUDA(cudaMemcpyAsync(Hm + (size_t)m * mh + m + 1, &one, sizeof(double), cudaMemcpyHostToDevice, c.stream));
    }
    double err_loc = tol;
    double ex[2] = {0.0, 0.0};
    while (true) {
      const int mx = mbrkdwn + k1;
      SG_TRY(pade_expm(c, Hm, mh, mx, sgn * t_step, 0, exph, nullptr, pscr, d_ns));
      if (k1 == 0) {
        err_loc = tol;
        break;
      }
      SG_CUDA(cudaMemcpyAsync(ex, exph + m, sizeof(double) * 2, cudaMemcpyDeviceToHost, c.stream));
      SG_CUDA(cudaStreamSynchronize(c.stream));
      const double p1 = std::fabs(ex[0]) * hst.beta;
      const double p2 = std::fabs(ex[1]) * hst.beta * hst.avnorm;
      if (p1 > 10.0 * p2) {
        err_loc = p2;
        xm = 1.0 / m;
      } else {
        err_loc = p1;
        xm = 1.0 / (m - 1);
      }
      if (err_loc > delta * t_step * tol) {  // reject, step down (mxreject = 0)
        t_step = gamma * t_step * std::pow(t_step * tol / err_loc, xm);
        const double q = std::pow(10.0, fortran_nint(std::log10(t_step) - sqr1) - 1);
        t_step = std::trunc(t_step / q + 0.55) * q;
        continue;
      }
      break;
    }
    const int mxu = mbrkdwn + std::max(0, k1 - 1);
    if (cluster) {
      SG_TRY(launch_gs_cluster(c, kry_update_cluster_kernel, kKryThreads, 0, false, V, n, (int)S, mxu, exph, (double*)w, dst));
    } else {
      kry_update_kernel<<<1, kKryThreads, 0, c.stream>>>(V, n, mxu, exph, (double*)w, dst);
      SG_LAUNCHED();
    }
    SG_CUDA(cudaMemcpyAsync(&hst, dst, sizeof(KryState), cudaMemcpyDeviceToHost, c.stream));
    SG_CUDA(cudaStreamSynchronize(c.stream));
    t_new = gamma * t_step * std::pow(t_step * tol / err_loc, xm);
    const double q = std::pow(10.0, fortran_nint(std::log10(t_new) - sqr1) - 1);
    t_new = std::trunc(t_new / q + 0.55) * q;
    if (t_new < t_step) t_new = t_step;
    t_now += t_step;
    if (nstep >= 1000) break;
  }
  *stepguess = nstep == 1 ? t_step : t_last;
  if (nstep_out) *nstep_out = nstep;
  if (nmult_out) *nmult_out = nmult;
  return SINCGPU_OK;
}

}  // namespace sincgpu
