// Coulomb convolution on half-length transforms (the FP64 form's default).
//
// Inputs and kept outputs of every line lie in [0, N), N <= M, so the transform of
// length L = 2M splits by the parity p of the frequency f = 2k + p:
//   X[2k + p] = sum_{n < M} (x[n] w_L^(n p)) w_M^(n k),       w_m = exp(-2 pi i / m)
//   y[n]      = sum_p conj(w_L)^(n p) sum_k Y[2k + p] conj(w_M)^(n k)
// i.e. two length-M transforms without zero padding, the odd one twisted (for odd M
// the twist is an alternating sign, half_freq).  The 3-D convolution runs as
//   X  : rows of rho -> both parities of kx -> W[pair][kx][places (z, y)]
//   YZY: one CTA per (pair, kx) holds one M x M plane in shared memory and does,
//        for each parity of ky in turn, the y transforms in place, then per column
//        the z transforms of both parities, the real kernel spectrum and the
//        inverse z transforms, then the inverse y transforms; the even parity's
//        result waits in V (L2) for the odd one's
//   XI : V rows along kx, both parities summed -> R (x < N)
// A line of M = M1 M2 points is transformed by S = max(M1, M2) threads in two
// steps with one exchange in place:
//   step 1: thread s < M2 owns n = s + M2 n1 and leaves k1 at position s + M2 k1
//   step 2: thread t < M1 owns positions M2 t + n2 and leaves frequency t + M1 k2
//           at position M2 t + k2
// The frequencies stay in that order: the kernel spectrum is stored in it, and the
// inverse runs the two steps backwards to natural order.  Thread t of the z
// columns holds the same frequencies after the forward transform and before the
// inverse one, so the spectrum is applied in registers.
// Coprime factors need no twiddles between the steps (Good and Thomas): with
// n = M2 n1 + M1 n2 - c M, c = 0 or 1, and f = r_i modulo 2 M_i (half_freq2),
//   w_L^(n f) = w_2M1^(n1 f) w_2M2^(n2 f) (-1)^(c f)
// so the y and z transforms of such M are two plain steps, for the odd parity with
// half-frequency transforms and the sign (-1)^c.  (The x passes keep the first form:
// its threads read consecutive x.)  The plane kernel's busiest unit is the shared-memory
// pipe (48^3: 90 % busy, a quarter of it bank conflicts; 81^3: 69 %, FP64 pipe 54 %, with 12
// warps an SM to cover latency and barriers), and the twiddles were a fifth of its
// wavefronts; for equal factors of odd M one set per thread serves both directions and
// parities and stays in registers.
//
// Why this form (81^3 grid, 16 orbitals, ms per evaluation): the five passes
// through HBM (coulomb_kernels.cuh) took 9.7 and were bound by the z pass (4.5), whose
// length-162 lines (18 x 9) idle half of their threads in half of the steps and
// keep two CTAs of 9 warps per SM.  Here the slab with both ky and kx transformed
// (68 MB per pair) is never stored, every line is the balanced 9 x 9, and lines
// belong to groups of two warps that synchronise among themselves, so only the
// three phases of a plane need the whole CTA: 6.1 in all (X 0.80, YZY 4.6, XI 0.67),
// against 1.6 that its bytes (W and V written and read once) take at the measured HBM
// rate and some 2.8 that its FP64 instructions take at the pipe's rate.
#pragma once
#include "context.hpp"
#include "coul_half.h"
#include "fft_reg.cuh"

namespace sincgpu {

struct HalfArgs {
  int N, nspf, herm;
  long long G, NS;    // NS: places of a plane (half_slots)
  const double2* tw;  // twiddles between the two steps (HalfPlan::TW)
  const double* kht;  // kernel spectrum / L^3 (half_spec_plane)
  double2* W;         // [pair][kx parity][kx position][place]
  double2* V;         // the same layout, after the plane kernel
  const int* pa;
  const int* pb;
  int pair0;
  int npair_total;
};

// the smallest transform length of the twiddle table that M divides
constexpr int const_roots_for(int M) {
  for (int i = 0; i < kNumFftLens; ++i)
    if (kFftLens[i] % M == 0) return kFftLens[i];
  return -1;
}

// DFT of length M in registers, with the half-frequency twist when ODD:
// forward: a[k] = sum_n a[n] w_2M^(n (2k + ODD)); inverse: a[n] = sum_k a[k] conj(w_2M)^(n (2k + ODD))
template <int M, bool INV, bool ODD>
__device__ __forceinline__ void half_dft(double2 (&a)[M]) {
  constexpr int P = const_roots_for(ODD ? 2 * M : M);
  static_assert(P > 0, "no twiddles for this length");
  const ConstRoots<P, double2> cr;
  if constexpr (ODD && !INV) {
#pragma unroll
    for (int n = 1; n < M; ++n) a[n] = cmul(a[n], cr[n * (P / (2 * M))]);
  }
  RegFFT<M, 1, INV, double2>::run(a, cr, P);
  if constexpr (ODD && INV) {
#pragma unroll
    for (int n = 1; n < M; ++n) a[n] = cmul(a[n], root<true>(cr, n * (P / (2 * M))));
  }
}

// a[] with the odd elements' signs changed
template <int M>
__device__ __forceinline__ void alternate(double2 (&a)[M]) {
#pragma unroll
  for (int n = 1; n < M; n += 2) a[n] = make_double2(-a[n].x, -a[n].y);
}
// The factor transforms of coprime plans: half-frequency when ODD, for an odd length
// as the plain transform of alternating signs (index k is then 2 k + M of 2 M)
template <int M, bool INV, bool ODD>
__device__ __forceinline__ void half_factor(double2 (&a)[M]) {
  if constexpr (M % 2 != 0) {
    if constexpr (ODD && !INV) alternate<M>(a);
    half_dft<M, INV, false>(a);
    if constexpr (ODD && INV) alternate<M>(a);
  } else {
    half_dft<M, INV, ODD>(a);
  }
}

// Thread and memory layout of lines of M = M1 M2 points.  Consecutive threads run
// along a line (row lines) or across lines (column lines); a plane row is PITCH
// values.  With 16-byte values eight lanes fill the banks, so consecutive threads
// should step the address by 1 modulo 8 across line ends too: for column lines
// PITCH = LG, for row lines PITCH = S (rows in order) or -S (a group's rows in
// reverse order), all modulo 8; both hold for S = 6, 7, 8, 9, 10.  Step 2 strides by
// ST2, made odd.
template <int M1_, int M2_>
struct HalfPlan {
  static constexpr int M1 = M1_, M2 = M2_, M = M1 * M2, L = 2 * M;
  static constexpr bool PFA = half_pfa(M1, M2);     // y and z without twiddles
  static constexpr bool ALT = M % 2 != 0;           // the odd parity's twist is (-1)^n
  static constexpr bool SQ = ALT && M1 == M2;       // the z twiddles stay in registers
  static constexpr int S = half_threads(M1, M2), LG = half_lines(M1, M2), BS = half_block(M1, M2);
  static constexpr int ST2 = M2 | 1;                // stored stride of step 2's blocks
  static constexpr int ROW = M1 * ST2;              // stored length of a line in a row
  static constexpr int want = (LG % 8 ? LG : S) % 8;
  static constexpr int PITCH = ROW + (want - ROW % 8 + 8) % 8;
  static constexpr bool REV = (LG % 8) != 0 && (8 - LG % 8) % 8 == S % 8;
  static constexpr int groups = half_col_groups(M1, M2);  // line groups of a plane
  static constexpr size_t plane_bytes = sizeof(double2) * ((size_t)(M - 1) * PITCH + ROW);
  // twiddles [parity][k1][s], rows of odd length, so that threads along s (forward)
  // and along k1 (inverse) both step through the banks
  static constexpr int TS = M2 | 1, TW = (ALT ? 1 : 2) * M1 * TS;
  static constexpr size_t smem = plane_bytes + sizeof(double2) * TW;
  static constexpr bool fits = smem + 1024 <= 228 * 1024;
  // registers a thread of the plane kernel needs without spilling (the input and the
  // even parity's result beside a working set, or beside a block and its spectrum;
  // the twisted transforms of even M take some more)
  static constexpr int REGS = (12 * M1 + 2 * M2 > 8 * M1 + 6 * M2 ? 12 * M1 + 2 * M2 : 8 * M1 + 6 * M2) + (PFA ? 46 : SQ ? 30 : 46);
  // thread groups per CTA: the count with the most busy groups on an SM (resident CTAs
  // by shared memory and by the 512 x 32 registers of each of the four schedulers,
  // groups idle in a plane's last round taken off), the most CTAs on ties, so that one
  // computes while another waits
  static constexpr int resident(int ng) {
    int r = (int)(228 * 1024 / (smem + 1024));
    while (r > 1 && 512 / ((2 * ng * r + 3) / 4) / 8 * 8 < REGS) --r;
    return r;
  }
  static constexpr int busy(int ng) {  // in 1/64
    const int rounds = (groups + ng - 1) / ng;
    return resident(ng) * groups * 64 / rounds;
  }
  static constexpr int best() {
    int b = 1;
    for (int ng = 2; ng <= 8; ++ng)
      if (busy(ng) > busy(b)) b = ng;
    return b;
  }
  static constexpr int NG = best(), T = 64 * NG, ctas = resident(NG);
  // x passes: two groups per CTA (four, or one, measured 2 % and 1 % slower in all at 81^3)
  static constexpr int XG = 2, XT = 64 * XG, XL = XG * LG, XC = M2 <= 7 ? 5 : 4;
  static constexpr size_t xbuf = sizeof(double2) * (size_t)XL * PITCH;

  // stored place in a row of position q (q = M2 t + k2)
  __device__ __forceinline__ static int at(int q) { return ST2 == M2 ? q : (q / M2) * ST2 + q % M2; }
  // row of the plane of line l of row group gi
  __device__ __forceinline__ static int row(int gi, int l) { return gi * LG + (REV ? LG - 1 - l : l); }
  // point of index s + M2 n1 of a y or z line
  __device__ __forceinline__ static int point(int i) {
    if constexpr (!PFA) return i;
    const int n1 = i / M2, t = M2 * n1 + M1 * (i - M2 * n1);
    return t < M ? t : t - M;
  }
  // the first n1 for which M2 n1 + M1 s wraps
  __device__ __forceinline__ static int wraps(int s) { return (M - M1 * s + M2 - 1) / M2; }
  // row groups and blocks of a group in W and V
  __device__ __forceinline__ static int row_groups(int N) { return PFA ? groups : (N + LG - 1) / LG; }
  __device__ __forceinline__ static int blocks(int N) { return PFA ? M1 : (N + M2 - 1) / M2; }
  // (z, y) of a place; false where the place holds nothing
  __device__ __forceinline__ static bool place(int slot, int N, int* z, int* y) {
    const int nb = blocks(N);
    const int blk = slot / BS, i = slot - blk * BS, gi = blk / nb, n1 = blk - gi * nb, l = i / M2, s = i - l * M2;
    if (l >= LG || row(gi, l) >= M) return false;
    *z = point(row(gi, l));
    *y = point(s + M2 * n1);
    return *z < N && *y < N;
  }
};

// waits for the 64 threads of group g
__device__ __forceinline__ void group_sync(int g) { asm volatile("bar.sync %0, 64;" ::"r"(g + 1) : "memory"); }

// v with its sign changed where m is the sign bit of the high word
__device__ __forceinline__ double2 flip(double2 v, unsigned m) {
  return make_double2(__hiloint2double(__double2hiint(v.x) ^ (int)m, __double2loint(v.x)),
                      __hiloint2double(__double2hiint(v.y) ^ (int)m, __double2loint(v.y)));
}
// sign masks of the values n = s + M2 n1 (n1 even, odd) of parity p for odd M
struct AltSign {
  unsigned even, odd;
  __device__ __forceinline__ AltSign(int s, int p) {
    even = p && (s & 1) ? 0x80000000u : 0u;
    odd = p && !(s & 1) ? 0x80000000u : 0u;
  }
};

// twiddle between the two steps: w_L^(s (2 k + p)), forward or conjugated
template <class PL, bool INV, int ODD>
__device__ __forceinline__ double2 half_tw(const double2* tw, int s, int k) {
  return root<INV>(tw, ((PL::ALT ? 0 : ODD) * PL::M1 + k) * PL::TS + s);
}

// the twiddles of thread s of forward step 1, and of thread t of inverse step 1
template <class PL, int ODD>
struct FwdTw {
  double2 v[PL::M1];
  __device__ __forceinline__ FwdTw(const double2* tw, int s) {
    if constexpr (PL::PFA) return;
    if (s >= PL::M2) s = 0;
#pragma unroll
    for (int k = 0; k < PL::M1; ++k) v[k] = half_tw<PL, false, ODD>(tw, s, k);
  }
  __device__ __forceinline__ double2 operator()(int k) const { return v[k]; }
};
template <class PL, int ODD>
struct InvTw {
  double2 v[PL::M2];
  __device__ __forceinline__ InvTw(const double2* tw, int t) {
    if constexpr (PL::PFA) return;
    if (t >= PL::M1) t = 0;
#pragma unroll
    for (int n2 = 0; n2 < PL::M2; ++n2) v[n2] = half_tw<PL, true, ODD>(tw, n2, t);
  }
  __device__ __forceinline__ double2 operator()(int n2) const { return v[n2]; }
};

// Steps of the twiddled form.  Forward step 1 on w[] (n = s + M2 n1), the result to
// positions s + M2 k1: put(k1, v).  ODD and sg: the parity, as a template for even M and
// as signs for odd M.
template <class PL, int ODD, class TWF, class PUT>
__device__ __forceinline__ void half_fwd1(double2 (&w)[PL::M1], AltSign sg, const TWF& tw, PUT put) {
  constexpr bool TWIST = ODD && !PL::ALT;
  if constexpr (PL::ALT) {
#pragma unroll
    for (int n1 = 0; n1 < PL::M1; ++n1) w[n1] = flip(w[n1], n1 & 1 ? sg.odd : sg.even);
  }
  half_dft<PL::M1, false, TWIST>(w);
#pragma unroll
  for (int k1 = 0; k1 < PL::M1; ++k1) {
    double2 v = w[k1];
    if (k1 > 0 || TWIST) v = cmul(v, tw(k1));
    put(k1, v);
  }
}
// inverse step 1 on b[] (frequencies t + M1 k2): put(n2, v)
template <class PL, class TWF, class PUT>
__device__ __forceinline__ void half_inv1(double2 (&b)[PL::M2], const TWF& tw, PUT put) {
  half_dft<PL::M2, true, false>(b);
#pragma unroll
  for (int n2 = 0; n2 < PL::M2; ++n2) {
    double2 v = b[n2];
    if (n2 > 0) v = cmul(v, tw(n2));
    put(n2, v);
  }
}
// inverse step 2 on w[] (positions s + M2 k1), to n = s + M2 n1
template <class PL, int ODD>
__device__ __forceinline__ void half_inv2(double2 (&w)[PL::M1], AltSign sg) {
  half_dft<PL::M1, true, ODD && !PL::ALT>(w);
  if constexpr (PL::ALT) {
#pragma unroll
    for (int n1 = 0; n1 < PL::M1; ++n1) w[n1] = flip(w[n1], n1 & 1 ? sg.odd : sg.even);
  }
}

// The y and z transforms' steps in either form.  ODD: the parity (for odd M of the
// twiddled form the parity is `sign`, ODD = 0, and both run the same code).
template <class PL, int ODD, class TWF, class PUT>
__device__ __forceinline__ void line_fwd1(double2 (&w)[PL::M1], int s, int sign, const TWF& tw, PUT put) {
  if constexpr (PL::PFA) {
    if constexpr (ODD) {
#pragma unroll
      for (int n1 = 1; n1 < PL::M1; ++n1) w[n1] = flip(w[n1], n1 >= PL::wraps(s) ? 0x80000000u : 0u);
    }
    half_factor<PL::M1, false, ODD != 0>(w);
#pragma unroll
    for (int k1 = 0; k1 < PL::M1; ++k1) put(k1, w[k1]);
  } else {
    half_fwd1<PL, ODD>(w, AltSign(s, sign), tw, put);
  }
}
template <class PL, int ODD>
__device__ __forceinline__ void line_fwd2(double2 (&b)[PL::M2]) {
  if constexpr (PL::PFA)
    half_factor<PL::M2, false, ODD != 0>(b);
  else
    half_dft<PL::M2, false, false>(b);
}
template <class PL, int ODD, class TWF, class PUT>
__device__ __forceinline__ void line_inv1(double2 (&b)[PL::M2], const TWF& tw, PUT put) {
  if constexpr (PL::PFA) {
    half_factor<PL::M2, true, ODD != 0>(b);
#pragma unroll
    for (int n2 = 0; n2 < PL::M2; ++n2) put(n2, b[n2]);
  } else {
    half_inv1<PL>(b, tw, put);
  }
}
template <class PL, int ODD>
__device__ __forceinline__ void line_inv2(double2 (&w)[PL::M1], int s, int sign) {
  if constexpr (PL::PFA) {
    half_factor<PL::M1, true, ODD != 0>(w);
    if constexpr (ODD) {
#pragma unroll
      for (int n1 = 1; n1 < PL::M1; ++n1) w[n1] = flip(w[n1], n1 >= PL::wraps(s) ? 0x80000000u : 0u);
    }
  } else {
    half_inv2<PL, ODD>(w, AltSign(s, sign));
  }
}

// X: rows of rho -> W[pair][parity][position][place].  XL places per CTA, LG per
// group; step 1 with the threads along a row, step 2 across the rows of the group, so
// that the frequencies leave in runs of LG places.
template <int M1, int M2, bool DENS>
__global__ void __launch_bounds__(HalfPlan<M1, M2>::XT, HalfPlan<M1, M2>::XC) half_fwd_x(const double2* __restrict__ phi1,
                                                                   const double2* __restrict__ phi2, HalfArgs ha) {
  using PL = HalfPlan<M1, M2>;
  constexpr int M = PL::M, S = PL::S;
  extern __shared__ __align__(16) double2 hsm[];
  double2* tw = hsm;
  const int N = ha.N, tid = threadIdx.x;
  for (int i = tid; i < PL::TW; i += PL::XT) tw[i] = ha.tw[i];
  const int g = tid >> 6, i = tid & 63;
  const int lr = i / S, sr = i - lr * S, sc = i / PL::LG, lc = i - sc * PL::LG;
  const int line = PL::REV ? PL::LG - 1 - lr : lr;
  double2* buf = hsm + PL::TW + g * PL::LG * PL::PITCH;
  // pairs fastest over the grid: the CTAs of one row block read the orbitals from L2
  const int p = blockIdx.x, c0 = blockIdx.y * PL::XL + g * PL::LG;
  int z, y;
  const bool row = lr < PL::LG && c0 + line < ha.NS && PL::place(c0 + line, N, &z, &y);
  const long long off = ((long long)z * N + y) * N;
  const double2 *s1, *s2 = nullptr;
  if (DENS) {
    s1 = phi1 + (long long)(ha.pair0 + p) * ha.G + off;
  } else {
    s1 = phi1 + (long long)ha.pa[p] * ha.G + off;
    s2 = phi2 + (long long)ha.pb[p] * ha.G + off;
  }
  double2 a[M1];
#pragma unroll
  for (int n1 = 0; n1 < M1; ++n1) {
    const int x = sr + M2 * n1;
    a[n1] = make_double2(0.0, 0.0);
    if (row && sr < M2 && x < N) a[n1] = DENS ? s1[x] : cmulc(s1[x], s2[x]);
  }
  const bool col = sc < M1 && c0 + lc < ha.NS;
  double2* out = ha.W + (long long)p * PL::L * ha.NS + (long long)(M2 * sc) * ha.NS + c0 + lc;
  __syncthreads();  // twiddles
  auto half = [&](auto odd) {
    constexpr int ODD = decltype(odd)::value;
    double2 w[M1];
#pragma unroll
    for (int n1 = 0; n1 < M1; ++n1) w[n1] = a[n1];
    if (lr < PL::LG && sr < M2)
      half_fwd1<PL, ODD>(w, AltSign(sr, ODD), [&](int k1) { return half_tw<PL, false, ODD>(tw, sr, k1); },
                         [&](int k1, double2 v) { buf[line * PL::PITCH + sr + PL::ST2 * k1] = v; });
    group_sync(g);
    if (col) {
      double2 b[M2];
#pragma unroll
      for (int n2 = 0; n2 < M2; ++n2) b[n2] = buf[lc * PL::PITCH + PL::ST2 * sc + n2];
      half_dft<M2, false, false>(b);
#pragma unroll
      for (int k2 = 0; k2 < M2; ++k2) out[(ODD * M + k2) * ha.NS] = b[k2];
    }
  };
  half(std::integral_constant<int, 0>{});
  group_sync(g);  // the buffer is read
  half(std::integral_constant<int, 1>{});
}

// the twiddles of the z transforms: from the table, or kept by the thread (equal factors
// of odd M: w_M^(s k) for both directions and parities)
template <class PL>
struct ZTw {
  const double2* tw;
  FwdTw<PL, 0> keep;
  int s;
  __device__ __forceinline__ ZTw(const double2* t, int s_) : tw(t), keep(t, PL::SQ ? s_ : 0), s(s_) {}
  template <int ODD>
  __device__ __forceinline__ double2 fwd(int k1) const {
    if constexpr (PL::SQ) return keep(k1);
    return half_tw<PL, false, ODD>(tw, s, k1);
  }
  template <int ODD>
  __device__ __forceinline__ double2 inv(int n2) const {
    if constexpr (PL::SQ) return cconj(keep(n2));
    return half_tw<PL, true, ODD>(tw, n2, s);
  }
};

// the z transforms of one column for one parity of kz: in: a[] (rows s + M2 n1), out:
// r[] (the same rows); pl: the column in the plane; w: this thread's spectrum, which
// is replaced by the one at `next` as soon as it is used
template <class PL, int ODD>
__device__ __forceinline__ void half_z(const double2 (&a)[PL::M1], double2 (&r)[PL::M1], bool act, int s, int g,
                                       double2* pl, double (&w)[PL::M2], const double* __restrict__ next,
                                       const ZTw<PL>& zt) {
  constexpr int M1 = PL::M1, M2 = PL::M2;
#pragma unroll
  for (int n1 = 0; n1 < M1; ++n1) r[n1] = a[n1];
  if (act && s < M2)
    line_fwd1<PL, ODD>(r, s, ODD, [&](int k1) { return zt.template fwd<ODD>(k1); },
                       [&](int k1, double2 v) { pl[(s + M2 * k1) * PL::PITCH] = v; });
  group_sync(g);
  if (act && s < M1) {
    double2 b[M2];
#pragma unroll
    for (int n2 = 0; n2 < M2; ++n2) b[n2] = pl[(M2 * s + n2) * PL::PITCH];
    line_fwd2<PL, ODD>(b);
#pragma unroll
    for (int k2 = 0; k2 < M2; ++k2) b[k2] = cscale(b[k2], w[k2]);
#pragma unroll
    for (int k2 = 0; k2 < M2; ++k2) w[k2] = __ldg(next + k2 * 64);
    line_inv1<PL, ODD>(b, [&](int n2) { return zt.template inv<ODD>(n2); },
                       [&](int n2, double2 v) { pl[(M2 * s + n2) * PL::PITCH] = v; });
  }
  group_sync(g);
  if (act && s < M2) {
#pragma unroll
    for (int k1 = 0; k1 < M1; ++k1) r[k1] = pl[(s + M2 * k1) * PL::PITCH];
    line_inv2<PL, ODD>(r, s, ODD);
  }
}

// YZY: one (pair, kx) plane
template <int M1, int M2>
__global__ void __launch_bounds__(HalfPlan<M1, M2>::T, HalfPlan<M1, M2>::ctas) half_yzy(HalfArgs ha) {
  using PL = HalfPlan<M1, M2>;
  constexpr int M = PL::M, S = PL::S;
  extern __shared__ __align__(16) double2 hsm[];
  double2* tw = hsm;
  double2* plane = hsm + PL::TW;
  const int N = ha.N, tid = threadIdx.x;
  if constexpr (!PL::PFA)
    for (int i = tid; i < PL::TW; i += PL::T) tw[i] = ha.tw[i];
  const int g = tid >> 6, i = tid & 63;
  const int lr = i / S, sr = i - lr * S;            // row lines: threads along the line
  const int sc = i / PL::LG, lc = i - sc * PL::LG;  // column lines: threads across lines
  const bool actr = lr < PL::LG, actc = sc < S;
  const int kx = blockIdx.x;  // parity * M + position
  const long long po = ((long long)blockIdx.y * PL::L + kx) * ha.NS + lr * M2 + sr;
  const double2* in = ha.W + po;
  double2* out = ha.V + po;
  const int nb = PL::blocks(N);
  const int px = kx >= M, qx = kx - px * M;
  const int fx = half_freq(M, qx / M2 + M1 * (qx % M2), px);
  const double* khx = ha.kht + (fx <= M ? fx : 2 * M - fx) * half_spec_plane(M1, M2) + i;
  __syncthreads();  // twiddles
  const int ngr = PL::row_groups(N);
  // y transforms of the plane's rows (zeros where z >= N)
  auto fwd_y = [&](auto odd, int py) {
    constexpr int ODD = decltype(odd)::value;
    const FwdTw<PL, ODD> ft(tw, sr);
    double2 nx[M1];  // the next round's values, on their way during this one
    auto fetch = [&](int gi) {
      const int row = PL::row(gi, lr);
      const bool ok = actr && sr < M2 && gi < ngr && row < M && PL::point(row) < N;
#pragma unroll
      for (int n1 = 0; n1 < M1; ++n1) nx[n1] = ok && n1 < nb ? in[(gi * nb + n1) * PL::BS] : make_double2(0.0, 0.0);
    };
    fetch(g);
#pragma unroll 1
    for (int gi = g; gi < PL::groups; gi += PL::NG) {
      const int row = PL::row(gi, lr);
      const bool ok = actr && row < M;
      double2* mine = plane + row * PL::PITCH;
      double2 w[M1];
#pragma unroll
      for (int n1 = 0; n1 < M1; ++n1) w[n1] = nx[n1];
      fetch(gi + PL::NG);
      if (ok && sr < M2)
        line_fwd1<PL, ODD>(w, sr, py, ft, [&](int k1, double2 v) { mine[sr + PL::ST2 * k1] = v; });
      group_sync(g);
      if (ok && sr < M1) {
        double2 b[M2];
#pragma unroll
        for (int n2 = 0; n2 < M2; ++n2) b[n2] = mine[PL::ST2 * sr + n2];
        line_fwd2<PL, ODD>(b);
#pragma unroll
        for (int k2 = 0; k2 < M2; ++k2) mine[PL::ST2 * sr + k2] = b[k2];
      }
    }
  };
  // inverse y transforms of the rows with z < N
  auto inv_y = [&](auto odd, int py) {
    constexpr int ODD = decltype(odd)::value;
    const InvTw<PL, ODD> it(tw, sr);
#pragma unroll 1
    for (int gi = g; gi < ngr; gi += PL::NG) {
      const int row = PL::row(gi, lr);
      const bool ok = actr && row < M && PL::point(row) < N;
      double2* mine = plane + row * PL::PITCH;
      if (ok && sr < M1) {
        double2 b[M2];
#pragma unroll
        for (int k2 = 0; k2 < M2; ++k2) b[k2] = mine[PL::ST2 * sr + k2];
        line_inv1<PL, ODD>(b, it, [&](int n2, double2 v) { mine[PL::ST2 * sr + n2] = v; });
      }
      double2* o = out + (long long)gi * nb * PL::BS;
      double2 v[M1];  // the even parity's result
#pragma unroll
      for (int n1 = 0; n1 < M1; ++n1)
        v[n1] = py && ok && sr < M2 && n1 < nb ? o[n1 * PL::BS] : make_double2(0.0, 0.0);
      group_sync(g);
      if (ok && sr < M2) {
        double2 w[M1];
#pragma unroll
        for (int k1 = 0; k1 < M1; ++k1) w[k1] = mine[sr + PL::ST2 * k1];
        line_inv2<PL, ODD>(w, sr, py);
#pragma unroll
        for (int n1 = 0; n1 < M1; ++n1)
          if (n1 < nb) o[n1 * PL::BS] = cadd(v[n1], w[n1]);
      }
    }
  };
  using Even = std::integral_constant<int, 0>;
  using Odd = std::integral_constant<int, 1>;
#pragma unroll 1
  for (int py = 0; py < 2; ++py) {
    if ((PL::ALT && !PL::PFA) || !py)
      fwd_y(Even{}, py);
    else
      fwd_y(Odd{}, 1);
    __syncthreads();
    // z transforms of the M columns
    const double* kh = khx + (2 * py) * PL::groups * (M2 * 64);
    const ZTw<PL> zt(tw, sc);
    double w[M2];
#pragma unroll
    for (int k2 = 0; k2 < M2; ++k2) w[k2] = __ldg(kh + g * (M2 * 64) + k2 * 64);
#pragma unroll 1
    for (int gi = g; gi < PL::groups; gi += PL::NG) {
      const int q = gi * PL::LG + lc;
      const bool ok = actc && q < M;
      double2* mine = plane + PL::at(q);
      const int gn = gi + PL::NG < PL::groups ? gi + PL::NG : gi;  // the next round's columns
      double2 a[M1], r[M1], r1[M1];
#pragma unroll
      for (int n1 = 0; n1 < M1; ++n1)
        a[n1] = ok && sc < M2 ? mine[(sc + M2 * n1) * PL::PITCH] : make_double2(0.0, 0.0);
      half_z<PL, 0>(a, r, ok, sc, g, mine, w, kh + (PL::groups + gi) * (M2 * 64), zt);
      half_z<PL, 1>(a, r1, ok, sc, g, mine, w, kh + gn * (M2 * 64), zt);
      if (ok && sc < M2) {
#pragma unroll
        for (int n1 = 0; n1 < M1; ++n1) mine[(sc + M2 * n1) * PL::PITCH] = cadd(r[n1], r1[n1]);
      }
    }
    __syncthreads();
    if ((PL::ALT && !PL::PFA) || !py)
      inv_y(Even{}, py);
    else
      inv_y(Odd{}, 1);
    if (!py) __syncthreads();  // the plane is read
  }
}

// XI: V[pair][parity][position][place] -> R, the X pass backwards: step 1 across the
// rows of a group (runs of LG places), step 2 along the rows
template <int M1, int M2, bool DENS>
__global__ void __launch_bounds__(HalfPlan<M1, M2>::XT, HalfPlan<M1, M2>::XC) half_inv_x(HalfArgs ha, double* __restrict__ Rpl,
                                                                   double2* __restrict__ full) {
  using PL = HalfPlan<M1, M2>;
  constexpr int M = PL::M, S = PL::S;
  extern __shared__ __align__(16) double2 hsm[];
  double2* tw = hsm;
  const int N = ha.N, tid = threadIdx.x;
  for (int i = tid; i < PL::TW; i += PL::XT) tw[i] = ha.tw[i];
  const int g = tid >> 6, i = tid & 63;
  const int lr = i / S, sr = i - lr * S, sc = i / PL::LG, lc = i - sc * PL::LG;
  const int line = PL::REV ? PL::LG - 1 - lr : lr;
  double2* buf = hsm + PL::TW + g * PL::LG * PL::PITCH;
  const int p = blockIdx.y, c0 = blockIdx.x * PL::XL + g * PL::LG;
  const bool col = sc < M1 && c0 + lc < ha.NS;
  const double2* in = ha.V + (long long)p * PL::L * ha.NS + (long long)(M2 * sc) * ha.NS + c0 + lc;
  double2 b[2][M2];  // both parities' frequencies on their way at once
#pragma unroll
  for (int odd = 0; odd < 2; ++odd)
#pragma unroll
    for (int k2 = 0; k2 < M2; ++k2)
      b[odd][k2] = col ? in[(odd * M + k2) * ha.NS] : make_double2(0.0, 0.0);
  int z, y;
  const bool row = lr < PL::LG && sr < M2 && c0 + line < ha.NS && PL::place(c0 + line, N, &z, &y);
  double2 r[M1];
  __syncthreads();  // twiddles
  auto half = [&](auto odd) {
    constexpr int ODD = decltype(odd)::value;
    if (col)
      half_inv1<PL>(b[ODD], [&](int n2) { return half_tw<PL, true, ODD>(tw, n2, sc); },
                    [&](int n2, double2 v) { buf[lc * PL::PITCH + PL::ST2 * sc + n2] = v; });
    group_sync(g);
    if (row) {
      double2 w[M1];
#pragma unroll
      for (int k1 = 0; k1 < M1; ++k1) w[k1] = buf[line * PL::PITCH + sr + PL::ST2 * k1];
      half_inv2<PL, ODD>(w, AltSign(sr, ODD));
#pragma unroll
      for (int n1 = 0; n1 < M1; ++n1) r[n1] = ODD ? cadd(r[n1], w[n1]) : w[n1];
    }
  };
  half(std::integral_constant<int, 0>{});
  group_sync(g);  // the buffer is read
  half(std::integral_constant<int, 1>{});
  if (!row) return;
  const long long G = ha.G, g0 = ((long long)z * N + y) * N;
  const int gp = ha.pair0 + p;
  long long off_ab, off_ba = 0;
  bool mirror = false;
  if (DENS) {
    off_ab = G * gp;
  } else {
    const int a = ha.pa[p], b = ha.pb[p];
    off_ab = G * ((long long)a + (long long)ha.nspf * b);
    off_ba = G * ((long long)b + (long long)ha.nspf * a);
    mirror = ha.herm && a != b;
  }
#pragma unroll
  for (int n1 = 0; n1 < M1; ++n1) {
    const int x = sr + M2 * n1;
    if (x >= N) continue;
    const long long at = g0 + x;
    if (Rpl) {
      Rpl[(long long)gp * G + at] = r[n1].x;
      Rpl[(long long)(ha.npair_total + gp) * G + at] = r[n1].y;
    }
    if (full) {
      full[off_ab + at] = r[n1];
      if (mirror) full[off_ba + at] = cconj(r[n1]);
    }
  }
}

// Launches the three passes for a chunk of np pairs.
template <int M1, int M2>
int half_launch(Ctx& c, const HalfArgs& ha, int np, bool dens, const double2* src1, const double2* src2, double* Rpl,
                double2* full) {
  using PL = HalfPlan<M1, M2>;
  static_assert(PL::fits, "the plane does not fit one SM");
  constexpr size_t xs = sizeof(double2) * PL::TW + PL::xbuf;
  // process-wide attributes, one fixed value each (thread-safe static initialisation)
  static const cudaError_t attr = [] {
    struct {
      const void* k;
      size_t b;
    } ks[] = {{(const void*)half_fwd_x<M1, M2, false>, xs}, {(const void*)half_fwd_x<M1, M2, true>, xs},
              {(const void*)half_inv_x<M1, M2, false>, xs}, {(const void*)half_inv_x<M1, M2, true>, xs},
              {(const void*)half_yzy<M1, M2>, PL::smem}};
    for (const auto& k : ks) {
      const cudaError_t e = cudaFuncSetAttribute(k.k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)k.b);
      if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
  }();
  SG_CUDA(attr);
  const int nrow = ceil_div(ha.NS, PL::XL);
  {
    ProfScope ps(c, ST_COUL_FWD_X);
    if (dens)
      half_fwd_x<M1, M2, true><<<dim3(np, nrow), PL::XT, xs, c.stream>>>(src1, nullptr, ha);
    else
      half_fwd_x<M1, M2, false><<<dim3(np, nrow), PL::XT, xs, c.stream>>>(src1, src2, ha);
    SG_LAUNCHED();
  }
  {
    ProfScope ps(c, ST_COUL_YZY);
    half_yzy<M1, M2><<<dim3(PL::L, np), PL::T, PL::smem, c.stream>>>(ha);
    SG_LAUNCHED();
  }
  {
    ProfScope ps(c, ST_COUL_INV_X);
    if (dens)
      half_inv_x<M1, M2, true><<<dim3(nrow, np), PL::XT, xs, c.stream>>>(ha, Rpl, full);
    else
      half_inv_x<M1, M2, false><<<dim3(nrow, np), PL::XT, xs, c.stream>>>(ha, Rpl, full);
    SG_LAUNCHED();
  }
  return SINCGPU_OK;
}

#define SINCGPU_HALF_DECLARE(M, A, B, NMIN)                                                                       \
  extern template int half_launch<A, B>(Ctx&, const HalfArgs&, int, bool, const double2*, const double2*, double*, \
                                        double2*);
SINCGPU_HALF_LENGTHS(SINCGPU_HALF_DECLARE)
#undef SINCGPU_HALF_DECLARE
#define SINCGPU_HALF_INSTANTIATE(A, B)                                                                    \
  template int half_launch<A, B>(Ctx&, const HalfArgs&, int, bool, const double2*, const double2*, double*, \
                                 double2*);

}  // namespace sincgpu
