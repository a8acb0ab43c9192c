// Half-lengths of the Coulomb passes (coulomb_half.cuh) and the layouts that the
// set-up tables share with them: (M, M1, M2, NMIN), M = M1 * M2, for grids of NMIN to M
// points a side; the padded axis has 2 M points.  Two near-equal factors, so that both
// steps of a transform keep their threads busy, M1 <= M2, which takes fewer registers.
// NMIN is where the half-length passes beat the five passes at those grids' padded
// length (coulomb.cu) by a tenth or more; grids between the entries keep the five
// passes, and so do those below 46 points: alone they gained up to a sixth, but beside
// other kernels (a batch's graphs, the second stream) their large shared memory made
// neighbours wait (39^3 in a batch of eight: 6 % slower in all, 41^3: 1 %).  Measured, us per
// pair, half-length against five passes: 20: 1.07 / 1.34 (length 42), 28: 2.6 / 3.1 (64),
// 31: 3.8 / 3.3 (64), 35: 4.0 / 4.7 (72), 41: 6.3 / 6.5 (81), 45: 8.8 / 8.4 (90),
// 49: 10.2 / 11.8 (100), 56: 17.0 / 20.9 (120), 57: 22 / 21 (120), 63: 22.4 / 33.1 (126),
// 64: 24.5 / 35.2 (144), 72: 35.1 / 39.0 (144), 81: 45.2 / 71.1 (162), 90: 99 / 77 (180),
// 100: 112 / 149 (216).
#pragma once

#define SINCGPU_HALF_LENGTHS(X)                                                   \
  X(49, 7, 7, 46) X(56, 7, 8, 55) X(63, 7, 9, 61) X(64, 8, 8, 64) X(72, 8, 9, 65) \
  X(81, 9, 9, 73) X(100, 10, 10, 97)

namespace sincgpu {

// the half-length of a grid of n points a side and its factors, or -1
inline int half_length_for(int n, int* m1, int* m2) {
#define SINCGPU_HALF_ENTRY(M, A, B, NMIN) \
  if (n >= NMIN && n <= M) {              \
    if (m1) *m1 = A;                      \
    if (m2) *m2 = B;                      \
    return M;                             \
  }
  SINCGPU_HALF_LENGTHS(SINCGPU_HALF_ENTRY)
#undef SINCGPU_HALF_ENTRY
  return -1;
}

// Lines of M1 M2 points: LG of them share a group of 64 threads, S threads each.
constexpr int half_threads(int m1, int m2) { return m1 > m2 ? m1 : m2; }
constexpr int half_lines(int m1, int m2) { return 64 / half_threads(m1, m2); }
// Frequency (of 2 M) of index k of parity p.  For even M the odd parity is the
// frequencies 2 k + 1; for odd M it is 2 k + M, the plain transform of the input
// with alternating signs.
constexpr int half_freq(int M, int k, int p) { return M % 2 ? (2 * k + p * M) % (2 * M) : 2 * k + p; }
// Coprime factors: the y and z transforms go by the Chinese remainder (coulomb_half.cuh)
constexpr int half_gcd(int a, int b) { return b ? half_gcd(b, a % b) : a; }
constexpr bool half_pfa(int m1, int m2) { return half_gcd(m1, m2) == 1; }
// Frequency of indices (k1, k2) of the y and z transforms.  Coprime factors: the f with
// f = r_i modulo 2 m_i, where r_i = 2 k_i + p, or 2 k_i + p m_i for an odd m_i (the plain
// transform of alternating signs); else half_freq of k1 + m1 k2.
inline
#ifdef __CUDACC__
__host__ __device__
#endif
int half_freq2(int m1, int m2, int k1, int k2, int p) {
  const int M = m1 * m2;
  if (half_pfa(m1, m2)) {
    const int r1 = half_freq(m1, k1, p), r2 = half_freq(m2, k2, p);
    for (int f = r1; f < 2 * M; f += 2 * m1)
      if (f % (2 * m2) == r2) return f;
    return 0;
  }
  return half_freq(M, k1 + m1 * k2, p);
}
// The kernel spectrum in the order in which the z transforms read it: [fx <= M]
// [parity of ky][parity of kz][group of columns][k2][64 threads]
constexpr int half_col_groups(int m1, int m2) { return (m1 * m2 + half_lines(m1, m2) - 1) / half_lines(m1, m2); }
constexpr long long half_spec_plane(int m1, int m2) { return 4LL * half_col_groups(m1, m2) * m2 * 64; }
// Point of index (n1, s) of a y or z line: s + M2 n1, or M2 n1 + M1 s modulo M for coprime
// factors.  The rows of a plane are kept in the order s + M2 n1 of their z.  Places of a
// plane in W and V: blocks of the rows of one group and the y of one n1, so that the
// threads of a group read and write runs; blocks without any point are left out where
// they come last
constexpr int half_block(int m1, int m2) { return (half_lines(m1, m2) * m2 + 7) / 8 * 8; }
constexpr long long half_slots(int n, int m1, int m2) {
  if (half_pfa(m1, m2)) return (long long)half_col_groups(m1, m2) * m1 * half_block(m1, m2);
  return (long long)((n + half_lines(m1, m2) - 1) / half_lines(m1, m2)) * ((n + m2 - 1) / m2) * half_block(m1, m2);
}

}  // namespace sincgpu
