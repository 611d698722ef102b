// Two-stage plane passes for N = P x Q, FP32 and FP64: every line transform is
// two register DFTs (length P, then Q) with one exchange through shared memory,
// run as tasks of one thread each (a line has Q tasks of the first and P of the
// second stage), so that any P x Q fills the warps, unlike a fixed group of
// lanes per line.
//
// A transformed line is kept as a P x QS table (QS = Q | 1: lanes of the second
// stage QS elements apart hit distinct banks):
//   forward order of use ("s"):  element q + Q r at [r][q]
//   after the two stages ("b"):  element k + P m at [k][m]
// and back, so each task writes where it read: no exchange buffer, no ordering
// inside a stage.  With n = q + Q r, j = k + P m:
//   s2b: X[k + P m] = sum_q W_Q^{q m} [W_N^{q k} sum_r x[q + Q r] W_P^{r k}]
//   b2s: Z[a + Q b] = sum_k W_P^{k b} [W_N^{k a} sum_m y[k + P m] W_Q^{m a}]
// (W conjugated for the inverse).  The C2R of a row pair ends in the registers
// of its second-stage tasks, where the density is accumulated or V_KS
// multiplied in, and the R2C starts from the same registers.
//
// Per (plane, state) item a block transforms the columns by block-wide tasks
// (pencil values found through a column map, so the plane is neither zeroed nor
// scattered), then each warp takes G row pairs at a time.  G and the warps per
// block are chosen so that G Q and G P tasks nearly fill rounds of 32 lanes and
// the blocks' warps nearly divide the N / 2 row pairs.
#pragma once
#include <algorithm>
#include "fft_smem.cuh"

// ---- register DFTs -------------------------------------------------------
// composite R = A B with coprime A, B by the prime-factor map (no twiddles):
// input (B n2 + A n1) mod R, output k with k1 = k mod B, k2 = k mod A
template <typename T, int R, bool INV>
__device__ __forceinline__ void rdft(cplx<T> (&v)[R]);

template <typename T, int A, int B, bool INV>
__device__ __forceinline__ void rdft_pfa(cplx<T> (&v)[A * B]) {
  constexpr int R = A * B;
  cplx<T> u[A][B];
#pragma unroll
  for (int n2 = 0; n2 < A; ++n2) {
#pragma unroll
    for (int n1 = 0; n1 < B; ++n1) u[n2][n1] = v[(B * n2 + A * n1) % R];
    rdft<T, B, INV>(u[n2]);
  }
#pragma unroll
  for (int k1 = 0; k1 < B; ++k1) {
    cplx<T> c[A];
#pragma unroll
    for (int n2 = 0; n2 < A; ++n2) c[n2] = u[n2][k1];
    rdft<T, A, INV>(c);
#pragma unroll
    for (int k = 0; k < R; ++k)
      if (k % B == k1) v[k] = c[k % A];
  }
}

// length 7 from its three symmetric and antisymmetric pairs
template <typename T, bool INV>
__device__ __forceinline__ void rdft7(cplx<T> (&v)[7]) {
  const T c[4] = {(T)1, (T)0.62348980185873353053, (T)-0.22252093395631440429,
                  (T)-0.90096886790241912624};
  const T s[4] = {(T)0, (T)0.78183148246802980871, (T)0.97492791218182360702,
                  (T)0.43388373911755812048};
  cplx<T> p[4], m[4];
#pragma unroll
  for (int j = 1; j < 4; ++j) {
    p[j] = v[j] + v[7 - j];
    m[j] = v[j] - v[7 - j];
  }
  const cplx<T> x0 = v[0];
  v[0] = (x0 + p[1]) + (p[2] + p[3]);
#pragma unroll
  for (int k = 1; k < 4; ++k) {
    cplx<T> a = x0, b = mk<T>(0, 0);
#pragma unroll
    for (int j = 1; j < 4; ++j) {
      const int q = (j * k) % 7, h = q > 3 ? 7 - q : q;
      a = a + cscale(p[j], c[h]);
      b = b + cscale(m[j], q > 3 ? -s[h] : s[h]);
    }
    const cplx<T> ib = mul_i(b, INV);  // forward: -i b
    v[k] = a + ib;
    v[7 - k] = a - ib;
  }
}

template <typename T, int R, bool INV>
__device__ __forceinline__ void rdft(cplx<T> (&v)[R]) {
  if constexpr (R == 6) rdft_pfa<T, 2, 3, INV>(v);
  else if constexpr (R == 7) rdft7<T, INV>(v);
  else if constexpr (R == 10) rdft_pfa<T, 2, 5, INV>(v);
  else if constexpr (R == 12) rdft_pfa<T, 4, 3, INV>(v);
  else if constexpr (R == 20) rdft_pfa<T, 4, 5, INV>(v);
  else Dft<T, R, INV>::template run<R>(v, nullptr);
}

// ---- shapes -----------------------------------------------------------------
// P, Q; G row pairs per warp and round; W warps per block; YS row splits of the
// density pass (its FP64 accumulators of a 200 x 200 plane exceed a register
// file: three blocks take a third of the rows each and repeat the columns).
// Of the factorings of a size the FP32 error decides before the time: 40 = 10 x 4 had a
// V.psi error of 3.05e-8 where the one-stage passes have 2.90e-8, 8 x 5 3.19e-8, 4 x 10
// 3.54e-8, 5 x 8 2.72e-8 (64 states, density + V.psi: 101 us as 10 x 4, 97 as 5 x 8).
template <int N> struct TwoCfg { static constexpr bool ok = false; };
#define CPSTEP_TWO(N_, P_, Q_, G_, W_, YS_)                                     \
  template <> struct TwoCfg<N_> {                                              \
    static constexpr bool ok = true;                                           \
    static constexpr int P = P_, Q = Q_, G = G_, W = W_, YS = YS_;              \
  }
CPSTEP_TWO(28, 7, 4, 8, 2, 1);
CPSTEP_TWO(32, 8, 4, 8, 2, 1);
CPSTEP_TWO(40, 5, 8, 4, 5, 1);
CPSTEP_TWO(42, 7, 6, 4, 6, 1);
CPSTEP_TWO(48, 8, 6, 4, 6, 1);
CPSTEP_TWO(60, 10, 6, 5, 6, 1);
CPSTEP_TWO(64, 8, 8, 4, 8, 1);
CPSTEP_TWO(80, 10, 8, 8, 5, 1);
CPSTEP_TWO(96, 12, 8, 8, 6, 1);
CPSTEP_TWO(120, 12, 10, 5, 12, 1);
CPSTEP_TWO(128, 16, 8, 4, 8, 1);
CPSTEP_TWO(200, 20, 10, 3, 12, 3);
#undef CPSTEP_TWO

template <typename T, int N, bool DENS = false>
struct TwoShape {
  using C = TwoCfg<N>;
  static constexpr int P = C::P, Q = C::Q, G = C::G, QS = Q | 1;
  // the FP32 density of a 128 x 128 plane: 16 warps, whose accumulators leave room
  // for two rounds of tasks (8 warps of twice the accumulators: 351 us, 16: 306 us
  // for 64 states)
  static constexpr int W = DENS && N == 128 && sizeof(T) == 4 ? 16 : C::W;
  static constexpr int THREADS = 32 * W;
  static constexpr int LL = P * QS;
  static constexpr int LC = LL | 1;  // column stride: lanes of consecutive kx on distinct banks
  // scratch line stride = Q mod 16 in FP32: the first stage's lanes (q, then the
  // next line) run through consecutive banks
  static constexpr int LS = sizeof(T) == 4 ? LL + (((Q - LL) % 16) + 16) % 16 : LL;
  static constexpr int PAIRS = N / 2;
  static constexpr int R1 = (G * Q + 31) / 32, R2 = (G * P + 31) / 32;  // rounds of tasks
  static constexpr int passes(int ys) { return (PAIRS + ys * W * G - 1) / (ys * W * G); }
  static constexpr size_t bytes(int nplx, int nlines) {
    return sizeof(cplx<T>) * (2 * (size_t)N + (size_t)nplx * LC + (size_t)W * G * LS +
                              (size_t)((nlines + 1) & ~1)) +
           (sizeof(unsigned short) * (size_t)nplx * N + 15) / 16 * 16;
  }
  // blocks per SM the registers are planned for: the larger DFT (with V_KS beside
  // the second one), the density's FP64 accumulators, addresses
  static constexpr int regs() {
    const int wd = (int)sizeof(T) / 4;
    return DENS ? 4 * passes(C::YS) * R2 * Q + 2 * wd * std::max(P, Q) + 40
                   : wd * std::max(2 * P, 4 * Q) + 40;
  }
  static constexpr int minb() {
    const int r = std::min(255, regs());
    return std::max(1, std::min(32, 65536 / ((r + 7) / 8 * 8 * THREADS)));
  }
};

// Real-space passes of single arrays (the density sphere): one block of 16 warps
// per plane; G row pairs per warp and round, fewer where the plane leaves less
// shared memory.
template <typename T, int N>
struct TwoReal {
  using S = TwoShape<T, N>;
  static constexpr int THREADS = 512, W = THREADS / 32;
  static constexpr size_t bytes_g(int nplx, int G) {
    return sizeof(cplx<T>) * (2 * (size_t)N + (size_t)nplx * S::LC + (size_t)W * G * S::LL);
  }
  static constexpr int g_fit(int G) {
    return G > 1 && bytes_g(N / 2, G) > 225 * 1024 ? g_fit(G - 1) : G;
  }
  static constexpr int G = g_fit((N / 2 + W - 1) / W);
  static constexpr size_t bytes(int nplx) { return bytes_g(nplx, G); }
};

template <int N>
struct TwoPos {
  static constexpr int P = TwoCfg<N>::P, Q = TwoCfg<N>::Q, QS = Q | 1;
  __device__ static __forceinline__ int s(int i) { return i / Q * QS + i % Q; }  // "s" order
  __device__ static __forceinline__ int b(int i) { return i % P * QS + i / P; }  // "b" order
};
