// PairCalculator products (FP64 path; the mixed-precision context sends
// them to the tensor-core kernels of paircalc_tc.cu where those apply).
//
//   overlap:      C(i,j) = alpha * sum_p wpt_p Re(conj a_i(p) b_j(p)) (+ beta C)
//                 = the reference's 2 * psi_r^T psi_r with Gx=0 rows scaled by
//                 1/sqrt(2) (ckPairCalculator.C:682-751, multiplyForward 'T','N'
//                 with alpha = 2 for double pack; scaling CP_State_GSpacePlane.C:
//                 1933-1954, :3120-3123).  C is column-major (ld = ldc).
//   backmultiply: out_i(p) = alpha * sum_j M(j,i) in_j(p) + beta * out_i(p),
//                 M column-major: psi.T ('N','N', ckPairCalculator.C:1314) and
//                 the gamma / lambda products (:1358, :1408, :1497).
//   dgemm:        column-major BLAS semantics, the myGEMM wrapper
//                 (ckPairCalculator.C:57-66).
//
// All three run on the FP64 tensor units; the overlap is split over K (the
// reference's numChunks K-split, pcCommManager.C:165-172) with a fixed-order
// reduction of the partial tiles, so results are deterministic.  The overlap that
// allocates nothing (cpstep_pc_overlap_noalloc) keeps its own scalar kernel,
// k_overlap_part, whose splits fit the fixed buffer.
#include <algorithm>
#include <mutex>
#include <cuda.h>
#include "ctx.cuh"
#include "dmma.cuh"

namespace pcalc {

constexpr int BM = 64, BN = 64, BK = 16, NT = 256;

// C_part[ks] (BM x BN tiles, column-major, ld = M) for the K-slab of split ks.
// A: [M][K] row-major (lda), B: [N][K] row-major (ldb), K counted in reals;
// w (per complex point) multiplies column k by w[k/2] when non-null.
__global__ void __launch_bounds__(NT)
k_overlap_part(const double* __restrict__ A, int lda, const double* __restrict__ B, int ldb,
               const double* __restrict__ w, int M, int N, int K, int kslab,
               double* __restrict__ part) {
  __shared__ double As[BK][BM + 1];
  __shared__ double Bs[BK][BN + 1];
  const int i0 = blockIdx.x * BM, j0 = blockIdx.y * BN, ks = blockIdx.z;
  const int kbeg = ks * kslab, kend = min(K, kbeg + kslab);
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  double acc[4][4] = {};
  for (int k0 = kbeg; k0 < kend; k0 += BK) {
    for (int e = threadIdx.x; e < BM * BK; e += NT) {
      int r = e / BK, c = e % BK;
      int k = k0 + c;
      double av = 0.0, bv = 0.0;
      if (k < kend) {
        if (i0 + r < M) {
          av = A[(size_t)(i0 + r) * lda + k];
          if (w) av *= w[k >> 1];
        }
        if (j0 + r < N) bv = B[(size_t)(j0 + r) * ldb + k];
      }
      As[c][r] = av;
      Bs[c][r] = bv;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      double a[4], b[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        a[q] = As[kk][ty + 16 * q];
        b[q] = Bs[kk][tx + 16 * q];
      }
#pragma unroll
      for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int r = 0; r < 4; ++r) acc[q][r] += a[q] * b[r];
    }
    __syncthreads();
  }
  double* P = part + (size_t)ks * M * N;
#pragma unroll
  for (int q = 0; q < 4; ++q)
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      int i = i0 + ty + 16 * q, j = j0 + tx + 16 * r;
      if (i < M && j < N) P[(size_t)j * M + i] = acc[q][r];
    }
}

// C = alpha sum_k part[k] + beta C; sym (M == N): the sum averaged with its
// transpose, taken in the same order for (i,j) and (j,i) so the result is exactly
// symmetric.  With G = 8 the partials of an element are added in eight groups by
// eight threads, then the groups in order: one thread per element over ~150
// partials is bound by the latency of its loads (two passes over them, groups
// first, took 18 us for 148 partials of 128 x 128, this one 5).
template <int G>
__global__ void __launch_bounds__(256)
k_splitk_reduce(const double* __restrict__ part, int nsplit, int M, int N, double alpha,
                double beta, double* __restrict__ C, int ldc, int sym,
                const double* __restrict__ diag) {
  constexpr int E = 256 / G;  // elements per block
  __shared__ double sh[2][G][E];
  const int tx = threadIdx.x % E, g = threadIdx.x / E;
  const long long e = (long long)blockIdx.x * E + tx;
  const bool in = e < (long long)M * N;
  const int j = in ? (int)(e / M) : 0, i = in ? (int)(e - (long long)j * M) : 0;
  const bool onlyd = diag && i == j;  // the diagonal summed in FP64 elsewhere
  double s1 = 0.0, s2 = 0.0;
  if (in && !onlyd) {
    const size_t mn = (size_t)M * N;
    const int k0 = nsplit * g / G, k1 = nsplit * (g + 1) / G;
    const size_t e1 = sym ? (size_t)min(i, j) * M + max(i, j) : (size_t)e;
    const size_t e2 = (size_t)max(i, j) * M + min(i, j);
#pragma unroll 8
    for (int k = k0; k < k1; ++k) s1 += part[(size_t)k * mn + e1];
    if (sym)
#pragma unroll 8
      for (int k = k0; k < k1; ++k) s2 += part[(size_t)k * mn + e2];
  }
  if (G > 1) {
    sh[0][g][tx] = s1;
    sh[1][g][tx] = s2;
    __syncthreads();
    if (g) return;
#pragma unroll
    for (int q = 1; q < G; ++q) {
      s1 += sh[0][q][tx];
      s2 += sh[1][q][tx];
    }
  }
  if (!in) return;
  const double s = onlyd ? diag[i] : (sym ? 0.5 * (s1 + s2) : s1);
  double* c = C + (size_t)j * ldc + i;
  *c = alpha * s + (beta == 0.0 ? 0.0 : beta * (*c));
}

template <typename... A>
static void splitk_reduce(cudaStream_t st, const double* part, int nsplit, int M, int N, A... a) {
  const long long mn = (long long)M * N;
  if (nsplit > 16)
    k_splitk_reduce<8><<<(unsigned)((mn + 31) / 32), 256, 0, st>>>(part, nsplit, M, N, a...);
  else
    k_splitk_reduce<1><<<(unsigned)((mn + 255) / 256), 256, 0, st>>>(part, nsplit, M, N, a...);
}

// column-major C = alpha op(A) op(B) + beta C (reference DGEMM semantics) on the
// FP64 tensor units: a 32 x 32 tile per block, its eight warps sharing out each
// 128-long K chunk (16 each) so that the S x S products of the step, 16 blocks at
// 128 states, still keep eight warps per tile busy; the warps' tiles are added in
// order.  An operand is kept as it lies: [x][k] where k is contiguous (op(A) = A^T,
// op(B) = B), [k][x] otherwise, both with strides that spread the fragment
// reads over the banks.  Sizes 128, 512, 2048: 27, 94, 1217 us on scalar FMAs in 64 x 64 tiles -> 14, 25, 1027.
constexpr int DT = 32, DK = 128, DLK = DK + 8, DLX = DT + 2;
constexpr int DOPND = DT * DLK;  // = DK * DLX doubles
static_assert(DOPND == DK * DLX, "one operand size for both layouts");

template <bool KC>  // k contiguous
__device__ __forceinline__ void dg_load(const double* __restrict__ X, int ldx, int x0, int nx,
                                        int k0, int k, double* s) {
  for (int q = threadIdx.x; q < DT * DK; q += NT) {
    const int x = KC ? q / DK : q % DT, l = KC ? q % DK : q / DT;
    const bool ok = x0 + x < nx && k0 + l < k;
    const size_t off = KC ? (size_t)(x0 + x) * ldx + k0 + l : (size_t)(k0 + l) * ldx + x0 + x;
    tc::cp8(s + (KC ? x * DLK + l : l * DLX + x), X + (ok ? off : 0), ok ? 8 : 0);
  }
}
template <bool KC>
__device__ __forceinline__ double2 dg_frag(const double* s, int x, int l) {
  if (KC) return *reinterpret_cast<const double2*>(s + x * DLK + l);
  return make_double2(s[l * DLX + x], s[(l + 1) * DLX + x]);
}

template <bool TA, bool TB>
__global__ void __launch_bounds__(NT)
k_dgemm(int m, int n, int k, double alpha, const double* __restrict__ A, int lda,
        const double* __restrict__ B, int ldb, double beta, double* __restrict__ C, int ldc) {
  extern __shared__ __align__(16) double sm[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int tm = (m + DT - 1) / DT, nc = (k + DK - 1) / DK;
  const int i0 = (int)(blockIdx.x % tm) * DT, j0 = (int)(blockIdx.x / tm) * DT;
  double acc[4][4][2];
  dm::zero(acc);
  auto load = [&](int st, int c) {
    double* s = sm + st * 2 * DOPND;
    dg_load<TA>(A, lda, i0, m, c * DK, k, s);
    dg_load<!TB>(B, ldb, j0, n, c * DK, k, s + DOPND);
    tc::cp_commit();
  };
  if (nc > 0) load(0, 0);
  for (int c = 0; c < nc; ++c) {
    tc::cp_wait<0>();
    __syncthreads();
    if (c + 1 < nc) load((c + 1) & 1, c + 1);
    if (c * DK + warp * 16 >= k) continue;
    const double* s = sm + (c & 1) * 2 * DOPND;
#pragma unroll
    for (int kk = 0; kk < 2; ++kk) {
      const int l = warp * 16 + kk * 8 + 2 * t;
      double2 a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        a[i] = dg_frag<TA>(s, i * 8 + g, l);
        b[i] = dg_frag<!TB>(s + DOPND, i * 8 + g, l);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) dm::mma884(acc[i][j], a[i].x, b[j].x);
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) dm::mma884(acc[i][j], a[i].y, b[j].y);
    }
  }
  __syncthreads();  // the stages become the eight partial tiles, column-major
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e)
        sm[warp * DT * DT + (j * 8 + 2 * t + e) * DT + i * 8 + g] = acc[i][j][e];
  __syncthreads();
#pragma unroll
  for (int q = 0; q < DT * DT / NT; ++q) {
    const int e = tid + NT * q, i = i0 + e % DT, j = j0 + e / DT;
    if (i >= m || j >= n) continue;
    double v = 0.0;
#pragma unroll
    for (int w = 0; w < NT / 32; ++w) v += sm[w * DT * DT + e];
    double* o = C + (size_t)j * ldc + i;
    *o = alpha * v + (beta == 0.0 ? 0.0 : beta * (*o));
  }
}

// ---------------------------------------------------------------------------
// FP64 products on the FP64 tensor units (dmma.cuh).  A block holds WM x WN
// warps of 32 x 32 outputs; 32-real chunks of both operands come in by cp.async
// into two stages, one barrier per chunk.  Blocks of 4 x 4 warps take one SM
// each (164 KB); sizes that fit 64 rows run blocks of 2 x 2 (overlap) or 2 x 4
// and 1 x 4 warps (back-multiply), whose padding costs less.  128 states, 65,736
// points: lambda and S 281 us each on FP64 FMAs (15 TFLOP/s) -> 130 us (33
// TFLOP/s; S's lower half is not formed), a back-multiply 293 -> 195 us (22
// TFLOP/s: four chunks per tile, whose epilogue is not overlapped).

template <int WM, int WN>
struct OvlCfg {
  static constexpr int TM = 32 * WM, TN = 32 * WN, THREADS = 32 * WM * WN;
  static constexpr size_t SMEM = sizeof(double) * 2 * dm::LDK * (TM + TN);
};

// C_part[ks] = A B^T over the split's chunks of 32 reals (A, B row-major
// [rows][K], K even; w per complex point scales A).  sym (A == B, M == N): only
// the tiles and, in a diagonal tile, the warp blocks on and above the diagonal
// are formed and written to both halves; a diagonal tile has one operand.
template <int WM, int WN>
__global__ void __launch_bounds__(OvlCfg<WM, WN>::THREADS)
k_overlap(const double* __restrict__ A, const double* __restrict__ B,
          const double* __restrict__ w, int M, int N, int K, int sym, int tn,
          double* __restrict__ part) {
  using C = OvlCfg<WM, WN>;
  extern __shared__ __align__(16) double sm[];
  double* As = sm;
  double* Bs = sm + 2 * C::TM * dm::LDK;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int ti, tj;
  if (sym) {  // blockIdx.x counts the tiles ti <= tj by rows
    int r = blockIdx.x;
    ti = 0;
    while (r >= tn - ti) {
      r -= tn - ti;
      ++ti;
    }
    tj = ti + r;
  } else {
    ti = blockIdx.x / tn;
    tj = blockIdx.x % tn;
  }
  const int i0 = ti * C::TM, j0 = tj * C::TN;
  const bool diag = sym && ti == tj;
  int wm = warp / WN, wn = warp % WN;
  bool work = true;
  if (diag) {  // warps 0, 1, .. take the blocks wm <= wn: spread over the schedulers
    int r = warp;
    wm = 0;
    while (wm < WM && r >= WN - wm) {
      r -= WN - wm;
      ++wm;
    }
    work = wm < WM;
    wn = wm + r;
    if (!work) wm = wn = 0;
  }
  const int nchunk = (K + 31) / 32;
  const int c0 = (int)((long long)nchunk * blockIdx.y / gridDim.y);
  const int c1 = (int)((long long)nchunk * (blockIdx.y + 1) / gridDim.y);
  double acc[4][4][2];
  dm::zero(acc);
  auto load = [&](int st, int c) {
    for (int q = tid; q < C::TM * 16; q += C::THREADS) {
      const int row = q >> 4, k = c * 32 + 2 * (q & 15);
      const bool ok = i0 + row < M && k < K;
      tc::cp16(As + (st * C::TM + row) * dm::LDK + 2 * (q & 15),
               A + (ok ? (size_t)(i0 + row) * K + k : 0), ok ? 16 : 0);
    }
    if (!diag)
      for (int q = tid; q < C::TN * 16; q += C::THREADS) {
        const int row = q >> 4, k = c * 32 + 2 * (q & 15);
        const bool ok = j0 + row < N && k < K;
        tc::cp16(Bs + (st * C::TN + row) * dm::LDK + 2 * (q & 15),
                 B + (ok ? (size_t)(j0 + row) * K + k : 0), ok ? 16 : 0);
      }
    tc::cp_commit();
  };
  if (c0 < c1) load(0, c0);
  const int g = lane >> 2, t = lane & 3;
  for (int c = c0; c < c1; ++c) {
    const int st = (c - c0) & 1;
    double wv[4];  // the weight of this thread's point in each group of 8 reals
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      const int p = c * 16 + kk * 4 + t;
      wv[kk] = (w && 2 * p < K) ? w[p] : 1.0;
    }
    tc::cp_wait<0>();
    __syncthreads();
    if (c + 1 < c1) load(st ^ 1, c + 1);
    if (!work) continue;
    const double* a0 = As + (st * C::TM + wm * 32 + g) * dm::LDK + 2 * t;
    const double* b0 =
        (diag ? As + (st * C::TM + wn * 32 + g) * dm::LDK : Bs + (st * C::TN + wn * 32 + g) * dm::LDK) +
        2 * t;
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      double2 a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        a[i] = *reinterpret_cast<const double2*>(a0 + i * 8 * dm::LDK + kk * 8);
        b[i] = *reinterpret_cast<const double2*>(b0 + i * 8 * dm::LDK + kk * 8);
        a[i].x *= wv[kk];
        a[i].y *= wv[kk];
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) dm::mma884(acc[i][j], a[i].x, b[j].x);
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) dm::mma884(acc[i][j], a[i].y, b[j].y);
    }
  }
  if (!work) return;
  double* P = part + (size_t)blockIdx.y * M * N;
  const bool both = sym && (!diag || wm != wn);
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int r = i0 + wm * 32 + i * 8 + g, cc = j0 + wn * 32 + j * 8 + 2 * t + e;
        if (r < M && cc < N) {
          P[(size_t)cc * M + r] = acc[i][j][e];
          if (both) P[(size_t)r * M + cc] = acc[i][j][e];
        }
      }
}

template <int WM>
struct BmCfg {
  static constexpr int TM = 32 * WM, THREADS = 128 * WM;
  static constexpr size_t SMEM = sizeof(double) * 2 * (dm::LDK * TM + 32 * dm::LDN);
};

// out[i][p] = alpha w[p/2] sum_j Mcm[j + i ldm] in[j][p] + beta out[i][p] on
// tiles of 32 WM rows x 128 reals; blocks walk the tiles (the row tiles of a
// point tile one after the other: in read once from HBM) with the next chunk's
// copies, the next tile's first one included, in flight behind the products.
// vec: out rows are 16-byte aligned.
template <int WM>
__global__ void __launch_bounds__(BmCfg<WM>::THREADS)
k_backmul(const double* __restrict__ Mcm, int ldm, const double* __restrict__ in, int ldi,
          double* __restrict__ out, int ldo, int nout, int nin, int K, double alpha, double beta,
          const double* __restrict__ w, int vec) {
  using C = BmCfg<WM>;
  extern __shared__ __align__(16) double sm[];
  double* As = sm;                      // [2][TM][LDK]: M rows i, j contiguous
  double* Bs = sm + 2 * C::TM * dm::LDK;  // [2][32][LDN]: in rows j
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = warp >> 2, wn = warp & 3;
  const int ni = (nout + C::TM - 1) / C::TM, nj = (nin + 31) / 32;
  const int ntile = ((K + 127) / 128) * ni;
  const int mine = (int)blockIdx.x < ntile ? (ntile - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
  const int total = mine * nj;
  double acc[4][4][2];
  dm::zero(acc);
  auto load = [&](int st, int it) {
    const int tile = (int)blockIdx.x + (it / nj) * (int)gridDim.x, j0 = (it % nj) * 32;
    const int p0 = (tile / ni) * 128, i0 = (tile % ni) * C::TM;
    for (int q = tid; q < C::TM * 32; q += C::THREADS) {
      const int row = q >> 5, j = q & 31;
      const bool ok = i0 + row < nout && j0 + j < nin;
      tc::cp8(As + (st * C::TM + row) * dm::LDK + j,
              Mcm + (ok ? (size_t)(i0 + row) * ldm + j0 + j : 0), ok ? 8 : 0);
    }
    for (int q = tid; q < 32 * 64; q += C::THREADS) {
      const int row = q >> 6, p = p0 + 2 * (q & 63);
      const bool ok = j0 + row < nin && p < K;  // K and p even: the pair is inside
      tc::cp16(Bs + (st * 32 + row) * dm::LDN + 2 * (q & 63),
               in + (ok ? (size_t)(j0 + row) * ldi + p : 0), ok ? 16 : 0);
    }
    tc::cp_commit();
  };
  if (total > 0) load(0, 0);
  for (int it = 0; it < total; ++it) {
    const int st = it & 1;
    tc::cp_wait<0>();
    __syncthreads();
    if (it + 1 < total) load(st ^ 1, it + 1);
    dm::chunk_kn(acc, As + (st * C::TM + wm * 32) * dm::LDK, Bs + st * 32 * dm::LDN + wn * 32,
                 lane);
    if (it % nj != nj - 1) continue;
    const int tile = (int)blockIdx.x + (it / nj) * (int)gridDim.x;
    const int i0 = (tile % ni) * C::TM + wm * 32 + (lane >> 2);
    const int q0 = (tile / ni) * 128 + wn * 32 + 2 * (lane & 3);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int p = q0 + 8 * j;
      const double a = (w && p < K) ? alpha * w[p >> 1] : alpha;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = i0 + 8 * i;
        double2 v = make_double2(a * acc[i][j][0], a * acc[i][j][1]);
        acc[i][j][0] = acc[i][j][1] = 0.0;
        if (r >= nout || p >= K) continue;
        double* o = out + (size_t)r * ldo + p;
        if (vec) {
          if (beta != 0.0) {
            const double2 u = *reinterpret_cast<const double2*>(o);
            v.x += beta * u.x;
            v.y += beta * u.y;
          }
          *reinterpret_cast<double2*>(o) = v;
        } else {
          o[0] = v.x + (beta == 0.0 ? 0.0 : beta * o[0]);
          o[1] = v.y + (beta == 0.0 ? 0.0 : beta * o[1]);
        }
      }
    }
  }
}

}  // namespace pcalc

// ---------------------------------------------------------------------------
// host side

int pc_part_reserve(cpstep_ctx* c, size_t need) {
  if (need > c->pc_part_elems) {
    graph_drop(c);  // a captured step may hold the old buffer
    cudaFree(c->d_pc_part);
    c->d_pc_part = nullptr;
    c->pc_part_elems = 0;
    CPSTEP_CUDA_TRY(cudaMalloc(&c->d_pc_part, need * sizeof(double)));
    c->pc_part_elems = need;
  }
  return CPSTEP_OK;
}

int lv_reserve(cpstep_ctx* c, size_t bytes) {
  if (bytes > c->lv_bytes) {
    graph_drop(c);  // a captured step may hold the old buffer
    cudaFree(c->d_lv);
    c->d_lv = nullptr;
    c->lv_bytes = 0;
    CPSTEP_CUDA_TRY(cudaMalloc(&c->d_lv, bytes));
    c->lv_bytes = bytes;
  }
  return CPSTEP_OK;
}

int split_reserve(cpstep_ctx* c, size_t bytes) {
  if (bytes > c->split_bytes) {
    graph_drop(c);  // a captured step may hold the old buffer
    cudaFree(c->d_split);
    c->d_split = nullptr;
    c->split_bytes = 0;
    CPSTEP_CUDA_TRY(cudaMalloc(&c->d_split, bytes));
    c->split_bytes = bytes;
  }
  return CPSTEP_OK;
}

size_t pc_part_need(int nsplit, size_t mn) { return (size_t)nsplit * mn; }

int pc_splitk_reduce_launch(cpstep_ctx* c, int nsplit, int M, int N, double alpha, double beta,
                            double* C, int ldc, int sym, const double* diag) {
  pcalc::splitk_reduce(c->stream, c->d_pc_part, nsplit, M, N, alpha, beta, C, ldc, sym, diag);
  CPSTEP_LAUNCH_CHECK();
  return CPSTEP_OK;
}

template <typename F>
static int dyn_smem(F kernel, size_t bytes) {
  CPSTEP_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)bytes));
  return CPSTEP_OK;
}

template <int WM, int WN>
static int overlap64(cpstep_ctx* c, const double* a, const double* b, int M, int N, int K,
                     const double* w, double alpha, double beta, double* C, int ldc, bool sym,
                     int per_sm) {
  using Cfg = pcalc::OvlCfg<WM, WN>;
  const int tm = cdiv(M, Cfg::TM), tn = cdiv(N, Cfg::TN);
  const int tiles = sym ? tm * (tm + 1) / 2 : tm * tn;
  const int nsplit = std::max(1, std::min(cdiv(K, 32), c->tune.pc_split * per_sm * c->num_sms / tiles));
  if (int rc = pc_part_reserve(c, pc_part_need(nsplit, (size_t)M * N))) return rc;
  if (int rc = dyn_smem(pcalc::k_overlap<WM, WN>, Cfg::SMEM)) return rc;
  pcalc::k_overlap<WM, WN><<<dim3(tiles, nsplit), Cfg::THREADS, Cfg::SMEM, c->stream>>>(
      a, b, w, M, N, K, sym ? 1 : 0, tn, c->d_pc_part);
  CPSTEP_LAUNCH_CHECK();
  return pc_splitk_reduce_launch(c, nsplit, M, N, alpha, beta, C, ldc, 0);
}

int pc_overlap_launch(cpstep_ctx* c, const double* a, const double* b, int M, int N, int K,
                      const double* w, double alpha, double beta, double* C, int ldc) {
  using namespace pcalc;
  bool used = false;
  if (int rc = pc_overlap_tc_launch(c, a, b, M, N, K, w, alpha, beta, C, ldc, &used)) return rc;
  if (used) return CPSTEP_OK;
  // both sides within 64 rows: 2 x 2 warps, two blocks per SM
  const bool sym = a == b && M == N;
  return (M <= 64 && N <= 64)
             ? overlap64<2, 2>(c, a, b, M, N, K, w, alpha, beta, C, ldc, sym, 2)
             : overlap64<4, 4>(c, a, b, M, N, K, w, alpha, beta, C, ldc, sym, 1);
}

template <int WM>
static int backmul64(cpstep_ctx* c, const double* Mcm, int ldm, const double* in, int ldi,
                     double* out, int ldo, int nout, int nin, int K, double alpha, double beta,
                     const double* w) {
  using Cfg = pcalc::BmCfg<WM>;
  if (int rc = dyn_smem(pcalc::k_backmul<WM>, Cfg::SMEM)) return rc;
  const int tiles = cdiv(K, 128) * cdiv(nout, Cfg::TM);
  const int per_sm = (int)std::max<size_t>(1, 227 * 1024 / (Cfg::SMEM + 1024));
  const int vec = (reinterpret_cast<uintptr_t>(out) & 15) == 0 && (ldo & 1) == 0;
  pcalc::k_backmul<WM><<<std::min(tiles, per_sm * c->num_sms), Cfg::THREADS, Cfg::SMEM, c->stream>>>(
      Mcm, ldm, in, ldi, out, ldo, nout, nin, K, alpha, beta, w, vec);
  CPSTEP_LAUNCH_CHECK();
  return CPSTEP_OK;
}

int pc_backmul_w_launch(cpstep_ctx* c, const double* Mcm, int ldm, const double* in, int ldi,
                        double* out, int ldo, int nout, int nin, int K, double alpha, double beta,
                        const double* w) {
  bool used = false;
  if (int rc = pc_backmul_tc_launch(c, Mcm, ldm, in, ldi, out, ldo, nout, nin, K, alpha, beta, w,
                                    &used))
    return rc;
  if (used) return CPSTEP_OK;
  // the fewest rows per tile that hold all outputs: padded rows cost as much as real ones
  if (nout <= 32) return backmul64<1>(c, Mcm, ldm, in, ldi, out, ldo, nout, nin, K, alpha, beta, w);
  if (nout <= 64) return backmul64<2>(c, Mcm, ldm, in, ldi, out, ldo, nout, nin, K, alpha, beta, w);
  return backmul64<4>(c, Mcm, ldm, in, ldi, out, ldo, nout, nin, K, alpha, beta, w);
}

int pc_backmul_launch(cpstep_ctx* c, const double* Mcm, int ldm, const double* in, int ldi,
                      double* out, int ldo, int nout, int nin, int K, double alpha, double beta) {
  return pc_backmul_w_launch(c, Mcm, ldm, in, ldi, out, ldo, nout, nin, K, alpha, beta, nullptr);
}

int dgemm_launch(cudaStream_t s, int ta, int tb, int m, int n, int k, double alpha,
                 const double* A, int lda, const double* B, int ldb, double beta, double* C,
                 int ldc) {
  using namespace pcalc;
  auto kern = ta ? (tb ? k_dgemm<true, true> : k_dgemm<true, false>)
                 : (tb ? k_dgemm<false, true> : k_dgemm<false, false>);
  const size_t smem = sizeof(double) * 2 * DOPND * (k > DK ? 2 : 1);
  if (int rc = dyn_smem(kern, sizeof(double) * 4 * DOPND)) return rc;
  const long long tiles = (long long)cdiv(m, DT) * cdiv(n, DT);
  kern<<<(unsigned)tiles, NT, smem, s>>>(m, n, k, alpha, A, lda, B, ldb, beta, C,
                                                        ldc);
  CPSTEP_LAUNCH_CHECK();
  return CPSTEP_OK;
}

// ---------------------------------------------------------------------------
// Allocation-free variant of the overlap product (cpstep_pc_overlap_noalloc).
//
// For callers that cannot allocate device memory: the split-K partial tiles go
// to a fixed array compiled into the library instead of context scratch.  The
// array exists on every GPU that loads the library, for the life of the
// process.  In host code `g_noalloc_part` names a host-side shadow, not device
// memory, so the kernels get the device address looked up below.

#define CPSTEP_NOALLOC_PART_DOUBLES (1 << 20)  // 8 MiB of partial tiles
static __device__ __align__(256) double g_noalloc_part[CPSTEP_NOALLOC_PART_DOUBLES];

namespace {
std::mutex g_noalloc_mu;
double* g_noalloc_addr[64] = {};            // device address of the array, per device
unsigned long long g_noalloc_ctx[64] = {};  // unique ID of the context it was looked up in
int g_noalloc_sms[64] = {};

// Unique ID of the calling thread's current context (cuCtxGetId: never reused
// within a process), 0 when none is current.  The driver entry points come
// through the runtime, so the library does not link the driver library.
typedef CUresult (*PfnCtxGetCurrent)(CUcontext*);
typedef CUresult (*PfnCtxGetId)(CUcontext, unsigned long long*);
unsigned long long current_ctx_id() {
  static PfnCtxGetCurrent get_cur = nullptr;
  static PfnCtxGetId get_id = nullptr;
  if (!get_cur || !get_id) {
    cudaDriverEntryPointQueryResult q1, q2;
    if (cudaGetDriverEntryPoint("cuCtxGetCurrent", reinterpret_cast<void**>(&get_cur),
                                cudaEnableDefault, &q1) != cudaSuccess ||
        cudaGetDriverEntryPoint("cuCtxGetId", reinterpret_cast<void**>(&get_id),
                                cudaEnableDefault, &q2) != cudaSuccess ||
        q1 != cudaDriverEntryPointSuccess || q2 != cudaDriverEntryPointSuccess) {
      cudaGetLastError();
      get_cur = nullptr;
      get_id = nullptr;
      return 0;
    }
  }
  CUcontext ctx = nullptr;
  unsigned long long id = 0;
  if (get_cur(&ctx) != CUDA_SUCCESS || !ctx || get_id(ctx, &id) != CUDA_SUCCESS) return 0;
  return id;
}
}  // namespace

extern "C" int cpstep_pc_overlap_noalloc(const double* d_a, const double* d_b, int na, int nb,
                                         int npts, const double* d_w, double alpha,
                                         double beta, double* d_c, int ldc, void* stream) {
  using namespace pcalc;
  if (!d_a || !d_b || !d_c || na <= 0 || nb <= 0 || npts <= 0 || ldc < na) {
    cpstep_set_error("pc_overlap_noalloc: bad argument");
    return CPSTEP_ERR_ARG;
  }
  if ((size_t)na * nb > CPSTEP_NOALLOC_PART_DOUBLES) {
    cpstep_set_error("pc_overlap_noalloc: na*nb = %zu exceeds the fixed scratch of %d doubles "
                     "(at most %d x %d); use cpstep_pc_overlap",
                     (size_t)na * nb, CPSTEP_NOALLOC_PART_DOUBLES, 1024, 1024);
    return CPSTEP_ERR_ARG;
  }
  int dev = 0;
  CPSTEP_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) {
    cpstep_set_error("pc_overlap_noalloc: device index %d out of range", dev);
    return CPSTEP_ERR_ARG;
  }
  double* part = nullptr;
  int nsm = 0;
  {
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    const unsigned long long id = current_ctx_id();
    if (!g_noalloc_addr[dev] || id == 0 || id != g_noalloc_ctx[dev]) {
      // once per device and context, with that device current: the address
      // is the array's copy in the current context (a reset of the device's
      // primary context, cudaDeviceReset, makes a new one)
      void* addr = nullptr;
      CPSTEP_CUDA_TRY(cudaGetSymbolAddress(&addr, g_noalloc_part));
      int sms = 0;
      CPSTEP_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
      g_noalloc_addr[dev] = static_cast<double*>(addr);
      g_noalloc_ctx[dev] = current_ctx_id();
      g_noalloc_sms[dev] = sms > 0 ? sms : 148;
    }
    part = g_noalloc_addr[dev];
    nsm = g_noalloc_sms[dev];
  }
  const int M = na, N = nb, K = 2 * npts;
  const int tm = cdiv(M, BM), tn = cdiv(N, BN);
  int want = std::max(1, (2 * nsm) / (tm * tn));
  const int fit = (int)std::max<size_t>(1, CPSTEP_NOALLOC_PART_DOUBLES / ((size_t)M * N));
  want = std::min(want, fit);
  int kslab = cdiv(cdiv(K, want), BK) * BK;
  int nsplit = cdiv(K, kslab);
  while ((size_t)nsplit * M * N > CPSTEP_NOALLOC_PART_DOUBLES) {  // rounding of kslab
    kslab += BK;
    nsplit = cdiv(K, kslab);
  }
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  // every partial the reduction reads is written by this call: nothing to clear
  k_overlap_part<<<dim3(tm, tn, nsplit), NT, 0, s>>>(d_a, K, d_b, K, d_w, M, N, K, kslab, part);
  CPSTEP_LAUNCH_CHECK();
  splitk_reduce(s, part, nsplit, M, N, alpha, beta, d_c, ldc, 0, (const double*)nullptr);
  CPSTEP_LAUNCH_CHECK();
  return CPSTEP_OK;
}
