// Ortho: T = (S/2)^(-1/2) by the reference's coupled Schulz iteration, as one
// cooperative kernel (grid-wide barriers between the GEMM phases, so the whole
// iteration is a single launch and the host never synchronises in between).
//
//   CPORTHOG::get_iter_Tmat  src_piny_physics_v1.0/abinito_physics/cp_orthog/cp_lowdin.C:180-265
//   Ortho::start_calc / do_iteration / step_2 / step_3 / tolerance_check /
//   collect_error            src_charm_driver/orthog_ctrl/ortho.C:153-269, :862-985, :109-145
//   A = I, B = S/2;  C = 3I - A B^T;  B <- B C^T / 2;  A <- C A^T / 2;
//   stop when rms(A_old - A_new) <= tol (1e-15) or after max_iter (10) iterations;
//   the reference aborts on failure (cp_lowdin.C:243-250), here a status code.
//
// Mixed precision: the same FP64 iteration to a looser tolerance, then a
// correction against S restores T^T (S/2) T = I to rounding.  (FP32 tiles were
// no faster: up to a few hundred states the barriers and the latency of one
// tile bound the iteration, beyond that the FP64 tensor units.)
// Optional spectral scaling (mixed path only): B = S/sigma with sigma an upper
// bound of the spectrum (Gershgorin), T = A (sigma/2)^(-1/2); it extends the
// convergence region beyond the reference's eig(S/2) < 2 condition.
//
// Every loop in the kernel has a fixed iteration bound; the only waits are the
// cooperative-groups grid barriers of a cooperative launch.
#include <cooperative_groups.h>
#include <algorithm>
#include <cmath>
#include "ctx.cuh"
#include "dmma.cuh"

namespace cg = cooperative_groups;

namespace orth {

constexpr int TS = 32;          // output tile
constexpr int NT = 256;         // 8 warps: each takes a sixteenth of a 128-long K chunk twice
constexpr int KC = 128;         // K chunk
constexpr int LDO = KC + 8;     // row stride: 64 mod 128 bytes (dmma.cuh, LDK)
constexpr int STAGE = 2 * TS * LDO;  // doubles of one stage: 32 rows of X and of Y

// sum_k X[i][k] Y[j][k] for the 32 x 32 tile (i0, j0) of n x n row-major matrices
// on the FP64 tensor units.  The eight warps split K (16 of every 128), so that
// a small n keeps all of them busy, and add their tiles through shared memory in
// warp order; out(i, j, sum) is called once per element inside the matrices.
// With n <= 128 the tile's whole operands are one round of copies.
template <typename Out>
__device__ __forceinline__ void tile_abt(const double* __restrict__ X,
                                         const double* __restrict__ Y, int n, int vec, int i0,
                                         int j0, double* sm, Out out) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int nc = (n + KC - 1) / KC;
  auto load = [&](int st, int c) {
    double* xs = sm + st * STAGE;
    double* ys = xs + TS * LDO;
    if (vec) {
      for (int q = tid; q < TS * (KC / 2); q += NT) {
        const int r = q / (KC / 2), k = 2 * (q % (KC / 2)), kk = c * KC + k;
        const bool kx = kk < n, ox = kx && i0 + r < n, oy = kx && j0 + r < n;
        tc::cp16(xs + r * LDO + k, X + (ox ? (size_t)(i0 + r) * n + kk : 0), ox ? 16 : 0);
        tc::cp16(ys + r * LDO + k, Y + (oy ? (size_t)(j0 + r) * n + kk : 0), oy ? 16 : 0);
      }
    } else {
      for (int q = tid; q < TS * KC; q += NT) {
        const int r = q / KC, k = q % KC, kk = c * KC + k;
        const bool kx = kk < n, ox = kx && i0 + r < n, oy = kx && j0 + r < n;
        tc::cp8(xs + r * LDO + k, X + (ox ? (size_t)(i0 + r) * n + kk : 0), ox ? 8 : 0);
        tc::cp8(ys + r * LDO + k, Y + (oy ? (size_t)(j0 + r) * n + kk : 0), oy ? 8 : 0);
      }
    }
    tc::cp_commit();
  };
  double acc[4][4][2];
  dm::zero(acc);
  load(0, 0);
  for (int c = 0; c < nc; ++c) {
    tc::cp_wait<0>();
    __syncthreads();
    if (c + 1 < nc) load((c + 1) & 1, c + 1);
    if (c * KC + warp * 16 >= n) continue;  // a K slice past the end is zero
    const double* xs = sm + (c & 1) * STAGE + g * LDO + warp * 16 + 2 * t;
    const double* ys = xs + TS * LDO;
#pragma unroll
    for (int kk = 0; kk < 2; ++kk) {
      double2 a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        a[i] = *reinterpret_cast<const double2*>(xs + i * 8 * LDO + kk * 8);
        b[i] = *reinterpret_cast<const double2*>(ys + i * 8 * LDO + kk * 8);
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
  __syncthreads();  // the stages become the eight partial tiles
  const int nw = n <= 16 * (NT / 32) ? (n + 15) / 16 : NT / 32;  // warps with a K slice
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
      *reinterpret_cast<double2*>(sm + warp * TS * TS + (i * 8 + g) * TS + j * 8 + 2 * t) =
          make_double2(acc[i][j][0], acc[i][j][1]);
  __syncthreads();
#pragma unroll
  for (int q = 0; q < TS * TS / NT; ++q) {
    const int e = tid + NT * q, i = i0 + e / TS, j = j0 + e % TS;
    double v = 0.0;
    for (int w = 0; w < nw; ++w) v += sm[w * TS * TS + e];
    if (i < n && j < n) out(i, j, v);
  }
  __syncthreads();  // before the next tile's copies
}

struct Work {
  int n, max_iter, vec;
  double tol;
  const double* S;  // [n][n] (symmetric)
  double *A, *B, *C, *A2, *B2;
  double *X, *Y, *E, *P;      // correction buffers (mixed)
  double* partial;            // [2][gridDim.x]
  double* T;                  // output [n][n]
  int* status;                // [0] iterations, [1] converged flag
  double* rms;                // final rms
  double sigma;               // spectral scale (2 = reference)
  int newton;                 // correction after the iteration (the mixed path's rule)
};

// One cooperative launch.  An iteration is two phases of tiles with a grid
// barrier after each; the update's norm is taken from the tiles of A as they
// are formed.  The first iteration, with A = I, needs B B^T alone.
__global__ void __launch_bounds__(NT) k_ortho(Work w) {
  cg::grid_group grid = cg::this_grid();
  extern __shared__ __align__(16) double sm[];
  __shared__ double red[32];
  __shared__ double rms_s;
  const int n = w.n, nn = n * n, nt = (n + TS - 1) / TS, ntiles = nt * nt;
  double *A = w.A, *B = w.B, *C = w.C, *A2 = w.A2, *B2 = w.B2;
  const size_t gtid = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const size_t gstride = (size_t)gridDim.x * blockDim.x;
  const double is = 1.0 / w.sigma;
  int it = 0;
  double tol_now = 1.0, prev = 1e300;
  while (tol_now > w.tol && it < w.max_iter) {
    ++it;
    double loc = 0.0;
    if (it == 1) {  // B = S / sigma, C = 3I - B:  B2 = B C^T / 2, A2 = C / 2
      for (int t = blockIdx.x; t < ntiles; t += gridDim.x)
        tile_abt(w.S, w.S, n, w.vec, t / nt * TS, t % nt * TS, sm, [&](int i, int j, double v) {
          const size_t e = (size_t)i * n + j;
          const double b = w.S[e] * is, a = 0.5 * ((i == j ? 3.0 : 0.0) - b);
          B2[e] = 0.5 * (3.0 * b - v * is * is);
          A2[e] = a;
          const double d = (i == j ? 1.0 : 0.0) - a;
          loc += d * d;
        });
    } else {
      // C = 3I - A B^T
      for (int t = blockIdx.x; t < ntiles; t += gridDim.x)
        tile_abt(A, B, n, w.vec, t / nt * TS, t % nt * TS, sm, [&](int i, int j, double v) {
          C[(size_t)i * n + j] = (i == j ? 3.0 : 0.0) - v;
        });
      grid.sync();
      // A2 = C A^T / 2 ;  B2 = B C^T / 2
      for (int t = blockIdx.x; t < 2 * ntiles; t += gridDim.x) {
        const int u = t < ntiles ? t : t - ntiles;
        if (t < ntiles)
          tile_abt(C, A, n, w.vec, u / nt * TS, u % nt * TS, sm, [&](int i, int j, double v) {
            const size_t e = (size_t)i * n + j;
            A2[e] = 0.5 * v;
            const double d = A[e] - 0.5 * v;
            loc += d * d;
          });
        else
          tile_abt(B, C, n, w.vec, u / nt * TS, u % nt * TS, sm,
                   [&](int i, int j, double v) { B2[(size_t)i * n + j] = 0.5 * v; });
      }
    }
    double* part = w.partial + (it & 1) * gridDim.x;  // the other half may still be read
    const double bs = block_sum(loc, red);
    if (threadIdx.x == 0) part[blockIdx.x] = bs;
    grid.sync();
    if (threadIdx.x < 32) {  // the same order in every block
      double s = 0.0;
      for (int b = threadIdx.x; b < (int)gridDim.x; b += 32) s += part[b];
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (threadIdx.x == 0) rms_s = sqrt(s / (double)nn);
    }
    __syncthreads();
    const double r = rms_s;
    __syncthreads();
    // the mixed path's rule: near the end a rise of the update means the coupled
    // iteration has reached its rounding; keep the previous iterate (the
    // correction polishes it).  The FP64 path keeps the reference's rule.
    if (w.newton && prev < 1e-3 && !(r < prev)) break;
    prev = r;
    tol_now = r;
    double* t1 = A; A = A2; A2 = t1;
    double* t2 = B; B = B2; B2 = t2;
  }
  // T = A (sigma/2)^(-1/2); before the correction it is symmetrised, so that
  // W = X (S/2) X below is the matrix T^T (S/2) T tests
  const double post = sqrt(2.0 / w.sigma);
  double* X = w.newton ? w.X : w.T;
  for (size_t e = gtid; e < (size_t)nn; e += gstride) {
    const int i = e / n, j = e % n;
    if (it == 0) X[e] = i == j ? post : 0.0;  // tol >= 1: no iteration, A = I
    else X[e] = w.newton ? 0.5 * (A[e] + A[(size_t)j * n + i]) * post : A[e] * post;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    w.status[0] = it;
    // mixed: converged once the iteration has stagnated below 1e-3 (the
    // correction takes it from there)
    w.status[1] = (tol_now <= w.tol || (w.newton && tol_now < 1e-3)) ? 1 : 0;
    *w.rms = tol_now;
  }
  if (!w.newton) return;
  // Correction: with X symmetric and W = X (S/2) X near I, T = X W^(-1/2),
  // W^(-1/2) = I - R/2 + 3R^2/8 + O(R^3), R = W - I, satisfies T^T (S/2) T = I
  // to FP64 rounding.
  auto phase = [&](const double* Xm, const double* Ym, auto out) {
    grid.sync();
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x)
      tile_abt(Xm, Ym, n, w.vec, t / nt * TS, t % nt * TS, sm, out);
  };
  phase(w.X, w.S, [&](int i, int j, double v) { w.Y[(size_t)i * n + j] = 0.5 * v; });
  phase(w.Y, w.X, [&](int i, int j, double v) { w.E[(size_t)i * n + j] = v - (i == j ? 1.0 : 0.0); });
  phase(w.E, w.E, [&](int i, int j, double v) {
    w.P[(size_t)i * n + j] = (i == j ? 1.0 : 0.0) - 0.5 * w.E[(size_t)i * n + j] + 0.375 * v;
  });
  phase(w.X, w.P, [&](int i, int j, double v) { w.T[(size_t)i * n + j] = v; });
}

// Up to 64 states: one block, every matrix in shared memory.  A warp forms a
// 16 x 16 tile with the whole K; the phases are as in k_ortho, with block
// barriers.
constexpr int SNT = 512, SN = 64, SLD = SN + 8;
__global__ void __launch_bounds__(SNT) k_ortho_small(Work w) {
  extern __shared__ __align__(16) double sm[];
  __shared__ double red[32];
  __shared__ double rms_s;
  const int n = w.n, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, t = lane & 3, nt = (n + 15) / 16;
  double *A = sm, *B = sm + SN * SLD, *C = sm + 2 * SN * SLD, *A2 = sm + 3 * SN * SLD,
         *B2 = sm + 4 * SN * SLD;
  // sum_k X[i][k] Y[j][k] (rows and columns past n are zero in every matrix)
  auto product = [&](const double* X, const double* Y, auto out) {
    if (warp < nt * nt) {
      const int i0 = warp / nt * 16, j0 = warp % nt * 16;
      double acc[2][2][2] = {};
      const double* xs = X + (i0 + g) * SLD + 2 * t;
      const double* ys = Y + (j0 + g) * SLD + 2 * t;
      for (int k = 0; k < n; k += 8) {
        double2 a[2], b[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          a[i] = *reinterpret_cast<const double2*>(xs + i * 8 * SLD + k);
          b[i] = *reinterpret_cast<const double2*>(ys + i * 8 * SLD + k);
        }
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int j = 0; j < 2; ++j) dm::mma884(acc[i][j], a[i].x, b[j].x);
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int j = 0; j < 2; ++j) dm::mma884(acc[i][j], a[i].y, b[j].y);
      }
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int r = i0 + 8 * i + g, c = j0 + 8 * j + 2 * t + e;
            if (r < n && c < n) out(r, c, acc[i][j][e]);
          }
    }
  };
  auto load_S = [&](double* D) {
    for (int e = tid; e < n * n; e += SNT) D[e / n * SLD + e % n] = w.S[e];
  };
  for (int e = tid; e < 5 * SN * SLD; e += SNT) sm[e] = 0.0;
  __syncthreads();
  load_S(B);
  __syncthreads();
  const double is = 1.0 / w.sigma;
  int it = 0;
  double tol_now = 1.0, prev = 1e300;
  while (tol_now > w.tol && it < w.max_iter) {
    ++it;
    double loc = 0.0;
    if (it == 1) {
      product(B, B, [&](int i, int j, double v) {
        const double b = B[i * SLD + j] * is, a = 0.5 * ((i == j ? 3.0 : 0.0) - b);
        B2[i * SLD + j] = 0.5 * (3.0 * b - v * is * is);
        A2[i * SLD + j] = a;
        const double d = (i == j ? 1.0 : 0.0) - a;
        loc += d * d;
      });
    } else {
      product(A, B, [&](int i, int j, double v) { C[i * SLD + j] = (i == j ? 3.0 : 0.0) - v; });
      __syncthreads();
      product(C, A, [&](int i, int j, double v) {
        A2[i * SLD + j] = 0.5 * v;
        const double d = A[i * SLD + j] - 0.5 * v;
        loc += d * d;
      });
      product(B, C, [&](int i, int j, double v) { B2[i * SLD + j] = 0.5 * v; });
    }
    const double bs = block_sum(loc, red);
    if (tid == 0) rms_s = sqrt(bs / (double)(n * n));
    __syncthreads();
    const double r = rms_s;
    if (w.newton && prev < 1e-3 && !(r < prev)) break;  // as in k_ortho
    prev = r;
    tol_now = r;
    double* t1 = A; A = A2; A2 = t1;
    double* t2 = B; B = B2; B2 = t2;
  }
  if (it == 0) {  // tol >= 1: no iteration, A = I
    if (tid < n) A[tid * SLD + tid] = 1.0;
    __syncthreads();
  }
  if (tid == 0) {
    w.status[0] = it;
    w.status[1] = (tol_now <= w.tol || (w.newton && tol_now < 1e-3)) ? 1 : 0;
    *w.rms = tol_now;
  }
  const double post = sqrt(2.0 / w.sigma);
  if (!w.newton) {
    for (int e = tid; e < n * n; e += SNT) w.T[e] = A[e / n * SLD + e % n] * post;
    return;
  }
  __syncthreads();
  double *X = C, *S = B2, *Y = A2, *E = A, *P = B;
  for (int e = tid; e < n * n; e += SNT) {
    const int i = e / n, j = e % n;
    X[i * SLD + j] = 0.5 * (A[i * SLD + j] + A[j * SLD + i]) * post;
  }
  load_S(S);
  __syncthreads();
  product(X, S, [&](int i, int j, double v) { Y[i * SLD + j] = 0.5 * v; });
  __syncthreads();
  product(Y, X, [&](int i, int j, double v) { E[i * SLD + j] = v - (i == j ? 1.0 : 0.0); });
  __syncthreads();
  product(E, E, [&](int i, int j, double v) {
    P[i * SLD + j] = (i == j ? 1.0 : 0.0) - 0.5 * E[i * SLD + j] + 0.375 * v;
  });
  __syncthreads();
  product(X, P, [&](int i, int j, double v) { w.T[i * n + j] = v; });
}

// Gershgorin bound of the spectrum: sigma = max_i sum_j |S_ij|
__global__ void k_gershgorin(const double* __restrict__ S, int n, double* __restrict__ out) {
  __shared__ double red[32];
  double m = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    double s = 0.0;
    for (int j = 0; j < n; ++j) s += fabs(S[(size_t)i * n + j]);
    m = fmax(m, s);
  }
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    double r = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) r = fmax(r, red[w]);
    *out = r;
  }
}

}  // namespace orth

// ---------------------------------------------------------------------------

static int ensure(cpstep_ctx* c, double** p, size_t* have, size_t need) {
  if (*have >= need) return CPSTEP_OK;
  graph_drop(c);  // a captured step may hold the old buffer
  cudaFree(*p);
  *p = nullptr;
  CPSTEP_CUDA_TRY(cudaMalloc(p, need * sizeof(double)));
  *have = need;
  return CPSTEP_OK;
}

// T = (S/2)^(-1/2); S, T device [n][n] FP64 (symmetric, so row/column-major agree).
// mixed: the iteration to a looser tolerance, then the correction; scale: Gershgorin
// spectral scaling.
int ortho_tmat(cpstep_ctx* c, const double* S, double* T, int n, int mixed, int scale,
               double tol, int max_iter, int* iters_out, double* rms_out, int check_host) {
  using namespace orth;
  const size_t nn = ((size_t)n * n + 1) / 2 * 2;  // matrices on 16-byte boundaries
  // workspace: 9 matrices, two sets of block partials, the status words
  constexpr size_t NPART = 2 * 4096;
  if (int rc = ensure(c, &c->d_ortho_ws, &c->ortho_ws_elems, 9 * nn + NPART + 8)) return rc;
  double* ws = c->d_ortho_ws;
  Work w;
  w.n = n;
  w.max_iter = max_iter;
  w.tol = tol;
  w.S = S;
  w.A = ws;
  w.B = ws + nn;
  w.C = ws + 2 * nn;
  w.A2 = ws + 3 * nn;
  w.B2 = ws + 4 * nn;
  w.X = ws + 5 * nn;
  w.Y = ws + 6 * nn;
  w.E = ws + 7 * nn;
  w.P = ws + 8 * nn;
  w.partial = ws + 9 * nn;
  w.T = T;
  w.status = reinterpret_cast<int*>(ws + 9 * nn + NPART);
  w.rms = ws + 9 * nn + NPART + 2;
  w.newton = mixed ? 1 : 0;
  w.sigma = 2.0;
  // 16-byte copies need even rows and an aligned S (the workspace is)
  w.vec = (n & 1) == 0 && (reinterpret_cast<uintptr_t>(S) & 15) == 0;
  double* d_sigma = ws + 9 * nn + NPART + 4;
  if (scale) {
    orth::k_gershgorin<<<1, 1024, 0, c->stream>>>(S, n, d_sigma);
    CPSTEP_LAUNCH_CHECK();
    double sg = 0.0;
    CPSTEP_CUDA_TRY(cudaMemcpyAsync(&sg, d_sigma, sizeof(double), cudaMemcpyDeviceToHost, c->stream));
    CPSTEP_CUDA_TRY(cudaStreamSynchronize(c->stream));
    w.sigma = std::max(2.0, sg * 1.0001);
  }
  const int ntiles = cdiv(n, TS) * cdiv(n, TS);
  if (c->ortho_wait) CPSTEP_CUDA_TRY(cudaStreamWaitEvent(c->stream, c->ortho_wait, 0));
  if (n <= SN) {
    const size_t smem = sizeof(double) * 5 * SN * SLD;
    CPSTEP_CUDA_TRY(cudaFuncSetAttribute(k_ortho_small, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)smem));
    k_ortho_small<<<1, SNT, smem, c->stream>>>(w);
    CPSTEP_LAUNCH_CHECK();
    if (c->ortho_signal) CPSTEP_CUDA_TRY(cudaEventRecord(c->ortho_signal, c->stream));
  } else {
    const size_t smem = sizeof(double) * STAGE * (n > KC ? 2 : 1);
    CPSTEP_CUDA_TRY(cudaFuncSetAttribute(k_ortho, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)(sizeof(double) * STAGE * 2)));
    int per_sm = 0;
    void* args[] = {&w};
    CPSTEP_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_ortho, NT, smem));
    const int nb = std::max(1, std::min(std::min(2 * ntiles, 4096), per_sm * c->num_sms));
    CPSTEP_CUDA_TRY(cudaLaunchCooperativeKernel((void*)k_ortho, nb, NT, args, smem, c->stream));
    CPSTEP_LAUNCH_CHECK();
    if (c->ortho_signal) CPSTEP_CUDA_TRY(cudaEventRecord(c->ortho_signal, c->stream));
  }
  c->d_ortho_status = w.status;
  if (check_host) {
    int st[2] = {0, 0};
    double r = 0.0;
    CPSTEP_CUDA_TRY(cudaMemcpyAsync(st, w.status, sizeof(st), cudaMemcpyDeviceToHost, c->stream));
    CPSTEP_CUDA_TRY(cudaMemcpyAsync(&r, w.rms, sizeof(double), cudaMemcpyDeviceToHost, c->stream));
    CPSTEP_CUDA_TRY(cudaStreamSynchronize(c->stream));
    if (iters_out) *iters_out = st[0];
    if (rms_out) *rms_out = r;
    if (!st[1]) {
      cpstep_set_error("Ortho: S^-1/2 iteration not converged in %d iterations (rms %g > %g)",
                       st[0], r, tol);
      return CPSTEP_ERR_NOCONV;
    }
  }
  return CPSTEP_OK;
}
