// The EES non-local pass of an FP64 context in G space, on the FP64 tensor
// units (dmma.cuh): the same sums as the NL-grid path of ees.cu by Parseval
// (see k_ees_sep there).  With the columns (atom a, channel c) of
//   B_ac(p) = w_p conj(dyp_c(p)) S_a(p),  S_a(p) = s_x(kx) s_y(ky) s_z(kz)
// over the real view of the points,
//   Z(s, ac)   = psi . B^T                                   k_sums
//   F_psi(s)  -= sum_ac zs(s, ac) B_ac,  zs = 2 vn occ Z     k_psi_force
//   F_a,d     -= sum_p w Re(conj(sum_c dyp_c G_ac) dS_a,d),  G_ac = sum_s zs(s, ac) psi_s
//                                                            k_atom_force
// The derivative sums are taken after the sum over states (G_ac), one product
// of the size of Z where three dMn products per channel would be needed.
// B is formed in the product kernels as its tile goes to shared memory, from
// the atoms' separable transforms: 46 flops per (atom, point) for four columns
// against 16 per state of the products, so no S matrix is stored or read.
//
// Each product is 2 (4 natm) S (2 npts) flops; the FP64 mma rate bounds all
// three.  192 atoms, 128 states, 65,736 points: 25.8 GFLOP each.
#include <algorithm>
#include "ctx.cuh"
#include "dmma.cuh"

namespace e64 {

constexpr int NT = 128;  // columns (k_sums, k_atom_force) or reals of points (k_psi_force)

struct Geo {
  const double2* sep;      // [natm][3][2][2 km + 1]
  const int *kx, *ky, *kz;
  const double* w;
  const double2* dyp;      // [nchan][npts]
  const int* tch;          // [ntyp][4] channels of a type, -1 unused
  const int* act;          // [na] atoms with projectors, in type order
  const int* typ;
  int npts, km, na;
};

__device__ __forceinline__ double2 cm(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// the atom of rank r (-1: none) and its type's channels
__device__ __forceinline__ int atom_of(const Geo& G, int r, int4& ch) {
  const int a = r < G.na ? G.act[r] : -1;
  ch = a >= 0 ? *reinterpret_cast<const int4*>(G.tch + 4 * G.typ[a]) : make_int4(-1, -1, -1, -1);
  return a;
}

// the four columns of atom a (< 0: none) with channels ch4 at point p
__device__ __forceinline__ void columns(const Geo& G, int a, int4 ch4, int p, double2 (&b)[4]) {
#pragma unroll
  for (int k = 0; k < 4; ++k) b[k] = make_double2(0.0, 0.0);
  if (a < 0 || p >= G.npts) return;
  const int nk = 2 * G.km + 1;
  const int ch[4] = {ch4.x, ch4.y, ch4.z, ch4.w};
  const double2* T = G.sep + (size_t)a * 6 * nk + G.km;
  double2 S = cm(T[G.kx[p]], cm(T[2 * nk + G.ky[p]], T[4 * nk + G.kz[p]]));
  const double w = G.w[p];
  S.x *= w;
  S.y *= w;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int c = ch[k];
    if (c < 0) continue;
    const double2 d = G.dyp[(size_t)c * G.npts + p];
    b[k] = make_double2(d.x * S.x + d.y * S.y, d.x * S.y - d.y * S.x);
  }
}

// Z partials: a tile of MT states x 128 columns (32 atoms) over a range of
// 16-point chunks; part[split][col][s].  psi comes in by cp.async, the columns
// are formed by all threads, half of each scheduler's warps before and half
// after their mma's, so that the formation's loads overlap the other half's
// products (one barrier per chunk, two stages).
template <int MT>
__global__ void __launch_bounds__(MT * 4) k_sums(const double2* __restrict__ psi, int S, Geo G,
                                                 int nchunk, double* __restrict__ part, int ncolp,
                                                 int Sp) {
  constexpr int THREADS = MT * 4;
  extern __shared__ __align__(16) double sm[];
  double* As = sm;                       // [2][MT][LDK]
  double* Bs = sm + 2 * MT * dm::LDK;    // [2][128][LDK]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = warp >> 2, wn = warp & 3;
  const int r0 = blockIdx.x * 32, s0 = blockIdx.y * MT;
  const int c0 = (int)((long long)nchunk * blockIdx.z / gridDim.z);
  const int c1 = (int)((long long)nchunk * (blockIdx.z + 1) / gridDim.z);
  __shared__ int4 ch_s[32];
  __shared__ int act_s[32];
  if (tid < 32) act_s[tid] = atom_of(G, r0 + tid, ch_s[tid]);
  __syncthreads();
  double acc[4][4][2];
  dm::zero(acc);
  auto load = [&](int st, int c) {
    for (int q = tid; q < MT * 16; q += THREADS) {
      const int row = q >> 4, pt = q & 15, s = s0 + row, p = c * 16 + pt;
      const bool ok = s < S && p < G.npts;
      tc::cp16(As + (st * MT + row) * dm::LDK + 2 * pt,
                     psi + (ok ? (size_t)s * G.npts + p : 0), ok ? 16 : 0);
    }
    tc::cp_commit();
  };
  auto form = [&](int st, int c) {
    for (int q = tid; q < 512; q += THREADS) {
      const int pt = q & 15, al = q >> 4;
      double2 b[4];
      columns(G, act_s[al], ch_s[al], c * 16 + pt, b);
#pragma unroll
      for (int k = 0; k < 4; ++k)
        *reinterpret_cast<double2*>(Bs + (st * NT + 4 * al + k) * dm::LDK + 2 * pt) = b[k];
    }
  };
  const bool early = (warp >> 2) & 1;
  if (c0 < c1) {
    load(0, c0);
    form(0, c0);
  }
  for (int c = c0; c < c1; ++c) {
    const int st = (c - c0) & 1;
    tc::cp_wait<0>();
    __syncthreads();
    const bool more = c + 1 < c1;
    if (more) load(st ^ 1, c + 1);
    if (more && early) form(st ^ 1, c + 1);
    dm::chunk_nk(acc, As + (st * MT + wm * 32) * dm::LDK, Bs + (st * NT + wn * 32) * dm::LDK,
                 lane);
    if (more && !early) form(st ^ 1, c + 1);
  }
  double* out = part + (size_t)blockIdx.z * ncolp * Sp;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int s = s0 + wm * 32 + i * 8 + (lane >> 2);
    if (s >= Sp) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int col = blockIdx.x * NT + wn * 32 + j * 8 + 2 * (lane & 3);
      out[(size_t)col * Sp + s] = acc[i][j][0];
      out[(size_t)(col + 1) * Sp + s] = acc[i][j][1];
    }
  }
}

// Z from its partials (split order), E_NL partials, and zs = 2 vn occ Z in both
// layouts, zero past the states and the columns in use
__global__ void k_scale(const double* __restrict__ part, int nsplit, int ncolp, int Sp, int S,
                        Geo G, const double* __restrict__ vn, const double* __restrict__ occ,
                        double* __restrict__ zs, double* __restrict__ zst,
                        double* __restrict__ epart) {
  const int col = blockIdx.x * 8 + threadIdx.y, s = blockIdx.y * 32 + threadIdx.x;
  const int r = col >> 2;
  int c = -1;
  if (r < G.na) c = G.tch[4 * G.typ[G.act[r]] + (col & 3)];
  double e = 0.0, z = 0.0;
  if (c >= 0 && s < S) {
    const size_t step = (size_t)ncolp * Sp;
    const double* q = part + (size_t)col * Sp + s;
#pragma unroll 8
    for (int k = 0; k < nsplit; ++k) z += q[k * step];
    const double f = vn[c] * occ[s];
    e = z * z * f;
    z *= 2.0 * f;
  }
  zst[(size_t)col * Sp + s] = z;
  zs[(size_t)s * ncolp + col] = z;
  for (int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
  if (threadIdx.x == 0) epart[(size_t)col * gridDim.y + blockIdx.y] = e;
}

// F_psi -= zs B: a tile of MT states x 64 points, the columns in chunks of 32
// (8 atoms)
template <int MT>
__global__ void __launch_bounds__(MT * 4) k_psi_force(const double* __restrict__ zs, int ncolp,
                                                      int S, Geo G, double2* __restrict__ f) {
  constexpr int THREADS = MT * 4;
  extern __shared__ __align__(16) double sm[];
  double* As = sm;                       // [2][MT][LDK]
  double* Bs = sm + 2 * MT * dm::LDK;    // [2][32][LDN]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = warp >> 2, wn = warp & 3;
  const int p0 = blockIdx.x * 64, s0 = blockIdx.y * MT;
  const int nchunk = (4 * G.na + 31) / 32;
  double acc[4][4][2];
  dm::zero(acc);
  auto load = [&](int st, int c) {
    for (int q = tid; q < MT * 16; q += THREADS) {
      const int row = q >> 4, k = 2 * (q & 15), s = s0 + row;
      const bool ok = s < S;
      tc::cp16(As + (st * MT + row) * dm::LDK + k,
                     zs + (ok ? (size_t)s * ncolp + c * 32 + k : 0), ok ? 16 : 0);
    }
    tc::cp_commit();
  };
  auto form = [&](int st, int c) {
    for (int q = tid; q < 512; q += THREADS) {
      const int pt = q & 63, al = q >> 6;
      double2 b[4];
      int4 ch;
      const int a = atom_of(G, c * 8 + al, ch);
      columns(G, a, ch, p0 + pt, b);
#pragma unroll
      for (int k = 0; k < 4; ++k)
        *reinterpret_cast<double2*>(Bs + (st * 32 + 4 * al + k) * dm::LDN + 2 * pt) = b[k];
    }
  };
  const bool early = (warp >> 2) & 1;
  load(0, 0);
  form(0, 0);
  for (int c = 0; c < nchunk; ++c) {
    const int st = c & 1;
    tc::cp_wait<0>();
    __syncthreads();
    const bool more = c + 1 < nchunk;
    if (more) load(st ^ 1, c + 1);
    if (more && early) form(st ^ 1, c + 1);
    dm::chunk_kn(acc, As + (st * MT + wm * 32) * dm::LDK, Bs + st * 32 * dm::LDN + wn * 32, lane);
    if (more && !early) form(st ^ 1, c + 1);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int s = s0 + wm * 32 + i * 8 + (lane >> 2);
    if (s >= S) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int p = p0 + wn * 16 + j * 4 + (lane & 3);
      if (p >= G.npts) continue;
      double2 v = f[(size_t)s * G.npts + p];
      v.x -= acc[i][j][0];
      v.y -= acc[i][j][1];
      f[(size_t)s * G.npts + p] = v;
    }
  }
}

// Atom-force sums: G_ac = sum_s zs psi_s for 32 atoms x 64 points, then
// sum_p Re(w conj(sum_c dyp_c G_ac) dS_a,d) per lattice axis d.  A block walks
// the point tiles blockIdx.y, blockIdx.y + gridDim.y, ... of its 32 atoms with
// the sums in registers: fpart[blockIdx.y][a][3].  The four channel lanes of
// an atom share its sum over channels; lane d < 3 of them takes axis d.
__global__ void __launch_bounds__(512) k_atom_force(const double* __restrict__ zst, int Sp,
                                                    const double2* __restrict__ psi, int S, Geo G,
                                                    double* __restrict__ fpart) {
  extern __shared__ __align__(16) double sm[];
  double* As = sm;                       // [2][128][LDK]
  double* Bs = sm + 2 * NT * dm::LDK;    // [2][32][LDN]
  __shared__ double red[4][4][32];       // [wn][axis][atom]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = warp >> 2, wn = warp & 3;
  const int r0 = blockIdx.x * 32;
  const int nkc = Sp / 32, ntile = (G.npts + 63) / 64;
  const int mine = ((int)blockIdx.y < ntile) ? (ntile - 1 - (int)blockIdx.y) / (int)gridDim.y + 1 : 0;
  const int total = mine * nkc;
  double acc[4][4][2], fa[4] = {0.0, 0.0, 0.0, 0.0};
  dm::zero(acc);
  auto load = [&](int st, int it) {
    const int p0 = ((int)blockIdx.y + (it / nkc) * (int)gridDim.y) * 64, sb = (it % nkc) * 32;
    for (int q = tid; q < NT * 16; q += 512) {
      const int row = q >> 4, k = 2 * (q & 15);
      tc::cp16(As + (st * NT + row) * dm::LDK + k,
                     zst + (size_t)(blockIdx.x * NT + row) * Sp + sb + k, 16);
    }
    for (int q = tid; q < 32 * 64; q += 512) {
      const int row = q >> 6, pt = q & 63, s = sb + row, p = p0 + pt;
      const bool ok = s < S && p < G.npts;
      tc::cp16(Bs + (st * 32 + row) * dm::LDN + 2 * pt,
                     psi + (ok ? (size_t)s * G.npts + p : 0), ok ? 16 : 0);
    }
    tc::cp_commit();
  };
  const int g = lane >> 2, t = lane & 3, ch = g & 3, nk = 2 * G.km + 1;
  if (total > 0) load(0, 0);
  for (int it = 0; it < total; ++it) {
    const int st = it & 1;
    tc::cp_wait<0>();
    __syncthreads();
    if (it + 1 < total) load(st ^ 1, it + 1);
    dm::chunk_kn(acc, As + (st * NT + wm * 32) * dm::LDK, Bs + st * 32 * dm::LDN + wn * 32, lane);
    if (it % nkc != nkc - 1) continue;
    const int p0 = ((int)blockIdx.y + (it / nkc) * (int)gridDim.y) * 64;
    // two points of an atom at a time, the loads of both in flight before the
    // first is used; past the ends they read valid entries that count for nothing
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      int pt[2], kx[2], ky[2], kz[2];
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        pt[j] = min(p0 + wn * 16 + (2 * h + j) * 4 + t, G.npts - 1);
        kx[j] = __ldg(G.kx + pt[j]);
        ky[j] = __ldg(G.ky + pt[j]);
        kz[j] = __ldg(G.kz + pt[j]);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = r0 + wm * 8 + i * 2 + (g >> 2);
        const int a = r < G.na ? __ldg(G.act + r) : -1;
        const int c = a >= 0 ? __ldg(G.tch + 4 * G.typ[a] + ch) : -1;
        const double2* T = G.sep + (size_t)max(a, 0) * 6 * nk + G.km;
        const double2* Tx = T + (ch == 0 ? nk : 0);
        const double2* Ty = T + (ch == 1 ? 3 : 2) * nk;
        const double2* Tz = T + (ch == 2 ? 5 : 4) * nk;
        const double2* dyp = G.dyp + (size_t)max(c, 0) * G.npts;
        double2 d[2], x[2], y[2], z[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          d[j] = __ldg(dyp + pt[j]);
          x[j] = __ldg(Tx + kx[j]);
          y[j] = __ldg(Ty + ky[j]);
          z[j] = __ldg(Tz + kz[j]);
        }
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          double2 q = cm(d[j], make_double2(acc[i][2 * h + j][0], acc[i][2 * h + j][1]));
          if (c < 0) q = make_double2(0.0, 0.0);
          acc[i][2 * h + j][0] = acc[i][2 * h + j][1] = 0.0;
#pragma unroll
          for (int o = 4; o <= 8; o <<= 1) {
            q.x += __shfl_xor_sync(0xffffffffu, q.x, o);
            q.y += __shfl_xor_sync(0xffffffffu, q.y, o);
          }
          if (ch < 3 && a >= 0 && p0 + wn * 16 + (2 * h + j) * 4 + t < G.npts) {
            const double2 D = cm(x[j], cm(y[j], z[j]));
            fa[i] += __ldg(G.w + pt[j]) * (q.x * D.x + q.y * D.y);
          }
        }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    fa[i] += __shfl_xor_sync(0xffffffffu, fa[i], 1);
    fa[i] += __shfl_xor_sync(0xffffffffu, fa[i], 2);
    if (t == 0) red[wn][ch][wm * 8 + i * 2 + (g >> 2)] = fa[i];
  }
  __syncthreads();
  if (tid < 96) {
    const int al = tid / 3, d = tid % 3, r = r0 + al;
    if (r < G.na)
      fpart[((size_t)blockIdx.y * G.na + r) * 3 + d] =
          (red[0][d][al] + red[1][d][al]) + (red[2][d][al] + red[3][d][al]);
  }
}

struct Cell {
  double h[9];
  double grid;
};

// energies[NL] (block 0) and the Cartesian atom forces (one warp per atom: a thread
// each took 20 us over 74 partials, latency after latency)
__global__ void k_finish(const double* __restrict__ epart, int ne, double* __restrict__ energies,
                         const double* __restrict__ fpart, int nblk, Geo G, Cell C,
                         double* __restrict__ fatm) {
  __shared__ double red[32];
  if (blockIdx.x == 0) {
    double e = 0.0;
    for (int i = threadIdx.x; i < ne; i += blockDim.x) e += epart[i];
    e = block_sum(e, red);
    if (threadIdx.x == 0 && energies) energies[CPSTEP_E_NL] = e;
    return;
  }
  const int r = (int)((blockIdx.x - 1) * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (r >= G.na) return;
  double f[3] = {0.0, 0.0, 0.0};
  for (int b = lane; b < nblk; b += 32)
#pragma unroll
    for (int d = 0; d < 3; ++d) f[d] += fpart[((size_t)b * G.na + r) * 3 + d];
#pragma unroll
  for (int d = 0; d < 3; ++d)
    for (int o = 16; o > 0; o >>= 1) f[d] += __shfl_xor_sync(0xffffffffu, f[d], o);
  if (lane >= 3) return;
  fatm[3 * (size_t)G.act[r] + lane] -=
      C.grid * (f[0] * C.h[3 * lane] + f[1] * C.h[3 * lane + 1] + f[2] * C.h[3 * lane + 2]);
}

template <typename K>
int smem(K k, size_t bytes) {
  CPSTEP_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
  return CPSTEP_OK;
}

template <int MT>
int sums(cpstep_ctx* c, const double2* psi, const Geo& G, int nsplit, int ncolp, int Sp) {
  const size_t b = sizeof(double) * 2 * dm::LDK * (MT + NT);
  if (int rc = smem(k_sums<MT>, b)) return rc;
  k_sums<MT><<<dim3(ncolp / NT, cdiv(c->nstates, MT), nsplit), MT * 4, b, c->stream>>>(
      psi, c->nstates, G, cdiv(G.npts, 16), c->nl.e64_part, ncolp, Sp);
  CPSTEP_LAUNCH_CHECK();
  return CPSTEP_OK;
}

template <int MT>
int psi_force(cpstep_ctx* c, const Geo& G, int ncolp, double2* f) {
  const size_t b = sizeof(double) * 2 * (MT * dm::LDK + 32 * dm::LDN);
  if (int rc = smem(k_psi_force<MT>, b)) return rc;
  k_psi_force<MT><<<dim3(cdiv(G.npts, 64), cdiv(c->nstates, MT)), MT * 4, b, c->stream>>>(
      c->nl.e64_zs, ncolp, c->nstates, G, f);
  CPSTEP_LAUNCH_CHECK();
  return CPSTEP_OK;
}

// rows of states per tile: the smallest of 32, 64, 128 that holds them all
int tile_rows(int S) { return S <= 32 ? 32 : (S <= 64 ? 64 : 128); }

// K splits of k_sums: the fewest chunks one after the other (block rounds times the
// chunks of a split) plus the splits' own cost in k_scale's sum, about a twentieth
// of a chunk each (a chunk of 128 states takes 5.4 us, a partial's load 0.1 to 0.2);
// four chunks at least.  54 atoms, 101 states of 14,835 points: 22 splits 237 us,
// 72 80 us.
int splits(int sms, int tiles, int nchunk) {
  int best = 1;
  double cost = 1e30;
  for (int k = 1; k <= std::max(1, std::min(sms, nchunk / 4)); ++k) {
    if ((long long)tiles * k > 4LL * sms && k > 1) break;
    const double cst = (double)((tiles * k + sms - 1) / sms) * ((nchunk + k - 1) / k) + 0.05 * k;
    if (cst < cost) {
      cost = cst;
      best = k;
    }
  }
  return best;
}

}  // namespace e64

// Active atoms (type order), channel table and scratch of the FP64 G-space
// pass; n.gspace64 stays 0 when a type has more than four channels.
int ees64_set(cpstep_ctx* c, const std::vector<int>& order) {
  NlData& n = c->nl;
  const AtomData& at = c->atoms;
  for (int t = 0; t < at.ntyp; ++t)
    if (n.tch[t].size() > 4) return CPSTEP_OK;
  std::vector<int> act, tch((size_t)at.ntyp * 4, -1);
  for (int t = 0; t < at.ntyp; ++t) {
    for (size_t k = 0; k < n.tch[t].size(); ++k) tch[(size_t)t * 4 + k] = n.tch[t][k];
    if (n.tch[t].empty()) continue;
    for (int r = at.tstart[t]; r < at.tstart[t + 1]; ++r) act.push_back(order[r]);
  }
  n.e64_na = (int)act.size();
  if (!n.e64_na) return CPSTEP_OK;
  const int S = c->nstates, ntile = cdiv(n.e64_na, 32), ncolp = ntile * e64::NT;
  const int Sp = cdiv(S, 32) * 32;
  n.e64_split = e64::splits(c->num_sms, ntile * cdiv(S, e64::tile_rows(S)), cdiv(c->npts, 16));
  n.e64_nblk = std::max(1, std::min(cdiv(c->npts, 64), c->num_sms / ntile));
  CPSTEP_CUDA_TRY(cudaMalloc(&n.sep, sizeof(double2) * at.natm * 6 * (2 * (size_t)n.km + 1)));
  CPSTEP_CUDA_TRY(cudaMalloc(&n.e64_part, sizeof(double) * n.e64_split * ncolp * (size_t)Sp));
  CPSTEP_CUDA_TRY(cudaMalloc(&n.e64_zs, sizeof(double) * 2 * ncolp * (size_t)Sp));
  CPSTEP_CUDA_TRY(cudaMalloc(&n.e64_e, sizeof(double) * ncolp * (Sp / 32)));
  CPSTEP_CUDA_TRY(cudaMalloc(&n.e64_f, sizeof(double) * n.e64_nblk * n.e64_na * 3));
  CPSTEP_CUDA_TRY(cudaMalloc(&n.e64_act, sizeof(int) * act.size()));
  CPSTEP_CUDA_TRY(cudaMemcpy(n.e64_act, act.data(), sizeof(int) * act.size(),
                             cudaMemcpyHostToDevice));
  CPSTEP_CUDA_TRY(cudaMalloc(&n.d_tch, sizeof(int) * tch.size()));
  CPSTEP_CUDA_TRY(cudaMemcpy(n.d_tch, tch.data(), sizeof(int) * tch.size(),
                             cudaMemcpyHostToDevice));
  CPSTEP_CUDA_TRY(cudaMalloc(&n.d_vn, sizeof(double) * n.nchan));
  CPSTEP_CUDA_TRY(cudaMemcpy(n.d_vn, n.ch_vn.data(), sizeof(double) * n.nchan,
                             cudaMemcpyHostToDevice));
  n.gspace64 = 1;
  return CPSTEP_OK;
}

// Whether the G-space pass is the faster one.  Its three products cost 48 flops per
// (atom, point, state), states and atoms padded to whole tiles, at the rates the
// tiles reach (an estimate of the whole pass, launches included); the NL-grid form
// a transform pair per channel and state, slower where the line length has no
// shuffle form or a plane leaves room for one block per SM, and the stencils of
// each atom.  ms, G-space / grid form:
//   195 atoms, 65,736 points, NL 80^3: 1.63/0.50 with 1 state, 1.63/0.87 with 8,
//   1.64/1.57 with 16, 1.92/2.58 with 33, 3.4/8.9 with 128; 600 atoms there, 64
//   states: 5.6/6.0, 900 atoms 8.1/6.8
//   405 atoms, 136,092 points, NL 96^3: 7.6/11.3 with 64
//   771 atoms, 258,510 points, NL 120^3: 20/12.5 with 16, 29/24 with 33, 29/48 with
//   64, 96/189 with 256
//   27 atoms, 2,575 points, NL 28^3: 0.09/0.48 with 1
bool ees64_faster(const cpstep_ctx* c) {
  const NlData& n = c->nl;
  const int S = c->nstates, mt = e64::tile_rows(S);
  const double rate = mt == 32 ? 1.5e13 : (mt == 64 ? 2.2e13 : 2.65e13);
  const double rows = (double)cdiv(S, mt) * mt, atoms = 32.0 * cdiv(n.e64_na, 32);
  const double tg = 80e-6 + 48.0 * atoms * c->npts * rows / rate;
  const bool one = 2 * (n.ops.nl_smem(c->nplane_x) + 1024) > 228 * 1024;  // plane blocks per SM
  const double line = (n.ops.shfl_lines ? 1.1e-11 : 1.9e-11) * (one ? 1.6 : 1.0);
  const double tf =
      55e-6 * n.nchan + S * (line * n.nchan * (double)n.nkf * n.nkf * n.nkf + 7e-8 * n.e64_na);
  return tg < tf;
}

int ees64_front(cpstep_ctx* c, const double* psi, const double* occ, bool forces) {
  NlData& n = c->nl;
  const int S = c->nstates;
  e64::Geo G{n.sep,   c->d_kx,   c->d_ky,       c->d_kz, c->d_wpt, n.dyp,
             n.d_tch, n.e64_act, c->atoms.typ,  c->npts, n.km,     n.e64_na};
  const int ntile = cdiv(n.e64_na, 32), ncolp = ntile * e64::NT, Sp = cdiv(S, 32) * 32;
  const double2* ps = reinterpret_cast<const double2*>(psi);
  double* zst = n.e64_zs + (size_t)ncolp * Sp;
  int rc;
  switch (e64::tile_rows(S)) {
    case 32: rc = e64::sums<32>(c, ps, G, n.e64_split, ncolp, Sp); break;
    case 64: rc = e64::sums<64>(c, ps, G, n.e64_split, ncolp, Sp); break;
    default: rc = e64::sums<128>(c, ps, G, n.e64_split, ncolp, Sp); break;
  }
  if (rc) return rc;
  e64::k_scale<<<dim3(ncolp / 8, Sp / 32), dim3(32, 8), 0, c->stream>>>(
      n.e64_part, n.e64_split, ncolp, Sp, S, G, n.d_vn, occ, n.e64_zs, zst, n.e64_e);
  CPSTEP_LAUNCH_CHECK();
  if (forces) {
    const size_t b = sizeof(double) * 2 * (e64::NT * dm::LDK + 32 * dm::LDN);
    if ((rc = e64::smem(e64::k_atom_force, b))) return rc;
    e64::k_atom_force<<<dim3(ntile, n.e64_nblk), 512, b, c->stream>>>(zst, Sp, ps, S, G, n.e64_f);
    CPSTEP_LAUNCH_CHECK();
  }
  return CPSTEP_OK;
}

int ees64_back(cpstep_ctx* c, double* fpsi, double* energies, double* fatm) {
  NlData& n = c->nl;
  const int S = c->nstates;
  e64::Geo G{n.sep,   c->d_kx,   c->d_ky,       c->d_kz, c->d_wpt, n.dyp,
             n.d_tch, n.e64_act, c->atoms.typ,  c->npts, n.km,     n.e64_na};
  const int ncolp = cdiv(n.e64_na, 32) * e64::NT, Sp = cdiv(S, 32) * 32;
  double2* f = reinterpret_cast<double2*>(fpsi);
  int rc;
  switch (e64::tile_rows(S)) {
    case 32: rc = e64::psi_force<32>(c, G, ncolp, f); break;
    case 64: rc = e64::psi_force<64>(c, G, ncolp, f); break;
    default: rc = e64::psi_force<128>(c, G, ncolp, f); break;
  }
  if (rc) return rc;
  e64::Cell C;
  for (int k = 0; k < 9; ++k) C.h[k] = c->hmati[k];
  C.grid = (double)n.nkf;
  e64::k_finish<<<1 + (fatm ? cdiv(n.e64_na, 4) : 0), 128, 0, c->stream>>>(
      n.e64_e, ncolp * (Sp / 32), energies, n.e64_f, n.e64_nblk, G, C, fatm);
  CPSTEP_LAUNCH_CHECK();
  return CPSTEP_OK;
}
