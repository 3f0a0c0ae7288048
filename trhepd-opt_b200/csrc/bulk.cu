// Bulk reflection matrices on the GPU: blkref (sim-trhepd-rheed/src/bulk.f90:7-128)
// for every (angle, beam group) at once.
//
// The reference forms each slice's transfer matrix from the eigendecomposition
// of the slice Hamiltonian H (trmatg.f90:6-59):
//     T = [tau e, rho e^-1; rho e, tau e^-1] [tau rho; rho tau]^-1,
//     tau = (gamma_i + kappa_j) u_ij,  rho = (gamma_i - kappa_j) u_ij.
// With w = (psi, psi') and c = S w, S = [G, -iI; G, iI] (G = diag gamma), the
// right factor maps mode amplitudes to c and the left one advances them by dz, so
//     T = S exp(dz [0 I; -H 0]) S^-1,
//     exp(dz [0 I; -H 0]) = [C, s; -H s, C],  C = cos(sqrt(H) dz),
//                                               s = sin(sqrt(H) dz)/sqrt(H).
// C and s come from a degree-8 Taylor series in X = -H h^2 on h = dz / 2^m
// (||X|| <= 1/4) followed by m double-angle steps C <- 2C^2 - I, s <- 2 s C:
// batched complex GEMMs, no eigensolver.  Each slice's propagator is converted
// to mode space and the slices are chained there, as the reference chains its
// slice transfer matrices (bulk.f90:67-79): chaining in w-space and converting
// once would form the decaying blocks of strongly evanescent beams (e^{-kappa c},
// ~1e-20 over a layer) as differences of ~1e20 entries.  Then the layer
// recursion R <- (T12 + T11 R)(T22 + T21 R)^-1 with the reference's convergence
// exit (bulk.f90:95-119).
#include <cuda_runtime.h>

#include <cmath>

#include "bulk.h"
#include "kernels.h"
#include "launch_attr.h"

namespace trhepd {

// ============================================================ batched complex GEMM
// C_b = alpha A_b B_b + beta C_b (row-major, FP64 DMMA), beta in {0, 1}.
namespace bgemm {
constexpr int BM = 64, BN = 64, BK = 16, STAGES = 3;
constexpr int ASTR = BK + 4, BSTR = BN + 2;
constexpr int A_TILE = BM * ASTR, B_TILE = BK * BSTR;
constexpr size_t SMEM = (size_t)STAGES * (A_TILE + B_TILE) * sizeof(cd);
}  // namespace bgemm

__device__ __forceinline__ void b_cp_async16(void* smem, const void* gmem, bool pred) {
  unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  int sz = pred ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(sz));
}
__device__ __forceinline__ void b_dmma(double& c0, double& c1, double& c2, double& c3, double a0,
                                       double a1, double b0) {
  asm volatile(
      "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, "
      "{%0,%1,%2,%3};\n"
      : "+d"(c0), "+d"(c1), "+d"(c2), "+d"(c3)
      : "d"(a0), "d"(a1), "d"(b0));
}

__global__ void __launch_bounds__(128, 2)
    k_zgemm_batched(BatchedGemm g) {
  using namespace bgemm;
  const int b = blockIdx.z;
  if (g.active && !g.active[b]) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cd* As = reinterpret_cast<cd*>(smem_raw);
  cd* Bs = As + STAGES * A_TILE;
  const cd* A = g.A + (size_t)b * g.sA;
  const cd* B = g.B + (size_t)b * g.sB;
  cd* C = g.C + (size_t)b * g.sC;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int gq = lane >> 2, t = lane & 3;
  const int wm = (warp >> 1) * 32, wn = (warp & 1) * 32;
  const int bm = blockIdx.y * BM, bn = blockIdx.x * BN;
  auto load_stage = [&](int s, int k0) {
    cd* a = As + s * A_TILE;
    cd* bb = Bs + s * B_TILE;
#pragma unroll
    for (int it = 0; it < (BM * BK) / 128; ++it) {
      int e = tid + it * 128;
      int r = e / BK, kk = e % BK;
      bool ok = bm + r < g.M && k0 + kk < g.K;
      b_cp_async16(a + r * ASTR + kk, ok ? A + (size_t)(bm + r) * g.lda + k0 + kk : A, ok);
    }
#pragma unroll
    for (int it = 0; it < (BK * BN) / 128; ++it) {
      int e = tid + it * 128;
      int kk = e / BN, c = e % BN;
      bool ok = k0 + kk < g.K && bn + c < g.N;
      b_cp_async16(bb + kk * BSTR + c, ok ? B + (size_t)(k0 + kk) * g.ldb + bn + c : B, ok);
    }
  };
  double cr[2][4][4], ci[2][4][4];
#pragma unroll
  for (int mi = 0; mi < 2; ++mi)
#pragma unroll
    for (int ni = 0; ni < 4; ++ni)
#pragma unroll
      for (int e = 0; e < 4; ++e) cr[mi][ni][e] = ci[mi][ni][e] = 0.0;
  const int nk = (g.K + BK - 1) / BK;
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) {
    if (s < nk) load_stage(s, s * BK);
    asm volatile("cp.async.commit_group;\n" ::);
  }
  for (int kt = 0; kt < nk; ++kt) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(STAGES - 2));
    __syncthreads();
    int nxt = kt + STAGES - 1;
    if (nxt < nk) load_stage(nxt % STAGES, nxt * BK);
    asm volatile("cp.async.commit_group;\n" ::);
    const cd* a = As + (kt % STAGES) * A_TILE;
    const cd* bb = Bs + (kt % STAGES) * B_TILE;
#pragma unroll
    for (int kk = 0; kk < BK; kk += 4) {
      cd af[2][2], bf[4];
#pragma unroll
      for (int mi = 0; mi < 2; ++mi) {
        af[mi][0] = a[(wm + mi * 16 + gq) * ASTR + kk + t];
        af[mi][1] = a[(wm + mi * 16 + gq + 8) * ASTR + kk + t];
      }
#pragma unroll
      for (int ni = 0; ni < 4; ++ni) bf[ni] = bb[(kk + t) * BSTR + wn + ni * 8 + gq];
#pragma unroll
      for (int mi = 0; mi < 2; ++mi)
#pragma unroll
        for (int ni = 0; ni < 4; ++ni) {
          double* R = cr[mi][ni];
          double* I = ci[mi][ni];
          b_dmma(R[0], R[1], R[2], R[3], af[mi][0].x, af[mi][1].x, bf[ni].x);
          b_dmma(R[0], R[1], R[2], R[3], -af[mi][0].y, -af[mi][1].y, bf[ni].y);
          b_dmma(I[0], I[1], I[2], I[3], af[mi][0].x, af[mi][1].x, bf[ni].y);
          b_dmma(I[0], I[1], I[2], I[3], af[mi][0].y, af[mi][1].y, bf[ni].x);
        }
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::);
#pragma unroll
  for (int mi = 0; mi < 2; ++mi)
#pragma unroll
    for (int ni = 0; ni < 4; ++ni)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        int r = bm + wm + mi * 16 + gq + ((e >= 2) ? 8 : 0);
        int c = bn + wn + ni * 8 + 2 * t + (e & 1);
        if (r < g.M && c < g.N) {
          cd v = g.alpha * cd{cr[mi][ni][e], ci[mi][ni][e]};
          size_t o = (size_t)r * g.ldc + c;
          C[o] = g.beta ? C[o] + v : v;
        }
      }
}

void launch_zgemm_batched(const BatchedGemm& g, cudaStream_t st) {
  using namespace bgemm;
  static SmemOptIn attr;
  attr.ensure((const void*)k_zgemm_batched, SMEM);
  dim3 grid(ceil_div(g.N, BN), ceil_div(g.M, BM), g.batch);
  k_zgemm_batched<<<grid, 128, SMEM, st>>>(g);
}

// ============================================================ bulk element kernels
// Element (i, j) of H = V(slice) + diag(gamma^2) for an item of m beams, padded to n:
// H(i,i) = u0 + g_i^2; H(j,i) = u(e) (j > i); H(i,j) = conj(w(e)), e = iv(j,i)
// (trmatg.f90:150-157).  pg: the group's iv(max, min) - 1; g: the item's gammas.
__device__ __forceinline__ cd bulk_h(const TableEntry* __restrict__ tcol,
                                     const int* __restrict__ pg, const cd* __restrict__ gam, int m,
                                     int n, int i, int j) {
  cd v = cd{0.0, 0.0};
  if (i < m && j < m) {
    if (i == j) {
      cd g = gam[i];
      v = tcol[0].u + g * g;
    } else if (i > j) {  // H(i, j), i > j: u(iv(i, j))
      v = tcol[pg[j * n + i]].u;
    } else {             // H(i, j), i < j: conj(w(iv(j, i)))
      v = conj(tcol[pg[i * n + j]].w);
    }
  }
  return v;
}
// c1 x + c2 x2 + c3 x3
__device__ __forceinline__ cd bulk_poly3(double c1, cd x, double c2, cd x2, double c3, cd x3) {
  return c1 * x + c2 * x2 + c3 * x3;
}
// Blocks of T = S E S^-1 (see file header) at (i, j), times the phase of column j.
__device__ __forceinline__ void bulk_mode(cd gi, cd gj, cd ph, cd e11, cd e12, cd e21, cd e22,
                                          cd& t11, cd& t12, cd& t21, cd& t22) {
  const cd I = cd{0.0, 1.0};
  cd A = gi * e11 - I * e21, B = gi * e12 - I * e22;
  cd Cc = gi * e11 + I * e21, D = gi * e12 + I * e22;
  cd ig = cdiv(cd{1.0, 0.0}, gj);
  t11 = ph * (0.5 * (A * ig + I * B));
  t12 = ph * (0.5 * (A * ig - I * B));
  t21 = ph * (0.5 * (Cc * ig + I * D));
  t22 = ph * (0.5 * (Cc * ig - I * D));
}

// X = -H h^2 for every item; keeps H for the -H s term.
__global__ void k_bulk_hamiltonian(const TableEntry* __restrict__ tcol, const int* __restrict__ pair,
                                   const cd* __restrict__ gam, const int* __restrict__ gsize,
                                   int ngr, int n, int ld, double h2, cd* __restrict__ H,
                                   cd* __restrict__ X) {
  const int b = blockIdx.y;
  const int grp = b % ngr;
  const int m = gsize[grp];
  const int* pg = pair + (size_t)grp * n * n;  // symmetric: iv(max, min) - 1 of the group
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n * n; e += gridDim.x * blockDim.x) {
    int i = e / n, j = e % n;
    const cd v = bulk_h(tcol, pg, gam + (size_t)b * n, m, n, i, j);
    size_t o = ((size_t)b * n + i) * ld + j;
    H[o] = v;
    X[o] = -h2 * v;
  }
}

// out = c0 I + c1 X + c2 X2 + c3 X3 + c4 X4 (X4 may be null)
__global__ void k_bulk_poly(const cd* __restrict__ X, const cd* __restrict__ X2,
                            const cd* __restrict__ X3, const cd* __restrict__ X4, double c0,
                            double c1, double c2, double c3, double c4, int n, int ld, int batch,
                            cd* __restrict__ out) {
  size_t total = (size_t)batch * n * n;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < total;
       e += (size_t)gridDim.x * blockDim.x) {
    size_t b = e / ((size_t)n * n);
    int r = (int)(e % ((size_t)n * n));
    int i = r / n, j = r % n;
    size_t o = (b * n + i) * ld + j;
    cd v = bulk_poly3(c1, X[o], c2, X2[o], c3, X3[o]);
    if (X4) v = v + c4 * X4[o];
    if (i == j) v.x += c0;
    out[o] = v;
  }
}

// A <- alpha * A + beta * B (+ gamma on the diagonal)
__global__ void k_bulk_axpby(cd* __restrict__ A, const cd* __restrict__ B, double alpha,
                             double beta, double diag, int n, int ld, int batch) {
  size_t total = (size_t)batch * n * n;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < total;
       e += (size_t)gridDim.x * blockDim.x) {
    size_t b = e / ((size_t)n * n);
    int r = (int)(e % ((size_t)n * n));
    int i = r / n, j = r % n;
    size_t o = (b * n + i) * ld + j;
    cd v = alpha * A[o] + (B ? beta * B[o] : cd{0.0, 0.0});
    if (i == j) v.x += diag;
    A[o] = v;
  }
}

// E = [C, s; -Hs, C] (2n x 2n, ld2)
__global__ void k_bulk_build_e(const cd* __restrict__ C, const cd* __restrict__ S,
                               const cd* __restrict__ Hs, int n, int ld, int ld2, int batch,
                               cd* __restrict__ E) {
  size_t total = (size_t)batch * n * n;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < total;
       e += (size_t)gridDim.x * blockDim.x) {
    size_t b = e / ((size_t)n * n);
    int r = (int)(e % ((size_t)n * n));
    int i = r / n, j = r % n;
    size_t o = (b * n + i) * ld + j;
    cd* Eb = E + b * 2 * n * ld2;
    Eb[(size_t)i * ld2 + j] = C[o];
    Eb[(size_t)i * ld2 + n + j] = S[o];
    Eb[(size_t)(n + i) * ld2 + j] = -Hs[o];
    Eb[(size_t)(n + i) * ld2 + n + j] = C[o];
  }
}

// T = S E S^-1 (see file header), times the unit-layer phase shift of columns
// j, j+n (bulk.f90:83-93) when `phase` is given; padded beams use gamma = 1.
__global__ void k_bulk_similarity(const cd* __restrict__ E, const cd* __restrict__ gam,
                                  const cd* __restrict__ phase, const int* __restrict__ gsize,
                                  int ngr, int n, int ld2, int batch, cd* __restrict__ T) {
  size_t total = (size_t)batch * n * n;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < total;
       e += (size_t)gridDim.x * blockDim.x) {
    size_t b = e / ((size_t)n * n);
    int r = (int)(e % ((size_t)n * n));
    int i = r / n, j = r % n;
    const int m = gsize[b % ngr];
    const cd* Eb = E + b * 2 * n * ld2;
    cd gi = (i < m) ? gam[b * n + i] : cd{1.0, 0.0};
    cd gj = (j < m) ? gam[b * n + j] : cd{1.0, 0.0};
    cd ph = (phase && j < m) ? phase[b * n + j] : cd{1.0, 0.0};
    cd* Tb = T + b * 2 * n * ld2;
    bulk_mode(gi, gj, ph, Eb[(size_t)i * ld2 + j], Eb[(size_t)i * ld2 + n + j],
              Eb[(size_t)(n + i) * ld2 + j], Eb[(size_t)(n + i) * ld2 + n + j],
              Tb[(size_t)i * ld2 + j], Tb[(size_t)i * ld2 + n + j],
              Tb[(size_t)(n + i) * ld2 + j], Tb[(size_t)(n + i) * ld2 + n + j]);
  }
}

// Unit-layer phase shift (bulk.f90:83-93): columns j and j+n of T times ph_j.
__global__ void k_bulk_phase_cols(cd* __restrict__ T, const cd* __restrict__ phase,
                                  const int* __restrict__ gsize, int ngr, int n, int ld2,
                                  int batch) {
  size_t total = (size_t)batch * 2 * n * n;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < total;
       e += (size_t)gridDim.x * blockDim.x) {
    size_t b = e / ((size_t)2 * n * n);
    int r = (int)(e % ((size_t)2 * n * n));
    int i = r / n, j = r % n;
    if (j >= gsize[b % ngr]) continue;
    const cd ph = phase[b * n + j];
    cd* Tb = T + b * 2 * n * ld2 + (size_t)i * ld2;
    Tb[j] = ph * Tb[j];
    Tb[n + j] = ph * Tb[n + j];
  }
}

// t1 = T12, t2 = T22 (first layer), for active items
__global__ void k_bulk_layer_init(const cd* __restrict__ T, const int* __restrict__ active, int n,
                                  int ld, int ld2, int batch, cd* __restrict__ t1,
                                  cd* __restrict__ t2) {
  size_t total = (size_t)batch * n * n;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < total;
       e += (size_t)gridDim.x * blockDim.x) {
    size_t b = e / ((size_t)n * n);
    if (!active[b]) continue;
    int r = (int)(e % ((size_t)n * n));
    int i = r / n, j = r % n;
    const cd* Tb = T + b * 2 * n * ld2;
    t1[(b * n + i) * ld + j] = Tb[(size_t)i * ld2 + n + j];
    t2[(b * n + i) * ld + j] = Tb[(size_t)(n + i) * ld2 + n + j];
  }
}

// Q = t2^T, P = t1^T (right division through the left solve); padded beams get
// an identity block so the solve stays regular.
__global__ void k_bulk_transpose_pair(const cd* __restrict__ t1, const cd* __restrict__ t2,
                                      const int* __restrict__ active, const int* __restrict__ gsize,
                                      int ngr, int n, int ld, int batch, cd* __restrict__ Q,
                                      cd* __restrict__ P) {
  size_t total = (size_t)batch * n * n;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < total;
       e += (size_t)gridDim.x * blockDim.x) {
    size_t b = e / ((size_t)n * n);
    if (!active[b]) continue;
    int r = (int)(e % ((size_t)n * n));
    int i = r / n, j = r % n;
    const int m = gsize[b % ngr];
    size_t o = (b * n + i) * ld + j, ot = (b * n + j) * ld + i;
    if (i < m && j < m) {
      Q[o] = t2[ot];
      P[o] = t1[ot];
    } else {
      Q[o] = cd{(i == j) ? 1.0 : 0.0, 0.0};
      P[o] = cd{0.0, 0.0};
    }
  }
}

// R = P^T; convergence test of the reference (bulk.f90:105-118): at layer 20 keep
// |R_ii|^2, after it stop the item once max_i ||R_ii|^2 - previous| < epsb.
__global__ void k_bulk_layer_finish(const cd* __restrict__ P, int* __restrict__ active,
                                    const int* __restrict__ gsize, int ngr, int n, int ld,
                                    int layer, double epsb, double* __restrict__ r20,
                                    cd* __restrict__ R) {
  const int b = blockIdx.x;
  if (!active[b]) return;
  const int m = gsize[b % ngr];
  for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
    int i = e / n, j = e % n;
    R[((size_t)b * n + i) * ld + j] = P[((size_t)b * n + j) * ld + i];
  }
  __syncthreads();
  if (layer < 20) return;
  __shared__ double red[32];
  double rmax = 0.0;
  for (int i = threadIdx.x; i < m; i += blockDim.x) {
    cd d = R[((size_t)b * n + i) * ld + i];
    double r2 = (d * conj(d)).x;
    if (layer > 20) rmax = fmax(rmax, fabs(r2 - r20[(size_t)b * n + i]));
    r20[(size_t)b * n + i] = r2;
  }
  for (int o = 16; o > 0; o >>= 1) rmax = fmax(rmax, __shfl_xor_sync(0xffffffffu, rmax, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = rmax;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) rmax = fmax(rmax, red[w]);
    if (layer > 20 && rmax < epsb) active[b] = 0;
  }
}

// ============================================================ small groups
// The whole reflection matrix of an item in one launch, for groups of up to 8 beams (a
// 7 x 7 surface cell has 3 to 7): a warp per item holds every matrix in shared memory
// through all slices and layers.  Products are single MMA tiles (m16n8k4, the operand
// order of k_zgemm_batched), the element formulas are those of the kernels above and the
// layer solve repeats k_gj_panel / k_gj_update (one panel), so the records are theirs bit
// for bit; what it saves is their launches, 15 to 20 of 3 to 15 us per slice for 4 x 4
// matrices in 64 x 64 tiles and 7 per layer with a readback: the N = 23 reference grid
// (483 items, 314 slices, 94 layers) took 52 ms, 8.4 ms with only the slices here.
constexpr int kSmallBulk = 8, kB1 = 9, kB2 = 17;        // row strides of n and 2n matrices
constexpr int kBulkWarps = 4;
constexpr int kBulkElems = 8 * 8 * kB1 + 3 * 16 * kB2;  // complex values per warp

struct BulkSmallArgs {
  const TableEntry* table;
  const int* pair;
  const cd* gam;
  const int* gsize;
  int nv, ns, ngr, n, nitem, m;
  double h, c1[4], c2[5], s1[4], s2[5];
  const cd* phase;  // unit-layer phase shift of the columns (nitem x n), or null
  int ml;           // layers at most
  double epsb;
  cd* R;            // nitem x n x ld
  int ld;
  int* layers;      // most layers of any item
  unsigned* status;
};

// C[i][j] (+)= (A B)(i, j) for the first `rows` rows and `cols` columns, K = k; rows and
// columns of A and B past their sizes hold zeros up to the tile.
template <int kTiles>
__device__ __forceinline__ void bulk_mm(const cd* A, int sa, const cd* B, int sb, int k, cd* C,
                                        int sc, int rows, int cols, bool add) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int nt = 0; nt < kTiles; ++nt) {
    double R[4] = {0.0, 0.0, 0.0, 0.0}, I[4] = {0.0, 0.0, 0.0, 0.0};
    for (int k0 = 0; k0 < k; k0 += 4) {
      const cd a0 = A[g * sa + k0 + t];
      const cd a1 = kTiles == 2 ? A[(g + 8) * sa + k0 + t] : cd{0.0, 0.0};
      const cd b = B[(k0 + t) * sb + nt * 8 + g];
      b_dmma(R[0], R[1], R[2], R[3], a0.x, a1.x, b.x);
      b_dmma(R[0], R[1], R[2], R[3], -a0.y, -a1.y, b.y);
      b_dmma(I[0], I[1], I[2], I[3], a0.x, a1.x, b.y);
      b_dmma(I[0], I[1], I[2], I[3], a0.y, a1.y, b.x);
    }
    __syncwarp();
#pragma unroll
    for (int e = 0; e < 2 * kTiles; ++e) {
      const int i = g + (e >= 2 ? 8 : 0), j = nt * 8 + 2 * t + (e & 1);
      if (i < rows && j < cols) {
        const cd v = cd{R[e], I[e]};
        C[i * sc + j] = add ? C[i * sc + j] + v : v;
      }
    }
  }
  __syncwarp();
}

__global__ void __launch_bounds__(32 * kBulkWarps) k_bulk_small(const BulkSmallArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int b = blockIdx.x * kBulkWarps + warp;
  cd* mem = reinterpret_cast<cd*>(smem_raw) + (size_t)warp * kBulkElems;
  if (b >= a.nitem) return;
  for (int e = lane; e < kBulkElems; e += 32) mem[e] = cd{0.0, 0.0};
  __syncwarp();
  auto m1 = [&](int k) { return mem + k * 8 * kB1; };
  cd *H = m1(0), *X = m1(1), *X2 = m1(2), *X3 = m1(3), *X4 = m1(4), *C = m1(5), *S = m1(6);
  cd* W = m1(7);
  cd *E = mem + 8 * 8 * kB1, *Tt = E + 16 * kB2, *Tn = Tt + 16 * kB2;
  const int n = a.n, n2 = 2 * n, nn = n * n, grp = b % a.ngr, m = a.gsize[grp];
  const int* pg = a.pair + (size_t)grp * nn;
  const cd* gam = a.gam + (size_t)b * n;
  const double h2 = a.h * a.h;
  // at most two elements per lane: e = lane, lane + 32
  cd hv[2];
  auto load = [&](int l) {
    const TableEntry* tc = a.table + (size_t)l * a.nv;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int e = lane + 32 * q;
      hv[q] = e < nn ? bulk_h(tc, pg, gam, m, n, e / n, e % n) : cd{0.0, 0.0};
    }
  };
  auto each = [&](auto&& f) {
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int e = lane + 32 * q;
      if (e < nn) f(e / n, e % n, (e / n) * kB1 + e % n, q);
    }
    __syncwarp();
  };
  auto mm1 = [&](const cd* A, const cd* B, cd* D, bool add) {
    bulk_mm<1>(A, kB1, B, kB1, n, D, kB1, n, n, add);
  };
  load(0);
  for (int l = 0; l < a.ns; ++l) {
    each([&](int, int, int o, int q) {
      H[o] = hv[q];
      X[o] = -h2 * hv[q];
    });
    if (l + 1 < a.ns) load(l + 1);
    mm1(X, X, X2, false);
    mm1(X2, X, X3, false);
    mm1(X2, X2, X4, false);
    each([&](int i, int j, int o, int) {
      cd c = bulk_poly3(a.c1[1], X[o], a.c1[2], X2[o], a.c1[3], X3[o]);
      cd w = bulk_poly3(a.c2[1], X[o], a.c2[2], X2[o], a.c2[3], X3[o]);
      w = w + a.c2[4] * X4[o];
      if (i == j) {
        c.x += a.c1[0];
        w.x += a.c2[0];
      }
      C[o] = c;
      W[o] = w;
    });
    mm1(X4, W, C, true);   // C = P1 + X^4 P2
    each([&](int i, int j, int o, int) {
      cd c = bulk_poly3(a.s1[1], X[o], a.s1[2], X2[o], a.s1[3], X3[o]);
      cd w = bulk_poly3(a.s2[1], X[o], a.s2[2], X2[o], a.s2[3], X3[o]);
      w = w + a.s2[4] * X4[o];
      if (i == j) {
        c.x += a.s1[0];
        w.x += a.s2[0];
      }
      S[o] = c;
      W[o] = w;
    });
    mm1(X4, W, S, true);
    each([&](int, int, int o, int) { S[o] = a.h * S[o]; });  // s = h * series
    for (int q = 0; q < a.m; ++q) {  // C <- 2C^2 - I, s <- 2 s C
      mm1(S, C, X2, false);
      mm1(C, C, W, false);
      each([&](int i, int j, int o, int) {
        cd c = 2.0 * W[o];
        if (i == j) c.x += -1.0;
        C[o] = c;
        S[o] = 2.0 * X2[o];
      });
    }
    mm1(H, S, W, false);
    // the slice's transfer matrix in mode space; T <- T_l T
    cd* D = l == 0 ? Tt : E;
    each([&](int i, int j, int o, int) {
      const cd gi = i < m ? gam[i] : cd{1.0, 0.0}, gj = j < m ? gam[j] : cd{1.0, 0.0};
      bulk_mode(gi, gj, cd{1.0, 0.0}, C[o], S[o], -W[o], C[o], D[i * kB2 + j],
                D[i * kB2 + n + j], D[(n + i) * kB2 + j], D[(n + i) * kB2 + n + j]);
    });
    if (l > 0) {
      if (n2 <= 8) bulk_mm<1>(E, kB2, Tt, kB2, n2, Tn, kB2, n2, n2, false);
      else bulk_mm<2>(E, kB2, Tt, kB2, n2, Tn, kB2, n2, n2, false);
      cd* const tmp = Tt;
      Tt = Tn;
      Tn = tmp;
    }
  }
  if (a.phase) {  // columns j and j + n of T (bulk.f90:83-93)
    for (int e = lane; e < n2 * n; e += 32) {
      const int i = e / n, j = e % n;
      if (j >= m) continue;
      const cd ph = a.phase[(size_t)b * n + j];
      Tt[i * kB2 + j] = ph * Tt[i * kB2 + j];
      Tt[i * kB2 + n + j] = ph * Tt[i * kB2 + n + j];
    }
    __syncwarp();
  }
  // layer recursion R <- (T12 + T11 R)(T22 + T21 R)^-1 (bulk.f90:95-119)
  cd *T11 = H, *T21 = X, *t1 = X2, *t2 = X3, *Q = X4, *P = C, *R = S;
  cd *Linv = E, *Uinv = E + 8 * kB1;  // E, Tn: free now
  cd *W1 = Tn;
  for (int e = lane; e < 8 * kB1; e += 32) T11[e] = T21[e] = R[e] = cd{0.0, 0.0};
  __syncwarp();
  each([&](int i, int j, int o, int) {
    T11[o] = Tt[i * kB2 + j];
    T21[o] = Tt[(n + i) * kB2 + j];
  });
  double r20 = 0.0;
  int layer = 1;
  for (; layer <= a.ml; ++layer) {
    each([&](int i, int j, int o, int) {
      t1[o] = Tt[i * kB2 + n + j];
      t2[o] = Tt[(n + i) * kB2 + n + j];
    });
    if (layer > 1) {
      mm1(T11, R, t1, true);
      mm1(T21, R, t2, true);
    }
    each([&](int i, int j, int o, int) {  // padded beams: an identity block
      const bool in = i < m && j < m;
      Q[o] = in ? t2[j * kB1 + i] : cd{i == j ? 1.0 : 0.0, 0.0};
      P[o] = in ? t1[j * kB1 + i] : cd{0.0, 0.0};
    });
    // LU of Q with partial pivoting, the row swaps also on P
    for (int c = 0; c < n; ++c) {
      double best = -1.0;
      int p = c;
      for (int i = c; i < n; ++i) {
        const double v = cabs1(Q[i * kB1 + c]);
        if (v > best) {
          best = v;
          p = i;
        }
      }
      __syncwarp();
      if (p != c && lane < 2 * n) {
        cd* M = lane < n ? Q : P;
        const int k = lane < n ? lane : lane - n;
        const cd x = M[c * kB1 + k];
        M[c * kB1 + k] = M[p * kB1 + k];
        M[p * kB1 + k] = x;
      }
      __syncwarp();
      const cd d = Q[c * kB1 + c];
      if (d.x == 0.0 && d.y == 0.0 && lane == 0) atomicOr(a.status, kStatusZeroPivot);
      const cd rinv = cdiv(cd{1.0, 0.0}, d);
      if (lane > c && lane < n) Q[lane * kB1 + c] = Q[lane * kB1 + c] * rinv;
      __syncwarp();
      each([&](int i, int j, int o, int) {
        if (i > c && j > c) Q[o] = Q[o] - Q[i * kB1 + c] * Q[c * kB1 + j];
      });
    }
    if (lane < n) {  // column `lane` of the inverses of L and U
      for (int i = 0; i < n; ++i) {
        cd v = cd{i == lane ? 1.0 : 0.0, 0.0};
        for (int q = 0; q < i; ++q) v = v - Q[i * kB1 + q] * Linv[q * kB1 + lane];
        Linv[i * kB1 + lane] = v;
      }
      for (int i = n - 1; i >= 0; --i) {
        cd v = cd{i == lane ? 1.0 : 0.0, 0.0};
        for (int q = i + 1; q < n; ++q) v = v - Q[i * kB1 + q] * Uinv[q * kB1 + lane];
        Uinv[i * kB1 + lane] = cdiv(v, Q[i * kB1 + i]);
      }
    }
    __syncwarp();
    each([&](int i, int j, int o, int) {
      cd v = cd{0.0, 0.0};
      for (int q = 0; q < n; ++q) v = v + Uinv[i * kB1 + q] * Linv[q * kB1 + j];
      W1[o] = v;
    });
    each([&](int i, int j, int, int) {  // R = (W1 P)^T
      cd v = cd{0.0, 0.0};
      for (int q = 0; q < n; ++q) v = v + W1[i * kB1 + q] * P[q * kB1 + j];
      R[j * kB1 + i] = v;
    });
    if (layer >= 20) {
      double change = 0.0;
      if (lane < m) {
        const cd d = R[lane * kB1 + lane];
        const double r2 = (d * conj(d)).x;
        if (layer > 20) change = fabs(r2 - r20);
        r20 = r2;
      }
      for (int o = 16; o > 0; o >>= 1)
        change = fmax(change, __shfl_xor_sync(0xffffffffu, change, o));
      if (layer > 20 && change < a.epsb) break;
    }
  }
  if (lane == 0) atomicMax(a.layers, min(layer, a.ml));
  for (int e = lane; e < nn; e += 32)
    a.R[((size_t)b * n + e / n) * a.ld + e % n] = R[(e / n) * kB1 + e % n];
}

bool bulk_small_fits(int n) { return n <= kSmallBulk; }

void launch_bulk_small(const TableEntry* table, int nv, int ns, const int* pair, const cd* gam,
                       const int* gsize, int ngr, int n, int nitem, int m, double h,
                       const double* fc, const double* fs, const cd* phase, int ml, double epsb,
                       cd* R, int ld, int* layers, unsigned* status, cudaStream_t st) {
  BulkSmallArgs a{};
  a.table = table;
  a.pair = pair;
  a.gam = gam;
  a.gsize = gsize;
  a.nv = nv;
  a.ns = ns;
  a.ngr = ngr;
  a.n = n;
  a.nitem = nitem;
  a.m = m;
  a.h = h;
  for (int k = 0; k < 4; ++k) {
    a.c1[k] = fc[k];
    a.s1[k] = fs[k];
  }
  for (int k = 0; k < 5; ++k) {
    a.c2[k] = fc[4 + k];
    a.s2[k] = fs[4 + k];
  }
  a.phase = phase;
  a.ml = ml;
  a.epsb = epsb;
  a.R = R;
  a.ld = ld;
  a.layers = layers;
  a.status = status;
  static SmemOptIn attr;
  const size_t smem = (size_t)kBulkWarps * kBulkElems * sizeof(cd);
  attr.ensure((const void*)k_bulk_small, smem);
  k_bulk_small<<<ceil_div(nitem, kBulkWarps), 32 * kBulkWarps, smem, st>>>(a);
}

static int grid_for(size_t total) {
  size_t g = (total + 255) / 256;
  return (int)(g > 148 * 16 ? 148 * 16 : (g ? g : 1));
}

void launch_bulk_hamiltonian(const TableEntry* tcol, const int* pair, const cd* gam,
                             const int* gsize, int ngr, int n, int ld, int batch, double h2, cd* H,
                             cd* X, cudaStream_t st) {
  dim3 grid(ceil_div(n * n, 256), batch);
  k_bulk_hamiltonian<<<grid, 256, 0, st>>>(tcol, pair, gam, gsize, ngr, n, ld, h2, H, X);
}
void launch_bulk_poly(const cd* X, const cd* X2, const cd* X3, const cd* X4, const double* c,
                      int n, int ld, int batch, cd* out, cudaStream_t st) {
  size_t total = (size_t)batch * n * n;
  k_bulk_poly<<<grid_for(total), 256, 0, st>>>(X, X2, X3, X4, c[0], c[1], c[2], c[3], c[4], n, ld,
                                                batch, out);
}
void launch_bulk_axpby(cd* A, const cd* B, double alpha, double beta, double diag, int n, int ld,
                       int batch, cudaStream_t st) {
  size_t total = (size_t)batch * n * n;
  k_bulk_axpby<<<grid_for(total), 256, 0, st>>>(A, B, alpha, beta, diag, n, ld, batch);
}
void launch_bulk_build_e(const cd* C, const cd* S, const cd* Hs, int n, int ld, int ld2, int batch,
                         cd* E, cudaStream_t st) {
  size_t total = (size_t)batch * n * n;
  k_bulk_build_e<<<grid_for(total), 256, 0, st>>>(C, S, Hs, n, ld, ld2, batch, E);
}
void launch_bulk_similarity(const cd* E, const cd* gam, const cd* phase, const int* gsize, int ngr,
                            int n, int ld2, int batch, cd* T, cudaStream_t st) {
  size_t total = (size_t)batch * n * n;
  k_bulk_similarity<<<grid_for(total), 256, 0, st>>>(E, gam, phase, gsize, ngr, n, ld2, batch, T);
}
void launch_bulk_phase_cols(cd* T, const cd* phase, const int* gsize, int ngr, int n, int ld2,
                            int batch, cudaStream_t st) {
  size_t total = (size_t)batch * 2 * n * n;
  k_bulk_phase_cols<<<grid_for(total), 256, 0, st>>>(T, phase, gsize, ngr, n, ld2, batch);
}
void launch_bulk_layer_init(const cd* T, const int* active, int n, int ld, int ld2, int batch,
                            cd* t1, cd* t2, cudaStream_t st) {
  size_t total = (size_t)batch * n * n;
  k_bulk_layer_init<<<grid_for(total), 256, 0, st>>>(T, active, n, ld, ld2, batch, t1, t2);
}
void launch_bulk_transpose_pair(const cd* t1, const cd* t2, const int* active, const int* gsize,
                                int ngr, int n, int ld, int batch, cd* Q, cd* P,
                                cudaStream_t st) {
  size_t total = (size_t)batch * n * n;
  k_bulk_transpose_pair<<<grid_for(total), 256, 0, st>>>(t1, t2, active, gsize, ngr, n, ld, batch,
                                                          Q, P);
}
void launch_bulk_layer_finish(const cd* P, int* active, const int* gsize, int ngr, int n, int ld,
                              int batch, int layer, double epsb, double* r20, cd* R,
                              cudaStream_t st) {
  k_bulk_layer_finish<<<batch, 256, 0, st>>>(P, active, gsize, ngr, n, ld, layer, epsb, r20, R);
}

}  // namespace trhepd
