// Renormalisation of the surface solve (sm_100a): the Gershgorin estimate
// (cond_est, sim-trhepd-rheed/src/matcomp.f90:498-528) and Q^{-1} P (matAbdivB,
// matcomp.f90:53-69) of every flagged angle, as a Gauss-Jordan elimination of
// [Q | P] on thread-block clusters and the FP64 tensor path.
//
// Pivoting is implicit: rows never move.  The pivot of column c is the row with the
// largest |re|+|im| (to 2^-11) among those that have not been a pivot yet; order[row]
// = c remembers it, and the finished P is permuted once at the end.  So neither the
// panels nor the trailing updates exchange rows.
//
// Sixteen columns ("sub-panel") are one CTA's, in its registers.  In-place elimination
// of a sub-panel leaves E: new rows = (pivot row of this sub-panel ? 0 : row) + E C1,
// C1 the sub-panel's pivot rows before it.  The CTAs of a cluster hold neighbouring
// sub-panels and apply the earlier ones' E (read from L2) to their own registers, so a
// cluster of S CTAs eliminates 16 S columns in one launch.
//
// * n <= 128: one cluster of ceil(n/16) <= 8 CTAs holds all of [Q | P], a sub-panel of
//   each in every CTA: one launch per renormalisation, state read and written once.
// * larger: per block of 16 S columns a cluster launch (its sub-panels' E), a small one
//   for the pivot rows those apply to, and one rank-16 S update of the trailing columns
//   by FP64 MMAs, numerically S rank-16 updates in turn; at the end the row permutation
//   of P.
#include <cuda_runtime.h>

#include <algorithm>
#include <stdexcept>
#include <type_traits>

#include "kernels.h"
#include "launch_attr.h"

namespace trhepd {
namespace gj {

constexpr int kW = 16;        // columns per CTA
constexpr int kMaxBlock = 8;  // CTAs of a cluster (the portable size)

__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ cd ldcg(const cd* p) {
  const double2 v = __ldcg(reinterpret_cast<const double2*>(p));
  return cd{v.x, v.y};
}
__device__ __forceinline__ void stcg(cd* p, cd v) {
  __stcg(reinterpret_cast<double2*>(p), make_double2(v.x, v.y));
}

struct BlockArgs {
  cd* Q;
  cd* P;
  const int* flag;
  int n, ld, c0, w;   // the block's columns c0 .. c0+w-1 (whole: 0 and n)
  int nsub;           // sub-panels of the block = ceil(w / 16)
  int* order;         // nang x n: the column a row was pivot of, -1 before
  int* piv;           // nang x n: the pivot row of each column
  cd* E;              // nang x n x ew
  int ew;
  cd* C1;             // nang x 16 S x ldc: the block's pivot rows, trailing columns
  int ldc;
  long long c1stride;
  unsigned* status;
};

__device__ __forceinline__ void mma64(double& c0, double& c1, double& c2, double& c3, double a0,
                                      double a1, double b0) {
  asm volatile(
      "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, "
      "{%0,%1,%2,%3};\n"
      : "+d"(c0), "+d"(c1), "+d"(c2), "+d"(c3)
      : "d"(a0), "d"(a1), "d"(b0));
}

__device__ __forceinline__ void cp16(void* smem, const void* gmem, bool pred) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(gmem),
               "r"(pred ? 16 : 0));
}

// One cluster of `ctas` CTAs per angle.  kG = 1: CTA s holds the block's columns 16 s ..;
// kG = 2 (the whole of [Q | P], c0 = 0, w = n): also P's columns 16 s .., and the
// elimination is finished here (permuted P, Q = I).
//
// A warp holds 16 kRT rows in the accumulator layout of the FP64 MMA: lane (g, t) has
// rows g, g+8, g+16, .. and columns t, t+4, t+8, t+12, so a column step needs 4 values of
// the pivot row per lane (a row per thread needed all 16, and the shared-memory
// broadcasts, 17 warps x 16 x 512 B, took twice the time of the arithmetic), and
// another CTA's E is applied with MMAs straight on the registers: complex numbers as
// (re, im) column pairs, K ordered so that lane t's A values of two k-steps are the
// parts of one complex E entry.
//
// The step chain (key, reduction, candidate rows, barrier, reciprocal, update; 1.1 K
// clocks at n = 47, 2.6 K at n = 521) bounds a sub-panel.  One redux.sync on a 32-bit key:
// the exponent and 11 leading mantissa bits of |re|+|im| over the row number, so the
// pivot is the largest to within 2^-11, which bounds the multipliers by 1.0005 instead of
// 1.  The column group at hand is always x[.][0], the groups rotate: one copy of the step
// in the instruction stream for the taller warps.
template <int kG, int kRT, int kMaxT, int kMinB>
__global__ void __launch_bounds__(kMaxT, kMinB) k_gj_block(const BlockArgs g, int ctas) {
  const int a = blockIdx.x / ctas, s = blockIdx.x - a * ctas;
  if (g.flag && !g.flag[a]) return;  // the whole cluster
  constexpr int kWarps = kMaxT / 32, kCStr = kW * kG + 4, kR = 2 * kRT, kWarpRows = 16 * kRT;
  __shared__ __align__(16) unsigned keys[2][32];
  __shared__ cd urow[2][kWarps][kW];
  __shared__ cd c1s[kW][kCStr];
  __shared__ int pivs[kW];
  __shared__ signed char slot[kWarps * kWarpRows];  // row -> pivot step of the E being applied
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int gq = lane >> 2, t4 = lane & 3;
  const int n = g.n, row0 = warp * kWarpRows + gq;  // this lane's rows are row0 + 8 r
  const unsigned full = 0xffffffffu;
  int* const order = g.order + (size_t)a * n;
  int* const piv = g.piv + (size_t)a * n;
  cd* const E = g.E + (size_t)a * n * g.ew;
  const size_t abase = (size_t)a * n * g.ld + g.c0 + s * kW;  // this CTA's columns
  const int cols = min(kW, g.w - s * kW);
  cd x[kR][4 * kG];   // [row][column / 4]; the second half P's
  unsigned used = 0;  // bit r: row r is no candidate (a pivot before, or past n)
#pragma unroll
  for (int r = 0; r < kR; ++r) {
    const int row = row0 + 8 * r;
    if (row >= n || (g.c0 > 0 && order[row] >= 0)) used |= 1u << r;
    if (g.c0 == 0 && s == 0 && t4 == 0 && row < n) order[row] = -1;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const bool ok = row < n && q * 4 + t4 < cols;
      const size_t o = abase + (size_t)row * g.ld + q * 4 + t4;
      x[r][q] = ok ? g.Q[o] : cd{0.0, 0.0};
      if constexpr (kG == 2) x[r][q + 4] = ok ? g.P[o] : cd{0.0, 0.0};
    }
  }
  for (int e = tid; e < 64; e += blockDim.x) keys[e >> 5][e & 31] = 0;
  for (int r = tid; r < kWarps * kWarpRows; r += blockDim.x) slot[r] = -1;
  __syncthreads();

  for (int t = 0; t < g.nsub; ++t) {
    const int cbase = g.c0 + t * kW;
    if (s == t) {
#pragma unroll (kRT == 1 ? 4 : 1)
      for (int q = 0; q < 4; ++q) {
#pragma unroll 1
        for (int tj = 0; tj < 4; ++tj) {
          const int jj = q * 4 + tj;
          if (jj >= cols) break;
          const int buf = jj & 1;
          unsigned key = 0;  // a candidate's key is positive
          if (t4 == tj) {
#pragma unroll
            for (int r = 0; r < kR; ++r) {
              const unsigned hi = (unsigned)__double2hiint(cabs1(x[r][0]));
              const unsigned k = ((hi << 1) & ~1023u) | (unsigned)(1023 - (row0 + 8 * r));
              if (!((used >> r) & 1u)) key = max(key, k);
            }
          }
          key = __reduce_max_sync(full, key);
          if (lane == 0) keys[buf][warp] = key;
          // every warp publishes its candidate row before the one barrier
          const int own = 1023 - (int)(key & 1023u) - warp * kWarpRows;
          const int cr = key != 0 && gq == (own & 7) ? own >> 3 : -1;
#pragma unroll
          for (int r = 0; r < kR; ++r)
            if (r == cr) {
#pragma unroll
              for (int k = 0; k < 4; ++k) urow[buf][warp][((q + k) & 3) * 4 + t4] = x[r][k];
            }
          __syncthreads();
          unsigned top = 0;
#pragma unroll
          for (int w = 0; w < kWarps; w += 4) {
            const uint4 v = *reinterpret_cast<const uint4*>(&keys[buf][w]);
            top = max(max(max(top, v.x), max(v.y, v.z)), v.w);
          }
          const int p = 1023 - (int)(top & 1023u);
          const int pw = p / kWarpRows, pl = p - warp * kWarpRows;  // its warp; within this one
          const cd* up = urow[buf][pw];
          const cd d = up[jj];
          cd u[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) u[k] = up[((q + k) & 3) * 4 + t4];
          const cd rc = crecip(d);
#pragma unroll
          for (int r = 0; r < kR; ++r) {
            // the row's entry of column jj is lane (gq, tj)'s
            const cd f = cd{__shfl_sync(full, x[r][0].x, tj, 4),
                            __shfl_sync(full, x[r][0].y, tj, 4)} * rc;
#pragma unroll
            for (int k = 0; k < 4; ++k) x[r][k] = cfms(f, u[k], x[r][k]);
            if (t4 == tj) x[r][0] = -f;
          }
          if (pl >= 0 && pl < kWarpRows && gq == (pl & 7)) {  // the pivot row is scaled instead
            const int pr = pl >> 3;
            used |= 1u << pr;
#pragma unroll
            for (int r = 0; r < kR; ++r)
              if (r == pr) {
#pragma unroll
                for (int k = 0; k < 4; ++k) x[r][k] = u[k] * rc;
                if (t4 == tj) x[r][0] = rc;
              }
            if (t4 == tj) {
              pivs[jj] = p;
              if (d.x == 0.0 && d.y == 0.0) atomicOr(g.status, kStatusZeroPivot);
            }
          }
          __syncwarp();
        }
#pragma unroll
        for (int r = 0; r < kR; ++r) {
          const cd f = x[r][0];
#pragma unroll
          for (int k = 1; k < 4; ++k) x[r][k - 1] = x[r][k];
          x[r][3] = f;
        }
      }
      // the pivots leave in one go: a global store per step would hold up its barrier
      __syncthreads();
      if (tid < cols) {
        piv[cbase + tid] = pivs[tid];
        order[pivs[tid]] = cbase + tid;
      }
#pragma unroll
      for (int r = 0; r < kR; ++r)
        if (row0 + 8 * r < n) {
          cd* e = E + (size_t)(row0 + 8 * r) * g.ew + t * kW + t4;
#pragma unroll
          for (int q = 0; q < 4; ++q) stcg(e + q * 4, x[r][q]);
        }
    }
    cluster_sync();  // E, the pivots: written before, read after
    if (kG == 1 && s == t) return;  // published: later E reach these rows in the update
    if (tid < kW) {
      const int p = cbase + tid < g.c0 + g.w ? __ldcg(piv + cbase + tid) : -1;
      pivs[tid] = p;
      if (p >= 0) slot[p] = (signed char)tid;
      else  // a partial sub-panel: its missing pivot rows are 0
        for (int k = 0; k < kW * kG; ++k) c1s[tid][k] = cd{0.0, 0.0};
    }
    __syncthreads();
    // columns this E applies to: Q's unless the CTA's sub-panel is done and final
    const int q0 = (kG == 2 && s <= t) ? 4 : 0;
#pragma unroll
    for (int r = 0; r < kR; ++r) {
      const int m = slot[row0 + 8 * r];
      if (m >= 0) {
        used |= 1u << r;
#pragma unroll
        for (int q = 0; q < 4 * kG; ++q) {
          if (q >= q0) {
            c1s[m][q * 4 + t4] = x[r][q];
            x[r][q] = cd{0.0, 0.0};
          }
        }
      }
    }
    __syncthreads();
    if (tid < kW && pivs[tid] >= 0) slot[pivs[tid]] = -1;
#pragma unroll 1
    for (int m0 = 0; m0 < 4; ++m0) {  // 4 complex of K per step
      cd ev[kR];
#pragma unroll
      for (int r = 0; r < kR; ++r)
        ev[r] = ldcg(E + (size_t)min(row0 + 8 * r, n - 1) * g.ew + t * kW + m0 * 4 + t4);
#pragma unroll
      for (int q = 0; q < 4 * kG; ++q) {
        if (kG == 2 && q < q0) continue;
        const cd b = c1s[m0 * 4 + t4][q * 4 + (gq >> 1)];
        const double be = (gq & 1) ? b.y : b.x, bo = (gq & 1) ? b.x : -b.y;
#pragma unroll
        for (int h = 0; h < kR; h += 2) {
          mma64(x[h][q].x, x[h][q].y, x[h + 1][q].x, x[h + 1][q].y, ev[h].x, ev[h + 1].x, be);
          mma64(x[h][q].x, x[h][q].y, x[h + 1][q].x, x[h + 1][q].y, ev[h].y, ev[h + 1].y, bo);
        }
      }
    }
  }

  if constexpr (kG == 2) {
    // every CTA has loaded its columns before the first cluster barrier
#pragma unroll
    for (int r = 0; r < kR; ++r) {
      const int row = row0 + 8 * r;
      if (row >= n) continue;
      const size_t oq = abase + (size_t)row * g.ld + t4;
      const size_t op = abase + (size_t)__ldcg(order + row) * g.ld + t4;
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (q * 4 + t4 < cols) {
          g.P[op + q * 4] = x[r][q + 4];
          g.Q[oq + q * 4] = cd{s * kW + q * 4 + t4 == row ? 1.0 : 0.0, 0.0};
        }
    }
  }
}

// The pivot rows a block's E apply to, over 32 trailing columns of one angle: those of
// sub-panel t as they stand when it is eliminated, C1_t = C[p_t] + sum_{u < t} E_u[p_t]
// C1_u.  (Folding the sub-panels' E into one E of the block instead would need no such
// chain, but its entries grow with the block: 8e-11 instead of 2e-11 of the row maximum
// on the reference's N = 521 case at 0.68 A with sp6.)
// The rows and the E they take (nsub (nsub - 1) / 2 blocks of 16 x 16) are all copied into
// shared memory first: one memory latency instead of one per few k steps.
constexpr int kC1Cols = 32, kC1Str = kC1Cols + 4, kEStr = 20;
static size_t c1_bytes(int nsub) {
  return ((size_t)nsub * kW * kC1Str + (size_t)nsub * (nsub - 1) / 2 * kW * kEStr) * sizeof(cd);
}
__global__ void __launch_bounds__(128) k_gj_c1(const BlockArgs g) {
  const int a = blockIdx.y;
  if (g.flag && !g.flag[a]) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, gq = lane >> 2, t4 = lane & 3;
  const int n = g.n, rows = g.nsub * kW, vc0 = blockIdx.x * kC1Cols;
  cd* c1 = reinterpret_cast<cd*>(smem_raw);  // 16 nsub x kC1Str
  cd* es = c1 + rows * kC1Str;               // block (t, u < t): t (t - 1) / 2 + u, 16 x kEStr
  const int n0 = n - g.c0 - g.w, total = n0 + n;
  const cd* E = g.E + (size_t)a * n * g.ew;
  const cd* Qa = g.Q + (size_t)a * n * g.ld + g.c0 + g.w;
  const cd* Pa = g.P + (size_t)a * n * g.ld;
  const int* piv = g.piv + (size_t)a * n + g.c0;
  {
    const int vc = vc0 + lane;
    const cd* src = vc < n0 ? Qa + vc : Pa + (vc - n0);
#pragma unroll 4
    for (int m = warp; m < rows; m += 4) {
      const bool ok = m < g.w && vc < total;
      cp16(c1 + m * kC1Str + lane, ok ? src + (size_t)piv[m] * g.ld : g.Q, ok);
    }
    for (int t = 1; t < g.nsub; ++t)
#pragma unroll 4
      for (int e = tid; e < t * kW * kW; e += 128) {
        const int u = e / (kW * kW), r = (e / kW) % kW, k = e % kW, m = t * kW + r;
        const bool ok = m < g.w;  // a missing pivot row's result is unused
        cp16(es + ((size_t)(t * (t - 1) / 2 + u) * kW + r) * kEStr + k,
             ok ? E + (size_t)piv[m] * g.ew + u * kW + k : E, ok);
      }
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
  }
  __syncthreads();
  const int cw = warp * 8;  // this warp's columns
  for (int t = 1; t < g.nsub; ++t) {
    cd acc[2][2];  // [row half][4-column group]
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int q = 0; q < 2; ++q)
        acc[h][q] = c1[(t * kW + gq + 8 * h) * kC1Str + cw + q * 4 + t4];
    for (int u = 0; u < t; ++u) {
      const cd* eb = es + ((size_t)(t * (t - 1) / 2 + u) * kW + gq) * kEStr + t4;
#pragma unroll
      for (int k = 0; k < kW; k += 4) {
        const cd e0 = eb[k], e1 = eb[8 * kEStr + k];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const cd b = c1[(u * kW + k + t4) * kC1Str + cw + q * 4 + (gq >> 1)];
          const double be = (gq & 1) ? b.y : b.x, bo = (gq & 1) ? b.x : -b.y;
          mma64(acc[0][q].x, acc[0][q].y, acc[1][q].x, acc[1][q].y, e0.x, e1.x, be);
          mma64(acc[0][q].x, acc[0][q].y, acc[1][q].x, acc[1][q].y, e0.y, e1.y, bo);
        }
      }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int q = 0; q < 2; ++q)
        c1[(t * kW + gq + 8 * h) * kC1Str + cw + q * 4 + t4] = acc[h][q];
    __syncwarp();  // a warp reads only its own columns
  }
  __syncthreads();
  cd* C1 = g.C1 + (size_t)a * g.c1stride;
  if (vc0 + lane < g.ldc)
    for (int m = warp; m < rows; m += 4)
      C1[(size_t)m * g.ldc + vc0 + lane] = c1[m * kC1Str + lane];
}

// Trailing update C = (pivot row of the block ? 0 : C) + E C1, K = 16 S <= 128, where a
// pivot row of sub-panel t takes no E of the sub-panels before t: 64 x 64 complex tiles, 4 warps of 32 x 32 on m16n8k4 FP64 MMAs (k_gj_block's layout: a lane's
// accumulator pair is one complex, so a warp reads and writes whole 64-byte pieces of
// rows), K in chunks of 16 through a 3-stage cp.async ring as the stage product.
// At K = 64 a tile has 16 K clocks of FP64 tensor work for 131 KB of C read and written.
// n = 521, 31 angles, first block: 405 us with a row-tile test at every MMA and the complex
// B values selected in registers (55 % of the FP64 rate), 363 us as it is (61 %).
constexpr int BM = 64, BN = 64, BK = 16, STAGES = 3;
constexpr int ASTR = BK + 4, BSTR = BN + 4;
constexpr int A_TILE = BM * ASTR, B_TILE = BK * BSTR;
constexpr size_t UPD_SMEM = (size_t)STAGES * (A_TILE + B_TILE) * sizeof(cd);

__global__ void __launch_bounds__(128, 2) k_gj_update(const BlockArgs g) {
  const int a = blockIdx.z;
  if (g.flag && !g.flag[a]) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cd* As = reinterpret_cast<cd*>(smem_raw);
  cd* Bs = As + STAGES * A_TILE;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int gq = lane >> 2, t = lane & 3;
  const int wm = (warp >> 1) * 32, wn = (warp & 1) * 32;
  const int n = g.n, bm = blockIdx.y * BM, bn = blockIdx.x * BN;
  const cd* E = g.E + (size_t)a * n * g.ew;
  const cd* C1 = g.C1 + (size_t)a * g.c1stride;
  __shared__ int first[BM];  // the first K chunk a row takes (past the last: rows past n)
  if (tid < BM) {
    int f = g.nsub;
    if (bm + tid < n) {
      const int o = g.order[(size_t)a * n + bm + tid];
      f = (o >= g.c0 && o < g.c0 + g.w) ? (o - g.c0) / kW : 0;
    }
    first[tid] = f;
  }
  __syncthreads();
  const int n0 = n - g.c0 - g.w, total = n0 + n;
  cd* const Qa = g.Q + (size_t)a * n * g.ld + g.c0 + g.w;
  cd* const Pa = g.P + (size_t)a * n * g.ld - n0;
  auto load_stage = [&](int s, int k0) {
    cd* as = As + s * A_TILE;
    cd* bs = Bs + s * B_TILE;
#pragma unroll
    for (int it = 0; it < BM * BK / 128; ++it) {
      const int e = tid + it * 128, r = e / BK, kk = e % BK;
      cp16(as + r * ASTR + kk, E + (size_t)min(bm + r, n - 1) * g.ew + k0 + kk,
           k0 >= first[r] * BK);
    }
#pragma unroll
    for (int it = 0; it < BK * BN / 128; ++it) {
      const int e = tid + it * 128, kk = e / BN, c = e % BN;
      const bool ok = bn + c < g.ldc;
      cp16(bs + kk * BSTR + c, C1 + (size_t)(k0 + kk) * g.ldc + (ok ? bn + c : 0), ok);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  const int nk = g.nsub;
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) {
    if (s < nk) load_stage(s, s * BK);
    else asm volatile("cp.async.commit_group;" ::: "memory");
  }
  // this warp's row tiles with rows below n (none where its columns are past the last)
  const int mlim = bn + wn < total ? min(max(ceil_div(n - bm - wm, 16), 0), 2) : 0;
  const int flip = (gq & 1) ? 0 : (int)0x80000000;
  cd acc[2][2][8];  // [row tile][row half][4-column group]: lane (g, t) column 4 ni + t
  size_t off[2][2];
#pragma unroll
  for (int mi = 0; mi < 2; ++mi)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int r = bm + wm + mi * 16 + gq + 8 * h;
      off[mi][h] = (size_t)min(r, n - 1) * g.ld;
      bool live = false;
      if (r < n) {
        const int o = g.order[(size_t)a * n + r];
        live = !(o >= g.c0 && o < g.c0 + g.w);
      }
#pragma unroll
      for (int ni = 0; ni < 8; ++ni) {
        const int c = bn + wn + ni * 4 + t;
        acc[mi][h][ni] = (live && c < total) ? (c < n0 ? Qa : Pa)[off[mi][h] + c] : cd{0.0, 0.0};
      }
    }
  for (int kt = 0; kt < nk; ++kt) {
    asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
    __syncthreads();
    const int nxt = kt + STAGES - 1;
    if (nxt < nk) load_stage(nxt % STAGES, nxt * BK);
    else asm volatile("cp.async.commit_group;" ::: "memory");
    const cd* as = As + (kt % STAGES) * A_TILE;
    const cd* bs = Bs + (kt % STAGES) * B_TILE;
    // whole row tiles only: a test per MMA would keep the next fragments' loads behind it
    auto chunk = [&](auto tiles) {
      constexpr int kTiles = decltype(tiles)::value;
#pragma unroll
      for (int kk = 0; kk < BK; kk += 4) {
        cd af[kTiles][2];
#pragma unroll
        for (int mi = 0; mi < kTiles; ++mi)
#pragma unroll
          for (int h = 0; h < 2; ++h)
            af[mi][h] = as[(wm + mi * 16 + gq + 8 * h) * ASTR + kk + t];
        // this lane's column of the (re, im) pairs, and its partner with the sign of i^2
        const double* brow = reinterpret_cast<const double*>(bs + (kk + t) * BSTR + wn);
#pragma unroll
        for (int ni = 0; ni < 8; ++ni) {
          const double be = brow[8 * ni + gq], bp = brow[8 * ni + (gq ^ 1)];
          const double bo = __hiloint2double(__double2hiint(bp) ^ flip, __double2loint(bp));
#pragma unroll
          for (int mi = 0; mi < kTiles; ++mi) {
            cd& c0 = acc[mi][0][ni];
            cd& c1 = acc[mi][1][ni];
            mma64(c0.x, c0.y, c1.x, c1.y, af[mi][0].x, af[mi][1].x, be);
          }
#pragma unroll
          for (int mi = 0; mi < kTiles; ++mi) {
            cd& c0 = acc[mi][0][ni];
            cd& c1 = acc[mi][1][ni];
            mma64(c0.x, c0.y, c1.x, c1.y, af[mi][0].y, af[mi][1].y, bo);
          }
        }
      }
    };
    if (mlim == 2) chunk(std::integral_constant<int, 2>{});
    else if (mlim == 1) chunk(std::integral_constant<int, 1>{});
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
  for (int mi = 0; mi < 2; ++mi)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (bm + wm + mi * 16 + gq + 8 * h >= n) continue;
#pragma unroll
      for (int ni = 0; ni < 8; ++ni) {
        const int c = bn + wn + ni * 4 + t;
        if (c < total) (c < n0 ? Qa : Pa)[off[mi][h] + c] = acc[mi][h][ni];
      }
    }
}

// P's rows into pivot order (row r becomes row order[r]) and Q = I, 8 columns per CTA:
// the columns pass through shared memory, so P is permuted in place.
constexpr int kPermCols = 8;
__global__ void __launch_bounds__(256) k_gj_finish(const BlockArgs g) {
  const int a = blockIdx.y;
  if (g.flag && !g.flag[a]) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cd* S = reinterpret_cast<cd*>(smem_raw);
  const int n = g.n, c0 = blockIdx.x * kPermCols, cols = min(kPermCols, n - c0);
  cd* Pa = g.P + (size_t)a * n * g.ld + c0;
  cd* Qa = g.Q + (size_t)a * n * g.ld + c0;
  const int* piv = g.piv + (size_t)a * n;
  for (int e = threadIdx.x; e < n * kPermCols; e += blockDim.x) {
    const int r = e / kPermCols, k = e % kPermCols;
    if (k < cols) {
      S[e] = Pa[(size_t)r * g.ld + k];
      Qa[(size_t)r * g.ld + k] = cd{c0 + k == r ? 1.0 : 0.0, 0.0};
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < n * kPermCols; e += blockDim.x) {
    const int r = e / kPermCols, k = e % kPermCols;
    if (k < cols) Pa[(size_t)r * g.ld + k] = S[piv[r] * kPermCols + k];
  }
}

static bool whole(int n) { return n <= kMaxBlock * kW; }  // one launch

// Sub-panels per block.  More of them means fewer passes over the trailing columns but
// an SM each, idle while another's sub-panel is eliminated, so: six up to 18 angles,
// else four.  Whole elimination at n = 521 (one CTA per SM) with 2 / 4 / 6 / 8 sub-panels
// per block: 1 angle 1.40 / 1.33 / 1.34 / 1.36 ms, 16 angles 3.22 / 2.72 / 2.55 / 2.79, 31
// angles 4.95 / 4.07 / 4.44 / 4.87, 61 angles 8.28 / 7.73 / 7.93 / 8.47 (now 1.22, 2.40,
// 3.75, 7.10; rank-32 updates with physical row swaps and a launch per 16 columns took 4.2,
// 5.9, 6.8, 10.7 ms).  The line holds from 150 to 600 beams, also where an SM takes two
// CTAs: the time with four over that with six, at 16 / 24 / 31 / 61 angles: n = 150 1.02 /
// 1.05 / 0.92 / 0.94, 191 1.05 / 0.90 / 0.94 / 0.86, 250 1.00 / 0.89 / 0.91 / 0.91, 400
// 1.03 / 1.03 / 0.91 / 0.99, 600 1.02 / 0.92 / 0.87 / 0.92 (n = 191, 31 angles: 415 -> 390 us).
static int block_ctas(int nang, int n) {
  const int sub = ceil_div(n, kW);
  if (whole(n)) return sub;
  const int s = nang <= 18 ? 6 : 4;
  return ceil_div(sub, ceil_div(sub, s));  // blocks of equal size
}

template <int kG, int kRT, int kMaxT, int kMinB>
static void launch_block(const BlockArgs& g, int nang, int ctas, cudaStream_t st) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(nang * ctas));
  cfg.blockDim = dim3((unsigned)(32 * ceil_div(g.n, 16 * kRT)));
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)ctas;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, k_gj_block<kG, kRT, kMaxT, kMinB>, g, ctas);
}

}  // namespace gj

namespace {
struct ClusterScratch {
  size_t order, piv, E, C1, total;
  int ew, ldc, rows;
};
ClusterScratch cluster_layout(int nang, int n) {
  ClusterScratch s{};
  const int ctas = gj::block_ctas(nang, n);
  s.ew = gj::kW * ctas;
  s.rows = gj::kW * ctas;
  s.ldc = round_up(2 * n, 4);
  auto up = [](size_t b) { return (b + 255) & ~size_t(255); };
  s.order = 0;
  s.piv = up((size_t)nang * n * sizeof(int));
  s.E = s.piv + up((size_t)nang * n * sizeof(int));
  s.C1 = s.E + up((size_t)nang * n * s.ew * sizeof(cd));
  s.total = s.C1 + (gj::whole(n) ? 0 : up((size_t)nang * s.rows * s.ldc * sizeof(cd)));
  return s;
}
}  // namespace

size_t gj_cluster_scratch_bytes(int nang, int n) { return cluster_layout(nang, n).total + 256; }

int launch_gj_cluster(cd* Q, cd* P, const int* flag, int nang, int n, int ld, void* scratch,
                      unsigned* status, cudaStream_t st) {
  using namespace gj;
  const ClusterScratch L = cluster_layout(nang, n);
  char* base = reinterpret_cast<char*>(scratch);
  BlockArgs g{};
  g.Q = Q;
  g.P = P;
  g.flag = flag;
  g.n = n;
  g.ld = ld;
  g.order = reinterpret_cast<int*>(base + L.order);
  g.piv = reinterpret_cast<int*>(base + L.piv);
  g.E = reinterpret_cast<cd*>(base + L.E);
  g.ew = L.ew;
  g.C1 = reinterpret_cast<cd*>(base + L.C1);
  g.ldc = L.ldc;
  g.c1stride = (long long)L.rows * L.ldc;
  g.status = status;
  const int ctas = block_ctas(nang, n);
  if (whole(n)) {
    g.c0 = 0;
    g.w = n;
    g.nsub = ctas;
    if (n <= 96) launch_block<2, 1, 192, 3>(g, nang, ctas, st);
    else launch_block<2, 1, 256, 2>(g, nang, ctas, st);
    return 1;
  }
  static SmemOptIn upd, fin, cone;
  cone.ensure((const void*)k_gj_c1, c1_bytes(kMaxBlock));
  upd.ensure((const void*)k_gj_update, UPD_SMEM);
  const size_t fin_smem = (size_t)n * kPermCols * sizeof(cd);
  fin.ensure((const void*)k_gj_finish, fin_smem);
  int launches = 0;
  for (int c0 = 0; c0 < n; c0 += ctas * kW) {
    g.c0 = c0;
    g.w = std::min(ctas * kW, n - c0);
    g.nsub = ceil_div(g.w, kW);
    g.ldc = round_up(2 * n - c0 - g.w, 4);
    // rows of a warp: 16 up to 128 beams (above; a cluster shares its SMs with others), 32 up
    // to 256, 48 up to 576 (at n = 521 eleven warps of 168 registers; 17 warps of 32 rows
    // leave 96 registers and an uneven fifth warp on one scheduler)
    if (n <= 256) launch_block<1, 2, 256, 2>(g, nang, g.nsub, st);
    else if (n <= 576) launch_block<1, 3, 384, 1>(g, nang, g.nsub, st);
    else launch_block<1, 4, 320, 1>(g, nang, g.nsub, st);
    const int total = 2 * n - c0 - g.w;
    for (int a0 = 0; a0 < nang; a0 += 65535) {  // angles on z
      BlockArgs h = g;
      h.Q += (size_t)a0 * n * ld;
      h.P += (size_t)a0 * n * ld;
      if (h.flag) h.flag += a0;
      h.order += (size_t)a0 * n;
      h.piv += (size_t)a0 * n;
      h.E += (size_t)a0 * n * g.ew;
      h.C1 += (size_t)a0 * g.c1stride;
      const int na = std::min(nang - a0, 65535);
      k_gj_c1<<<dim3(ceil_div(total, kC1Cols), na), 128, c1_bytes(g.nsub), st>>>(h);
      k_gj_update<<<dim3(ceil_div(total, BN), ceil_div(n, BM), na), 128, UPD_SMEM, st>>>(h);
      launches += 2;
    }
    ++launches;
  }
  for (int a0 = 0; a0 < nang; a0 += 65535) {
    BlockArgs h = g;
    h.Q += (size_t)a0 * n * ld;
    h.P += (size_t)a0 * n * ld;
    if (h.flag) h.flag += a0;
    h.piv += (size_t)a0 * n;
    k_gj_finish<<<dim3(ceil_div(n, kPermCols), std::min(nang - a0, 65535)), 256, fin_smem, st>>>(h);
    ++launches;
  }
  return launches;
}

// ============================================================ Gershgorin estimate
// cond_est per angle (matcomp.f90:498-528): a cluster of `parts` CTAs per angle sums
// |Q(i, j)| of its share of the rows per column; CTA 0 adds the shares over the
// cluster's shared memory and takes the extremes.  (One CTA per angle walked all n rows
// serially: 230 us at n = 521.)
__global__ void __launch_bounds__(kGjClusterMaxRows)
    k_cond_est(const cd* __restrict__ Q, int n, int ld, int force, int parts,
               int* __restrict__ flag, double* __restrict__ dval) {
  const int a = blockIdx.x / parts, part = blockIdx.x - a * parts;
  extern __shared__ double csum[];  // n column sums of this share
  __shared__ double smn[32], smx[32];
  const cd* A = Q + (size_t)a * n * ld;
  const int r0 = (int)((long long)n * part / parts), r1 = (int)((long long)n * (part + 1) / parts);
  for (int j = threadIdx.x; j < n; j += blockDim.x) {
    double t = 0.0;
#pragma unroll 8
    for (int i = r0; i < r1; ++i) {
      const cd v = A[(size_t)i * ld + j];
      t += (i != j) ? sqrt(v.x * v.x + v.y * v.y) : 0.0;
    }
    csum[j] = t;
  }
  gj::cluster_sync();
  if (part == 0) {
    double mn = INFINITY, mx = 0.0;
    for (int j = threadIdx.x; j < n; j += blockDim.x) {
      double t = csum[j];
      for (int q = 1; q < parts; ++q) {
        unsigned remote;
        const unsigned local = (unsigned)__cvta_generic_to_shared(&csum[j]);
        double v;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(q));
        asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(remote) : "memory");
        t += v;
      }
      const cd dj = A[(size_t)j * ld + j];
      const double ad = hypot(dj.x, dj.y);
      mn = fmin(mn, ad - t);
      mx = fmax(mx, ad + t);
    }
    for (int o = 16; o > 0; o >>= 1) {
      mn = fmin(mn, __shfl_xor_sync(0xffffffffu, mn, o));
      mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) {
      smn[w] = mn;
      smx[w] = mx;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      const int nw = blockDim.x >> 5;
      for (int i = 1; i < nw; ++i) {
        mn = fmin(mn, smn[i]);
        mx = fmax(mx, smx[i]);
      }
      const cd a11 = A[0];
      mx = fmax(mx, hypot(a11.x, a11.y));
      const double d = (mn < 0.0) ? 1e100 : mx / mn;
      if (dval) dval[a] = d;
      flag[a] = (force || d > 1e3) ? 1 : 0;
    }
  }
  gj::cluster_sync();  // the shares stay until CTA 0 has read them
}

void launch_cond_est(const cd* Q, int nang, int n, int ld, int force, int* flag, double* dval,
                     cudaStream_t st) {
  const int parts = n <= 32 ? 1 : n <= 64 ? 2 : n <= 128 ? 4 : 8;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(nang * parts));
  cfg.blockDim = dim3((unsigned)std::min(round_up(n, 32), kGjClusterMaxRows));
  cfg.dynamicSmemBytes = (size_t)n * sizeof(double);
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)parts;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, k_cond_est, Q, n, ld, force, parts, flag, dval);
}

}  // namespace trhepd
