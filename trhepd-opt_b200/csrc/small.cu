// Fused small-beam RKN integration (hp_int_spa, sim-trhepd-rheed/src/surf_prkn.f90:278-330).
//
// For N <= 64 beams a whole angle fits one SM, so the solve is one launch, one CTA of
// four warps per angle, through all s*ns stages:
//   * the stage columns of the potential table (nv entries) are copied into shared memory
//     three stages ahead; the product reads the matrix entries
//     straight from it (V(k, j) is an entry of pair(k, j), conjugated or not: the
//     fragments' entry numbers stay packed in registers), so no stage matrix is formed;
//   * the product Q V runs on the FP64 tensor cores (mma.sync m16n8k4 on (re, im) column
//     pairs): a warp owns whole 16-row tiles times every WC-th group of four columns, so
//     the four schedulers get equal shares, and a lane holds whole complex elements;
//   * the epilogue is the RKN update of the stacked path: P += cb (Q V + Q o D_a),
//     Q <- Q + ca P; P stays in registers (shared memory beyond 48 beams); Q = I enters
//     as data;
//   * at the end of a slice the renormalisation (policy 0: Gershgorin estimate
//     cond_est, matcomp.f90:498-528, > 1e3; policy 1: every `interval` slices;
//     always on the last) is a Gauss-Jordan elimination of [Q | P] (matAbdivB,
//     matcomp.f90:53-69) with implicit pivoting in 16-column sub-panels, as renorm.cu:
//     the panel's rows in registers, its E in the panel's own columns of Q, the other
//     columns updated by MMAs.
// The stage order, merged half kicks and coefficients are those of run_rkn.  What bounds
// it: at N = 47 the FP64 pipe (6.9 K clocks a product), at N = 23 the chain of barriers,
// shared-memory latency and 1.2 K clocks of MMAs.
// One launch can carry several problems (their own tables, beam counts up to
// the launch's limit, slice counts and renormalisation intervals): each CTA finds
// its problem in the launch parameters.
#include <cuda_runtime.h>

#include <algorithm>
#include <stdexcept>

#include "small.h"
#include "launch_attr.h"

namespace trhepd {
namespace fused {

constexpr int kThreads = 128;
constexpr int kTabBufs = 4;  // table columns in flight where shared memory allows
constexpr int kMaxEntries = (1 << 14) - 1;  // the fragment codes have 15 bits of position

// RT row tiles; GW column groups per warp.  kRk4: the classical RK4 steps of rk4_int
// (surf_rk.f90:27-91) instead of the RKN kicks: Q, P, the stage point's Q and the two
// weighted sums in shared memory (elements of them touched by their own lane only), the
// stage point's P in registers.
template <int RT, int GW, bool kRk4>
struct Cfg {
  static constexpr int NP = 16 * RT;
  static constexpr int WC = RT == 2 ? 2 : 4;        // warps along the columns
  static constexpr int WR = 4 / WC;                 // and along the row tiles
  static constexpr int TW = RT / WR;                // row tiles per warp
  static constexpr int KS = 4 * RT;                 // k steps of a product
  static constexpr bool PREG = RT <= 3 && !kRk4;    // P in registers
  static constexpr int QB = RT <= 2 && !kRk4 ? 2 : 1;  // Q buffers (one barrier per stage less)
  static constexpr int STR = NP + 4;                // 4 mod 8 complex: conflict-free fragments
  static constexpr int MINB = kRk4 ? (RT <= 2 ? 2 : 1) : RT <= 2 ? 3 : RT == 3 ? 2 : 1;
  // complex values of Q, P, the RK4 arrays or else the pivot rows (which share the first
  // RK4 sum: it is dead at the end of a slice), and the fragment codes (8 bytes per lane and
  // k step)
  static constexpr size_t extra = kRk4 ? (size_t)3 * NP * STR : (size_t)16 * STR;
  // beyond 48 beams a single column buffer also holds the pivot rows
  static constexpr bool SHARE = RT > 3 && !kRk4;
  static constexpr size_t elems =
      (size_t)(QB + (PREG ? 0 : 1)) * NP * STR + extra + KS * kThreads / 2;
};

__device__ __forceinline__ unsigned smem_addr(const void* p) {
  return (unsigned)__cvta_generic_to_shared(p);
}
// Waits for a phase of a barrier, two seconds at most.
__device__ __forceinline__ bool wait_parity(const unsigned long long* bar, int parity) {
  unsigned long long t0 = 0;
  for (unsigned it = 0;; ++it) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    if (ok) return true;
    if ((it & 255) == 255) {
      unsigned long long t;
      asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
      if (t0 == 0) t0 = t;
      else if (t - t0 > 2000000000ull) return false;
    }
  }
}

__device__ __forceinline__ void fmma(cd& c0, cd& c1, double a0, double a1, double b0) {
  asm volatile(
      "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, "
      "{%0,%1,%2,%3};\n"
      : "+d"(c0.x), "+d"(c0.y), "+d"(c1.x), "+d"(c1.y)
      : "d"(a0), "d"(a1), "d"(b0));
}

template <int RT, int GW, bool kRk4>
__global__ void __launch_bounds__(kThreads, Cfg<RT, GW, kRk4>::MINB)
    k_fused_rkn(const __grid_constant__ FusedLaunch L, int nbuf, int tab_stride) {
  using C = Cfg<RT, GW, kRk4>;
  constexpr int NP = C::NP, STR = C::STR, TW = C::TW;
  // this CTA's problem: the last whose first CTA is <= blockIdx.x
  int pi = 0;
  for (int q = 1; q < L.nprob; ++q)
    if (L.p[q].first_cta <= (int)blockIdx.x) pi = q;
  const FusedProblem& a = L.p[pi];
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cd* Qs = reinterpret_cast<cd*>(smem_raw);             // the current Q
  cd* Qo = Qs + (C::QB - 1) * NP * STR;                 // the other (the same for QB = 1)
  cd* const Ps = Qs + C::QB * NP * STR;                 // PREG = false only
  cd* const SQ = Ps + (C::PREG ? 0 : NP * STR);         // kRk4 only, as the next two
  cd* const SP = SQ + NP * STR;
  cd* const Qt = SP + NP * STR;
  const bool one = C::SHARE && nbuf == 1;  // the pivot rows share the only column buffer
  cd* const codes_at = SQ + (one ? 0 : C::extra);
  uint2* const codes = reinterpret_cast<uint2*>(codes_at);  // [KS][kThreads]
  cd* const tab = codes_at + C::KS * kThreads / 2;          // [nbuf][tab_stride]
  cd* const c1s = one ? tab : SQ;                           // 16 pivot rows
  __shared__ double csum[kThreads];
  __shared__ double red_d[2][4];
  __shared__ unsigned keys[2][32];
  __shared__ cd urow[2][16];
  __shared__ int order[NP], piv[NP], renorm_sh;
  __shared__ signed char slot[NP];
  __shared__ __align__(8) unsigned long long bars[kTabBufs];
  const unsigned full = 0xffffffffu;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int gq = lane >> 2, t4 = lane & 3;
  const int wr = warp / C::WC, wc = warp % C::WC;
  const int n = a.n, ld = a.ld, nv = a.nv, ang = blockIdx.x - a.first_cta;
  const int row0 = wr * TW * 16 + gq;                   // rows row0 + 16 i + 8 h
  auto col = [&](int j) { return 4 * (j * C::WC + wc) + t4; };
  cd* const Qg = a.Q + (size_t)ang * n * ld;
  cd* const Pg = a.P + (size_t)ang * n * ld;

  cd preg[C::PREG ? TW * 2 * GW : 1];
  auto P = [&](int i, int h, int j) -> cd& {
    if constexpr (C::PREG) return preg[(i * 2 + h) * GW + j];
    else return Ps[(row0 + 16 * i + 8 * h) * STR + col(j)];
  };
  for (int e = tid; e < NP * STR; e += kThreads) {
    const int i = e / STR, j = e % STR;
    const bool ok = i < n && j < n;
    Qs[e] = ok ? Qg[(size_t)i * ld + j] : cd{0.0, 0.0};
    if (C::QB == 2) Qo[e] = cd{0.0, 0.0};
    if (kRk4) Qt[e] = cd{0.0, 0.0};
  }
  double dreg[GW];
#pragma unroll
  for (int j = 0; j < GW; ++j) {
    dreg[j] = col(j) < n ? a.D[(size_t)ang * ld + col(j)].x : 0.0;  // D = -gamma^2 is real
#pragma unroll
    for (int i = 0; i < TW; ++i)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int r = row0 + 16 * i + 8 * h;
        P(i, h, j) = (r < n && col(j) < n) ? Pg[(size_t)r * ld + col(j)] : cd{0.0, 0.0};
      }
  }
  // The B fragments' matrix entries: lane (g, t) of k step ks and group j takes V(4 ks + t,
  // 4 cg + g / 2), as -V: an upper entry (k < j, and the diagonal's entry 0) is conj(u), a
  // lower one w, so only the imaginary part can change sign.  Even lanes use (re, -im) as
  // the two k rows, odd ones (im, re): 15 bits of position (16-byte words of the table
  // column; the zero entry is nv) and the sign.
  for (int ks = 0; ks < C::KS; ++ks) {
    unsigned code[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int k = 4 * ks + t4, c = 4 * (j * C::WC + wc) + (gq >> 1);
      unsigned pos = 2 * nv, lower = 0;
      if (j < GW && k < n && c < n) {
        lower = k > c;
        pos = 2 * (k == c ? 0 : a.pair[k * n + c]) + lower;
      }
      code[j] = pos | ((gq & 1) ? 1u - lower : lower) << 15;
    }
    codes[ks * kThreads + tid] = make_uint2(code[0] | code[1] << 16, code[2] | code[3] << 16);
  }
  const int ng = (n + 3) / 4;  // column groups (and k steps) that hold beams
  for (int b = 0; b < nbuf; ++b)
    if (tid < 2) tab[b * tab_stride + 2 * nv + tid] = cd{0.0, 0.0};
  const int s = L.s, ns = a.ns;
  const double dz = a.dz;
  // The next column of the table into the next buffer: one bulk copy by thread 0 (16-byte
  // copies by every thread took 500 clocks of a stage).  Every issued column is consumed.
  const int ncol = s * ns + 1;
  if (tid == 0) {
    for (int b = 0; b < nbuf; ++b)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&bars[b])) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  int issued = 0, in = 0;           // columns on their way or consumed (thread 0)
  int consumed = 0, out = 0, parity = 0;
  bool dead = false;                // a copy that never came: reported, not waited for again
  auto fetch = [&]() {
    if (tid == 0 && issued < ncol && !dead) {
      const unsigned bar = smem_addr(&bars[in]), bytes = 32u * nv;
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
                   : "memory");
      asm volatile(
          "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
          ::"r"(smem_addr(tab + in * tab_stride)), "l"(a.table + (size_t)issued * nv), "r"(bytes),
          "r"(bar)
          : "memory");
      in = in + 1 < nbuf ? in + 1 : 0;
      ++issued;
    }
  };
  auto arrived = [&]() {  // waits for the next column
    if (!dead && !wait_parity(&bars[out], parity)) {
      dead = true;
      atomicOr(a.status, kStatusTimeout);
    }
    ++consumed;
    if (++out == nbuf) {
      out = 0;
      parity ^= 1;
    }
  };
  for (int c = 0; c < max(nbuf - 1, 1); ++c) fetch();
  cd acc[TW][2][GW];
  // acc = -Qin V with the column at tc
  auto product = [&](const cd* Qin, const cd* tc) {
#pragma unroll
    for (int i = 0; i < TW; ++i)
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int j = 0; j < GW; ++j) acc[i][h][j] = cd{0.0, 0.0};
    // two k steps a turn, each one's fragments loaded before the other's MMAs; steps past
    // the beams meet zero entries
    cd af[2][TW][2], bf[2][GW];
    auto load = [&](int ks, cd (&x)[TW][2], cd (&y)[GW]) {
      const uint2 code = codes[ks * kThreads + tid];
#pragma unroll
      for (int i = 0; i < TW; ++i)
#pragma unroll
        for (int h = 0; h < 2; ++h) x[i][h] = Qin[(row0 + 16 * i + 8 * h) * STR + 4 * ks + t4];
#pragma unroll
      for (int j = 0; j < GW; ++j) {
        const unsigned w = j < 2 ? code.x : code.y, cj = (j & 1) ? w >> 16 : w & 0xffffu;
        const cd b = tc[cj & 0x7fffu];
        const double im = __hiloint2double(__double2hiint(b.y) ^ (int)((cj & 0x8000u) << 16),
                                           __double2loint(b.y));
        y[j] = (gq & 1) ? cd{im, b.x} : cd{b.x, im};
      }
    };
    auto mma = [&](const cd (&x)[TW][2], const cd (&y)[GW]) {
#pragma unroll
      for (int j = 0; j < GW; ++j)
#pragma unroll
        for (int i = 0; i < TW; ++i)
          fmma(acc[i][0][j], acc[i][1][j], x[i][0].x, x[i][1].x, y[j].x);
#pragma unroll
      for (int j = 0; j < GW; ++j)
#pragma unroll
        for (int i = 0; i < TW; ++i)
          fmma(acc[i][0][j], acc[i][1][j], x[i][0].y, x[i][1].y, y[j].y);
    };
    load(0, af[0], bf[0]);
#pragma unroll 1
    for (int ks = 0; ks < ng; ks += 2) {
      load(ks + 1, af[1], bf[1]);
      mma(af[0], bf[0]);
      load(min(ks + 2, C::KS - 1), af[0], bf[0]);
      mma(af[1], bf[1]);
    }
  };
  // P += cb (Q V + Q o D), Q <- Q + ca P with the next table column; ends without a barrier.
  // hold: an elimination may follow, a column that shares its buffer is fetched after it.
  auto stage = [&](double cb, double ca, bool hold) {
    const cd* tc = tab + out * tab_stride;
    arrived();
    __syncthreads();  // Q is there too
    if (nbuf > 1) fetch();
    product(Qs, tc);
    if (C::QB == 1 || nbuf == 1) __syncthreads();  // every read of Q and the column done
    if (nbuf == 1 && !(one && hold)) fetch();
#pragma unroll
    for (int i = 0; i < TW; ++i)
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int j = 0; j < GW; ++j) {
          const int o = (row0 + 16 * i + 8 * h) * STR + col(j);
          const cd q = Qs[o], z = acc[i][h][j];  // z = -Q V
          cd p = P(i, h, j);
          p = cd{fma(cb, fma(q.x, dreg[j], -z.x), p.x), fma(cb, fma(q.y, dreg[j], -z.y), p.y)};
          P(i, h, j) = p;
          Qo[o] = cd{fma(ca, p.x, q.x), fma(ca, p.y, q.y)};
        }
    if (C::QB == 2) {
      cd* const tmp = Qs;
      Qs = Qo;
      Qo = tmp;
    }
  };
  // Gershgorin estimate of Q (cond_est) > 1e3
  auto needs_renorm = [&]() -> bool {
    constexpr int parts = kThreads / NP;
    const int j = tid % NP, part = tid / NP;
    __syncthreads();
    double t = 0.0;
    if (part < parts && j < n)
      for (int i = part; i < n; i += parts)
        if (i != j) {
          const cd v = Qs[i * STR + j];
          t += sqrt(v.x * v.x + v.y * v.y);
        }
    csum[tid] = t;
    __syncthreads();
    double mn = INFINITY, mx = 0.0;
    if (tid < n) {
      for (int q = 1; q < parts; ++q) t += csum[q * NP + tid];
      const cd dj = Qs[tid * STR + tid];
      const double ad = hypot(dj.x, dj.y);
      mn = ad - t;
      mx = ad + t;
    }
    for (int o = 16; o > 0; o >>= 1) {
      mn = fmin(mn, __shfl_xor_sync(full, mn, o));
      mx = fmax(mx, __shfl_xor_sync(full, mx, o));
    }
    if (lane == 0) {
      red_d[0][warp] = mn;
      red_d[1][warp] = mx;
    }
    __syncthreads();
    if (tid == 0) {
      for (int w = 1; w < 4; ++w) {
        mn = fmin(mn, red_d[0][w]);
        mx = fmax(mx, red_d[1][w]);
      }
      const cd a11 = Qs[0];
      mx = fmax(mx, hypot(a11.x, a11.y));
      const double d = (mn < 0.0) ? 1e100 : mx / mn;
      renorm_sh = d > 1e3;
    }
    __syncthreads();
    return renorm_sh != 0;
  };
  // [Q | P] -> [I | Q^{-1} P]
  auto gauss_jordan = [&]() {
    for (int e = tid; e < NP; e += kThreads) slot[e] = -1;
    if (tid < 64) keys[tid >> 5][tid & 31] = 0;
    unsigned used = 0;  // rows warp * 16 + gq (+ 8) of the panel: pivots before, or past n
    const int prow = warp * 16 + gq;
    if (prow >= n) used |= 1u;
    if (prow + 8 >= n) used |= 2u;
    __syncthreads();
    for (int t = 0; 16 * t < n; ++t) {
      const int cols = min(16, n - 16 * t);
      cd x[2][4];
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int q = 0; q < 4; ++q)
          x[h][q] = warp < RT ? Qs[(prow + 8 * h) * STR + 16 * t + 4 * q + t4] : cd{0.0, 0.0};
#pragma unroll
      for (int q = 0; q < 4; ++q) {
#pragma unroll 1
        for (int tj = 0; tj < 4; ++tj) {
          const int jj = 4 * q + tj, kb = jj & 1;
          if (jj >= cols) break;
          unsigned key = 0;  // see renorm.cu
          if (t4 == tj) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const unsigned hi = (unsigned)__double2hiint(cabs1(x[h][q]));
              const unsigned k = ((hi << 1) & ~1023u) | (unsigned)(1023 - (prow + 8 * h));
              if (!((used >> h) & 1u)) key = max(key, k);
            }
          }
          key = __reduce_max_sync(full, key);
          if (lane == 0) keys[kb][warp] = key;
          __syncthreads();
          const int p = 1023 - (int)(max(max(keys[kb][0], keys[kb][1]),
                                         max(keys[kb][2], keys[kb][3])) & 1023u);
          const bool holder = warp == (p >> 4) && gq == (p & 7);
          const int ph = (p >> 3) & 1;
          if (holder) {
#pragma unroll
            for (int h = 0; h < 2; ++h)
              if (h == ph) {
#pragma unroll
                for (int k = 0; k < 4; ++k) urow[kb][k * 4 + t4] = x[h][k];
                used |= 1u << h;
                if (t4 == tj) {
                  piv[16 * t + jj] = p;
                  order[p] = 16 * t + jj;
                  slot[p] = (signed char)jj;
                  if (x[h][q].x == 0.0 && x[h][q].y == 0.0) atomicOr(a.status, kStatusZeroPivot);
                }
              }
          }
          __syncthreads();
          const cd d = urow[kb][jj];
          cd u[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) u[k] = urow[kb][k * 4 + t4];
          const cd rc = crecip(d);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const cd f = cd{__shfl_sync(full, x[h][q].x, tj, 4),
                            __shfl_sync(full, x[h][q].y, tj, 4)} * rc;
#pragma unroll
            for (int k = 0; k < 4; ++k) x[h][k] = cfms(f, u[k], x[h][k]);
            if (t4 == tj) x[h][q] = -f;
          }
          if (holder) {  // the pivot row is scaled instead
#pragma unroll
            for (int h = 0; h < 2; ++h)
              if (h == ph) {
#pragma unroll
                for (int k = 0; k < 4; ++k) x[h][k] = u[k] * rc;
                if (t4 == tj) x[h][q] = rc;
              }
          }
          __syncwarp();
        }
      }
      if (warp < RT) {  // E, in the panel's columns
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int q = 0; q < 4; ++q) Qs[(prow + 8 * h) * STR + 16 * t + 4 * q + t4] = x[h][q];
      }
      __syncthreads();
      // the other columns: Q's right of the panel, then P's; 16 t + 16 .. of Q first
#pragma unroll 1
      for (int pass = 0; pass < 2; ++pass) {
        const int jmin = pass == 0 ? 16 * t + 16 : 0;  // first column
        if (jmin >= n) continue;
#pragma unroll
        for (int i = 0; i < TW; ++i)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int r = row0 + 16 * i + 8 * h, m = slot[r];
            if (m >= 0) {
#pragma unroll
              for (int j = 0; j < GW; ++j)
                if (4 * (j * C::WC + wc) >= jmin) {
                  cd& v = pass == 0 ? Qs[r * STR + col(j)] : P(i, h, j);
                  c1s[m * STR + col(j)] = v;
                  v = cd{0.0, 0.0};
                }
            }
          }
        if (cols < 16)
          for (int e = tid; e < (16 - cols) * STR; e += kThreads)
            c1s[cols * STR + e] = cd{0.0, 0.0};
        __syncthreads();
#pragma unroll
        for (int j = 0; j < GW; ++j) {
          const int cg = j * C::WC + wc;
          if (4 * cg < jmin || cg >= ng) continue;
          cd v[TW][2];
#pragma unroll
          for (int i = 0; i < TW; ++i)
#pragma unroll
            for (int h = 0; h < 2; ++h)
              v[i][h] = pass == 0 ? Qs[(row0 + 16 * i + 8 * h) * STR + col(j)] : P(i, h, j);
#pragma unroll
          for (int m0 = 0; m0 < 4; ++m0) {
            const cd b = c1s[(4 * m0 + t4) * STR + 4 * cg + (gq >> 1)];
            const double be = (gq & 1) ? b.y : b.x, bo = (gq & 1) ? b.x : -b.y;
#pragma unroll
            for (int i = 0; i < TW; ++i) {
              const cd e0 = Qs[(row0 + 16 * i) * STR + 16 * t + 4 * m0 + t4];
              const cd e1 = Qs[(row0 + 16 * i + 8) * STR + 16 * t + 4 * m0 + t4];
              fmma(v[i][0], v[i][1], e0.x, e1.x, be);
              fmma(v[i][0], v[i][1], e0.y, e1.y, bo);
            }
          }
#pragma unroll
          for (int i = 0; i < TW; ++i)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              if (pass == 0) Qs[(row0 + 16 * i + 8 * h) * STR + col(j)] = v[i][h];
              else P(i, h, j) = v[i][h];
            }
        }
        __syncthreads();  // the pivot rows' buffer, Q's next panel
      }
      if (tid < cols) slot[piv[16 * t + tid]] = -1;
      __syncthreads();
    }
    // P's rows into pivot order, through Q's buffer; Q = I
#pragma unroll
    for (int i = 0; i < TW; ++i)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int r = row0 + 16 * i + 8 * h;
        if (r < n) {
#pragma unroll
          for (int j = 0; j < GW; ++j) Qs[order[r] * STR + col(j)] = P(i, h, j);
        }
      }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < TW; ++i)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int r = row0 + 16 * i + 8 * h;
#pragma unroll
        for (int j = 0; j < GW; ++j) {
          const int o = r * STR + col(j);
          if (r < n) P(i, h, j) = Qs[o];
          Qs[o] = cd{r < n && r == col(j) ? 1.0 : 0.0, 0.0};
        }
      }
  };

  auto end_of_slice = [&](int l) {
    bool renorm = l == ns;
    if (!renorm) renorm = (L.policy == 0) ? needs_renorm() : (l % a.interval) == 0;
    if (renorm) {
      __syncthreads();
      gauss_jordan();
    }
    if (one) {
      if (renorm) {  // the pivot rows may have passed over the zero entry
        if (tid < 2) tab[2 * nv + tid] = cd{0.0, 0.0};
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // before the copy's writes
        __syncthreads();
      }
      fetch();
    }
  };
  if constexpr (kRk4) {
    // stage j: weight of k_j in the sum, step to the next stage point; the middle column
    // serves two stages, the last one the next slice's first
    cd pt[TW * 2 * GW];
    const cd* tc = nullptr;
    for (int l = 1; l <= ns; ++l) {
#pragma unroll 1
      for (int st = 0; st < 4; ++st) {
        const double w = (st == 1 || st == 2) ? 2.0 : 1.0, step = st < 2 ? 0.5 * dz : dz;
        const bool next = (st & 1) || (st == 0 && l == 1);
        if (next) {
          tc = tab + out * tab_stride;
          arrived();
        }
        __syncthreads();  // the stage point is there
        if (next) fetch();
        const cd* Qin = st == 0 ? Qs : Qt;
        product(Qin, tc);
        __syncthreads();  // every read of the stage point done
#pragma unroll
        for (int i = 0; i < TW; ++i)
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int j = 0; j < GW; ++j) {
              const int o = (row0 + 16 * i + 8 * h) * STR + col(j);
              cd& ps = pt[(i * 2 + h) * GW + j];
              const cd q = Qin[o], z = acc[i][h][j], p0 = Ps[o];  // z = -Q V
              const cd kp = cd{fma(q.x, dreg[j], -z.x), fma(q.y, dreg[j], -z.y)};
              const cd kq = st == 0 ? p0 : ps;
              cd sq = kq, sp = kp;
              if (st > 0) {
                sq = SQ[o] + w * kq;
                sp = SP[o] + w * kp;
              }
              if (st < 3) {
                SQ[o] = sq;
                SP[o] = sp;
                Qt[o] = Qs[o] + step * kq;
                ps = p0 + step * kp;
              } else {
                Qs[o] = Qs[o] + (dz / 6) * sq;
                Ps[o] = p0 + (dz / 6) * sp;
              }
            }
      }
      end_of_slice(l);
    }
  } else {
    for (int l = 1; l <= ns; ++l) {
      for (int k = 1; k <= s; ++k) {
        // k == 1 merges the end-of-slice half kick of slice l-1 with the first kick
        const double cb = (k == 1) ? (l == 1 ? 1.0 : 2.0) * L.bab[0] * dz : L.bab[2 * k - 2] * dz;
        stage(cb, L.bab[2 * k - 1] * dz, k == s);
      }
      end_of_slice(l);
    }
    // final half kick with Q = I: P += b1 dz M(end)
    stage(L.bab[0] * dz, 0.0, false);
  }
  if (tid == 0 && dead)  // copies still on their way (as long as they may take)
    while (consumed < issued) {
      wait_parity(&bars[out], parity);
      ++consumed;
      if (++out == nbuf) {
        out = 0;
        parity ^= 1;
      }
    }
  __syncthreads();
  for (int e = tid; e < n * n; e += kThreads) {
    const int i = e / n, j = e % n;
    Qg[(size_t)i * ld + j] = Qs[i * STR + j];
  }
#pragma unroll
  for (int i = 0; i < TW; ++i)
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int j = 0; j < GW; ++j) {
        const int r = row0 + 16 * i + 8 * h;
        if (r < n && col(j) < n) Pg[(size_t)r * ld + col(j)] = P(i, h, j);
      }
}

// Shared memory of a launch: four column buffers where they leave the CTAs per SM the
// registers allow, else two or one (a column's copy takes longer than a stage of a small
// problem).  A single buffer is longer than the 16 pivot rows that share it: so every set
// of 64 beams fits (2017 entries, 31 angles: 51 ms; 156 with a launch per stage, 95 with
// gathered matrices in place of the table column).
template <int RT, int GW, bool kRk4>
constexpr int buffers(int stride, size_t& smem) {
  using C = Cfg<RT, GW, kRk4>;
  auto bytes = [&](int b) {
    return (C::elems - (b == 1 && C::SHARE ? C::extra : 0) + (size_t)b * stride) * sizeof(cd);
  };
  int nbuf = bytes(kTabBufs) <= size_t(227 * 1024) / C::MINB - 4096 ? kTabBufs : 2;
  if (bytes(nbuf) > 224 * 1024) nbuf = 1;
  smem = bytes(nbuf);
  return smem <= 224 * 1024 ? nbuf : 0;
}
// Whether nv table entries a column fit; RK4 keeps a column through two stages.
template <int RT, int GW, bool kRk4>
constexpr bool fits(int nv) {
  size_t smem = 0;
  return nv >= 1 && nv <= kMaxEntries &&
         buffers<RT, GW, kRk4>(2 * (nv + 1), smem) >= (kRk4 ? 2 : 1);
}
// the limits small.h states
static_assert(fits<3, 3, false>(48 * 47 / 2 + 1));
static_assert(fits<4, 4, false>(2303) && !fits<4, 4, false>(2304));
static_assert(fits<3, 3, true>(271) && !fits<3, 3, true>(272));

// A launch that fits.
template <int RT, int GW, bool kRk4 = false>
void launch(const FusedLaunch& L, int nvmax, cudaStream_t st) {
  static SmemOptIn attr;
  const int stride = 2 * (nvmax + 1);
  size_t smem = 0;
  const int nbuf = buffers<RT, GW, kRk4>(stride, smem);
  attr.ensure((const void*)k_fused_rkn<RT, GW, kRk4>, smem);
  k_fused_rkn<RT, GW, kRk4><<<L.total_ctas, kThreads, smem, st>>>(L, nbuf, stride);
}

}  // namespace fused

namespace {
// Checks a launch; returns the largest beam and entry counts.
void check(const FusedLaunch& L, int& nmax, int& nvmax) {
  if (L.nprob < 1 || L.nprob > kFusedMaxProblems || L.s < 1 || L.s > 11)
    throw std::invalid_argument("fused integration: bad launch");
  int ctas = 0;
  nmax = nvmax = 0;
  for (int q = 0; q < L.nprob; ++q) {
    const FusedProblem& a = L.p[q];
    if (a.n < 2 || a.n > kFusedMaxBeams || a.ns < 1 || a.interval < 1 || a.nang < 1 ||
        a.first_cta != ctas || a.nv < 1)
      throw std::invalid_argument("fused integration: unsupported problem");
    ctas += a.nang;
    nmax = std::max(nmax, a.n);
    nvmax = std::max(nvmax, a.nv);
  }
  if (ctas != L.total_ctas) throw std::invalid_argument("fused integration: CTA count");
}
}  // namespace

bool fused_rkn_fits(int n, int nv) {
  return n >= 2 && n <= kFusedMaxBeams &&
         (n <= 16   ? fused::fits<1, 1, false>(nv)
          : n <= 24 ? fused::fits<2, 3, false>(nv)
          : n <= 32 ? fused::fits<2, 4, false>(nv)
          : n <= 48 ? fused::fits<3, 3, false>(nv)
                    : fused::fits<4, 4, false>(nv));
}

int launch_fused_rkn(const FusedLaunch& L, cudaStream_t st) {
  int nmax = 0, nvmax = 0;
  check(L, nmax, nvmax);
  if (!fused_rkn_fits(nmax, nvmax)) throw std::invalid_argument("fused integration: shared memory");
  if (nmax <= 16) fused::launch<1, 1>(L, nvmax, st);
  else if (nmax <= 24) fused::launch<2, 3>(L, nvmax, st);
  else if (nmax <= 32) fused::launch<2, 4>(L, nvmax, st);
  else if (nmax <= 48) fused::launch<3, 3>(L, nvmax, st);
  else fused::launch<4, 4>(L, nvmax, st);
  return 1;
}

bool fused_rk4_fits(int n, int nv) {
  return n >= 2 && n <= kFusedRk4MaxBeams &&
         (n <= 16   ? fused::fits<1, 1, true>(nv)
          : n <= 24 ? fused::fits<2, 3, true>(nv)
          : n <= 32 ? fused::fits<2, 4, true>(nv)
                    : fused::fits<3, 3, true>(nv));
}

int launch_fused_rk4(const FusedLaunch& L, cudaStream_t st) {
  int nmax = 0, nvmax = 0;
  check(L, nmax, nvmax);
  if (L.s != 2 || !fused_rk4_fits(nmax, nvmax))
    throw std::invalid_argument("fused RK4: unsupported problem");
  if (nmax <= 16) fused::launch<1, 1, true>(L, nvmax, st);
  else if (nmax <= 24) fused::launch<2, 3, true>(L, nvmax, st);
  else if (nmax <= 32) fused::launch<2, 4, true>(L, nvmax, st);
  else fused::launch<3, 3, true>(L, nvmax, st);
  return 1;
}

}  // namespace trhepd
