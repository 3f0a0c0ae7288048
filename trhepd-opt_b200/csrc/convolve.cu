// Stage products as convolutions over the beam grid (hp_pinth / hp_qinth,
// sim-trhepd-rheed/src/surf_prkn.f90:222-276, with vvi2mate's matrix,
// matcomp.f90:253-279), sm_100a.
//
// The stage matrix is V(k, j) = T(g_j - g_k): a row of Q times V is a convolution of
// the row, laid out on the beams' index grid, with the Fourier components T of the
// potential.  For the 521 beams of a disc (26 x 26 grid) that is 1.7e5 FP64 operations
// a row and stage by DFTs against 1.1e6 by the dense product.  Rows are independent
// until the next renormalisation, so a CTA keeps its rows' Q and P in shared memory
// through all the stages of one launch: no state traffic to HBM between stages, no
// gathered matrices, one launch instead of two to five per stage.
//
// Linear convolution needs 2m points for m grid points.  A 2m-point DFT of a half-empty
// line is two m-point DFTs, of the line (even frequencies) and of the line times
// e^{-i pi x / m} (odd ones), and only the first m outputs of the inverse are wanted:
// the sum of the two inverses, the odd one turned back.  All transforms are m-point, in
// one thread's registers (dft.cuh).  Per stage:
//   A  line y, parity s:  q(., y) -> W[s][y][fx]                       (x transform)
//   B  column fx of s:    both y parities: transform, times the spectrum, inverse, sum
//   C  line y, parity s:  inverse over fx; the two parities (neighbouring lanes)
//      exchange halves, and each updates P and Q on its half of the line.
// C and the next A touch a line by the same pair of lanes, so a stage has two barriers.
#include <cuda_runtime.h>

#include <algorithm>
#include <stdexcept>

#include "convolve.h"
#include "dft.cuh"
#include "launch_attr.h"

namespace trhepd {

namespace {

// Threads of a CTA and CTAs per SM.  Small CTAs: their phases drift apart, so one's
// transforms (FP64 pipe) cover another's shared-memory traffic and barriers.  Measured
// per stage, us (threads x CTAs): n = 521, 31 angles: 313 (128 x 2), 323 (64 x 4), 343
// (256 x 1), 377 (64 x 5, spills); n = 300, 61 angles: 163 / 217 / 185; n = 191, 61
// angles: 54 (64 x 8), 58 (128 x 4), 74 (256 x 1); n = 95, 61 angles: 14.5 (96 x 5),
// 16.2 (64 x 8), 18.4 (256 x 1); n = 70: 9.6 (128 x 5), 12.5 (256 x 1).  Launches of six
// stages (an elimination after every slice) and slower machines of the kind: n = 191 62.
template <int M>
struct Shape {
  static constexpr int kThreads = M <= 10 ? 128 : M <= 12 ? 96 : M <= 16 ? 64 : 128;
  static constexpr int kMinB = M <= 12 ? 5 : M <= 16 ? 8 : 2;
};

template <int M>
__global__ void __launch_bounds__(Shape<M>::kThreads, Shape<M>::kMinB)
    k_conv_stages(const __grid_constant__ ConvStages a, int R, int blocks_b) {
  constexpr int XS = M | 1;            // odd line stride (16-byte words): no bank conflicts
  constexpr int H = (M + 1) / 2;       // a lane's half of a line
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int WL = M * XS;
  const int sy = a.sy, line = sy * XS;
  cd* const Qs = reinterpret_cast<cd*>(smem_raw);
  cd* const Ps = Qs + R * line;
  cd* const Ws = Ps + R * line;        // [row][s][y < M][fx]
  const int tid = threadIdx.x, nt = blockDim.x;
  const size_t elems = (size_t)4 * M * M;

  for (int blk = blockIdx.x;; blk += gridDim.x) {
    const int pb = blk / blocks_b;
    const int r0 = pb * a.rows_b + (blk - pb * blocks_b) * R;
    if (r0 >= a.rows) return;
    const int nr = min(R, min(a.rows, (pb + 1) * a.rows_b) - r0);
    const cd* spec0 = a.spec + (size_t)pb * a.spec_stride;
    __syncthreads();
    for (int e = tid; e < 2 * R * line; e += nt) Qs[e] = cd{0.0, 0.0};
    __syncthreads();
    for (int r = 0; r < nr; ++r)
      for (int j = tid; j < a.n; j += nt) {
        const int c = a.cell[j], o = r * line + (c >> 8) * XS + (c & 255);
        Qs[o] = a.Q[(size_t)(r0 + r) * a.ld + j];
        Ps[o] = a.P[(size_t)(r0 + r) * a.ld + j];
      }
    __syncthreads();
    const int na = 2 * nr * sy, nb = 2 * nr * M;  // (row, line, parity), (row, parity, column)
    for (int i = 0, k = 0; i < a.nstage; ++i, k = (k + 1 == a.s) ? 0 : k + 1) {
      const double cb = i == 0 ? a.cb0 : a.cb[k], ca = a.ca[k];
      // ---- A
      for (int t = tid; t < na; t += nt) {
        const int s = t & 1, y = (t >> 1) % sy, r = (t >> 1) / sy;
        const cd* q = Qs + r * line + y * XS;
        cd* w = Ws + (2 * r + s) * WL + y * XS;
        cd v[M];
#pragma unroll
        for (int x = 0; x < M; ++x) v[x] = q[x];
        if (s) {
#pragma unroll
          for (int x = 1; x < M; ++x) v[x] = dft::twiddle<2 * M, false>(v[x], x);
        }
        dft::Dft<M>::fwd(v);
#pragma unroll
        for (int p = 0; p < M; ++p) w[dft::freq<M>(p)] = v[p];
      }
      for (int e = tid; e < 2 * nr * (M - sy) * XS; e += nt) {  // the lines past sy
        const int rs = e / ((M - sy) * XS);
        Ws[rs * WL + line + e - rs * ((M - sy) * XS)] = cd{0.0, 0.0};
      }
      __syncthreads();
      // ---- B
      const cd* spec = spec0 + (size_t)i * elems;  // [sy parity][fy][s][fx]
      for (int t = tid; t < nb; t += nt) {
        const int fx = t % M, rs = t / M;
        cd* w = Ws + rs * WL + fx;
        const cd* sp = spec + (rs & 1) * M + fx;
        cd v[M];
#pragma unroll
        for (int y = 0; y < M; ++y) v[y] = w[y * XS];
#pragma unroll 1
        for (int h = 0; h < 2; ++h) {
          dft::Dft<M>::fwd(v);
#pragma unroll
          for (int p = 0; p < M; ++p) {
            const double2 c = __ldg(reinterpret_cast<const double2*>(
                sp + (size_t)(h * M + dft::freq<M>(p)) * 2 * M));
            v[p] = cd{fma(v[p].x, c.x, -(v[p].y * c.y)), fma(v[p].x, c.y, v[p].y * c.x)};
            if (p % 8 == 7) asm volatile("" ::: "memory");  // bounds the loads in flight
          }
          dft::Dft<M>::inv(v);
          if (h == 0) {  // the even part waits in W while the line comes back, turned
#pragma unroll
            for (int y = 0; y < M; ++y) {
              const cd u = w[y * XS];
              w[y * XS] = v[y];
              v[y] = dft::twiddle<2 * M, false>(u, y);
            }
          }
        }
#pragma unroll
        for (int y = 0; y < M; ++y)
          w[y * XS] = w[y * XS] + dft::twiddle<2 * M, true>(v[y], y);
      }
      __syncthreads();
      // ---- C
      for (int t0 = tid & ~31; t0 < na; t0 += nt) {  // whole warps: lanes exchange below
        const int t = min(t0 + (tid & 31), na - 1);  // na is even: pairs stay together
        const bool live = t0 + (tid & 31) < na;
        const int s = t & 1, y = (t >> 1) % sy, r = (t >> 1) / sy;
        const cd* w = Ws + (2 * r + s) * WL + y * XS;
        cd v[M];
#pragma unroll
        for (int p = 0; p < M; ++p) v[p] = w[dft::freq<M>(p)];
        dft::Dft<M>::inv(v);
        if (s) {
#pragma unroll
          for (int x = 1; x < M; ++x) v[x] = dft::twiddle<2 * M, true>(v[x], x);
        }
        const unsigned mask = a.mask[y] >> (s ? H : 0);
        const double* d = a.D + ((size_t)((r0 + r) / a.n) * sy + y) * M + (s ? H : 0);
        cd* q = Qs + r * line + y * XS + (s ? H : 0);
        cd* p = Ps + r * line + y * XS + (s ? H : 0);
#pragma unroll
        for (int x = 0; x < H; ++x) {
          const cd hi = x + H < M ? v[x + H < M ? x + H : x] : cd{0.0, 0.0};
          const cd give = s ? v[x] : hi, keep = s ? hi : v[x];
          cd z = keep + cd{__shfl_xor_sync(0xffffffffu, give.x, 1),
                           __shfl_xor_sync(0xffffffffu, give.y, 1)};
          // cells without a beam stay zero (bits cleared: no predicate per cell)
          const int on = (int)(mask << (31 - x)) >> 31;
          z.x = __hiloint2double(__double2hiint(z.x) & on, __double2loint(z.x) & on);
          z.y = __hiloint2double(__double2hiint(z.y) & on, __double2loint(z.y) & on);
          if (live && (x + H < M || !s)) {
            const cd qv = q[x];
            const double dv = __ldg(d + x);
            cd pv = p[x];
            pv = cd{fma(cb, fma(qv.x, dv, z.x), pv.x), fma(cb, fma(qv.y, dv, z.y), pv.y)};
            p[x] = pv;
            q[x] = cd{fma(ca, pv.x, qv.x), fma(ca, pv.y, qv.y)};
          }
          if (x % 4 == 3) asm volatile("" ::: "memory");
        }
        __syncwarp();
      }
      // the next A reads the lines this C wrote by the same pair of lanes
    }
    __syncthreads();
    for (int r = 0; r < nr; ++r)
      for (int j = tid; j < a.n; j += nt) {
        const int c = a.cell[j], o = r * line + (c >> 8) * XS + (c & 255);
        a.Q[(size_t)(r0 + r) * a.ld + j] = Qs[o];
        a.P[(size_t)(r0 + r) * a.ld + j] = Ps[o];
      }
  }
}

template <int M>
size_t row_bytes(int sy) {
  return (size_t)2 * (sy + M) * (M | 1) * sizeof(cd);
}

template <int M>
void launch_stages(const ConvStages& a, int max_ctas, cudaStream_t st) {
  using S = Shape<M>;
  static SmemOptIn attr;
  const size_t limit = 227 * 1024 / S::kMinB - 1024;  // 1 KB of each CTA is the system's
  // rows a CTA can hold: tasks of one round, shared memory
  const int rmax = std::max(1, std::min(S::kThreads / (2 * M), (int)(limit / row_bytes<M>(a.sy))));
  const int nprob = ceil_div(a.rows, a.rows_b);
  // rows per CTA: as few waves as the most rows give, then as few rows as those allow
  const int slots = 148 * S::kMinB;
  auto waves = [&](int r) { return ceil_div(nprob * ceil_div(a.rows_b, r), slots); };
  int R = rmax;
  while (R > 1 && waves(R - 1) == waves(rmax)) --R;
  const size_t smem = (size_t)R * row_bytes<M>(a.sy);
  attr.ensure((const void*)k_conv_stages<M>, smem);
  const int blocks_b = ceil_div(a.rows_b, R), blocks = nprob * blocks_b;
  const int grid = max_ctas > 0 ? std::min(blocks, max_ctas * S::kMinB) : blocks;
  const int threads = std::min(round_up(2 * R * M, 32), S::kThreads);
  k_conv_stages<M><<<grid, threads, smem, st>>>(a, R, blocks_b);
}

// One CTA per column and problem: the 2m x 2m difference grid from the table, its DFT
// by direct sums (x, then y), scaled by 1 / (2m)^2.  A few 1e-3 of the stages' own time.
__global__ void __launch_bounds__(256)
    k_conv_spectra(const TableEntry* __restrict__ table, const TableEntry* const* __restrict__ tables,
                   size_t col0, int nv, const int* __restrict__ entry, int m, int sx, int sy,
                   cd* __restrict__ spec, size_t spec_stride) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int L = 2 * m, nx = 2 * sx - 1, ny = 2 * sy - 1;
  cd* g = reinterpret_cast<cd*>(smem_raw);  // [ny][nx], differences -(s-1) .. s-1
  cd* h = g + nx * ny;                      // [ny][L]
  cd* w = h + ny * L;                       // e^{-2 pi i k / L}
  const TableEntry* tc = (tables ? tables[blockIdx.y] : table) + (col0 + blockIdx.x) * (size_t)nv;
  for (int k = threadIdx.x; k < L; k += blockDim.x) {
    double s, c;
    sincospi(2.0 * k / L, &s, &c);
    w[k] = cd{c, -s};
  }
  const double scale = 1.0 / ((double)L * L);
  for (int e = threadIdx.x; e < nx * ny; e += blockDim.x) {
    const int dx = e % nx - (sx - 1), dy = e / nx - (sy - 1);
    const int t = entry[((dy + L) % L) * L + (dx + L) % L];
    cd v = cd{0.0, 0.0};
    if (t > 0) v = -conj(tc[t - 1].u);
    else if (t < 0) v = -tc[-t - 1].w;
    g[e] = scale * v;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < ny * L; e += blockDim.x) {
    const int kx = e % L, y = e / L;
    cd s = cd{0.0, 0.0};
    int ph = (kx * (L - (sx - 1))) % L;
    for (int x = 0; x < nx; ++x) {
      s = cfma(g[y * nx + x], w[ph], s);
      ph += kx;
      if (ph >= L) ph -= L;
    }
    h[e] = s;
  }
  __syncthreads();
  cd* out = spec + (size_t)blockIdx.y * spec_stride + (size_t)blockIdx.x * L * L;
  for (int e = threadIdx.x; e < L * L; e += blockDim.x) {
    const int kx = e % L, ky = e / L;
    cd s = cd{0.0, 0.0};
    int ph = (ky * (L - (sy - 1))) % L;
    for (int y = 0; y < ny; ++y) {
      s = cfma(h[y * L + kx], w[ph], s);
      ph += ky;
      if (ph >= L) ph -= L;
    }
    out[((size_t)((ky & 1) * m + (ky >> 1)) * 2 + (kx & 1)) * m + (kx >> 1)] = s;
  }
}

__global__ void k_conv_check(const TableEntry* __restrict__ table, int ncol, int nv,
                             const int* __restrict__ twins, int ntwins, int* __restrict__ bad) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= ntwins) return;
  const int e1 = twins[2 * t], e2 = twins[2 * t + 1];
  for (int c = blockIdx.y; c < ncol; c += gridDim.y) {
    const TableEntry* tc = table + (size_t)c * nv;
    const cd u = tc[e1].u, w = tc[e2].w, u0 = tc[0].u;
    const double tol = 1e-14 * (fabs(u0.x) + fabs(u0.y));
    if (!(fabs(u.x - w.x) <= tol && fabs(u.y + w.y) <= tol)) *bad = 1;
  }
}

}  // namespace

size_t conv_spectrum_elems(int m) { return (size_t)4 * m * m; }

void launch_conv_spectra(const TableEntry* table, const TableEntry* const* tables, int nprob,
                         size_t col0, int ncol, int nv, const int* entry, int m, int sx, int sy,
                         cd* spec, size_t spec_stride, cudaStream_t st) {
  static SmemOptIn attr;
  const size_t L = 2 * m, nx = 2 * sx - 1, ny = 2 * sy - 1;
  const size_t smem = (nx * ny + ny * L + L) * sizeof(cd);
  attr.ensure((const void*)k_conv_spectra, smem);
  k_conv_spectra<<<dim3((unsigned)ncol, (unsigned)nprob), 256, smem, st>>>(
      table, tables, col0, nv, entry, m, sx, sy, spec, spec_stride);
}

void launch_conv_check(const TableEntry* table, int ncol, int nv, const int* twins, int ntwins,
                       int* bad, cudaStream_t st) {
  if (ntwins <= 0) return;
  k_conv_check<<<dim3(ceil_div(ntwins, 128), std::min(ncol, 1024)), 128, 0, st>>>(
      table, ncol, nv, twins, ntwins, bad);
}

void launch_conv_stages(const ConvStages& a, int max_ctas, cudaStream_t st) {
  switch (a.m) {
    case 9: return launch_stages<9>(a, max_ctas, st);
    case 10: return launch_stages<10>(a, max_ctas, st);
    case 12: return launch_stages<12>(a, max_ctas, st);
    case 15: return launch_stages<15>(a, max_ctas, st);
    case 16: return launch_stages<16>(a, max_ctas, st);
    case 20: return launch_stages<20>(a, max_ctas, st);
    case 25: return launch_stages<25>(a, max_ctas, st);
    case 27: return launch_stages<27>(a, max_ctas, st);
    case 32: return launch_stages<32>(a, max_ctas, st);
    default: throw std::invalid_argument("convolution: transform length");
  }
}

}  // namespace trhepd
