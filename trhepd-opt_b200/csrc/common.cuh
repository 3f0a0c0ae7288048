// Shared device helpers for the multislice surface solve (sm_100a).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <cmath>

namespace trhepd {

struct cd {  // complex double, layout-compatible with Fortran complex(8) / double _Complex
  double x, y;
};

__host__ __device__ __forceinline__ cd mk(double x, double y) { return cd{x, y}; }
__host__ __device__ __forceinline__ cd operator+(cd a, cd b) { return cd{a.x + b.x, a.y + b.y}; }
__host__ __device__ __forceinline__ cd operator-(cd a, cd b) { return cd{a.x - b.x, a.y - b.y}; }
__host__ __device__ __forceinline__ cd operator-(cd a) { return cd{-a.x, -a.y}; }
__host__ __device__ __forceinline__ cd operator*(cd a, cd b) {
  return cd{a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x};
}
__host__ __device__ __forceinline__ cd operator*(double s, cd a) { return cd{s * a.x, s * a.y}; }
__host__ __device__ __forceinline__ cd conj(cd a) { return cd{a.x, -a.y}; }
// acc + a b and acc - a b as four fused multiply-adds (rounds differently from
// acc + (a * b) with the product formed first)
__host__ __device__ __forceinline__ cd cfma(cd a, cd b, cd acc) {
  return cd{fma(a.x, b.x, fma(-a.y, b.y, acc.x)), fma(a.x, b.y, fma(a.y, b.x, acc.y))};
}
__host__ __device__ __forceinline__ cd cfms(cd a, cd b, cd acc) {
  return cd{fma(-a.x, b.x, fma(a.y, b.y, acc.x)), fma(-a.x, b.y, fma(-a.y, b.x, acc.y))};
}
__host__ __device__ __forceinline__ double cabs1(cd a) { return fabs(a.x) + fabs(a.y); }
// a / b with the scaling of Smith's algorithm
__host__ __device__ __forceinline__ cd cdiv(cd a, cd b) {
  if (fabs(b.x) >= fabs(b.y)) {
    double r = b.y / b.x, den = b.x + b.y * r;
    return cd{(a.x + a.y * r) / den, (a.y - a.x * r) / den};
  } else {
    double r = b.x / b.y, den = b.x * r + b.y;
    return cd{(a.x * r + a.y) / den, (a.y * r - a.x) / den};
  }
}
#ifdef __CUDACC__
// 1 / d = conj(d) / |d|^2, d scaled by a power of two first: |d|^2 neither overflows nor
// underflows, and the scaling rounds nothing.  1 / |d|^2 by two Newton-Raphson steps
// y <- y + y (1 - x y) on the hardware's approximation, good to its last bit or two where
// x is a normal number, as it is here (2^-102 for the least subnormal d, else 1 to 8).
// Each part to 6 * 2^-53.  Without a branch (cdiv: two divisions and one), and without a
// call, around which the 96-register elimination spills: n = 95, 61 angles, 253 slices
// take 63.2 ms with __drcp_rn, 61.4 so, 60.6 unscaled.
__device__ __forceinline__ cd crecip(cd d) {
  constexpr int kExp = 0x7ff00000;  // the exponent's bits of the high word
  const int e = max(__double2hiint(d.x) & kExp, __double2hiint(d.y) & kExp);
  const double s = __hiloint2double(max(0x7fe00000 - e, 0x00100000), 0);
  d = s * d;
  const cd ds = s * d;  // beside the chain of r: the scale of the result
  const double x = fma(d.x, d.x, d.y * d.y);
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  r = fma(r, fma(-x, r, 1.0), r);
  r = fma(r, fma(-x, r, 1.0), r);
  return cd{ds.x * r, -ds.y * r};
}
#endif

__host__ __device__ __forceinline__ int ceil_div(int a, int b) { return (a + b - 1) / b; }
__host__ __device__ __forceinline__ int round_up(int a, int b) { return ceil_div(a, b) * b; }

// Device status word bits (read back by the host after each solve).
enum : unsigned {
  kStatusNonFinite = 1u << 0,
  kStatusZeroPivot = 1u << 1,
  kStatusTimeout = 1u << 2,
};

}  // namespace trhepd
