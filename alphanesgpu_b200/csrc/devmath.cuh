// Device helpers of the sweeps (sweep.cuh) and the operators (ops.cu); included inside namespace stafb.
#pragma once

// exp(x) in double precision, table-driven (P. T. P. Tang, ACM TOMS 15, 1989): with n = round(16 x / ln 2), x = n ln2/16 +
// r, |r| <= ln2/32, exp(x) = 2^(n div 16) * 2^((n mod 16)/16) * e^r and e^r - 1 = r + r^2 q(r), q the degree-4 Chebyshev
// interpolant of (e^r - 1 - r)/r^2 (error 2.8e-17).  Eleven double operations; the table is sixteen doubles in shared
// memory = all 32 banks once, so lanes with different n never conflict.  The sweeps in double precision evaluate
// little else: the library's exp takes 58 issue cycles per warp on this GPU, a double fma 2.  The exponent saturates
// (below 2^-1022; above 2^1024 as a NaN, never a finite value); no branch, which would keep the exponentials of a
// pair's channels from overlapping.
__device__ const double EXP16_TABLE[16] = {
    1.0,                1.0442737824274138, 1.0905077326652577, 1.1387886347566916, 1.189207115002721,  1.241857812073484,
    1.2968395546510096, 1.3542555469368927, 1.4142135623730951, 1.4768261459394993, 1.5422108254079407, 1.6104903319492543,
    1.681792830507429,  1.7562521603732995, 1.8340080864093424, 1.9152065613971474};
__device__ __forceinline__ double exp_table16(double x, const double* tab) {
  const double magic = 6755399441055744.0;  // 1.5 * 2^52: the integer lands in the low word
  const double t = fma(x, 23.083120654223414, magic);
  const int n = __double2loint(t);
  const double nf = t - magic;
  double r = fma(nf, -0.043321698780346196, x);  // ln2/16 with 33 bits: exact products
  r = fma(nf, -4.650385693757748e-12, r);
  double q = fma(0.0013889034348599464, r, 0.008333449701253456);
  q = fma(q, r, 0.04166666666496045);
  q = fma(q, r, 0.1666666666530169);
  q = fma(q, r, 0.5);
  const double T0 = tab[n & 15];
  const double e = fma(T0, fma(r * r, q, r), T0);
  const int k = max(-1022, min(n >> 4, 1024));
  return __hiloint2double(__double2hiint(e) + (k << 20), __double2loint(e));
}

// Sums NV per-lane values over the 32 lanes of a warp.  Every step halves the number of values a lane
// still carries (lanes with the step's bit set keep the upper half and hand over the lower one), so
// NV-1 shuffles replace 5*NV; once one value is left the remaining steps are a plain butterfly.
// On return lane L holds the total of value index L >> log2(32 / NV).  NV is a power of two <= 32.
template <class T, int NV>
__device__ __forceinline__ T multi_reduce(T (&v)[NV], int lane) {
  static_assert(NV == 1 || NV == 2 || NV == 4 || NV == 8 || NV == 16 || NV == 32, "NV must be a power of two");
  int off = 16;
#pragma unroll
  for (int half = NV / 2; half >= 1; half >>= 1) {
    const bool up = (lane & off) != 0;
#pragma unroll
    for (int i = 0; i < half; i++) {
      const T keep = up ? v[i + half] : v[i];
      const T send = up ? v[i] : v[i + half];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
    }
    off >>= 1;
  }
  T r = v[0];
  for (; off >= 1; off >>= 1) r += __shfl_xor_sync(0xffffffffu, r, off);
  return r;
}
