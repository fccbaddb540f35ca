// Elementary functions of the device code in double precision.
#pragma once

namespace wds {
namespace {

// 1 / x for a normal x in (0, 2^1021) within 0.51 units in the last place (0 and
// infinity give NaN): the hardware's 23-bit approximation and two Newton steps
// (48 cycles of latency against 77 of the correctly rounded __drcp_rn, measured
// on dependent chains).
__device__ __forceinline__ double recip(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  y = fma(y, fma(-x, y, 1.0), y);
  return fma(y, fma(-x, y, 1.0), y);
}

// a / b with rb = recip(b), from a product and one residual step: within
// 0.51 units in the last place, so not always the rounded quotient (a and the
// residual normal).
__device__ __forceinline__ double quotient(double a, double b, double rb) {
  const double q = a * rb;
  return fma(fma(-q, b, a), rb, q);
}

__device__ __noinline__ double pow_any(double x, double y) { return pow(x, y); }

// x^y.  Every link takes one power per iteration, the largest part of the link
// pass, and CUDA's pow costs 274 cycles of a scheduler per warp (768 threads
// per SM, 791 cycles alone); this one 184 (446), and its largest error over
// 38 000 points (x 1e-30 to 1e6, y 0.852, 1, 2 and -1 to 2) is 0.60 units in
// the last place against 1.21; at exponents to 30 in size 1.3.  x = 2^e m with
// m in [sqrt(1/2), sqrt(2)): log2 m = (2 / ln 2) atanh((m - 1) / (m + 1)) from the odd series, the leading
// term as an unevaluated sum of two doubles (Dekker's exact products by fma);
// then y (e + log2 m) = n + g and 2^g = e^(g ln 2) likewise.  The coefficients
// are Chebyshev interpolants of (atanh(s) / s - 1) / s^2 on [0, 0.0295] in s^2
// (as rounded, 2^-60.6 of log2 m) and of (e^t - 1 - t) / t^2 on +-ln(2) / 2
// (2^-61.3 of the result).  Arguments that are not positive, normal and finite,
// and results near the ends of the range, take CUDA's function.
__device__ __forceinline__ double pow_pos(double x, double y) {
  const int hx = __double2hiint(x);
  if ((unsigned)(hx - 0x00100000) >= 0x7fe00000u) return pow_any(x, y);
  const int e = (hx - 0x3fe6a09f) >> 20;
  const double m = __hiloint2double(hx - (e << 20), __double2loint(x));
  const double f = m - 1.0, d = f + 2.0, dl = f - (d - 2.0);  // m + 1 = d + dl
  const double r = recip(d);
  const double s = f * r, sl = fma(-s, dl, fma(-s, d, f)) * r;
  const double z = s * s;
  double p = 0x1.0c03cc5bc65f5p-4;
  p = fma(p, z, 0x1.0fbe913e56768p-4);
  p = fma(p, z, 0x1.3b1c35868035bp-4);
  p = fma(p, z, 0x1.745cf903bf098p-4);
  p = fma(p, z, 0x1.c71c72015b06fp-4);
  p = fma(p, z, 0x1.2492492476cbap-3);
  p = fma(p, z, 0x1.9999999999a38p-3);
  p = fma(p, z, 0x1.5555555555555p-2);
  const double u = fma(s * z, p, sl);
  const double c = 0x1.71547652b82fep+1, cl = 0x1.777d0ffda0d24p-55;  // 2 / ln 2
  const double hi = c * s, lo = fma(c, u, fma(cl, s, fma(c, s, -hi)));
  // e as a double: its bits below 2^52 + 2^31
  const double E = __hiloint2double(0x43300000, (int)((unsigned)e ^ 0x80000000u)) - 0x1.000008p52;
  const double b0 = E + hi, b1 = ((E - b0) + hi) + lo;
  const double b = b0 + b1, bl = (b0 - b) + b1;  // log2 x
  const double ph = y * b, pl = fma(y, bl, fma(y, b, -ph));
  if (!(fabs(ph) < 1000.0)) return pow_any(x, y);
  const double nm = ph + 0x1.8p52;
  const int n = __double2loint(nm);  // ph to the nearest integer
  const double g = ph - (nm - 0x1.8p52);
  const double l2 = 0x1.62e42fefa39efp-1, l2l = 0x1.abc9e3b39803fp-56;  // ln 2
  const double t = l2 * g, tl = fma(l2, g, -t) + fma(l2l, g, l2 * pl);
  double q = 0x1.1f730349868cep-29;
  q = fma(q, t, 0x1.af4de97ca4194p-26);
  q = fma(q, t, 0x1.27e4db646b17ep-22);
  q = fma(q, t, 0x1.71de0231960ebp-19);
  q = fma(q, t, 0x1.a01a01a6d889cp-16);
  q = fma(q, t, 0x1.a01a01abe7fe1p-13);
  q = fma(q, t, 0x1.6c16c16c162d4p-10);
  q = fma(q, t, 0x1.11111111100dcp-7);
  q = fma(q, t, 0x1.5555555555556p-5);
  q = fma(q, t, 0x1.5555555555557p-3);
  q = fma(q, t, 0x1.0000000000000p-1);
  const double a = 1.0 + t, w = t * t * q;
  const double v = a + fma(tl, a + w, ((1.0 - a) + t) + w);
  return __hiloint2double(__double2hiint(v) + (n << 20), __double2loint(v));
}

}  // namespace
}  // namespace wds
