// Device helpers shared by the precompiled kernels and the run-time
// specialised (NVRTC) kernels: 64-bit division by an invariant divisor and
// float-float ("df64") arithmetic.  Self-contained: no system headers, so the
// same text compiles under nvcc and NVRTC.
//
// Why df64: on GB300 the FP64 pipe issues ~0.6 T DFMA/s (measured 1.19
// TFLOP/s) against 6.7 TB/s of HBM, i.e. ~1.3 FP64 ops per streamed element.
// Rows of a PTM with more terms than that are computed on the FP32 pipes
// (~58x faster) as pairs of floats with a 48-bit significand, well inside the
// 1e-12 agreement required against float64 numpy.
#ifndef QSGB_DEVICE_CUH_
#define QSGB_DEVICE_CUH_

typedef unsigned long long qsgb_u64;
typedef long long qsgb_i64;

// Start of a kernel launched as a programmatic dependent: wait for the
// preceding grid, then let the next one be launched.  Its blocks come in as
// this grid's leave and wait here in turn, which takes the launch latency
// (1 to 1.5 us between small kernels) off the stream.
__device__ __forceinline__ void qsgb_pdl_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Unsigned 64-bit division by an invariant divisor d (Granlund & Montgomery,
// "Division by invariant integers using multiplication", PLDI 1994, Fig. 4.1,
// N = 64): q = (t + ((n - t) >> 1)) >> (l - 1), t = mulhi(m, n), with
// l = ceil(log2 d) and m = floor(2^64 (2^l - d) / d) + 1; l == 0 encodes d = 1.
__device__ __forceinline__ qsgb_u64 qsgb_fdiv(qsgb_u64 n, qsgb_u64 m, int l) {
  if (l == 0) return n;
  const qsgb_u64 t = __umul64hi(m, n);
  return (t + ((n - t) >> 1)) >> (l - 1);
}

// Split an IEEE double into hi + lo floats with integer operations and one
// I2F (the FP64<->FP32 converters run on the slow FP64 pipe on GB300, I2F at
// 16 T/s).  hi is x rounded to 24 significant bits (ties away).  The 29 bits
// below, read as a signed integer, are then exactly x - hi in units of
// 2^(E-52): I2F rounds them to nearest even and a power of two scales them, so
// hi + lo agrees with x to 2^-49 of its binade, without bias (a bias would
// accumulate linearly over a long circuit where unbiased errors grow as a
// square root), and |lo| <= 2^-24 |hi| keeps the cross terms and the dropped
// lo * lo small.  Inputs the float pair cannot carry to that precision set
// `bad`: a non-zero |x| < 2^-102 and |x| >= 2^127, inf and nan; hi and lo are
// then meaningless, and callers recompute the affected results in native FP64.
// E0 and N: the exponents taken, e in [E0, E0 + N).
template <unsigned E0 = 921u, unsigned N = 229u>
__device__ __forceinline__ void qsgb_split_f64(double x, float& hi, float& lo, unsigned& bad) {
  const unsigned h = (unsigned)__double2hiint(x);
  const unsigned l = (unsigned)__double2loint(x);
  // bits 30..23 <- e[7:0], 22..0 <- m[51:29]; rebias e-1023+127 = e-896,
  // which on the low 8 exponent bits is an xor with 0x80 (bit 30)
  const unsigned t = __funnelshift_l(l, h, 3);
  const unsigned hb = ((t & 0x7fffffffu) | (h & 0x80000000u)) ^ 0x40000000u;
  // x's sign and 2^(E-24); with the 2^-31 the scale of the integer l << 3
  const float scale = __uint_as_float((hb & 0xff800000u) - (24u << 23));
  lo = (__int2float_rn((int)(l << 3)) * 0x1p-31f) * scale;
  // e in [921, 1149] is 2^-102 <= |x| < 2^127; zero is carried exactly
  const bool out = h + h - (E0 << 21) >= (N << 21);
  hi = out ? 0.0f : __uint_as_float(hb + ((l >> 28) & 1u));
  if (out) bad |= (h + h) | l;
}

// A float-float row result whose leading float s is outside the range where
// the pair keeps 48 significant bits: 0 < |s| < 2^-70 (products whose error
// terms may have fallen below the normal floats) or |s| >= 2^126 (near
// overflow), inf or nan.  s == 0 is exact when every input of the row is
// (inputs below 2^-102 are flagged by qsgb_split_f64).  Callers recompute
// such rows in native FP64.
__device__ __forceinline__ unsigned qsgb_df_suspect(float s) {
  const float a = fabsf(s);
  return (!(a < 0x1p126f) || (a < 0x1p-70f && s != 0.0f)) ? 1u : 0u;
}

// acc (s, c) += (ph + pl) * (xh + xl); pl*xl (2^-49 relative) is dropped.
// The two-sum of s and the rounded product p is Knuth's; its correction on
// p's side and the product's rounding error are one fma, ph xh - bp, where bp
// is what the sum took of p.  The small cross term is added first, so that
// one rounding only is made at the size of the large one.  10 operations; the
// product error and the correction apart took 12.  (Letting the fma add s to
// the exact product as well, 9 operations, loses the low half whenever the
// signs differ.)  With the split above and qsgb_df_round, on GB300: a fused
// 13-qubit noisy circuit (44 passes of 3 to 8 terms per row, bound by
// instruction issue) 10.86 -> 10.00 ms, one layer of a 14-qubit one (near the
// HBM rate) 14.64 -> 14.40 ms; the RMS error of a row against long double
// falls by 40 % at 2 and 3 terms, 30 % at 6, 10 to 16 % at 16.
__device__ __forceinline__ void qsgb_df_fma(float& s, float& c, float ph, float pl, float xh, float xl) {
  const float p = __fmul_rn(ph, xh);  // _rn: never contracted with the sum below
  const float s2 = s + p;
  const float bp = s2 - s;
  float e = fmaf(ph, xh, -bp);
  e += s - (s2 - bp);
  e = fmaf(pl, xh, e);
  e = fmaf(ph, xl, e);
  s = s2;
  c += e;
}

// first term of a row: (s, c) = (ph + pl) * (xh + xl)
__device__ __forceinline__ void qsgb_df_mul(float& s, float& c, float ph, float pl, float xh, float xl) {
  const float p = __fmul_rn(ph, xh);
  float e = fmaf(ph, xh, -p);
  e = fmaf(pl, xh, e);
  c = fmaf(ph, xl, e);
  s = p;
}

// Round s + t to the nearest double for a row that qsgb_df_suspect(s) does
// not flag (a flagged row's value is discarded), with integer operations and
// one float->int conversion: as qsgb_df_to_double below without its range
// selects.  The sign of r goes into the scale, so that the correction T is in
// the magnitude's direction.  Where r is below 2^-76 and unflagged, s is 0
// and the two-sum is exact (u = 0): T is 0 also where the scale wraps to an
// infinity (an exponent field of 51 in r), for 0 * inf is a nan and a nan
// converts to the integer 0.  A subnormal r (rows whose leading floats cancel
// at 2^-102) comes out within 2^-126 of its value.
__device__ __forceinline__ double qsgb_df_round(float s, float t) {
  const float r = s + t;  // two-sum: no ordering assumption on |s|, |t|
  const float bt = r - s;
  const float u = (s - (r - bt)) + (t - bt);
  const unsigned rb = __float_as_uint(r);
  unsigned sc = (306u << 23) - (rb & 0x7f800000u);
  // a power of two with u toward zero: the next ulp is half as large
  if ((rb & 0x7fffffu) == 0u && (int)(__float_as_uint(u) ^ rb) < 0) sc += 1u << 23;
  const int T = __float2int_rn(u * __uint_as_float(sc ^ (rb & 0x80000000u)));  // in ulps of the result
  unsigned h = ((unsigned)((int)rb >> 3) & 0x8fffffffu) + (896u << 20);
  if (r == 0.0f) h = 0u;
  const qsgb_u64 bits = (((qsgb_u64)h << 32) | (qsgb_u64)(rb << 29)) + (qsgb_u64)(qsgb_i64)T;
  return __longlong_as_double((long long)bits);
}

// Round s + t (any magnitudes) to the nearest double, with integer
// operations and one float->int conversion.  After a two-sum (r, u) with
// |u| <= ulp_f(r)/2, the double is bits(r) + round(u / ulp_d(r)) ulps; when r
// is a power of two and u points toward zero the next ulp is half as large.
// |r| < 2^-74 keeps r only; r == 0 or denormal gives +-0.
__device__ __forceinline__ double qsgb_df_to_double(float s, float t) {
  const float r = s + t;  // two-sum: no ordering assumption on |s|, |t|
  const float bt = r - s;
  const float u = (s - (r - bt)) + (t - bt);
  const unsigned rb = __float_as_uint(r);
  const unsigned er = (rb >> 23) & 0xffu;
  const unsigned m = rb & 0x7fffffu;
  const unsigned sgn = rb & 0x80000000u;
  const bool toward0 = ((__float_as_uint(u) ^ rb) & 0x80000000u) != 0u;
  const unsigned sc = 306u - er + ((m == 0u && toward0) ? 1u : 0u);
  const float scale = (er >= 54u) ? __uint_as_float(sc << 23) : 0.0f;
  int T = __float2int_rn(u * scale);  // u in units of the target ulp
  if (sgn) T = -T;                   // magnitude domain
  const qsgb_u64 mag = ((qsgb_u64)(((er + 896u) << 20) | (m >> 3)) << 32) | (qsgb_u64)(m << 29);
  qsgb_u64 bits = mag + (qsgb_u64)(qsgb_i64)T;
  if (er == 0u) bits = 0;
  if (er == 255u) bits = 0x7ff8000000000000ull;
  return __longlong_as_double((long long)(bits | ((qsgb_u64)sgn << 32)));
}

#endif  // QSGB_DEVICE_CUH_
