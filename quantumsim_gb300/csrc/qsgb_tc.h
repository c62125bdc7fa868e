// Interface between the apply entry points and the tensor-core kernel for
// dense 16 x 16 PTMs (qsgb_tc.cu).
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "qsgb_common.cuh"

namespace qsgb {
namespace tc {

// ------------------------------------------------ base-256 digits
// The split of the tcgen05 kernels and of the PTM gradient: a value against
// a block exponent as a signed 55-bit fixed-point integer F in seven balanced
// base-256 digits, each exactly an FP16 number.  Byte digits cost one byte
// permute and one three-input logic operation per pair of values and digit
// (base 1024, six digits: two shifts, a permute and a logic operation), their
// products are at most 2^14, and every level sum of K <= 16 terms stays below
// 2^21, so that all levels are exact in FP32, leave it by adding 1.5 * 2^23
// (no F2I, which runs at a quarter rate) and combine pairwise in 32 bits.
// With digit pairs up to i + j = 7 the error is about half of base 1024's with
// i + j <= 5 (exact integer model, 16 terms: 6.1e-17 against 1.45e-16
// relative for inputs of one scale, 2.1e-16 against 3.8e-16 over three
// decades).
constexpr int kPlanes = 7;  // digits
constexpr int kLevels = 8;  // levels i + j = 0 .. 7
constexpr unsigned long long kBias8 = 0x0080808080808080ull;
// biased exponents below this are not scaled by: a block whose values are all
// smaller is recomputed in native FP64 (zeros are exact)
constexpr unsigned kMinExp = 64;

// |F| + B for x = (hi, lo) against the block exponent, given in place (eh =
// biased exponent << 20, >= kMinExp << 20): |F| <= 2^55; values with exponent 0
// (zero, subnormals) and those 2^-54 below the block give 0.  The sign goes
// onto the digits (Signs).
__device__ __forceinline__ unsigned long long fixed8(unsigned hi, unsigned lo, unsigned eh) {
  const unsigned s = (eh - (hi & 0x7ff00000u)) >> 20;
  const unsigned long long m = ((unsigned long long)((hi & 0xfffffu) | 0x100000u) << 32 | lo) << 2;
  unsigned long long f;
  asm("shr.u64 %0, %1, %2;" : "=l"(f) : "l"(m), "r"(s));  // shifts of 64 and more give 0
  return f + kBias8;
}

// (+-1, +-1) and -1152 (+-1, +-1) as FP16x2: the signs of two values
struct Signs {
  unsigned one, bias;
};
__device__ __forceinline__ Signs signs_of(unsigned hi_a, unsigned hi_b) {
  const unsigned q = __byte_perm(hi_a, hi_b, 0x7632) & 0x80008000u;
  return {q | 0x3c003c00u, q ^ 0xe480e480u};
}

// FP16x2 of digit j (0 the most significant) of two values: byte 6 - j, the
// top digit with its carry bit (16 bits), as 0x6400 | v = 1024 + v, minus
// 1152, with the value's sign
template <int J>
__device__ __forceinline__ unsigned digit8_pair(unsigned long long ua, unsigned long long ub, const Signs& s) {
  constexpr int byte = 6 - J;
  unsigned r;
  if (byte == 6) {
    r = __byte_perm((unsigned)(ua >> 32), (unsigned)(ub >> 32), 0x7632) | 0x64006400u;
  } else if (byte >= 4) {
    r = __byte_perm((unsigned)(ua >> 32), (unsigned)(ub >> 32), byte == 4 ? 0x0400 : 0x0501);
    r = (r & 0x00ff00ffu) | 0x64006400u;
  } else {
    constexpr unsigned sel = (unsigned)(byte | ((byte + 4) << 8));
    r = __byte_perm((unsigned)ua, (unsigned)ub, sel);
    r = (r & 0x00ff00ffu) | 0x64006400u;
  }
  unsigned out;
  asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(out) : "r"(r), "r"(s.one), "r"(s.bias));
  return out;
}

// Eight values of one row of a digit plane, every plane: 16 bytes at
// dst + J * STRIDE
template <int J, int STRIDE>
__device__ __forceinline__ void store_digits8(unsigned char* dst, const unsigned long long (&u)[8],
                                              const Signs (&s)[4]) {
  if constexpr (J < kPlanes) {
    *reinterpret_cast<uint4*>(dst + J * STRIDE) =
        make_uint4(digit8_pair<J>(u[0], u[1], s[0]), digit8_pair<J>(u[2], u[3], s[1]),
                   digit8_pair<J>(u[4], u[5], s[2]), digit8_pair<J>(u[6], u[7], s[3]));
    store_digits8<J + 1, STRIDE>(dst, u, s);
  }
}
template <int STRIDE>
__device__ __forceinline__ void split8(unsigned char* dst, const double* x, const unsigned* eh) {
  unsigned long long u[8];
  Signs s[4];
#pragma unroll
  for (int k = 0; k < 8; ++k) u[k] = fixed8((unsigned)__double2hiint(x[k]), (unsigned)__double2loint(x[k]), eh[k]);
#pragma unroll
  for (int k = 0; k < 4; ++k)
    s[k] = signs_of((unsigned)__double2hiint(x[2 * k]), (unsigned)__double2hiint(x[2 * k + 1]));
  store_digits8<0, STRIDE>(dst, u, s);
}

// An FP32 level sum, an integer below 2^22, as an integer plus kMagic
constexpr unsigned kMagic = 0x4b400000u;  // bits of 1.5 * 2^23
__device__ __forceinline__ unsigned level_bits(float a) { return __float_as_uint(a + 12582912.0f); }
// Two consecutive levels as one 32-bit integer: 256 a + b
__device__ __forceinline__ int level_pair(float a, float b) {
  return (int)((level_bits(a) << 8) + level_bits(b) - ((kMagic << 8) + kMagic));
}
// sum_L A_L 2^(56 - 8 L) / 2^14 of eight levels, given as pairs, in 64 bits.
// NARROW: 4 p45 fits 32 bits (sums over 16 products, not over 32).
template <bool NARROW = true>
__device__ __forceinline__ long long combine8(int p01, int p23, int p45, int p67) {
  const long long low = NARROW ? (long long)(p45 * 4 + (p67 >> 14)) : (long long)p45 * 4 + (p67 >> 14);
  return (long long)p23 * 262144ll + low + ((long long)p01 << 34);
}
// v 2^sc as a double, sc given as sc << 20.  For v = combine8 of values split
// against ex and PTM entries against ep (biased exponents),
// sc = ex + ep - kScale8; scale8_ok(sc) says that every result is zero or a
// normal double (1 <= |v| < 2^61), so that the results need no test of their
// own: blocks for which it fails are recomputed in native FP64.
constexpr int kScale8 = 2100;
__host__ __device__ constexpr bool scale8_ok(int sc) { return sc >= 1 - 1023 && sc <= 2046 - 1023 - 61; }
__device__ __forceinline__ double scale8(long long v, unsigned sc20) {
  const double d = __ll2double_rn(v);
  unsigned hi = (unsigned)__double2hiint(d);
  if (hi != 0u) hi += sc20;
  return __hiloint2double((int)hi, __double2loint(d));
}

// ------------------------------------------------ base-1024 digits
// digit planes of the split of the warp-level kernel (six balanced base-1024
// digits of a 57-bit fixed-point value plus sign)
constexpr int kDigits = 6;
constexpr unsigned long long kDigitBias =
    512ull * (1ull + (1ull << 10) + (1ull << 20) + (1ull << 30) + (1ull << 40) + (1ull << 50));

// Biased exponent of x as used for scaling (subnormals and zero count as 1)
// and its 53-bit significand (implicit bit included for normal numbers).
__device__ __forceinline__ unsigned exp_eff(unsigned hi) {
  const unsigned e = (hi >> 20) & 0x7ffu;
  return e == 0u ? 1u : e;
}

// F + B for input x = (hi, lo) against group exponent emax (biased, >= e):
// F = sign(x) * (m << 4) >> (emax - e), |F| < 2^57.
__device__ __forceinline__ unsigned long long fixed_biased(unsigned hi, unsigned lo, unsigned emax) {
  const unsigned e = (hi >> 20) & 0x7ffu;
  const unsigned mh = (hi & 0xfffffu) | (e != 0u ? 0x100000u : 0u);
  const unsigned long long m = ((unsigned long long)mh << 32 | lo) << 4;
  const unsigned s = emax - (e == 0u ? 1u : e);
  unsigned long long f = s < 64u ? (m >> s) : 0ull;
  if (hi & 0x80000000u) f = 0ull - f;
  return f + kDigitBias;
}

// FP16x2 register of digit plane j (bit position p = 10 (5 - j)) of two
// inputs: (v_a - 512, v_b - 512) built from 0x6400 | v = 1024 + v.
__device__ __forceinline__ unsigned digit_pair(unsigned long long ua, unsigned long long ub, int p) {
  const unsigned a = (unsigned)(ua >> p) & 0x3ffu;
  const unsigned b = (unsigned)(ub >> p) & 0x3ffu;
  const unsigned r = a | (b << 16) | 0x64006400u;
  unsigned out;
  asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(out) : "r"(r), "r"(0x66006600u));  // - (1536, 1536)
  return out;
}

// d += a b for one m16n8k16 tile: FP16 operands, FP32 accumulators (the
// fragment layouts of mma.sync.aligned.m16n8k16.row.col)
__device__ __forceinline__ void mma16816(float* d, const unsigned* a, const unsigned* b) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

struct TcParams {
  const double* in;
  double* out;
  unsigned* status;
  uint64_t n_groups, n_tiles;
  FastDiv div_z, div_y;
  int64_t sxi, syi, sai, sbi;  // strides of (x, a, y, b) in elements; z stride 1
  int64_t sxo, syo, sao, sbo;
  int pair_store;  // groups 2c, 2c+1 are adjacent and 16-byte aligned
  int vec_z1;      // Z == 1 and both tensors 32-byte aligned: a group's
                   // runs along the last target move as 32-byte vectors
  const double* dptm;  // device PTM (launch_device)
  int dlayout;         // its storage (QSGB_PTM_SWAPPED / QSGB_PTM_TRANSPOSED bits)
  double ptm[16][16];  // the op matrix of a host PTM
};
// the warp-level kernel's: the PTM split on the host
struct TcWarpParams : TcParams {
  int row_exp[16];                         // Ep_r - 1022 - 54 per row
  unsigned short digits[kDigits][16][16];  // FP16 digit planes e_i[r][k]
};

static_assert(sizeof(TcWarpParams) <= 32764, "kernel parameter limit");

// The op matrix is 16 x 16 without inf or nan.
bool eligible(const double* op, int kin, int kout);
// Apply the 16 x 16 op matrix `op` (row-major, rows = (ra, rb), columns =
// (ka, kb), qudit a more significant) to an FP64 tensor viewed as
// (X, 4, Y, 4, Z).
int launch(const double* op, const void* in, void* out, uint64_t X, uint64_t Y, uint64_t Z, unsigned* status,
           cudaStream_t stream);
// The same for a 16 x 16 PTM in device memory, stored in `layout`
// (QSGB_PTM_SWAPPED / QSGB_PTM_TRANSPOSED bits): every block reads and
// splits it (nothing is read on the host); inf or nan entries send every
// group to the native FP64 path.
int launch_device(const double* dptm, int layout, const void* in, void* out, uint64_t X, uint64_t Y, uint64_t Z,
                  unsigned* status, cudaStream_t stream);

// Larger dense PTMs (Kin, Kout <= kWideMax) in device memory, FP64 or FP32
// vectors (qsgb_tcw.cu); dimensions and strides as for launch_device.  A PTM
// with holes is not applied: `out` is marked for the generic kernel, which has
// to be launched behind (ApplyParams::only_marked).
constexpr int kWideMax = 96;
int launch_wide(const double* dptm, int layout, const void* in, void* out, int dtype, int da_out, int db_out,
                int da_in, int db_in, uint64_t X, uint64_t Y, uint64_t Z, unsigned* status, cudaStream_t stream);

// The mark is a nan that no arithmetic gives, in the first row of every group.
// (A state that holds this very nan would at worst be computed twice.)
__device__ __forceinline__ void mark_holes(double* o) {
  *reinterpret_cast<unsigned long long*>(o) = 0xfff8dead0badf00dull;
}
__device__ __forceinline__ void mark_holes(float* o) { *reinterpret_cast<unsigned*>(o) = 0xffc0deadu; }
__device__ __forceinline__ bool holes_marked(const double* o) {
  return *reinterpret_cast<const volatile unsigned long long*>(o) == 0xfff8dead0badf00dull;
}
__device__ __forceinline__ bool holes_marked(const float* o) {
  return *reinterpret_cast<const volatile unsigned*>(o) == 0xffc0deadu;
}

}  // namespace tc
}  // namespace qsgb
