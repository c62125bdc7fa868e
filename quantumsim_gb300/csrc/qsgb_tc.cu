// Dense two-qubit PTMs (16 x 16, FP64 storage) on the tensor cores.
//
// A dense PTM row has 16 terms: in float-float on the FP32 pipes that is
// ~12 instructions per term, and the kernel is bound by instruction issue at
// a quarter of the HBM rate; in native FP64 it is bound by the FP64 pipe
// (~0.6 T FMA/s on GB300).  These kernels compute the contraction exactly
// enough for FP64 parity on the FP16 tensor cores instead, with an
// error-free splitting in the spirit of the Ozaki scheme (Ozaki, Ogita,
// Oishi and Rump, "Error-free transformations of matrix multiplication by
// using fast routines of matrix multiplication and its applications",
// Numer. Algorithms 59, 2012):
//
//  * Each group of 16 inputs (one bystander index) and each PTM row is scaled
//    by its largest binary exponent and written as fixed-point integers, with
//    integer operations on the double's bit pattern, in balanced digits that
//    are exact FP16 numbers.
//  * For pairs of digit planes (i, j) up to a last level the tensor cores add
//    sum_k e_ik d_jk to the FP32 accumulator of level L = i + j.
//  * The level sums are combined in 64-bit integer arithmetic, converted to
//    double once and scaled on the exponent field.
//
// The tcgen05 kernel (the second half of this file, used by default) has
// seven base-256 digits and levels 0 .. 7, all exact integer sums; the digits
// and their error are described in qsgb_tc.h.  The warp-level kernel that
// follows here (QSGB_TC_KERNEL=mma_sync) has six base-1024 digits of a 57-bit
// F: with B = 512 * sum_j 2^(10 j), F + B is a non-negative 60-bit integer
// whose digits v_j give d_j = v_j - 512; a product of two is at most 2^18, a
// K = 16 sum at most 2^22, levels 0 .. 3 are exact and 4 and 5 may round their
// last bit, 2^-40 below level 0.  Its error is about 2^-47.7 * max_k |P_rk| *
// max_k |x_k| of the row and group, the tcgen05 kernel's below 2^-49 of it
// (typically 2^-54), against 16 * 2^-53 * sum_k |P_rk| |x_k| for an FP64
// dot product.  Groups whose inputs hold inf or nan, or whose results leave
// the normal double range, are recomputed in native FP64.
//
// Warp-level work mapping: a warp takes tiles of 8 groups (the N of the MMA).
// Lane (g, c) = (lane / 4, lane % 4) loads inputs k in {2c, 2c+1, 2c+8, 2c+9}
// of group g (the B fragment layout of m16n8k16), and ends with outputs rows
// {g, g+8} of groups {2c, 2c+1} (the accumulator layout).  The PTM digit
// planes (the A fragments) are loaded into registers once per warp.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <type_traits>

#include "qsgb_common.cuh"
#include "qsgb_tc.h"

namespace qsgb {
namespace tc {
namespace {

constexpr int kBlock = 256;


// 2^sc * sum_L A_L 2^(10 (4 - L)); bad |= 1 when the result is not a normal
// double (or zero).
__device__ __forceinline__ double combine(const float (&acc)[kDigits][4], int s, int sc, unsigned& bad) {
  long long v = (long long)__float2int_rn(acc[0][s]) << 40;
  v += (long long)__float2int_rn(acc[1][s]) << 30;
  v += (long long)__float2int_rn(acc[2][s]) << 20;
  v += (long long)__float2int_rn(acc[3][s]) << 10;
  v += (long long)__float2int_rn(acc[4][s]);
  v += (long long)(__float2int_rn(acc[5][s]) >> 10);
  if (v == 0) return 0.0;
  const double d = __ll2double_rn(v);
  const int hi = __double2hiint(d);
  const int e = ((hi >> 20) & 0x7ff) + sc;
  bad |= (e < 1 || e > 2046) ? 1u : 0u;
  return __hiloint2double(hi + (sc << 20), __double2loint(d));
}

template <bool CONTIG>
__global__ void __launch_bounds__(kBlock) apply16_tc_kernel(const __grid_constant__ TcWarpParams p) {
  const int lane = threadIdx.x & 31;
  const int g = lane >> 2, c = lane & 3;
  const int warps = kBlock / 32;
  // A fragments of every digit plane: rows {g, g+8}, columns {2c, 2c+1} and
  // {2c+8, 2c+9}
  unsigned A[kDigits][4];
#pragma unroll
  for (int i = 0; i < kDigits; ++i) {
    const unsigned short* d = &p.digits[i][0][0];
    A[i][0] = d[g * 16 + 2 * c] | ((unsigned)d[g * 16 + 2 * c + 1] << 16);
    A[i][1] = d[(g + 8) * 16 + 2 * c] | ((unsigned)d[(g + 8) * 16 + 2 * c + 1] << 16);
    A[i][2] = d[g * 16 + 2 * c + 8] | ((unsigned)d[g * 16 + 2 * c + 9] << 16);
    A[i][3] = d[(g + 8) * 16 + 2 * c + 8] | ((unsigned)d[(g + 8) * 16 + 2 * c + 9] << 16);
  }
  const int rsc0 = p.row_exp[g], rsc1 = p.row_exp[g + 8];
  // this lane's inputs k = (ka, kb): 2c -> (c/2, 2(c%2)), +1 -> kb + 1,
  // +8 -> ka + 2
  const int ka = c >> 1, kb = 2 * (c & 1);
  const int64_t in_off0 = ka * p.sai + kb * p.sbi;
  const int64_t in_off2 = in_off0 + 2 * p.sai;
  // this lane's outputs: rows g = (g/4, g%4) and g + 8 = (g/4 + 2, g%4)
  const int64_t out_off0 = (g >> 2) * p.sao + (g & 3) * p.sbo;
  const int64_t out_off1 = out_off0 + 2 * p.sao;

  auto base = [&](uint64_t grp, int64_t sx, int64_t sy) -> int64_t {
    const uint64_t t1 = fdiv(grp, p.div_z);
    const uint64_t z = grp - t1 * p.div_z.d;
    const uint64_t x = fdiv(t1, p.div_y);
    const uint64_t y = t1 - x * p.div_y.d;
    return (int64_t)x * sx + (int64_t)y * sy + (int64_t)z;
  };

  const uint64_t wstride = (uint64_t)gridDim.x * warps;
  for (uint64_t tile = (uint64_t)blockIdx.x * warps + (threadIdx.x >> 5); tile < p.n_tiles; tile += wstride) {
    const uint64_t g0 = tile * 8;
    const uint64_t gi = g0 + g;  // this lane's input group
    const bool live = gi < p.n_groups;
    int64_t bi;
    if (CONTIG) {
      // 8 consecutive groups are 8 consecutive z of one (x, y)
      bi = base(g0, p.sxi, p.syi) + g;
    } else {
      bi = live ? base(gi, p.sxi, p.syi) : 0;
    }
    double x[4] = {0.0, 0.0, 0.0, 0.0};
    if (live) {
      x[0] = p.in[bi + in_off0];
      x[1] = p.in[bi + in_off0 + p.sbi];
      x[2] = p.in[bi + in_off2];
      x[3] = p.in[bi + in_off2 + p.sbi];
    }
    unsigned hi[4], lo[4];
    unsigned emax = 1u, bad = 0u;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      hi[i] = (unsigned)__double2hiint(x[i]);
      lo[i] = (unsigned)__double2loint(x[i]);
      emax = max(emax, exp_eff(hi[i]));
      bad |= ((hi[i] >> 20) & 0x7ffu) == 0x7ffu ? 1u : 0u;  // inf, nan
    }
    emax = max(emax, __shfl_xor_sync(0xffffffffu, emax, 1));
    emax = max(emax, __shfl_xor_sync(0xffffffffu, emax, 2));
    unsigned long long u[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) u[i] = fixed_biased(hi[i], lo[i], emax);
    unsigned B[kDigits][2];
#pragma unroll
    for (int j = 0; j < kDigits; ++j) {
      B[j][0] = digit_pair(u[0], u[1], 10 * (kDigits - 1 - j));
      B[j][1] = digit_pair(u[2], u[3], 10 * (kDigits - 1 - j));
    }
    float acc[kDigits][4];
#pragma unroll
    for (int l = 0; l < kDigits; ++l) acc[l][0] = acc[l][1] = acc[l][2] = acc[l][3] = 0.f;
#pragma unroll
    for (int i = 0; i < kDigits; ++i)
#pragma unroll
      for (int j = 0; i + j < kDigits; ++j) mma16816(acc[i + j], A[i], B[j]);
    // output groups 2c and 2c+1: their exponents live in lanes 8c and 8c+4
    const int ex0 = (int)__shfl_sync(0xffffffffu, emax, 8 * c) - 1022;
    const int ex1 = (int)__shfl_sync(0xffffffffu, emax, 8 * c + 4) - 1022;
    double y[4];
    y[0] = combine(acc, 0, ex0 + rsc0, bad);  // row g, group 2c
    y[1] = combine(acc, 1, ex1 + rsc0, bad);  // row g, group 2c+1
    y[2] = combine(acc, 2, ex0 + rsc1, bad);  // row g+8, group 2c
    y[3] = combine(acc, 3, ex1 + rsc1, bad);  // row g+8, group 2c+1
    const uint64_t go0 = g0 + 2 * c, go1 = go0 + 1;
    int64_t bo0, bo1;
    if (CONTIG) {
      bo0 = base(g0, p.sxo, p.syo) + 2 * c;
      bo1 = bo0 + 1;
    } else {
      bo0 = go0 < p.n_groups ? base(go0, p.sxo, p.syo) : 0;
      bo1 = go1 < p.n_groups ? base(go1, p.sxo, p.syo) : 0;
    }
    if (__any_sync(0xffffffffu, bad)) {
      // inf / nan inputs or results outside the normal range: the tile's
      // outputs in native FP64 (lane: rows g, g+8 of groups 2c, 2c+1); the
      // loops over q and h are unrolled so that y[] stays in registers
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const uint64_t gq = q ? go1 : go0;
        if (gq < p.n_groups) {
          const int64_t b_in = base(gq, p.sxi, p.syi);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int r = g + 8 * h;
            double a = 0.0;
#pragma unroll 1
            for (int k = 0; k < 16; ++k)
              a = fma(p.ptm[r][k], p.in[b_in + (k >> 2) * p.sai + (k & 3) * p.sbi], a);
            y[2 * h + q] = a;
          }
        }
      }
    }
    if (CONTIG && p.pair_store) {
      // groups 2c, 2c+1 are adjacent: 16-byte stores
      *reinterpret_cast<double2*>(p.out + bo0 + out_off0) = make_double2(y[0], y[1]);
      *reinterpret_cast<double2*>(p.out + bo0 + out_off1) = make_double2(y[2], y[3]);
    } else {
      if (go0 < p.n_groups) {
        p.out[bo0 + out_off0] = y[0];
        p.out[bo0 + out_off1] = y[2];
      }
      if (go1 < p.n_groups) {
        p.out[bo1 + out_off0] = y[1];
        p.out[bo1 + out_off1] = y[3];
      }
    }
  }
}

// ---------------------------------------------------------------------------
// tcgen05 form: one thread per group, 128 groups per tile (the M of one
// tcgen05.mma), the eight level accumulators in tensor memory.
//
// Per tile, each thread splits its group's 16 inputs and writes its row of the
// seven input digit planes (the A operand, 128 x 16 FP16 each) to shared
// memory; then it loads its inputs of the next tile.  One thread issues seven
// tcgen05.mma.kind::f16, one per input plane j: the B operand is PTM planes
// 0 .. 7 - j stacked along N (plane 7 is zero), and since level i + j is
// accumulator column block i + j, their levels are adjacent columns.  One MMA
// per pair of planes (34 of N = 16) read the input planes five times as often
// from shared memory.  After the commit's mbarrier each warp reads its 32
// lanes (groups) of the accumulators with tcgen05.ld and recombines its
// outputs.  Shared-memory operands use the canonical K-major layout without
// swizzling: core matrices of 8 rows x 16 bytes (8 FP16 along K) at
// (row / 8) * 256 + (k / 8) * 128, so the descriptors carry a leading (K) byte
// offset of 128 and a stride (8-row) byte offset of 256.
//
// What bounds it: the serial chain of a tile (load, split, barrier, MMAs,
// recombination, ~85 instructions per element) over the 4 blocks of an SM that
// tensor memory allows; issue is half busy, the FP64 pipe 73 % with one
// conversion per output (ncu, 12 qubits).  Measured on GB300, dense PTMs, us (start of this
// design: base-1024 digits, 21 MMAs, two barriers a tile): 13 qubits 349 ->
// 263 (3.07 -> 4.08 TB/s), 12 qubits 92.7 -> 71.4, 10 qubits 14.3 -> 10.2,
// last two of 12 qubits 103.8 -> 75.1.  Of the 21 us at 12 qubits, byte digits
// and fewer selects gave 11, the stacked MMAs 10.  Two threads a group (256
// threads a block) measured 74.6 at 12 qubits.
constexpr int kUBlock = 128;
constexpr int kPlaneA = 128 * 16 * 2;  // one input digit plane: 128 rows x 16 FP16
constexpr int kPlaneB = 16 * 16 * 2;   // one PTM digit plane: 16 rows x 16 FP16
constexpr int kSmemB = kPlanes * kPlaneA;             // 28672
constexpr int kSmemBar = kSmemB + kLevels * kPlaneB;  // 32768: the PTM's planes and one of zeros
constexpr int kSmemTmem = kSmemBar + 8;
constexpr int kSmemRowExp = kSmemBar + 32;  // int[16] (device PTMs)
static_assert(kSmemRowExp % 16 == 0 && kSmemRowExp + 64 <= 56 * 1024, "shared-memory layout");
// the dynamic allocation is padded so that at most 4 blocks share an SM:
// 4 x 128 tensor-memory columns fill its 512
constexpr int kUmmaSmem = 56 * 1024;
constexpr unsigned kTmemCols = 16 * kLevels;  // 128, a power of two
// kind::f16 instruction descriptor: D F32 (bits 4-5 = 1), A and B F16 (0),
// both K-major, M / 16 at bits 24-28; N / 8 (bits 17-22) is added
constexpr uint32_t kIdesc0 = (1u << 4) | ((128u >> 4) << 24);
constexpr long long kSpinLimit = 1ll << 26;

__host__ __device__ constexpr int core_off(int row, int k) {
  return (row >> 3) * 256 + (k >> 3) * 128 + (row & 7) * 16 + (k & 7) * 2;
}

// shared-memory matrix descriptor: start >> 4 (bits 0-13), leading byte
// offset >> 4 (16-29), stride byte offset >> 4 (32-45), version 1 (46-47),
// no swizzling (61-63 = 0)
__device__ __forceinline__ unsigned long long smem_desc(uint32_t saddr) {
  return (unsigned long long)((saddr >> 4) & 0x3fffu) | ((unsigned long long)(128 >> 4) << 16) |
         ((unsigned long long)(256 >> 4) << 32) | (1ull << 46);
}

__device__ __forceinline__ uint32_t tmem_ld4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
  return 0;
}

// Offset of op element (r, k) in a 16 x 16 two-qubit PTM stored in `layout`.
__device__ __forceinline__ int dev_index(int layout, int r, int k) {
  const int ra = r >> 2, rb = r & 3, ka = k >> 2, kb = k & 3;
  switch (layout & 3) {
    case 0:
      return r * 16 + k;
    case QSGB_PTM_SWAPPED:  // (rb, ra, kb, ka)
      return ((rb * 4 + ra) * 4 + kb) * 4 + ka;
    case QSGB_PTM_TRANSPOSED:  // forward (ka, kb, ra, rb)
      return k * 16 + r;
    default:  // forward swapped (kb, ka, rb, ra)
      return ((kb * 4 + ka) * 4 + rb) * 4 + ra;
  }
}

// DEVP: the PTM is in device memory (p.dptm), else in the parameters (p.ptm).
// Every block splits it into the B operand planes and the row scales, in
// shared memory: that costs less than carrying the planes in the parameters
// (3.5 KB more a launch, read back with divergent constant loads: 11.9 against
// 10.2 us on 10 qubits) and leaves the host nothing to split.
template <bool CONTIG, bool DEVP>
__global__ void __launch_bounds__(kUBlock) apply16_umma_kernel(const __grid_constant__ TcParams p) {
  extern __shared__ __align__(1024) unsigned char smem[];
  const int t = threadIdx.x, warp = t >> 5;
  const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(smem);
  const uint32_t sA = sbase, sB = sbase + kSmemB, bar = sbase + kSmemBar;
  volatile uint32_t* tslot = reinterpret_cast<volatile uint32_t*>(smem + kSmemTmem);
  const int64_t sai = p.sai, sbi = p.sbi;

  auto base = [&](uint64_t grp) -> int64_t {
    const uint64_t t1 = fdiv(grp, p.div_z);
    const uint64_t z = grp - t1 * p.div_z.d;
    const uint64_t x = fdiv(t1, p.div_y);
    const uint64_t y = t1 - x * p.div_y.d;
    return (int64_t)x * p.sxi + (int64_t)y * p.syi + (int64_t)z;
  };

  // a tile's inputs: this thread's group, 16 values; with unit stride along
  // the last target (Z == 1, tensors 32-byte aligned) as 4 32-byte loads: lanes
  // are 128 bytes apart there, and each access costs one sector a lane
  // (last two of 12 qubits: 95.3 against 75.1 us with 16-byte accesses)
  auto load_tile = [&](uint64_t tile, double (&x)[16], int64_t& b, bool& live) {
    const uint64_t gi = tile * kUBlock + t;
    live = tile < p.n_tiles && gi < p.n_groups;
    b = 0;
    if (CONTIG) {
      if (tile < p.n_tiles) b = base(tile * kUBlock) + t;  // 128 consecutive z of one (x, y)
    } else if (live) {
      b = base(gi);
    }
    if (!live) {
#pragma unroll
      for (int k = 0; k < 16; ++k) x[k] = 0.0;
    } else if (p.vec_z1) {
#pragma unroll
      for (int ka = 0; ka < 4; ++ka)
        asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];"
                     : "=d"(x[4 * ka]), "=d"(x[4 * ka + 1]), "=d"(x[4 * ka + 2]), "=d"(x[4 * ka + 3])
                     : "l"(p.in + b + ka * sai));
    } else {
#pragma unroll
      for (int k = 0; k < 16; ++k) x[k] = p.in[b + (k >> 2) * sai + (k & 3) * sbi];
    }
  };

  uint32_t phase = 0;
  bool timed_out = false;
  double x[16];
  int64_t b;
  bool live;
  uint64_t tile = blockIdx.x;
  // set-up that reads no memory, while the preceding kernel finishes
  if (t < kPlaneB / 16) *reinterpret_cast<uint4*>(smem + kSmemB + kPlanes * kPlaneB + 16 * t) = make_uint4(0, 0, 0, 0);
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sbase + kSmemTmem),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (t == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();  // this block has its tensor memory before a dependent's may ask for any
  pdl_wait();
  load_tile(tile, x, b, live);  // in flight during the split of the PTM
  int* srow = reinterpret_cast<int*>(smem + kSmemRowExp);
  int ptm_bad = 0;  // inf or nan entries, or a row too small to scale by (this thread's pair)
  {
    // 8 threads per row (lanes 8r' .. 8r'+7 of a warp), two entries each
    const int r = t >> 3, k = 2 * (t & 7);
    const double v0 = DEVP ? p.dptm[dev_index(p.dlayout, r, k)] : p.ptm[r][k];
    const double v1 = DEVP ? p.dptm[dev_index(p.dlayout, r, k + 1)] : p.ptm[r][k + 1];
    const unsigned h0 = (unsigned)__double2hiint(v0), h1 = (unsigned)__double2hiint(v1);
    unsigned emax = max((h0 >> 20) & 0x7ffu, (h1 >> 20) & 0x7ffu);
    emax = max(emax, __shfl_xor_sync(0xffffffffu, emax, 1));
    emax = max(emax, __shfl_xor_sync(0xffffffffu, emax, 2));
    emax = max(emax, __shfl_xor_sync(0xffffffffu, emax, 4));
    // inf, nan, or a non-zero row below the smallest scale
    ptm_bad = (emax == 0x7ffu || (emax < kMinExp && (v0 != 0.0 || v1 != 0.0))) ? 1 : 0;
    if (emax < kMinExp) emax = 1023u;  // any scale serves a row of zeros
    const unsigned long long u0 = fixed8(h0, (unsigned)__double2loint(v0), emax << 20);
    const unsigned long long u1 = fixed8(h1, (unsigned)__double2loint(v1), emax << 20);
    const Signs sg = signs_of(h0, h1);
    unsigned char* dst = smem + kSmemB + core_off(r, k);
    *reinterpret_cast<unsigned*>(dst + 0 * kPlaneB) = digit8_pair<0>(u0, u1, sg);
    *reinterpret_cast<unsigned*>(dst + 1 * kPlaneB) = digit8_pair<1>(u0, u1, sg);
    *reinterpret_cast<unsigned*>(dst + 2 * kPlaneB) = digit8_pair<2>(u0, u1, sg);
    *reinterpret_cast<unsigned*>(dst + 3 * kPlaneB) = digit8_pair<3>(u0, u1, sg);
    *reinterpret_cast<unsigned*>(dst + 4 * kPlaneB) = digit8_pair<4>(u0, u1, sg);
    *reinterpret_cast<unsigned*>(dst + 5 * kPlaneB) = digit8_pair<5>(u0, u1, sg);
    *reinterpret_cast<unsigned*>(dst + 6 * kPlaneB) = digit8_pair<6>(u0, u1, sg);
    if ((t & 7) == 0) srow[r] = (int)emax - kScale8;
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  ptm_bad = __syncthreads_or(ptm_bad);
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tslot;
  const uint32_t tlane = tmem + ((uint32_t)(32 * warp) << 16);
  int rmin = srow[0], rmax = srow[0];  // row scales, least and greatest
#pragma unroll
  for (int r = 1; r < 16; ++r) {
    rmin = min(rmin, srow[r]);
    rmax = max(rmax, srow[r]);
  }
  bool done = true;  // this thread saw the last tile's MMAs complete
  for (; tile < p.n_tiles; tile += gridDim.x) {
    unsigned eh = 0u;
#pragma unroll
    for (int k = 0; k < 16; ++k) eh = max(eh, (unsigned)__double2hiint(x[k]) & 0x7ff00000u);
    unsigned emax = eh >> 20;
    unsigned bad = (ptm_bad || emax == 0x7ffu) ? 1u : 0u;  // inf, nan
    if (emax < kMinExp) {  // all zero, or all below the smallest scale
#pragma unroll
      for (int k = 0; k < 16; ++k) bad |= x[k] != 0.0 ? 1u : 0u;
      emax = 1023u;  // any scale serves zeros
    }
    bad |= (scale8_ok((int)emax + rmin) && scale8_ok((int)emax + rmax)) ? 0u : 1u;
    eh = emax << 20;
    // this thread's row of the seven input digit planes, 8 inputs at a time
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const unsigned e8[8] = {eh, eh, eh, eh, eh, eh, eh, eh};
      split8<kPlaneA>(smem + core_off(t, 8 * c), x + 8 * c, e8);
    }
    // the next tile's inputs load while the tensor cores and the
    // recombination work on this one
    const int64_t bc = b;
    const bool livec = live;
    load_tile(tile + gridDim.x, x, b, live);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    if (__syncthreads_or(done ? 0 : 1)) {
      timed_out = true;
      break;
    }
    if (t == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const unsigned long long bdesc = smem_desc(sB);
#pragma unroll
      for (int j = 0; j < kPlanes; ++j) {
        // input plane j against PTM planes 0 .. 7 - j, whose levels j .. 7 are
        // adjacent accumulator columns; plane 7 is zero (j = 0 clears level 7)
        const unsigned long long adesc = smem_desc(sA + j * kPlaneA);
        const uint32_t idesc = kIdesc0 | ((16u * (uint32_t)(kLevels - j) >> 3) << 17);
        asm volatile(
            "{ .reg .pred q; setp.ne.u32 q, %4, 0; "
            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, q; }" ::"r"(tmem + 16u * (uint32_t)j),
            "l"(adesc), "l"(bdesc), "r"(idesc), "r"(j)
            : "memory");
      }
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
                   : "memory");
    }
    // every thread waits for the MMAs itself (bounded); a time-out ends the
    // block at its next barrier
    {
      uint32_t seen = 0;
      for (long long spin = 0; spin < kSpinLimit && !seen; ++spin)
        asm volatile(
            "{ .reg .pred q; mbarrier.try_wait.parity.shared::cta.b64 q, [%1], %2; selp.u32 %0, 1, 0, q; }"
            : "=r"(seen)
            : "r"(bar), "r"(phase)
            : "memory");
      done = seen != 0u;
    }
    phase ^= 1u;
    __syncwarp();  // the tensor-memory loads below are warp-wide
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    // outputs: rows r = 4c .. 4c + 3 = (ra = c, rb = 0 .. 3), eight levels each
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      uint32_t w[kLevels][4];
#pragma unroll
      for (int l = 0; l < kLevels; ++l) tmem_ld4(tlane + 16u * l + 4u * c, w[l]);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      double y[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        int pr[kLevels / 2];
#pragma unroll
        for (int l = 0; l < kLevels; l += 2)
          pr[l / 2] = level_pair(__uint_as_float(w[l][q]), __uint_as_float(w[l + 1][q]));
        y[q] = scale8(combine8(pr[0], pr[1], pr[2], pr[3]),
                      eh + ((unsigned)srow[4 * c + q] << 20));
      }
      if (livec) {
        if (p.vec_z1) {
          asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p.out + bc + c * p.sao), "d"(y[0]), "d"(y[1]),
                       "d"(y[2]), "d"(y[3])
                       : "memory");
        } else {
#pragma unroll
          for (int q = 0; q < 4; ++q) p.out[bc + c * p.sao + q * p.sbo] = y[q];
        }
      }
    }
    if (bad && livec) {
      // inf / nan inputs or results outside the normal range: this group's
      // outputs again in native FP64
#pragma unroll 1
      for (int r = 0; r < 16; ++r) {
        double a = 0.0;
#pragma unroll 1
        for (int k = 0; k < 16; ++k) {
          const double pk = DEVP ? p.dptm[dev_index(p.dlayout, r, k)] : p.ptm[r][k];
          a = fma(pk, p.in[bc + (k >> 2) * sai + (k & 3) * sbi], a);
        }
        p.out[bc + (r >> 2) * p.sao + (r & 3) * p.sbo] = a;
      }
    }
  }
  timed_out = __syncthreads_or(timed_out || !done ? 1 : 0) != 0;
  if (timed_out && t == 0) {
    if (p.status) atomicOr(p.status, QSGB_DEV_TIMEOUT);
    // bounded wait for the MMAs still in flight before the memory is freed
    uint32_t seen = 0;
    for (long long spin = 0; spin < kSpinLimit && !seen; ++spin)
      asm volatile(
          "{ .reg .pred q; mbarrier.try_wait.parity.shared::cta.b64 q, [%1], %2; selp.u32 %0, 1, 0, q; }"
          : "=r"(seen)
          : "r"(bar), "r"(phase ^ 1u)
          : "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
  }
}

// FP16 bit pattern of an integer |v| <= 2048 (exact).
unsigned short half_bits(int v) {
  if (v == 0) return 0;
  const unsigned sgn = v < 0 ? 0x8000u : 0u;
  unsigned a = (unsigned)std::abs(v);
  int e = 31 - __builtin_clz(a);  // a in [2^e, 2^(e+1))
  const unsigned mant = (a << (10 - e)) & 0x3ffu;
  return (unsigned short)(sgn | ((unsigned)(e + 15) << 10) | mant);
}

// Host split of one PTM row (same fixed point as the device inputs).
void split_row(const double* row, unsigned short (*dig)[16][16], int r, int* row_exp) {
  unsigned emax = 1;
  for (int k = 0; k < 16; ++k) {
    uint64_t b;
    std::memcpy(&b, &row[k], 8);
    const unsigned e = (unsigned)(b >> 52) & 0x7ffu;
    emax = std::max(emax, e == 0u ? 1u : e);
  }
  for (int k = 0; k < 16; ++k) {
    uint64_t b;
    std::memcpy(&b, &row[k], 8);
    const unsigned e = (unsigned)(b >> 52) & 0x7ffu;
    const uint64_t m = ((b & 0xfffffffffffffull) | (e != 0u ? (1ull << 52) : 0ull)) << 4;
    const unsigned s = emax - (e == 0u ? 1u : e);
    uint64_t f = s < 64u ? (m >> s) : 0ull;
    if (b >> 63) f = 0ull - f;
    const uint64_t u = f + kDigitBias;
    for (int j = 0; j < kDigits; ++j) {
      const int v = (int)((u >> (10 * (kDigits - 1 - j))) & 0x3ffu) - 512;
      dig[j][r][k] = half_bits(v);
    }
  }
  row_exp[r] = (int)emax - 1022 - 54;
}

}  // namespace

bool eligible(const double* ptm_host, int kin, int kout) {
  if (kin != 16 || kout != 16) return false;
  for (int i = 0; i < 256; ++i) {
    uint64_t b;
    std::memcpy(&b, &ptm_host[i], 8);
    if (((b >> 52) & 0x7ffu) == 0x7ffu) return false;  // inf, nan
  }
  return true;
}

namespace {

void set_geometry(TcParams& p, const void* in, void* out, uint64_t X, uint64_t Y, uint64_t Z, unsigned* status) {
  p.in = static_cast<const double*>(in);
  p.out = static_cast<double*>(out);
  p.status = status;
  p.n_groups = X * Y * Z;
  p.n_tiles = (p.n_groups + 7) / 8;
  p.div_z = make_fastdiv(Z);
  p.div_y = make_fastdiv(Y);
  p.sbi = (int64_t)Z;
  p.sai = (int64_t)(Y * 4 * Z);
  p.syi = 4 * (int64_t)Z;
  p.sxi = 16 * (int64_t)(Y * Z);
  p.sbo = p.sbi;
  p.sao = p.sai;
  p.syo = p.syi;
  p.sxo = p.sxi;
}

template <bool DEVP>
int launch_umma(TcParams& p, const void* in, void* out, uint64_t Z, cudaStream_t stream) {
  // tcgen05 form: tiles of 128 groups per block, at most 4 blocks per SM
  p.n_tiles = (p.n_groups + kUBlock - 1) / kUBlock;
  const bool contig = Z % kUBlock == 0;
  p.vec_z1 = Z == 1 && (uintptr_t)in % 32 == 0 && (uintptr_t)out % 32 == 0 ? 1 : 0;
  auto kern = contig ? apply16_umma_kernel<true, DEVP> : apply16_umma_kernel<false, DEVP>;
  const int st = allow_dynamic_smem((const void*)kern, kUmmaSmem);
  if (st != QSGB_OK) return st;
  const unsigned grid = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(p.n_tiles, (uint64_t)sm_count() * 4));
  return launch_pdl(kern, grid, kUBlock, kUmmaSmem, stream, p);
}

}  // namespace

int launch(const double* op, const void* in, void* out, uint64_t X, uint64_t Y, uint64_t Z, unsigned* status,
           cudaStream_t stream) {
  static const bool mma_sync = [] {
    const char* v = std::getenv("QSGB_TC_KERNEL");
    return v && std::strcmp(v, "mma_sync") == 0;
  }();
  if (mma_sync) {
    // warp-level form: tiles of 8 groups per warp
    TcWarpParams p{};
    std::memcpy(p.ptm, op, sizeof p.ptm);
    set_geometry(p, in, out, X, Y, Z, status);
    for (int r = 0; r < 16; ++r) split_row(op + 16 * r, p.digits, r, p.row_exp);
    const bool contig = Z % 8 == 0;
    p.pair_store = contig && (uintptr_t)out % 16 == 0 ? 1 : 0;
    const uint64_t blocks = (p.n_tiles + kBlock / 32 - 1) / (kBlock / 32);
    const unsigned grid = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(blocks, (uint64_t)sm_count() * 8));
    if (contig)
      apply16_tc_kernel<true><<<grid, kBlock, 0, stream>>>(p);
    else
      apply16_tc_kernel<false><<<grid, kBlock, 0, stream>>>(p);
    return launch_status();
  }
  TcParams p{};
  std::memcpy(p.ptm, op, sizeof p.ptm);
  set_geometry(p, in, out, X, Y, Z, status);
  return launch_umma<false>(p, in, out, Z, stream);
}

int launch_device(const double* dptm, int layout, const void* in, void* out, uint64_t X, uint64_t Y, uint64_t Z,
                  unsigned* status, cudaStream_t stream) {
  TcParams p{};
  p.dptm = dptm;
  p.dlayout = layout & 3;
  set_geometry(p, in, out, X, Y, Z, status);
  return launch_umma<true>(p, in, out, Z, stream);
}

}  // namespace tc
}  // namespace qsgb
