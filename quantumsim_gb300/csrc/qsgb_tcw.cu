// Dense PTMs larger than 16 x 16 (two qutrits: 81 x 81; a qubit and a qutrit:
// 36 x 36; rectangular ones up to 96 x 96) on the tensor cores.
//
// A dense 81 x 81 PTM costs 81 multiply-adds per output.  The generic kernel
// interprets term lists (1.21 ms on 7 qutrits, 38 MB in and out); float-float
// on the FP32 pipes would be bound by ~10 operations per term.  Here the
// contraction runs in the error-free digit split of qsgb_tc.cu (after Ozaki,
// Ogita, Oishi and Rump, Numer. Algorithms 59, 2012) with digits fitted to the
// longer sums:
//
//  * Each group's inputs and each PTM row are scaled by their largest binary
//    exponent and written as signed fixed-point integers in ND balanced
//    base-512 digits, exact FP16 numbers in [-256, 256]: ND = 6 (54 bits) for
//    FP64 storage, ND = 4 (36 bits) for FP32.  A product of two digits is at
//    most 2^16 and a K = 81 sum at most 2^22.4, so that a level (all digit
//    pairs i + j = L) of up to three pairs (two for K = 96) stays below 2^24,
//    where FP32 sums of integers are exact for any input; the deeper levels
//    hold up to six pairs, and only sums that use their whole range could
//    round there, in the last bit of a level 2^-27 below the first.
//  * The levels are combined in int64 and rounded to the storage type once.
//    The dropped levels (i + j >= ND) bound the error by about
//    5 K 2^-54 max_k |P_rk| max_k |x_k| for FP64 (typically 2^-51 of that
//    product); for FP32 it is far below one rounding of the result.
//  * Groups that hold inf or nan, and FP64 results outside the normal range,
//    are recomputed in plain arithmetic by their own threads.
//
// Work split: one block of 256 threads per SM takes tiles of 128 groups (the M
// of one MMA); two threads share a group, half of the inputs and half of the
// outputs each.  All digit planes of the inputs do not fit shared memory
// beside those of the PTM (147 + 110 KB for 81 x 81), so the input planes, the
// A operand, live in tensor memory: ND x 48 columns, plus two accumulator
// buffers of N columns (288 + 192 of the 512).  The levels are computed one
// after another, L + 1 digit pairs of N = 96 wide MMAs each, alternating the
// two buffers: while the tensor cores work on level L + 1, the threads read
// level L and add it to their int64 sums.
//
// When the less significant target is the last qudit (Z == 1) a thread's group
// is not adjacent to its neighbour's; the tile then goes through shared memory
// both ways, copied in runs of consecutive elements.
#include <algorithm>

#include "qsgb_common.cuh"
#include "qsgb_tc.h"

namespace qsgb {
namespace tc {
namespace {

constexpr int kWBlock = 256;
constexpr int kWGroups = 128;  // groups per tile
constexpr long long kWSpinLimit = 1ll << 26;

struct WideParams {
  const void* in;
  void* out;
  const double* ptm;  // device
  unsigned* status;
  int kin, kout;
  int da_in, db_in, da_out, db_out;
  int layout;        // QSGB_PTM_SWAPPED / QSGB_PTM_TRANSPOSED bits
  int npad, ksteps;  // N of the MMA (multiple of 16), K steps of 16
  int staged;        // Z == 1: tiles through shared memory
  int off_stage;     // shared-memory offset of the staged tile
  uint64_t n_groups, n_tiles;
  FastDiv div_z, div_y;
  int64_t sxi, syi, sai, sbi;
  int64_t sxo, syo, sao, sbo;
};

// shared-memory byte offsets before the PTM planes
constexpr int kWMaxK = 96;
constexpr int kWOffBar = 0;                          // two mbarriers
constexpr int kWOffTmem = 16;                        // tensor-memory base
constexpr int kWOffRow = 32;                         // int[96]: row exponents
constexpr int kWOffEmax = kWOffRow + 4 * kWMaxK;     // unsigned[2][128]: half-group exponents
constexpr int kWOffIn = kWOffEmax + 8 * kWGroups;    // int64[96]: input offsets
constexpr int kWOffOut = kWOffIn + 8 * kWMaxK;       // int64[96]: output offsets
constexpr int kWOffSin = kWOffOut + 8 * kWMaxK;      // int[96]: staged input offsets
constexpr int kWOffSout = kWOffSin + 4 * kWMaxK;     // int[96]: staged output offsets
constexpr int kWOffGin = kWOffSout + 4 * kWMaxK;     // int64[128]: group bases, in
constexpr int kWOffGout = kWOffGin + 8 * kWGroups;   // int64[128]: group bases, out
constexpr int kWOffB = (kWOffGout + 8 * kWGroups + 127) / 128 * 128;

// biased exponent and significand (implicit bit included) of a value
struct Parts {
  unsigned e;
  unsigned neg;
  unsigned long long m;
};
__device__ __forceinline__ Parts parts(double v) {
  const unsigned h = (unsigned)__double2hiint(v);
  Parts r;
  r.e = (h >> 20) & 0x7ffu;
  r.neg = h >> 31;
  r.m = ((unsigned long long)((h & 0xfffffu) | (r.e ? 0x100000u : 0u)) << 32) | (unsigned)__double2loint(v);
  return r;
}
__device__ __forceinline__ Parts parts(float v) {
  const unsigned b = __float_as_uint(v);
  Parts r;
  r.e = (b >> 23) & 0xffu;
  r.neg = b >> 31;
  r.m = (b & 0x7fffffu) | (r.e ? 0x800000u : 0u);
  return r;
}
__device__ __forceinline__ unsigned exp_of(double v) { return ((unsigned)__double2hiint(v) >> 20) & 0x7ffu; }
__device__ __forceinline__ unsigned exp_of(float v) { return (__float_as_uint(v) >> 23) & 0xffu; }
template <typename T>
constexpr unsigned kExpAll = sizeof(T) == 8 ? 0x7ffu : 0xffu;

// F + B: the value as a (9 ND)-bit non-negative integer against exponent emax
// (F = sign * m aligned, |F| < 2^(9 ND - 1); B = 256 in every base-512 digit)
template <int ND, int MBITS>
__device__ __forceinline__ unsigned long long fixed9(const Parts& p, unsigned emax) {
  constexpr int kUp = 9 * ND - 1 - MBITS;  // alignment of an MBITS significand
  constexpr unsigned long long kBias = 256ull * (((1ull << (9 * ND)) - 1ull) / 511ull);
  const unsigned s = emax - (p.e ? p.e : 1u) + (kUp < 0 ? (unsigned)-kUp : 0u);
  const unsigned long long m = kUp > 0 ? p.m << (kUp > 0 ? kUp : 0) : p.m;
  unsigned long long f = s < 64u ? m >> s : 0ull;
  if (p.neg) f = 0ull - f;
  return f + kBias;
}

// FP16x2 of one base-512 digit (bit position pos) of two values: 0x6400 | v
// is 1024 + v; minus 1280
__device__ __forceinline__ unsigned digit9_pair(unsigned long long ua, unsigned long long ub, int pos, unsigned mask) {
  const unsigned a = (unsigned)(ua >> pos) & mask;
  const unsigned b = (unsigned)(ub >> pos) & mask;
  const unsigned r = a | (b << 16) | 0x64006400u;
  unsigned out;
  asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(out) : "r"(r), "r"(0x65006500u));
  return out;
}

// shared-memory matrix descriptor of a K-major plane without swizzling whose
// 8-column (K) slabs of npad rows x 16 bytes follow one another: leading (K)
// byte offset 16 npad, stride (8 rows) 128
__device__ __forceinline__ unsigned long long wide_desc(uint32_t saddr, int npad) {
  return (unsigned long long)((saddr >> 4) & 0x3fffu) | ((unsigned long long)npad << 16) |
         ((unsigned long long)(128 >> 4) << 32) | (1ull << 46);
}

__device__ __forceinline__ void tmem_st4(uint32_t addr, const unsigned (&r)[4]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(r[0]), "r"(r[1]),
               "r"(r[2]), "r"(r[3])
               : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t addr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(addr));
}

// T: storage type; KH: K and N are at most 16 KH, a thread owns 8 KH inputs
// and 8 KH outputs of its group
template <typename T, int KH>
__global__ void __launch_bounds__(kWBlock, 1) apply_wide_kernel(const __grid_constant__ WideParams p) {
  constexpr bool F64 = sizeof(T) == 8;
  constexpr int ND = F64 ? 6 : 4;
  constexpr int MB = F64 ? 53 : 24;
  constexpr int kHalf = 8 * KH;             // inputs (outputs) of a thread
  constexpr int kPlaneCols = 8 * KH;        // tensor-memory columns of an input plane
  constexpr int kDCol = ND * kPlaneCols;    // first accumulator column
  constexpr unsigned kCols = kDCol + 32 * KH <= 256 ? 256u : 512u;
  extern __shared__ __align__(1024) unsigned char smem[];
  const int t = threadIdx.x, warp = t >> 5;
  const int gl = t & (kWGroups - 1), h = t >> 7;  // group of the tile, half
  const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(smem);
  const uint32_t bar = sbase + kWOffBar;
  int* srow = reinterpret_cast<int*>(smem + kWOffRow);
  unsigned* semax = reinterpret_cast<unsigned*>(smem + kWOffEmax);
  int64_t* goff_in = reinterpret_cast<int64_t*>(smem + kWOffIn);
  int64_t* goff_out = reinterpret_cast<int64_t*>(smem + kWOffOut);
  int* soff_in = reinterpret_cast<int*>(smem + kWOffSin);
  int* soff_out = reinterpret_cast<int*>(smem + kWOffSout);
  int64_t* gin = reinterpret_cast<int64_t*>(smem + kWOffGin);
  int64_t* gout = reinterpret_cast<int64_t*>(smem + kWOffGout);
  T* stage = reinterpret_cast<T*>(smem + p.off_stage);
  const T* __restrict__ in = static_cast<const T*>(p.in);
  T* __restrict__ out = static_cast<T*>(p.out);
  const int dbi = p.db_in | 1, dbo = p.db_out | 1;  // odd: staged rows without bank conflicts

  pdl_wait();
  for (int k = t; k < kWMaxK; k += kWBlock) {
    if (k < p.kin) {
      const int ka = k / p.db_in, kb = k - ka * p.db_in;
      goff_in[k] = ka * p.sai + kb * p.sbi;
      soff_in[k] = ka * kWGroups * dbi + kb;
    }
    if (k < p.kout) {
      const int ra = k / p.db_out, rb = k - ra * p.db_out;
      goff_out[k] = ra * p.sao + rb * p.sbo;
      soff_out[k] = ra * kWGroups * dbo + rb;
    }
  }

  // ---- the PTM's digit planes (the B operand), once per block.  A stored
  // offset is a row part plus a column part in every layout.
  auto row_off = [&](int r) {
    const int ra = r / p.db_out, rb = r - ra * p.db_out;
    switch (p.layout & 3) {
      case 0: return r * p.kin;
      case QSGB_PTM_SWAPPED: return (rb * p.da_out + ra) * p.kin;
      case QSGB_PTM_TRANSPOSED: return r;
      default: return rb * p.da_out + ra;
    }
  };
  auto col_off = [&](int k) {
    const int ka = k / p.db_in, kb = k - ka * p.db_in;
    switch (p.layout & 3) {
      case 0: return k;
      case QSGB_PTM_SWAPPED: return kb * p.da_in + ka;
      case QSGB_PTM_TRANSPOSED: return k * p.kout;
      default: return (kb * p.da_in + ka) * p.kout;
    }
  };
  int ptm_bad = 0;
  for (int r = warp; r < p.npad; r += kWBlock / 32) {
    unsigned e = 1u;
    if (r < p.kout) {
      const int ro = row_off(r);
      for (int k = t & 31; k < p.kin; k += 32) e = max(e, exp_of(p.ptm[ro + col_off(k)]));
    }
    for (int o = 16; o > 0; o >>= 1) e = max(e, __shfl_xor_sync(0xffffffffu, e, o));
    if (e == 0x7ffu) ptm_bad = 1;
    if ((t & 31) == 0) srow[r] = (int)e;
  }
  __syncthreads();
  const int plane_b = p.ksteps * 2 * p.npad * 16;  // bytes
  for (int u = t; u < p.npad * p.ksteps * 2; u += kWBlock) {
    const int kc = u / p.npad, r = u - kc * p.npad;  // 8 columns of row r
    unsigned long long f[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int k = kc * 8 + q;
      const double v = (r < p.kout && k < p.kin) ? p.ptm[row_off(r) + col_off(k)] : 0.0;
      f[q] = fixed9<ND, 53>(parts(v), (unsigned)srow[r]);
    }
#pragma unroll
    for (int j = 0; j < ND; ++j) {
      uint4 w;
      const int pos = 9 * (ND - 1 - j);
      const unsigned mask = j == 0 ? 0x3ffu : 0x1ffu;
      w.x = digit9_pair(f[0], f[1], pos, mask);
      w.y = digit9_pair(f[2], f[3], pos, mask);
      w.z = digit9_pair(f[4], f[5], pos, mask);
      w.w = digit9_pair(f[6], f[7], pos, mask);
      *reinterpret_cast<uint4*>(smem + kWOffB + j * plane_b + (kc * p.npad + r) * 16) = w;
    }
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sbase + kWOffTmem),
                 "r"(kCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (t == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar + 8) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  ptm_bad = __syncthreads_or(ptm_bad);
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(smem + kWOffTmem);
  const uint32_t tlane = tmem + ((uint32_t)(32 * (warp & 3)) << 16);
  const uint32_t idesc =
      (1u << 4) | ((uint32_t)(p.npad >> 3) << 17) | ((128u >> 4) << 24);  // D F32, A and B F16, K-major

  // level L: every digit pair i + j = L over all K steps into buffer L & 1
  auto issue_level = [&](int L) {
    const uint32_t d = tmem + (uint32_t)(kDCol + (L & 1) * p.npad);
    for (int i = 0; i <= L; ++i) {  // PTM plane i, input plane L - i
      const uint32_t a0 = tmem + (uint32_t)((L - i) * kPlaneCols);
      const uint32_t b0 = sbase + kWOffB + i * plane_b;
      for (int ks = 0; ks < p.ksteps; ++ks) {
        const unsigned long long bdesc = wide_desc(b0 + ks * 2 * p.npad * 16, p.npad);
        const uint32_t accumulate = (i | ks) ? 1u : 0u;
        asm volatile(
            "{ .reg .pred q; setp.ne.u32 q, %4, 0; "
            "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, q; }" ::"r"(d),
            "r"(a0 + 8u * (uint32_t)ks), "l"(bdesc), "r"(idesc), "r"(accumulate)
            : "memory");
      }
    }
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar + 8 * (L & 1))
                 : "memory");
  };
  uint32_t phases = 0u;  // bit b: parity of barrier b's next completion
  auto wait_bar = [&](int b) -> bool {
    uint32_t done = 0;
    for (long long spin = 0; spin < kWSpinLimit && !done; ++spin)
      asm volatile(
          "{ .reg .pred q; mbarrier.try_wait.parity.shared::cta.b64 q, [%1], %2; selp.u32 %0, 1, 0, q; }"
          : "=r"(done)
          : "r"(bar + 8 * b), "r"((phases >> b) & 1u)
          : "memory");
    phases ^= 1u << b;
    __syncwarp();  // the tensor-memory loads that follow are warp-wide
    return done != 0u;
  };
  // copies of a staged tile: element e of the run of ka (all groups of the
  // tile, db consecutive elements each), thread by thread
  auto staged_copy = [&](bool load, int nv) {
    const int da = load ? p.da_in : p.da_out, db = load ? p.db_in : p.db_out, dbs = load ? dbi : dbo;
    const int64_t sa = load ? p.sai : p.sao;
    const int64_t* g = load ? gin : gout;
    const int di = kWBlock / db, dk = kWBlock - di * db;
    for (int ka = 0; ka < da; ++ka) {
      int i = t / db, kb = t - i * db;
      T* s = stage + ka * kWGroups * dbs;
      while (i < nv) {
        if (load)
          s[i * dbs + kb] = in[g[i] + ka * sa + kb];
        else
          out[g[i] + ka * sa + kb] = s[i * dbs + kb];
        i += di;
        kb += dk;
        if (kb >= db) {
          kb -= db;
          ++i;
        }
      }
    }
  };

  bool timed_out = false;
  for (uint64_t tile = blockIdx.x; tile < p.n_tiles; tile += gridDim.x) {
    const uint64_t gi = tile * kWGroups + gl;
    const bool live = gi < p.n_groups;
    int64_t bi = 0, bo = 0;
    if (live) {
      const uint64_t t1 = fdiv(gi, p.div_z);
      const uint64_t z = gi - t1 * p.div_z.d;
      const uint64_t x = fdiv(t1, p.div_y);
      const uint64_t y = t1 - x * p.div_y.d;
      bi = (int64_t)x * p.sxi + (int64_t)y * p.syi + (int64_t)z;
      bo = (int64_t)x * p.sxo + (int64_t)y * p.syo + (int64_t)z;
    }
    const uint64_t left = p.n_groups - tile * kWGroups;
    const int nv = left < (uint64_t)kWGroups ? (int)left : kWGroups;
    if (p.staged) {
      if (h == 0) {
        gin[gl] = bi;
        gout[gl] = bo;
      }
      __syncthreads();
      staged_copy(true, nv);
      __syncthreads();
    }
    // ---- this thread's inputs, the group's exponent, the digits
    unsigned emax = 1u;
    {
      T x[kHalf];
#pragma unroll
      for (int j = 0; j < kHalf; ++j) {
        const int k = h * kHalf + j;
        x[j] = (T)0;
        if (live && k < p.kin) x[j] = p.staged ? stage[soff_in[k] + gl * dbi] : in[bi + goff_in[k]];
        emax = max(emax, exp_of(x[j]));
      }
      semax[h * kWGroups + gl] = emax;
      __syncthreads();
      emax = max(emax, semax[(h ^ 1) * kWGroups + gl]);
#pragma unroll
      for (int b = 0; b < KH; ++b) {  // 8 inputs: 4 columns of every plane
        unsigned long long u[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) u[q] = fixed9<ND, MB>(parts(x[8 * b + q]), emax);
#pragma unroll
        for (int j = 0; j < ND; ++j) {
          const int pos = 9 * (ND - 1 - j);
          const unsigned mask = j == 0 ? 0x3ffu : 0x1ffu;
          unsigned w[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) w[q] = digit9_pair(u[2 * q], u[2 * q + 1], pos, mask);
          tmem_st4(tlane + (uint32_t)(j * kPlaneCols + h * 4 * KH + 4 * b), w);
        }
      }
    }
    unsigned bad = (ptm_bad || emax == kExpAll<T>) ? 1u : 0u;
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (t == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      issue_level(0);
      issue_level(1);
    }
    // ---- levels: V = sum_L A_L 2^(top - 9 L)
    long long v[kHalf];
#pragma unroll
    for (int j = 0; j < kHalf; ++j) v[j] = 0;
#pragma unroll 1
    for (int L = 0; L < ND; ++L) {
      const bool done = wait_bar(L & 1);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int sh = (F64 ? 40 : 27) - 9 * L;  // F64: 40, 31, 22, 13, 4, -5
      const uint32_t col = tlane + (uint32_t)(kDCol + (L & 1) * p.npad + h * kHalf);
#pragma unroll
      for (int b = 0; b < KH; ++b) {
        if (h * kHalf + 8 * b < p.kout) {
          uint32_t w[8];
          tmem_ld8(col + 8 * b, w);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          if (sh >= 0) {
#pragma unroll
            for (int q = 0; q < 8; ++q) v[8 * b + q] += (long long)__float2int_rn(__uint_as_float(w[q])) << sh;
          } else {
#pragma unroll
            for (int q = 0; q < 8; ++q) v[8 * b + q] += (long long)(__float2int_rn(__uint_as_float(w[q])) >> -sh);
          }
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      if (__syncthreads_or(done ? 0 : 1)) {
        timed_out = true;
        phases ^= 1u << (L & 1);  // this level's commit was not seen
        break;
      }
      if (t == 0 && L + 2 < ND) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        issue_level(L + 2);
      }
    }
    if (timed_out) {
      // bounded waits for the MMAs in flight (this level's and the next
      // one's) before the tensor memory is freed
      if (t == 0 && p.status) atomicOr(p.status, QSGB_DEV_TIMEOUT);
      wait_bar(0);
      wait_bar(1);
      break;
    }
    // ---- results
    const int sc0 = (int)emax - (F64 ? 2100 : 1191);
#pragma unroll
    for (int j = 0; j < kHalf; ++j) {
      const int r = h * kHalf + j;
      if (r < p.kout) {
        T y = (T)0;
        if (v[j] != 0) {
          const int sc = sc0 + srow[r];
          if constexpr (F64) {
            const double d = __ll2double_rn(v[j]);
            const int hi = __double2hiint(d);
            const int e = ((hi >> 20) & 0x7ff) + sc;
            bad |= (e < 1 || e > 2046) ? 1u : 0u;
            y = __hiloint2double(hi + (sc << 20), __double2loint(d));
          } else {
            y = ldexpf(__ll2float_rn(v[j]), sc);
          }
        }
        if (p.staged)
          stage[soff_out[r] + gl * dbo] = y;
        else if (live)
          out[bo + goff_out[r]] = y;
      }
    }
    if (bad && live) {
      // inf or nan inputs or results outside the normal range: this thread's
      // outputs again, in the storage type's plain arithmetic
#pragma unroll 1
      for (int r = h * kHalf; r < (h + 1) * kHalf && r < p.kout; ++r) {
        T a = (T)0;
        const int ro = row_off(r);
#pragma unroll 1
        for (int k = 0; k < p.kin; ++k) a = fma((T)p.ptm[ro + col_off(k)], in[bi + goff_in[k]], a);
        if (p.staged)
          stage[soff_out[r] + gl * dbo] = a;
        else
          out[bo + goff_out[r]] = a;
      }
    }
    if (p.staged) {
      __syncthreads();
      staged_copy(false, nv);
      __syncthreads();  // the tables and the tile are free
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kCols) : "memory");
  }
}

template <typename T, int KH>
int wide_launch(WideParams& p, cudaStream_t stream) {
  constexpr int ND = sizeof(T) == 8 ? 6 : 4;
  const int planes = ND * p.ksteps * 2 * p.npad * 16;
  p.off_stage = kWOffB + planes;
  int smem = p.off_stage;
  if (p.staged) {
    const int run = std::max(p.da_in * (p.db_in | 1), p.da_out * (p.db_out | 1));
    const int bytes = run * kWGroups * (int)sizeof(T);
    if (smem + bytes <= 227 * 1024)
      smem += bytes;
    else
      p.staged = 0;
  }
  const int st = allow_dynamic_smem((const void*)apply_wide_kernel<T, KH>, smem);
  if (st != QSGB_OK) return st;
  const unsigned grid = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(p.n_tiles, (uint64_t)sm_count()));
  return launch_pdl(apply_wide_kernel<T, KH>, grid, kWBlock, smem, stream, p);
}

}  // namespace

int launch_wide(const double* dptm, int layout, const void* in, void* out, int dtype, int da_out, int db_out,
                int da_in, int db_in, uint64_t X, uint64_t Y, uint64_t Z, unsigned* status, cudaStream_t stream) {
  WideParams p{};
  p.in = in;
  p.out = out;
  p.ptm = dptm;
  p.status = status;
  p.kin = da_in * db_in;
  p.kout = da_out * db_out;
  p.da_in = da_in;
  p.db_in = db_in;
  p.da_out = da_out;
  p.db_out = db_out;
  p.layout = layout & 3;
  p.npad = (p.kout + 15) / 16 * 16;
  p.ksteps = (p.kin + 15) / 16;
  p.staged = Z == 1 ? 1 : 0;
  p.n_groups = X * Y * Z;
  p.n_tiles = (p.n_groups + kWGroups - 1) / kWGroups;
  p.div_z = make_fastdiv(Z);
  p.div_y = make_fastdiv(Y);
  p.sbi = (int64_t)Z;
  p.syi = db_in * (int64_t)Z;
  p.sai = (int64_t)(Y * db_in * Z);
  p.sxi = (int64_t)da_in * p.sai;
  p.sbo = (int64_t)Z;
  p.syo = db_out * (int64_t)Z;
  p.sao = (int64_t)(Y * db_out * Z);
  p.sxo = (int64_t)da_out * p.sao;
  const bool small = p.npad <= 48 && p.ksteps <= 3;
  if (dtype == QSGB_F64) return small ? wide_launch<double, 3>(p, stream) : wide_launch<double, 6>(p, stream);
  return small ? wide_launch<float, 3>(p, stream) : wide_launch<float, 6>(p, stream);
}

}  // namespace tc
}  // namespace qsgb
