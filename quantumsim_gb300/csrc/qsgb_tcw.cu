// Dense PTMs larger than 16 x 16 (two qutrits: 81 x 81; a qubit and a qutrit:
// 36 x 36; rectangular ones up to 96 x 96) on the tensor cores.
//
// A dense 81 x 81 PTM costs 81 multiply-adds per output.  The generic kernel
// interprets term lists (1.21 ms on 7 qutrits, 38 MB in and out); float-float
// on the FP32 pipes would be bound by ~10 operations per term.  Here the
// contraction runs in the error-free base-256 digit split of the 16 x 16
// kernel (qsgb_tc.h; after Ozaki, Ogita, Oishi and Rump, Numer. Algorithms 59,
// 2012):
//
//  * Each group's inputs and each PTM row are scaled by their largest binary
//    exponent and written as 55-bit fixed-point integers in seven balanced
//    byte digits, exact FP16 numbers.  A product of two digits is at most 2^14
//    and a K = 96 sum at most 2^20.6, so a level (all digit pairs i + j = L < 8;
//    at most seven pairs) stays below 2^24, where FP32 sums of integers are
//    exact.
//  * Levels pair up in 32-bit integers, are combined in int64 and rounded to
//    the storage type once.  Truncation and the dropped levels bound the error
//    by about 2^-47 max_k |P_rk| max_k |x_k| at K = 81 (typically 2^-53 of that
//    product; for FP32 vectors far below one rounding).
//  * That bound says little about a row that leaves out the group's largest
//    components.  So a PTM with holes (a zero, or an entry below 2^-24 of its
//    row's largest, in a row that is not all zero) is left to the generic
//    kernel, whose rows keep every term's precision: this one, which has the
//    PTM's exponents at hand, then only marks the output, and the generic
//    kernel, always launched behind it, works if it finds the mark.  Without
//    holes every row has a share of its group's largest product.
//  * Groups that hold inf or nan, or whose scales leave the range where every
//    result is a normal number, are recomputed, too: in the storage type's
//    plain arithmetic by their own threads.
//
// Work split: one block of 512 threads per SM takes tiles of 128 groups (the M
// of one MMA); four threads share a group, a quarter of the inputs and of each
// half of the outputs each.  All digit planes of the inputs do not fit shared
// memory beside those of the PTM, so the input planes, the A operand, live in
// tensor memory: 7 x 48 columns, plus three accumulator buffers of 48 columns
// (336 + 144 of the 512).  The outputs are computed in two halves of up to 48
// rows; a group of three levels at a time is accumulated, one buffer each, with
// the MMAs of the three interleaved; while the threads add a group to their
// sums, the tensor cores work on the next.
//
// When the less significant target is the last qudit (Z == 1) a thread's group
// is not adjacent to its neighbour's; the tile then goes through shared memory
// both ways, copied in runs of consecutive elements.
//
// Measured on GB300, dense 81 x 81 on 7 qutrits (461 tiles, 38 MB), in a graph:
// 76 us a pass (2.5 of them the generic kernel that finds no mark), 106 on the
// last two qutrits, against 1200 us in the generic kernel, with 1/60 of its
// error; FP32 vectors 74 us against 227 (with five planes, 39 bits, it was 56:
// but FP32 inputs below 2^-15 of the largest kept fewer bits than they have).
// With zeros in the PTM 977 us, as much as the generic kernel alone.  A first
// form of this kernel (base-512 digits, six levels of N = 96 one after another,
// 256 threads) took 140 us; this one with a level per commit 113 us, and 162 us
// with its MMAs issued by one thread from rolled loops.  What bounds it now:
// latency, over 408 small MMAs and ~175 instructions per output on one block
// of 16 warps; issue is a third busy
// (ncu, 7 qutrits).
#include <algorithm>

#include "qsgb_common.cuh"
#include "qsgb_tc.h"

namespace qsgb {
namespace tc {
namespace {

constexpr int kWBlock = 512;
constexpr int kWWarps = kWBlock / 32;
constexpr int kWGroups = 128;  // groups per tile
constexpr int kWParts = kWBlock / kWGroups;
constexpr int kWBufs = 3;      // accumulator buffers
constexpr long long kWSpinLimit = 1ll << 26;

struct WideParams {
  const void* in;
  void* out;
  const double* ptm;  // device
  unsigned* status;
  int kin, kout;
  int da_in, db_in, da_out, db_out;
  int layout;     // QSGB_PTM_SWAPPED / QSGB_PTM_TRANSPOSED bits
  int nhalf;      // N of the MMA: 16, 32 or 48 (two halves cover kout)
  int ksteps;     // K steps of 16
  int staged;     // Z == 1: tiles through shared memory
  int off_stage;  // shared-memory offset of the staged tile
  uint64_t n_groups, n_tiles;
  FastDiv div_z, div_y;
  int64_t sxi, syi, sai, sbi;
  int64_t sxo, syo, sao, sbo;
};

// shared-memory byte offsets before the PTM planes
constexpr int kWMaxK = 96;
constexpr int kWOffFull = 0;                             // mbarrier: accumulators ready
constexpr int kWOffEmpty = 8;                            // mbarrier: accumulators read
constexpr int kWOffTmem = 16;                            // tensor-memory base
constexpr int kWOffRow = 64;                             // int[96]: row scales
constexpr int kWOffEmax = kWOffRow + 4 * kWMaxK;         // unsigned[4][128]: quarter-group exponents
constexpr int kWOffIn = kWOffEmax + 4 * kWParts * kWGroups;  // int64[96]: input offsets
constexpr int kWOffOut = kWOffIn + 8 * kWMaxK;           // int64[96]: output offsets
constexpr int kWOffSin = kWOffOut + 8 * kWMaxK;          // int[96]: staged input offsets
constexpr int kWOffSout = kWOffSin + 4 * kWMaxK;         // int[96]: staged output offsets
constexpr int kWOffProw = kWOffSout + 4 * kWMaxK;        // int[96]: PTM offsets of rows
constexpr int kWOffPcol = kWOffProw + 4 * kWMaxK;        // int[96]: PTM offsets of columns
constexpr int kWOffGin = kWOffPcol + 4 * kWMaxK;         // int64[128]: group bases, in
constexpr int kWOffGout = kWOffGin + 8 * kWGroups;       // int64[128]: group bases, out
constexpr int kWOffB = (kWOffGout + 8 * kWGroups + 127) / 128 * 128;

__device__ __forceinline__ unsigned exp_of(double v) { return ((unsigned)__double2hiint(v) >> 20) & 0x7ffu; }
__device__ __forceinline__ unsigned exp_of(float v) { return (__float_as_uint(v) >> 23) & 0xffu; }
// a row whose largest entry has biased exponent e has one of exponent `least`
// (zeros and subnormals count 0) that is a hole; inf and nan beside others
// make holes of those
__device__ __forceinline__ bool hole(unsigned least, unsigned e) { return least + 24u < e; }
__device__ __forceinline__ unsigned sign_word(double v) { return (unsigned)__double2hiint(v); }
__device__ __forceinline__ unsigned sign_word(float v) { return __float_as_uint(v); }

// |F| + B against the block exponent e: F has 55 bits; exponent-0 values (zero,
// subnormals) give 0 when the block's exponent is kMinX or more
__device__ __forceinline__ unsigned long long fixed_bytes(double v, unsigned e) {
  return fixed8((unsigned)__double2hiint(v), (unsigned)__double2loint(v), e << 20);
}
__device__ __forceinline__ unsigned long long fixed_bytes(float v, unsigned e) {
  const unsigned b = __float_as_uint(v);
  const unsigned long long m = (unsigned long long)((b & 0x7fffffu) | 0x800000u) << (55 - 24);
  unsigned long long f;
  asm("shr.u64 %0, %1, %2;" : "=l"(f) : "l"(m), "r"(e - ((b >> 23) & 0xffu)));
  return f + kBias8;
}
// shared-memory matrix descriptor of a K-major plane without swizzling whose
// 8-column (K) slabs of `rows` rows x 16 bytes follow one another: leading (K)
// byte offset 16 rows, stride (8 rows) 128
__device__ __forceinline__ unsigned long long wide_desc(uint32_t saddr, int rows) {
  return (unsigned long long)((saddr >> 4) & 0x3fffu) | ((unsigned long long)rows << 16) |
         ((unsigned long long)(128 >> 4) << 32) | (1ull << 46);
}

__device__ __forceinline__ void tmem_st4(uint32_t addr, const unsigned (&r)[4]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(r[0]), "r"(r[1]),
               "r"(r[2]), "r"(r[3])
               : "memory");
}
__device__ __forceinline__ void tmem_ld4(uint32_t addr, float (&r)[4]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
               : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3])
               : "r"(addr));
}

// the digits of 8 inputs: 4 columns of every input plane (stride `plane`)
template <int J = 0>
__device__ __forceinline__ void store_planes(uint32_t addr, uint32_t plane, const unsigned long long (&u)[8],
                                             const Signs (&s)[4]) {
  if constexpr (J < kPlanes) {
    const unsigned w[4] = {digit8_pair<J>(u[0], u[1], s[0]), digit8_pair<J>(u[2], u[3], s[1]),
                           digit8_pair<J>(u[4], u[5], s[2]), digit8_pair<J>(u[6], u[7], s[3])};
    tmem_st4(addr, w);
    store_planes<J + 1>(addr + plane, plane, u, s);
  }
}
template <int J = 0>
__device__ __forceinline__ void store_ptm_planes(unsigned char* dst, int plane, const unsigned long long (&u)[8],
                                                 const Signs (&s)[4]) {
  if constexpr (J < kPlanes) {
    *reinterpret_cast<uint4*>(dst) =
        make_uint4(digit8_pair<J>(u[0], u[1], s[0]), digit8_pair<J>(u[2], u[3], s[1]),
                   digit8_pair<J>(u[4], u[5], s[2]), digit8_pair<J>(u[6], u[7], s[3]));
    store_ptm_planes<J + 1>(dst + plane, plane, u, s);
  }
}

// The mark of a PTM with holes
template <typename T>
__device__ void mark_all(const WideParams& p) {
  for (uint64_t g = (uint64_t)blockIdx.x * kWBlock + threadIdx.x; g < p.n_groups; g += (uint64_t)gridDim.x * kWBlock) {
    const uint64_t t1 = fdiv(g, p.div_z);
    const uint64_t x = fdiv(t1, p.div_y);
    mark_holes(static_cast<T*>(p.out) + (int64_t)x * p.sxo + (int64_t)(t1 - x * p.div_y.d) * p.syo +
               (int64_t)(g - t1 * p.div_z.d));
  }
}

// T: storage type; a thread owns KQ inputs (K <= 4 KQ) and up to KQ outputs
template <typename T, int KQ>
__global__ void __launch_bounds__(kWBlock, 1) apply_wide_kernel(const __grid_constant__ WideParams p) {
  constexpr bool F64 = sizeof(T) == 8;
  constexpr int PL = kPlanes, LV = kLevels;
  constexpr unsigned kExpAll = F64 ? 0x7ffu : 0xffu;
  constexpr unsigned kMinX = F64 ? kMinExp : 56u;  // least block exponent of the inputs
  constexpr int kPlaneCols = 2 * KQ;         // tensor-memory columns of an input plane
  constexpr int kDCol = PL * kPlaneCols;     // first accumulator column
  static_assert(kDCol + kWBufs * 48 <= 512, "tensor memory");
  constexpr unsigned kCols = 512u;
  constexpr int kMaxOut = 12;                // outputs of a thread per half: nhalf / 4
  extern __shared__ __align__(1024) unsigned char smem[];
  const int t = threadIdx.x, warp = t >> 5;
  const int gl = t & (kWGroups - 1), h = t >> 7;  // group of the tile, quarter
  const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(smem);
  const uint32_t full = sbase + kWOffFull, empty = sbase + kWOffEmpty;
  int* srow = reinterpret_cast<int*>(smem + kWOffRow);
  unsigned* semax = reinterpret_cast<unsigned*>(smem + kWOffEmax);
  int64_t* goff_in = reinterpret_cast<int64_t*>(smem + kWOffIn);
  int64_t* goff_out = reinterpret_cast<int64_t*>(smem + kWOffOut);
  int* soff_in = reinterpret_cast<int*>(smem + kWOffSin);
  int* soff_out = reinterpret_cast<int*>(smem + kWOffSout);
  int* prow = reinterpret_cast<int*>(smem + kWOffProw);
  int* pcol = reinterpret_cast<int*>(smem + kWOffPcol);
  int64_t* gin = reinterpret_cast<int64_t*>(smem + kWOffGin);
  int64_t* gout = reinterpret_cast<int64_t*>(smem + kWOffGout);
  T* stage = reinterpret_cast<T*>(smem + p.off_stage);
  const T* in = static_cast<const T*>(p.in);
  T* __restrict__ out = static_cast<T*>(p.out);
  const int dbi = p.db_in | 1, dbo = p.db_out | 1;  // odd: staged rows without bank conflicts
  const int nhalf = p.nhalf, npad = 2 * nhalf;

  // ---- set-up that reads no memory, while the preceding kernel finishes
  if (t < kWMaxK) {
    // element offsets of inputs, outputs, and of the PTM: a stored offset is a
    // row part plus a column part in every layout
    if (t < p.kin) {
      const int ka = t / p.db_in, kb = t - ka * p.db_in;
      goff_in[t] = ka * p.sai + kb * p.sbi;
      soff_in[t] = ka * kWGroups * dbi + kb;
      switch (p.layout & 3) {
        case 0: pcol[t] = t; break;
        case QSGB_PTM_SWAPPED: pcol[t] = kb * p.da_in + ka; break;
        case QSGB_PTM_TRANSPOSED: pcol[t] = t * p.kout; break;
        default: pcol[t] = (kb * p.da_in + ka) * p.kout; break;
      }
    }
    if (t < p.kout) {
      const int ra = t / p.db_out, rb = t - ra * p.db_out;
      goff_out[t] = ra * p.sao + rb * p.sbo;
      soff_out[t] = ra * kWGroups * dbo + rb;
      switch (p.layout & 3) {
        case 0: prow[t] = t * p.kin; break;
        case QSGB_PTM_SWAPPED: prow[t] = (rb * p.da_out + ra) * p.kin; break;
        case QSGB_PTM_TRANSPOSED: prow[t] = t; break;
        default: prow[t] = rb * p.da_out + ra; break;
      }
    }
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sbase + kWOffTmem),
                 "r"(kCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (t == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(full) : "memory");
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(empty), "r"(kWWarps) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();  // this block has its tensor memory before a dependent's may ask for any
  pdl_wait();

  // ---- the PTM's digit planes (the B operand), once per block
  int ptm_bad = 0;
  int holes = 0;
#pragma unroll 3
  for (int r = warp; r < npad; r += kWWarps) {
    unsigned e = 0u, nz = 0u, least = 0x7ffu;
    if (r < p.kout) {
      const int ro = prow[r];
      double v[kWMaxK / 32];
#pragma unroll
      for (int i = 0; i < kWMaxK / 32; ++i) {  // past the last column: the first one again
        const int k = (t & 31) + 32 * i;
        v[i] = p.ptm[ro + pcol[k < p.kin ? k : 0]];
      }
#pragma unroll
      for (int i = 0; i < kWMaxK / 32; ++i) {
        const unsigned ev = exp_of(v[i]);
        e = max(e, ev);
        least = min(least, ev);
        nz |= v[i] != 0.0 ? 1u : 0u;
      }
    }
    e = __reduce_max_sync(0xffffffffu, e);
    nz = __reduce_or_sync(0xffffffffu, nz);
    least = __reduce_min_sync(0xffffffffu, least);
    // inf, nan, or a non-zero row below the smallest scale
    if (e == 0x7ffu || (e < kMinExp && nz)) ptm_bad = 1;
    if (nz && hole(least, e)) holes = 1;
    if (e < kMinExp) e = 1023u;  // any scale serves a row of zeros
    if ((t & 31) == 0) srow[r] = (int)e;
  }
  // (the shuffle tells the compiler that the answer is the warp's: without it the
  // MMAs' operands are not warp-uniform to it, 75 -> 97 us on 7 qutrits)
  const bool leave = __shfl_sync(0xffffffffu, __syncthreads_or(holes), 0) != 0;
  if (leave) mark_all<T>(p);
  const int plane_b = p.ksteps * 2 * npad * 16;  // bytes
  for (int u = leave ? npad * p.ksteps * 2 : t; u < npad * p.ksteps * 2; u += kWBlock) {
    const int kc = u / npad, r = u - kc * npad;  // 8 columns of row r
    double v[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int k = kc * 8 + q;
      v[q] = (r < p.kout && k < p.kin) ? p.ptm[prow[r] + pcol[k]] : 0.0;
    }
    unsigned long long f[8];
    Signs s[4];
#pragma unroll
    for (int q = 0; q < 8; ++q) f[q] = fixed_bytes(v[q], (unsigned)srow[r]);
#pragma unroll
    for (int q = 0; q < 4; ++q) s[q] = signs_of(sign_word(v[2 * q]), sign_word(v[2 * q + 1]));
    store_ptm_planes(smem + kWOffB + (kc * npad + r) * 16, plane_b, f, s);
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  ptm_bad = __syncthreads_or(ptm_bad);
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  int rmin = srow[0], rmax = srow[0];  // row scales, least and greatest
  for (int r = 1; r < p.kout; ++r) {
    rmin = min(rmin, srow[r]);
    rmax = max(rmax, srow[r]);
  }
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(smem + kWOffTmem);
  const uint32_t utmem = __shfl_sync(0xffffffffu, tmem, 0);  // warp-uniform
  const int uwarp = __shfl_sync(0xffffffffu, warp, 0);
  const uint32_t tlane = tmem + ((uint32_t)(32 * (warp & 3)) << 16);
  const uint32_t idesc =
      (1u << 4) | ((uint32_t)(nhalf >> 3) << 17) | ((128u >> 4) << 24);  // D F32, A and B F16, K-major

  bool dead = false;  // a wait of this thread ran out
  auto wait_bar = [&](uint32_t bar, uint32_t parity) {
    uint32_t done = dead ? 1u : 0u;
    for (long long spin = 0; spin < kWSpinLimit && !done; ++spin)
      asm volatile(
          "{ .reg .pred q; mbarrier.try_wait.parity.shared::cta.b64 q, [%1], %2; selp.u32 %0, 1, 0, q; }"
          : "=r"(done)
          : "r"(bar), "r"(parity)
          : "memory");
    dead = dead || !done;
  };
  // Group g of the block (kGroups per half of the outputs, tile after tile):
  // up to three consecutive levels, one accumulator buffer each, their MMAs
  // interleaved: an MMA that adds to the accumulator of the one before waits
  // for it (~130 cycles at N = 48).  The whole of warp 0 runs this, so that the
  // operands stay warp-uniform, and one elected lane issues; loops are unrolled
  // over the K steps, whose descriptors differ by a constant.
  auto issue_group = [&](uint32_t g, int half, int L0) {
    if (g > 0) wait_bar(empty, (g - 1) & 1u);  // the buffers' last contents have been read
    __syncwarp();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const unsigned long long dk = (unsigned long long)(2 * npad);      // per K step, in 16-byte units
    const unsigned long long dp = (unsigned long long)(plane_b >> 4);  // per plane
    uint32_t a0[kWBufs];
    unsigned long long b0[kWBufs];
    int cnt[kWBufs];
#pragma unroll
    for (int l = 0; l < kWBufs; ++l) {  // PTM planes i0 .. i1 with input planes L - i
      const int L = L0 + l;
      const int i0 = L > PL - 1 ? L - (PL - 1) : 0, i1 = L < PL - 1 ? L : PL - 1;
      cnt[l] = L < LV ? i1 - i0 + 1 : 0;
      a0[l] = utmem + (uint32_t)((L - i0) * kPlaneCols);
      b0[l] = wide_desc(sbase + kWOffB + i0 * plane_b + half * nhalf * 16, npad);
    }
    for (int i = 0; i < PL; ++i) {
#pragma unroll
      for (int ks = 0; ks < KQ / 4; ++ks) {
        if (ks < p.ksteps) {
#pragma unroll
          for (int l = 0; l < kWBufs; ++l)
            if (i < cnt[l])
              asm volatile(
                  "{ .reg .pred e, q; elect.sync _|e, 0xffffffff; setp.ne.u32 q, %4, 0; "
                  "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, q; }" ::"r"(utmem + (uint32_t)(kDCol + 48 * l)),
                  "r"(a0[l] + 8u * (uint32_t)ks), "l"(b0[l] + dk * (unsigned)ks), "r"(idesc), "r"(i > 0 || ks > 0 ? 1 : 0)
                  : "memory");
        }
      }
#pragma unroll
      for (int l = 0; l < kWBufs; ++l) {
        a0[l] -= (uint32_t)kPlaneCols;
        b0[l] += dp;
      }
    }
    asm volatile(
        "{ .reg .pred e; elect.sync _|e, 0xffffffff; "
        "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0]; }" ::"r"(full)
        : "memory");
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

  constexpr int kGroups = (LV + kWBufs - 1) / kWBufs;  // of levels, per half
  uint32_t group = 0;  // groups issued so far
  for (uint64_t tile = leave ? p.n_tiles : blockIdx.x; tile < p.n_tiles; tile += gridDim.x) {
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
    unsigned emax = 0u;
    {
      T x[KQ];
#pragma unroll
      for (int j = 0; j < KQ; ++j) {
        const int k = h * KQ + j;
        x[j] = (T)0;
        if (live && k < p.kin) x[j] = p.staged ? stage[soff_in[k] + gl * dbi] : in[bi + goff_in[k]];
      }
#pragma unroll
      for (int j = 0; j < KQ; ++j) emax = max(emax, exp_of(x[j]));
      if (emax < kMinX) {  // bit 16: a non-zero value
#pragma unroll
        for (int j = 0; j < KQ; ++j) emax |= x[j] != (T)0 ? 0x10000u : 0u;
      }
      semax[h * kWGroups + gl] = emax;
      __syncthreads();
      unsigned some = 0u;
      emax = 0u;
#pragma unroll
      for (int q = 0; q < kWParts; ++q) {
        const unsigned e = semax[q * kWGroups + gl];
        some |= e;
        emax = max(emax, e & 0xffffu);
      }
      // below the smallest scale: recomputed; all zero: any scale serves
      if (emax < kMinX) emax = some >= 0x10000u ? kExpAll : (F64 ? 1023u : 127u);
      if (h * KQ < 16 * p.ksteps) {
#pragma unroll
        for (int b = 0; b < KQ / 8; ++b) {  // 8 inputs: 4 columns of every plane
          unsigned long long u[8];
          Signs s[4];
#pragma unroll
          for (int q = 0; q < 8; ++q) u[q] = fixed_bytes(x[8 * b + q], emax);
#pragma unroll
          for (int q = 0; q < 4; ++q) s[q] = signs_of(sign_word(x[8 * b + 2 * q]), sign_word(x[8 * b + 2 * q + 1]));
          store_planes(tlane + (uint32_t)((h * KQ + 8 * b) / 2), (uint32_t)kPlaneCols, u, s);
        }
      }
    }
    // inf, nan, too small a scale, or results that may leave the normal range
    bool bad = ptm_bad || emax == kExpAll;
    // (|v| < 2^63 here, 2 bits more than scale8_ok allows for)
    if (F64) bad = bad || !scale8_ok((int)emax + rmin - kScale8) || !scale8_ok((int)emax + rmax + 2 - kScale8);
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (uwarp == 0) issue_group(group, 0, 0);
    // ---- the outputs, half after half, level group after level group
#pragma unroll 1
    for (int half = 0; half < 2; ++half) {
      long long v[kMaxOut];
      int pr[kMaxOut];
#pragma unroll
      for (int j = 0; j < kMaxOut; ++j) v[j] = 0;
      const int col = h * (nhalf >> 2);  // this thread's first column of the half
#pragma unroll
      for (int G = 0; G < kGroups; ++G) {
        wait_bar(full, group & 1u);
        __syncwarp();  // the tensor-memory loads are warp-wide
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        float w[kWBufs][3][4];
#pragma unroll
        for (int l = 0; l < kWBufs; ++l)
#pragma unroll
          for (int c = 0; c < 3; ++c)
            if (G * kWBufs + l < LV && 16 * c < nhalf)
              tmem_ld4(tlane + (uint32_t)(kDCol + 48 * l + col + 4 * c), w[l][c]);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        if ((t & 31) == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(empty) : "memory");
        ++group;
        if (uwarp == 0 && (G + 1 < kGroups || half == 0))
          issue_group(group, G + 1 < kGroups ? half : 1, G + 1 < kGroups ? (G + 1) * kWBufs : 0);
        // levels 0 and 1 stay below 2^22: the magic number; F2I for the others
#pragma unroll
        for (int l = 0; l < kWBufs; ++l) {
          const int L = G * kWBufs + l;
          if (L < LV) {
#pragma unroll
            for (int j = 0; j < kMaxOut; ++j) {
              const float a = w[l][j >> 2][j & 3];
              const int i = L <= 1 ? (int)(level_bits(a) - kMagic) : __float2int_rn(a);
              if (L == 6)  // seven pairs of K = 96 may fill 32 bits: scaled first
                pr[j] = i >> 6;
              else if (L == 7)
                pr[j] += i >> 14;
              else
                pr[j] = (L & 1) ? pr[j] + i : i << 8;
              // V = sum_L A_L 2^(top - 8 L)
              if (L == 1) v[j] = (long long)pr[j] << 34;
              if (L == 3) v[j] += (long long)pr[j] * 262144ll;
              if (L == 5) v[j] += (long long)pr[j] * 4ll;
              if (L == 7) v[j] += (long long)pr[j];
            }
          }
        }
      }
      // ---- results of this half
#pragma unroll
      for (int j = 0; j < kMaxOut; ++j) {
        const int r = half * nhalf + col + j;
        if (j < (nhalf >> 2) && r < p.kout) {
          T y;
          if constexpr (F64)
            y = scale8(v[j], (unsigned)((int)emax + srow[r] - kScale8) << 20);
          else
            y = ldexpf(__ll2float_rn(v[j]), (int)emax + srow[r] - (kScale8 - 1023 + 127));
          if (p.staged)
            stage[soff_out[r] + gl * dbo] = y;
          else if (live)
            out[bo + goff_out[r]] = y;
        }
      }
      if (bad && live) {
        // this thread's outputs again, in the storage type's plain arithmetic
#pragma unroll 1
        for (int j = 0; j < (nhalf >> 2); ++j) {
          const int r = half * nhalf + col + j;
          if (r >= p.kout) break;
          T a = (T)0;
#pragma unroll 1
          for (int k = 0; k < p.kin; ++k) a = fma((T)p.ptm[prow[r] + pcol[k]], in[bi + goff_in[k]], a);
          if (p.staged)
            stage[soff_out[r] + gl * dbo] = a;
          else
            out[bo + goff_out[r]] = a;
        }
      }
    }
    if (__syncthreads_or(dead ? 1 : 0)) {
      dead = true;
      break;
    }
    if (p.staged) {
      staged_copy(false, nv);
      __syncthreads();  // the tables and the tile are free
    }
  }
  if (dead) {
    // a wait ran out: bounded waits for the MMAs that may be in flight before
    // the tensor memory is freed
    if (t == 0 && p.status) atomicOr(p.status, QSGB_DEV_TIMEOUT);
    dead = false;
    wait_bar(full, group & 1u);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kCols) : "memory");
  }
}

template <typename T, int KQ>
int wide_launch(WideParams& p, cudaStream_t stream) {
  const int planes = kPlanes * p.ksteps * 2 * 2 * p.nhalf * 16;
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
  const int st = allow_dynamic_smem((const void*)apply_wide_kernel<T, KQ>, smem);
  if (st != QSGB_OK) return st;
  const unsigned grid = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(p.n_tiles, (uint64_t)sm_count()));
  return launch_pdl(apply_wide_kernel<T, KQ>, grid, kWBlock, smem, stream, p);
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
  p.nhalf = (p.kout + 31) / 32 * 16;
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
  const bool small = p.ksteps <= 4;
  if (dtype == QSGB_F64) return small ? wide_launch<double, 16>(p, stream) : wide_launch<double, 24>(p, stream);
  return small ? wide_launch<float, 16>(p, stream) : wide_launch<float, 24>(p, stream);
}

}  // namespace tc
}  // namespace qsgb
