// Batched forward + adjoint of many independent circuits in one persistent
// launch (FP32 Pauli vectors, FP64 reductions).
//
// Work model: a program is a sequence of stages; each stage holds work items
// (one op of one instance on a range of groups or elements).  Items of a
// stage belong to independent instances, so persistent blocks take them from
// the stage's atomic counter in any order; a grid barrier separates stages.
// Small instances finish in one item, large ones are split into tiles, so a
// few hundred blocks keep busy across instances of 4..16 qubits.
//
// Adjoint without stored intermediates: an op's input state is rebuilt from
// its output with the inverse PTM (rotations, controlled phases and damping
// are invertible and well conditioned), while the adjoint state moves back
// through P^T; the host refreshes the state from checkpoints every few
// layers.  One ADJOINT item therefore reads x_out and g_out once, writes x_in
// and g_in, and accumulates its share of dL/dP = sum g_out (x) x_in.  The
// two-qubit ADJOINT does its three small products per 32-group warp tile on
// the warp-level tensor cores (mma.sync m16n8k8, TF32 operands split hi/lo);
// every other body runs on the FP32 pipes.  An op here is whatever the host
// planned as a unit (a CZ may carry the rotations before it).
//
// Every grid barrier polls a bounded number of times; on expiry the kernel
// flags QSGB_DEV_TIMEOUT and all blocks return.
#include <cooperative_groups.h>

#include <algorithm>

#include "qsgb_common.cuh"

namespace qsgb {
namespace {

constexpr int kBatchBlock = 256;
// floats per row of a warp's 16 x 32 adjoint tiles: 32 groups + 4 of
// padding, so that the fragment loads and the 16-byte stores of X_in in the
// two-qubit ADJOINT fall in distinct banks
constexpr int kAdjStride = 36;
constexpr int kWarps = kBatchBlock / 32;

struct BatchSmem {
  float P[256];
  float PT[256];  // P transposed (ADJOINT: g_in = P^T g_out)
  float Pi[256];
  // two-qubit ADJOINT tiles, one pair per warp: x (X_in) and g (G_out), 16
  // rows of kAdjStride floats; reused for the FP64 cross-warp sums of the dP
  // partials
  union {
    struct {
      float g[kWarps][16 * kAdjStride];
      float x[kWarps][16 * kAdjStride];
    } t;
    double red[kWarps][256];
  } u __attribute__((aligned(16)));
  double acc[kBatchBlock][16];  // per-thread FP64 dP partials (ADJOINT)
  int item;
  int ok;
  double lsum[kBatchBlock / 32];
};

}  // namespace

// The block's dynamic shared memory, at namespace scope so that the op
// bodies (separate functions) address it as shared memory.
extern __shared__ __align__(16) unsigned char batch_dsm[];

namespace {

__device__ __forceinline__ BatchSmem& smem() { return *reinterpret_cast<BatchSmem*>(batch_dsm); }

__device__ __forceinline__ volatile uint32_t* vol(uint32_t* p) { return p; }

// Grid barrier (sense by generation).  Returns false when the wait expired
// or another block aborted.
__device__ bool grid_barrier(uint32_t* count, uint32_t* gen, uint32_t* abort_flag, long long limit,
                             unsigned* status, BatchSmem& sm) {
  __syncthreads();
  if (threadIdx.x == 0) {
    sm.ok = 1;
    const uint32_t g0 = *vol(gen);
    __threadfence();
    if (atomicAdd(count, 1u) == gridDim.x - 1) {
      atomicExch(count, 0u);
      __threadfence();
      atomicAdd(gen, 1u);
    } else {
      long long it = 0;
      while (*vol(gen) == g0) {
        if (*vol(abort_flag) || ++it > limit) {
          sm.ok = 0;
          if (it > limit && status) atomicOr(status, QSGB_DEV_TIMEOUT);
          atomicExch(abort_flag, 1u);
          break;
        }
        __nanosleep(64);
      }
    }
    __threadfence();
  }
  __syncthreads();
  return sm.ok != 0;
}

// ---------------------------------------------------------------- geometry
struct Geo {
  int k;          // 4 or 16 inputs per group
  int lz, ly;     // log2 of Z and Y (powers of 4)
};

__device__ __forceinline__ Geo geometry(int n, int q0, int q1) {
  Geo g;
  if (q1 < 0) {
    g.k = 4;
    g.lz = 2 * (n - 1 - q0);
    g.ly = 0;
  } else {
    g.k = 16;
    g.lz = 2 * (n - 1 - q1);
    g.ly = 2 * (q1 - q0 - 1);
  }
  return g;
}

// base element of group `gi` and offset of input k
__device__ __forceinline__ int64_t group_base(const Geo& g, int64_t gi) {
  const int64_t z = gi & ((1ll << g.lz) - 1);
  const int64_t t = gi >> g.lz;
  if (g.k == 4) return ((t << (g.lz + 2)) | z);
  const int64_t y = t & ((1ll << g.ly) - 1);
  const int64_t x = t >> g.ly;
  return (x << (g.lz + g.ly + 4)) + (y << (g.lz + 2)) + z;
}

// (32-bit: instances have at most 15 qubits, so an offset inside a group
// stays below 3 * 4^14; fewer registers than 64-bit addresses per input)
template <int K>
__device__ __forceinline__ int in_offset(const Geo& g, int k) {
  if (K == 4) return k << g.lz;
  return ((k >> 2) << (g.lz + g.ly + 2)) + ((k & 3) << g.lz);
}

// ---------------------------------------------------------------- items
// Vectorised in-place apply.  Z >= 4: a thread takes V consecutive groups
// (z .. z+V-1, 16- or 8-byte accesses per input); Z == 1: the K inputs of a
// group along the less significant qubit are contiguous (16-byte accesses).
// The per-op bodies are not inlined into the kernel: each gets its own
// register allocation under the kernel's 128-register cap, so one op's
// pressure does not spill into the others.
template <int K>
__device__ __noinline__ void apply_vec(float* __restrict__ x, const Geo& geo, int64_t beg, int64_t end, const float* P) {
  if (geo.lz >= 2) {
    constexpr int V = 4;
    for (int64_t gi = beg + (int64_t)threadIdx.x * V; gi < end; gi += (int64_t)blockDim.x * V) {
      const int64_t b = group_base(geo, gi);
      float v[K][V];
#pragma unroll
      for (int k = 0; k < K; ++k) {
        const float* src = x + b + in_offset<K>(geo, k);
        if (V == 4) {
          const float4 t = *reinterpret_cast<const float4*>(src);
          v[k][0] = t.x; v[k][1] = t.y; v[k][2 % V] = t.z; v[k][3 % V] = t.w;
        } else {
          const float2 t = *reinterpret_cast<const float2*>(src);
          v[k][0] = t.x; v[k][1] = t.y;
        }
      }
#pragma unroll 1
      for (int r = 0; r < K; ++r) {
        float y[V];
#pragma unroll
        for (int l = 0; l < V; ++l) y[l] = 0.f;
#pragma unroll
        for (int k = 0; k < K; ++k) {
          const float pk = P[r * K + k];
#pragma unroll
          for (int l = 0; l < V; ++l) y[l] = fmaf(pk, v[k][l], y[l]);
        }
        float* dst = x + b + in_offset<K>(geo, r);
        if (V == 4)
          *reinterpret_cast<float4*>(dst) = make_float4(y[0], y[1], y[2 % V], y[3 % V]);
        else
          *reinterpret_cast<float2*>(dst) = make_float2(y[0], y[1]);
      }
    }
  } else {
    for (int64_t gi = beg + threadIdx.x; gi < end; gi += blockDim.x) {
      const int64_t b = group_base(geo, gi);
      float v[K], y[K];
#pragma unroll
      for (int k = 0; k < K; k += 4) {
        const float4 t = *reinterpret_cast<const float4*>(x + b + in_offset<K>(geo, k));
        v[k] = t.x; v[k + 1] = t.y; v[k + 2] = t.z; v[k + 3] = t.w;
      }
#pragma unroll
      for (int r = 0; r < K; ++r) {
        float a = 0.f;
#pragma unroll
        for (int k = 0; k < K; ++k) a = fmaf(P[r * K + k], v[k], a);
        y[r] = a;
      }
#pragma unroll
      for (int k = 0; k < K; k += 4)
        *reinterpret_cast<float4*>(x + b + in_offset<K>(geo, k)) = make_float4(y[k], y[k + 1], y[k + 2], y[k + 3]);
    }
  }
}

// FP32 sums into FP64 ones (the first ones of an item as they are).  On GB300 a
// warp's conversion or addition in FP64 takes ~62 cycles of its sub-partition:
// an item of four tiles per warp is not folded a second time at its end.
// (Conversions by integer operations on the bit patterns: 58.2 -> 59.0 ms for
// the step of 64 10-qubit circuits.)
template <int N>
__device__ __forceinline__ void fold_fp64(double* acc, float (&v)[N], bool first) {
#pragma unroll
  for (int e = 0; e < N; ++e) {
    acc[e] = first ? (double)v[e] : acc[e] + (double)v[e];
    v[e] = 0.f;
  }
}

// One-qubit adjoint (pairs of groups when Z >= 4, one contiguous group when
// Z == 1): x = P^-1 x, g = P^T g, and
// dP[r][k] = sum g_out[r] x_in[k] accumulated in FP32 registers, folded to
// FP64 every 16 groups, reduced over the block and written to dst (16
// doubles).
__device__ __noinline__ void adjoint1_vec(float* __restrict__ x, float* __restrict__ gv, const Geo& geo, int64_t beg,
                             int64_t end, const float* P, const float* Pi, BatchSmem& sm, double* __restrict__ dst) {
  float acc[16];
  double* accd = sm.acc[threadIdx.x];  // FP64 running sums live in shared memory
#pragma unroll
  for (int e = 0; e < 16; ++e) acc[e] = 0.f;
  auto one = [&](const float* xo, const float* go, float* xi, float* gn) {
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      float a = 0.f, c = 0.f;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        a = fmaf(Pi[r * 4 + k], xo[k], a);
        c = fmaf(P[k * 4 + r], go[k], c);
      }
      xi[r] = a;
      gn[r] = c;
    }
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int k = 0; k < 4; ++k) acc[r * 4 + k] = fmaf(go[r], xi[k], acc[r * 4 + k]);
  };
  int since = 0;
  bool first = true;
  if (geo.lz >= 2) {  // pairs of groups (z, z+1): 8-byte accesses
    for (int64_t gi = beg + (int64_t)threadIdx.x * 2; gi < end; gi += (int64_t)blockDim.x * 2) {
      const int64_t b = group_base(geo, gi);
      float xv[4][2], gvv[4][2];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float2 a = *reinterpret_cast<const float2*>(x + b + in_offset<4>(geo, k));
        const float2 c = *reinterpret_cast<const float2*>(gv + b + in_offset<4>(geo, k));
        xv[k][0] = a.x; xv[k][1] = a.y;
        gvv[k][0] = c.x; gvv[k][1] = c.y;
      }
      float xi[4][2], gn[4][2];
#pragma unroll
      for (int l = 0; l < 2; ++l) {
        const float xo[4] = {xv[0][l], xv[1][l], xv[2][l], xv[3][l]};
        const float go[4] = {gvv[0][l], gvv[1][l], gvv[2][l], gvv[3][l]};
        float a[4], c[4];
        one(xo, go, a, c);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          xi[r][l] = a[r];
          gn[r][l] = c[r];
        }
      }
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        *reinterpret_cast<float2*>(x + b + in_offset<4>(geo, r)) = make_float2(xi[r][0], xi[r][1]);
        *reinterpret_cast<float2*>(gv + b + in_offset<4>(geo, r)) = make_float2(gn[r][0], gn[r][1]);
      }
      if (++since == 8) {
        fold_fp64(accd, acc, first);
        first = false;
        since = 0;
      }
    }
  } else {
    for (int64_t gi = beg + threadIdx.x; gi < end; gi += blockDim.x) {
      const int64_t b = group_base(geo, gi);
      const float4 a = *reinterpret_cast<const float4*>(x + b);
      const float4 c = *reinterpret_cast<const float4*>(gv + b);
      const float xo[4] = {a.x, a.y, a.z, a.w};
      const float go[4] = {c.x, c.y, c.z, c.w};
      float xi[4], gn[4];
      one(xo, go, xi, gn);
      *reinterpret_cast<float4*>(x + b) = make_float4(xi[0], xi[1], xi[2], xi[3]);
      *reinterpret_cast<float4*>(gv + b) = make_float4(gn[0], gn[1], gn[2], gn[3]);
      if (++since == 16) {
        fold_fp64(accd, acc, first);
        first = false;
        since = 0;
      }
    }
  }
  if (since || first) fold_fp64(accd, acc, first);
  // block reduction: over a warp by exchanges that halve the entries a lane
  // holds (16 FP64 additions a lane; a butterfly per entry, the same sums,
  // takes 80), then across warps in shared memory.  With the fold above: 64
  // circuits of 10 qubits 64.4 -> 58.2 ms, 20 circuits of 4 to 12 93.6 -> 90.8.
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double v[16];
#pragma unroll
  for (int e = 0; e < 16; ++e) v[e] = accd[e];
#pragma unroll
  for (int h = 8; h > 0; h >>= 1) {
    const bool up = (lane & (2 * h)) != 0;  // keeps the upper half
#pragma unroll
    for (int e = 0; e < h; ++e) {
      const double send = up ? v[e] : v[e + h], keep = up ? v[e + h] : v[e];
      v[e] = keep + __shfl_xor_sync(0xffffffffu, send, 2 * h);
    }
  }
  v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
  if ((lane & 1) == 0) sm.u.red[w][lane >> 1] = v[0];
  __syncthreads();
  if (threadIdx.x < 16) {
    double s = 0.0;
    for (int ww = 0; ww < (int)(blockDim.x >> 5); ++ww) s += sm.u.red[ww][threadIdx.x];
    dst[threadIdx.x] = s;
  }
  __syncthreads();
}

// ---- warp-level tensor-core helpers (mma.sync m16n8k8, TF32 operands)
// The FP32 value x is carried as hi + lo, both TF32 (cvt.rna keeps the top
// 11 significant bits): hi = tf32(x), lo = tf32(x - hi).  A product is taken
// as A_lo B_hi + A_hi B_lo + A_hi B_hi (the lo * lo term is below the
// representation error of the split, ~2^-22 relative), accumulated in FP32.
__device__ __forceinline__ uint32_t to_tf32(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return r;
}

__device__ __forceinline__ void split_tf32(float x, uint32_t& hi, uint32_t& lo) {
  hi = to_tf32(x);
  lo = to_tf32(x - __uint_as_float(hi));
}

// d += a * b for one m16n8k8 tile: a = 16 x 8 (row-major fragment a0..a3),
// b = 8 x 8 (column fragment b0, b1), d = 16 x 8 FP32
__device__ __forceinline__ void mma_tf32(float* d, const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
      "{%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// d += A B with A given as split fragments (ah, al) and B as FP32 values
__device__ __forceinline__ void mma3(float* d, const uint32_t (&ah)[4], const uint32_t (&al)[4], float b0,
                                     float b1) {
  uint32_t bh0, bl0, bh1, bl1;
  split_tf32(b0, bh0, bl0);
  split_tf32(b1, bh1, bl1);
  mma_tf32(d, al, bh0, bh1);
  mma_tf32(d, ah, bl0, bl1);
  mma_tf32(d, ah, bh0, bh1);
}

// 32 bytes (8 floats), 32-byte aligned
__device__ __forceinline__ void store8(float* dst, const float (&v)[8]) {
  asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst), "f"(v[0]), "f"(v[1]), "f"(v[2]),
               "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
               : "memory");
}

// Two-qubit ADJOINT on the warp-level tensor cores.  A warp takes tiles of 32
// consecutive groups:
//   X_in = P^-1 X_out and G_in = P^T G_out   (M 16, N 32, K 16: 8 mma each)
//   dP  += G_out X_in^T                      (M 16, N 16, K 32: 8 mma)
// each mma in 3xTF32 (24 per product).  Lane l = (gid, tig) = (l / 4, l % 4)
// holds components 4 j + tig (j = 0..3) of column gid of every n-tile as right
// operands, and gets components row(gid, 0 / 1) of columns 2 tig and 2 tig + 1.
// Which group a column stands for, and which component a row, is free, and is
// chosen for both to be whole runs of memory, so that the first two products
// need no exchange between lanes:
//  * Z > 1: column c of n-tile nt is group 4 c + nt.  The lane's four groups
//    of a component are 16 bytes, its eight results 32.
//  * Z == 1: group 8 nt + c / 2 + 4 (c % 2), rows 2 gid and 2 gid + 1.  A load
//    of the warp is 128 consecutive bytes, a lane's results are pairs.
// G_out and X_in go through the warp's two 16 x 32 tiles in shared memory
// ([component][group]) for the third product alone, which sums over groups.
// Its fragments are carried in FP32 over 4 tiles, then folded into the
// thread's FP64 sums in shared memory; at the end the warps' sums are added
// in a fixed order and written to dst (256 doubles).
//
// Bound by the latency of its loads on 16 warps per SM.  With a group per lane
// and every product's operands and results staged (96 shared-memory accesses
// and 64 global ones of 4 bytes per tile, against 56 and 12 here) the step of
// 512 circuits took 1.198 s, that of 20 circuits 106.4 ms; here 1.087 s and
// 96.5 ms, with the same bits (G_out read a second time in the third product's
// order instead of staged: 101.7 ms and other FP32 sums).
__device__ __noinline__ void adjoint2_warp(float* __restrict__ x, float* __restrict__ gv, const Geo& geo, int64_t beg,
                                           int64_t end, double* __restrict__ dst) {
  constexpr int K = 16;
  constexpr int S = kAdjStride;
  BatchSmem& sm = smem();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nwarps = blockDim.x >> 5;
  const int gid = lane >> 2, tig = lane & 3;
  float* ta = sm.u.t.x[warp];  // X_in
  float* tb = sm.u.t.g[warp];  // G_out
  const int lz = geo.lz, la = geo.lz + geo.ly + 2;  // log2 strides of b and a (component 4 a + b)
  const bool last = lz == 0;
  const bool aligned = (((uintptr_t)x | (uintptr_t)gv) & 31) == 0;
  auto column = [&](int nt, int c) { return last ? 8 * nt + (c >> 1) + 4 * (c & 1) : 4 * c + nt; };
  const int r0 = last ? 2 * gid : gid, r1 = last ? 2 * gid + 1 : gid + 8;
  // A fragments of P^-1 and P^T (two k-steps each), split into TF32 hi / lo
  uint32_t pih[2][4], pil[2][4], pth[2][4], ptl[2][4];
#pragma unroll
  for (int ks = 0; ks < 2; ++ks)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int e = ((i & 1) ? r1 : r0) * K + 8 * ks + 4 * (i >> 1) + tig;
      split_tf32(sm.Pi[e], pih[ks][i], pil[ks][i]);
      split_tf32(sm.PT[e], pth[ks][i], ptl[ks][i]);
    }
  float dp[8];  // dP fragments: [4 nb + i], rows gid, gid + 8; columns 8 nb + 2 tig (+1)
#pragma unroll
  for (int i = 0; i < 8; ++i) dp[i] = 0.f;
  double* acc = sm.acc[threadIdx.x];  // FP64 running sums in shared memory
  int tiles = 0;
  // offsets inside a group: component tig, the result rows
  const int in0 = tig << lz, out0 = in_offset<K>(geo, r0), out1 = in_offset<K>(geo, r1);
  for (int64_t t0 = beg + (int64_t)warp * 32; t0 < end; t0 += (int64_t)nwarps * 32) {
    // four consecutive groups along z per access, or eight (32 bytes); else
    // group by group (Z == 1, the end of an item, a start inside a run)
    const bool full = t0 + 32 <= end;
    const bool quads = full && lz >= 2 && (t0 & 3) == 0;
    const bool wide = quads && aligned && lz >= 4 && (t0 & 7) == 0;
    float xv[4][4], gq[4][4];  // [component 4 j + tig][n-tile]
    if (quads) {
      const int64_t b = group_base(geo, t0 + 4 * gid) + in0;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float4 u = *reinterpret_cast<const float4*>(x + b + (j << la));
        const float4 w = *reinterpret_cast<const float4*>(gv + b + (j << la));
        xv[j][0] = u.x; xv[j][1] = u.y; xv[j][2] = u.z; xv[j][3] = u.w;
        gq[j][0] = w.x; gq[j][1] = w.y; gq[j][2] = w.z; gq[j][3] = w.w;
      }
    } else {
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) {
        const int64_t gi = t0 + column(nt, gid);
        const bool have = gi < end;
        const int64_t b = (have ? group_base(geo, gi) : 0) + in0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          xv[j][nt] = have ? x[b + (j << la)] : 0.f;
          gq[j][nt] = have ? gv[b + (j << la)] : 0.f;
        }
      }
    }
    {
      // this warp's next tile into L2 while the current one is computed (the
      // loads are bound by their latency): lane l takes tensor l / 16 and, for
      // Z >= 16, component l % 16 at the tile's first and last group (one
      // 128-byte run each when the groups are consecutive along z); for Z == 1
      // and Z == 4, where a row of the tile's 32 groups is 512 contiguous bytes
      // unless they change x, line l % 4 of chunk row (l / 4) % 4.  Addresses are those of groups inside the item.
      const int64_t tn = t0 + (int64_t)nwarps * 32;
      if (tn < end) {
        const float* base = (lane < 16) ? x : gv;
        if (lz >= 4) {
          const int off = in_offset<K>(geo, lane & 15);
          const int64_t fin = tn + 31 < end ? tn + 31 : end - 1;
          asm volatile("prefetch.global.L2 [%0];" ::"l"(base + group_base(geo, tn) + off));
          asm volatile("prefetch.global.L2 [%0];" ::"l"(base + group_base(geo, fin) + off));
        } else if (tn + 31 < end) {
          const int64_t b0 = group_base(geo, tn), b1 = group_base(geo, tn + 31);
          if (b1 - b0 == (last ? 31 * 4 : 7 * 16 + 3)) {  // the 32 groups share x: rows are contiguous
            const int q = (lane >> 2) & 3;
            asm volatile("prefetch.global.L2 [%0];" ::"l"(base + b0 + in_offset<K>(geo, 4 * q) + 32 * (lane & 3)));
          }
        }
      }
    }
    // G_out into its tile
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float* row = tb + (4 * j + tig) * S;
      if (last) {
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) row[column(nt, gid)] = gq[j][nt];
      } else {
        *reinterpret_cast<float4*>(row + 4 * gid) = make_float4(gq[j][0], gq[j][1], gq[j][2], gq[j][3]);
      }
    }
    // X_in = P^-1 X_out: four n-tiles of 8 groups
    float xi[4][4], gn[4][4];
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
#pragma unroll
      for (int i = 0; i < 4; ++i) xi[nt][i] = 0.f;
#pragma unroll
      for (int ks = 0; ks < 2; ++ks) mma3(xi[nt], pih[ks], pil[ks], xv[2 * ks][nt], xv[2 * ks + 1][nt]);
    }
    // X_in into its tile (before the second product: the two interleaved hold
    // more registers, 96.4 against 94.8 ms for the step of 20 circuits; all
    // stores behind both products: X_in's before the second, 100.0 ms)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float* row = ta + (h ? r1 : r0) * S;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        if (last) {
#pragma unroll
          for (int nt = 0; nt < 4; ++nt) row[8 * nt + tig + 4 * c] = xi[nt][2 * h + c];
        } else {
          *reinterpret_cast<float4*>(row + 8 * tig + 4 * c) =
              make_float4(xi[0][2 * h + c], xi[1][2 * h + c], xi[2][2 * h + c], xi[3][2 * h + c]);
        }
      }
    }
    // G_in = P^T G_out
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
#pragma unroll
      for (int i = 0; i < 4; ++i) gn[nt][i] = 0.f;
#pragma unroll
      for (int ks = 0; ks < 2; ++ks) mma3(gn[nt], pth[ks], ptl[ks], gq[2 * ks][nt], gq[2 * ks + 1][nt]);
    }
    __syncwarp();  // the tiles are written, and every lane has read what the others overwrite
    if (wide) {
      const int64_t b = group_base(geo, t0 + 8 * tig);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float v[8], w[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          v[i] = xi[i & 3][2 * h + (i >> 2)];
          w[i] = gn[i & 3][2 * h + (i >> 2)];
        }
        store8(x + b + (h ? out1 : out0), v);
        store8(gv + b + (h ? out1 : out0), w);
      }
    } else if (quads) {
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int64_t b = group_base(geo, t0 + 8 * tig + 4 * c);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int i = 2 * h + c, o = h ? out1 : out0;
          *reinterpret_cast<float4*>(x + b + o) = make_float4(xi[0][i], xi[1][i], xi[2][i], xi[3][i]);
          *reinterpret_cast<float4*>(gv + b + o) = make_float4(gn[0][i], gn[1][i], gn[2][i], gn[3][i]);
        }
      }
    } else {
#pragma unroll
      for (int nt = 0; nt < 4; ++nt)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const int64_t gi = t0 + column(nt, 2 * tig + c);
          if (gi < end) {
            const int64_t b = group_base(geo, gi);
            if (last) {
              *reinterpret_cast<float2*>(x + b + out0) = make_float2(xi[nt][c], xi[nt][2 + c]);
              *reinterpret_cast<float2*>(gv + b + out0) = make_float2(gn[nt][c], gn[nt][2 + c]);
            } else {
              x[b + out0] = xi[nt][c];
              x[b + out1] = xi[nt][2 + c];
              gv[b + out0] = gn[nt][c];
              gv[b + out1] = gn[nt][2 + c];
            }
          }
        }
    }
    // dP += G_out X_in^T: A[r][group], B[group][k] = X_in[k][group]
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
      const int c = 8 * ks + tig;
      const float ga[4] = {tb[gid * S + c], tb[(gid + 8) * S + c], tb[gid * S + c + 4], tb[(gid + 8) * S + c + 4]};
      uint32_t ah[4], al[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) split_tf32(ga[i], ah[i], al[i]);
#pragma unroll
      for (int nb = 0; nb < 2; ++nb) mma3(dp + 4 * nb, ah, al, ta[(8 * nb + gid) * S + c], ta[(8 * nb + gid) * S + c + 4]);
    }
    __syncwarp();
    if ((++tiles & 3) == 0) fold_fp64(acc, dp, tiles == 4);
  }
  if (tiles < 4 || (tiles & 3)) fold_fp64(acc, dp, tiles < 4);
  __syncthreads();  // every warp is done with the tile: reuse it for the sums
#pragma unroll
  for (int nb = 0; nb < 2; ++nb)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = gid + 8 * (i >> 1), k = 8 * nb + 2 * tig + (i & 1);
      sm.u.red[warp][r * 16 + k] = acc[nb * 4 + i];
    }
  __syncthreads();
  for (int e = threadIdx.x; e < K * K; e += blockDim.x) {
    double t = 0.0;
    for (int w = 0; w < nwarps; ++w) t += sm.u.red[w][e];
    dst[e] = t;
  }
  __syncthreads();
}

__device__ __noinline__ void loss_item(const qsgb_batch_program& p, const qsgb_batch_instance& in, int inst, BatchSmem& sm) {
  const int n = in.n_qubits;
  const int64_t D = 1ll << n;
  double part = 0.0;
  for (int64_t j = threadIdx.x; j < D; j += blockDim.x) {
    // element of the diagonal entry j: bit q of j (from the top) selects
    // Pauli element 0 (|0><0|) or 1 (|1><1|) of qubit q
    int64_t idx = 0;
    for (int q = 0; q < n; ++q) idx |= ((j >> (n - 1 - q)) & 1ll) << (2 * (n - 1 - q));
    const double pr = (double)in.x[idx];
    const double t = p.target[in.diag_offset + j];
    p.prob[in.diag_offset + j] = pr;
    const double pe = pr > 1e-300 ? pr : 1e-300;
    if (t > 0) {
      part += t * (log(t) - log(pe));
      in.g[idx] = (float)(-t / pe);
    } else {
      in.g[idx] = 0.f;
    }
  }
  for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
  if ((threadIdx.x & 31) == 0) sm.lsum[threadIdx.x >> 5] = part;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += sm.lsum[w];
    p.loss[inst] = s;
  }
  __syncthreads();
}

// An item's fields against its instance: a known op, targets inside the
// instance (two distinct, ordered qubits for two-qubit ops), ranges inside
// the vector (in groups for APPLY / ADJOINT), a non-negative PTM or
// checkpoint index, an instance below the program's count.  Malformed items
// are skipped and reported as QSGB_DEV_BADITEM instead of being allowed to
// address memory they do not own.
__device__ __forceinline__ bool item_ok(const qsgb_batch_program& p, const qsgb_batch_item& it) {
  if (it.op < QSGB_BOP_INIT || it.op > QSGB_BOP_GRADSUM || it.inst < 0 || it.inst >= p.n_instances) return false;
  if (it.op == QSGB_BOP_GRADSUM) return it.beg >= 0 && it.end >= it.beg && it.ptm >= 0;
  const qsgb_batch_instance in = p.instances[it.inst];
  const int n = in.n_qubits;
  if (n < 1 || n > 15 || in.size != (1ll << (2 * n))) return false;
  if (it.op == QSGB_BOP_LOSS) return true;
  if (it.beg < 0 || it.ptm < 0) return false;
  if (it.op == QSGB_BOP_APPLY || it.op == QSGB_BOP_ADJOINT) {
    if (it.q0 < 0 || it.q0 >= n) return false;
    if (it.q1 >= 0 && (it.q1 <= it.q0 || it.q1 >= n)) return false;
    return it.end <= (in.size >> (it.q1 < 0 ? 2 : 4));
  }
  return it.end <= in.size && (it.beg & 3) == 0 && (it.end & 3) == 0;
}

__device__ void process(const qsgb_batch_program& p, const qsgb_batch_item& it, BatchSmem& sm) {
  const qsgb_batch_instance in = p.instances[it.inst];
  switch (it.op) {
    // element ranges start and end on multiples of 4 (item_ok): 16-byte accesses
    case QSGB_BOP_INIT:
      for (int64_t e = it.beg + 4 * (int64_t)threadIdx.x; e < it.end; e += 4 * (int64_t)blockDim.x)
        *reinterpret_cast<float4*>(in.x + e) = make_float4(e == 0 ? 1.f : 0.f, 0.f, 0.f, 0.f);
      break;
    case QSGB_BOP_ZERO_G:
      for (int64_t e = it.beg + 4 * (int64_t)threadIdx.x; e < it.end; e += 4 * (int64_t)blockDim.x)
        *reinterpret_cast<float4*>(in.g + e) = make_float4(0.f, 0.f, 0.f, 0.f);
      break;
    case QSGB_BOP_SAVE: {
      float* dst = in.ckpt + (int64_t)it.ptm * in.size;
      for (int64_t e = it.beg + 4 * (int64_t)threadIdx.x; e < it.end; e += 4 * (int64_t)blockDim.x)
        *reinterpret_cast<float4*>(dst + e) = *reinterpret_cast<const float4*>(in.x + e);
      break;
    }
    case QSGB_BOP_RESTORE: {
      const float* src = in.ckpt + (int64_t)it.ptm * in.size;
      for (int64_t e = it.beg + 4 * (int64_t)threadIdx.x; e < it.end; e += 4 * (int64_t)blockDim.x)
        *reinterpret_cast<float4*>(in.x + e) = *reinterpret_cast<const float4*>(src + e);
      break;
    }
    case QSGB_BOP_APPLY:
    case QSGB_BOP_ADJOINT: {
      const Geo geo = geometry(in.n_qubits, it.q0, it.q1);
      const int kk = geo.k * geo.k;
      for (int e = threadIdx.x; e < kk; e += blockDim.x) {
        const float v = p.ptm[(int64_t)it.ptm * 256 + e];
        sm.P[e] = v;
        if (it.op == QSGB_BOP_ADJOINT) {
          sm.PT[(e % geo.k) * geo.k + e / geo.k] = v;
          sm.Pi[e] = p.ptm_inv[(int64_t)it.ptm * 256 + e];
        }
      }
      __syncthreads();
      if (it.op == QSGB_BOP_APPLY) {
        if (geo.k == 4)
          apply_vec<4>(in.x, geo, it.beg, it.end, sm.P);
        else
          apply_vec<16>(in.x, geo, it.beg, it.end, sm.P);
      } else if (geo.k == 4) {
        adjoint1_vec(in.x, in.g, geo, it.beg, it.end, sm.P, sm.Pi, sm, p.grad_partial + (int64_t)it.slot * 256);
      } else {
        adjoint2_warp(in.x, in.g, geo, it.beg, it.end, p.grad_partial + (int64_t)it.slot * 256);
      }
      __syncthreads();
      break;
    }
    case QSGB_BOP_LOSS:
      loss_item(p, in, it.inst, sm);
      break;
    case QSGB_BOP_GRADSUM:
      for (int e = threadIdx.x; e < 256; e += blockDim.x) {
        double s = 0.0;
        for (int64_t sl = it.beg; sl < it.end; ++sl) s += p.grad_partial[sl * 256 + e];
        p.grad[(int64_t)it.ptm * 256 + e] = s;
      }
      break;
    default:
      if (threadIdx.x == 0 && p.work) atomicExch(&p.work[p.n_stages + 2], 1u);
      break;
  }
}

__global__ void __launch_bounds__(kBatchBlock, 2) batch_kernel(const __grid_constant__ qsgb_batch_program p,
                                                               unsigned* status, long long spin_limit) {
  extern __shared__ __align__(16) unsigned char dsm[];
  BatchSmem& sm = *reinterpret_cast<BatchSmem*>(dsm);
  uint32_t* bar_count = p.work + p.n_stages;
  uint32_t* bar_gen = p.work + p.n_stages + 1;
  uint32_t* abort_flag = p.work + p.n_stages + 2;
  for (int s = 0; s < p.n_stages; ++s) {
    const int beg = p.stage_begin[s], end = p.stage_begin[s + 1];
    while (true) {
      __syncthreads();
      if (threadIdx.x == 0) sm.item = beg + (int)atomicAdd(&p.work[s], 1u);
      __syncthreads();
      const int i = sm.item;
      if (i >= end) break;
      const qsgb_batch_item it = p.items[i];
      if (!item_ok(p, it)) {
        if (threadIdx.x == 0 && status) atomicOr(status, QSGB_DEV_BADITEM);
        continue;
      }
      process(p, it, sm);
    }
    if (s + 1 < p.n_stages && !grid_barrier(bar_count, bar_gen, abort_flag, spin_limit, status, sm)) return;
  }
}

}  // namespace
}  // namespace qsgb

static int batch_smem_setup() {
  const int bytes = (int)sizeof(qsgb::BatchSmem);
  if (cudaFuncSetAttribute(qsgb::batch_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess) {
    cudaGetLastError();
    return -1;
  }
  return bytes;
}

extern "C" int qsgb_batch_max_grid(int block) {
  if (block != qsgb::kBatchBlock) return 0;
  const int smem = batch_smem_setup();
  if (smem < 0) return 0;
  int occ = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, qsgb::batch_kernel, block, smem) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return occ * qsgb::sm_count();
}

extern "C" int qsgb_batch_run(const qsgb_batch_program* prog, int grid, int block, int cooperative,
                              unsigned* dev_status, int64_t spin_limit, void* stream) {
  if (!prog || !prog->instances || !prog->items || !prog->stage_begin || !prog->work || !prog->ptm)
    return QSGB_ERR_INVALID;
  if (block != qsgb::kBatchBlock || grid < 1 || prog->n_stages < 1 || prog->n_instances < 1 || spin_limit < 1)
    return QSGB_ERR_INVALID;
  const int maxg = qsgb_batch_max_grid(block);
  if (maxg < 1) return QSGB_ERR_CUDA;
  if (grid > maxg) return QSGB_ERR_INVALID;  // every block must be resident for the barriers
  qsgb_batch_program p = *prog;
  long long lim = (long long)spin_limit;
  cudaStream_t s = qsgb::as_stream(stream);
  void* args[] = {(void*)&p, (void*)&dev_status, (void*)&lim};
  cudaError_t e;
  const size_t smem = sizeof(qsgb::BatchSmem);
  if (cooperative)
    e = cudaLaunchCooperativeKernel((const void*)qsgb::batch_kernel, dim3(grid), dim3(block), args, smem, s);
  else
    e = cudaLaunchKernel((const void*)qsgb::batch_kernel, dim3(grid), dim3(block), args, smem, s);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return QSGB_ERR_CUDA;
  }
  return QSGB_OK;
}
