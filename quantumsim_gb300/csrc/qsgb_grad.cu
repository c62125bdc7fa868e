// Reverse-mode kernels for apply_ptm: the gradient with respect to the PTM,
//   dP[r, k] = sum over bystander groups g of g_out[g, r] * x_in[g, k],
// a tall-skinny (Kout x Kin) reduction over all groups.  (The gradient with
// respect to the state is apply_ptm with the transposed PTM, see
// qsgb_apply.cu.)  The reference has no differentiation; the operation is
// the adjoint of quantumsim/pauli_vectors/numpy.py:50-64.
//
// The reduction has Kout * Kin multiply-adds per group: 256 for a two-qubit
// PTM, ~16 per streamed element.  On GB300 the FP64 pipe issues ~0.6 T FMA/s,
// so native FP64 products cap the kernel near 0.3 TB/s; the products here run
// on the FP32 pipes in float-float ("df64") arithmetic instead:
//
// Stage 1: each block walks tiles of `tg` groups.  The tile's inputs and
// output-gradients are loaded (the next tile's into registers while the
// current one is computed), split into float pairs hi + lo (48 significant
// bits, qsgb_split_f64) and staged in shared memory group-major.  Each thread
// owns a 4 x 4 micro-tile of (r, k) entries and a slice of the tile's groups
// and accumulates exact products hi*hi + the cross terms in float-float
// (qsgb_df_fma: error ~2^-47 per product, relative).  At the end of the block
// the slices' float-float sums are added in a fixed order and rounded to
// one double per entry (integer operations, qsgb_df_to_double).
//
// A tile holding a non-zero value outside [2^-100, 2^40] (where products or
// their sums could leave the float range) is computed in native FP64 instead,
// from global memory, into FP64 accumulators in shared memory that join the
// block's sums at the end.  Products of in-range values below the float
// range (< 2^-126) lose their low bits: the absolute error per product stays
// below 2^-149.
//
// Stage 2 adds the per-block partials of each entry in a fixed order
// (deterministic).
#include <algorithm>
#include <cstdlib>
#include <cstring>

#include "qsgb_common.cuh"
#include "qsgb_tc.h"

namespace qsgb {
namespace {

constexpr int kGradBlock = 256;
constexpr int kLoads = 8;  // (Kin + Kout) * tg <= kLoads * kGradBlock
constexpr int kStage2Entries = 32;
constexpr int kStage2Slices = 32;

struct GradParams {
  const void* x;
  const void* g;
  int kin, kout, db_in, db_out;
  int kpi, kpo;    // float2 row lengths of the staged inputs / gradients
  int tg;          // groups per tile (a power of two dividing kGradBlock)
  int nmt_c, nmt;  // 4 x 4 micro-tiles along k, in total
  int slices;      // group slices of a tile (micro-tiles <= kGradBlock)
  uint64_t n_groups, n_tiles;
  FastDiv div_z, div_y;
  int64_t sxi, syi, sai, sbi;
  int64_t sxo, syo, sao, sbo;
  // shared-memory byte offsets
  int off_gb, off_offs, off_fb, off_red2, off_flag, smem;
  int vec_z1;  // 16 x 16: the second qudit's four elements are one 32-byte word
};

unsigned grad_blocks(uint64_t n_groups, int tg) {
  const uint64_t tiles = (n_groups + tg - 1) / tg;
  return (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(tiles, (uint64_t)sm_count() * 2));
}

// groups per tile: the largest power of two <= kGradBlock with
// rows * tg <= kLoads * kGradBlock
int grad_tile(int rows) {
  int tg = kGradBlock;
  while (tg > 1 && rows * tg > kLoads * kGradBlock) tg >>= 1;
  return tg;
}

__device__ __forceinline__ unsigned out_of_band(double v) {
  const unsigned h = (unsigned)__double2hiint(v);
  const unsigned e = (h >> 20) & 0x7ffu;
  const bool nz = ((h << 1) | (unsigned)__double2loint(v)) != 0u;
  return (nz && (e < 923u || e > 1063u)) ? 1u : 0u;  // 2^-100 <= |v| <= 2^40
}

__device__ __forceinline__ unsigned out_of_band(float v) {
  const unsigned b = __float_as_uint(v) & 0x7fffffffu;
  const unsigned e = b >> 23;
  return (b != 0u && (e < 27u || e > 167u)) ? 1u : 0u;
}

__device__ __forceinline__ float2 split_pair(double v) {
  float h, l;
  unsigned ignored = 0;
  qsgb_split_f64(v, h, l, ignored);
  return make_float2(h, l);
}

__device__ __forceinline__ float2 split_pair(float v) { return make_float2(v, 0.0f); }

// (s, c) += (s2, c2), float-float
__device__ __forceinline__ void df_add(float& s, float& c, float s2, float c2) {
  const float r = s + s2;
  const float bp = r - s;
  const float err = (s - (r - bp)) + (s2 - bp);
  s = r;
  c += err + c2;
}

template <typename T, int MPT>
__global__ void __launch_bounds__(kGradBlock) grad_stage1(const __grid_constant__ GradParams p,
                                                          double* __restrict__ part) {
  extern __shared__ __align__(16) unsigned char smem[];
  float2* sx = reinterpret_cast<float2*>(smem);  // [tg][kpi]
  float2* sg = sx + p.tg * p.kpi;                // [tg][kpo]
  int64_t* gb = reinterpret_cast<int64_t*>(smem + p.off_gb);      // [2][tg]: group bases (in, out), -1 idle
  int64_t* offs = reinterpret_cast<int64_t*>(smem + p.off_offs);  // [kin + kout] row offsets
  double* fb = reinterpret_cast<double*>(smem + p.off_fb);        // [kGradBlock][MPT][16] FP64 tiles
  int* fb_any = reinterpret_cast<int*>(smem + p.off_flag);
  const T* X = static_cast<const T*>(p.x);
  const T* G = static_cast<const T*>(p.g);
  const int t = threadIdx.x;
  const int R = p.kin + p.kout;

  // zero the staging area (padding rows stay zero) and the FP64 sums
  {
    float4* z = reinterpret_cast<float4*>(smem);
    for (int i = t; i < p.off_gb / 16; i += kGradBlock) z[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    double* f = fb;
    for (int i = t; i < kGradBlock * MPT * 16; i += kGradBlock) f[i] = 0.0;
  }
  for (int r = t; r < R; r += kGradBlock) {
    if (r < p.kin) {
      const int ka = r / p.db_in, kb = r - ka * p.db_in;
      offs[r] = ka * p.sai + kb * p.sbi;
    } else {
      const int rr = r - p.kin, ra = rr / p.db_out, rb = rr - ra * p.db_out;
      offs[r] = ra * p.sao + rb * p.sbo;
    }
  }
  if (t == 0) *fb_any = 0;
  pdl_wait();
  __syncthreads();

  // loader role: group gg_ld of the tile, rows r0_ld + j * rstep
  const int gg_ld = t & (p.tg - 1);
  const int r0_ld = t / p.tg, rstep = kGradBlock / p.tg;
  T v[kLoads];
  int64_t bin = -1, bout = -1;
  auto fetch = [&](uint64_t tile) {
    const uint64_t g = tile * p.tg + gg_ld;
    const bool live = tile < p.n_tiles && g < p.n_groups;
    bin = bout = -1;
    if (live) {
      const uint64_t t1 = fdiv(g, p.div_z);
      const uint64_t z = g - t1 * p.div_z.d;
      const uint64_t x = fdiv(t1, p.div_y);
      const uint64_t y = t1 - x * p.div_y.d;
      bin = (int64_t)x * p.sxi + (int64_t)y * p.syi + (int64_t)z;
      bout = (int64_t)x * p.sxo + (int64_t)y * p.syo + (int64_t)z;
    }
#pragma unroll
    for (int j = 0; j < kLoads; ++j) {
      const int r = r0_ld + j * rstep;
      v[j] = (T)0;
      if (live && r < R) v[j] = r < p.kin ? X[bin + offs[r]] : G[bout + offs[r]];
    }
  };
  auto stage = [&]() -> unsigned {
    unsigned bad = 0;
#pragma unroll
    for (int j = 0; j < kLoads; ++j) {
      const int r = r0_ld + j * rstep;
      if (r < R) {
        bad |= out_of_band(v[j]);
        const float2 s = split_pair(v[j]);
        if (r < p.kin)
          sx[gg_ld * p.kpi + r] = s;
        else
          sg[gg_ld * p.kpo + (r - p.kin)] = s;
      }
    }
    if (r0_ld == 0) {
      gb[gg_ld] = bin;
      gb[p.tg + gg_ld] = bout;
    }
    return bad;
  };

  // compute role: micro-tiles and group slice
  int mt[MPT], r0[MPT], k0[MPT];
  bool act[MPT];
  int slice;
  if (MPT == 1) {
    mt[0] = t % p.nmt;
    slice = t / p.nmt;
    act[0] = slice < p.slices;
  } else {
    slice = 0;
#pragma unroll
    for (int m = 0; m < MPT; ++m) {
      mt[m] = t + m * kGradBlock;
      act[m] = mt[m] < p.nmt;
    }
  }
#pragma unroll
  for (int m = 0; m < MPT; ++m) {
    r0[m] = (mt[m] / p.nmt_c) * 4;
    k0[m] = (mt[m] % p.nmt_c) * 4;
  }
  float s[MPT][16], c[MPT][16];
#pragma unroll
  for (int m = 0; m < MPT; ++m)
#pragma unroll
    for (int q = 0; q < 16; ++q) s[m][q] = c[m][q] = 0.0f;

  fetch(blockIdx.x);
  for (uint64_t tile = blockIdx.x; tile < p.n_tiles; tile += gridDim.x) {
    __syncthreads();  // the previous tile is consumed
    const int bad = __syncthreads_or((int)stage());
    fetch(tile + gridDim.x);  // in flight while this tile is computed
    if (!bad) {
#pragma unroll
      for (int m = 0; m < MPT; ++m) {
        if (!act[m]) continue;
        for (int gg = slice; gg < p.tg; gg += p.slices) {
          const float4 a01 = *reinterpret_cast<const float4*>(sg + gg * p.kpo + r0[m]);
          const float4 a23 = *reinterpret_cast<const float4*>(sg + gg * p.kpo + r0[m] + 2);
          const float4 b01 = *reinterpret_cast<const float4*>(sx + gg * p.kpi + k0[m]);
          const float4 b23 = *reinterpret_cast<const float4*>(sx + gg * p.kpi + k0[m] + 2);
          const float ah[4] = {a01.x, a01.z, a23.x, a23.z}, al[4] = {a01.y, a01.w, a23.y, a23.w};
          const float bh[4] = {b01.x, b01.z, b23.x, b23.z}, bl[4] = {b01.y, b01.w, b23.y, b23.w};
#pragma unroll
          for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) qsgb_df_fma(s[m][4 * i + j], c[m][4 * i + j], ah[i], al[i], bh[j], bl[j]);
        }
      }
    } else {
      // a value outside the float-float band: this tile in native FP64
      if (t == 0) *fb_any = 1;
#pragma unroll 1
      for (int m = 0; m < MPT; ++m) {
        if (!act[m]) continue;
        double* acc = fb + ((int64_t)t * MPT + m) * 16;
#pragma unroll 1
        for (int gg = slice; gg < p.tg; gg += p.slices) {
          const int64_t bi = gb[gg], bo = gb[p.tg + gg];
          if (bi < 0) continue;
          double a[4], b[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            a[i] = r0[m] + i < p.kout ? (double)G[bo + offs[p.kin + r0[m] + i]] : 0.0;
            b[i] = k0[m] + i < p.kin ? (double)X[bi + offs[k0[m] + i]] : 0.0;
          }
#pragma unroll
          for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[4 * i + j] = fma(a[i], b[j], acc[4 * i + j]);
        }
      }
    }
  }

  // block sums: slices in a fixed order, one double per entry
  __syncthreads();
  float2* red = reinterpret_cast<float2*>(smem);  // [kGradBlock][MPT][16], over the staging area
#pragma unroll
  for (int m = 0; m < MPT; ++m)
#pragma unroll
    for (int q = 0; q < 16; ++q) red[((int64_t)t * MPT + m) * 16 + q] = make_float2(s[m][q], c[m][q]);
  __syncthreads();
  const bool any_fb = *fb_any != 0;
  const int E = p.kin * p.kout;
  const int EP = p.nmt * 16;  // padded entries
  float2* red2 = reinterpret_cast<float2*>(smem + p.off_red2);  // [chunks][EP] (MPT == 1)
  double* fb2 = reinterpret_cast<double*>(smem + p.off_red2 + kGradBlock * sizeof(float2));
  if constexpr (MPT == 1) {
    // level 1: entry qp, slice chunk ch (slices ch, ch + nch, ...); with
    // many slices (small PTMs) the chunks spread the sums over the block
    const int nch = EP < kGradBlock ? kGradBlock / EP : 1;
    for (int tq = t; tq < nch * EP; tq += kGradBlock) {
      const int qp = tq % EP, ch = tq / EP;
      const int mtq = qp >> 4, q = qp & 15;
      float S = 0.0f, C = 0.0f;
      double F = 0.0;
      for (int sl = ch; sl < p.slices; sl += nch) {
        const int64_t idx = ((int64_t)(sl * p.nmt + mtq)) * 16 + q;
        const float2 v2 = red[idx];
        df_add(S, C, v2.x, v2.y);
        if (any_fb) F += fb[idx];
      }
      if (nch > 1) {
        red2[ch * EP + qp] = make_float2(S, C);
        fb2[ch * EP + qp] = F;
      } else {
        const int r = (mtq / p.nmt_c) * 4 + (q >> 2), k = (mtq % p.nmt_c) * 4 + (q & 3);
        double d = qsgb_df_to_double(S, C);
        if (any_fb) d += F;
        if (r < p.kout && k < p.kin) part[(int64_t)blockIdx.x * E + r * p.kin + k] = d;
      }
    }
    if (nch > 1) {
      __syncthreads();
      // level 2: the chunks of entry qp in order
      for (int qp = t; qp < EP; qp += kGradBlock) {
        const int mtq = qp >> 4, q = qp & 15;
        float S = 0.0f, C = 0.0f;
        double F = 0.0;
        for (int ch = 0; ch < nch; ++ch) {
          const float2 v2 = red2[ch * EP + qp];
          df_add(S, C, v2.x, v2.y);
          if (any_fb) F += fb2[ch * EP + qp];
        }
        const int r = (mtq / p.nmt_c) * 4 + (q >> 2), k = (mtq % p.nmt_c) * 4 + (q & 3);
        double d = qsgb_df_to_double(S, C);
        if (any_fb) d += F;
        if (r < p.kout && k < p.kin) part[(int64_t)blockIdx.x * E + r * p.kin + k] = d;
      }
    }
  } else {
  for (int qp = t; qp < EP; qp += kGradBlock) {
    const int mtq = qp >> 4, q = qp & 15;
    const int r = (mtq / p.nmt_c) * 4 + (q >> 2), k = (mtq % p.nmt_c) * 4 + (q & 3);
    float S = 0.0f, C = 0.0f;
    double F = 0.0;
    {
      const int tt = mtq % kGradBlock, m = mtq / kGradBlock;
      const int64_t idx = ((int64_t)tt * MPT + m) * 16 + q;
      const float2 v2 = red[idx];
      S = v2.x;
      C = v2.y;
      if (any_fb) F = fb[idx];
    }
    double d = qsgb_df_to_double(S, C);
    if (any_fb) d += F;
    if (r < p.kout && k < p.kin) part[(int64_t)blockIdx.x * E + r * p.kin + k] = d;
  }
  }
}

// ---------------------------------------------------------------------------
// One qudit of at most four Pauli elements: a group per thread
// ---------------------------------------------------------------------------
// At up to 4 x 4 entries a group's whole outer product fits a thread: its (up
// to) eight values come straight into registers, the next group's while this
// one is multiplied, and nothing is staged in shared memory or shared between
// threads until the sums are complete.  The same float-float products and band
// as in stage 1 above; a group with a value outside the band is multiplied in
// native FP64, into sums of its thread in shared memory (12 qubits, us: none 69,
// one value in 10^5 74, one in 1000 86, all 148; with the whole block's groups
// done again 68, 191, 191, 192; the staged kernel 150, 167, 434, 523).  The warps' sums are scattered over their lanes
// by exchanges (16 entries: 16 shuffles of a pair instead of 80) and the block's
// added in warp order.  Bound by instruction issue (about 400 a group, 160 of
// them the products) and the latency of one group ahead per thread; a ring of
// asynchronous copies three groups ahead gave 4 % at 12 qubits and took 5 % at
// 10.  A gradient with its second stage, against the staged kernel above: 10
// qubits (2^18 groups) 19.8 -> 11.3 us, 11 qubits 47 -> 22, 12 qubits 150 -> 69
// (3.9 TB/s); FP32 vectors of 12 qubits 132 -> 48.
// A thread's walk over its groups: the place in the two tensors, moved by a
// fixed number of groups at a time without a division.
struct Grad4Walk {
  int64_t z, x, o;       // place along the inner bystander, offsets of the group
  int64_t dz, dx, dxo;   // a step, while z stays below its length
  __device__ __forceinline__ Grad4Walk(const GradParams& p, uint64_t g, uint64_t stride) {
    uint64_t y = fdiv(g, p.div_z);
    z = (int64_t)(g - y * p.div_z.d);
    x = (int64_t)y * p.syi + z;
    o = (int64_t)y * p.syo + z;
    y = fdiv(stride, p.div_z);
    dz = (int64_t)(stride - y * p.div_z.d);
    dx = (int64_t)y * p.syi + dz;
    dxo = (int64_t)y * p.syo + dz;
  }
  __device__ __forceinline__ void step(const GradParams& p) {
    z += dz;
    x += dx;
    o += dxo;
    if (z >= (int64_t)p.div_z.d) {
      z -= (int64_t)p.div_z.d;
      x += p.syi - (int64_t)p.div_z.d;
      o += p.syo - (int64_t)p.div_z.d;
    }
  }
};

// FULL: four input and four output elements
template <typename T, bool FULL>
__device__ __forceinline__ void grad4_load(T (&v)[8], const T* X, const T* G, const GradParams& p, const Grad4Walk& w) {
  const T* x = X + w.x;
  const T* o = G + w.o;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    v[k] = FULL || k < p.kin ? x[k * p.sbi] : (T)0;
    v[4 + k] = FULL || k < p.kout ? o[k * p.sbo] : (T)0;
  }
}

__device__ __forceinline__ void split_band(double v, float& h, float& l, unsigned& bad) {
  qsgb_split_f64<923u, 141u>(v, h, l, bad);  // 2^-100 <= |v| < 2^41
}
__device__ __forceinline__ void split_band(float v, float& h, float& l, unsigned& bad) {
  bad |= out_of_band(v);
  h = v;
  l = 0.0f;
}

// lanes 2H apart share the sums of entries [0, 2H): each keeps H of them
template <int H>
__device__ __forceinline__ void grad4_halve(float (&s)[16], float (&c)[16], int lane) {
  const bool up = (lane & (2 * H)) != 0;  // keeps the upper ones
#pragma unroll
  for (int q = 0; q < H; ++q) {
    const float ss = up ? s[q] : s[q + H], sc = up ? c[q] : c[q + H];
    s[q] = up ? s[q + H] : s[q];
    c[q] = up ? c[q + H] : c[q];
    df_add(s[q], c[q], __shfl_xor_sync(0xffffffffu, ss, 2 * H), __shfl_xor_sync(0xffffffffu, sc, 2 * H));
  }
}

template <typename T, bool FULL>
__global__ void __launch_bounds__(kGradBlock, 2) grad4_kernel(const __grid_constant__ GradParams p,
                                                              double* __restrict__ part) {
  __shared__ double sums[kGradBlock / 32][16];
  __shared__ double f64[16][kGradBlock];  // products of groups outside the band, a thread's own
  const T* X = static_cast<const T*>(p.x);
  const T* G = static_cast<const T*>(p.g);
  const int t = threadIdx.x, lane = t & 31;
  const uint64_t first = (uint64_t)blockIdx.x * kGradBlock + t, stride = (uint64_t)gridDim.x * kGradBlock;
  float s[16], c[16];
#pragma unroll
  for (int q = 0; q < 16; ++q) s[q] = c[q] = 0.0f;
  bool met = false;  // this thread has had such a group
  pdl_wait();
  T v[8];
  Grad4Walk walk(p, first, stride);
  if (first < p.n_groups) grad4_load<T, FULL>(v, X, G, p, walk);
  for (uint64_t g = first; g < p.n_groups; g += stride) {
    float h[8], l[8];
    unsigned bad = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) split_band(v[k], h[k], l[k], bad);
    if (bad) {  // this group in native FP64
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          double* f = &f64[4 * r + k][t];
          *f = fma((double)v[4 + r], (double)v[k], met ? *f : 0.0);
        }
      met = true;
#pragma unroll
      for (int k = 0; k < 8; ++k) h[k] = l[k] = 0.0f;
    }
    if (g + stride < p.n_groups) {
      walk.step(p);
      grad4_load<T, FULL>(v, X, G, p, walk);
    }
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int q = 4 * r + k;
        if constexpr (sizeof(T) == 8) {
          qsgb_df_fma(s[q], c[q], h[4 + r], l[4 + r], h[k], l[k]);
        } else {  // the same without the low parts
          const float s2 = s[q] + __fmul_rn(h[4 + r], h[k]);
          const float bp = s2 - s[q];
          c[q] += fmaf(h[4 + r], h[k], -bp) + (s[q] - (s2 - bp));
          s[q] = s2;
        }
      }
  }
  grad4_halve<8>(s, c, lane);
  grad4_halve<4>(s, c, lane);
  grad4_halve<2>(s, c, lane);
  grad4_halve<1>(s, c, lane);
  const float s2 = __shfl_xor_sync(0xffffffffu, s[0], 1), c2 = __shfl_xor_sync(0xffffffffu, c[0], 1);
  df_add(s[0], c[0], s2, c2);
  double d = qsgb_df_to_double(s[0], c[0]);  // entry lane / 2 of this warp
  if (__any_sync(0xffffffffu, met)) {
#pragma unroll 1
    for (int q = 0; q < 16; ++q) {
      double f = met ? f64[q][t] : 0.0;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) f += __shfl_xor_sync(0xffffffffu, f, o);
      if ((lane >> 1) == q) d += f;
    }
  }
  if ((lane & 1) == 0) sums[t >> 5][lane >> 1] = d;
  __syncthreads();
  if (t < 16) {
    const int r = t >> 2, k = t & 3;
    double r0 = 0.0;
    for (int w = 0; w < kGradBlock / 32; ++w) r0 += sums[w][t];
    if (r < p.kout && k < p.kin) part[(int64_t)blockIdx.x * (p.kin * p.kout) + r * p.kin + k] = r0;
  }
}

// out[e] = sum over blocks b of part[b][e]: kStage2Entries entries x
// kStage2Slices block slices per thread block, slices added in order
__global__ void __launch_bounds__(kStage2Entries* kStage2Slices)
    grad_stage2(const double* part, int nblocks, int E, double* __restrict__ out) {
  __shared__ double red[kStage2Slices][kStage2Entries + 1];
  const int el = threadIdx.x % kStage2Entries, sl = threadIdx.x / kStage2Entries;
  const int e = blockIdx.x * kStage2Entries + el;
  double acc = 0.0;
  pdl_wait();
  if (e < E) {
#pragma unroll 8
    for (int b = sl; b < nblocks; b += kStage2Slices) acc += part[(int64_t)b * E + e];
  }
  red[sl][el] = acc;
  __syncthreads();
  if (sl == 0 && e < E) {
    double s = 0.0;
    for (int i = 0; i < kStage2Slices; ++i) s += red[i][el];
    out[e] = s;
  }
}

// ---------------------------------------------------------------------------
// 16 x 16 gradients on FP64 vectors: the tensor cores
// ---------------------------------------------------------------------------
// The same reduction as a product over groups, dP = G^T X per chunk of 16
// groups, on mma.sync.m16n8k16 (FP16 operands, FP32 accumulators) with the
// error-free digit split of the apply kernel (qsgb_tc.h): within a chunk,
// row r of A = G^T is scaled by its largest exponent over the chunk's
// groups and column k of B = X by its own, each value written as a 55-bit
// fixed-point integer in seven balanced base-256 FP16 digits.  For every digit
// pair (i, j) with i + j <= 7 two MMAs (n = 0..7, 8..15) add into level
// i + j; all level sums are exact FP32 integers.  The eight levels of each
// entry are combined in int64, scaled by 2^(E_r + E_k - kScale8) and added to
// FP64 accumulators in chunk order.  Error per chunk: below
// 2^-49 max_g |g_out[g, r]| max_g |x_in[g, k]| over the chunk's groups,
// typically 2^-54.  A chunk holding inf or nan, values all below
// 2^-959, or a result outside the normal double range, is recomputed in native
// FP64 from global memory.
//
// A warp takes chunks; lane l = (h, i) = (l / 16, l % 16) loads group i of
// the chunk, rows r = 8h .. 8h+7 of g_out and k = 8h .. 8h+7 of x_in, and
// writes each digit of its 8 rows as one 16-byte half row into the warp's
// planes A[d][g][r] and B[d][g][k] (the half rows of groups 4..7 and 12..15
// exchanged, so that 8 groups' half rows fall into different banks).  The
// fragments come back transposed (ldmatrix.trans): lane
// (gid, tig) = (l / 4, l % 4) ends with entries
// (r, k) = (gid or gid + 8, nt * 8 + 2 tig + {0, 1}).
//
// H = 2: a chunk of 32 groups, two such halves with common exponents whose
// level sums are added as integers (a bit more each).  Exponent search,
// recombination and the FP64 sums (16 operations of a pipe that takes a warp
// 16 cycles) are paid once for both, and twice the loads are in flight; the
// planes of 16 warps fill an SM's shared memory in one block.  With no more
// chunks of 16 than resident warps, H = 1 spreads the work further.
//
// Bound by instruction issue and latency: at 12 qubits 2.0 TB/s.  Measured on
// GB300, a gradient with its second stage, at 10 and 12 qubits (4096 and 65536
// chunks of 16): base-1024 digits 21.8 and 173 us, base 256 with H = 1 19.9 and
// 144, H = 2 17.3 and 131; on the last two qudits, with 32-byte loads instead
// of 8-byte ones, 25.0 and 174 -> 18.6 and 138.
constexpr int kTcgBlock = 256;
constexpr int kTcgWarps = kTcgBlock / 32;
constexpr int kTcgPlane = 16 * 16 * 2;  // bytes per digit plane

template <int H>
struct TcgWarpSmem {
  unsigned char a[H][tc::kPlanes * kTcgPlane];  // digits of g_out: [g][r]
  unsigned char b[H][tc::kPlanes * kTcgPlane];  // digits of x_in: [g][k]
  int er[16], ek[16];                           // chunk exponents of rows, columns
};
template <int H>
struct TcgSmem {
  TcgWarpSmem<H> warp[kTcgWarps * H];
  int64_t oin[16], oout[16];  // row offsets of x_in and g_out
};

__device__ __forceinline__ void ldmatrix4_trans(unsigned (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}

__device__ __forceinline__ void load4(double* v, const double* src) {
  asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]), "=d"(v[3]) : "l"(src));
}

template <int H>
__global__ void __launch_bounds__(kTcgBlock* H, 2 / H) grad16_tc_kernel(const __grid_constant__ GradParams p,
                                                              double* __restrict__ part) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  TcgSmem<H>& sm = *reinterpret_cast<TcgSmem<H>*>(smem);
  TcgWarpSmem<H>& ws = sm.warp[w];
  const double* X = static_cast<const double*>(p.x);
  const double* G = static_cast<const double*>(p.g);
  const int h = lane >> 4, i = lane & 15;
  const int gid = lane >> 2, tig = lane & 3;
  if (threadIdx.x < 16) {
    const int k = threadIdx.x;
    const int ka = k / p.db_in, kb = k - ka * p.db_in;
    sm.oin[k] = ka * p.sai + kb * p.sbi;
    const int ra = k / p.db_out, rb = k - ra * p.db_out;
    sm.oout[k] = ra * p.sao + rb * p.sbo;
  }
  pdl_wait();
  __syncthreads();
  // byte offset of half row c of group g in a plane
  auto half_row = [](int g, int c) { return g * 32 + ((c ^ ((g >> 2) & 1)) << 4); };
  // ldmatrix source rows: A tiles (g 0-7 | r 0-7), (0-7 | 8-15), (8-15 | 0-7), (8-15 | 8-15);
  // B tiles (g 0-7 | k 0-7), (8-15 | 0-7), (0-7 | 8-15), (8-15 | 8-15)
  const int lr = lane & 7, t1b = (lane >> 3) & 1, t2b = lane >> 4;
  const uint32_t sa = (uint32_t)__cvta_generic_to_shared(ws.a[0]) + half_row(lr + 8 * t2b, t1b);
  const uint32_t sb = (uint32_t)__cvta_generic_to_shared(ws.b[0]) + half_row(lr + 8 * t1b, t2b);
  auto bases = [&](uint64_t g, int64_t& bi, int64_t& bo) {
    const uint64_t t1 = fdiv(g, p.div_z);
    const uint64_t z = g - t1 * p.div_z.d;
    const uint64_t x = fdiv(t1, p.div_y);
    const uint64_t y = t1 - x * p.div_y.d;
    bi = (int64_t)x * p.sxi + (int64_t)y * p.syi + (int64_t)z;
    bo = (int64_t)x * p.sxo + (int64_t)y * p.syo + (int64_t)z;
  };
  double acc[2][4];
#pragma unroll
  for (int nt = 0; nt < 2; ++nt)
#pragma unroll
    for (int q = 0; q < 4; ++q) acc[nt][q] = 0.0;

  const uint64_t n_chunks = (p.n_groups + 16 * H - 1) / (16 * H);
  const uint64_t wstride = (uint64_t)gridDim.x * kTcgWarps * H;
  for (uint64_t c = (uint64_t)blockIdx.x * kTcgWarps * H + w; c < n_chunks; c += wstride) {
    double gv[H][8], xv[H][8];
#pragma unroll
    for (int hf = 0; hf < H; ++hf) {
      const uint64_t g = c * (16 * H) + 16 * hf + i;
      if (g < p.n_groups) {
        int64_t bi, bo;
        bases(g, bi, bo);
        if (p.vec_z1) {
#pragma unroll
          for (int j = 0; j < 8; j += 4) {
            load4(gv[hf] + j, G + bo + sm.oout[8 * h + j]);
            load4(xv[hf] + j, X + bi + sm.oin[8 * h + j]);
          }
        } else {
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            gv[hf][j] = G[bo + sm.oout[8 * h + j]];
            xv[hf][j] = X[bi + sm.oin[8 * h + j]];
          }
        }
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) gv[hf][j] = xv[hf][j] = 0.0;
      }
    }
    // chunk exponents of rows 8h+j (g_out, low half word) and columns 8h+j
    // (x_in, high half word): maxima over the 16 lanes of this half
    unsigned e2[8], nonfinite = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      e2[j] = 0u;
#pragma unroll
      for (int hf = 0; hf < H; ++hf) {
        const unsigned hg = (unsigned)__double2hiint(gv[hf][j]), hx = (unsigned)__double2hiint(xv[hf][j]);
        e2[j] = __vmaxu2(e2[j], ((hg >> 20) & 0x7ffu) | ((hx >> 4) & 0x7ff0000u));
      }
    }
#pragma unroll
    for (int o = 1; o < 16; o <<= 1)
#pragma unroll
      for (int j = 0; j < 8; ++j) e2[j] = __vmaxu2(e2[j], __shfl_xor_sync(0xffffffffu, e2[j], o));
    {
      unsigned top = 0u, low = 0xffffffffu;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        top = __vmaxu2(top, e2[j]);
        low = __vminu2(low, e2[j]);
      }
      nonfinite = ((top & 0xffffu) == 0x7ffu || (top >> 16) == 0x7ffu) ? 1u : 0u;
      if ((low & 0xffffu) < tc::kMinExp || (low >> 16) < tc::kMinExp) {
        // a row or column that is all zero (exact) or below the smallest scale
#pragma unroll
        for (int j = 0; j < 8; ++j) {
#pragma unroll
          for (int hf = 0; hf < H; ++hf) {
            if ((e2[j] & 0xffffu) < tc::kMinExp && gv[hf][j] != 0.0) nonfinite = 1u;
            if ((e2[j] >> 16) < tc::kMinExp && xv[hf][j] != 0.0) nonfinite = 1u;
          }
          // any scale serves zeros
          if ((e2[j] & 0xffffu) < tc::kMinExp) e2[j] = (e2[j] & 0xffff0000u) | 1023u;
          if ((e2[j] >> 16) < tc::kMinExp) e2[j] = (e2[j] & 0xffffu) | (1023u << 16);
        }
      }
    }
    if (i == 0) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        ws.er[8 * h + j] = (int)(e2[j] & 0xffffu);
        ws.ek[8 * h + j] = (int)(e2[j] >> 16);
      }
    }
    {
      unsigned eh[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) eh[j] = (e2[j] & 0xffffu) << 20;
#pragma unroll
      for (int hf = 0; hf < H; ++hf) tc::split8<kTcgPlane>(ws.a[hf] + half_row(i, h), gv[hf], eh);
#pragma unroll
      for (int j = 0; j < 8; ++j) eh[j] = (e2[j] & 0xffff0000u) << 4;
#pragma unroll
      for (int hf = 0; hf < H; ++hf) tc::split8<kTcgPlane>(ws.b[hf] + half_row(i, h), xv[hf], eh);
    }
    const bool chunk_bad = __any_sync(0xffffffffu, nonfinite != 0u);
    __syncwarp();
    int pr[2][4][tc::kLevels / 2];  // two levels each, of all halves
#pragma unroll
    for (int hf = 0; hf < H; ++hf) {
      unsigned fa[tc::kPlanes][4], fb[tc::kPlanes][4];
#pragma unroll
      for (int d = 0; d < tc::kPlanes; ++d) {
        ldmatrix4_trans(fa[d], sa + (hf * tc::kPlanes + d) * kTcgPlane);
        ldmatrix4_trans(fb[d], sb + (hf * tc::kPlanes + d) * kTcgPlane);
      }
#pragma unroll
      for (int L = 0; L < tc::kLevels; L += 2)
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
          float d[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
          for (int a = 0; a < tc::kPlanes; ++a) {
            if (L - a >= 0 && L - a < tc::kPlanes) tc::mma16816(d[0], fa[a], fb[L - a] + 2 * nt);
            if (L + 1 - a >= 0 && L + 1 - a < tc::kPlanes) tc::mma16816(d[1], fa[a], fb[L + 1 - a] + 2 * nt);
          }
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int pair = tc::level_pair(d[0][q], d[1][q]);
            pr[nt][q][L / 2] = hf == 0 ? pair : pr[nt][q][L / 2] + pair;
          }
        }
    }
    // scale and accumulate (in FP64 from global memory when the chunk or a
    // result is out of range)
    double y[2][4];
    unsigned bad = 0;
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int r = gid + (q >= 2 ? 8 : 0), k = nt * 8 + 2 * tig + (q & 1);
        const int sc = ws.er[r] + ws.ek[k] - tc::kScale8;
        // twice the groups: a bit more
        bad |= tc::scale8_ok(sc) && tc::scale8_ok(sc + H - 1) ? 0u : 1u;
        y[nt][q] = tc::scale8(tc::combine8<H == 1>(pr[nt][q][0], pr[nt][q][1], pr[nt][q][2], pr[nt][q][3]),
                              (unsigned)sc << 20);
      }
    if (chunk_bad || __any_sync(0xffffffffu, bad != 0u)) {
#pragma unroll
      for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int r = gid + (q >= 2 ? 8 : 0), k = nt * 8 + 2 * tig + (q & 1);
          const int ka = k / p.db_in, kb = k - ka * p.db_in, ra = r / p.db_out, rb = r - ra * p.db_out;
          const int64_t ok = ka * p.sai + kb * p.sbi, orr = ra * p.sao + rb * p.sbo;
          double s2 = 0.0;
#pragma unroll 1
          for (int gg = 0; gg < 16 * H; ++gg) {
            const uint64_t g2 = c * (16 * H) + gg;
            if (g2 >= p.n_groups) break;
            int64_t bi, bo;
            bases(g2, bi, bo);
            s2 = fma(G[bo + orr], X[bi + ok], s2);
          }
          y[nt][q] = s2;
        }
    }
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[nt][q] += y[nt][q];
    __syncwarp();  // the planes are rewritten by the next chunk
  }
  // block sums over the warps, in warp order
  __syncthreads();
  double* red = reinterpret_cast<double*>(smem);  // [warps][256], over the planes
#pragma unroll
  for (int nt = 0; nt < 2; ++nt)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int r = gid + (q >= 2 ? 8 : 0), k = nt * 8 + 2 * tig + (q & 1);
      red[w * 256 + r * 16 + k] = acc[nt][q];
    }
  __syncthreads();
  if (threadIdx.x < 256) {
    const int e = threadIdx.x;
    double s2 = 0.0;
    for (int ww = 0; ww < kTcgWarps * H; ++ww) s2 += red[ww * 256 + e];
    part[(int64_t)blockIdx.x * 256 + e] = s2;
  }
}

unsigned tcg_blocks(uint64_t n_groups) {
  const uint64_t chunks = (n_groups + 15) / 16;
  const uint64_t blocks = (chunks + kTcgWarps - 1) / kTcgWarps;
  return (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(blocks, (uint64_t)sm_count() * 2));
}

template <int H>
int launch_grad16(const GradParams& p, unsigned nb, double* part, cudaStream_t s) {
  const int smem = std::max((int)sizeof(TcgSmem<H>), kTcgWarps * H * 256 * (int)sizeof(double));
  const int st = allow_dynamic_smem((const void*)grad16_tc_kernel<H>, smem);
  if (st != QSGB_OK) return st;
  return launch_pdl(grad16_tc_kernel<H>, nb, (unsigned)(kTcgBlock * H), (size_t)smem, s, p, part);
}

// 16 x 16 FP64 gradients go to the tensor cores unless QSGB_TC_GRAD=0
bool tc_grad_enabled() {
  static const bool on = [] {
    const char* v = std::getenv("QSGB_TC_GRAD");
    return !(v && std::strcmp(v, "0") == 0);
  }();
  return on;
}

GradParams make_params(const void* x_in, const void* g_out, int64_t da_out, int64_t db_out, int64_t da_in,
                       int64_t db_in, int64_t X, int64_t Y, int64_t Z) {
  GradParams p{};
  p.x = x_in;
  p.g = g_out;
  const int kin = (int)(da_in * db_in), kout = (int)(da_out * db_out);
  p.kin = kin;
  p.kout = kout;
  p.db_in = (int)db_in;
  p.db_out = (int)db_out;
  const int pi = (kin + 3) / 4 * 4, po = (kout + 3) / 4 * 4;
  p.kpi = pi + 2;  // + 16 bytes: consecutive groups start 4 banks apart
  p.kpo = po + 2;
  p.tg = grad_tile(kin + kout);
  p.nmt_c = pi / 4;
  p.nmt = (pi / 4) * (po / 4);
  p.slices = p.nmt <= kGradBlock ? kGradBlock / p.nmt : 1;
  p.n_groups = (uint64_t)X * Y * Z;
  p.n_tiles = (p.n_groups + p.tg - 1) / p.tg;
  p.div_z = make_fastdiv((uint64_t)Z);
  p.div_y = make_fastdiv((uint64_t)Y);
  p.sbi = Z;
  p.syi = db_in * Z;
  p.sai = Y * db_in * Z;
  p.sxi = da_in * Y * db_in * Z;
  p.sbo = Z;
  p.syo = db_out * Z;
  p.sao = Y * db_out * Z;
  p.sxo = da_out * Y * db_out * Z;
  const int mpt = p.nmt <= kGradBlock ? 1 : 2;
  const size_t stagebytes = (size_t)p.tg * (p.kpi + p.kpo) * sizeof(float2);
  const size_t redbytes = (size_t)kGradBlock * mpt * 16 * sizeof(float2);
  size_t o = (std::max(stagebytes, redbytes) + 15) / 16 * 16;
  p.off_gb = (int)o;
  o += 2 * (size_t)p.tg * sizeof(int64_t);
  p.off_offs = (int)o;
  o += ((size_t)(kin + kout) * sizeof(int64_t) + 15) / 16 * 16;
  p.off_fb = (int)o;
  o += (size_t)kGradBlock * mpt * 16 * sizeof(double);
  p.off_red2 = (int)o;  // level-1 sums: kGradBlock float2 + kGradBlock double
  o += (size_t)kGradBlock * (sizeof(float2) + sizeof(double));
  p.off_flag = (int)o;
  o += 16;
  p.smem = (int)o;
  return p;
}

template <typename T, int MPT>
int launch_stage1(const GradParams& p, unsigned nb, double* part, cudaStream_t s) {
  auto kern = grad_stage1<T, MPT>;
  const int st = allow_dynamic_smem((const void*)kern, p.smem);
  if (st != QSGB_OK) return st;
  return launch_pdl(kern, nb, kGradBlock, (size_t)p.smem, s, p, part);
}

int launch_stage2(const double* part, int nblocks, int E, double* dptm, cudaStream_t s) {
  return launch_pdl(grad_stage2, (unsigned)((E + kStage2Entries - 1) / kStage2Entries),
                    (unsigned)(kStage2Entries * kStage2Slices), 0, s, part, nblocks, E, dptm);
}

int grad_common(const void* x_in, const void* g_out, double* dptm, int64_t da_out, int64_t db_out, int64_t da_in,
                int64_t db_in, int64_t X, int64_t Y, int64_t Z, int dtype, void* scratch, int64_t scratch_bytes,
                void* stream) {
  if (!x_in || !g_out || !dptm) return QSGB_ERR_INVALID;
  if (da_out < 1 || db_out < 1 || da_in < 1 || db_in < 1 || X < 1 || Y < 1 || Z < 1) return QSGB_ERR_INVALID;
  if (dtype != QSGB_F64 && dtype != QSGB_F32) return QSGB_ERR_INVALID;
  const int64_t kin = da_in * db_in, kout = da_out * db_out;
  // 4 x 4 micro-tiles: at most 2 per thread
  if (kin > 256 || kout > 256 || ((kin + 3) / 4) * ((kout + 3) / 4) > 2 * kGradBlock)
    return QSGB_ERR_UNSUPPORTED;
  GradParams p = make_params(x_in, g_out, da_out, db_out, da_in, db_in, X, Y, Z);
  const unsigned nb = grad_blocks(p.n_groups, p.tg);
  const int E = (int)(kin * kout);
  if (!scratch || scratch_bytes < (int64_t)nb * E * (int64_t)sizeof(double)) return QSGB_ERR_SCRATCH;
  cudaStream_t s = as_stream(stream);
  double* part = static_cast<double*>(scratch);
  if (dtype == QSGB_F64 && kin == 16 && kout == 16 && tc_grad_enabled()) {
    p.vec_z1 = Z == 1 && db_in == 4 && db_out == 4 && ((uintptr_t)x_in | (uintptr_t)g_out) % 32 == 0;
    // chunks of 32 groups when those of 16 are more than the resident warps;
    // the scratch holds the partials of tcg_blocks <= nb blocks either way
    const bool wide = p.n_groups > (uint64_t)sm_count() * 2 * kTcgWarps * 16;
    const unsigned nbt = wide ? (unsigned)sm_count() : tcg_blocks(p.n_groups);
    const int s1 = wide ? launch_grad16<2>(p, nbt, part, s) : launch_grad16<1>(p, nbt, part, s);
    return s1 != QSGB_OK ? s1 : launch_stage2(part, (int)nbt, E, dptm, s);
  }
  // one qudit (a group's rows lie a stride apart) of at most 4 elements: a
  // thread's registers hold the outer product
  if (da_in == 1 && da_out == 1 && X == 1 && kin <= 4 && kout <= 4) {
    const bool full = kin == 4 && kout == 4;
    const auto kern = dtype == QSGB_F64 ? (full ? grad4_kernel<double, true> : grad4_kernel<double, false>)
                                        : (full ? grad4_kernel<float, true> : grad4_kernel<float, false>);
    const int s1 = launch_pdl(kern, nb, (unsigned)kGradBlock, 0, s, p, part);
    return s1 != QSGB_OK ? s1 : launch_stage2(part, (int)nb, E, dptm, s);
  }
  const bool two = p.nmt > kGradBlock;
  int st;
  if (dtype == QSGB_F64)
    st = two ? launch_stage1<double, 2>(p, nb, part, s) : launch_stage1<double, 1>(p, nb, part, s);
  else
    st = two ? launch_stage1<float, 2>(p, nb, part, s) : launch_stage1<float, 1>(p, nb, part, s);
  if (st != QSGB_OK) return st;
  return launch_stage2(part, (int)nb, E, dptm, s);
}

}  // namespace
}  // namespace qsgb

extern "C" int64_t qsgb_ptm_grad_scratch_bytes(int64_t n_groups, int64_t k_out, int64_t k_in) {
  if (n_groups < 1 || k_out < 1 || k_in < 1) return 0;
  const int tg = qsgb::grad_tile((int)std::min<int64_t>(k_out + k_in, 1 << 20));
  return (int64_t)qsgb::grad_blocks((uint64_t)n_groups, tg) * k_out * k_in * (int64_t)sizeof(double);
}

extern "C" int qsgb_ptm_grad1(const void* x_in, const void* g_out, double* dptm, int64_t d_out, int64_t d_in,
                              int64_t dim_y, int64_t dim_z, int dtype, void* scratch, int64_t scratch_bytes,
                              void* stream) {
  return qsgb::grad_common(x_in, g_out, dptm, 1, d_out, 1, d_in, 1, dim_y, dim_z, dtype, scratch, scratch_bytes,
                           stream);
}

extern "C" int qsgb_ptm_grad2(const void* x_in, const void* g_out, double* dptm, int64_t d0_out, int64_t d1_out,
                              int64_t d0_in, int64_t d1_in, int64_t dim_x, int64_t dim_y, int64_t dim_z, int dtype,
                              void* scratch, int64_t scratch_bytes, void* stream) {
  return qsgb::grad_common(x_in, g_out, dptm, d0_out, d1_out, d0_in, d1_in, dim_x, dim_y, dim_z, dtype, scratch,
                           scratch_bytes, stream);
}
