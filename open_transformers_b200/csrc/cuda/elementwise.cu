// Memory-bound kernels of the transformer block for sm_100a: RMSNorm fwd/bwd, gain-free QK-norm
// fused with RoPE fwd/bwd, SwiGLU fwd/bwd, fused cross-entropy + z-loss fwd+bwd, embedding
// gather and its deterministic backward, canonical sums.
//
// Every reduction follows csrc/common/det_reduce.h and every transcendental comes from
// csrc/common/det_math.h, so csrc/cpu/ref_ops.cpp returns the same bits.
// Activations are templated on T in {bf16, float}; arithmetic is always fp32 with one
// rounding to T at the store.
//
// Reference roles: repop rms_norm (src/pretrain/model/modules/norm_repop.py:19-22), silu
// (ffn_repop.py:52-54), apply_rope (rope.py:103-125), fused_ce_z_loss (model/fused_loss.py:40-104),
// deterministic embedding backward (embedding_repop.py:3-10).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"
#include "det_math.h"
#include "entries.cuh"
#include "ew_common.cuh"
#include "tc05.cuh"

namespace {


// ------------------------------------------------------------------ RMSNorm
// One warp per row; lane_tree with VW = 8. The row stays in registers (as loaded) between the sum of squares and the
// scaling, so all of its loads are in flight at once and x is read once. MAXC = max number of 8-wide column chunks per
// lane (D <= 256 * MAXC).
template <typename T, int MAXC>
__global__ void __launch_bounds__(256) rmsnorm_fwd_kernel(const T* x, const T* w, T* __restrict__ y,
                                                         float* __restrict__ rstd_out, long rows, int D, float inv_d, float eps) {
  after_predecessor();
  const long row = (long)blockIdx.x * 8 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (row >= rows) return;
  const T* xr = x + row * D;
  Raw8<T> raw[MAXC];
#pragma unroll
  for (int j = 0; j < MAXC; ++j) {
    const int c = lane * 8 + j * 256;
    if (c < D) raw[j].load(xr + c);
  }
  float acc = 0.0f;
#pragma unroll
  for (int j = 0; j < MAXC; ++j) {
    if (lane * 8 + j * 256 < D) {
      float f[8];
      raw[j].unpack(f);
#pragma unroll
      for (int e = 0; e < 8; ++e) acc = __fmaf_rn(f[e], f[e], acc);
    }
  }
  const float ss = warp_butterfly(acc);
  const float rstd = det_rsqrtf(__fadd_rn(__fmul_rn(ss, inv_d), eps));
  if (lane == 0) rstd_out[row] = rstd;
  T* yr = y + row * D;
#pragma unroll
  for (int j = 0; j < MAXC; ++j) {
    const int c = lane * 8 + j * 256;
    if (c < D) {
      float f[8], o[8];
      raw[j].unpack(f);
      if (w) {
        float g[8];
        Vec8<T>::load(w + c, g);
#pragma unroll
        for (int e = 0; e < 8; ++e) o[e] = __fmul_rn(__fmul_rn(f[e], rstd), g[e]);
      } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) o[e] = __fmul_rn(f[e], rstd);
      }
      Vec8<T>::store(yr + c, o);
    }
  }
}
// The same row of any width: x is read twice, the second time from the nearer caches, U groups of eight columns per lane and turn,
// all loaded before any is stored (behind a store the next turn's loads would wait).
template <typename T, int U>
__global__ void __launch_bounds__(256) rmsnorm_fwd_wide_kernel(const T* x, const T* w, T* __restrict__ y, float* __restrict__ rstd_out, long rows,
                                                              int D, float inv_d, float eps) {
  after_predecessor();
  const long row = (long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (row >= rows) return;
  const T* xr = x + row * D;
  float acc = 0.0f;
  for (int c = lane * 8; c < D; c += 256) {
    float f[8];
    Vec8<T>::load(xr + c, f);
#pragma unroll
    for (int e = 0; e < 8; ++e) acc = __fmaf_rn(f[e], f[e], acc);
  }
  const float ss = warp_butterfly(acc);
  const float rstd = det_rsqrtf(__fadd_rn(__fmul_rn(ss, inv_d), eps));
  if (lane == 0) rstd_out[row] = rstd;
  T* yr = y + row * D;
  for (int c0 = lane * 8; c0 < D; c0 += 256 * U) {
    Raw8<T> rx[U], rw[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int c = c0 + u * 256;
      if (c < D) {
        rx[u].load(xr + c);
        if (w) rw[u].load(w + c);
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int c = c0 + u * 256;
      if (c < D) {
        float f[8], o[8];
        rx[u].unpack(f);
        if (w) {
          float g[8];
          rw[u].unpack(g);
#pragma unroll
          for (int e = 0; e < 8; ++e) o[e] = __fmul_rn(__fmul_rn(f[e], rstd), g[e]);
        } else {
#pragma unroll
          for (int e = 0; e < 8; ++e) o[e] = __fmul_rn(f[e], rstd);
        }
        Vec8<T>::store(yr + c, o);
      }
    }
  }
}

// Where the row stays in registers. The second reading of a bf16 row is cheap (L1) and a warp that holds a long row has less to
// overlap, so bf16 rows of 1024 columns and more gain only where that reading misses, in long rows of a tensor far above the
// L2; fp32 rows, twice the bytes, gain at every width. us, two readings and registers: bf16 64 x 2048 3.6 and 4.5, 1200 x 1024
// 2.95 and 3.3, 8192 x 2048 9.2 and 10.4, 16384 x 2048 23.0 and 24.7, 4096 x 4096 10.3 and 13.9, 16384 x 4096 57.6 and 50.1; 1200 x
// 768 3.15 and 3.05; fp32 64 x 2048 5.2 and 4.7, 16384 x 2048 64 and 53.
inline bool rmsnorm_in_registers(long rows, int D, bool bf16) {
  if (D > 4096) return false;
  return !bf16 || D <= 768 || (D > 2048 && rows >= 12288);
}

// One CTA of SLAB warps per slab of SLAB rows, one warp per row: the row stays in registers (as loaded, 16-byte
// vectors) between the dot product and the dx pass, so x and dy are read once. dgamma partial [slab][D] is the
// ascending-row fold inside the slab: every warp leaves its row's dy * xhat products in shared memory and, after one
// barrier, the CTA adds the SLAB rows of each column in row order (the same chain a single warp would have run).
// MAXC = max number of 8-wide column chunks per lane (D <= 256 * MAXC).
constexpr int NORM_SLAB = 8;
template <typename T, int MAXC>
__global__ void __launch_bounds__(NORM_SLAB * 32) rmsnorm_bwd_kernel(const T* dy, const T* x, const T* w,
                                                                    const float* rstd_in, T* __restrict__ dx,
                                                                    float* __restrict__ dgamma_partial, long rows, int D, float inv_d) {
  wait_for_predecessor();
  extern __shared__ float prod[];  // [NORM_SLAB][MAXC * 256] when dgamma is wanted
  const long slab = blockIdx.x;
  const int lane = threadIdx.x & 31, wrow = threadIdx.x >> 5;
  const long row = slab * NORM_SLAB + wrow;
  const bool live = row < rows;
  if (live) {
    const float rstd = rstd_in[row];
    const T* xr = x + row * D;
    const T* dyr = dy + row * D;
    Raw8<T> xraw[MAXC], draw[MAXC];
#pragma unroll
    for (int j = 0; j < MAXC; ++j) {
      const int c = lane * 8 + j * 256;
      if (c < D) {
        xraw[j].load(xr + c);
        draw[j].load(dyr + c);
      }
    }
    float acc = 0.0f;
#pragma unroll
    for (int j = 0; j < MAXC; ++j) {
      const int c = lane * 8 + j * 256;
      if (c < D) {
        float xf[8], df[8], g[8];
        xraw[j].unpack(xf);
        draw[j].unpack(df);
        if (w) Vec8<T>::load(w + c, g);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const float xh = __fmul_rn(xf[e], rstd);
          const float gy = w ? __fmul_rn(df[e], g[e]) : df[e];
          acc = __fmaf_rn(gy, xh, acc);
          if (dgamma_partial) prod[wrow * (MAXC * 256) + j * 256 + e * 32 + lane] = __fmul_rn(df[e], xh);  // lanes side by side: no bank conflict
        }
      }
    }
    const float cs = __fmul_rn(warp_butterfly(acc), inv_d);
    T* dxr = dx + row * D;
#pragma unroll
    for (int j = 0; j < MAXC; ++j) {
      const int c = lane * 8 + j * 256;
      if (c < D) {
        float xf[8], df[8], g[8], o[8];
        xraw[j].unpack(xf);
        draw[j].unpack(df);
        if (w) Vec8<T>::load(w + c, g);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const float xh = __fmul_rn(xf[e], rstd);
          const float gy = w ? __fmul_rn(df[e], g[e]) : df[e];
          o[e] = __fmul_rn(rstd, __fmaf_rn(-xh, cs, gy));
        }
        Vec8<T>::store(dxr + c, o);
      }
    }
  }
  if (dgamma_partial) {
    __syncthreads();
    const int nrow = (int)((rows - slab * NORM_SLAB < NORM_SLAB) ? rows - slab * NORM_SLAB : NORM_SLAB);
    float* out = dgamma_partial + slab * D;
    for (int j = wrow; j < MAXC; j += NORM_SLAB) {  // warp j folds column chunk j; a lane owns the same 8 columns as above
      const int c = lane * 8 + j * 256;
      if (c < D) {
        float a[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          float t = 0.0f;
          for (int r = 0; r < nrow; ++r) t = __fadd_rn(t, prod[r * (MAXC * 256) + j * 256 + e * 32 + lane]);
          a[e] = t;
        }
        *reinterpret_cast<float4*>(out + c) = make_float4(a[0], a[1], a[2], a[3]);
        *reinterpret_cast<float4*>(out + c + 4) = make_float4(a[4], a[5], a[6], a[7]);
      }
    }
  }
}

// pair_tree over the leading dimension of v[n][D], in place; result in row 0.
// The tree "for s = 1, 2, 4..: v[i] += v[i+s] for i multiple of 2s, i+s < n" only ever pairs rows inside a
// 2s-aligned group, so groups of 64 rows are reduced independently in shared memory (levels s = 1..32) and the
// same kernel is then applied to the 64-strided group roots (levels 64..2048), and so on: identical association,
// log-depth instead of a serial chain. Logical row j lives at v[j * row_stride * D]. A missing partner leaves the
// value untouched (never "+ 0.0", which would turn -0.0 into +0.0).
__global__ void __launch_bounds__(256) pair_tree_cols_stage_kernel(float* v, long n, long row_stride, int D) {
  wait_for_predecessor();
  __shared__ float sm[64][33];
  const int c = threadIdx.x & 31, r = threadIdx.x >> 5;  // 32 columns x 8 row-threads
  const int col = blockIdx.x * 32 + c;
  const long g0 = (long)blockIdx.y * 64;                // first logical row of this group
  const long rows_here = min((long)64, n - g0);
  if (col < D)
    for (int rr = r; rr < rows_here; rr += 8) sm[rr][c] = v[(g0 + rr) * row_stride * D + col];
  __syncthreads();
  for (int s = 1; s < 64; s *= 2) {
    for (int i = r * 2 * s; i + s < rows_here; i += 16 * s) sm[i][c] = __fadd_rn(sm[i][c], sm[i + s][c]);
    __syncthreads();
  }
  if (col < D && r == 0) v[g0 * row_stride * D + col] = sm[0][c];
}

inline int pair_tree_cols_launch(float* v, long n, int D, cudaStream_t s) {
  long stride = 1;
  while (n > 1) {
    const long groups = (n + 63) / 64;
    dim3 grid((D + 31) / 32, (unsigned)groups);
    if (const int rc = otb_launch_early(pair_tree_cols_stage_kernel, grid, 256, 0, s, v, n, stride, D)) return rc;
    n = groups;
    stride *= 64;
  }
  return 0;
}

// ------------------------------------------------------------ per-head RMSNorm with gain
// The RMSNorm of every head of a [tokens, ld] buffer (head h in columns h*D .. h*D + D - 1, D <= 128, multiple of 8), read
// and written in place of its columns: the same sums as the row kernels above on [tokens * heads, D] (lane_tree with VW = 8
// uses 16 of its 32 lanes at this width; the other sixteen add +0.0 once), without copies that make the heads contiguous and
// copies that join them again. Sixteen lanes per row, so a warp works on two.
__device__ __forceinline__ float half_butterfly(float v) {
  v = __fadd_rn(v, 0.0f);  // the partner at distance 16 holds no element
#pragma unroll
  for (int off = 8; off >= 1; off >>= 1) v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, off));
  return v;
}
template <typename T>
__global__ void __launch_bounds__(256) head_rmsnorm_fwd_kernel(const T* x, long ldx, const T* w, T* __restrict__ y, long ldy,
                                                              float* __restrict__ rstd_out, long rows, int heads, int D, float inv_d, float eps) {
  wait_for_predecessor();
  const long row = (long)blockIdx.x * 16 + (threadIdx.x >> 4);
  const int c = (threadIdx.x & 15) * 8;
  const bool on = row < rows && c < D;
  const long tok = row / heads;
  const long at = (row - tok * heads) * D + c;
  Raw8<T> raw;
  float acc = 0.0f;
  if (on) {
    raw.load(x + tok * ldx + at);
    float f[8];
    raw.unpack(f);
#pragma unroll
    for (int e = 0; e < 8; ++e) acc = __fmaf_rn(f[e], f[e], acc);
  }
  const float ss = half_butterfly(acc);
  const float rstd = det_rsqrtf(__fadd_rn(__fmul_rn(ss, inv_d), eps));
  if (on) {
    if (c == 0) rstd_out[row] = rstd;
    float f[8], g[8], o[8];
    raw.unpack(f);
    Vec8<T>::load(w + c, g);
#pragma unroll
    for (int e = 0; e < 8; ++e) o[e] = __fmul_rn(__fmul_rn(f[e], rstd), g[e]);
    Vec8<T>::store(y + tok * ldy + at, o);
  }
}
// dx and the dgamma partials of NORM_SLAB-row slabs (rows = (token, head) pairs); two slabs per CTA.
template <typename T>
__global__ void __launch_bounds__(256) head_rmsnorm_bwd_kernel(const T* dy, long lddy, const T* x, long ldx, const T* w,
                                                              const float* rstd_in, T* __restrict__ dx, long lddx,
                                                              float* __restrict__ dgamma_partial, long rows, int heads, int D, float inv_d) {
  wait_for_predecessor();
  __shared__ float prod[16][128];
  const int r = threadIdx.x >> 4, c = (threadIdx.x & 15) * 8;
  const long row = (long)blockIdx.x * 16 + r;
  const bool on = row < rows && c < D;
  const long tok = row / heads;
  const long at = (row - tok * heads) * D + c;
  float xh[8], gy[8], acc = 0.0f, rstd = 0.0f;
  if (on) {
    rstd = rstd_in[row];
    float xf[8], df[8], g[8];
    Vec8<T>::load(x + tok * ldx + at, xf);
    Vec8<T>::load(dy + tok * lddy + at, df);
    Vec8<T>::load(w + c, g);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      xh[e] = __fmul_rn(xf[e], rstd);
      gy[e] = __fmul_rn(df[e], g[e]);
      acc = __fmaf_rn(gy[e], xh[e], acc);
      if (dgamma_partial) prod[r][c + e] = __fmul_rn(df[e], xh[e]);
    }
  }
  const float cs = __fmul_rn(half_butterfly(acc), inv_d);
  if (on) {
    float o[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) o[e] = __fmul_rn(rstd, __fmaf_rn(-xh[e], cs, gy[e]));
    Vec8<T>::store(dx + tok * lddx + at, o);
  }
  if (dgamma_partial) {
    __syncthreads();
    const int slab = threadIdx.x >> 7, col = threadIdx.x & 127;
    const long first = (long)blockIdx.x * 16 + slab * NORM_SLAB;
    if (first < rows && col < D) {
      const int n = (int)min((long)NORM_SLAB, rows - first);
      float t = 0.0f;
      for (int i = 0; i < n; ++i) t = __fadd_rn(t, prod[slab * NORM_SLAB + i][col]);
      dgamma_partial[(first / NORM_SLAB) * D + col] = t;
    }
  }
}

// --------------------------------------------------- gain-free QK-norm + RoPE
// Over the first `heads` heads of a [rows, ld_in] buffer with head width D (<= 128, multiple of 4): lane l of a warp holds
// elements 4l..4l+3 of a head (two rotation pairs). out[row, head*D + i]; rstd[row*heads + head]. lane_tree with VW = 4.
// A warp takes NH heads of one token: the token's cos / sin are read once for all of them and their loads (8 bytes
// per lane in bf16) are in flight together; one head per warp with 2-byte loads and two 64-bit divisions per warp was bound
// by its instructions (76 us forward, 86 us backward at 16384 tokens x 20 heads x 128; with the row sums of the attention
// backward regrouped the same way, that layer's pass went from 864 to 761 us with a 512-key window). VEC: bases and pitches allow the four-element accesses.
// Four heads per warp need enough heads to fill the chip: us, one and four per warp, 100 tokens x 5 heads x 128 2.5 and 2.9,
// 300 x 16 3.0 and 3.0, 1000 x 5 3.2 and 3.1, 2000 x 5 4.5 and 3.9; a single head per token leaves three quarters of the registers
// unused (32768 x 1 x 64 backward: 9.5 and 11.5).
constexpr int ROPE_HEADS = 4;
inline bool rope_one_head(long rows, int heads) { return heads == 1 || rows * heads < 4800; }
template <typename T, bool VEC> struct Vec4;
template <> struct Vec4<__nv_bfloat16, true> {
  uint2 v;
  __device__ __forceinline__ void load(const __nv_bfloat16* p) { v = *reinterpret_cast<const uint2*>(p); }
  __device__ __forceinline__ void unpack(float (&f)[4]) const {
    f[0] = __uint_as_float(v.x << 16); f[1] = __uint_as_float(v.x & 0xFFFF0000u);
    f[2] = __uint_as_float(v.y << 16); f[3] = __uint_as_float(v.y & 0xFFFF0000u);
  }
  static __device__ __forceinline__ void store(__nv_bfloat16* p, const float (&f)[4]) {
    __nv_bfloat162 a = __floats2bfloat162_rn(f[0], f[1]), b = __floats2bfloat162_rn(f[2], f[3]);
    *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<uint32_t*>(&a), *reinterpret_cast<uint32_t*>(&b));
  }
};
template <> struct Vec4<float, true> {
  float4 v;
  __device__ __forceinline__ void load(const float* p) { v = *reinterpret_cast<const float4*>(p); }
  __device__ __forceinline__ void unpack(float (&f)[4]) const { f[0] = v.x; f[1] = v.y; f[2] = v.z; f[3] = v.w; }
  static __device__ __forceinline__ void store(float* p, const float (&f)[4]) { *reinterpret_cast<float4*>(p) = make_float4(f[0], f[1], f[2], f[3]); }
};
template <typename T> struct Vec4<T, false> {
  T v[4];
  __device__ __forceinline__ void load(const T* p) {
#pragma unroll
    for (int e = 0; e < 4; ++e) v[e] = p[e];
  }
  __device__ __forceinline__ void unpack(float (&f)[4]) const {
#pragma unroll
    for (int e = 0; e < 4; ++e) f[e] = to_f<T>(v[e]);
  }
  static __device__ __forceinline__ void store(T* p, const float (&f)[4]) {
#pragma unroll
    for (int e = 0; e < 4; ++e) p[e] = from_f<T>(f[e]);
  }
};
// warp -> (token, first head); false past the end
template <int NH>
__device__ __forceinline__ bool rope_place(long rows, int heads, long& row, int& head0) {
  const int groups = (heads + NH - 1) / NH;
  const long wid = (long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (wid >= rows * groups) return false;
  row = (rows * groups) >> 31 ? wid / groups : (long)((unsigned)wid / (unsigned)groups);
  head0 = (int)(wid - row * groups) * NH;
  return true;
}
__device__ __forceinline__ int rope_pos(long row, int seq_len) { return row >> 31 ? (int)(row % seq_len) : (int)((unsigned)row % (unsigned)seq_len); }

template <typename T, bool VEC, int NH>
__global__ void __launch_bounds__(256) qknorm_rope_fwd_kernel(const T* in, long ld_in, T* __restrict__ out, long ld_out,
                                       float* __restrict__ rstd_out, const float* cosb,
                                       const float* sinb, long rows, int heads, int D, int seq_len,
                                       int do_norm, float inv_d, float eps) {
  after_predecessor();
  long row;
  int head0;
  if (!rope_place<NH>(rows, heads, row, head0)) return;
  const int lane = threadIdx.x & 31;
  const bool active = lane * 4 < D;
  const int n = min(NH, heads - head0);
  Vec4<T, VEC> raw[NH];
  const T* p = in + row * ld_in + (long)head0 * D + lane * 4;
#pragma unroll
  for (int i = 0; i < NH; ++i)
    if (active && i < n) raw[i].load(p + i * D);
  float c[2] = {0.f, 0.f}, s[2] = {0.f, 0.f};
  if (active) {
    const long at = (long)rope_pos(row, seq_len) * (D >> 1) + lane * 2;
#pragma unroll
    for (int pr = 0; pr < 2; ++pr) { c[pr] = cosb[at + pr]; s[pr] = sinb[at + pr]; }
  }
  // The heads' sums first, then lane i finds the root of head i: one square root and division for all of them. (Every lane finding every
  // head's: 16384 tokens x 20 heads x 128 38.9 us, so 35.6; 1000 x 16 x 64 4.8 and 4.2.)
  float rstd = 0.0f;
  if (do_norm) {
    float mine = 0.0f;
#pragma unroll
    for (int i = 0; i < NH; ++i) {
      float f[4] = {0.f, 0.f, 0.f, 0.f}, acc = 0.0f;
      if (active && i < n) raw[i].unpack(f);
#pragma unroll
      for (int e = 0; e < 4; ++e) acc = __fmaf_rn(f[e], f[e], acc);
      const float ss = warp_butterfly(acc);
      if (lane == i) mine = ss;
    }
    rstd = det_rsqrtf(__fadd_rn(__fmul_rn(mine, inv_d), eps));
    if (lane < n) rstd_out[row * heads + head0 + lane] = rstd;
  }
  T* o = out + row * ld_out + (long)head0 * D + lane * 4;
#pragma unroll
  for (int i = 0; i < NH; ++i) {
    if (i >= n) break;  // (the same for the whole warp)
    float f[4] = {0.f, 0.f, 0.f, 0.f};
    if (active) raw[i].unpack(f);
    if (do_norm) {
      const float r = __shfl_sync(0xffffffffu, rstd, i);
#pragma unroll
      for (int e = 0; e < 4; ++e) f[e] = __fmul_rn(f[e], r);
    }
    if (active) {
      float r[4];
#pragma unroll
      for (int pr = 0; pr < 2; ++pr) {
        const float xe = f[2 * pr], xo = f[2 * pr + 1];
        r[2 * pr] = __fmaf_rn(xe, c[pr], -__fmul_rn(xo, s[pr]));
        r[2 * pr + 1] = __fmaf_rn(xe, s[pr], __fmul_rn(xo, c[pr]));
      }
      Vec4<T, VEC>::store(o + i * D, r);
    }
  }
}

template <typename T, bool VEC, int NH>
__global__ void __launch_bounds__(256) qknorm_rope_bwd_kernel(const T* dout, long ld_dout, const T* in, long ld_in,
                                       const float* rstd_in, T* __restrict__ din, long ld_din,
                                       const float* cosb, const float* sinb, long rows,
                                       int heads, int D, int seq_len, int do_norm, float inv_d) {
  after_predecessor();
  long row;
  int head0;
  if (!rope_place<NH>(rows, heads, row, head0)) return;
  const int lane = threadIdx.x & 31;
  const bool active = lane * 4 < D;
  const int n = min(NH, heads - head0);
  Vec4<T, VEC> rd[NH], rx[NH];
  float rstd[NH];
  const T* pd = dout + row * ld_dout + (long)head0 * D + lane * 4;
  const T* px = in + row * ld_in + (long)head0 * D + lane * 4;
#pragma unroll
  for (int i = 0; i < NH; ++i) {
    if (active && i < n) {
      rd[i].load(pd + i * D);
      if (do_norm) rx[i].load(px + i * D);
    }
    rstd[i] = do_norm && i < n ? rstd_in[row * heads + head0 + i] : 0.0f;
  }
  float c[2] = {0.f, 0.f}, s[2] = {0.f, 0.f};
  if (active) {
    const long at = (long)rope_pos(row, seq_len) * (D >> 1) + lane * 2;
#pragma unroll
    for (int pr = 0; pr < 2; ++pr) { c[pr] = cosb[at + pr]; s[pr] = sinb[at + pr]; }
  }
  T* o = din + row * ld_din + (long)head0 * D + lane * 4;
#pragma unroll
  for (int i = 0; i < NH; ++i) {
    if (i >= n) break;
    float g[4] = {0.f, 0.f, 0.f, 0.f};
    if (active) {
      float d[4];
      rd[i].unpack(d);
#pragma unroll
      for (int pr = 0; pr < 2; ++pr) {
        const float de = d[2 * pr], dd = d[2 * pr + 1];
        g[2 * pr] = __fmaf_rn(de, c[pr], __fmul_rn(dd, s[pr]));
        g[2 * pr + 1] = __fmaf_rn(dd, c[pr], -__fmul_rn(de, s[pr]));
      }
    }
    if (do_norm) {
      float xh[4] = {0.f, 0.f, 0.f, 0.f};
      if (active) {
        rx[i].unpack(xh);
#pragma unroll
        for (int e = 0; e < 4; ++e) xh[e] = __fmul_rn(xh[e], rstd[i]);
      }
      float acc = 0.0f;
#pragma unroll
      for (int e = 0; e < 4; ++e) acc = __fmaf_rn(g[e], xh[e], acc);
      const float cs = __fmul_rn(warp_butterfly(acc), inv_d);
#pragma unroll
      for (int e = 0; e < 4; ++e) g[e] = __fmul_rn(rstd[i], __fmaf_rn(-xh[e], cs, g[e]));
    }
    if (active) Vec4<T, VEC>::store(o + i * D, g);
  }
}

// ------------------------------------------------------------------- SwiGLU
// gate_up [rows, 2F] (gate = cols [0,F), up = cols [F,2F)) -> h [rows, F] = silu(gate) * up
// silu(g) * u of eight elements, and its gradient (dg, du) from d
template <typename T>
__device__ __forceinline__ void swiglu8(const Raw8<T>& rg, const Raw8<T>& ru, T* h) {
  float g[8], u[8], o[8];
  rg.unpack(g);
  ru.unpack(u);
#pragma unroll
  for (int e = 0; e < 8; e += 2) {
    const tc05::f2 g2 = tc05::pack2(g[e], g[e + 1]);
    tc05::unpack2(tc05::mul2(tc05::mul2(g2, tc05::sigmoid_fast2(g2)), tc05::pack2(u[e], u[e + 1])), o[e], o[e + 1]);
  }
  Vec8<T>::store(h, o);
}
template <typename T>
__device__ __forceinline__ void swiglu8_bwd(const Raw8<T>& rg, const Raw8<T>& ru, const Raw8<T>& rd, T* dg, T* du) {
  using namespace tc05;
  float g[8], u[8], d[8], og[8], ou[8];
  rg.unpack(g);
  ru.unpack(u);
  rd.unpack(d);
#pragma unroll
  for (int e = 0; e < 8; e += 2) {
    const f2 g2 = pack2(g[e], g[e + 1]), u2 = pack2(u[e], u[e + 1]), d2 = pack2(d[e], d[e + 1]);
    const f2 sg = sigmoid_fast2(g2);
    const f2 silu = mul2(g2, sg);
    // d silu / dg = sg * (1 + g (1 - sg))
    const f2 one = pack2(1.0f, 1.0f);
    const f2 dsilu = mul2(sg, fma2(g2, add2(one, mul2(sg, pack2(-1.0f, -1.0f))), one));
    unpack2(mul2(mul2(d2, u2), dsilu), og[e], og[e + 1]);
    unpack2(mul2(d2, silu), ou[e], ou[e + 1]);
  }
  Vec8<T>::store(dg, og);
  Vec8<T>::store(du, ou);
}
// One thread per group of eight, wherever its row is.
template <typename T>
__global__ void __launch_bounds__(256) swiglu_fwd_flat_kernel(const T* gu, T* __restrict__ h, long rows, int F) {
  after_predecessor();
  const long idx = ((long)blockIdx.x * blockDim.x + threadIdx.x) * 8;
  if (idx >= rows * F) return;
  const long row = idx / F;
  const T* gr = gu + row * 2 * F + (idx - row * F);
  Raw8<T> g, u;
  g.load(gr);
  u.load(gr + F);
  swiglu8(g, u, h + idx);
}
template <typename T>
__global__ void __launch_bounds__(256) swiglu_bwd_flat_kernel(const T* gu, const T* dh, T* __restrict__ dgu, long rows, int F) {
  after_predecessor();
  const long idx = ((long)blockIdx.x * blockDim.x + threadIdx.x) * 8;
  if (idx >= rows * F) return;
  const long row = idx / F, at = row * 2 * F + (idx - row * F);
  Raw8<T> g, u, d;
  g.load(gu + at);
  u.load(gu + at + F);
  d.load(dh + idx);
  swiglu8_bwd(g, u, d, dgu + at, dgu + at + F);
}
// One CTA per row, two groups per thread and sweep with all their loads in flight: no index division (a 64-bit one per group
// costs as much as the activation), and enough bytes in flight per SM to hold the memory's rate. It needs rows that fill its
// warps and enough of them; narrow rows leave lanes idle and end up as many CTAs with next to nothing to do, and a few wide rows
// leave SMs idle. bf16, flat and per row, us, forward: 20000 x 5632 120 and 101, 10000 x 2048 24.1 and 20.5, 4800 x 1024 6.7
// and 6.3; 20000 x 704 16.0 and 19.2, 20000 x 352 8.8 and 12.4, 1048576 x 64 73 and 544; 64 x 5632 2.4 and 2.8, 600 x 16384
// 11.4 and 12.5, 1200 x 1024 3.0 and 3.3. (Backward alike, its gain smaller: 20000 x 5632 164 and 160.)
constexpr int SWIGLU_MAX_THREADS = 384;
inline bool swiglu_per_row(long rows, int F) { return F >= 1024 && rows >= 2048 && rows <= 0x7fffffffL; }
template <typename T>
__global__ void __launch_bounds__(SWIGLU_MAX_THREADS) swiglu_fwd_kernel(const T* gu, T* __restrict__ h, int F) {
  after_predecessor();
  const T* gr = gu + (long)blockIdx.x * 2 * F;
  T* hr = h + (long)blockIdx.x * F;
  for (int c0 = threadIdx.x * 8; c0 < F; c0 += blockDim.x * 16) {
    Raw8<T> rg[2], ru[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int c = c0 + u * blockDim.x * 8;
      if (c < F) {
        rg[u].load(gr + c);
        ru[u].load(gr + F + c);
      }
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int c = c0 + u * blockDim.x * 8;
      if (c < F) swiglu8(rg[u], ru[u], hr + c);
    }
  }
}
// d_gate_up [rows, 2F] from dh [rows, F]
template <typename T>
__global__ void __launch_bounds__(SWIGLU_MAX_THREADS) swiglu_bwd_kernel(const T* gu, const T* dh, T* __restrict__ dgu, int F) {
  after_predecessor();
  const T* gr = gu + (long)blockIdx.x * 2 * F;
  const T* dr = dh + (long)blockIdx.x * F;
  T* or_ = dgu + (long)blockIdx.x * 2 * F;
  for (int c0 = threadIdx.x * 8; c0 < F; c0 += blockDim.x * 16) {
    Raw8<T> rg[2], ru[2], rd[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int c = c0 + u * blockDim.x * 8;
      if (c < F) {
        rg[u].load(gr + c);
        ru[u].load(gr + F + c);
        rd[u].load(dr + c);
      }
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int c = c0 + u * blockDim.x * 8;
      if (c < F) swiglu8_bwd(rg[u], ru[u], rd[u], or_ + c, or_ + F + c);
    }
  }
}
// threads per row: the row's groups split evenly over the sweeps of two groups per thread
inline int swiglu_threads(int F) {
  const int groups = F / 8, sweeps = (groups + 2 * SWIGLU_MAX_THREADS - 1) / (2 * SWIGLU_MAX_THREADS);
  const int t = (groups + 2 * sweeps - 1) / (2 * sweeps);
  return (t + 31) / 32 * 32;
}

// --------------------------------------------------------- fused CE + z-loss
// One CTA per row of logits [rows, V] (V % 8 == 0), of 512 threads or, for rows of fewer than 512 groups of 8, of fewer. With m = max of the row and L = log2(e):
//   e_i = exp2(fma(x_i, L, -(m * L)))        (det_exp2_acc, evaluated two at a time with packed fp32 arithmetic)
//   s   = sum e_i: the 8-element group g = i / 8 belongs to thread g % 512; a thread keeps two ascending chains, the
//         even and the odd elements of its groups, adds them, and the 512 thread sums go through block_tree_sum
//   lse = log(s) + m,  ce[row] = lse - x[label],  lse_out[row] = lse
// and the row is overwritten with d loss / d logits = e_i * k - onehot * scale, k = ((1 + 2 z lse) / s) * scale
// (scale = 1 / (tokens * accum), host reciprocal; the label's element is fma(e, k, -scale)).
// Rows with label < 0 are ignored: zero loss, zero gradient.
// Rows too long for the registers (the form below) are read three times, once from memory. They are bound by instructions, not by
// the reads (the maximum of bf16 logits is taken two at a time as bf16). Two things help the longest and cost others registers, and with
// them CTAs per SM (ce_form chooses):
//   TEST: the first pass finds the smallest logit too, and where it is near enough the exponent's clamp is left out;
//   UNROLL groups per thread are in flight.
// us for 16384 rows with their gradient; neither / TEST / TEST and four groups: bf16 V 32768 525 / 516 / 568, 65536 986 / 967 / 1073, 98304
// 1714 / 1672 / 1552; 4000 rows of 128256 622 / 624 / 542. fp32, 4000 rows: 16384 99 / 104 / 135, 32768 256 / 198 / 225, 65536 611 / 584 / 448;
// with a few rows per SM neither helps (64 rows of 128256: 30 / 34 / 37, 149: 52 / - / 60, 600: 222 / 231 / 209).
constexpr int CE_THREADS = 512, CE_SWEEP = CE_THREADS * 8;
template <typename T, int CE_UNROLL>
__device__ __forceinline__ void ce_fetch(Raw8<T> (&raw)[CE_UNROLL], const T* __restrict__ xr, int c0, int V) {
#pragma unroll
  for (int u = 0; u < CE_UNROLL; ++u)
    if (c0 + u * CE_SWEEP < V) raw[u].load(xr + c0 + u * CE_SWEEP);
}
// the thread's even and odd chains of sum e_i
template <typename T, int CE_UNROLL, bool CLAMP>
__device__ __forceinline__ tc05::f2 ce_sum(const T* __restrict__ xr, int V, tc05::f2 l2, tc05::f2 nm2) {
  using namespace tc05;
  Raw8<T> raw[CE_UNROLL];
  f2 acc2 = pack2(0.0f, 0.0f);
  for (int c0 = threadIdx.x * 8; c0 < V; c0 += CE_UNROLL * CE_SWEEP) {
    ce_fetch(raw, xr, c0, V);
#pragma unroll
    for (int u = 0; u < CE_UNROLL; ++u) {
      if (c0 + u * CE_SWEEP >= V) break;
      float f[8];
      raw[u].unpack(f);
#pragma unroll
      for (int e = 0; e < 8; e += 2) acc2 = add2(acc2, exp2_acc2<CLAMP>(fma2(pack2(f[e], f[e + 1]), l2, nm2)));
    }
  }
  return acc2;
}
// the thread's groups of the row become e_i * k; the owner of the label's group rewrites that one element
template <typename T, int CE_UNROLL, bool CLAMP>
__device__ __forceinline__ void ce_grad(T* __restrict__ xr, int V, tc05::f2 l2, tc05::f2 nm2, tc05::f2 k2, long label, float at_label) {
  using namespace tc05;
  Raw8<T> raw[CE_UNROLL];
  for (int c0 = threadIdx.x * 8; c0 < V; c0 += CE_UNROLL * CE_SWEEP) {
    ce_fetch(raw, xr, c0, V);
#pragma unroll
    for (int u = 0; u < CE_UNROLL; ++u) {
      const int c = c0 + u * CE_SWEEP;
      if (c >= V) break;
      float f[8], o[8];
      raw[u].unpack(f);
#pragma unroll
      for (int e = 0; e < 8; e += 2) unpack2(mul2(exp2_acc2<CLAMP>(fma2(pack2(f[e], f[e + 1]), l2, nm2)), k2), o[e], o[e + 1]);
      Vec8<T>::store(xr + c, o);
      if (label >= c && label < c + 8) xr[label] = from_f<T>(at_label);
    }
  }
}
template <typename T, int CE_UNROLL, bool TEST>
__global__ void __launch_bounds__(CE_THREADS) ce_zloss_kernel(T* logits, const long* labels,
                                                              float* __restrict__ ce_out, float* __restrict__ lse_out,
                                                              long rows, int V, float two_z, float scale, int write_grad) {
  after_predecessor();
  using namespace tc05;
  __shared__ float sh[32];
  const long row = blockIdx.x;
  T* xr = logits + row * V;
  const long label = labels[row];
  if (label < 0) {
    if (threadIdx.x == 0) { ce_out[row] = 0.0f; lse_out[row] = 0.0f; }
    if (write_grad) {
      float z[8] = {0, 0, 0, 0, 0, 0, 0, 0};
      for (int c = threadIdx.x * 8; c < V; c += CE_SWEEP) Vec8<T>::store(xr + c, z);
    }
    return;
  }
  const float x_label = to_f<T>(xr[label]);
  float mx = -INFINITY, mn = INFINITY;
  {
    Raw8<T> raw[CE_UNROLL];
    for (int c0 = threadIdx.x * 8; c0 < V; c0 += CE_UNROLL * CE_SWEEP) {
      ce_fetch(raw, xr, c0, V);
#pragma unroll
      for (int u = 0; u < CE_UNROLL; ++u) {
        if (c0 + u * CE_SWEEP >= V) break;
        raw[u].largest(mx);
        if (TEST) raw[u].smallest(mn);
      }
    }
  }
  mx = block_max(mx, sh);
  const float LOG2E = 1.44269504088896341f;
  const f2 l2 = pack2(LOG2E, LOG2E);
  const float nm = -__fmul_rn(mx, LOG2E);
  const f2 nm2 = pack2(nm, nm);
  // The exponent's clamp at -126 does nothing in a row whose smallest logit is above it (the exponent grows with the logit;
  // a NaN or an infinity fails the test): such rows, all of them in practice, leave it out, one instruction in eight.
  bool inside = false;
  if constexpr (TEST) inside = __syncthreads_and(__fmaf_rn(mn, LOG2E, nm) >= -126.0f);
  const f2 acc2 = inside ? ce_sum<T, CE_UNROLL, false>(xr, V, l2, nm2) : ce_sum<T, CE_UNROLL, true>(xr, V, l2, nm2);
  float a0, a1;
  unpack2(acc2, a0, a1);
  const float s = block_tree_sum(__fadd_rn(a0, a1), sh);
  const float lse = __fadd_rn(det_logf(s), mx);
  if (threadIdx.x == 0) {
    ce_out[row] = __fadd_rn(lse, -x_label);
    lse_out[row] = lse;
  }
  if (!write_grad) return;
  __syncthreads();  // every thread has its copy of the label logit before anyone overwrites the row
  const float k = __fmul_rn(__fdiv_rn(__fmaf_rn(two_z, lse, 1.0f), s), scale);
  const f2 k2 = pack2(k, k);
  const float at_label = __fmaf_rn(det_exp2_acc(__fmaf_rn(x_label, LOG2E, nm)), k, -scale);
  if (inside) ce_grad<T, CE_UNROLL, false>(xr, V, l2, nm2, k2, label, at_label);
  else ce_grad<T, CE_UNROLL, true>(xr, V, l2, nm2, k2, label, at_label);
}

// Rows of up to GROUPS groups per thread: the row is read once and its e_i stay in registers from the sum to the gradient, which
// halves both the reading passes and the exponentials. Same chains and trees, so the same bits; rows of fewer than 512 groups
// take a CTA of fewer threads (the sums that are missing from the tree are zeros in the other form). Bound by memory and, below
// 2048 columns, by the row's two reductions. us, three passes and so: bf16 64 x 1024 3.4 and 2.5, 16384 x 1024 89 and 21, 8192 x 2048
// 52 and 22, 8192 x 4096 67 and 46, 8192 x 8192 108 and 64 (4.2 TB/s), 8192 x 12288 139 and 104, 16384 x 16384 296 and 239; fp32 2048 x 1024
// 12.5 and 5.1, 8192 x 4096 81 and 58, 4000 x 8192 60 and 52, but 4000 x 16384 99 and 108: four groups of fp32 leave too few rows on an SM.
template <typename T, int GROUPS>
__global__ void __launch_bounds__(CE_THREADS) ce_zloss_short_kernel(T* logits, const long* labels, float* __restrict__ ce_out, float* __restrict__ lse_out,
                                                                    int V, float two_z, float scale, int write_grad) {
  after_predecessor();
  using namespace tc05;
  __shared__ float sh[32];
  const long row = blockIdx.x;
  T* xr = logits + row * V;
  const int c0 = threadIdx.x * 8;
  Raw8<T> raw[GROUPS];
  ce_fetch(raw, xr, c0, V);
  const long label = labels[row];
  if (label < 0) {
    if (threadIdx.x == 0) { ce_out[row] = 0.0f; lse_out[row] = 0.0f; }
    if (write_grad) {
      float z[8] = {0, 0, 0, 0, 0, 0, 0, 0};
      for (int c = c0; c < V; c += CE_SWEEP) Vec8<T>::store(xr + c, z);
    }
    return;
  }
  const float x_label = to_f<T>(xr[label]);
  float mx = -INFINITY;
#pragma unroll
  for (int u = 0; u < GROUPS; ++u)
    if (c0 + u * CE_SWEEP < V) raw[u].largest(mx);
  mx = block_max(mx, sh);
  const float LOG2E = 1.44269504088896341f;
  const f2 l2 = pack2(LOG2E, LOG2E);
  const float nm = -__fmul_rn(mx, LOG2E);
  const f2 nm2 = pack2(nm, nm);
  f2 e2[GROUPS][4], acc2 = pack2(0.0f, 0.0f);
#pragma unroll
  for (int u = 0; u < GROUPS; ++u) {
    if (c0 + u * CE_SWEEP < V) {
      float f[8];
      raw[u].unpack(f);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        e2[u][e] = exp2_acc2(fma2(pack2(f[2 * e], f[2 * e + 1]), l2, nm2));
        acc2 = add2(acc2, e2[u][e]);
      }
    }
  }
  float a0, a1;
  unpack2(acc2, a0, a1);
  const float s = block_tree_sum(__fadd_rn(a0, a1), sh);
  const float lse = __fadd_rn(det_logf(s), mx);
  if (threadIdx.x == 0) {
    ce_out[row] = __fadd_rn(lse, -x_label);
    lse_out[row] = lse;
  }
  if (!write_grad) return;
  const float k = __fmul_rn(__fdiv_rn(__fmaf_rn(two_z, lse, 1.0f), s), scale);
  const f2 k2 = pack2(k, k);
  const float at_label = __fmaf_rn(det_exp2_acc(__fmaf_rn(x_label, LOG2E, nm)), k, -scale);
#pragma unroll
  for (int u = 0; u < GROUPS; ++u) {
    const int c = c0 + u * CE_SWEEP;
    if (c < V) {
      float o[8];
#pragma unroll
      for (int e = 0; e < 4; ++e) unpack2(mul2(e2[u][e], k2), o[2 * e], o[2 * e + 1]);
      Vec8<T>::store(xr + c, o);
      if (label >= c && label < c + 8) xr[label] = from_f<T>(at_label);
    }
  }
}
// threads of a short row's CTA: a power of two of at least one warp
inline unsigned ce_short_threads(int V) {
  unsigned t = CE_THREADS;
  while (t > 32 && (int)(t / 2) * 8 >= V) t /= 2;
  return t;
}

// Form of the loss kernel for longer rows: 0 neither, 1 TEST, 4 TEST and four groups in flight. The lines lie where the figures above cross.
inline int ce_form(long rows, int V, bool bf16) {
  if (bf16) return V <= 20 * CE_SWEEP ? 1 : 4;
  return V <= 6 * CE_SWEEP || rows <= 4 * otb_sm_count() ? 0 : V <= 8 * CE_SWEEP ? 1 : 4;
}

// sum (or sum of squares) of n floats: element i -> thread i % 1024, ascending fold, block_tree_sum.
// mode 0: sum x, 1: sum x*x (fma chain). out[0] = result * post_scale.
__global__ void __launch_bounds__(1024) det_sum_kernel(const float* x, long n, int mode, float post_scale,
                                                        float* __restrict__ out) {
  wait_for_predecessor();
  __shared__ float sh[32];
  float acc = 0.0f;
  for (long i = threadIdx.x; i < n; i += 1024) {
    const float v = x[i];
    acc = mode ? __fmaf_rn(v, v, acc) : __fadd_rn(acc, v);
  }
  const float s = block_tree_sum(acc, sh);
  if (threadIdx.x == 0) out[0] = __fmul_rn(s, post_scale);
}

// ---------------------------------------------------------------- embedding
template <typename T>
__global__ void embedding_fwd_kernel(const long* __restrict__ ids, const T* __restrict__ table, T* __restrict__ out,
                                     long rows, int D) {
  const long row = blockIdx.x;
  const long id = ids[row];
  const uint4* src = reinterpret_cast<const uint4*>(table + id * D);
  uint4* dst = reinterpret_cast<uint4*>(out + row * D);
  const int nvec = D * (int)sizeof(T) / 16;
  for (int i = threadIdx.x; i < nvec; i += blockDim.x) dst[i] = src[i];
}
// sorted_ids: the n token ids in ascending order (stable sort); sorted_tok: the token position of each. One CTA per
// sorted position: the CTA at the HEAD of a run of equal ids owns that id's row, the others exit at once, so the
// launch needs no count of distinct ids (no device-to-host read of a data-dependent size).
// dW[id, :] (+)= sum over the run in ascending token position, fp32.
template <typename T>
__global__ void embedding_bwd_kernel(const T* __restrict__ dy, const long* __restrict__ sorted_ids,
                                     const long* __restrict__ sorted_tok, long n, float* __restrict__ dW, int D,
                                     int accumulate) {
  const long b = blockIdx.x;
  const long id = sorted_ids[b];
  if (b > 0 && sorted_ids[b - 1] == id) return;
  long e = b + 1;
  while (e < n && sorted_ids[e] == id) ++e;
  float* out = dW + id * D;
  for (int c = threadIdx.x; c < D; c += blockDim.x) {
    float acc = 0.0f;
    for (long i = b; i < e; ++i) acc = __fadd_rn(acc, to_f<T>(dy[sorted_tok[i] * D + c]));
    out[c] = accumulate ? __fadd_rn(out[c], acc) : acc;
  }
}
// The same sums, eight columns a thread (16 bytes of bf16), the rows of a run in flight four at a time. D % 8 == 0 and 16-byte
// aligned operands. us, a column a thread and so (bf16, tokens x columns into a table of): 2048 x 256 into 1024 5.5 and 4.0, 8192 x
// 2048 into 8192 45 and 19.5, 8192 x 768 into 128256 24 and 10.3, 16384 x 2048 into 128256 155 and 71.
template <typename T>
__global__ void embedding_bwd8_kernel(const T* __restrict__ dy, const long* __restrict__ sorted_ids, const long* __restrict__ sorted_tok, long n,
                                      float* __restrict__ dW, int D, int accumulate) {
  const long b = blockIdx.x;
  const long id = sorted_ids[b];
  if (b > 0 && sorted_ids[b - 1] == id) return;
  long e = b + 1;
  while (e < n && sorted_ids[e] == id) ++e;
  float* out = dW + id * D;
  for (int c = threadIdx.x * 8; c < D; c += blockDim.x * 8) {
    float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (long i = b; i < e; i += 4) {
      Raw8<T> raw[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (i + u < e) raw[u].load(dy + sorted_tok[i + u] * D + c);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (i + u < e) {
          float f[8];
          raw[u].unpack(f);
#pragma unroll
          for (int x = 0; x < 8; ++x) acc[x] = __fadd_rn(acc[x], f[x]);
        }
      }
    }
    if (accumulate) {
      float o[8];
      Vec8<float>::load(out + c, o);
#pragma unroll
      for (int x = 0; x < 8; ++x) acc[x] = __fadd_rn(o[x], acc[x]);
    }
    Vec8<float>::store(out + c, acc);
  }
}

// elementwise helpers ---------------------------------------------------------
template <typename TI, typename TO>
__global__ void cast_kernel(const TI* __restrict__ in, TO* __restrict__ out, long n) {
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = from_f<TO>(to_f<TI>(in[i]));
}
template <typename T>
__global__ void add_kernel(const T* __restrict__ a, const T* __restrict__ b, T* __restrict__ out, long n) {
  const long i = ((long)blockIdx.x * blockDim.x + threadIdx.x) * 8;
  if (i >= n) return;
  float x[8], y[8], o[8];
  Vec8<T>::load(a + i, x);
  Vec8<T>::load(b + i, y);
#pragma unroll
  for (int e = 0; e < 8; ++e) o[e] = __fadd_rn(x[e], y[e]);
  Vec8<T>::store(out + i, o);
}

inline unsigned blocks_for(long n, int per) { return (unsigned)((n + per - 1) / per); }
// whether four elements of any row that start at a multiple of four are one aligned access
inline bool four_aligned(const void* p, long ld, int bf16) { return ld % 4 == 0 && reinterpret_cast<uintptr_t>(p) % (bf16 ? 8 : 16) == 0; }

}  // namespace

#define S(stream) reinterpret_cast<cudaStream_t>(stream)
#define DISPATCH_T(is_bf16, ...)                       \
  if (is_bf16) { using T = __nv_bfloat16; __VA_ARGS__ } \
  else { using T = float; __VA_ARGS__ }

// dtype: 1 = bf16, 0 = fp32 for every activation pointer. All row widths multiples of 8.
extern "C" int otb_rmsnorm_fwd(const void* x, const void* w, void* y, float* rstd, long rows, int D, float inv_d,
                               float eps, int dtype, void* stream) {
  if (D % 8) return -2;
#define RF(KERN) return otb_launch_early(KERN, blocks_for(rows, 8), 256, 0, S(stream), (const T*)x, (const T*)w, (T*)y, rstd, rows, D, inv_d, eps)
#define RFC(MAXC) RF((rmsnorm_fwd_kernel<T, MAXC>))
  if (!rmsnorm_in_registers(rows, D, dtype)) {
    // four groups per turn take more registers, which large tensors need for rows in flight (us, two and four: 64 x 2048 3.3 and 3.2, 4096 x
    // 2048 7.0 and 5.5, 8192 x 2048 9.6 and 9.2, 8192 x 5120 40.2 and 31.4; 16384 x 2048 23.1 and 24.6, 16384 x 1024 8.9 and 9.4)
    if (rows <= 64L * otb_sm_count()) { DISPATCH_T(dtype, RF((rmsnorm_fwd_wide_kernel<T, 4>));) } else { DISPATCH_T(dtype, RF((rmsnorm_fwd_wide_kernel<T, 2>));) }
  } else if (dtype) {
    using T = __nv_bfloat16;
    if (D <= 256) RFC(1); else if (D <= 768) RFC(3); else RFC(16);
  } else {
    using T = float;
    if (D <= 256) RFC(1); else if (D <= 1024) RFC(4); else if (D <= 2048) RFC(8); else RFC(16);
  }
#undef RFC
#undef RF
}
extern "C" int otb_rmsnorm_bwd(const void* dy, const void* x, const void* w, const float* rstd, void* dx,
                               float* dgamma_partial, long rows, int D, float inv_d, int dtype, void* stream) {
  if (D % 8 || D > 256 * 16) return -2;
  int launched = 0;
  const long slabs = (rows + NORM_SLAB - 1) / NORM_SLAB;
#define RB(MAXC)                                                                                                          \
  DISPATCH_T(dtype, {                                                                                                     \
    if (const int rc = otb_allow_smem<rmsnorm_bwd_kernel<T, MAXC>>(NORM_SLAB * 256 * MAXC * 4)) return rc;                   \
    launched = otb_launch_early(rmsnorm_bwd_kernel<T, MAXC>, (unsigned)slabs, NORM_SLAB * 32, dgamma_partial ? NORM_SLAB * 256 * MAXC * 4 : 0, S(stream), (const T*)dy, (const T*)x, (const T*)w, rstd, (T*)dx, \
                                                                                     dgamma_partial, rows, D, inv_d);     \
  })
  if (D <= 256) { RB(1) } else if (D <= 1024) { RB(4) } else if (D <= 2048) { RB(8) } else { RB(16) }
#undef RB
  if (launched || !dgamma_partial) return launched;
  return pair_tree_cols_launch(dgamma_partial, slabs, D, S(stream));
}
// x, y, dy, dx: 16-byte aligned, pitches (in elements) that keep every row so; D <= 128, multiple of 8. rows = tokens * heads.
extern "C" int otb_head_rmsnorm_fwd(const void* x, long ldx, const void* w, void* y, long ldy, float* rstd, long rows, int heads, int D,
                                    float inv_d, float eps, int dtype, void* stream) {
  if (D % 8 || D > 128 || ldx % 8 || ldy % 8) return -2;
  DISPATCH_T(dtype, return otb_launch_early(head_rmsnorm_fwd_kernel<T>, blocks_for(rows, 16), 256, 0, S(stream), (const T*)x, ldx, (const T*)w, (T*)y, ldy, rstd, rows, heads,
                                                                                          D, inv_d, eps);)
}
extern "C" int otb_head_rmsnorm_bwd(const void* dy, long lddy, const void* x, long ldx, const void* w, const float* rstd, void* dx, long lddx,
                                    float* dgamma_partial, long rows, int heads, int D, float inv_d, int dtype, void* stream) {
  if (D % 8 || D > 128 || lddy % 8 || ldx % 8 || lddx % 8) return -2;
  int launched = 0;
  DISPATCH_T(dtype, launched = otb_launch_early(head_rmsnorm_bwd_kernel<T>, blocks_for(rows, 16), 256, 0, S(stream), (const T*)dy, lddy, (const T*)x, ldx, (const T*)w, rstd,
                                                                                          (T*)dx, lddx, dgamma_partial, rows, heads, D, inv_d);)
  if (launched || !dgamma_partial) return launched;
  return pair_tree_cols_launch(dgamma_partial, (rows + NORM_SLAB - 1) / NORM_SLAB, D, S(stream));
}
extern "C" long otb_rmsnorm_slabs(long rows) { return (rows + NORM_SLAB - 1) / NORM_SLAB; }

extern "C" int otb_pair_tree_cols(float* v, long n, int D, void* stream) {
  return pair_tree_cols_launch(v, n, D, S(stream));
}

extern "C" int otb_qknorm_rope_fwd(const void* in, long ld_in, void* out, long ld_out, float* rstd, const float* cosb,
                                   const float* sinb, long rows, int heads, int D, int seq_len, int do_norm,
                                   float inv_d, float eps, int dtype, void* stream) {
  if (D % 4 || D > 128) return -2;
  const bool vec = four_aligned(in, ld_in, dtype) && four_aligned(out, ld_out, dtype);
#define QF(V, NH) DISPATCH_T(dtype, return otb_launch_early(qknorm_rope_fwd_kernel<T, V, NH>, blocks_for(rows * ((heads + NH - 1) / NH), 8), 256, 0, S(stream),  \
                        (const T*)in, ld_in, (T*)out, ld_out, rstd, cosb, sinb, rows, heads, D, seq_len, do_norm, inv_d, eps);)
  if (rope_one_head(rows, heads)) {
    if (vec) { QF(true, 1) } else { QF(false, 1) }
  } else {
    if (vec) { QF(true, ROPE_HEADS) } else { QF(false, ROPE_HEADS) }
  }
#undef QF
}
extern "C" int otb_qknorm_rope_bwd(const void* dout, long ld_dout, const void* in, long ld_in, const float* rstd,
                                   void* din, long ld_din, const float* cosb, const float* sinb, long rows, int heads,
                                   int D, int seq_len, int do_norm, float inv_d, int dtype, void* stream) {
  if (D % 4 || D > 128) return -2;
  const bool vec = four_aligned(dout, ld_dout, dtype) && four_aligned(in, ld_in, dtype) && four_aligned(din, ld_din, dtype);
#define QB(V, NH) DISPATCH_T(dtype, return otb_launch_early(qknorm_rope_bwd_kernel<T, V, NH>, blocks_for(rows * ((heads + NH - 1) / NH), 8), 256, 0, S(stream),  \
                        (const T*)dout, ld_dout, (const T*)in, ld_in, rstd, (T*)din, ld_din, cosb, sinb, rows, heads, D, seq_len, do_norm, inv_d);)
  if (rope_one_head(rows, heads)) {
    if (vec) { QB(true, 1) } else { QB(false, 1) }
  } else {
    if (vec) { QB(true, ROPE_HEADS) } else { QB(false, ROPE_HEADS) }
  }
#undef QB
}
extern "C" int otb_swiglu_fwd(const void* gu, void* h, long rows, int F, int dtype, void* stream) {
  if (F % 8) return -2;
  if (swiglu_per_row(rows, F)) {
    DISPATCH_T(dtype, return otb_launch_early(swiglu_fwd_kernel<T>, (unsigned)rows, swiglu_threads(F), 0, S(stream), (const T*)gu, (T*)h, F);)
  } else {
    DISPATCH_T(dtype, return otb_launch_early(swiglu_fwd_flat_kernel<T>, blocks_for(rows * F / 8, 256), 256, 0, S(stream), (const T*)gu, (T*)h, rows, F);)
  }
}
extern "C" int otb_swiglu_bwd(const void* gu, const void* dh, void* dgu, long rows, int F, int dtype, void* stream) {
  if (F % 8) return -2;
  if (swiglu_per_row(rows, F)) {
    DISPATCH_T(dtype, return otb_launch_early(swiglu_bwd_kernel<T>, (unsigned)rows, swiglu_threads(F), 0, S(stream), (const T*)gu, (const T*)dh, (T*)dgu, F);)
  } else {
    DISPATCH_T(dtype, return otb_launch_early(swiglu_bwd_flat_kernel<T>, blocks_for(rows * F / 8, 256), 256, 0, S(stream), (const T*)gu, (const T*)dh, (T*)dgu, rows, F);)
  }
}
extern "C" int otb_ce_zloss(void* logits, const long* labels, float* ce, float* lse, long rows, int V, float two_z,
                            float scale, int write_grad, int dtype, void* stream) {
  if (V % 8) return -2;
  using bf16 = __nv_bfloat16;
#define CE(T, U, TEST) \
  return otb_launch_early(ce_zloss_kernel<T, U, TEST>, (unsigned)rows, CE_THREADS, 0, S(stream), (T*)logits, labels, ce, lse, rows, V, two_z, scale, write_grad)
#define CE_SHORT(T, GROUPS) \
  return otb_launch_early(ce_zloss_short_kernel<T, GROUPS>, (unsigned)rows, ce_short_threads(V), 0, S(stream), (T*)logits, labels, ce, lse, V, two_z, scale, write_grad)
  if (dtype) {
    if (V <= CE_SWEEP) CE_SHORT(bf16, 1);
    if (V <= 2 * CE_SWEEP) CE_SHORT(bf16, 2);
    if (V <= 4 * CE_SWEEP) CE_SHORT(bf16, 4);
    if (ce_form(rows, V, true) == 1) CE(bf16, 1, true);
    CE(bf16, 4, true);
  }
  if (V <= CE_SWEEP) CE_SHORT(float, 1);
  if (V <= 2 * CE_SWEEP) CE_SHORT(float, 2);
  const int form = ce_form(rows, V, false);
  if (form == 0) CE(float, 1, false);
  if (form == 1) CE(float, 1, true);
  CE(float, 4, true);
#undef CE_SHORT
#undef CE
}
extern "C" int otb_det_sum(const float* x, long n, int mode, float post_scale, float* out, void* stream) {
  return otb_launch_early(det_sum_kernel, 1, 1024, 0, S(stream), x, n, mode, post_scale, out);
}
extern "C" int otb_embedding_fwd(const long* ids, const void* table, void* out, long rows, int D, int dtype,
                                 void* stream) {
  if (D % 8) return -2;
  DISPATCH_T(dtype, return otb_launch(embedding_fwd_kernel<T>, (unsigned)rows, 128, 0, S(stream), ids, (const T*)table, (T*)out, rows,
                                                                                    D);)
}
extern "C" int otb_embedding_bwd(const void* dy, const long* sorted_ids, const long* sorted_tok, long n, float* dW, int D,
                                 int accumulate, int dtype, void* stream) {
  if (n <= 0) return 0;
  const bool wide = D > 0 && D % 8 == 0 && ((reinterpret_cast<uintptr_t>(dy) | reinterpret_cast<uintptr_t>(dW)) & 15) == 0;
  const unsigned threads = wide ? (unsigned)(D < 2048 ? (D / 8 + 31) / 32 * 32 : 256) : 256u;
  DISPATCH_T(dtype, return otb_launch(wide ? embedding_bwd8_kernel<T> : embedding_bwd_kernel<T>, (unsigned)n, threads, 0, S(stream), (const T*)dy,
                                      sorted_ids, sorted_tok, n, dW, D, accumulate);)
}
extern "C" int otb_cast(const void* in, void* out, long n, int in_bf16, int out_bf16, void* stream) {
  const unsigned g = blocks_for(n, 256);
  if (in_bf16 && !out_bf16) cast_kernel<__nv_bfloat16, float><<<g, 256, 0, S(stream)>>>((const __nv_bfloat16*)in, (float*)out, n);
  else if (!in_bf16 && out_bf16) cast_kernel<float, __nv_bfloat16><<<g, 256, 0, S(stream)>>>((const float*)in, (__nv_bfloat16*)out, n);
  else return -2;
  return (int)cudaGetLastError();
}
extern "C" int otb_add(const void* a, const void* b, void* out, long n, int dtype, void* stream) {
  if (n % 8) return -2;
  DISPATCH_T(dtype, add_kernel<T><<<blocks_for(n / 8, 256), 256, 0, S(stream)>>>((const T*)a, (const T*)b, (T*)out, n);)
  return (int)cudaGetLastError();
}

OTB_PACKED(otb_rmsnorm_fwd)
OTB_PACKED(otb_rmsnorm_bwd)
OTB_PACKED(otb_head_rmsnorm_fwd)
OTB_PACKED(otb_head_rmsnorm_bwd)
OTB_PACKED(otb_qknorm_rope_fwd)
OTB_PACKED(otb_qknorm_rope_bwd)
OTB_PACKED(otb_swiglu_fwd)
OTB_PACKED(otb_swiglu_bwd)
OTB_PACKED(otb_ce_zloss)
OTB_PACKED(otb_det_sum)
OTB_PACKED(otb_embedding_fwd)
OTB_PACKED(otb_embedding_bwd)
