// Exact fp32 family on CUDA cores: GEMM and attention whose every dot product is the single chain
//   acc = fma(a_k, b_k, acc), k ascending, acc starting at +0
// i.e. bit-identical to csrc/cpu/ref_gemm_attn.cpp. Used when activations are fp32
// (run.mixed_precision = false: the tiny reproducibility configs, the fp32 audit replay); the
// throughput path is the tcgen05 family.
#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"
#include "det_math.h"
#include "entries.cuh"

namespace {

inline bool aligned16(const void* p, long ld) { return ((reinterpret_cast<uintptr_t>(p) | (uintptr_t)(ld * 4)) & 15) == 0; }

// ------------------------------------------------------------------------------ GEMM
// TM x TN tile of C per CTA, RM x RN chains per thread, k-slabs double-buffered in shared memory as [k][row] (the next
// slabs travel through registers while this one is multiplied). The chains are independent, so the tile shape only
// decides how many CTAs there are and how many shared-memory words a multiply-add costs:
//   128 x 128 (8 x 8 per thread: 4 float4 per 64 multiply-adds), 64 x 64 and 32 x 32 (4 x 4: 2 per 16).
// The rule takes the largest tile that still gives every SM a CTA (two for the 128-wide one, whose last wave costs most).
// Bound by the serial chains of the few tiles a small product has, then by shared-memory words per multiply-add. A 2-layer,
// 256-wide micro-batch of 4 x 512 tokens spent 5.1 ms in these products with one 64 x 64 tile shape, scalar shared-memory
// reads and no overlap of load and multiply, 6.8 ms in attention; the whole pass went from 11.47 to 2.69 ms, and with the deeper fetch of the small tiles (and
// cheaper launches) to 2.31.
template <int TM, int TN, int RM, int RN>
struct F32Tile {
  static constexpr int NT = (TM / RM) * (TN / RN);
  // The small tiles have too few multiply-adds per slab to cover a load from L2 or DRAM (a 2048 x 256 x 768 product took 58 us
  // with slabs of 16 fetched one ahead): they take slabs of 32 and fetch two ahead.
  static constexpr int GK = TM >= 128 ? 16 : 32;
  static constexpr int AHEAD = TM >= 128 ? 1 : 2;
};

// v = *p where `in`, else v stays: a predicated load. A branch around it would make the loaded value meet the zeros of the
// other side in a move, which waits for the load there and then instead of two slabs later.
__device__ __forceinline__ void load_if(float4& v, const float* p, bool in) {
  asm("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %5, 0;\n\t@q ld.global.v4.f32 {%0, %1, %2, %3}, [%4];\n\t}\n"
      : "+f"(v.x), "+f"(v.y), "+f"(v.z), "+f"(v.w)
      : "l"(p), "r"((int)in));
}
// One operand's share of a k-slab, held in registers between the global load and the shared-memory store. WHOLE: every float4
// is aligned and lies inside the operand or outside it as a whole.
template <int TR, int NT, bool MN, int GK, bool WHOLE>
struct Slab {
  static constexpr int PER = TR * GK / 4 / NT;  // float4 per thread
  static_assert(TR * GK / 4 % NT == 0, "the slab splits evenly over the CTA");
  float4 v[PER];
  __device__ __forceinline__ void load(const float* __restrict__ X, long ld, int r0, int R, int k0, int K, bool vec) {
#pragma unroll
    for (int p = 0; p < PER; ++p) {
      const int i = threadIdx.x + p * NT;
      // MN-major: four rows of one k; K-major: four k of one row (lanes along the rows: conflict-free stores)
      const int r = r0 + (MN ? (i % (TR / 4)) * 4 : i % TR), k = k0 + (MN ? i / (TR / 4) : (i / TR) * 4);
      const bool in = r < R && k < K;
      if constexpr (WHOLE) {
        v[p] = make_float4(0.f, 0.f, 0.f, 0.f);
        load_if(v[p], X + (MN ? (long)k * ld + r : (long)r * ld + k), in);
        continue;
      }
      float f[4] = {0.f, 0.f, 0.f, 0.f};
      if (in) {
        const float* q = X + (MN ? (long)k * ld + r : (long)r * ld + k);
        if (vec && (MN ? r + 4 <= R : k + 4 <= K)) {
          const float4 w = *reinterpret_cast<const float4*>(q);
          f[0] = w.x; f[1] = w.y; f[2] = w.z; f[3] = w.w;
        } else {
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (MN ? r + e < R : k + e < K) f[e] = q[e];
        }
      }
      v[p] = make_float4(f[0], f[1], f[2], f[3]);
    }
  }
  __device__ __forceinline__ void store(float (&s)[GK][TR + 4]) const {
#pragma unroll
    for (int p = 0; p < PER; ++p) {
      const int i = threadIdx.x + p * NT;
      if (MN) {
        *reinterpret_cast<float4*>(&s[i / (TR / 4)][(i % (TR / 4)) * 4]) = v[p];
      } else {
        const int r = i % TR, k = (i / TR) * 4;
        s[k][r] = v[p].x; s[k + 1][r] = v[p].y; s[k + 2][r] = v[p].z; s[k + 3][r] = v[p].w;
      }
    }
  }
};

// RES: CTAs that an SM holds at least, at the cost of spilled registers (0: as the compiler likes).
template <int TM, int TN, int RM, int RN, int RES, bool A_MN, bool B_MN, int EPI, bool WHOLE>
__global__ void __launch_bounds__(F32Tile<TM, TN, RM, RN>::NT, RES)
gemm_f32_kernel(const float* __restrict__ A, const float* __restrict__ B, float* __restrict__ C,
                const float* __restrict__ R, int M, int N, int K, long lda, long ldb, long ldc, long ldr, int vec) {
  using Tile = F32Tile<TM, TN, RM, RN>;
  constexpr int NT = Tile::NT, GX = TN / RN, GK = Tile::GK, AHEAD = Tile::AHEAD;
  __shared__ __align__(16) float sa[2][GK][TM + 4], sb[2][GK][TN + 4];
  const int tx = threadIdx.x % GX, ty = threadIdx.x / GX;
  const int m0 = blockIdx.y * TM, n0 = blockIdx.x * TN;
  // a thread's rows / columns come in groups of four, half a tile apart when there are two groups
  auto mrow = [&](int i) { return m0 + (i >> 2) * (TM / 2) + ty * 4 + (i & 3); };
  auto ncol = [&](int j) { return n0 + (j >> 2) * (TN / 2) + tx * 4 + (j & 3); };
  float acc[RM][RN];
#pragma unroll
  for (int i = 0; i < RM; ++i)
#pragma unroll
    for (int j = 0; j < RN; ++j)
      // the accumulating epilogue continues the chain from the value already in C
      acc[i][j] = (EPI == 2 && mrow(i) < M && ncol(j) < N) ? C[(long)mrow(i) * ldc + ncol(j)] : 0.0f;
  Slab<TM, NT, A_MN, GK, WHOLE> la[AHEAD];
  Slab<TN, NT, B_MN, GK, WHOLE> lb[AHEAD];
  const bool va = vec & 1, vb = vec & 2, vc = vec & 4;
  la[0].load(A, lda, m0, M, 0, K, va);
  lb[0].load(B, ldb, n0, N, 0, K, vb);
  la[0].store(sa[0]);
  lb[0].store(sb[0]);
  if (AHEAD == 2) {
    la[AHEAD - 1].load(A, lda, m0, M, GK, K, va);
    lb[AHEAD - 1].load(B, ldb, n0, N, GK, K, vb);
  }
  __syncthreads();
  auto step = [&](int buf, int k) {
    float a[RM], b[RN];
#pragma unroll
    for (int i = 0; i < RM; i += 4) {
      const float4 f = *reinterpret_cast<const float4*>(&sa[buf][k][(i >> 2) * (TM / 2) + ty * 4]);
      a[i] = f.x; a[i + 1] = f.y; a[i + 2] = f.z; a[i + 3] = f.w;
    }
#pragma unroll
    for (int j = 0; j < RN; j += 4) {
      const float4 f = *reinterpret_cast<const float4*>(&sb[buf][k][(j >> 2) * (TN / 2) + tx * 4]);
      b[j] = f.x; b[j + 1] = f.y; b[j + 2] = f.z; b[j + 3] = f.w;
    }
#pragma unroll
    for (int i = 0; i < RM; ++i)
#pragma unroll
      for (int j = 0; j < RN; ++j) acc[i][j] = __fmaf_rn(a[i], b[j], acc[i][j]);
  };
  for (int k00 = 0; k00 < K; k00 += 2 * GK) {
#pragma unroll
    for (int u = 0; u < 2; ++u) {  // slab k0 / GK has parity u: so do its buffer and, two ahead, its registers
      const int k0 = k00 + u * GK;
      if (k0 >= K) break;
      if (k0 + AHEAD * GK < K) {
        la[AHEAD == 2 ? u : 0].load(A, lda, m0, M, k0 + AHEAD * GK, K, va);
        lb[AHEAD == 2 ? u : 0].load(B, ldb, n0, N, k0 + AHEAD * GK, K, vb);
      }
      if (k0 + GK <= K) {
#pragma unroll
        for (int k = 0; k < GK; ++k) step(u, k);
      } else {  // the chain ends at K: no links of padding
        for (int k = 0; k < K - k0; ++k) step(u, k);
      }
      if (k0 + GK < K) {
        la[AHEAD == 2 ? u ^ 1 : 0].store(sa[u ^ 1]);  // that buffer was last read before the barrier that ended the previous slab
        lb[AHEAD == 2 ? u ^ 1 : 0].store(sb[u ^ 1]);
      }
      __syncthreads();
    }
  }
#pragma unroll
  for (int i = 0; i < RM; ++i) {
    const int m = mrow(i);
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < RN; j += 4) {
      const int n = ncol(j);
      float v[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        v[e] = acc[i][j + e];
        if (EPI == 3 && n + e < N) v[e] = __fadd_rn(v[e], R[(long)m * ldr + n + e]);
      }
      if (vc && n + 4 <= N) {
        *reinterpret_cast<float4*>(C + (long)m * ldc + n) = make_float4(v[0], v[1], v[2], v[3]);
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (n + e < N) C[(long)m * ldc + n + e] = v[e];
      }
    }
  }
}

template <int TM, int TN, int RM, int RN, int RES = 0>
int launch_gemm_f32(const float* A, const float* B, float* C, const float* R, int M, int N, int K, long lda, long ldb, long ldc, long ldr,
                    int a_mn, int b_mn, int epi, int vec, cudaStream_t s, bool predicate = true) {
  const dim3 grid((N + TN - 1) / TN, (M + TM - 1) / TM);
  // Predicated loads, us, branches and predicated. They pay with two MN-major operands, the weight gradients, in 32-wide tiles (704 x 256 x
  // 2048 72.1 and 46.6, accumulating 70.3 and 57.3; 128 x 128 x 64 4.4 and 3.3), in 64-wide ones (but see the caller), and in 128-wide
  // ones that store (4096 x 4096 x 512 411 and 376, 8192 x 4096 x 256 411 and 375), not in those that accumulate (450 and 472, 477 and
  // 514); and with two K-major ones that store from 64-wide tiles (2048 x 1408 x 256 66.1 and 61.2, 768 x 2048 x 1000 129.9 and
  // 125.0), not accumulating (38.7 and 39.9, 125.5 and 128.5) nor in 128-wide ones (464 and 480). Elsewhere they differ in both directions.
  const bool whole = predicate && (vec & 3) == 3 && (a_mn ? M : K) % 4 == 0 && (b_mn ? N : K) % 4 == 0;
#define GF(AM, BM, E)                                                                                    \
  do {                                                                                                   \
    constexpr bool PAYS = E == 2 ? AM && BM && TM < 128 : AM == BM && (AM || TM == 64);                  \
    auto kern = whole && PAYS ? gemm_f32_kernel<TM, TN, RM, RN, RES, AM, BM, E, PAYS>                    \
                              : gemm_f32_kernel<TM, TN, RM, RN, RES, AM, BM, E, false>;                  \
    kern<<<grid, F32Tile<TM, TN, RM, RN>::NT, 0, s>>>(A, B, C, R, M, N, K, lda, ldb, ldc, ldr, vec);     \
  } while (0)
#define GE(AM, BM)                                      \
  switch (epi) {                                         \
    case 0: case 1: GF(AM, BM, 0); break;                \
    case 2: GF(AM, BM, 2); break;                        \
    case 3: GF(AM, BM, 3); break;                        \
    default: return -3;                                  \
  }
  if (!a_mn && !b_mn) { GE(false, false) } else if (!a_mn && b_mn) { GE(false, true) }
  else if (a_mn && b_mn) { GE(true, true) } else { GE(true, false) }
#undef GE
#undef GF
  return (int)cudaGetLastError();
}

// ------------------------------------------------------------------------- attention
// The three main kernels work on 64-row tiles whose operands sit TRANSPOSED in shared memory ([d][64 + 4]): a product over d
// reads one float4 of rows and one of columns per step for 4 x 4 (or 4 x 8) chains, and the accumulations over queries /
// keys read the same arrays as float4 along the row index, four links of each chain at a time. Before (one warp per row,
// every operand straight from global memory, one key per lane) each multiply-add cost a strided load:
// 0.71 ms forward and 2.68 ms backward per layer at 4 x 512 tokens, 4 heads x 64, causal.
__device__ __forceinline__ bool masked(int qi, int kj, int window) { return kj > qi || (window > 0 && kj <= qi - window); }

constexpr int AT = 64;         // rows of a tile
constexpr int ALD = AT + 4;    // pitch of a transposed 64-row tile (multiple of 4: float4 rows)
constexpr int FKB = 128;       // keys per softmax block of the forward (the block the running maximum moves by)
constexpr int FLD = FKB + 4;

// dst[d][r] = src[(row0 + r) * ld + d] for r < rows, d < D; rows at or past `limit` read as zero. Lanes run along r, so the
// stores are conflict-free; a lane takes four d at a time (one 16-byte load when the operand allows it).
__device__ __forceinline__ void load_t(float* __restrict__ dst, int pitch, int rows, const float* __restrict__ src, long ld, long row0,
                                       int have, int D, bool vec) {
  for (int i = threadIdx.x; i < rows * ((D + 3) / 4); i += 256) {
    const int r = i % rows, d = (i / rows) * 4;
    float v[4] = {0.f, 0.f, 0.f, 0.f};
    if (r < have) {
      const float* p = src + (row0 + r) * ld + d;
      if (vec) {
        const float4 f = *reinterpret_cast<const float4*>(p);
        v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (d + e < D) v[e] = p[e];
      }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (d + e < D) dst[(d + e) * pitch + r] = v[e];
  }
}
// CTA -> (64-row tile, head, sequence); tiles vary slowest, so that the longest ones of every head start first
__device__ __forceinline__ void tile_of(int T, int heads, int& tile, int& head, int& b) {
  const long per = gridDim.x / ((T + AT - 1) / AT);  // heads x sequences
  const long w = blockIdx.x % per;
  tile = (int)(blockIdx.x / per);
  head = (int)(w % heads);
  b = (int)(w / heads);
}
__device__ __forceinline__ void ld4(const float* p, float (&v)[4]) {
  const float4 f = *reinterpret_cast<const float4*>(p);
  v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
}

// One CTA per (64 queries, head, sequence). A key block is 128 wide: scores by all threads (4 queries x 8 keys each) into
// sS[key][query]; softmax with thread = (query, 32-key quarter); P V with thread = (4 queries, D / 16 columns).
template <int DM>
__global__ void __launch_bounds__(256)
attn_f32_fwd_kernel(const float* __restrict__ qk, long ldqk, const float* __restrict__ qkv, long ldqkv,
                    float* __restrict__ O, long ldo, float* __restrict__ lse, int B, int T, int H, int Hkv, int D,
                    int window, float c_log2, int vec) {
  extern __shared__ float4 smem4[];
  float* sQ = reinterpret_cast<float*>(smem4);   // [DM][ALD]
  float* sKV = sQ + DM * ALD;                    // K: [DM][FLD], then V: [FKB][DM + 4]
  float* sS = sKV + (DM * FLD > FKB * (DM + 4) ? DM * FLD : FKB * (DM + 4));  // [FKB][ALD]
  float* sX = sS + FKB * ALD;                    // [4][64] quarter maxima, later quarter sums
  float* sA = sX + 4 * AT;                       // [64] alpha
  constexpr int VLD = DM + 4, U = DM / 16;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int row = threadIdx.x & 63, quarter = threadIdx.x >> 6;
  int qt, h, b;
  tile_of(T, H, qt, h, b);
  const int q0 = ((T + AT - 1) / AT - 1 - qt) * AT;  // long rows first
  const int g = h / (H / Hkv);
  const int qhave = min(AT, T - q0);
  load_t(sQ, ALD, AT, qk + (long)h * D, ldqk, (long)b * T + q0, qhave, D, vec);
  const int qb0 = (q0 / 128) * 128, jmax = q0 / 128;
  const int jmin = (window > 0 && qb0 - window + 1 > 0) ? (qb0 - window + 1) / 128 : 0;
  const int qi = q0 + row;
  float o[4][U];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int u = 0; u < U; ++u) o[i][u] = 0.0f;
  float m_run = -INFINITY, l_part = 0.0f;
  for (int j = jmin; j <= jmax; ++j) {
    const int k0 = j * FKB, khave = min(FKB, T - k0);
    __syncthreads();
    load_t(sKV, FLD, FKB, qk + (long)(H + g) * D, ldqk, (long)b * T + k0, khave, D, vec);
    __syncthreads();
    float s[4][8];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int e = 0; e < 8; ++e) s[i][e] = 0.0f;
#pragma unroll 4
    for (int d = 0; d < D; ++d) {
      float a[4], k1[4], k2[4];
      ld4(sQ + d * ALD + ty * 4, a);
      ld4(sKV + d * FLD + tx * 4, k1);
      ld4(sKV + d * FLD + 64 + tx * 4, k2);
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          s[i][e] = __fmaf_rn(a[i], k1[e], s[i][e]);
          s[i][4 + e] = __fmaf_rn(a[i], k2[e], s[i][4 + e]);
        }
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int kk = (e >> 2) * 64 + tx * 4 + (e & 3);
      *reinterpret_cast<float4*>(sS + kk * ALD + ty * 4) = make_float4(s[0][e], s[1][e], s[2][e], s[3][e]);
    }
    __syncthreads();
    // V replaces K while the softmax runs on sS
    for (int i = threadIdx.x; i < FKB * ((D + 3) / 4); i += 256) {
      const int nv = (D + 3) / 4, r = i / nv, d = (i % nv) * 4;
      float v[4] = {0.f, 0.f, 0.f, 0.f};
      if (r < khave) {
        const float* p = qkv + ((long)b * T + k0 + r) * ldqkv + (long)(H + Hkv + g) * D + d;
        if (vec) ld4(p, v);
        else {
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (d + e < D) v[e] = p[e];
        }
      }
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (d + e < D) sKV[r * VLD + d + e] = v[e];
    }
    float mx = -INFINITY;
#pragma unroll 8
    for (int e = 0; e < 32; ++e) {
      const int kj = k0 + quarter * 32 + e;
      const float v = sS[(quarter * 32 + e) * ALD + row];
      if (!masked(qi, kj, window) && kj < T) mx = fmaxf(mx, v);
    }
    sX[quarter * AT + row] = mx;
    __syncthreads();
    mx = fmaxf(fmaxf(sX[row], sX[AT + row]), fmaxf(sX[2 * AT + row], sX[3 * AT + row]));
    const float m_new = fmaxf(m_run, __fmul_rn(mx, c_log2));
    const float m_safe = (m_new == -INFINITY) ? 0.0f : m_new;
    const float alpha = det_exp2_attn(__fadd_rn(m_run, -m_safe));
    float le = 0.0f, lo = 0.0f;  // the quarter's row sum: even and odd keys are ascending chains, then added
#pragma unroll 4
    for (int e = 0; e < 32; ++e) {
      const int kj = k0 + quarter * 32 + e;
      const float v = sS[(quarter * 32 + e) * ALD + row];
      const bool dead = masked(qi, kj, window) || kj >= T || v == -INFINITY;
      const float p = dead ? 0.0f : det_exp2_attn(__fmaf_rn(v, c_log2, -m_safe));
      sS[(quarter * 32 + e) * ALD + row] = p;
      if (e & 1) lo = __fadd_rn(lo, p);
      else le = __fadd_rn(le, p);
    }
    l_part = __fmaf_rn(l_part, alpha, __fadd_rn(le, lo));
    if (quarter == 0) sA[row] = alpha;
    m_run = m_new;
    __syncthreads();
    float pv[4][U];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int u = 0; u < U; ++u) pv[i][u] = 0.0f;
#pragma unroll 4
    for (int e = 0; e < FKB; ++e) {
      float p[4];
      ld4(sS + e * ALD + ty * 4, p);
#pragma unroll
      for (int w = 0; w < U / 4; ++w) {
        float v[4];
        ld4(sKV + e * VLD + w * 64 + tx * 4, v);
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (p[i] != 0.0f) {  // hidden keys take no part in the chain
#pragma unroll
            for (int x = 0; x < 4; ++x) pv[i][w * 4 + x] = __fmaf_rn(p[i], v[x], pv[i][w * 4 + x]);
          }
      }
    }
    float al[4];
    ld4(sA + ty * 4, al);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int u = 0; u < U; ++u) o[i][u] = __fmaf_rn(o[i][u], al[i], pv[i][u]);
  }
  __syncthreads();
  sX[quarter * AT + row] = l_part;
  __syncthreads();
  if (quarter == 0) {
    const float l_tot = __fadd_rn(__fadd_rn(__fadd_rn(sX[row], sX[AT + row]), sX[2 * AT + row]), sX[3 * AT + row]);
    sA[row] = l_tot;
    if (qi < T) lse[((long)b * H + h) * T + qi] = __fmaf_rn(det_logf(l_tot), 1.44269504088896341f, m_run);
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = ty * 4 + i;
    if (r >= qhave) continue;
    const float l_tot = sA[r];
    float* orow = O + ((long)b * T + q0 + r) * ldo + (long)h * D;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int d = (u >> 2) * 64 + tx * 4 + (u & 3);
      if (d < D) orow[d] = __fdiv_rn(o[i][u], l_tot);
    }
  }
}

__global__ void attn_f32_delta_kernel(const float* __restrict__ dO, long lddo, const float* __restrict__ O, long ldo,
                                      float* __restrict__ delta, int B, int T, int H, int D) {
  const long wid = (long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (wid >= (long)B * T * H) return;
  const long row = wid / H;
  const int h = (int)(wid - row * H);
  float acc = 0.0f;
  for (int e = 0; e < 4; ++e) {
    const int d = lane * 4 + e;
    if (d < D) acc = __fmaf_rn(dO[row * lddo + (long)h * D + d], O[row * ldo + (long)h * D + d], acc);
  }
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) acc = __fadd_rn(acc, __shfl_xor_sync(0xffffffffu, acc, off));
  if (lane == 0) {
    const long bb = row / T, t = row - bb * T;
    delta[(bb * H + h) * T + t] = acc;
  }
}

// ---- sequences far shorter than a tile: one warp per query, or per key in dK / dV, and one pair per lane; no block of keys
// ever moves the running maximum (T <= FKB). Same chains, same bits. The tiles above spend as long on one query as on 64 (4
// heads, us, this form and tiles: forward 1 token x 64 5.5 and 15.8, 16 tokens 9.7 and 17.4, 33 tokens 15.8 and 18.5, x 128 19.9
// and 28.7; 48 tokens 27.6 and 18.5; backward 1 token x 64 13.7 and 27.2, 16 tokens 20.2 and 29.2, 32 tokens 31.2 and 30.1).
__device__ __forceinline__ float chain(const float* __restrict__ a, const float* __restrict__ b, int D) {
  float s = 0.0f;
  for (int d = 0; d < D; ++d) s = __fmaf_rn(a[d], b[d], s);
  return s;
}
__global__ void __launch_bounds__(128)
attn_f32_fwd_short_kernel(const float* __restrict__ qk, long ldqk, const float* __restrict__ qkv, long ldqkv, float* __restrict__ O, long ldo,
                          float* __restrict__ lse, int B, int T, int H, int Hkv, int D, int window, float c_log2) {
  __shared__ float sp[4][FKB];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long wid = (long)blockIdx.x * 4 + w;
  if (wid >= (long)B * H * T) return;
  const int qi = (int)(wid % T), h = (int)((wid / T) % H), g = h / (H / Hkv);
  const long row0 = wid / ((long)T * H) * T, qrow = row0 + qi;  // first row of the sequence; this query's
  float s[4], mx = -INFINITY;
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int kj = lane + 32 * u;
    s[u] = kj < T && !masked(qi, kj, window) ? chain(qk + qrow * ldqk + (long)h * D, qk + (row0 + kj) * ldqk + (long)(H + g) * D, D) : -INFINITY;
    mx = fmaxf(mx, s[u]);
  }
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
  const float m_run = __fmul_rn(mx, c_log2);
  const float m_safe = (m_run == -INFINITY) ? 0.0f : m_run;
#pragma unroll
  for (int u = 0; u < 4; ++u) sp[w][lane + 32 * u] = (s[u] == -INFINITY) ? 0.0f : det_exp2_attn(__fmaf_rn(s[u], c_log2, -m_safe));
  __syncwarp();
  float l_part = 0.0f;
  if (lane < 4) {  // the four quarter-row sums: even and odd keys are ascending chains, then added
    float le = 0.0f, lo = 0.0f;
    for (int e = lane * 32; e < lane * 32 + 32; e += 2) { le = __fadd_rn(le, sp[w][e]); lo = __fadd_rn(lo, sp[w][e + 1]); }
    l_part = __fadd_rn(le, lo);
  }
  float pv[4] = {0.f, 0.f, 0.f, 0.f};
  for (int e = 0; e < T; ++e) {
    const float p = sp[w][e];
    if (p == 0.0f) continue;
    const float* vr = qkv + (row0 + e) * ldqkv + (long)(H + Hkv + g) * D;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int d = lane + 32 * u;
      if (d < D) pv[u] = __fmaf_rn(p, vr[d], pv[u]);
    }
  }
  const float l0 = __shfl_sync(0xffffffffu, l_part, 0), l1 = __shfl_sync(0xffffffffu, l_part, 1);
  const float l2 = __shfl_sync(0xffffffffu, l_part, 2), l3 = __shfl_sync(0xffffffffu, l_part, 3);
  const float l_tot = __fadd_rn(__fadd_rn(__fadd_rn(l0, l1), l2), l3);
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int d = lane + 32 * u;
    if (d < D) O[qrow * ldo + (long)h * D + d] = __fdiv_rn(__fadd_rn(0.0f, pv[u]), l_tot);  // (0: the output before this block)
  }
  if (lane == 0) lse[(wid / T) * T + qi] = __fmaf_rn(det_logf(l_tot), 1.44269504088896341f, m_run);
}
// p and ds of one (query, key) pair
__device__ __forceinline__ void pair_p_ds(const float* __restrict__ q, const float* __restrict__ k, const float* __restrict__ dor,
                                          const float* __restrict__ v, float l2, float dl, int D, float c_log2, float scale, float& p, float& ds) {
  p = det_exp2_attn(__fmaf_rn(chain(q, k, D), c_log2, -l2));
  ds = __fmul_rn(__fmul_rn(p, __fadd_rn(chain(dor, v, D), -dl)), scale);
}
__global__ void __launch_bounds__(128)
attn_f32_bwd_kv_short_kernel(const float* __restrict__ qk, long ldqk, const float* __restrict__ qkv, long ldqkv, const float* __restrict__ dO, long lddo,
                             const float* __restrict__ lse, const float* __restrict__ delta, float* __restrict__ dqk, long lddqk,
                             float* __restrict__ dqkv, long lddqkv, int B, int T, int H, int Hkv, int D, int window, float c_log2, float scale) {
  __shared__ float sp[4][32], sds[4][32];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long wid = (long)blockIdx.x * 4 + w;
  if (wid >= (long)B * Hkv * T) return;
  const int kj = (int)(wid % T), g = (int)((wid / T) % Hkv), G = H / Hkv;
  const long b = wid / ((long)T * Hkv), krow = b * T + kj;
  const float* k = qk + krow * ldqk + (long)(H + g) * D;
  const float* v = qkv + krow * ldqkv + (long)(H + Hkv + g) * D;
  float dk[4] = {0.f, 0.f, 0.f, 0.f}, dv[4] = {0.f, 0.f, 0.f, 0.f};
  for (int h = g * G; h < (g + 1) * G; ++h) {
    for (int qb = kj / 32 * 32; qb < T; qb += 32) {
      const int qi = qb + lane;
      const long qrow = b * T + qi, st = (b * H + h) * T + qi;
      float p = 0.0f, ds = 0.0f;
      if (qi < T && !masked(qi, kj, window))
        pair_p_ds(qk + qrow * ldqk + (long)h * D, k, dO + qrow * lddo + (long)h * D, v, lse[st], delta[st], D, c_log2, scale, p, ds);
      sp[w][lane] = p;
      sds[w][lane] = ds;
      __syncwarp();
      for (int e = 0; e < 32 && qb + e < T; ++e) {
        if (masked(qb + e, kj, window)) continue;
        const long row = b * T + qb + e;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int d = lane + 32 * u;
          if (d < D) {
            dv[u] = __fmaf_rn(sp[w][e], dO[row * lddo + (long)h * D + d], dv[u]);
            dk[u] = __fmaf_rn(sds[w][e], qk[row * ldqk + (long)h * D + d], dk[u]);
          }
        }
      }
      __syncwarp();
    }
  }
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int d = lane + 32 * u;
    if (d < D) {
      dqk[krow * lddqk + (long)(H + g) * D + d] = dk[u];
      dqkv[krow * lddqkv + (long)(H + Hkv + g) * D + d] = dv[u];
    }
  }
}
__global__ void __launch_bounds__(128)
attn_f32_bwd_q_short_kernel(const float* __restrict__ qk, long ldqk, const float* __restrict__ qkv, long ldqkv, const float* __restrict__ dO, long lddo,
                            const float* __restrict__ lse, const float* __restrict__ delta, float* __restrict__ dqk, long lddqk, int B, int T, int H,
                            int Hkv, int D, int window, float c_log2, float scale) {
  __shared__ float sds[4][32];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long wid = (long)blockIdx.x * 4 + w;
  if (wid >= (long)B * H * T) return;
  const int qi = (int)(wid % T), h = (int)((wid / T) % H), g = h / (H / Hkv);
  const long row0 = wid / ((long)T * H) * T, qrow = row0 + qi;
  float dq[4] = {0.f, 0.f, 0.f, 0.f};
  for (int kb = 0; kb <= qi; kb += 32) {
    const int kj = kb + lane;
    float p = 0.0f, ds = 0.0f;
    if (kj < T && !masked(qi, kj, window))
      pair_p_ds(qk + qrow * ldqk + (long)h * D, qk + (row0 + kj) * ldqk + (long)(H + g) * D, dO + qrow * lddo + (long)h * D,
                qkv + (row0 + kj) * ldqkv + (long)(H + Hkv + g) * D, lse[(wid / T) * T + qi], delta[(wid / T) * T + qi], D, c_log2, scale, p, ds);
    sds[w][lane] = ds;
    __syncwarp();
    for (int e = 0; e < 32 && kb + e <= qi; ++e) {
      if (masked(qi, kb + e, window)) continue;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int d = lane + 32 * u;
        if (d < D) dq[u] = __fmaf_rn(sds[w][e], qk[(row0 + kb + e) * ldqk + (long)(H + g) * D + d], dq[u]);
      }
    }
    __syncwarp();
  }
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int d = lane + 32 * u;
    if (d < D) dqk[qrow * lddqk + (long)h * D + d] = dq[u];
  }
}
// Whether a call takes these: where the tiles leave SMs idle up to 40 tokens (backward 31); with more tiles than SMs, whose rate
// then counts, up to 16 (8): 256 heads of 16 tokens x 64 forward 23.7 and 25.6, of 31 57 and 27; backward 4 tokens 15 and 41, 16
// tokens 72 and 43; 2048 heads of 8 tokens 36 and 155, backward 106 and 251, of 16 331 and 267.
inline bool short_rows(int T, long heads, bool backward) {
  static_assert(FKB >= 40, "one block of keys");
  if (heads <= otb_sm_count()) return T <= (backward ? 31 : 40);
  return T <= (backward ? 8 : 16);
}

// s and dp of a 4 x 4 patch (rows from tiles R1 / R2, columns from C1 / C2), each one chain ascending in d
__device__ __forceinline__ void patch(const float* __restrict__ R1, const float* __restrict__ C1, const float* __restrict__ R2,
                                      const float* __restrict__ C2, int D, int ty, int tx, float (&s)[4][4], float (&dp)[4][4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) { s[i][e] = 0.0f; dp[i][e] = 0.0f; }
#pragma unroll 4
  for (int d = 0; d < D; ++d) {
    float a[4], c[4], a2[4], c2[4];
    ld4(R1 + d * ALD + ty * 4, a);
    ld4(C1 + d * ALD + tx * 4, c);
    ld4(R2 + d * ALD + ty * 4, a2);
    ld4(C2 + d * ALD + tx * 4, c2);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        s[i][e] = __fmaf_rn(a[i], c[e], s[i][e]);
        dp[i][e] = __fmaf_rn(a2[i], c2[e], dp[i][e]);
      }
  }
}

// dV, dK chains of 4 keys x U columns over a tile's queries; TEST: leave out hidden pairs and queries past the sequence
template <bool TEST, int U>
__device__ __forceinline__ void chains_kv(const float* __restrict__ sP, const float* __restrict__ sD, const float* __restrict__ sO,
                                          const float* __restrict__ sQ, int ty, int tx, int qhave, int q0, int k0, int window,
                                          float (&dv)[4][U], float (&dk)[4][U]) {
#pragma unroll 1
  for (int q = 0; q < AT; q += 4) {
    float ov[U][4], qv[U][4];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      ld4(sO + (tx + 16 * u) * ALD + q, ov[u]);
      ld4(sQ + (tx + 16 * u) * ALD + q, qv[u]);
    }
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      float p[4], ds[4];
      ld4(sP + (q + x) * ALD + ty * 4, p);
      ld4(sD + (q + x) * ALD + ty * 4, ds);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (TEST && (q + x >= qhave || masked(q0 + q + x, k0 + ty * 4 + i, window))) continue;
#pragma unroll
        for (int u = 0; u < U; ++u) {
          dv[i][u] = __fmaf_rn(p[i], ov[u][x], dv[i][u]);
          dk[i][u] = __fmaf_rn(ds[i], qv[u][x], dk[i][u]);
        }
      }
    }
  }
}
// dQ chains of 4 queries x U columns over a tile's keys
template <bool TEST, int U>
__device__ __forceinline__ void chains_q(const float* __restrict__ sD, const float* __restrict__ sK, int ty, int tx, int q0, int k0, int window,
                                         float (&dq)[4][U]) {
#pragma unroll 1
  for (int k = 0; k < AT; k += 4) {
    float kv[U][4];
#pragma unroll
    for (int u = 0; u < U; ++u) ld4(sK + (tx + 16 * u) * ALD + k, kv[u]);
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      float ds[4];
      ld4(sD + (k + x) * ALD + ty * 4, ds);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (TEST && masked(q0 + ty * 4 + i, k0 + k + x, window)) continue;
#pragma unroll
        for (int u = 0; u < U; ++u) dq[i][u] = __fmaf_rn(ds[i], kv[u][x], dq[i][u]);
      }
    }
  }
}

// dK, dV of 64 keys of one key/value head: the chain of every element runs over the group's query heads, then ascending
// queries, hidden pairs left out. Thread = (4 keys, D / 16 columns).
template <int DM>
__global__ void __launch_bounds__(256)
attn_f32_bwd_kv_kernel(const float* __restrict__ qk, long ldqk, const float* __restrict__ qkv, long ldqkv,
                       const float* __restrict__ dO, long lddo, const float* __restrict__ lse,
                       const float* __restrict__ delta, float* __restrict__ dqk, long lddqk, float* __restrict__ dqkv,
                       long lddqkv, int B, int T, int H, int Hkv, int D, int window, float c_log2, float scale, int vec) {
  extern __shared__ float4 smem4[];
  float* sK = reinterpret_cast<float*>(smem4);
  float* sV = sK + DM * ALD;
  float* sQ = sV + DM * ALD;
  float* sO = sQ + DM * ALD;
  float* sP = sO + DM * ALD;    // [query][ALD] over keys
  float* sD = sP + AT * ALD;
  constexpr int U = DM / 16;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  int kt, g, b;
  tile_of(T, Hkv, kt, g, b);
  const int k0 = kt * AT, G = H / Hkv;
  const int khave = min(AT, T - k0);
  load_t(sK, ALD, AT, qk + (long)(H + g) * D, ldqk, (long)b * T + k0, khave, D, vec);
  load_t(sV, ALD, AT, qkv + (long)(H + Hkv + g) * D, ldqkv, (long)b * T + k0, khave, D, vec);
  float dk[4][U], dv[4][U];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int u = 0; u < U; ++u) { dk[i][u] = 0.0f; dv[i][u] = 0.0f; }
  const int qend = window > 0 ? min(T, k0 + AT - 1 + window) : T;  // queries that see any of these keys
  for (int hh = 0; hh < G; ++hh) {
    const int h = g * G + hh;
    const float* lrow = lse + ((long)b * H + h) * T;
    const float* drow = delta + ((long)b * H + h) * T;
    for (int q0 = k0; q0 < qend; q0 += AT) {
      const int qhave = min(AT, T - q0);
      __syncthreads();
      load_t(sQ, ALD, AT, qk + (long)h * D, ldqk, (long)b * T + q0, qhave, D, vec);
      load_t(sO, ALD, AT, dO + (long)h * D, lddo, (long)b * T + q0, qhave, D, vec);
      __syncthreads();
      float s[4][4], dp[4][4];
      patch(sQ, sK, sO, sV, D, ty, tx, s, dp);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int qi = q0 + ty * 4 + i;
        const float l2 = qi < T ? lrow[qi] : 0.0f, dl = qi < T ? drow[qi] : 0.0f;
        float p[4], ds[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          p[e] = det_exp2_attn(__fmaf_rn(s[i][e], c_log2, -l2));
          ds[e] = __fmul_rn(__fmul_rn(p[e], __fadd_rn(dp[i][e], -dl)), scale);
        }
        *reinterpret_cast<float4*>(sP + (ty * 4 + i) * ALD + tx * 4) = make_float4(p[0], p[1], p[2], p[3]);
        *reinterpret_cast<float4*>(sD + (ty * 4 + i) * ALD + tx * 4) = make_float4(ds[0], ds[1], ds[2], ds[3]);
      }
      __syncthreads();
      // whether every (query, key) of the tile takes part: no tests inside the chains then
      const bool all = q0 >= k0 + AT - 1 && qhave == AT && (window == 0 || q0 + AT - 1 < k0 + window);
      if (all) chains_kv<false, U>(sP, sD, sO, sQ, ty, tx, qhave, q0, k0, window, dv, dk);
      else chains_kv<true, U>(sP, sD, sO, sQ, ty, tx, qhave, q0, k0, window, dv, dk);
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (ty * 4 + i >= khave) continue;
    const long krow = (long)b * T + k0 + ty * 4 + i;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int d = tx + 16 * u;
      if (d < D) {
        dqk[krow * lddqk + (long)(H + g) * D + d] = dk[i][u];
        dqkv[krow * lddqkv + (long)(H + Hkv + g) * D + d] = dv[i][u];
      }
    }
  }
}

// dQ of 64 queries of one head: chains over ascending keys, hidden pairs left out. Thread = (4 queries, D / 16 columns).
template <int DM>
__global__ void __launch_bounds__(256)
attn_f32_bwd_q_kernel(const float* __restrict__ qk, long ldqk, const float* __restrict__ qkv, long ldqkv,
                      const float* __restrict__ dO, long lddo, const float* __restrict__ lse,
                      const float* __restrict__ delta, float* __restrict__ dqk, long lddqk, int B, int T, int H, int Hkv,
                      int D, int window, float c_log2, float scale, int vec) {
  extern __shared__ float4 smem4[];
  float* sQ = reinterpret_cast<float*>(smem4);
  float* sO = sQ + DM * ALD;
  float* sK = sO + DM * ALD;
  float* sV = sK + DM * ALD;
  float* sD = sV + DM * ALD;    // [key][ALD] over queries
  constexpr int U = DM / 16;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  int qt, h, b;
  tile_of(T, H, qt, h, b);
  const int q0 = ((T + AT - 1) / AT - 1 - qt) * AT, g = h / (H / Hkv);
  const int qhave = min(AT, T - q0);
  load_t(sQ, ALD, AT, qk + (long)h * D, ldqk, (long)b * T + q0, qhave, D, vec);
  load_t(sO, ALD, AT, dO + (long)h * D, lddo, (long)b * T + q0, qhave, D, vec);
  float dq[4][U];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int u = 0; u < U; ++u) dq[i][u] = 0.0f;
  float l2[4], dl[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const int qi = q0 + tx * 4 + e;
    l2[e] = qi < T ? lse[((long)b * H + h) * T + qi] : 0.0f;
    dl[e] = qi < T ? delta[((long)b * H + h) * T + qi] : 0.0f;
  }
  const int kfirst = (window > 0 && q0 - window + 1 > 0) ? (q0 - window + 1) / AT * AT : 0;
  for (int k0 = kfirst; k0 <= q0; k0 += AT) {
    const int khave = min(AT, T - k0);
    __syncthreads();
    load_t(sK, ALD, AT, qk + (long)(H + g) * D, ldqk, (long)b * T + k0, khave, D, vec);
    load_t(sV, ALD, AT, qkv + (long)(H + Hkv + g) * D, ldqkv, (long)b * T + k0, khave, D, vec);
    __syncthreads();
    float s[4][4], dp[4][4];  // rows: keys, columns: queries
    patch(sK, sQ, sV, sO, D, ty, tx, s, dp);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float ds[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float p = det_exp2_attn(__fmaf_rn(s[i][e], c_log2, -l2[e]));
        ds[e] = __fmul_rn(__fmul_rn(p, __fadd_rn(dp[i][e], -dl[e])), scale);
      }
      *reinterpret_cast<float4*>(sD + (ty * 4 + i) * ALD + tx * 4) = make_float4(ds[0], ds[1], ds[2], ds[3]);
    }
    __syncthreads();
    const bool all = k0 + AT - 1 <= q0 && (window == 0 || q0 + AT - 1 < k0 + window);
    if (all) chains_q<false, U>(sD, sK, ty, tx, q0, k0, window, dq);
    else chains_q<true, U>(sD, sK, ty, tx, q0, k0, window, dq);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (ty * 4 + i >= qhave) continue;
    const long qrow = (long)b * T + q0 + ty * 4 + i;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int d = tx + 16 * u;
      if (d < D) dqk[qrow * lddqk + (long)h * D + d] = dq[i][u];
    }
  }
}

}  // namespace

extern "C" int otb_gemm_f32(const float* A, const float* B, float* C, const float* R, int M, int N, int K, long lda,
                            long ldb, long ldc, long ldr, int a_mn, int b_mn, int epi, void* stream) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  // 16-byte accesses where the operand's base and pitch allow them (bit 0: A, 1: B, 2: C)
  const int vec = (aligned16(A, lda) ? 1 : 0) | (aligned16(B, ldb) ? 2 : 0) | (aligned16(C, ldc) ? 4 : 0);
  const long sms = otb_sm_count();
  auto tiles = [&](int t) { return (long)((M + t - 1) / t) * ((N + t - 1) / t); };
  if (tiles(128) >= 2 * sms) return launch_gemm_f32<128, 128, 8, 8>(A, B, C, R, M, N, K, lda, ldb, ldc, ldr, a_mn, b_mn, epi, vec, s);
  if (tiles(64) >= sms) {
    // Two 64-wide tiles are resident on an SM, or three with some registers spilled; r tiles take r times as long as one, so
    // the smaller r x waves wins (K-major, 1429 x 1214 x 2307, 437 tiles: 502 us with two, 365 with three; 1337 x 1734 x 696, 588
    // tiles: 127 and 154). An MN-major B takes fewer registers and fits three as it is, but for the accumulating epilogue.
    auto cost = [&](long r) { return r * ((tiles(64) + r * sms - 1) / (r * sms)); };
    if ((!b_mn || epi == 2) && cost(3) < cost(2)) return launch_gemm_f32<64, 64, 4, 4, 3>(A, B, C, R, M, N, K, lda, ldb, ldc, ldr, a_mn, b_mn, epi, vec, s);
    // With predicated loads a store of two MN-major operands has registers for two tiles per SM only, which pays where that many make
    // clearly fewer turns (branches and three, predicated and two, us: 456 tiles 37.9 and 35.1, 588 114 and 92; but 384 tiles 95 and
    // 128, 704 50.0 and 51.3, 896 60.5 and 62.2, 1152 67.5 and 68.1).
    const bool predicate = !a_mn || !b_mn || epi == 2 || 4 * cost(2) <= 3 * cost(3);
    return launch_gemm_f32<64, 64, 4, 4>(A, B, C, R, M, N, K, lda, ldb, ldc, ldr, a_mn, b_mn, epi, vec, s, predicate);
  }
  return launch_gemm_f32<32, 32, 4, 4>(A, B, C, R, M, N, K, lda, ldb, ldc, ldr, a_mn, b_mn, epi, vec, s);
}

namespace {
template <int DM>
int attn_f32_fwd(const float* qk, long ldqk, const float* qkv, long ldqkv, float* O, long ldo, float* lse, int B, int T, int H, int Hkv, int D,
                 int window, float c_log2, int vec, cudaStream_t s) {
  constexpr int KV = DM * FLD > FKB * (DM + 4) ? DM * FLD : FKB * (DM + 4);
  constexpr int bytes = 4 * (DM * ALD + KV + FKB * ALD + 5 * AT);
  if (const int rc = otb_allow_smem<attn_f32_fwd_kernel<DM>>(bytes)) return rc;
  attn_f32_fwd_kernel<DM><<<(unsigned)((T + AT - 1) / AT * (long)H * B), 256, bytes, s>>>(qk, ldqk, qkv, ldqkv, O, ldo, lse, B, T, H, Hkv, D, window, c_log2, vec);
  return (int)cudaGetLastError();
}
template <int DM>
int attn_f32_bwd(const float* qk, long ldqk, const float* qkv, long ldqkv, const float* dO, long lddo, const float* lse, const float* delta,
                 float* dqk, long lddqk, float* dqkv, long lddqkv, int B, int T, int H, int Hkv, int D, int window, float c_log2, float scale,
                 int vec, cudaStream_t s) {
  constexpr int kv_bytes = 4 * (4 * DM * ALD + 2 * AT * ALD), q_bytes = 4 * (4 * DM * ALD + AT * ALD);
  if (const int rc = otb_allow_smem<attn_f32_bwd_kv_kernel<DM>>(kv_bytes)) return rc;
  if (const int rc = otb_allow_smem<attn_f32_bwd_q_kernel<DM>>(q_bytes)) return rc;
  const long nt = (T + AT - 1) / AT;
  attn_f32_bwd_kv_kernel<DM><<<(unsigned)(nt * Hkv * B), 256, kv_bytes, s>>>(qk, ldqk, qkv, ldqkv, dO, lddo, lse, delta, dqk, lddqk, dqkv, lddqkv, B, T, H,
                                                                     Hkv, D, window, c_log2, scale, vec);
  attn_f32_bwd_q_kernel<DM><<<(unsigned)(nt * H * B), 256, q_bytes, s>>>(qk, ldqk, qkv, ldqkv, dO, lddo, lse, delta, dqk, lddqk, B, T, H, Hkv, D, window,
                                                                 c_log2, scale, vec);
  return (int)cudaGetLastError();
}
}  // namespace

extern "C" int otb_attn_f32_fwd(const float* qk, long ldqk, const float* qkv, long ldqkv, float* O, long ldo, float* lse,
                                int B, int T, int H, int Hkv, int D, int window, float scale, void* stream) {
  if (D > 128 || H % Hkv) return -2;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  const float c_log2 = (float)((double)scale * 1.4426950408889634);
  if (short_rows(T, (long)B * H, false)) {
    attn_f32_fwd_short_kernel<<<(unsigned)(((long)B * H * T + 3) / 4), 128, 0, s>>>(qk, ldqk, qkv, ldqkv, O, ldo, lse, B, T, H, Hkv, D, window, c_log2);
    return (int)cudaGetLastError();
  }
  const int vec = D % 4 == 0 && aligned16(qk, ldqk) && aligned16(qkv, ldqkv);
  if (D <= 64) return attn_f32_fwd<64>(qk, ldqk, qkv, ldqkv, O, ldo, lse, B, T, H, Hkv, D, window, c_log2, vec, s);
  return attn_f32_fwd<128>(qk, ldqk, qkv, ldqkv, O, ldo, lse, B, T, H, Hkv, D, window, c_log2, vec, s);
}
extern "C" int otb_attn_f32_bwd(const float* qk, long ldqk, const float* qkv, long ldqkv, const float* O, long ldo,
                                const float* dO, long lddo, const float* lse, float* delta, float* dqk, long lddqk,
                                float* dqkv, long lddqkv, int B, int T, int H, int Hkv, int D, int window, float scale,
                                void* stream) {
  if (D > 128 || H % Hkv) return -2;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  const float c_log2 = (float)((double)scale * 1.4426950408889634);
  const long w1 = (long)B * T * H;
  attn_f32_delta_kernel<<<(unsigned)((w1 + 7) / 8), 256, 0, s>>>(dO, lddo, O, ldo, delta, B, T, H, D);
  if (short_rows(T, (long)B * H, true)) {
    attn_f32_bwd_kv_short_kernel<<<(unsigned)(((long)B * Hkv * T + 3) / 4), 128, 0, s>>>(qk, ldqk, qkv, ldqkv, dO, lddo, lse, delta, dqk, lddqk, dqkv, lddqkv,
                                                                                        B, T, H, Hkv, D, window, c_log2, scale);
    attn_f32_bwd_q_short_kernel<<<(unsigned)((w1 + 3) / 4), 128, 0, s>>>(qk, ldqk, qkv, ldqkv, dO, lddo, lse, delta, dqk, lddqk, B, T, H, Hkv, D, window,
                                                                        c_log2, scale);
    return (int)cudaGetLastError();
  }
  const int vec = D % 4 == 0 && aligned16(qk, ldqk) && aligned16(qkv, ldqkv) && aligned16(dO, lddo);
  if (D <= 64)
    return attn_f32_bwd<64>(qk, ldqk, qkv, ldqkv, dO, lddo, lse, delta, dqk, lddqk, dqkv, lddqkv, B, T, H, Hkv, D, window, c_log2, scale, vec, s);
  return attn_f32_bwd<128>(qk, ldqk, qkv, ldqkv, dO, lddo, lse, delta, dqk, lddqk, dqkv, lddqkv, B, T, H, Hkv, D, window, c_log2, scale, vec, s);
}

OTB_PACKED(otb_gemm_f32)
OTB_PACKED(otb_attn_f32_fwd)
OTB_PACKED(otb_attn_f32_bwd)
