// Causal / sliding-window flash attention for sm_100a on tcgen05 tensor cores, GQA-native.
//
// Kernels (all: warp 0 = TMA producer, warp 1 = tcgen05.mma issuer, the rest = element warps working straight out of
// tensor memory; a warp may touch TMEM lanes 32*(w%4)..+31 only):
//
//   attn_fwd2     CTA = (batch, query head, TWO 128-row query tiles); one thread per row; S = Q K^T (TMEM) -> online
//                 softmax -> P written back over S as bf16 (the A operand of P V) -> O accumulates in TMEM.
//   attn_bwd_kv3  CTA = (batch, KV head, 128 keys); scores formed transposed (S^T, dP^T: lanes are keys), P^T / dS^T
//                 written back in place, dV += P^T dO and dK += dS^T Q with the A operand in TMEM; 128-query steps over
//                 the heads of the group and the query blocks that see these keys, both ascending; any T.
//   attn_bwd_q2   CTA = (batch, query head, two query tiles); two threads per row; dS written back over S;
//                 dQ += dS K with dS in TMEM; 64-key steps ascending.
//   attn_fwd_i8pv the forward with P V in int8: one tile per CTA, four threads per row, P through shared memory, O in
//                 registers.
//
// No atomics, no split accumulation: every output element has one owner CTA and a fixed
// summation order, so results are identical for any grid, stream or GPU count. The window rule
// is "key in (query - window, query]" (window = 0: full causal). Scores are used in the log2
// domain: y = fma(s, c, -m) with c = scale*log2(e), p = det_exp2_attn(y) (shared with the CPU
// twin), masked scores are -inf. The saved row statistic `lse` is m + log2(l) in that domain.
// Row sums: each 32-key quarter keeps two ascending chains (even / odd keys) that are added per block;
// the four quarter sums are combined ((l0 + l1) + l2) + l3 at the end.
//
// int8-PV variant of the forward: V is quantised beforehand to int8 per (KV head, 128-key block) with one
// fp32 step per block (quant_v_kernel), the probabilities are quantised on the fly to q = rint(127 p), P V runs on
// the int8 tensor cores (tcgen05 kind::i8, exact int32 sums over the 128 keys of a block) and is dequantised in
// fp32: O = O*alpha + float(sum) * (step / 127). Softmax statistics stay fp32 on the unquantised probabilities;
// the backward is the straight-through float shadow (the ordinary backward kernels on the bf16 q, k, v).
// Reference role: int8pv_causal_flash_attention (attention_repop.py:52; docs/MODEL_OP_DTYPE_TRACE.md:80,117-119).
//
// Layouts: q/k come from one [B*T, ld] bf16 buffer (post-RoPE; head h at column h*D, KV head g
// at column (H+g)*D); v comes from the packed qkv buffer; O is [B*T, H*D]; lse and delta are
// [B, H, T] fp32. Reference role: repop causal_flash_attention fwd/bwd
// (src/pretrain/model/modules/attention_repop.py:38-53).
#include "tc05.cuh"
#include "common.cuh"
#include "det_math.h"
#include "entries.cuh"

using namespace tc05;

namespace {

// Launch-order permutation for the race tests: block x works as block (x + g_attn_rotation) mod gridDim.x, and the persistent
// kernels permute the tiles in their list of items the same way. A block owns
// its query tile (or key block) and sums in a fixed order, so any rotation must give the same bytes (0 in production).
__device__ int g_attn_rotation = 0;
// index i of n under the permutation (unsigned: any rotation that the setter takes may be added)
__device__ __forceinline__ int rotated(int i, int n) { return (int)(((unsigned)i + (unsigned)g_attn_rotation) % (unsigned)n); }

constexpr int BQ = 128;   // query rows per tile
constexpr int BKV = 128;  // keys per block
constexpr int NSPLIT = 4;                 // threads per row
constexpr int KPT = 128 / NSPLIT;         // keys per thread and block
constexpr int SOFTMAX_THREADS = 128 * NSPLIT;
constexpr int ATT_THREADS = 64 + SOFTMAX_THREADS;
constexpr int SOFTMAX_WARPS = SOFTMAX_THREADS / 32;

// The four warps that share the rows of a TMEM lane quadrant. (With one barrier for all sixteen warps 4 x 4096 tokens took 784 us, so 768, when
// the kernel still used the divider and spilled; 651 now.)
__device__ __forceinline__ void quadrant_bar(int quad) { asm volatile("bar.sync %0, %1;" ::"r"(quad + 1), "n"(32 * NSPLIT) : "memory"); }

// N (16 or 32) consecutive TMEM columns of this thread's lane
template <int N>
__device__ __forceinline__ void tmem_ld_cols(uint32_t taddr, uint32_t (&v)[N]) {
  if constexpr (N == 32) tmem_ld_32x32b_x32(taddr, v);
  else tmem_ld_32x32b_x16(taddr, v);
}

struct Bars {
  uint64_t b[24];
  uint32_t tmem_slot;
  uint32_t abort_flag;
};
struct BarsX : Bars {
  float xch[2][NSPLIT][128];  // [parity][part][row] exchange between the threads of a row
};

__device__ __forceinline__ uint8_t* align1024(uint8_t* p) {
  return reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(p) + 1023) & ~uintptr_t(1023));
}
// The bf16 forward, dQ and dK/dV kernels are persistent, one CTA per SM (the int8 P V forward is not): every role walks the same list of work
// items, barrier phases and ring positions running on, so the loads and first products of an item are under way while the previous
// one's results are read out of tensor memory and stored. (As one CTA per item, set-up, first loads and the epilogue of each, about
// 8 us, were exposed: a quarter of an item's time with a 512-key window. When it was made, forward and backward of 4 x 4096 tokens, 16 heads
// x 128, went from 1790 to 1612 us full causal, 744 to 691 windowed. Where every item has a CTA of its own the walk costs 1 to 5 % of the
// forward: 1 x 2048 56 and 59 us, 1 x 333 x 12 heads x 64 14.6 and 15.1, then; those take 52 and 11.5 now.) Item r * gridDim + c of the list goes to CTA c in even turns
// r and to the mirrored CTA in odd ones; the list is sorted by falling work (but for a lone last tile, which comes first), so
// the sums come out nearly even.
__device__ __forceinline__ int work_item(int turn) {
  return turn * (int)gridDim.x + (turn & 1 ? (int)(gridDim.x - 1 - blockIdx.x) : (int)blockIdx.x);
}
// A lane of an element warp never leaves an item alone where a bounded wait gives up: it would be missing from the tensor-memory accesses,
// votes and shuffles that follow, and the others would wait for it without a limit. dK/dV votes at each wait (mbar_wait_warp). In the
// forward kernels and dQ a warp goes on with whatever values are there, and votes at the item's end whether to store them and go on: by
// its lanes' own answers, which then wait no more, or in dQ by the abort word. Each kernel has the form that costs it least. us
// against waits that lanes left one by one, 4 x 4096 tokens, 16 heads x 128: dK/dV and dQ 944 and 936, windowed (512 keys) 344 and 346; with
// answers kept in dQ and the abort word in dK/dV 352. Forward 350 and 352; 2 % more with the abort word at a few hundred tokens.
// byte offset of the 16-byte chunk `ch` (0..7) of row r in a [rows][128 B] 128B-swizzled tile
__device__ __forceinline__ uint32_t swz(uint32_t r, uint32_t ch) { return r * 128u + ((ch ^ (r & 7u)) << 4); }

// K-major operand, tile made of [128 rows][64 elems] sub-tiles 16 KB apart; k-step kk = 16 elems
__device__ __forceinline__ uint64_t desc_k(uint32_t base, int kk) {
  return desc_plus(make_smem_desc(base, 16, 1024), (kk >> 2) * 16384 + (kk & 3) * 32);
}
// MN-major operand, tile made of [128 k-rows][64 mn elems] chunks 16 KB apart; k-step kk = 16 rows
__device__ __forceinline__ uint64_t desc_mn(uint32_t base, int kk) {
  return desc_plus(make_smem_desc(base, 16384, 1024), kk * 2048);
}

template <int D>
__device__ __forceinline__ void load_tile(uint8_t* dst, const CUtensorMap* tm, uint64_t* bar, int col, int row, int b) {
#pragma unroll
  for (int c = 0; c < D / 64; ++c) tma_load_3d(dst + c * 16384, tm, bar, col + c * 64, row, b);
}

__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
// key kj is hidden from query qi (causal, and the sliding window when window > 0)
__device__ __forceinline__ bool key_hidden(int kj, int qi, int window) { return kj > qi || (window > 0 && kj <= qi - window); }

// How much of a patch of keys [klo, khi] x queries [qlo, qhi] is visible. Steps on the diagonal or the window's edge hold few
// patches with both kinds of pair; the others need no position tests, or no arithmetic at all (P = dS = 0). A warp looks at
// its own 32 rows, so the answer is the same for all its lanes.
enum Seen : int { HIDDEN = 0, MIXED = 1, VISIBLE = 2 };
__device__ __forceinline__ Seen seen(int klo, int khi, int qlo, int qhi, int window) {
  if (klo > qhi || (window > 0 && khi <= qlo - window)) return HIDDEN;
  return khi <= qlo && (window == 0 || klo > qhi - window) ? VISIBLE : MIXED;
}

// Maximum of a thread's KPT raw scores. MASK = false is the common (fully visible) block: no position tests at all.
template <bool MASK>
__device__ __forceinline__ float scores_max(const uint32_t (&sv)[KPT], int kbase, int qi, int window) {
  float mx = -INFINITY;
  if constexpr (MASK) {
#pragma unroll
    for (int e = 0; e < KPT; ++e) mx = fmaxf(mx, key_hidden(kbase + e, qi, window) ? -INFINITY : __uint_as_float(sv[e]));
  } else {
#pragma unroll
    for (int e = 0; e < KPT; e += 2) mx = max3(mx, __uint_as_float(sv[e]), __uint_as_float(sv[e + 1]));
  }
  return mx;
}

// p = exp2(s * c - m) for the thread's KPT scores, packed for the P V product (bf16 pairs, or int8 quadruples when I8),
// and the two ascending row-sum chains (even keys, odd keys) as one packed value.
template <bool MASK, bool I8>
__device__ __forceinline__ f2 probs_pack(const uint32_t (&sv)[KPT], float c_log2, float m_safe, int kbase, int qi, int window,
                                         uint32_t (&pk)[KPT / 2]) {
  const f2 c2 = pack2(c_log2, c_log2), nm2 = pack2(-m_safe, -m_safe);
  f2 lsum2 = pack2(0.0f, 0.0f);
#pragma unroll
  for (int e = 0; e < KPT; e += 2) {
    f2 p2 = exp2_attn2(fma2(pack2(__uint_as_float(sv[e]), __uint_as_float(sv[e + 1])), c2, nm2));
    float p0, p1;
    unpack2(p2, p0, p1);
    if constexpr (MASK) {
      if (key_hidden(kbase + e, qi, window)) p0 = 0.0f;
      if (key_hidden(kbase + e + 1, qi, window)) p1 = 0.0f;
      p2 = pack2(p0, p1);
    }
    lsum2 = add2(lsum2, p2);
    if constexpr (I8) {
      // rint(127 p) sits in the low byte of 127 p + 1.5 * 2^23. (The product is rounded first, by itself: as packed instructions
      // the two come out as one multiply-add, whose ties are others.)
      float t0, t1;
      unpack2(add2(pack2(__fmul_rn(p0, 127.0f), __fmul_rn(p1, 127.0f)), pack2(12582912.0f, 12582912.0f)), t0, t1);
      const uint32_t two = __byte_perm(__float_as_uint(t0), __float_as_uint(t1), 0x0040);
      pk[e >> 2] = (e & 3) == 0 ? two : __byte_perm(pk[e >> 2], two, 0x5410);
    } else {
      pk[e >> 1] = pack_bf16(p0, p1);
    }
  }
  return lsum2;
}

// Stores of NCH (2 or 4) 16-byte chunks of each lane's row, rows of a warp being `pitch` bytes apart and `rows` the number of them (counted from
// lane 0's) that exist. NCH neighbouring lanes first exchange chunks, so that a lane writes chunk (lane % NCH) of each of their rows: an
// instruction then touches 32 / NCH lines instead of 32: the results of an item with a 512-key window took a tenth of its time. Backward, us,
// each lane its own row and so: 1 x 2048 tokens 134.7 and 130.6, 4 x 4096 1053 and 1037, with a 512-key window 365 to 388 and 350 to 372. (The
// forward, whose one thread a row has no registers left for it, takes 2 % longer so.)
template <int NCH>
__device__ __forceinline__ void store_rows(uint4 (&c)[NCH], void* mine, long pitch, int rows, int lane) {
#pragma unroll
  for (int s = 1; s < NCH; s *= 2) {
    const bool up = lane & s;
#pragma unroll
    for (int j = 0; j < NCH; ++j) {
      if (j & s) continue;
      uint4 &lo = c[j], &hi = c[j ^ s];
      const uint4 send = up ? lo : hi;
      uint4 got;
      got.x = __shfl_xor_sync(0xffffffffu, send.x, s);
      got.y = __shfl_xor_sync(0xffffffffu, send.y, s);
      got.z = __shfl_xor_sync(0xffffffffu, send.z, s);
      got.w = __shfl_xor_sync(0xffffffffu, send.w, s);
      if (up) lo = got; else hi = got;
    }
  }
  const int i = lane % NCH;
  uint8_t* first = static_cast<uint8_t*>(mine) - i * pitch + i * 16;
#pragma unroll
  for (int k = 0; k < NCH; ++k)
    if (lane - i + k < rows) *reinterpret_cast<uint4*>(first + k * pitch) = c[k];
}

// N outputs of a row divided by its sum l, packed to bf16 pairs; y = 1 / l correctly rounded. IEEE divisions without the divider: two
// steps q <- q + (a - q l) y from q = a y give the correctly rounded quotient where nothing over- or underflows (Markstein, IBM J. Res.
// Dev. 34, 1990); a warp with a value outside those bounds (a zero, whose sign the steps may lose, an infinity or a NaN among them)
// divides. Called by whole warps. (The divider's checks keep its instructions from overlapping: with it the 128 of a row took 10 thousand
// clocks, a third of an item with a 512-key window. us, divider and so: forward 1 x 16 tokens 8.6 and 6.9, 1 x 333 13.6 and 11.9, 1 x 2048 57
// and 54, 4 x 4096 388 and 362, with a 512-key window 176 and 163; int8 P V 1 x 2048 89 and 82, 4 x 4096 768 and 701, window 334 and 309.)
template <int N>
__device__ __forceinline__ void divide_pack(const float (&a)[N], float l, float y, uint32_t (&pk)[N / 2]) {
  float lo = fabsf(a[0]), hi = lo;
#pragma unroll
  for (int e = 1; e < N; ++e) {
    lo = fminf(lo, fabsf(a[e]));
    asm("max.NaN.f32 %0, %0, %1;" : "+f"(hi) : "f"(fabsf(a[e])));
  }
  if (__all_sync(0xffffffffu, l >= 0x1p-20f && l <= 0x1p40f && lo >= 0x1p-60f && hi <= 0x1p80f)) {
    const f2 y2 = pack2(y, y), nl2 = pack2(-l, -l);
#pragma unroll
    for (int e = 0; e < N; e += 2) {
      const f2 a2 = pack2(a[e], a[e + 1]);
      f2 q = mul2(a2, y2);
      q = fma2(fma2(q, nl2, a2), y2, q);
      q = fma2(fma2(q, nl2, a2), y2, q);
      float q0, q1;
      unpack2(q, q0, q1);
      pk[e >> 1] = pack_bf16(q0, q1);
    }
  } else {
#pragma unroll
    for (int e = 0; e < N; e += 2) pk[e >> 1] = pack_bf16(__fdiv_rn(a[e], l), __fdiv_rn(a[e + 1], l));
  }
}

// ------------------------------------------------- forward with P V in int8
__global__ void __launch_bounds__(ATT_THREADS, 1)
attn_fwd_i8pv_kernel(const __grid_constant__ CUtensorMap tmQK, const __grid_constant__ CUtensorMap tmV, __nv_bfloat16* __restrict__ O, long ldo,
                     float* __restrict__ lse_out, int T, int H, int Hkv, int window, float c_log2, const float* __restrict__ vstep,
                     uint32_t* __restrict__ status) {
  constexpr int D = 128;  // 128-byte value rows
  constexpr int TILE = BQ * D * 2;
  constexpr int ST = 2;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align1024(smem_raw);
  uint8_t* sQ = smem;
  uint8_t* sP = sQ + TILE;
  uint8_t* sK = sP + BQ * BKV * 2;
  uint8_t* sV = sK + ST * TILE;
  BarsX* bars = reinterpret_cast<BarsX*>(sV + ST * TILE);
  uint64_t* q_full = &bars->b[0];
  uint64_t* k_full = &bars->b[1];    // [ST]
  uint64_t* k_empty = &bars->b[3];   // [ST]
  uint64_t* v_full = &bars->b[5];    // [ST]
  uint64_t* v_empty = &bars->b[7];   // [ST]
  uint64_t* s_full = &bars->b[9];    // [2]
  uint64_t* s_empty = &bars->b[11];  // [2]
  uint64_t* p_ready = &bars->b[13];
  uint64_t* pv_full = &bars->b[14];
  volatile uint32_t* abort_flag = &bars->abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nq = (T + BQ - 1) / BQ;
  const int qt = nq - 1 - (int)((blockIdx.x + g_attn_rotation) % gridDim.x);  // heavy tiles first
  const int h = blockIdx.y, b = blockIdx.z;
  const int g = h / (H / Hkv);
  const int q0 = qt * BQ;
  const int jmax = qt;
  const int jmin = (window > 0 && q0 - window + 1 > 0) ? (q0 - window + 1) / BKV : 0;
  const int n = jmax - jmin + 1;

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int s = 0; s < ST; ++s) {
      mbar_init(&k_full[s], 1); mbar_init(&k_empty[s], 1); mbar_init(&v_full[s], 1); mbar_init(&v_empty[s], 1);
    }
    for (int s = 0; s < 2; ++s) { mbar_init(&s_full[s], 1); mbar_init(&s_empty[s], SOFTMAX_WARPS); }
    mbar_init(p_ready, SOFTMAX_WARPS);
    mbar_init(pv_full, 1);
    bars->abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) { tmem_alloc(&bars->tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = bars->tmem_slot;
  const uint32_t tS = tmem, tPV = tmem + 256;

  if (warp == 0) {
    if (elect_one()) {
      mbar_expect_tx(q_full, TILE);
      load_tile<D>(sQ, &tmQK, q_full, h * D, q0, b);
      for (int i = 0; i < n; ++i) {
        const int st = i % ST;
        const uint32_t ph = (i / ST) & 1;
        const int k0 = (jmin + i) * BKV;
        if (!mbar_wait(&k_empty[st], ph ^ 1, abort_flag)) break;
        mbar_expect_tx(&k_full[st], TILE);
        load_tile<D>(sK + st * TILE, &tmQK, &k_full[st], (H + g) * D, k0, b);
        if (!mbar_wait(&v_empty[st], ph ^ 1, abort_flag)) break;
        mbar_expect_tx(&v_full[st], BKV * D);  // int8 values: [128 keys][D bytes], one swizzle row per key
        tma_load_3d(sV + st * TILE, &tmV, &v_full[st], g * D, k0, b);
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      constexpr uint32_t idS = make_idesc(128, BKV, 0, 0);
      constexpr uint32_t idPV = make_idesc(128, D, 0, 1, 2, 1);
      const uint32_t aQ = smem_u32(sQ), aP = smem_u32(sP);
      bool ok = mbar_wait(q_full, 0, abort_flag);
      auto issue_S = [&](int i) {
        const int st = i % ST;
        if (!mbar_wait(&k_full[st], (i / ST) & 1, abort_flag)) return false;
        if (!mbar_wait(&s_empty[i & 1], ((i >> 1) & 1) ^ 1, abort_flag)) return false;
        tc_fence_after();
        const uint32_t aK = smem_u32(sK + st * TILE);
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) mma_f16_ss(tS + (i & 1) * 128, desc_k(aQ, kk), desc_k(aK, kk), idS, kk != 0);
        mma_commit(&s_full[i & 1]);
        mma_commit(&k_empty[st]);
        return true;
      };
      if (ok) ok = issue_S(0);
      for (int i = 0; i < n && ok; ++i) {
        if (i + 1 < n) { if (!issue_S(i + 1)) { ok = false; break; } }
        const int st = i % ST;
        if (!mbar_wait(p_ready, i & 1, abort_flag)) { ok = false; break; }
        if (!mbar_wait(&v_full[st], (i / ST) & 1, abort_flag)) { ok = false; break; }
        tc_fence_after();
        const uint32_t aV = smem_u32(sV + st * TILE);
        // P: [128 rows][128 int8 keys] K-major, 32 keys per instruction; V: [128 keys][128 int8] MN-major, 32 key rows per instruction
#pragma unroll
        for (int kk = 0; kk < BKV / 32; ++kk)
          mma_i8_ss(tPV, make_smem_desc(aP + kk * 32, 16, 1024), make_smem_desc(aV + kk * 4096, 16384, 1024), idPV, kk != 0);
        mma_commit(pv_full);
        mma_commit(&v_empty[st]);
      }
    }
  } else {
    constexpr int DH = D / NSPLIT;            // output columns per thread
    constexpr int CW = 16;                    // TMEM columns per load of the PV accumulator (short loads keep registers free)
    const int qd = warp & 3;
    const int part = (warp - 2) >> 2;
    const int r = qd * 32 + lane;          // row inside the tile == TMEM lane
    const int qi = q0 + r;                 // query position
    const uint32_t lane_off = uint32_t(qd * 32) << 16;
    float m_run = -INFINITY, l_run = 0.0f, alpha_prev = 0.0f;
    float c_prev = 0.0f;  // dequantisation factor (value step / 127) of the block whose P V is pending
    const int nblk = (T + BKV - 1) / BKV;
    // two accumulator words -> fp32 contributions; the integers (below 2^22) become floats by one addition to the bits of 1.5 * 2^23
    // and one subtraction, both exact. (This and the same for the probabilities, instead of the conversion pipe, a quarter as wide:
    // 4 x 4096 tokens, 16 heads, 812 -> 784 us; 1 x 2048 94 -> 91.)
    auto pv_vals = [&](uint32_t w0, uint32_t w1) {
      const f2 x = add2(pack2(__uint_as_float(w0 + 0x4B400000u), __uint_as_float(w1 + 0x4B400000u)), pack2(-12582912.0f, -12582912.0f));
      return mul2(x, pack2(c_prev, c_prev));
    };
    f2 o[DH / 2];
#pragma unroll
    for (int d = 0; d < DH / 2; ++d) o[d] = pack2(0.0f, 0.0f);
    bool ok = true;
    for (int i = 0; i < n; ++i) {
      const int j = jmin + i;
      const int kbase = j * BKV + part * KPT;
      const bool need_mask = (j == jmax) || (window > 0 && j * BKV < q0 + BQ - window);
      ok = ok && mbar_wait(&s_full[i & 1], (i >> 1) & 1, abort_flag);
      tc_fence_after();
      const uint32_t tSb = tS + (i & 1) * 128 + part * KPT + lane_off;
      // the thread's 32 raw scores stay in registers for both passes; once they are there the S buffer is free
      uint32_t sv[KPT];
      tmem_ld_32x32b_x32(tSb, sv);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&s_empty[i & 1]);
      float mx = need_mask ? scores_max<true>(sv, kbase, qi, window) : scores_max<false>(sv, kbase, qi, window);
      bars->xch[i & 1][part][r] = mx;
      quadrant_bar(qd);
#pragma unroll
      for (int pp = 0; pp < NSPLIT; ++pp) mx = fmaxf(mx, bars->xch[i & 1][pp][r]);
      const float m_new = fmaxf(m_run, __fmul_rn(mx, c_log2));
      const float m_safe = (m_new == -INFINITY) ? 0.0f : m_new;
      const float alpha = det_exp2_attn(__fadd_rn(m_run, -m_safe));
      // probabilities and the quarter-row sum first (independent of O), while the tensor core finishes the previous P V
      uint32_t pk[KPT / 2];
      const f2 lsum2 = need_mask ? probs_pack<true, true>(sv, c_log2, m_safe, kbase, qi, window, pk)
                                 : probs_pack<false, true>(sv, c_log2, m_safe, kbase, qi, window, pk);
      // deferred accumulation of the previous block's P V (its completion also frees the P buffer)
      if (i > 0) {
        ok = ok && mbar_wait(pv_full, (i - 1) & 1, abort_flag);
        tc_fence_after();
        const f2 a2 = pack2(alpha_prev, alpha_prev);
#pragma unroll
        for (int c = 0; c < DH / CW; ++c) {
          uint32_t v[CW];
          tmem_ld_cols<CW>(tPV + lane_off + part * DH + c * CW, v);
          tmem_ld_wait();
#pragma unroll
          for (int e = 0; e < CW; e += 2)
            o[(c * CW + e) >> 1] = fma2(o[(c * CW + e) >> 1], a2, pv_vals(v[e], v[e + 1]));
        }
      }
      // keys part*32 .. +31 are bytes part*32 .. +31 of the 128-byte row: chunks part*2, part*2 + 1
#pragma unroll
      for (int w = 0; w < 2; ++w)
        *reinterpret_cast<uint4*>(sP + swz(r, part * 2 + w)) = make_uint4(pk[4 * w], pk[4 * w + 1], pk[4 * w + 2], pk[4 * w + 3]);
      float ls0, ls1;
      unpack2(lsum2, ls0, ls1);
      const float lsum = __fadd_rn(ls0, ls1);
      l_run = __fmaf_rn(l_run, alpha, lsum);
      m_run = m_new;
      alpha_prev = alpha;
      c_prev = __fmul_rn(vstep[((long)b * Hkv + g) * nblk + j], 1.0f / 127.0f);
      fence_proxy_async_smem();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_ready);
    }
    ok = ok && mbar_wait(pv_full, (n - 1) & 1, abort_flag);
    ok = __all_sync(0xffffffffu, ok);
    tc_fence_after();
    bars->xch[n & 1][part][r] = l_run;
    quadrant_bar(qd);
    float l_tot = bars->xch[n & 1][0][r];
#pragma unroll
    for (int pp = 1; pp < NSPLIT; ++pp) l_tot = __fadd_rn(l_tot, bars->xch[n & 1][pp][r]);
    if (ok) {
      const bool in_range = qi < T;
      const float y = __frcp_rn(l_tot);
      __nv_bfloat16* orow = O + ((long)b * T + qi) * ldo + (long)h * D + part * DH;
#pragma unroll
      for (int c = 0; c < DH / CW; ++c) {
        uint32_t v[CW];
        tmem_ld_cols<CW>(tPV + lane_off + part * DH + c * CW, v);
        tmem_ld_wait();
        uint32_t pk[CW / 2];
        float a[CW];
#pragma unroll
        for (int e = 0; e < CW; e += 2) unpack2(fma2(o[(c * CW + e) >> 1], pack2(alpha_prev, alpha_prev), pv_vals(v[e], v[e + 1])), a[e], a[e + 1]);
        divide_pack<CW>(a, l_tot, y, pk);
        if (in_range) {
#pragma unroll
          for (int w = 0; w < CW / 8; ++w)
            reinterpret_cast<uint4*>(orow + c * CW)[w] = make_uint4(pk[4 * w], pk[4 * w + 1], pk[4 * w + 2], pk[4 * w + 3]);
        }
      }
      if (in_range && part == 0)
        lse_out[((long)b * H + h) * T + qi] = __fmaf_rn(det_logf(l_tot), 1.44269504088896341f, m_run);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && bars->abort_flag && status) atomicExch(status, 2u);
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem, 512); }
}

// ------------------------------------------------- forward, two query tiles per CTA
// The bf16 forward. One CTA owns TWO adjacent 128-row query tiles (A, B) of one (batch, head) and walks the key blocks
// both need; warp 0 loads K and V once for both tiles, warp 1 issues every tensor-core product, warps 2..5 are tile A's
// softmax (ONE THREAD PER ROW, so no value ever crosses threads) and warps 6..9 tile B's. While one tile's softmax
// runs, the tensor core works for the other tile. Tensor memory: S_A | S_B | O_A | O_B, 128 columns each.
//   S = Q K^T lands in S_X; the row's thread reads it twice (maximum, then probabilities) and overwrites its first 64
//   columns with P as bf16 pairs, which is the A operand of P V (tcgen05.mma with A in tensor memory); O_X is the
//   accumulator of P V over all key blocks: before block i > first the thread multiplies its O row by
//   alpha = exp2(m_old - m_new) in place (skipped, with identical bits, when alpha == 1 for the whole warp), then the
//   tensor core adds the block's 8 k-steps to it. The row sum keeps the four 32-key quarter chains of the CPU twin.
constexpr int F2_THREADS = 64 + 256;

struct Bars2 {
  uint64_t q_full, q_empty, k_full[2], k_empty[2], v_full[2], v_empty[2], s_full[2], p_ready[2], o_done[2];
  uint32_t tmem_slot;
  uint32_t abort_flag;
};

template <int D>
__global__ void __launch_bounds__(F2_THREADS, 1)
attn_fwd2_kernel(const __grid_constant__ CUtensorMap tmQK, const __grid_constant__ CUtensorMap tmV,
                 __nv_bfloat16* __restrict__ O, long ldo, float* __restrict__ lse_out, int B, int T, int H, int Hkv, int window,
                 float c_log2, uint32_t* __restrict__ status) {
  constexpr int TILE = BQ * D * 2;
  constexpr int ST = 2;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align1024(smem_raw);
  uint8_t* sQ = smem;                  // [2] tiles A, B
  uint8_t* sK = sQ + 2 * TILE;         // [ST]
  uint8_t* sV = sK + ST * TILE;        // [ST]
  Bars2* bars = reinterpret_cast<Bars2*>(sV + ST * TILE);
  volatile uint32_t* abort_flag = &bars->abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nq = (T + BQ - 1) / BQ, npairs = (nq + 1) / 2, heads = B * H;
  const int items = npairs * heads;
  // Item -> pair of tiles (heavy pairs first), head, sequence, and the key blocks: [jlo_X, jhi_X] of tile X; the CTA walks
  // [jlo_A, jhi_B] (jlo_A <= jlo_B, jhi_A < jhi_B)
  struct Item {
    int tile0, h, b, g, jlo, n, jhiA, jloB, jhiB;
    bool hasB;
    __device__ __forceinline__ bool act(int X, int j) const { return X == 0 ? j <= jhiA : (hasB && j >= jloB && j <= jhiB); }
  };
  auto item_of = [&](int w) {
    Item it;
    const int hb = w % heads;
    it.tile0 = 2 * (npairs - 1 - rotated(w / heads, npairs));
    it.h = hb % H;
    it.b = hb / H;
    it.g = it.h / (H / Hkv);
    it.hasB = it.tile0 + 1 < nq;
    auto jlo_of = [&](int t) { const int q0 = t * BQ; return (window > 0 && q0 - window + 1 > 0) ? (q0 - window + 1) / BKV : 0; };
    it.jlo = jlo_of(it.tile0);
    it.jhiA = it.tile0;
    it.jloB = it.hasB ? jlo_of(it.tile0 + 1) : 0;
    it.jhiB = it.tile0 + 1;
    it.n = (it.hasB ? it.jhiB : it.jhiA) - it.jlo + 1;
    return it;
  };

  if (threadIdx.x == 0) {
    mbar_init(&bars->q_full, 1);
    mbar_init(&bars->q_empty, 1);
    for (int s = 0; s < ST; ++s) {
      mbar_init(&bars->k_full[s], 1); mbar_init(&bars->k_empty[s], 1); mbar_init(&bars->v_full[s], 1); mbar_init(&bars->v_empty[s], 1);
    }
    for (int x = 0; x < 2; ++x) { mbar_init(&bars->s_full[x], 1); mbar_init(&bars->p_ready[x], 4); mbar_init(&bars->o_done[x], 1); }
    bars->abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) { tmem_alloc(&bars->tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  after_predecessor();
  const uint32_t tmem = bars->tmem_slot;

  if (warp == 0) {
    if (elect_one()) {
      uint32_t ring = 0;  // key blocks loaded so far
      bool ok = true;
      for (int turn = 0, w; ok && (w = work_item(turn)) < items; ++turn) {
        const Item it = item_of(w);
        if (!mbar_wait(&bars->q_empty, (turn & 1) ^ 1, abort_flag)) break;
        mbar_expect_tx(&bars->q_full, it.hasB ? 2 * TILE : TILE);
        load_tile<D>(sQ, &tmQK, &bars->q_full, it.h * D, it.tile0 * BQ, it.b);
        if (it.hasB) load_tile<D>(sQ + TILE, &tmQK, &bars->q_full, it.h * D, (it.tile0 + 1) * BQ, it.b);
        for (int i = 0; i < it.n; ++i, ++ring) {
          const int st = ring % ST;
          const uint32_t ph = (ring / ST) & 1;
          const int k0 = (it.jlo + i) * BKV;
          if (!(ok = mbar_wait(&bars->k_empty[st], ph ^ 1, abort_flag))) break;
          mbar_expect_tx(&bars->k_full[st], TILE);
          load_tile<D>(sK + st * TILE, &tmQK, &bars->k_full[st], (H + it.g) * D, k0, it.b);
          if (!(ok = mbar_wait(&bars->v_empty[st], ph ^ 1, abort_flag))) break;
          mbar_expect_tx(&bars->v_full[st], TILE);
          load_tile<D>(sV + st * TILE, &tmV, &bars->v_full[st], (H + Hkv + it.g) * D, k0, it.b);
        }
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      constexpr uint32_t idS = make_idesc(128, BKV, 0, 0);
      constexpr uint32_t idPV = make_idesc(128, D, 0, 1);
      // Scores are formed one step ahead, across the boundaries of items: the next item's first ones go right behind this one's last P V,
      // while the softmax warps still divide and store. us, from the next item's beginning and so: 1 x 2048 tokens 54.4 and 52.0, 4 x 4096
      // 363 and 357, with a 512-key window 163 and 152; 8 x 2048, 4 x 64 heads, 53.8 and 52.0. (The same in dQ: 1033 to 1046 for the whole
      // backward, windowed 366 to 360; not taken.)
      uint32_t ring = 0, blocks[2] = {0, 0};  // key blocks so far; those of each tile
      // this step's item and key block, and those of the step whose scores are formed now: one further, in the next item after the last
      Item it, ahead = item_of(work_item(0));
      int turn = -1, i = 0, ahead_i = 0;
      bool ok = true;
      for (bool first = true; ok; first = false) {
        bool scores = ahead_i < ahead.n, k_here = false;
        for (int X = 0; X < 2 && ok; ++X) {
          if (!first && it.act(X, it.jlo + i)) {
            const int j = it.jlo + i, st = (ring - 1) % ST;
            if (!(ok = mbar_wait(&bars->v_full[st], ((ring - 1) / ST) & 1, abort_flag) && mbar_wait(&bars->p_ready[X], blocks[X] & 1, abort_flag))) break;
            ++blocks[X];
            tc_fence_after();
            const uint32_t aV = smem_u32(sV + st * TILE);
            const bool fresh = j == (X == 0 ? it.jlo : it.jloB);
#pragma unroll
            for (int kk = 0; kk < BKV / 16; ++kk)
              mma_f16_ts(tmem + 256 + X * 128, tmem + X * 128 + kk * 8, desc_mn(aV, kk), idPV, !fresh || kk != 0);
            if (j == (X == 0 ? it.jhiA : it.jhiB)) mma_commit(&bars->o_done[X]);
          }
          // this tile's next S goes right behind its P V (it overwrites the P just consumed)
          if (scores && ahead.act(X, ahead.jlo + ahead_i)) {
            if (!k_here) {
              if (ahead_i == 0 && !(ok = mbar_wait(&bars->q_full, (turn + 1) & 1, abort_flag))) break;
              if (!(ok = mbar_wait(&bars->k_full[ring % ST], (ring / ST) & 1, abort_flag))) break;
              tc_fence_after();
              k_here = true;
            }
            const uint32_t aK = smem_u32(sK + (ring % ST) * TILE), aQ = smem_u32(sQ + X * TILE);
#pragma unroll
            for (int kk = 0; kk < D / 16; ++kk) mma_f16_ss(tmem + X * 128, desc_k(aQ, kk), desc_k(aK, kk), idS, kk != 0);
            mma_commit(&bars->s_full[X]);
          }
        }
        if (!ok) break;
        if (!first) mma_commit(&bars->v_empty[(ring - 1) % ST]);
        if (!scores) break;
        mma_commit(&bars->k_empty[ring % ST]);
        if (ahead_i == ahead.n - 1) mma_commit(&bars->q_empty);  // the item's last scores are on their way
        if (ahead_i == 0) {
          it = ahead;
          ++turn;
        }
        i = ahead_i;
        ++ring;
        if (++ahead_i == ahead.n) {
          const int w = work_item(turn + 1);
          if (w < items) {
            ahead = item_of(w);
            ahead_i = 0;
          }
        }
      }
    }
  } else {
    const int X = (warp - 2) >> 2;           // tile of this warp
    const int quad = warp & 3;               // TMEM lane quadrant this warp may touch
    const int r = quad * 32 + lane;          // row inside the tile == TMEM lane
    const uint32_t lane_off = uint32_t(quad * 32) << 16;
    const uint32_t tS = tmem + X * 128 + lane_off, tO = tmem + 256 + X * 128 + lane_off;
    uint32_t scores = 0, outputs = 0;  // score tiles and results of this tile so far (barrier phases)
    bool ok = true;
    for (int turn = 0, w; ok && (w = work_item(turn)) < items; ++turn) {
      const Item it = item_of(w);
      if (X == 1 && !it.hasB) continue;
      const int q0 = (it.tile0 + X) * BQ, qi = q0 + r, h = it.h, b = it.b;
      const int jloX = X == 0 ? it.jlo : it.jloB, jhiX = X == 0 ? it.jhiA : it.jhiB;
      float m_run = -INFINITY, l_run[NSPLIT] = {0.0f, 0.0f, 0.0f, 0.0f};
      for (int j = jloX; j <= jhiX; ++j) {
        const bool need_mask = (j == jhiX) || (window > 0 && j * BKV < q0 + BQ - window);
        ok = ok && mbar_wait(&bars->s_full[X], scores & 1, abort_flag);
        ++scores;
        tc_fence_after();
        // pass 1: row maximum. Fully visible blocks take the unrolled path with the next 32 columns already in flight
        // while the current ones are reduced; blocks on the diagonal or the window edge take a compact loop.
        float mx = -INFINITY;
        if (!need_mask) {
          uint32_t sa[KPT], sb[KPT];
          tmem_ld_32x32b_x32(tS, sa);
          tmem_ld_wait();
          tmem_ld_32x32b_x32(tS + KPT, sb);
          mx = scores_max<false>(sa, 0, 0, 0);
          tmem_ld_wait();
          tmem_ld_32x32b_x32(tS + 2 * KPT, sa);
          mx = fmaxf(mx, scores_max<false>(sb, 0, 0, 0));
          tmem_ld_wait();
          tmem_ld_32x32b_x32(tS + 3 * KPT, sb);
          mx = fmaxf(mx, scores_max<false>(sa, 0, 0, 0));
          tmem_ld_wait();
          mx = fmaxf(mx, scores_max<false>(sb, 0, 0, 0));
        } else {
#pragma unroll 1
          for (int c = 0; c < NSPLIT; ++c) {
            uint32_t sv[KPT];
            tmem_ld_32x32b_x32(tS + c * KPT, sv);
            tmem_ld_wait();
            mx = fmaxf(mx, scores_max<true>(sv, j * BKV + c * KPT, qi, window));
          }
        }
        const float m_new = fmaxf(m_run, __fmul_rn(mx, c_log2));
        const float m_safe = (m_new == -INFINITY) ? 0.0f : m_new;
        const float alpha = det_exp2_attn(__fadd_rn(m_run, -m_safe));
        // O row *= alpha (the previous P V is complete: its S product was issued behind it)
        if (j > jloX && __any_sync(0xffffffffu, alpha != 1.0f)) {
          const f2 a2 = pack2(alpha, alpha);
#pragma unroll
          for (int c = 0; c < D / 32; ++c) {
            uint32_t v[32];
            tmem_ld_32x32b_x32(tO + c * 32, v);
            tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 32; e += 2) {
              float a0, a1;
              unpack2(mul2(pack2(__uint_as_float(v[e]), __uint_as_float(v[e + 1])), a2), a0, a1);
              v[e] = __float_as_uint(a0);
              v[e + 1] = __float_as_uint(a1);
            }
            tmem_st_32x32b_x32(tO + c * 32, v);
          }
        }
        // pass 2: probabilities, quarter sums, P (bf16 pairs) over the first 64 columns of S (a P store only ever
        // covers columns whose scores have been read already)
        if (!need_mask) {
          uint32_t sa[KPT], sb[KPT], pk[KPT / 2];
          float ls0, ls1;
          tmem_ld_32x32b_x32(tS, sa);
          tmem_ld_wait();
          tmem_ld_32x32b_x32(tS + KPT, sb);
          unpack2(probs_pack<false, false>(sa, c_log2, m_safe, 0, 0, 0, pk), ls0, ls1);
          l_run[0] = __fmaf_rn(l_run[0], alpha, __fadd_rn(ls0, ls1));
          tmem_ld_wait();
          tmem_st_32x32b_x16(tS, pk);
          tmem_ld_32x32b_x32(tS + 2 * KPT, sa);
          unpack2(probs_pack<false, false>(sb, c_log2, m_safe, 0, 0, 0, pk), ls0, ls1);
          l_run[1] = __fmaf_rn(l_run[1], alpha, __fadd_rn(ls0, ls1));
          tmem_ld_wait();
          tmem_st_32x32b_x16(tS + KPT / 2, pk);
          tmem_ld_32x32b_x32(tS + 3 * KPT, sb);
          unpack2(probs_pack<false, false>(sa, c_log2, m_safe, 0, 0, 0, pk), ls0, ls1);
          l_run[2] = __fmaf_rn(l_run[2], alpha, __fadd_rn(ls0, ls1));
          tmem_ld_wait();
          tmem_st_32x32b_x16(tS + KPT, pk);
          unpack2(probs_pack<false, false>(sb, c_log2, m_safe, 0, 0, 0, pk), ls0, ls1);
          l_run[3] = __fmaf_rn(l_run[3], alpha, __fadd_rn(ls0, ls1));
          tmem_st_32x32b_x16(tS + 3 * (KPT / 2), pk);
        } else {
          float lq[NSPLIT];
#pragma unroll 1
          for (int c = 0; c < NSPLIT; ++c) {
            uint32_t sv[KPT], pk[KPT / 2];
            tmem_ld_32x32b_x32(tS + c * KPT, sv);
            tmem_ld_wait();
            float ls0, ls1;
            unpack2(probs_pack<true, false>(sv, c_log2, m_safe, j * BKV + c * KPT, qi, window, pk), ls0, ls1);
            const float lq_c = __fadd_rn(ls0, ls1);
            lq[0] = c == 0 ? lq_c : lq[0]; lq[1] = c == 1 ? lq_c : lq[1]; lq[2] = c == 2 ? lq_c : lq[2]; lq[3] = c == 3 ? lq_c : lq[3];
            tmem_st_32x32b_x16(tS + c * (KPT / 2), pk);
          }
#pragma unroll
          for (int c = 0; c < NSPLIT; ++c) l_run[c] = __fmaf_rn(l_run[c], alpha, lq[c]);
        }
        tmem_st_wait();
        m_run = m_new;
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars->p_ready[X]);
      }
      ok = ok && mbar_wait(&bars->o_done[X], outputs & 1, abort_flag);
      ok = __all_sync(0xffffffffu, ok);
      ++outputs;
      tc_fence_after();
      if (ok) {
        const float l_tot = __fadd_rn(__fadd_rn(__fadd_rn(l_run[0], l_run[1]), l_run[2]), l_run[3]);
        const bool in_range = qi < T;
        const float y = __frcp_rn(l_tot);
        __nv_bfloat16* orow = O + ((long)b * T + qi) * ldo + (long)h * D;
#pragma unroll
        for (int c = 0; c < D / 32; ++c) {
          uint32_t v[32];
          tmem_ld_32x32b_x32(tO + c * 32, v);
          tmem_ld_wait();
          uint32_t pk[16];
          float a[32];
#pragma unroll
          for (int e = 0; e < 32; ++e) a[e] = __uint_as_float(v[e]);
          divide_pack<32>(a, l_tot, y, pk);
          if (in_range) {
#pragma unroll
            for (int w = 0; w < 4; ++w)
              reinterpret_cast<uint4*>(orow + c * 32)[w] = make_uint4(pk[4 * w], pk[4 * w + 1], pk[4 * w + 2], pk[4 * w + 3]);
          }
        }
        if (in_range) lse_out[((long)b * H + h) * T + qi] = __fmaf_rn(det_logf(l_tot), 1.44269504088896341f, m_run);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && bars->abort_flag && status) atomicExch(status, 2u);
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem, 512); }
}

// Backward element math for a thread's KPT (score, dP) pairs: p = exp2(s * c - lse) (0 where hidden or the row is out of
// range), ds = (p * (dp - delta)) * scale; both packed to bf16 pairs.
template <bool MASK>
__device__ __forceinline__ void dscores(const uint32_t (&vs)[16], const uint32_t (&vd)[16], float c_log2, float lse_r, float dl_r,
                                        float scale, bool row_ok, int kbase, int qi, int window, uint32_t (&dsr)[8]) {
  const f2 c2 = pack2(c_log2, c_log2), nl2 = pack2(-lse_r, -lse_r), nd2 = pack2(-dl_r, -dl_r), sc2 = pack2(scale, scale);
#pragma unroll
  for (int e = 0; e < 16; e += 2) {
    f2 p2 = exp2_attn2(fma2(pack2(__uint_as_float(vs[e]), __uint_as_float(vs[e + 1])), c2, nl2));
    if constexpr (MASK) {
      float p0, p1;
      unpack2(p2, p0, p1);
      if (!row_ok || key_hidden(kbase + e, qi, window)) p0 = 0.0f;
      if (!row_ok || key_hidden(kbase + e + 1, qi, window)) p1 = 0.0f;
      p2 = pack2(p0, p1);
    }
    const f2 d2 = mul2(mul2(p2, add2(pack2(__uint_as_float(vd[e]), __uint_as_float(vd[e + 1])), nd2)), sc2);
    float d0, d1;
    unpack2(d2, d0, d1);
    dsr[e >> 1] = pack_bf16(d0, d1);
  }
}

// ------------------------------------------------ backward: dQ, two query tiles per CTA
// Same organisation as the forward: one CTA owns two adjacent 128-row query tiles, one thread per query row, and the
// tensor core serves one tile while the other tile's threads do the element math (two threads per row, each with half
// of the step's keys; nothing crosses threads in the backward). Keys advance in steps of 64: S = Q K^T and
// dP = dO V^T (128 x 64 each) land in tensor memory, the row's threads turn them into dS = p (dP - delta) scale, store
// it as bf16 pairs over their own score columns, and dQ += dS K runs with dS as the tensor-memory A operand. dQ accumulates over ascending keys in 16-key tensor-core steps, exactly as before.
// Tensor memory per tile: S 64 | dP 64 | dQ 128 columns.
constexpr int HK = 64;  // keys per step

template <int D, int ROWS>
__device__ __forceinline__ void load_tile_r(uint8_t* dst, const CUtensorMap* tm, uint64_t* bar, int col, int row, int b) {
#pragma unroll
  for (int c = 0; c < D / 64; ++c) tma_load_3d(dst + c * (ROWS * 128), tm, bar, col + c * 64, row, b);
}
// K-major / MN-major operand descriptors for tiles of ROWS rows ([ROWS][64 elems] sub-tiles ROWS * 128 bytes apart)
template <int ROWS>
__device__ __forceinline__ uint64_t desc_k_r(uint32_t base, int kk) {
  return desc_plus(make_smem_desc(base, 16, 1024), (kk >> 2) * (ROWS * 128) + (kk & 3) * 32);
}
template <int ROWS>
__device__ __forceinline__ uint64_t desc_mn_r(uint32_t base, int kk) {
  return desc_plus(make_smem_desc(base, ROWS * 128, 1024), kk * 2048);
}

struct BarsQ2 {
  uint64_t qdo_full, qdo_empty, kv_full[3], kv_empty[3], sdp_full[2], ds_ready[2], dq_done[2];
  uint32_t tmem_slot;
  uint32_t abort_flag;
};

template <int D>
__global__ void __launch_bounds__(ATT_THREADS, 1)
attn_bwd_q2_kernel(const __grid_constant__ CUtensorMap tmQK, const __grid_constant__ CUtensorMap tmDO,
                   const __grid_constant__ CUtensorMap tmK64, const __grid_constant__ CUtensorMap tmV64,
                   const float* __restrict__ lse, const float* __restrict__ delta, __nv_bfloat16* __restrict__ dQ, long lddq, int B, int T,
                   int H, int Hkv, int window, float scale, float c_log2, uint32_t* __restrict__ status) {
  constexpr int TILE = BQ * D * 2;    // a [128][D] query-side tile
  constexpr int KT = HK * D * 2;      // a [64][D] key-side tile
  constexpr int ST = 3;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align1024(smem_raw);
  uint8_t* sQ = smem;                 // [2]
  uint8_t* sDO = sQ + 2 * TILE;       // [2]
  uint8_t* sK = sDO + 2 * TILE;       // [ST]
  uint8_t* sV = sK + ST * KT;         // [ST]
  BarsQ2* bars = reinterpret_cast<BarsQ2*>(sV + ST * KT);
  volatile uint32_t* abort_flag = &bars->abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nq = (T + BQ - 1) / BQ, npairs = (nq + 1) / 2, heads = B * H;
  const int items = npairs * heads;
  // Item -> pair of tiles (heavy pairs first), head, sequence, and the 64-key steps [ulo_X, uhi_X] of tile X: every step that
  // holds a key some row of the tile can see
  struct Item {
    int tile0, h, b, g, ulo, n, uhiA, uloB, uhiB;
    bool hasB;
    __device__ __forceinline__ bool act(int X, int u) const { return X == 0 ? u <= uhiA : (hasB && u >= uloB && u <= uhiB); }
  };
  auto item_of = [&](int w) {
    Item it;
    const int hb = w % heads;
    it.tile0 = 2 * (npairs - 1 - rotated(w / heads, npairs));
    it.h = hb % H;
    it.b = hb / H;
    it.g = it.h / (H / Hkv);
    it.hasB = it.tile0 + 1 < nq;
    auto ulo_of = [&](int t) { const int q0 = t * BQ; return (window > 0 && q0 - window + 1 > 0) ? (q0 - window + 1) / HK : 0; };
    it.ulo = ulo_of(it.tile0);
    it.uhiA = 2 * it.tile0 + 1;
    it.uloB = it.hasB ? ulo_of(it.tile0 + 1) : 0;
    it.uhiB = 2 * it.tile0 + 3;
    it.n = (it.hasB ? it.uhiB : it.uhiA) - it.ulo + 1;
    return it;
  };

  if (threadIdx.x == 0) {
    mbar_init(&bars->qdo_full, 1);
    mbar_init(&bars->qdo_empty, 1);
    for (int s = 0; s < ST; ++s) { mbar_init(&bars->kv_full[s], 1); mbar_init(&bars->kv_empty[s], 1); }
    for (int x = 0; x < 2; ++x) { mbar_init(&bars->sdp_full[x], 1); mbar_init(&bars->ds_ready[x], 8); mbar_init(&bars->dq_done[x], 1); }
    bars->abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) { tmem_alloc(&bars->tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = bars->tmem_slot;

  if (warp == 0) {
    if (elect_one()) {
      uint32_t ring = 0;
      bool ok = true;
      for (int turn = 0, w; ok && (w = work_item(turn)) < items; ++turn) {
        const Item it = item_of(w);
        if (!mbar_wait(&bars->qdo_empty, (turn & 1) ^ 1, abort_flag)) break;
        mbar_expect_tx(&bars->qdo_full, (it.hasB ? 4 : 2) * TILE);
        for (int X = 0; X < (it.hasB ? 2 : 1); ++X) {
          load_tile<D>(sQ + X * TILE, &tmQK, &bars->qdo_full, it.h * D, (it.tile0 + X) * BQ, it.b);
          load_tile<D>(sDO + X * TILE, &tmDO, &bars->qdo_full, it.h * D, (it.tile0 + X) * BQ, it.b);
        }
        for (int i = 0; i < it.n; ++i, ++ring) {
          const int st = ring % ST;
          const int k0 = (it.ulo + i) * HK;
          if (!(ok = mbar_wait(&bars->kv_empty[st], ((ring / ST) & 1) ^ 1, abort_flag))) break;
          mbar_expect_tx(&bars->kv_full[st], 2 * KT);
          load_tile_r<D, HK>(sK + st * KT, &tmK64, &bars->kv_full[st], (H + it.g) * D, k0, it.b);
          load_tile_r<D, HK>(sV + st * KT, &tmV64, &bars->kv_full[st], (H + Hkv + it.g) * D, k0, it.b);
        }
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      constexpr uint32_t idS = make_idesc(128, HK, 0, 0);  // S = Q K^T, dP = dO V^T: 128 x 64
      constexpr uint32_t idQ = make_idesc(128, D, 0, 1);   // dQ = dS K: A in tensor memory, B MN-major
      bool ok = true;
      uint32_t ring = 0, parity[2] = {0, 0};  // key steps before this item; dS tiles consumed per tile
      for (int turn = 0, w; ok && (w = work_item(turn)) < items; ++turn) {
        const Item it = item_of(w);
        const int n = it.n;
        if (!(ok = mbar_wait(&bars->qdo_full, turn & 1, abort_flag))) break;
        bool first[2] = {true, true};
        auto kv_ready = [&](int i) { return mbar_wait(&bars->kv_full[(ring + i) % ST], ((ring + i) / ST) & 1, abort_flag); };
        auto issue_sdp = [&](int X, int i) {
          const uint32_t aK = smem_u32(sK + ((ring + i) % ST) * KT), aV = smem_u32(sV + ((ring + i) % ST) * KT);
          const uint32_t aQ = smem_u32(sQ + X * TILE), aDO = smem_u32(sDO + X * TILE);
#pragma unroll
          for (int kk = 0; kk < D / 16; ++kk) mma_f16_ss(tmem + X * 256, desc_k(aQ, kk), desc_k_r<HK>(aK, kk), idS, kk != 0);
#pragma unroll
          for (int kk = 0; kk < D / 16; ++kk) mma_f16_ss(tmem + X * 256 + 64, desc_k(aDO, kk), desc_k_r<HK>(aV, kk), idS, kk != 0);
          mma_commit(&bars->sdp_full[X]);
        };
        if (!(ok = kv_ready(0))) break;
        tc_fence_after();
        for (int X = 0; X < 2; ++X)
          if (it.act(X, it.ulo)) issue_sdp(X, 0);
        for (int i = 0; i < n && ok; ++i) {
          const int st = (ring + i) % ST, u = it.ulo + i;
          const bool more = i + 1 < n;
          bool kv_next = false;
          for (int X = 0; X < 2 && ok; ++X) {
            if (it.act(X, u)) {
              if (!(ok = mbar_wait(&bars->ds_ready[X], parity[X] & 1, abort_flag))) break;
              ++parity[X];
              tc_fence_after();
              const uint32_t aK = smem_u32(sK + st * KT);
#pragma unroll
              for (int kk = 0; kk < HK / 16; ++kk)
                mma_f16_ts(tmem + X * 256 + 128, tmem + X * 256 + (kk >> 1) * 32 + (kk & 1) * 8, desc_mn_r<HK>(aK, kk), idQ, !first[X] || kk != 0);
              first[X] = false;
              if (u == (X == 0 ? it.uhiA : it.uhiB)) mma_commit(&bars->dq_done[X]);
            }
            if (more && it.act(X, u + 1)) {
              if (!kv_next) {
                if (!(ok = kv_ready(i + 1))) break;
                tc_fence_after();
                kv_next = true;
              }
              issue_sdp(X, i + 1);
            }
          }
          if (!ok) break;
          mma_commit(&bars->kv_empty[st]);
          if (i + 2 == n) mma_commit(&bars->qdo_empty);  // the item's last scores are on their way (an item has two steps at least)
        }
        ring += n;
      }
    }
  } else {
    // sixteen element warps: two threads per query row (32 of the step's 64 keys each), 8 warps per tile
    const int X = (warp - 2) >> 3;
    const int quad = warp & 3;
    const int hf = ((warp - 2) & 7) >> 2;    // which half of the step's keys
    const int r = quad * 32 + lane;
    const uint32_t lane_off = uint32_t(quad * 32) << 16;
    const uint32_t tS = tmem + X * 256 + lane_off + hf * 32, tDP = tS + 64, tDQ = tmem + X * 256 + 128 + lane_off;
    uint32_t scores = 0, outputs = 0;  // score tiles and results of this tile so far (barrier phases)
    bool ok = true;
    for (int turn = 0, w; ok && (w = work_item(turn)) < items; ++turn) {
      const Item it = item_of(w);
      if (X == 1 && !it.hasB) continue;
      const int q0 = (it.tile0 + X) * BQ, qi = q0 + r, h = it.h, b = it.b;
      const bool row_ok = qi < T;
      const float lse_r = row_ok ? lse[((long)b * H + h) * T + qi] : 0.0f;
      const float dl_r = row_ok ? delta[((long)b * H + h) * T + qi] : 0.0f;
      const int uloX = X == 0 ? it.ulo : it.uloB, uhiX = X == 0 ? it.uhiA : it.uhiB;
      for (int u = uloX; u <= uhiX; ++u) {
        const int k0 = u * HK;
        // some (row, key) pair of this step is hidden, or the tile has rows past the end of the sequence
        const bool need_mask = (k0 + HK - 1 > q0) || (window > 0 && k0 <= q0 + BQ - 1 - window) || (q0 + BQ > T);
        mbar_wait(&bars->sdp_full[X], scores & 1, abort_flag);
        ++scores;
        tc_fence_after();
        // dS (bf16 pairs, 8 columns per 16 keys) goes over the thread's own score columns, which it has read by then
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint32_t sa[16], da[16], pk[8];
          tmem_ld_32x32b_x16(tS + c * 16, sa);
          tmem_ld_32x32b_x16(tDP + c * 16, da);
          tmem_ld_wait();
          if (need_mask) dscores<true>(sa, da, c_log2, lse_r, dl_r, scale, row_ok, k0 + hf * 32 + c * 16, qi, window, pk);
          else dscores<false>(sa, da, c_log2, lse_r, dl_r, scale, true, 0, 0, 0, pk);
          tmem_st_32x32b_x8(tS + c * 8, pk);
        }
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars->ds_ready[X]);
      }
      mbar_wait(&bars->dq_done[X], outputs & 1, abort_flag);
      ok = __all_sync(0xffffffffu, *abort_flag == 0);
      ++outputs;
      tc_fence_after();
      if (ok) {
        constexpr int DHALF = D / 2;
        __nv_bfloat16* dqrow = dQ + ((long)b * T + qi) * lddq + (long)h * D + hf * DHALF;
#pragma unroll
        for (int c = 0; c < DHALF / 32; ++c) {
          uint32_t v[32];
          tmem_ld_32x32b_x32(tDQ + hf * DHALF + c * 32, v);
          tmem_ld_wait();
          uint4 out[4];
#pragma unroll
          for (int w = 0; w < 4; ++w)
            out[w] = make_uint4(pack_bf16(__uint_as_float(v[8 * w]), __uint_as_float(v[8 * w + 1])),
                                pack_bf16(__uint_as_float(v[8 * w + 2]), __uint_as_float(v[8 * w + 3])),
                                pack_bf16(__uint_as_float(v[8 * w + 4]), __uint_as_float(v[8 * w + 5])),
                                pack_bf16(__uint_as_float(v[8 * w + 6]), __uint_as_float(v[8 * w + 7])));
          store_rows<4>(out, dqrow + c * 32, lddq * 2, T - q0 - quad * 32, lane);
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && blockIdx.x == 0) wait_for_predecessor();
  if (threadIdx.x == 0 && bars->abort_flag && status) atomicExch(status, 4u);
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem, 512); }
}

// ------------------------------------------- backward: dK and dV, transposed scores
// One CTA owns 128 keys of one KV head and walks, head by head of the group and in ascending query order, the 128-row
// query steps that see those keys. The products are formed TRANSPOSED, S^T = K Q^T and dP^T = V dO^T (128 keys x 128
// queries), so a tensor-memory lane is a key: the threads of a key row write P^T and dS^T back over their own columns
// as bf16 pairs and both accumulations, dV += P^T dO and dK += dS^T Q, take their A operand straight from tensor memory.
// dV and dK accumulate over (head, query) in 16-query tensor-core steps, as the CPU twin does.
// Steps are 128 queries wide because a product of two shared-memory operands reads all of A whatever its width (128 x 64 takes 60
// clocks a k-step, 128 x 128 64). That leaves tensor memory for one S^T and one dP^T, and the overlap comes from the order: while
// the sixteen element warps (four threads per key row, no value crosses threads) turn dP^T into dS^T, the tensor core runs dV and
// the next S^T; while they make the next P^T, it runs dK and the next dP^T. Each 64-query half of P^T and dS^T is handed over by
// itself; the probabilities stay in registers (fp32) from the one phase to the other.
// A 128 x 128 step takes 3720 clocks of the whole launch: P^T 1800 (1250 of the multiply-add pipe), dS^T 750, 600 and 170 waiting for S^T and
// dP^T, and 400 between these and in the items' results. A step of which only the first half holds queries takes as long as a whole one:
// 40 x 64 tokens, 16 heads on 4 of 128, 46.5 us with 64-query steps, 50.9 so. (Leaving the padding's arithmetic out: 49.8 there, but 923 -> 954
// for 4 x 4096 tokens, 16 heads on 8.)
// 4 x 4096 tokens, 16 x 128 heads: 538 -> 533 us against 64-query steps with two score buffers (products alone 2900 clocks there);
// lengths that are no multiple of 64 had a kernel of their own: backward of 333 tokens, 12 x 64, 39.5 -> 25.1 us, 2 x 1000 55.3 -> 36.1.
// Also measured: two groups of eight warps, one per 64-query buffer (537 us); P^T through shared memory, so that S^T is free early
// (611: three products of four then take all of the shared-memory bandwidth).
// Per-query statistics (-lse, -delta) are copied to shared memory by the loading warp, plain loads, so any T will do: rows past
// the end have dO = 0 and -delta = 0 and add nothing.
// Tensor memory: dV 128 | dK 128 | S^T 128 | dP^T 128.
constexpr int KV_QST = 3, KV_DOST = 2;  // Q lives until its dK product, dO until its dV product

struct BarsKV3 {
  uint64_t k_full, k_empty, v_full, v_empty, q_full[KV_QST], q_empty[KV_QST], do_full[KV_DOST], do_empty[KV_DOST], stat_full[2], s_full, dp_full,
      p_ready[2], ds_ready[2], acc_full, acc_empty;
  uint32_t tmem_slot;
  uint32_t abort_flag;
};

// P^T of 16 queries of the thread's key (0 where hidden), kept as fp32 pairs and packed to bf16. One copy of the arithmetic for
// pieces with and without hidden pairs: with a copy of each for all four pieces the kernel outgrew the instruction cache (85 K
// misses an SM at 4 x 4096 tokens, 716 us instead of 533).
__device__ __forceinline__ void probs_t(const uint32_t (&vs)[16], const float* nl, float c_log2, bool mixed, int kj, int qbase, int window, f2 (&p)[8],
                                        uint32_t (&pk)[8]) {
  const f2 c2 = pack2(c_log2, c_log2);
#pragma unroll
  for (int e = 0; e < 16; e += 4) {
    const float4 l4 = *reinterpret_cast<const float4*>(nl + e);
    p[e >> 1] = exp2_attn2(fma2(pack2(__uint_as_float(vs[e]), __uint_as_float(vs[e + 1])), c2, pack2(l4.x, l4.y)));
    p[(e >> 1) + 1] = exp2_attn2(fma2(pack2(__uint_as_float(vs[e + 2]), __uint_as_float(vs[e + 3])), c2, pack2(l4.z, l4.w)));
  }
  if (mixed) {
    const uint32_t reach = window > 0 ? (uint32_t)window : 0x7FFFFFFFu;  // the queries kj .. kj + reach - 1 see the key
#pragma unroll
    for (int e = 0; e < 16; e += 2) {
      float p0, p1;
      unpack2(p[e >> 1], p0, p1);
      if ((uint32_t)(qbase + e - kj) >= reach) p0 = 0.0f;
      if ((uint32_t)(qbase + e + 1 - kj) >= reach) p1 = 0.0f;
      p[e >> 1] = pack2(p0, p1);
    }
  }
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    float p0, p1;
    unpack2(p[e], p0, p1);
    pk[e] = pack_bf16(p0, p1);
  }
}
// dS^T = (P (dP - delta)) scale of the same 16 queries
__device__ __forceinline__ void dscores_t(const uint32_t (&vd)[16], const float* nd, const f2 (&p)[8], float scale, uint32_t (&pk)[8]) {
  const f2 sc2 = pack2(scale, scale);
#pragma unroll
  for (int e = 0; e < 16; e += 4) {
    const float4 d4 = *reinterpret_cast<const float4*>(nd + e);
#pragma unroll
    for (int w = 0; w < 4; w += 2) {
      const f2 d2 = mul2(mul2(p[(e + w) >> 1], add2(pack2(__uint_as_float(vd[e + w]), __uint_as_float(vd[e + w + 1])), w ? pack2(d4.z, d4.w) : pack2(d4.x, d4.y))), sc2);
      float d0, d1;
      unpack2(d2, d0, d1);
      pk[(e + w) >> 1] = pack_bf16(d0, d1);
    }
  }
}

template <int D>
__global__ void __launch_bounds__(ATT_THREADS, 1)
attn_bwd_kv3_kernel(const __grid_constant__ CUtensorMap tmQK, const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDO,
                    const float* __restrict__ nlse, const float* __restrict__ ndelta, __nv_bfloat16* __restrict__ dK, long lddk,
                    __nv_bfloat16* __restrict__ dV, long lddv, int B, int T, int H, int Hkv, int window, float scale, float c_log2,
                    uint32_t* __restrict__ status) {
  constexpr int TILE = BKV * D * 2;
  constexpr int QST = KV_QST, DOST = KV_DOST;
  let_successor_begin();
  extern __shared__ __align__(1024) uint8_t smem_kv[];
  if (smem_u32(smem_kv) & 1023u) {  // no room to align by hand; the first byte that a kernel without static shared memory gets is aligned so
    if (threadIdx.x == 0 && status) atomicExch(status, 3u);
    return;
  }
  uint8_t* sK = smem_kv;
  uint8_t* sV = sK + TILE;
  uint8_t* sQ = sV + TILE;            // [QST]
  uint8_t* sDO = sQ + QST * TILE;     // [DOST]
  float* sStat = reinterpret_cast<float*>(sDO + DOST * TILE);  // [2][2][128]: -lse, -delta of the step's queries
  BarsKV3* bars = reinterpret_cast<BarsKV3*>(sStat + 4 * BQ);
  volatile uint32_t* abort_flag = &bars->abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int G = H / Hkv, nkb = (T + BKV - 1) / BKV, heads = B * Hkv;
  const int items = nkb * heads;
  // Item -> key block (the first ones are seen by the most queries), KV head, sequence; the 64-query halves that see it, counted
  // from its own position, and the 128-query steps per head (of the last one, only the first half where the count is odd)
  struct Item { int k0, g, b, halves, nqi, n; };
  auto item_of = [&](int w) {
    Item it;
    it.k0 = rotated(w / heads, nkb) * BKV;
    it.g = w % heads % Hkv;
    it.b = w % heads / Hkv;
    int last = (T - 1) / 64;
    if (window > 0) last = min(last, (it.k0 + BKV - 1 + window - 1) / 64);
    it.halves = last - it.k0 / 64 + 1;
    it.nqi = (it.halves + 1) / 2;
    it.n = G * it.nqi;
    return it;
  };

  if (threadIdx.x == 0) {
    mbar_init(&bars->k_full, 1); mbar_init(&bars->k_empty, 1); mbar_init(&bars->v_full, 1); mbar_init(&bars->v_empty, 1);
    for (int s = 0; s < QST; ++s) { mbar_init(&bars->q_full[s], 1); mbar_init(&bars->q_empty[s], 1); }
    for (int s = 0; s < DOST; ++s) { mbar_init(&bars->do_full[s], 1); mbar_init(&bars->do_empty[s], 1); }
    for (int s = 0; s < 2; ++s) { mbar_init(&bars->stat_full[s], 1); mbar_init(&bars->p_ready[s], SOFTMAX_WARPS); mbar_init(&bars->ds_ready[s], SOFTMAX_WARPS); }
    mbar_init(&bars->s_full, 1); mbar_init(&bars->dp_full, 1);
    mbar_init(&bars->acc_full, 1); mbar_init(&bars->acc_empty, SOFTMAX_WARPS);
    bars->abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) { tmem_alloc(&bars->tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = bars->tmem_slot;
  const uint32_t tDV = tmem, tDK = tmem + 128, tS = tmem + 256, tDP = tmem + 384;

  if (warp == 0) {
    uint32_t c = 0;  // query steps loaded so far
    bool ok = true;
    for (int turn = 0, w; ok && (w = work_item(turn)) < items; ++turn) {
      const Item it = item_of(w);
      int h = it.g * G, q0 = it.k0;
      for (int i = 0; ok && i < it.n; ++i, ++c) {
        const int qs = c % QST, os = c % DOST;
        float st[2][4];
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          const int q = q0 + x * 32 + lane;
          const long at = ((long)it.b * H + h) * T + q;
          st[0][x] = q < T ? nlse[at] : 0.0f;
          st[1][x] = q < T ? ndelta[at] : 0.0f;
        }
        if (lane == 0) {
          if (i == 0 && (ok = mbar_wait(&bars->k_empty, (turn & 1) ^ 1, abort_flag))) {
            mbar_expect_tx(&bars->k_full, TILE);
            load_tile<D>(sK, &tmQK, &bars->k_full, (H + it.g) * D, it.k0, it.b);
          }
          if (ok && (ok = mbar_wait(&bars->q_empty[qs], ((c / QST) & 1) ^ 1, abort_flag))) {
            mbar_expect_tx(&bars->q_full[qs], TILE);
            load_tile<D>(sQ + qs * TILE, &tmQK, &bars->q_full[qs], h * D, q0, it.b);
          }
          if (ok && i == 0 && (ok = mbar_wait(&bars->v_empty, (turn & 1) ^ 1, abort_flag))) {
            mbar_expect_tx(&bars->v_full, TILE);
            load_tile<D>(sV, &tmV, &bars->v_full, (H + Hkv + it.g) * D, it.k0, it.b);
          }
          if (ok && (ok = mbar_wait(&bars->do_empty[os], ((c / DOST) & 1) ^ 1, abort_flag))) {
            mbar_expect_tx(&bars->do_full[os], TILE);
            load_tile<D>(sDO + os * TILE, &tmDO, &bars->do_full[os], h * D, q0, it.b);
          }
          // the statistics of two steps ago have been read once that step's dK product is done
          if (ok && c >= 2) ok = mbar_wait(&bars->q_empty[(c - 2) % QST], ((c - 2) / QST) & 1, abort_flag);
        }
        ok = __shfl_sync(0xffffffffu, (int)ok, 0);
        if (!ok) break;
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          sStat[(c & 1) * 2 * BQ + x * 32 + lane] = st[0][x];
          sStat[(c & 1) * 2 * BQ + BQ + x * 32 + lane] = st[1][x];
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars->stat_full[c & 1]);
        if ((q0 += BQ) == it.k0 + it.nqi * BQ) {
          q0 = it.k0;
          ++h;
        }
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      constexpr uint32_t idS = make_idesc(128, BQ, 0, 0);  // S^T = K Q^T, dP^T = V dO^T
      constexpr uint32_t idG = make_idesc(128, D, 0, 1);   // dV = P^T dO, dK = dS^T Q: A in tensor memory, B MN-major
      const uint32_t aK = smem_u32(sK), aV = smem_u32(sV);
      // two walks over the same steps: the score products are one step ahead
      struct Walk { int turn = 0, i = 0, n = 0, q = 0, nqi = 0, halves = 0; uint32_t c = 0; } a, d;  // n = 0: past the last item
      auto begin = [&](Walk& x) {
        const int w = work_item(x.turn);
        x.i = x.n = x.q = x.nqi = x.halves = 0;
        if (w < items) {
          const Item it = item_of(w);
          x.n = it.n;
          x.nqi = it.nqi;
          x.halves = it.halves;
        }
      };
      auto next = [&](Walk& x) {
        ++x.c;
        if (++x.q == x.nqi) x.q = 0;
        if (++x.i == x.n) {
          ++x.turn;
          begin(x);
        }
      };
      // operands are waited for ahead of the hand-over that the product also needs
      auto S_ready = [&]() {
        return !(a.i == 0 && !mbar_wait(&bars->k_full, a.turn & 1, abort_flag)) && mbar_wait(&bars->q_full[a.c % QST], (a.c / QST) & 1, abort_flag);
      };
      auto dP_ready = [&]() {
        return !(a.i == 0 && !mbar_wait(&bars->v_full, a.turn & 1, abort_flag)) && mbar_wait(&bars->do_full[a.c % DOST], (a.c / DOST) & 1, abort_flag);
      };
      auto issue_S = [&]() {
        const uint32_t aQ = smem_u32(sQ + (a.c % QST) * TILE);
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) mma_f16_ss(tS, desc_k(aK, kk), desc_k(aQ, kk), idS, kk != 0);
        mma_commit(&bars->s_full);
        if (a.i == a.n - 1) mma_commit(&bars->k_empty);
      };
      auto issue_dP = [&]() {
        const uint32_t aDO = smem_u32(sDO + (a.c % DOST) * TILE);
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) mma_f16_ss(tDP, desc_k(aV, kk), desc_k(aDO, kk), idS, kk != 0);
        mma_commit(&bars->dp_full);
        if (a.i == a.n - 1) mma_commit(&bars->v_empty);
      };
      // one accumulation over the step's queries, half by half as the element warps hand them over
      auto accumulate = [&](uint32_t tAcc, uint32_t tA, uint32_t aB, uint64_t* ready) {
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          if (!mbar_wait(&ready[half], d.c & 1, abort_flag)) return false;
          tc_fence_after();
          if (half == 0 || 2 * d.q + 1 < d.halves) {
#pragma unroll
            for (int kk = half * 4; kk < half * 4 + 4; ++kk)
              mma_f16_ts(tAcc, tA + kk * 16, desc_mn(aB, kk), idG, (d.i | kk) != 0);
          }
        }
        return true;
      };
      begin(a);
      d = a;
      bool ok = true;
      for (bool first = true; ok && (first || d.n); first = false) {
        if (a.n && !(ok = S_ready())) break;
        if (!first) {
          if (d.i == 0 && !(ok = mbar_wait(&bars->acc_empty, (d.turn & 1) ^ 1, abort_flag))) break;  // the last item's results are read
          if (!(ok = accumulate(tDV, tS, smem_u32(sDO + (d.c % DOST) * TILE), bars->p_ready))) break;
        }
        if (a.n) issue_S();  // over the P^T just consumed
        if (!first) mma_commit(&bars->do_empty[d.c % DOST]);
        if (a.n && !(ok = dP_ready())) break;
        if (!first && !(ok = accumulate(tDK, tDP, smem_u32(sQ + (d.c % QST) * TILE), bars->ds_ready))) break;
        if (a.n) {
          issue_dP();
          next(a);
        }
        if (!first) {
          mma_commit(&bars->q_empty[d.c % QST]);
          if (d.i == d.n - 1) mma_commit(&bars->acc_full);
          next(d);
        }
      }
    }
  } else {
    const int quad = warp & 3;
    const int part = (warp - 2) >> 2;        // which 16 queries of a 64-query half, and which quarter of the result's columns
    const int r = quad * 32 + lane;          // key row == TMEM lane
    const uint32_t lane_off = (uint32_t(quad * 32) << 16) + part * 16;
    uint32_t c = 0;
    bool ok = true;
    for (int turn = 0, w; ok && (w = work_item(turn)) < items; ++turn) {
      const Item it = item_of(w);
      const int kj = it.k0 + r, klo = it.k0 + quad * 32;
      int step = 0;
      for (int i = 0; i < it.n && ok; ++i, ++c, step = step + 1 == it.nqi ? 0 : step + 1) {
        const int q0 = it.k0 + step * BQ + part * 16;
        const float* nl = sStat + (c & 1) * 2 * BQ + part * 16;
        const float* nd = nl + BQ;
        // two pieces of 16 queries, the second one's values in flight under the first one's arithmetic
        Seen sn[2];
        f2 p[2][8];
        uint32_t v[2][16], pk[8];
#pragma unroll
        for (int x = 0; x < 2; ++x) sn[x] = seen(klo, klo + 31, q0 + x * 64, q0 + x * 64 + 15, window);
        if (!mbar_wait_warp(&bars->stat_full[c & 1], (c >> 1) & 1, abort_flag) || !mbar_wait_warp(&bars->s_full, c & 1, abort_flag)) { ok = false; break; }
        tc_fence_after();
        tmem_ld_32x32b_x16(tS + lane_off, v[0]);
#pragma unroll
        for (int x = 0; x < 2; ++x) {
          tmem_ld_wait();
          if (x == 0) tmem_ld_32x32b_x16(tS + lane_off + 64, v[1]);
          if (sn[x] != HIDDEN) probs_t(v[x], nl + x * 64, c_log2, sn[x] == MIXED, kj, q0 + x * 64, window, p[x], pk);
          else {
#pragma unroll
            for (int e = 0; e < 8; ++e) pk[e] = 0u;
          }
          tmem_st_32x32b_x8(tS + lane_off + x * 64, pk);
          tmem_st_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&bars->p_ready[x]);
        }
        if (!mbar_wait_warp(&bars->dp_full, c & 1, abort_flag)) { ok = false; break; }
        tc_fence_after();
        tmem_ld_32x32b_x16(tDP + lane_off, v[0]);
        tmem_ld_32x32b_x16(tDP + lane_off + 64, v[1]);
        tmem_ld_wait();
#pragma unroll
        for (int x = 0; x < 2; ++x) {
          if (sn[x] != HIDDEN) dscores_t(v[x], nd + x * 64, p[x], scale, pk);
          else {
#pragma unroll
            for (int e = 0; e < 8; ++e) pk[e] = 0u;
          }
          tmem_st_32x32b_x8(tDP + lane_off + x * 64, pk);
          tmem_st_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&bars->ds_ready[x]);
        }
      }
      ok = ok && mbar_wait_warp(&bars->acc_full, turn & 1, abort_flag);
      if (!ok) break;
      tc_fence_after();
      constexpr int DH = D / NSPLIT;
      const long row = (long)it.b * T + kj;
#pragma unroll
      for (int which = 0; which < 2; ++which) {
        uint32_t v[DH];
        tmem_ld_cols<DH>((which ? tDK : tDV) + (uint32_t(quad * 32) << 16) + part * DH, v);
        tmem_ld_wait();
        if (which == 1) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&bars->acc_empty);
        }
        uint4 out[DH / 8];
#pragma unroll
        for (int x = 0; x < DH / 8; ++x)
          out[x] = make_uint4(pack_bf16(__uint_as_float(v[8 * x]), __uint_as_float(v[8 * x + 1])),
                              pack_bf16(__uint_as_float(v[8 * x + 2]), __uint_as_float(v[8 * x + 3])),
                              pack_bf16(__uint_as_float(v[8 * x + 4]), __uint_as_float(v[8 * x + 5])),
                              pack_bf16(__uint_as_float(v[8 * x + 6]), __uint_as_float(v[8 * x + 7])));
        store_rows<DH / 8>(out, (which ? dK + row * lddk : dV + row * lddv) + (long)it.g * D + part * DH, (which ? lddk : lddv) * 2, T - klo, lane);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && bars->abort_flag && status) atomicExch(status, 3u);
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem, 512); }
}

// delta[b,h,t] = sum_d dO[t,h,d] * O[t,h,d], lane_tree with VW = 4. The scratch has three [B, H, T] planes: delta, -lse and
// -delta (the negated copies feed the transposed dK/dV kernel's packed arithmetic). A warp takes DELTA_ROWS consecutive
// rows of one head: all of their loads (8 bytes per lane) are in flight together and the rows' results leave as whole
// 32-byte sectors. Memory-bound then (134 MB at 4 x 4096 rows, 16 heads x 128); one row per warp with 2-byte loads, two
// 64-bit divisions and 4-byte stores took 56 us there. VEC: both operands allow the 8-byte loads.
constexpr int DELTA_ROWS = 8;
template <bool VEC>
__global__ void __launch_bounds__(256) attn_delta_kernel(const __nv_bfloat16* __restrict__ dO, long lddo, const __nv_bfloat16* __restrict__ O,
                                  long ldo, const float* __restrict__ lse, float* __restrict__ delta, int B, int T, int H, int D) {
  const long wid = (long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  const long rows = (long)B * T, groups = (rows + DELTA_ROWS - 1) / DELTA_ROWS;
  if (wid >= groups * H) return;
  const long grp = (groups * H) >> 31 ? wid / H : (long)((unsigned)wid / (unsigned)H);  // heads vary fastest: neighbouring warps read one row
  const int h = (int)(wid - grp * H);
  const long row0 = grp * DELTA_ROWS;
  const int n = (int)min((long)DELTA_ROWS, rows - row0);
  const bool active = lane * 4 < D;
  const __nv_bfloat16* pa = dO + row0 * lddo + (long)h * D + lane * 4;
  const __nv_bfloat16* po = O + row0 * ldo + (long)h * D + lane * 4;
  uint2 a[DELTA_ROWS], o[DELTA_ROWS];
#pragma unroll
  for (int r = 0; r < DELTA_ROWS; ++r) {
    a[r] = o[r] = make_uint2(0u, 0u);
    if (active && r < n) {
      if (VEC) {
        a[r] = *reinterpret_cast<const uint2*>(pa + r * lddo);
        o[r] = *reinterpret_cast<const uint2*>(po + r * ldo);
      } else {
        const uint16_t* x = reinterpret_cast<const uint16_t*>(pa + r * lddo);
        const uint16_t* y = reinterpret_cast<const uint16_t*>(po + r * ldo);
        a[r] = make_uint2(x[0] | (uint32_t)x[1] << 16, x[2] | (uint32_t)x[3] << 16);
        o[r] = make_uint2(y[0] | (uint32_t)y[1] << 16, y[2] | (uint32_t)y[3] << 16);
      }
    }
  }
  float mine = 0.0f;
#pragma unroll
  for (int r = 0; r < DELTA_ROWS; ++r) {
    float acc = 0.0f;
    if (active) {
      acc = __fmaf_rn(__uint_as_float(a[r].x << 16), __uint_as_float(o[r].x << 16), acc);
      acc = __fmaf_rn(__uint_as_float(a[r].x & 0xFFFF0000u), __uint_as_float(o[r].x & 0xFFFF0000u), acc);
      acc = __fmaf_rn(__uint_as_float(a[r].y << 16), __uint_as_float(o[r].y << 16), acc);
      acc = __fmaf_rn(__uint_as_float(a[r].y & 0xFFFF0000u), __uint_as_float(o[r].y & 0xFFFF0000u), acc);
    }
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) acc = __fadd_rn(acc, __shfl_xor_sync(0xffffffffu, acc, off));
    if (lane == r) mine = acc;
  }
  if (lane < n) {
    const long row = row0 + lane, bb = row >> 31 ? row / T : (long)((unsigned)row / (unsigned)T), t = row - bb * T;
    const long idx = (bb * H + h) * T + t, plane = (long)B * H * T;
    delta[idx] = mine;
    delta[plane + idx] = -lse[idx];
    delta[2 * plane + idx] = -mine;
  }
}

// One CTA per (128-key block, KV head, batch): step = max(max|V| / 127, FLT_MIN) over the block, V_q = clamp(rint(V / step)).
template <int D>
__global__ void quant_v_kernel(const __nv_bfloat16* __restrict__ qkv, long ldqkv, int vcol0, int8_t* __restrict__ vq, long ldvq,
                               float* __restrict__ vstep, int T, int Hkv) {
  __shared__ float sh[32];
  const int blk = blockIdx.x, g = blockIdx.y, b = blockIdx.z;
  const int nblk = gridDim.x;
  const int k0 = blk * BKV;
  constexpr int VPR = D / 8;  // 16-byte vectors per row
  float m = 0.0f;
  for (int i = threadIdx.x; i < BKV * VPR; i += blockDim.x) {
    const int r = i / VPR, c = (i % VPR) * 8;
    if (k0 + r >= T) continue;
    const uint4 v = *reinterpret_cast<const uint4*>(qkv + ((long)b * T + k0 + r) * ldqkv + vcol0 + g * D + c);
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      m = fmaxf(m, fabsf(__uint_as_float(w[e] << 16)));
      m = fmaxf(m, fabsf(__uint_as_float(w[e] & 0xFFFF0000u)));
    }
  }
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, off));
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = m;
  __syncthreads();
  m = 0.0f;
  for (int w = 0; w < (int)(blockDim.x >> 5); ++w) m = fmaxf(m, sh[w]);
  const float step = fmaxf(__fmul_rn(m, 1.0f / 127.0f), 1.17549435e-38f);
  if (threadIdx.x == 0) vstep[((long)b * Hkv + g) * nblk + blk] = step;
  for (int i = threadIdx.x; i < BKV * VPR; i += blockDim.x) {
    const int r = i / VPR, c = (i % VPR) * 8;
    if (k0 + r >= T) continue;
    const uint4 v = *reinterpret_cast<const uint4*>(qkv + ((long)b * T + k0 + r) * ldqkv + vcol0 + g * D + c);
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    uint32_t o[2] = {0, 0};
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float f = (e & 1) ? __uint_as_float(w[e >> 1] & 0xFFFF0000u) : __uint_as_float(w[e >> 1] << 16);
      const int qv = (int)fminf(fmaxf(rintf(__fdiv_rn(f, step)), -127.0f), 127.0f);
      o[e >> 2] |= (uint32_t)(qv & 0xFF) << (8 * (e & 3));
    }
    *reinterpret_cast<uint2*>(vq + ((long)b * T + k0 + r) * ldvq + g * D + c) = make_uint2(o[0], o[1]);
  }
}

CUresult encode_3d_u8(CUtensorMap* out, const void* ptr, uint64_t cols, uint64_t T, uint64_t B, uint64_t ld_bytes) {
  static PFN_encodeTiled fn = get_encode_tiled();
  if (!fn) return CUDA_ERROR_NOT_SUPPORTED;
  cuuint64_t dims[3] = {cols, T, B};
  cuuint64_t strides[2] = {ld_bytes, T * ld_bytes};
  cuuint32_t box[3] = {128, 128, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  return otb_encode([&] {
    return fn(out, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  });
}

CUresult encode_3d(CUtensorMap* out, const void* ptr, uint64_t cols, uint64_t T, uint64_t B, uint64_t ld_elems, uint32_t box_rows = 128) {
  static PFN_encodeTiled fn = get_encode_tiled();
  if (!fn) return CUDA_ERROR_NOT_SUPPORTED;
  cuuint64_t dims[3] = {cols, T, B};
  cuuint64_t strides[2] = {ld_elems * 2, T * ld_elems * 2};
  cuuint32_t box[3] = {64, box_rows, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  return otb_encode([&] {
    return fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(ptr), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  });
}

constexpr int attn_fwd_i8pv_smem_bytes() { return (1 + 2 * 2) * (BQ * 128 * 2) + BQ * BKV * 2 + 1024 + 512 + 4096; }

template <int D> constexpr int attn_bwd_q2_smem_bytes() { return 4 * (BQ * D * 2) + 2 * 3 * (HK * D * 2) + 1024 + 256; }
template <int D> constexpr int attn_bwd_kv3_smem_bytes() { return (2 + KV_QST + KV_DOST) * (BKV * D * 2) + 4 * BQ * 4 + (int)sizeof(BarsKV3); }
template <int D> constexpr int attn_fwd2_smem_bytes() { return (2 + 2 * 2) * (BQ * D * 2) + 1024 + 256; }

}  // namespace

// qk: [B*T, ldqk] bf16 holding H query heads then Hkv key heads (width D each); qkv: [B*T, ldqkv] bf16 whose
// value heads start at column (H + Hkv) * D; O: [B*T, ldo]; lse: [B, H, T] fp32. D in {64, 128}.
// one CTA per SM, fewer when there are fewer items
static inline unsigned persistent_grid(long items) { return (unsigned)(items < otb_sm_count() ? items : otb_sm_count()); }

extern "C" int otb_set_attn_rotation(int rotation) {
  if (rotation < 0) return -2;
  return (int)cudaMemcpyToSymbol(g_attn_rotation, &rotation, sizeof(rotation));
}
extern "C" int otb_attn_fwd(const void* qk, long ldqk, const void* qkv, long ldqkv, void* O, long ldo, float* lse, int B,
                            int T, int H, int Hkv, int D, int window, float scale, uint32_t* status, void* stream) {
  if ((D != 64 && D != 128) || H % Hkv || (ldqk & 7) || (ldqkv & 7) || (ldo & 7)) return -2;
  CUtensorMap tq, tv;
  CUresult r = encode_3d(&tq, qk, (uint64_t)ldqk, (uint64_t)T, (uint64_t)B, (uint64_t)ldqk);
  if (r != CUDA_SUCCESS) return 1000 + (int)r;
  r = encode_3d(&tv, qkv, (uint64_t)ldqkv, (uint64_t)T, (uint64_t)B, (uint64_t)ldqkv);
  if (r != CUDA_SUCCESS) return 1000 + (int)r;
  const float c_log2 = (float)((double)scale * 1.4426950408889634);
  const int nq = (T + BQ - 1) / BQ;
  const unsigned grid = persistent_grid((long)((nq + 1) / 2) * H * B);
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  // Early where most of the chip is free anyway (us, ordinary and early: 12 CTAs 9.0 and 8.4, 24 13.9 and 13.4, 48 24.5 and 23.8, 64
  // 33.8 and 33.2, each heads x pairs of query tiles); with 128 and 148 CTAs it loses (56.6 and 58.0, 406 and 420, windowed 176 and 179).
  const bool early = 2 * (int)grid <= otb_sm_count();
  if (D == 128) {
    const int rc = otb_allow_smem<attn_fwd2_kernel<128>>(attn_fwd2_smem_bytes<128>());
    if (rc) return rc;
    return otb_launch_if_early(early, attn_fwd2_kernel<128>, grid, F2_THREADS, attn_fwd2_smem_bytes<128>(), s, tq, tv, (__nv_bfloat16*)O, ldo, lse, B, T,
                               H, Hkv, window, c_log2, status);
  } else {
    const int rc = otb_allow_smem<attn_fwd2_kernel<64>>(attn_fwd2_smem_bytes<64>());
    if (rc) return rc;
    return otb_launch_if_early(early, attn_fwd2_kernel<64>, grid, F2_THREADS, attn_fwd2_smem_bytes<64>(), s, tq, tv, (__nv_bfloat16*)O, ldo, lse, B, T,
                               H, Hkv, window, c_log2, status);
  }
}

// Forward with P V on the int8 tensor cores (head_dim 128 only). vq: int8 scratch [B*T, Hkv*D]; vstep: fp32 scratch
// [B, Hkv, ceil(T/128)]; both are written here (the per-block value quantisation) and read by the attention kernel.
extern "C" int otb_attn_fwd_i8pv(const void* qk, long ldqk, const void* qkv, long ldqkv, void* O, long ldo, float* lse, void* vq,
                                 float* vstep, int B, int T, int H, int Hkv, int D, int window, float scale, uint32_t* status,
                                 void* stream) {
  if (D != 128 || H % Hkv || (ldqk & 7) || (ldqkv & 7) || (ldo & 7)) return -2;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  const int nblk = (T + BKV - 1) / BKV;
  const long ldvq = (long)Hkv * D;
  quant_v_kernel<128><<<dim3(nblk, Hkv, B), 256, 0, s>>>((const __nv_bfloat16*)qkv, ldqkv, (H + Hkv) * D, (int8_t*)vq, ldvq, vstep, T, Hkv);
  CUtensorMap tq, tv;
  CUresult r = encode_3d(&tq, qk, (uint64_t)ldqk, (uint64_t)T, (uint64_t)B, (uint64_t)ldqk);
  if (r != CUDA_SUCCESS) return 1000 + (int)r;
  r = encode_3d_u8(&tv, vq, (uint64_t)ldvq, (uint64_t)T, (uint64_t)B, (uint64_t)ldvq);
  if (r != CUDA_SUCCESS) return 1000 + (int)r;
  const float c_log2 = (float)((double)scale * 1.4426950408889634);
  dim3 grid((T + BQ - 1) / BQ, H, B);
  const int rc = otb_allow_smem<attn_fwd_i8pv_kernel>(attn_fwd_i8pv_smem_bytes());
  if (rc) return rc;
  attn_fwd_i8pv_kernel<<<grid, ATT_THREADS, attn_fwd_i8pv_smem_bytes(), s>>>(tq, tv, (__nv_bfloat16*)O, ldo, lse, T, H, Hkv, window, c_log2, vstep,
                                                                             status);
  return (int)cudaGetLastError();
}

// dO, O: [B*T, ld] bf16 (head h at column h*D). Outputs: dqk [B*T, lddqk] (dQ heads then dK heads),
// dV written at column (H + Hkv) * D of dqkv [B*T, lddqkv]; delta: [3, B, H, T] fp32 scratch (delta, -lse, -delta).
extern "C" int otb_attn_bwd(const void* qk, long ldqk, const void* qkv, long ldqkv, const void* O, long ldo,
                            const void* dO, long lddo, const float* lse, float* delta, void* dqk, long lddqk, void* dqkv,
                            long lddqkv, int B, int T, int H, int Hkv, int D, int window, float scale, uint32_t* status,
                            void* stream) {
  if ((D != 64 && D != 128) || H % Hkv || (ldqk & 7) || (ldqkv & 7) || (ldo & 7) || (lddo & 7) || (lddqk & 7) ||
      (lddqkv & 7))
    return -2;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  const float c_log2 = (float)((double)scale * 1.4426950408889634);
  CUtensorMap tq, tv, tdo;
  CUresult r = encode_3d(&tq, qk, (uint64_t)ldqk, (uint64_t)T, (uint64_t)B, (uint64_t)ldqk);
  if (r != CUDA_SUCCESS) return 1000 + (int)r;
  r = encode_3d(&tv, qkv, (uint64_t)ldqkv, (uint64_t)T, (uint64_t)B, (uint64_t)ldqkv);
  if (r != CUDA_SUCCESS) return 1000 + (int)r;
  r = encode_3d(&tdo, dO, (uint64_t)lddo, (uint64_t)T, (uint64_t)B, (uint64_t)lddo);
  if (r != CUDA_SUCCESS) return 1000 + (int)r;
  const long warps = ((long)B * T + DELTA_ROWS - 1) / DELTA_ROWS * H;
  const bool vec = ((reinterpret_cast<uintptr_t>(O) | reinterpret_cast<uintptr_t>(dO)) & 7) == 0;  // pitches are multiples of 8 elements
  auto delta_kernel = vec ? attn_delta_kernel<true> : attn_delta_kernel<false>;
  if (const int rc = otb_launch(delta_kernel, (unsigned)((warps + 7) / 8), 256, 0, s, (const __nv_bfloat16*)dO, lddo, (const __nv_bfloat16*)O, ldo, lse,
                               delta, B, T, H, D))
    return rc;
  __nv_bfloat16* dQp = (__nv_bfloat16*)dqk;
  __nv_bfloat16* dKp = dQp + (long)H * D;
  __nv_bfloat16* dVp = (__nv_bfloat16*)dqkv + (long)(H + Hkv) * D;
  CUtensorMap tk64, tv64;
  r = encode_3d(&tk64, qk, (uint64_t)ldqk, (uint64_t)T, (uint64_t)B, (uint64_t)ldqk, HK);
  if (r != CUDA_SUCCESS) return 1000 + (int)r;
  r = encode_3d(&tv64, qkv, (uint64_t)ldqkv, (uint64_t)T, (uint64_t)B, (uint64_t)ldqkv, HK);
  if (r != CUDA_SUCCESS) return 1000 + (int)r;
  const int nq = (T + BQ - 1) / BQ;
  const int nkb = (T + BKV - 1) / BKV;
  const unsigned gq = persistent_grid((long)((nq + 1) / 2) * H * B), gkv = persistent_grid((long)nkb * Hkv * B);
  // dQ runs beside dK/dV: its CTAs start on the SMs that the latter leaves free, or as its CTAs end (backward, us, one after the
  // other and so: 2 x 1000 tokens, 12 heads x 64, window 512 83 and 56; 1 x 2048, 16 x 128 198 and 141; 4 x 4096 1018 and 976).
  const long plane = (long)B * H * T;
  if (D == 128) {
    const int rc = otb_allow_smem<attn_bwd_kv3_kernel<128>>(attn_bwd_kv3_smem_bytes<128>()) | otb_allow_smem<attn_bwd_q2_kernel<128>>(attn_bwd_q2_smem_bytes<128>());
    if (rc) return rc;
    const int kv = otb_launch(attn_bwd_kv3_kernel<128>, gkv, ATT_THREADS, attn_bwd_kv3_smem_bytes<128>(), s, tq, tv, tdo, delta + plane, delta + 2 * plane, dKp,
                              lddqk, dVp, lddqkv, B, T, H, Hkv, window, scale, c_log2, status);
    if (kv) return kv;
    return otb_launch_early(attn_bwd_q2_kernel<128>, gq, ATT_THREADS, attn_bwd_q2_smem_bytes<128>(), s, tq, tdo, tk64, tv64, lse, delta, dQp, lddqk, B, T,
                            H, Hkv, window, scale, c_log2, status);
  } else {
    const int rc = otb_allow_smem<attn_bwd_kv3_kernel<64>>(attn_bwd_kv3_smem_bytes<64>()) | otb_allow_smem<attn_bwd_q2_kernel<64>>(attn_bwd_q2_smem_bytes<64>());
    if (rc) return rc;
    const int kv = otb_launch(attn_bwd_kv3_kernel<64>, gkv, ATT_THREADS, attn_bwd_kv3_smem_bytes<64>(), s, tq, tv, tdo, delta + plane, delta + 2 * plane, dKp,
                              lddqk, dVp, lddqkv, B, T, H, Hkv, window, scale, c_log2, status);
    if (kv) return kv;
    return otb_launch_early(attn_bwd_q2_kernel<64>, gq, ATT_THREADS, attn_bwd_q2_smem_bytes<64>(), s, tq, tdo, tk64, tv64, lse, delta, dQp, lddqk, B, T,
                            H, Hkv, window, scale, c_log2, status);
  }
}

OTB_PACKED(otb_attn_fwd)
OTB_PACKED(otb_attn_bwd)
OTB_PACKED(otb_attn_fwd_i8pv)
