// One decoder block without gradients as one host call: the nine launches of norm -> QKV product -> QK-norm / RoPE ->
// attention -> output product (+ residual) -> norm -> gate/up product -> SwiGLU -> down product (+ residual), each the kernel
// that the block's modules launch one by one, so the results are the same bits. What bounds the scoring of a short prompt is
// the host: module calls and autograd functions, about 250 us of Python a block for 50 us of kernels (333 tokens through the
// six-layer 100M model: 1584 -> 542 us, the launches' own changes included; 440 with the model's walk in train() and a table of scratch sizes).
#include "common.cuh"
#include "entries.cuh"

namespace {
constexpr long SCRATCH_ALIGN = 256;
inline long up(long bytes) { return (bytes + SCRATCH_ALIGN - 1) / SCRATCH_ALIGN * SCRATCH_ALIGN; }
// Byte offsets in the scratch buffer. The attention's buffers and the feed-forward's share their room: the former are read
// for the last time by the output product.
struct BlockScratch {
  long norm, rstd, mid, qkv, qk, o, lse, gu, act, total;
  BlockScratch(long rows, int d, int H, int Hkv, int D, int F, int e) {
    const long heads = H + Hkv;
    norm = 0;
    rstd = norm + up(rows * d * e);
    mid = rstd + up(rows * heads * 4);
    qkv = mid + up(rows * d * e);
    qk = qkv + up(rows * (heads + Hkv) * D * e);
    o = qk + up(rows * heads * D * e);
    lse = o + up(rows * H * D * e);
    const long attn_end = lse + up(rows * H * 4);
    gu = qkv;
    act = gu + up(rows * 2 * F * e);
    const long ffn_end = act + up(rows * F * e);
    total = attn_end > ffn_end ? attn_end : ffn_end;
  }
};
}  // namespace

extern "C" long otb_block_fwd_scratch(long rows, int d, int H, int Hkv, int D, int F, int bf16) {
  return BlockScratch(rows, d, H, Hkv, D, F, bf16 ? 2 : 4).total;
}

// x, y: [B*T, d]; w*: weights in the activations' type, row-major [out, in]; scratch: otb_block_fwd_scratch bytes, 256-byte
// aligned. Returns the first launch's error, if any. Never allocates, never synchronises.
extern "C" int otb_block_fwd(const void* x, void* y, void* scratch, const void* norm1, const void* wqkv, const void* wo, const void* norm2,
                             const void* wgu, const void* wdown, const float* cosb, const float* sinb, int B, int T, int d, int H, int Hkv,
                             int D, int F, int window, int qk_norm, float eps1, float eps2, float eps_qk, float scale, int bf16,
                             uint32_t* status, void* stream) {
  const long rows = (long)B * T;
  const BlockScratch s(rows, d, H, Hkv, D, F, bf16 ? 2 : 4);
  char* base = static_cast<char*>(scratch);
  void *h = base + s.norm, *mid = base + s.mid, *qkv = base + s.qkv, *qk = base + s.qk, *o = base + s.o, *gu = base + s.gu, *act = base + s.act;
  float *rstd = reinterpret_cast<float*>(base + s.rstd), *lse = reinterpret_cast<float*>(base + s.lse);
  const int heads = H + Hkv, nqkv = (heads + Hkv) * D;
  const float inv_d = (float)(1.0 / d);
  auto product = [&](const void* a, const void* w, void* c, const void* r, int N, int K) {
    const int epi = r ? 3 : 0;
    const long ldr = r ? N : 0;
    if (bf16) return otb_gemm_bf16(a, w, c, r, (int)rows, N, K, K, K, N, ldr, 0, 0, epi, status, 0, stream);
    return otb_gemm_f32((const float*)a, (const float*)w, (float*)c, (const float*)r, (int)rows, N, K, K, K, N, ldr, 0, 0, epi, stream);
  };
  int rc = otb_rmsnorm_fwd(x, norm1, h, rstd, rows, d, inv_d, eps1, bf16, stream);
  if (!rc) rc = product(h, wqkv, qkv, nullptr, nqkv, d);
  if (!rc) rc = otb_qknorm_rope_fwd(qkv, nqkv, qk, (long)heads * D, rstd, cosb, sinb, rows, heads, D, T, qk_norm, (float)(1.0 / D), eps_qk, bf16, stream);
  if (!rc)
    rc = bf16 ? otb_attn_fwd(qk, (long)heads * D, qkv, nqkv, o, (long)H * D, lse, B, T, H, Hkv, D, window, scale, status, stream)
              : otb_attn_f32_fwd((const float*)qk, (long)heads * D, (const float*)qkv, nqkv, (float*)o, (long)H * D, lse, B, T, H, Hkv, D, window,
                                 scale, stream);
  if (!rc) rc = product(o, wo, mid, x, d, H * D);
  if (!rc) rc = otb_rmsnorm_fwd(mid, norm2, h, rstd, rows, d, inv_d, eps2, bf16, stream);
  if (!rc) rc = product(h, wgu, gu, nullptr, 2 * F, d);
  if (!rc) rc = otb_swiglu_fwd(gu, act, rows, F, bf16, stream);
  if (!rc) rc = product(act, wdown, y, mid, d, F);
  return rc;
}
OTB_PACKED(otb_block_fwd)
