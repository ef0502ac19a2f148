// One pre-norm decoder block, forward in one call and backward in two: the launches that ops.rms_norm, linear, rope_qkv, flash_attention_packed
// and swiglu make one by one, in the same order, over buffers that are laid out here.
//
// What bounds a training step of a small model is the host: a block is 9 launches forward and 17 backward, and issuing each through Python,
// autograd and ctypes took 29 us of host time, where the GPU worked 2 - 10 (4 layers of width 256, 4 x 128 tokens: 4.2 ms a step, 0.65 of them
// kernels). From here: 1.59 ms.
#include "common.cuh"

#include <algorithm>

TSB_EXPORT int tsb_rmsnorm_fwd(const void* x, const void* res, const void* w, void* y, void* h_out, float* rstd, int rows, int D, float eps,
                               int dtype, void* stream);
TSB_EXPORT int tsb_rmsnorm_bwd_parts(int rows);
TSB_EXPORT int tsb_rmsnorm_bwd(const void* dy, const void* x, const void* w, const float* rstd, const void* dres, void* dx, void* dw,
                               float* partial, int rows, int D, int accumulate_dw, int dtype, void* stream);
TSB_EXPORT int tsb_swiglu_fwd(const void* gate_up, void* out, long long rows, int F, int dtype, void* stream);
TSB_EXPORT int tsb_swiglu_bwd_rows(const void* dout, long long ld_dout, const void* gate_up, void* dgate_up, long long rows, int F, int dtype,
                                   void* stream);
TSB_EXPORT int tsb_rope_qkv(void* qkv, const float* cos_t, const float* sin_t, const int* pos, long long tokens, int seq_len, int pos_offset,
                            int heads_rot, int heads_total, int D, float sign, int dtype, void* stream);
TSB_EXPORT int tsb_flash_fwd(const void* q, const void* k, const void* v, void* o, float* lse, int B, int Sq, int Sk, int H, int Hkv, int D,
                             long long q_sb, long long q_ss, long long q_sh, long long k_sb, long long k_ss, long long k_sh, long long v_sb,
                             long long v_ss, long long v_sh, long long o_sb, long long o_ss, long long o_sh, float scale, int causal,
                             void* stream);
TSB_EXPORT long long tsb_flash_bwd_scratch_bytes(int B, int Sq, int H, int D);
TSB_EXPORT int tsb_flash_bwd(const void* dO, const void* q, const void* k, const void* v, const void* o, const float* lse, void* dq, void* dk,
                             void* dv, void* scratch, int B, int Sq, int Sk, int H, int Hkv, int D, long long q_sb, long long q_ss,
                             long long q_sh, long long k_sb, long long k_ss, long long k_sh, long long v_sb, long long v_ss, long long v_sh,
                             long long g_sb, long long g_ss, long long g_sh, float scale, int causal, void* stream);
TSB_EXPORT int tsb_gemm_bf16(const void* A, const void* B, void* C, int M, int N, int K, long long lda, long long ldb, long long ldc, int a_mn,
                             int b_mn, int out_f32, int accumulate, int block_n, int max_ctas, void* stream);

namespace tsb {
namespace {

constexpr int kBf16 = 1;        // dtype code of the entry points above

struct BlockShape {
  int B, S, W, H, Hkv, D, F;
  long long rows() const { return static_cast<long long>(B) * S; }
  long long packed() const { return static_cast<long long>(H + 2 * Hkv) * D; }
  bool ok() const {
    return B > 0 && S > 0 && W > 0 && H > 0 && Hkv > 0 && F > 0 && H % Hkv == 0 && (D == 64 || D == 128) && W == H * D && W <= 8192 &&
           F % 8 == 0 && rows() < (1 << 30);
  }
};

// Pieces of one allocation, each from a multiple of 256 bytes on.
struct Cut {
  uint8_t* base;
  long long at = 0;
  uint8_t* take(long long bytes) {
    uint8_t* p = base + at;
    at += (bytes + 255) / 256 * 256;
    return p;
  }
};

// What the forward pass leaves for the backward pass, in two pieces: the second is done with halfway and given back then.
struct Saved {
  uint8_t *h1, *res1, *qkv, *o, *h2, *gu, *act;
  float *rstd1, *rstd2, *lse;
  long long bytes, mid_bytes;
  Saved(const BlockShape& s, void* base, void* mid, bool has_res) {
    Cut c{static_cast<uint8_t*>(base)}, m{static_cast<uint8_t*>(mid)};
    const long long T = s.rows();
    h1 = c.take(T * s.W * 2);
    res1 = has_res ? c.take(T * s.W * 2) : nullptr;
    qkv = c.take(T * s.packed() * 2);
    o = c.take(T * s.W * 2);
    h2 = c.take(T * s.W * 2);
    gu = m.take(T * 2 * s.F * 2);
    act = m.take(T * s.F * 2);
    rstd1 = reinterpret_cast<float*>(c.take(T * 4));
    rstd2 = reinterpret_cast<float*>(c.take(T * 4));
    lse = reinterpret_cast<float*>(c.take(T * s.H * 4));
    bytes = c.at;
    mid_bytes = m.at;
  }
};

// What the backward pass needs meanwhile, in two pieces. No more is held at any time than the modules hold one by one (16384 tokens, width 4096,
// 14336 between: 6.9 GB a step over the weights, where one piece for all and a buffer for each gradient took 7.6):
//   wide   the gradient of gate and up, in which that of the activation is formed first (in the columns of gate, which SwiGLU's backward pass
//          reads and writes in place); then what attention adds dQ up in; then the gradient of norm_1's output.
//   rest   the gradient of the stream between the halves, of q / k / v, and the norms' sums. Taken when `mid` has been given back.
// The gradients of norm_2's output and of attention's lie in dx, which is filled last.
struct Work {
  uint8_t *wide, *da, *dqkv;
  float* partial;
  long long wide_bytes, rest_bytes;
  Work(const BlockShape& s, void* wide_base, void* rest_base) {
    Cut c{static_cast<uint8_t*>(rest_base)};
    const long long T = s.rows();
    wide = static_cast<uint8_t*>(wide_base);
    wide_bytes = std::max({T * 2 * s.F * 2, T * s.W * 2, tsb_flash_bwd_scratch_bytes(s.B, s.S, s.H, s.D)});
    da = c.take(T * s.W * 2);
    dqkv = c.take(T * s.packed() * 2);
    partial = reinterpret_cast<float*>(c.take(static_cast<long long>(tsb_rmsnorm_bwd_parts(static_cast<int>(T))) * s.W * 4));
    rest_bytes = c.at;
  }
};

BlockShape shape_of(const long long* a) {
  return {static_cast<int>(a[0]), static_cast<int>(a[1]), static_cast<int>(a[2]), static_cast<int>(a[3]),
          static_cast<int>(a[4]), static_cast<int>(a[5]), static_cast<int>(a[6])};
}
template <typename T = void>
T* ptr(long long v) { return reinterpret_cast<T*>(v); }

}  // namespace
}  // namespace tsb

// Host arrays. shape: B, S, W, H, Hkv, D, F (W = H * D; D 64 or 128; F a multiple of 8).
// bytes: what a forward call keeps in `saved` and in `mid`, what a backward call needs in `wide` and in `rest`. -2 for other shapes.
TSB_EXPORT int tsb_block_bytes(const long long* shape, int has_res, long long* bytes) {
  using namespace tsb;
  const BlockShape s = shape_of(shape);
  if (!s.ok()) return -2;
  const Saved k(s, nullptr, nullptr, has_res != 0);
  const Work w(s, nullptr, nullptr);
  bytes[0] = k.bytes;
  bytes[1] = k.mid_bytes;
  bytes[2] = w.wide_bytes;
  bytes[3] = w.rest_bytes;
  return 0;
}

// out = down(silu(gate) * up) of the normed stream; res2 = x [+ res] + o_proj(attention). All bf16, contiguous, 16-byte aligned.
// p: x, res (0: none), norm_1, qkv weight, o weight, norm_2, gate and up weight, down weight, cos, sin, saved, mid, res2, out.
// f: eps of norm_1, eps of norm_2, softmax scale. Rows of weights are stacked (q, k, v; gate, up).
TSB_EXPORT int tsb_block_forward(const long long* shape, const long long* p, const float* f, int causal, void* stream) {
  using namespace tsb;
  const BlockShape s = shape_of(shape);
  if (!s.ok()) return -2;
  const Saved k(s, ptr(p[10]), ptr(p[11]), p[1] != 0);
  const int T = static_cast<int>(s.rows()), N = static_cast<int>(s.packed()), W = s.W, F = s.F, D = s.D;
  const long long row = N, seq = static_cast<long long>(s.S) * N, hd = static_cast<long long>(s.H) * D, vd = hd + static_cast<long long>(s.Hkv) * D;
  void *res2 = ptr(p[12]), *out = ptr(p[13]);
  auto product = [&](const void* x, long long w, void* y, int cols, int depth) {
    return tsb_gemm_bf16(x, ptr(w), y, T, cols, depth, depth, depth, cols, 0, 0, 0, 0, 0, 0, stream);
  };
  int rc = tsb_rmsnorm_fwd(ptr(p[0]), ptr(p[1]), ptr(p[2]), k.h1, k.res1, k.rstd1, T, W, f[0], kBf16, stream);
  if (rc) return rc;
  if ((rc = product(k.h1, p[3], k.qkv, N, W))) return rc;
  rc = tsb_rope_qkv(k.qkv, ptr<float>(p[8]), ptr<float>(p[9]), nullptr, T, s.S, 0, s.H + s.Hkv, s.H + 2 * s.Hkv, D, 1.f, kBf16, stream);
  if (rc) return rc;
  rc = tsb_flash_fwd(k.qkv, k.qkv + hd * 2, k.qkv + vd * 2, k.o, k.lse, s.B, s.S, s.S, s.H, s.Hkv, D, seq, row, D, seq, row, D, seq, row, D,
                     static_cast<long long>(s.S) * W, W, D, f[2], causal, stream);
  if (rc) return rc;
  // (the output of o_proj waits in `out`, which the down projection fills last)
  if ((rc = product(k.o, p[4], out, W, W))) return rc;
  rc = tsb_rmsnorm_fwd(out, p[1] ? k.res1 : ptr(p[0]), ptr(p[5]), k.h2, res2, k.rstd2, T, W, f[1], kBf16, stream);
  if (rc) return rc;
  if ((rc = product(k.h2, p[6], k.gu, 2 * F, W))) return rc;
  if ((rc = tsb_swiglu_fwd(k.gu, k.act, T, F, kBf16, stream))) return rc;
  return product(k.act, p[7], out, W, F);
}

// Gradients of the above, in two parts: 1, from the block's output to gate and up, after which what `mid` holds is not needed, then 2, the rest.
// p: x (where there was no res; else unused), norm_1, qkv, o, norm_2, gate and up, down (weights), cos, sin, saved, mid, res2, gradients of norm_1, qkv, o,
// norm_2, gate and up, down (added to; bf16), dout, dres2 (0: none), wide (kept between the parts), rest, dx (of x and of res). Part 1 touches
// neither rest nor dx, part 2 neither mid nor dout. f: as forward.
TSB_EXPORT int tsb_block_backward(const long long* shape, const long long* p, const float* f, int has_res, int causal, int part, void* stream) {
  using namespace tsb;
  const BlockShape s = shape_of(shape);
  if (!s.ok() || (part != 1 && part != 2)) return -2;
  const Saved k(s, ptr(p[9]), ptr(p[10]), has_res != 0);
  const Work w(s, ptr(p[20]), ptr(p[21]));
  const int T = static_cast<int>(s.rows()), N = static_cast<int>(s.packed()), W = s.W, F = s.F, D = s.D;
  auto input = [&](const void* dy, long long weight, void* d, int outs, int ins, long long ldd) {         // d = dy W
    return tsb_gemm_bf16(dy, ptr(weight), d, T, ins, outs, outs, ins, ldd, 0, 1, 0, 0, 0, 0, stream);
  };
  auto weight = [&](const void* dy, const void* x, long long d, int outs, int ins) {                      // dW += dy^T x
    return tsb_gemm_bf16(dy, x, ptr(d), outs, ins, T, outs, ins, ins, 1, 1, 0, 1, 0, 0, stream);
  };
  int rc = 0;
  if (part == 1) {
    const void* dout = ptr(p[18]);
    if ((rc = input(dout, p[6], w.wide, W, F, 2LL * F))) return rc;
    if ((rc = weight(dout, k.act, p[17], W, F))) return rc;
    return tsb_swiglu_bwd_rows(w.wide, 2LL * F, k.gu, w.wide, T, F, kBf16, stream);
  }
  const long long row = N, seq = static_cast<long long>(s.S) * N, hd = static_cast<long long>(s.H) * D, vd = hd + static_cast<long long>(s.Hkv) * D;
  void *dx = ptr(p[22]), *dh2 = dx, *d_o = dx, *dh1 = w.wide;
  if ((rc = input(w.wide, p[5], dh2, 2 * F, W, W))) return rc;
  if ((rc = weight(w.wide, k.h2, p[16], 2 * F, W))) return rc;
  if ((rc = tsb_rmsnorm_bwd(dh2, ptr(p[11]), ptr(p[4]), k.rstd2, ptr(p[19]), w.da, ptr(p[15]), w.partial, T, W, 1, kBf16, stream))) return rc;
  if ((rc = input(w.da, p[3], d_o, W, W, W))) return rc;
  if ((rc = weight(w.da, k.o, p[14], W, W))) return rc;
  rc = tsb_flash_bwd(d_o, k.qkv, k.qkv + hd * 2, k.qkv + vd * 2, k.o, k.lse, w.dqkv, w.dqkv + hd * 2, w.dqkv + vd * 2, w.wide, s.B, s.S, s.S,
                     s.H, s.Hkv, D, seq, row, D, seq, row, D, seq, row, D, seq, row, D, f[2], causal, stream);
  if (rc) return rc;
  rc = tsb_rope_qkv(w.dqkv, ptr<float>(p[7]), ptr<float>(p[8]), nullptr, T, s.S, 0, s.H + s.Hkv, s.H + 2 * s.Hkv, D, -1.f, kBf16, stream);
  if (rc) return rc;
  if ((rc = input(w.dqkv, p[2], dh1, N, W, W))) return rc;
  if ((rc = weight(w.dqkv, k.h1, p[13], N, W))) return rc;
  return tsb_rmsnorm_bwd(dh1, has_res ? k.res1 : ptr(p[0]), ptr(p[1]), k.rstd1, w.da, dx, ptr(p[12]), w.partial, T, W, 1, kBf16, stream);
}
