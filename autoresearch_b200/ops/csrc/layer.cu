// A transformer layer per call: the launch sequences of the forward and the backward pass of a dense layer that is not
// tensor-parallel, and of what precedes the experts of an expert layer.  Host code only.  The kernels are those that the separate
// entry points start, in the same order and on the same operands, with one exception: the weight gradients of a small layer
// (group_dw) leave in one launch at the end of the backward pass (gemm_sm100.cu), whose K splits add up in another order.
//
// Why: a dense layer is 7 launches forward (8 with the rotation as its own kernel) and 13 backward (15 with a value embedding; three
// fewer with grouped weight gradients).  Through one Python call and one autograd node per kernel a launch cost 25 us of host
// time, four times what a kernel of a small batch runs.  Measured, per step -> per layer (ungrouped): training pass of the 119.5 M model on one sequence of
// 2048 15.4 -> 8.6 ms (GPU work 7.4); small model, 512 tokens scored 0.95 -> 0.46 ms, 1024 tokens trained 2.70 -> 1.32 ms.
//
// Math and order: brain/src/forward.rs:359-739, brain/src/backward.rs:203-877.
#include "api.h"

namespace {

// The activations that a layer keeps, carved out of one buffer (bf16 [N, cols] each, then the fp32 row statistics).
// N * D is a multiple of 128 elements, so every bf16 part starts on a 256-byte boundary; the statistics are padded to four
// floats each, because the kernels read them as pairs.  The layer's input after scaling, xs, is read by the output projection and by
// nothing later (the backward pass forms it again from x and x0): it lies where an output of the call is written last.
struct Kept {
  char *xs, *xn, *qkv, *att, *xs2, *xn2, *act;
  float *lse, *rstd, *gate;
  explicit Kept(const ArbLayer& a) {
    const long long N = a.B * a.T, D = a.H * 128;
    char* p = static_cast<char*>(a.kept);
    auto take = [&](long long cols) { char* q = p; p += N * cols * 2; return q; };
    xs = static_cast<char*>(a.half ? a.out2 : a.out);
    if (a.scoring) {
      // no backward pass follows: q|k|v 3 D, xn D and, over it when the projection has read it, the attention's output; what comes
      // behind the attention lies over what is dead by then
      qkv = take(3 * D); xn = att = take(D);
      xs2 = qkv; xn2 = xs2 + N * D * 2; act = xn2 + N * D * 2;
    } else {
      xn = take(D); qkv = take(3 * D); att = take(D);
      xs2 = take(a.half ? 0 : D); xn2 = take(a.half ? 0 : D); act = take(a.half ? 0 : a.M);
    }
    const long long nh = (N * a.H + 3) / 4 * 4;
    lse = reinterpret_cast<float*>(p); rstd = lse + nh; gate = rstd + 2 * nh;
  }
};

// C[M, N] = A[M, K] op B, all dense; transposed operands as in arb_gemm_bf16
struct Gemm {
  int* err;
  cudaStream_t s;
  int nt(const void* a, const void* w, void* c, const void* aux, long long m, long long n, long long k, int epi) const {
    return arb_gemm_bf16(a, w, c, aux, int(m), int(n), int(k), 1, k, k, n, 0, 0, 0, 0, 0, epi, 0, 0.f, 0.f, 1.f, err, s);
  }
  int nn(const void* a, const void* w, void* c, const void* aux, long long m, long long n, long long k, int epi) const {
    return arb_gemm_bf16(a, w, c, aux, int(m), int(n), int(k), 1, k, n, n, 0, 0, 0, 0, 1, epi, 0, 0.f, 0.f, 1.f, err, s);
  }
  int dw(const void* dy, const void* x, void* w_grad, long long m, long long n, long long rows) const {
    return arb_gemm_bf16(dy, x, w_grad, nullptr, int(m), int(n), int(rows), 1, m, n, n, 0, 0, 0, 1, 1, EPI_ATOMIC_F32, 0, 0.f, 0.f,
                         1.f, err, s);
  }
};

bool bad_sizes(const ArbLayer& a) {
  return a.B <= 0 || a.T <= 0 || a.H <= 0 || (a.half ? a.M != 0 : a.M <= 0) || (a.M & 7) || a.B * a.T > 0x7fffffffll || a.H > 65535 || a.M > 0x7fffffffll;
}

}  // namespace

#define ARB_TRY(call) do { if (int arb_rc = (call)) return arb_rc; ++n; } while (0)

extern "C" int arb_layer_fwd(const ArbLayer* args, int* launches, cudaStream_t s) {
  const ArbLayer& a = *args;
  if (bad_sizes(a) || !a.kept || !a.out || (a.half && !a.out2)) return -3;
  const long long N = a.B * a.T, D = a.H * 128;
  const Kept k(a);
  const Gemm g{static_cast<int*>(a.err), s};
  const float eps = float(a.eps);
  const int* ids = static_cast<const int*>(a.ids);
  const int H = int(a.H), T = int(a.T), ch = int(a.gate_ch);
  int n = 0;
  ARB_TRY(arb_resid_scale_norm_fwd(a.x, a.x0, a.lam_r, a.lam_0, int(a.idx), k.xs, k.xn, N, int(D), eps, s));
  if (a.fuse_post) {
    ARB_TRY(arb_gemm_qkv_post_args(a.cos_t, a.sin_t, k.rstd, T, H, a.ve ? k.xn : nullptr, a.ve ? D : 0, a.ve ? ids : nullptr, a.ve,
                                   a.ve ? a.gate_w : nullptr, a.ve ? k.gate : nullptr, a.ve ? ch : 0, eps));
    ARB_TRY(g.nt(k.xn, a.wqkv, k.qkv, nullptr, N, 3 * D, D, EPI_QKV_POST));
  } else {
    ARB_TRY(g.nt(k.xn, a.wqkv, k.qkv, nullptr, N, 3 * D, D, EPI_STORE_BF16));
    ARB_TRY(arb_qkv_post_fwd(k.qkv, a.cos_t, a.sin_t, k.rstd, k.xn, ids, a.ve, a.ve ? a.gate_w : nullptr, a.ve ? k.gate : nullptr, N, T,
                             H, int(D), ch, eps, s));
  }
  ARB_TRY(arb_attn_fwd(k.qkv, k.qkv + 2 * D, k.qkv + 4 * D, k.att, k.lse, int(a.B), T, H, 3 * D, 3 * D, 3 * D, D, int(a.window),
                       float(a.scale), g.err, s));
  void *xs2 = a.half ? a.out : k.xs2, *xn2 = a.half ? a.out2 : k.xn2;
  ARB_TRY(g.nt(k.att, a.wo, xs2, k.xs, N, D, D, EPI_ADD_AUX));
  ARB_TRY(arb_rmsnorm_fwd(xs2, xn2, N, int(D), eps, s));
  if (!a.half) {
    ARB_TRY(g.nt(xn2, a.wfc, k.act, nullptr, N, a.M, D, EPI_RELU2));
    ARB_TRY(g.nt(k.act, a.wdn, a.out, xs2, N, D, a.M, EPI_ADD_AUX));
  }
  *launches = n;
  return 0;
}

// a.group_dw: the four weight gradients leave in one launch at the end; d_h then has a place of its own.
// a.work: bf16 [N, max(M, 4 D) + D] (with group_dw [N, M + 4 D + D], the value rows' gradients behind M + 3 D), then d_xn_gate
// [N, gate_ch], then (16-byte aligned, as is dgl) fp32 delta and dgl [N, H] each.  a.d_x also holds d_xn2, d_att and d_xn in turn.
// On return the value embedding's row gradients [N, D] lie behind the first 3 N D elements.
extern "C" int arb_layer_bwd(const ArbLayer* args, int* launches, cudaStream_t s) {
  const ArbLayer& a = *args;
  if (bad_sizes(a) || !a.kept || !a.work || !a.d_x || !a.d_x0 || !a.g || a.scoring || (a.half && (!a.out || !a.g_xn))) return -3;
  const long long N = a.B * a.T, D = a.H * 128;
  const Kept k(a);
  const Gemm g{static_cast<int*>(a.err), s};
  const float eps = float(a.eps);
  const int* ids = static_cast<const int*>(a.ids);
  const int H = int(a.H), T = int(a.T), ch = int(a.gate_ch);
  auto* w = static_cast<char*>(a.work);
  const long long wide = a.group_dw ? a.M + 4 * D : a.M > 4 * D ? a.M : 4 * D;
  char *dh = w, *dqkv = w + (a.group_dw ? N * a.M * 2 : 0);   // else d_h is dead when the attention backward writes d_qkv
  char* dve = dqkv + N * 3 * D * 2;
  char *t1 = static_cast<char*>(a.d_x), *g2 = w + N * wide * 2;
  char* dxg = g2 + N * D * 2;
  float *delta = reinterpret_cast<float*>(dxg + (N * ch * 2 + 15) / 16 * 16), *dgl = delta + (N * H + 3) / 4 * 4;
  int n = 0;
  if (a.half) {
    ARB_TRY(arb_rmsnorm_bwd(a.out, a.g_xn, a.g, g2, N, int(D), eps, s));
  } else {
    // MLP: out = xs2 + relu(xn2 wfc^T)^2 wdn^T
    ARB_TRY(g.nn(a.g, a.wdn, dh, k.act, N, a.M, D, EPI_RELU2_BWD));
    if (!a.group_dw) {
      ARB_TRY(g.dw(a.g, k.act, a.g_wdn, D, a.M, N));
      ARB_TRY(g.dw(dh, k.xn2, a.g_wfc, a.M, D, N));
    }
    ARB_TRY(g.nn(dh, a.wfc, t1, nullptr, N, D, a.M, EPI_STORE_BF16));
    ARB_TRY(arb_rmsnorm_bwd(k.xs2, t1, a.g, g2, N, int(D), eps, s));
  }
  // attention: xs2 = xs + att wo^T; g2 is the gradient of xs2
  ARB_TRY(g.nn(g2, a.wo, t1, nullptr, N, D, D, EPI_STORE_BF16));
  if (!a.group_dw) ARB_TRY(g.dw(g2, k.att, a.g_wo, D, D, N));
  ARB_TRY(arb_attn_bwd(k.qkv, k.qkv + 2 * D, k.qkv + 4 * D, k.att, t1, k.lse, dqkv, dqkv + 2 * D, dqkv + 4 * D, delta, nullptr, int(a.B),
                       T, H, 3 * D, 3 * D, 3 * D, D, D, 3 * D, 3 * D, 3 * D, int(a.window), float(a.scale), g.err, s));
  ARB_TRY(arb_qkv_post_bwd(dqkv, k.qkv, a.cos_t, a.sin_t, k.rstd, k.xn, ids, a.ve, a.ve ? a.gate_w : nullptr, a.ve ? k.gate : nullptr,
                           a.ve ? dve : nullptr, a.ve ? static_cast<float*>(a.g_gate) : nullptr, a.ve ? dxg : nullptr,
                           a.ve ? dgl : nullptr, N, T, H, int(D), ch, s));
  if (!a.group_dw) ARB_TRY(g.dw(dqkv, k.xn, a.g_wqkv, 3 * D, D, N));
  ARB_TRY(g.nn(dqkv, a.wqkv, t1, nullptr, N, D, 3 * D, EPI_STORE_BF16));
  if (a.ve) ARB_TRY(arb_add_cols(t1, D, dxg, N, ch, s));
  ARB_TRY(arb_resid_scale_norm_bwd(a.x, a.x0, a.lam_r, a.lam_0, int(a.idx), g2, t1, a.d_x, a.d_x0, a.d_x0_acc,
                                   static_cast<float*>(a.g_lam_r), static_cast<float*>(a.g_lam_0), N, int(D), eps, s));
  if (a.group_dw) {
    const void *dy[4] = {dqkv, g2, a.g, dh}, *x[4] = {k.xn, k.att, k.act, k.xn2};
    float* c[4] = {static_cast<float*>(a.g_wqkv), static_cast<float*>(a.g_wo), static_cast<float*>(a.g_wdn), static_cast<float*>(a.g_wfc)};
    const int d = int(D), f = int(a.M), rows[4] = {3 * d, d, d, f}, cols[4] = {d, d, f, d};
    ARB_TRY(arb_gemm_dw_group(dy, x, c, rows, cols, a.half ? 2 : 4, int(N), g.err, s));
  }
  *launches = n;
  return 0;
}
