// The host side of the ops that a layer is made of, as one extension module over the C ABI
// (include/b200_hstu.h): results and scratch are allocated, argument structs filled and the launches
// and library GEMMs of a stage queued in one call from Python.
//
// A layer on a small batch takes its kernels 40 us in inference and 390 us in training (forward and
// backward); with one Python call, a ctypes struct and a few tensor objects per launch its host side
// took 115 and 660 us, and the GPU waited.
#include <ATen/cuda/CUDAContext.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>

#include <optional>
#include <string>
#include <tuple>

#include "b200_hstu.h"

namespace {

using at::Tensor;
using MaybeTensor = std::optional<Tensor>;

// the message of _cabi.check()
void check(int rc, const char *what) {
  if (rc != 0)
    throw std::runtime_error(std::string(what) + " failed (status " + std::to_string(rc) + "): " + b200_hstu_last_error());
}

// the device of the launch and the current stream on it
struct Launch {
  c10::cuda::CUDAGuard guard;
  cudaStream_t stream;
  explicit Launch(const Tensor &t)
      : guard(t.device()), stream(at::cuda::getCurrentCUDAStream(t.device().index()).stream()) {}
};

// The library GEMMs go through the dispatcher, so under autocast they convert their operands.  The backwards
// are called with the types that the forward chose and keep them, wherever they are called.
struct NoAutocast {
  c10::impl::ExcludeDispatchKeyGuard guard{c10::autocast_dispatch_keyset};
};

// A kernel walks a buffer by the dtype code of the call: what a GEMM has made has to have that type.
const Tensor &of_type(const Tensor &t, at::ScalarType type) {
  TORCH_CHECK(t.scalar_type() == type, "a library GEMM gave ", t.scalar_type(), " where the next kernel reads ", type);
  return t;
}

Tensor empty_like_of(at::IntArrayRef shape, const Tensor &t) { return at::empty(shape, t.options()); }
Tensor floats(int64_t n, const Tensor &t) { return at::empty({n}, t.options().dtype(at::kFloat)); }
Tensor bytes(int64_t n, const Tensor &t) { return at::empty({n}, t.options().dtype(at::kByte)); }
template <typename T = void>
T *ptr(const Tensor &t) { return t.numel() == 0 ? nullptr : static_cast<T *>(t.data_ptr()); }
template <typename T = void>
T *ptr(const MaybeTensor &t) { return t.has_value() && t->defined() ? ptr<T>(*t) : nullptr; }
bool given(const MaybeTensor &t) { return t.has_value() && t->defined(); }

// ---------------------------------------------------------------------------------------
// attention
// ---------------------------------------------------------------------------------------
// what a call says besides its tensors
struct AttnConfig {
  int64_t max_seq_len;
  double alpha;
  int64_t max_attn_len, contextual_seq_len, min_full_attn_seq_len;
  int64_t impl, dtype;
};

void fill_attn(b200_hstu_attn_args &a, const Tensor &q, const Tensor &k, const Tensor &v, const Tensor &offsets,
               const MaybeTensor &targets, const MaybeTensor &scale, const MaybeTensor &bias, const AttnConfig &c,
               double dropout, const MaybeTensor &seed) {
  a.q = ptr(q);
  a.k = ptr(k);
  a.v = ptr(v);
  a.seq_offsets = ptr<const int32_t>(offsets);
  a.num_targets = ptr<const int32_t>(targets);
  if (given(scale)) {
    a.attn_scale = static_cast<const float *>(scale->data_ptr());
    a.attn_scale_numel = scale->numel();
  }
  a.q_row_stride = q.stride(0);
  a.q_head_stride = q.stride(1);
  a.k_row_stride = k.stride(0);
  a.k_head_stride = k.stride(1);
  a.v_row_stride = v.stride(0);
  a.v_head_stride = v.stride(1);
  a.total_L = k.size(0);
  a.B = (int32_t)(offsets.numel() - 1);
  a.H = (int32_t)q.size(1);
  a.dqk = (int32_t)q.size(2);
  a.dv = (int32_t)v.size(2);
  a.max_seq_len = (int32_t)c.max_seq_len;
  a.alpha = (float)c.alpha;
  a.max_attn_len = (int32_t)c.max_attn_len;
  a.contextual_seq_len = (int32_t)c.contextual_seq_len;
  a.min_full_attn_seq_len = (int32_t)c.min_full_attn_seq_len;
  a.dtype = (int32_t)c.dtype;
  a.impl = (int32_t)c.impl;
  if (offsets.scalar_type() == at::kLong) a.impl |= B200_HSTU_OFFSETS_I64;
  if (given(targets) && targets->scalar_type() == at::kLong) a.impl |= B200_HSTU_TARGETS_I64;
  if (given(bias)) {
    a.bias_by_distance = static_cast<const float *>(bias->data_ptr());
    a.bias_numel = (int32_t)bias->numel();
  }
  if (given(seed) && dropout > 0.0) {
    a.dropout_ratio = (float)dropout;
    a.dropout_seed = static_cast<const uint64_t *>(seed->data_ptr());
  }
}

MaybeTensor attn_workspace(b200_hstu_attn_args &a, int which, const Tensor &like) {
  const int64_t n = b200_hstu_attn_workspace_bytes(&a, which);
  if (n <= 0) return std::nullopt;
  Tensor ws = bytes(n, like);
  a.workspace = ws.data_ptr();
  a.workspace_bytes = n;
  return ws;
}

// After a launch, for debugging: waits for the stream and reads the status words of its work lists; a
// bounded wait that gave up inside the kernel becomes an error.
void check_status(const b200_hstu_attn_args &a, int which, cudaStream_t stream, const char *what) {
  Tensor host = at::zeros({3}, at::TensorOptions().dtype(at::kInt).pinned_memory(true));
  int32_t *s = static_cast<int32_t *>(host.data_ptr());
  check(b200_hstu_attn_status_async(&a, which, s, stream), "b200_hstu_attn_status_async");
  C10_CUDA_CHECK(cudaStreamSynchronize(stream));
  if (s[0] != 0 || s[1] != 0 || s[2] != 0)
    throw std::runtime_error(std::string(what) +
                             ": a bounded wait inside the kernel gave up (status forward / dK,dV / dQ = [" +
                             std::to_string(s[0]) + ", " + std::to_string(s[1]) + ", " + std::to_string(s[2]) +
                             "]); the output is incomplete");
}

// `delta` > 0: cached inference (q holds the last `delta` rows of every sequence); rows of sequences shorter than
// that are zero (`long_enough`: there are none).  Returns the output and the scratch (for the backward's plan, and the status words).
std::tuple<Tensor, MaybeTensor> attention_forward(const Tensor &q, const Tensor &k, const Tensor &v,
                                                  const Tensor &offsets, const MaybeTensor &targets,
                                                  const MaybeTensor &scale, const MaybeTensor &bias,
                                                  int64_t max_seq_len, double alpha, int64_t max_attn_len,
                                                  int64_t contextual_seq_len, int64_t min_full_attn_seq_len,
                                                  int64_t impl, int64_t dtype, bool plan, double dropout,
                                                  const MaybeTensor &seed, int64_t delta, bool long_enough,
                                                  bool status) {
  Tensor out = delta > 0 && !long_enough ? at::zeros({q.size(0), q.size(1), v.size(2)}, q.options())
                         : at::empty({q.size(0), q.size(1), v.size(2)}, q.options());
  b200_hstu_attn_args a = {};
  fill_attn(a, q, k, v, offsets, targets, scale, bias,
            {max_seq_len, alpha, max_attn_len, contextual_seq_len, min_full_attn_seq_len, impl, dtype}, dropout, seed);
  a.out = ptr(out);
  a.o_row_stride = out.stride(0);
  a.o_head_stride = out.stride(1);
  a.delta_size = (int32_t)delta;
  MaybeTensor ws = attn_workspace(a, plan ? 2 : 0, q);
  if (plan && given(ws)) a.plan_mode = B200_HSTU_PLAN_FOR_BACKWARD;
  Launch l(q);
  check(b200_hstu_attn_fwd(&a, l.stream), delta > 0 ? "b200_hstu_attn_fwd (delta)" : "b200_hstu_attn_fwd");
  if (status && given(ws))
    check_status(a, 0, l.stream, delta > 0 ? "b200_hstu_attn_fwd (delta)" : "b200_hstu_attn_fwd");
  return {out, ws};
}

// Fills dq, dk, dv (and adds to d_bias).
void attention_backward(const Tensor &dout, const Tensor &q, const Tensor &k, const Tensor &v,
                        const Tensor &offsets, const MaybeTensor &targets, const MaybeTensor &scale,
                        const MaybeTensor &bias, int64_t max_seq_len, double alpha, int64_t max_attn_len,
                        int64_t contextual_seq_len, int64_t min_full_attn_seq_len, int64_t impl, int64_t dtype,
                        const Tensor &dq, const Tensor &dk, const Tensor &dv, const MaybeTensor &planned,
                        const MaybeTensor &d_bias, double dropout, const MaybeTensor &seed, bool status) {
  b200_hstu_attn_args a = {};
  fill_attn(a, q, k, v, offsets, targets, scale, bias,
            {max_seq_len, alpha, max_attn_len, contextual_seq_len, min_full_attn_seq_len, impl, dtype}, dropout, seed);
  a.dout = dout.data_ptr();
  a.dq = dq.data_ptr();
  a.dk = dk.data_ptr();
  a.dv_ = dv.data_ptr();
  a.do_row_stride = dout.stride(0);
  a.do_head_stride = dout.stride(1);
  a.dq_row_stride = dq.stride(0);
  a.dq_head_stride = dq.stride(1);
  a.dk_row_stride = dk.stride(0);
  a.dk_head_stride = dk.stride(1);
  a.dv_row_stride = dv.stride(0);
  a.dv_head_stride = dv.stride(1);
  if (given(d_bias) && given(bias)) a.d_bias_by_distance = static_cast<float *>(d_bias->data_ptr());
  MaybeTensor ws;
  if (given(planned) && b200_hstu_attn_workspace_bytes(&a, 1) > 0) {
    a.plan_mode = B200_HSTU_PLAN_REUSE;
    a.workspace = planned->data_ptr();
    a.workspace_bytes = planned->numel();
  } else {
    ws = attn_workspace(a, 1, q);
  }
  Launch l(q);
  check(b200_hstu_attn_bwd(&a, l.stream), "b200_hstu_attn_bwd");
  if (status && a.workspace != nullptr)
    check_status(a, a.plan_mode == B200_HSTU_PLAN_REUSE ? 2 : 1, l.stream, "b200_hstu_attn_bwd");
}

// ---------------------------------------------------------------------------------------
// norm-mul
// ---------------------------------------------------------------------------------------
struct NormMulConfig {
  double eps;
  int64_t H, V;
  bool concat_u, concat_x;
  int64_t act;
  bool group_norm;
  double dropout;
};

void fill_norm_mul(b200_hstu_norm_mul_args &a, const Tensor &attn, const Tensor &u, const Tensor &weight,
                   const Tensor &bias, const NormMulConfig &c, int64_t dtype, const MaybeTensor &seed) {
  a.attn = attn.data_ptr();
  a.u = u.data_ptr();
  a.weight = weight.data_ptr();
  a.bias = bias.data_ptr();
  a.attn_row_stride = attn.stride(0);
  a.u_row_stride = u.stride(0);
  a.rows = attn.size(0);
  a.H = (int32_t)c.H;
  a.V = (int32_t)c.V;
  a.concat_u = c.concat_u;
  a.concat_x = c.concat_x;
  a.act = (int32_t)c.act;
  a.group_norm = c.group_norm;
  a.eps = (float)c.eps;
  a.dtype = (int32_t)dtype;
  if (given(seed) && c.dropout > 0.0) {
    a.dropout_ratio = (float)c.dropout;
    a.dropout_seed = static_cast<const int64_t *>(seed->data_ptr());
  }
}

// out, mean, rstd (`stats`), and the dropout mask as bits (`want_mask`, where the library can store it)
std::tuple<Tensor, MaybeTensor, MaybeTensor, MaybeTensor> norm_mul_forward(
    const Tensor &attn, const Tensor &u, const Tensor &weight, const Tensor &bias, double eps, int64_t H, int64_t V,
    bool concat_u, bool concat_x, int64_t act, bool group_norm, double dropout, const MaybeTensor &seed, int64_t dtype,
    bool want_mask, bool stats) {
  const int64_t rows = attn.size(0);
  const int64_t parts = group_norm ? (concat_u && concat_x ? 3 : 1) : 1 + (int)concat_u + (int)concat_x;
  Tensor out = empty_like_of({rows, parts * H * V}, attn);
  MaybeTensor mean, rstd, mask;
  b200_hstu_norm_mul_args a = {};
  fill_norm_mul(a, attn, u, weight, bias, {eps, H, V, concat_u, concat_x, act, group_norm, dropout}, dtype, seed);
  a.out = out.data_ptr();
  a.out_row_stride = out.stride(0);
  if (stats) {
    mean = floats(rows * (group_norm ? H : 1), attn);
    rstd = floats(rows * (group_norm ? H : 1), attn);
    a.mean = static_cast<float *>(mean->data_ptr());
    a.rstd = static_cast<float *>(rstd->data_ptr());
  }
  if (want_mask && a.dropout_seed != nullptr && rows > 0) {
    const int64_t n = b200_hstu_norm_mul_dropout_mask_bytes(&a);
    if (n > 0) {
      mask = bytes(n, attn);
      a.dropout_mask = static_cast<uint8_t *>(mask->data_ptr());
    }
  }
  if (rows > 0) {
    Launch l(attn);
    check(b200_hstu_norm_mul_fwd(&a, l.stream), "b200_hstu_norm_mul_fwd");
  }
  return {out, mean, rstd, mask};
}

// dattn, du, dweight, dbias.  `mask`: the bits the forward stored; without them the kernel regenerates the
// mask from the seed.
std::tuple<Tensor, Tensor, Tensor, Tensor> norm_mul_backward(
    const Tensor &dout_, const Tensor &attn, const Tensor &u, const Tensor &weight, const Tensor &bias,
    const Tensor &mean, const Tensor &rstd, double eps, int64_t H, int64_t V, bool concat_u, bool concat_x, int64_t act,
    bool group_norm, double dropout, const MaybeTensor &seed, const MaybeTensor &mask, int64_t dtype) {
  const Tensor dout = dout_.stride(-1) != 1 ? dout_.contiguous() : dout_;
  const int64_t rows = attn.size(0);
  Tensor dattn = empty_like_of({rows, H * V}, attn);
  Tensor du = empty_like_of({rows, H * V}, attn);
  Tensor dw = at::empty_like(weight), db = at::empty_like(bias);
  const int64_t n = b200_hstu_norm_mul_bwd_workspace_bytes((int32_t)H, (int32_t)V, group_norm);
  Tensor partial = bytes(n, attn);
  b200_hstu_norm_mul_args a = {};
  fill_norm_mul(a, attn, u, weight, bias, {eps, H, V, concat_u, concat_x, act, group_norm, dropout}, dtype, seed);
  a.mean = static_cast<float *>(mean.data_ptr());
  a.rstd = static_cast<float *>(rstd.data_ptr());
  a.dout = dout.data_ptr();
  a.dattn = dattn.data_ptr();
  a.du = du.data_ptr();
  a.dweight = dw.data_ptr();
  a.dbias = db.data_ptr();
  a.partial = partial.data_ptr();
  a.partial_bytes = n;
  a.dout_row_stride = dout.stride(0);
  a.dattn_row_stride = dattn.stride(0);
  a.du_row_stride = du.stride(0);
  if (a.dropout_seed != nullptr && given(mask) && reinterpret_cast<uintptr_t>(dout.data_ptr()) % 16 == 0 &&
      dout.stride(0) % 8 == 0)
    a.dropout_mask = static_cast<uint8_t *>(mask->data_ptr());
  Launch l(attn);
  check(b200_hstu_norm_mul_bwd(&a, l.stream), "b200_hstu_norm_mul_bwd");
  return {dattn, du, dw, db};
}

// ---------------------------------------------------------------------------------------
// output stage: x + norm_mul(attn, u) W
// ---------------------------------------------------------------------------------------
// `over_x`: the result goes over x.
std::tuple<Tensor, MaybeTensor, MaybeTensor> output_forward(const Tensor &attn, const Tensor &u, Tensor x,
                                                            const Tensor &weight, const Tensor &bias,
                                                            const Tensor &output_weight, double eps, int64_t H,
                                                            int64_t V, bool concat_u, bool concat_x, int64_t act,
                                                            bool group_norm, double dropout, const MaybeTensor &seed,
                                                            int64_t dtype, bool stats, bool over_x) {
  auto [y, mean, rstd, mask] = norm_mul_forward(attn, u, weight, bias, eps, H, V, concat_u, concat_x, act, group_norm,
                                                dropout, seed, dtype, false, stats);
  // (addmm copies x into its result first, a pass over memory: 1.26 ms of the 49 of four layers on 484 k rows of 1024)
  return {over_x ? x.addmm_(y, output_weight) : at::addmm(x, y, output_weight), mean, rstd};
}

// dattn, du, d_norm_weight, d_norm_bias, d_output_weight
std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor> output_backward(
    const Tensor &dout_, const Tensor &attn, const Tensor &u, const Tensor &weight, const Tensor &bias,
    const Tensor &output_weight, const Tensor &mean, const Tensor &rstd, double eps, int64_t H, int64_t V,
    bool concat_u, bool concat_x, int64_t act, bool group_norm, double dropout, const MaybeTensor &seed, int64_t dtype) {
  const NoAutocast no_autocast;
  Tensor d_wo;
  // (under autocast the forward's result may have another type than what went into it)
  const at::ScalarType type = attn.scalar_type();
  const Tensor dout = (dout_.stride(-1) != 1 ? dout_.contiguous() : dout_).to(type), wo = output_weight.to(type);
  {
    Tensor y = std::get<0>(norm_mul_forward(attn, u, weight, bias, eps, H, V, concat_u, concat_x, act, group_norm,
                                            dropout, seed, dtype, false, true));
    d_wo = at::mm(y.t(), dout);
  }
  const Tensor dy = at::mm(dout, wo.t());
  auto [dattn, du, dw, db] = norm_mul_backward(of_type(dy, type), attn, u, weight, bias, mean, rstd, eps, H, V, concat_u, concat_x,
                                               act, group_norm, dropout, seed, std::nullopt, dtype);
  return {dattn, du, dw, db, d_wo};
}

// ---------------------------------------------------------------------------------------
// uvqk stage: LayerNorm, linear, SiLU(u)
// ---------------------------------------------------------------------------------------
bool uvqk_supported(const Tensor &x, const Tensor &weight, int64_t hv, int64_t dtype) {
  if (x.stride(-1) != 1 || x.stride(0) % 8 != 0 || x.stride(0) < x.size(1) ||
      reinterpret_cast<uintptr_t>(x.data_ptr()) % 16 != 0)
    return false;
  return b200_hstu_ln_linear_supported((int32_t)weight.size(0), (int32_t)weight.size(1), (int32_t)hv, (int32_t)dtype) != 0;
}

struct Uvqk {
  Tensor uvqk, u;
  MaybeTensor mean, rstd;
};

Uvqk uvqk_launch(const Tensor &x, const Tensor &nw, const Tensor &nb, const Tensor &w, const Tensor &b, double eps,
                 int64_t hv, int64_t dtype, bool inference, const MaybeTensor &workspace, bool prepared) {
  const int64_t M = x.size(0), D = x.size(1), N = w.size(1);
  // (the kernel reads them, and sizes its workspace, by the width of x)
  TORCH_CHECK(w.size(0) == D && nw.numel() >= D && nb.numel() >= D && b.numel() >= N,
              "uvqk stage: parameters of another width than x");
  Uvqk r;
  r.uvqk = empty_like_of({M, N}, x);
  r.u = empty_like_of({M, hv}, x);
  b200_hstu_ln_linear_args a = {};
  if (!inference) {
    r.mean = floats(M, x);
    r.rstd = floats(M, x);
    a.mean = static_cast<float *>(r.mean->data_ptr());
    a.rstd = static_cast<float *>(r.rstd->data_ptr());
  }
  const int64_t n = b200_hstu_ln_linear_workspace_bytes((int32_t)D, (int32_t)N);
  const Tensor ws = given(workspace) ? *workspace : bytes(n, x);
  a.weights_prepared = prepared;
  a.skip_pre_activation = inference;
  a.x = x.data_ptr();
  a.norm_weight = nw.data_ptr();
  a.norm_bias = nb.data_ptr();
  a.weight = w.data_ptr();
  a.bias = b.data_ptr();
  a.out = r.uvqk.data_ptr();
  a.u = r.u.data_ptr();
  a.workspace = ws.data_ptr();
  a.workspace_bytes = n;
  a.x_row_stride = x.stride(0);
  a.out_row_stride = r.uvqk.stride(0);
  a.u_row_stride = r.u.stride(0);
  a.M = M;
  a.D = (int32_t)D;
  a.N = (int32_t)N;
  a.silu_cols = (int32_t)hv;
  a.eps = (float)eps;
  a.dtype = (int32_t)dtype;
  Launch l(x);
  check(b200_hstu_ln_linear_silu_fwd(&a, l.stream), "b200_hstu_ln_linear_silu_fwd");
  return r;
}

// (q, k, v) as [M, H, d] views of the uvqk buffer, columns [u | v | q | k]
struct Qkv {
  Tensor q, k, v;
};
Qkv qkv_views(const Tensor &uvqk, int64_t H, int64_t A, int64_t V) {
  const int64_t M = uvqk.size(0), N = uvqk.stride(0), off = uvqk.storage_offset();
  return {uvqk.as_strided({M, H, A}, {N, A, 1}, off + 2 * H * V), uvqk.as_strided({M, H, A}, {N, A, 1}, off + 2 * H * V + H * A),
          uvqk.as_strided({M, H, V}, {N, V, 1}, off + H * V)};
}

// u, attention output, k, v where no gradient is wanted
std::tuple<Tensor, Tensor, Tensor, Tensor> uvqk_attention_inference(
    const Tensor &x, const Tensor &nw, const Tensor &nb, const Tensor &w, const Tensor &b, double eps, int64_t H,
    int64_t A, int64_t V, const Tensor &workspace, bool prepared, const Tensor &offsets, const MaybeTensor &targets,
    const MaybeTensor &bias, int64_t max_seq_len, double alpha, int64_t max_attn_len, int64_t contextual_seq_len,
    int64_t impl, int64_t dtype, bool status) {
  const Uvqk s = uvqk_launch(x, nw, nb, w, b, eps, H * V, dtype, true, workspace, prepared);
  const Qkv t = qkv_views(s.uvqk, H, A, V);
  Tensor out = std::get<0>(attention_forward(t.q, t.k, t.v, offsets, targets, std::nullopt, bias, max_seq_len, alpha,
                                             max_attn_len, contextual_seq_len, 0, impl, dtype, false, 0.0, std::nullopt, 0,
                                             true, status));
  return {s.u, out.view({x.size(0), H * V}), t.k, t.v};
}

// The same from the separate stages: LayerNorm, library GEMM, SiLU
std::tuple<Tensor, Tensor, Tensor, Tensor> separate_attention_inference(
    const Tensor &x, const Tensor &nw, const Tensor &nb, const Tensor &w, const Tensor &b, double eps, int64_t H,
    int64_t A, int64_t V, const Tensor &offsets, const MaybeTensor &targets, const MaybeTensor &bias,
    int64_t max_seq_len, double alpha, int64_t max_attn_len, int64_t contextual_seq_len, int64_t impl, int64_t dtype,
    bool status) {
  Tensor uvqk, u = empty_like_of({x.size(0), H * V}, x);
  {
    Tensor normed = empty_like_of({x.size(0), x.size(1)}, x);
    Launch l(x);
    check(b200_hstu_layer_norm_fwd(x.data_ptr(), x.stride(0), nw.data_ptr(), nb.data_ptr(), normed.data_ptr(),
                                   normed.stride(0), nullptr, nullptr, x.size(0), (int32_t)x.size(1), (float)eps,
                                   (int32_t)dtype, l.stream),
          "b200_hstu_layer_norm_fwd");
    uvqk = of_type(at::addmm(b, normed, w), x.scalar_type());
    check(b200_hstu_silu_fwd(uvqk.data_ptr(), uvqk.stride(0), u.data_ptr(), u.stride(0), x.size(0), (int32_t)(H * V),
                             (int32_t)dtype, l.stream),
          "b200_hstu_silu_fwd");
  }
  const Qkv t = qkv_views(uvqk, H, A, V);
  Tensor out = std::get<0>(attention_forward(t.q, t.k, t.v, offsets, targets, std::nullopt, bias, max_seq_len, alpha,
                                             max_attn_len, contextual_seq_len, 0, impl, dtype, false, 0.0, std::nullopt, 0,
                                             true, status));
  return {u, out.view({x.size(0), H * V}), t.k, t.v};
}

// Whether cached_attention() takes these: one launch appends to K and V, which have the same rows
bool cached_supported(const Tensor &x, const Tensor &weight, int64_t hv, int64_t ha, const Tensor &k_cache,
                      const Tensor &v_cache, const Tensor &cache_offsets) {
  const auto fits = [&](const Tensor &t, int64_t width) {
    return t.dim() == 2 && t.size(0) == k_cache.size(0) && t.size(1) == width && t.scalar_type() == x.scalar_type() &&
           t.is_contiguous();
  };
  if (x.dim() != 2 || x.size(0) == 0 || (x.scalar_type() != at::kBFloat16 && x.scalar_type() != at::kHalf) ||
      cache_offsets.scalar_type() != at::kLong || !cache_offsets.is_contiguous() || !fits(k_cache, ha) || !fits(v_cache, hv))
    return false;
  return uvqk_supported(x, weight, hv, x.scalar_type() == at::kBFloat16 ? B200_HSTU_BF16 : B200_HSTU_F16);
}

// Cached inference: uvqk stage on the new rows, their K and V behind the cached ones, attention of the new rows.
// Returns u, attention output, k, v, offsets of k and v.
std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor> cached_attention(
    const Tensor &x, const Tensor &nw, const Tensor &nb, const Tensor &w, const Tensor &b, double eps, int64_t H,
    int64_t A, int64_t V, const Tensor &workspace, bool prepared, const Tensor &k_cache, const Tensor &v_cache,
    const Tensor &cache_offsets, const MaybeTensor &targets, int64_t max_seq_len, double alpha, int64_t max_attn_len,
    int64_t contextual_seq_len, int64_t impl, int64_t dtype, bool status) {
  const int64_t B = cache_offsets.numel() - 1, delta = x.size(0) / B, rows = k_cache.size(0) + x.size(0);
  TORCH_CHECK(!given(targets) || targets->numel() >= B, "num_targets must have one entry per sequence");
  const Uvqk s = uvqk_launch(x, nw, nb, w, b, eps, H * V, dtype, true, workspace, prepared);
  const Qkv t = qkv_views(s.uvqk, H, A, V);
  Tensor k = empty_like_of({rows, H, A}, x), v = empty_like_of({rows, H, V}, x);
  Tensor offsets = at::empty({B + 1}, cache_offsets.options());
  b200_hstu_append_kv_args a = {};
  a.k_cache = ptr(k_cache);
  a.v_cache = ptr(v_cache);
  a.k_new = ptr(t.k);
  a.v_new = ptr(t.v);
  a.k = ptr(k);
  a.v = ptr(v);
  a.offsets = static_cast<const int64_t *>(cache_offsets.data_ptr());
  a.full_offsets = static_cast<int64_t *>(offsets.data_ptr());
  a.k_row_bytes = H * A * x.element_size();
  a.v_row_bytes = H * V * x.element_size();
  a.k_new_stride_bytes = t.k.stride(0) * x.element_size();
  a.v_new_stride_bytes = t.v.stride(0) * x.element_size();
  a.cached_rows = k_cache.size(0);
  a.B = (int32_t)B;
  a.delta = (int32_t)delta;
  Launch l(x);
  check(b200_hstu_append_kv(&a, l.stream), "b200_hstu_append_kv");
  Tensor out = std::get<0>(attention_forward(t.q, k, v, offsets, targets, std::nullopt, std::nullopt, max_seq_len, alpha,
                                             max_attn_len, contextual_seq_len, 0, impl, dtype, false, 0.0, std::nullopt,
                                             delta, true, status));
  return {s.u, out.view({x.size(0), H * V}), k, v, offsets};
}

// u, attention output, k, v, uvqk, mean, rstd, scratch with the backward's plan
std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor, Tensor, Tensor, MaybeTensor> uvqk_attention_forward(
    const Tensor &x, const Tensor &nw, const Tensor &nb, const Tensor &w, const Tensor &b, double eps, int64_t H,
    int64_t A, int64_t V, const Tensor &offsets, const MaybeTensor &targets, const MaybeTensor &bias,
    int64_t max_seq_len, double alpha, int64_t max_attn_len, int64_t contextual_seq_len, int64_t impl, int64_t dtype,
    bool plan, bool status) {
  const Uvqk s = uvqk_launch(x, nw, nb, w, b, eps, H * V, dtype, false, std::nullopt, false);
  const Qkv t = qkv_views(s.uvqk, H, A, V);
  auto [out, ws] = attention_forward(t.q, t.k, t.v, offsets, targets, std::nullopt, bias, max_seq_len, alpha, max_attn_len,
                                     contextual_seq_len, 0, impl, dtype, plan, 0.0, std::nullopt, 0, true, status);
  return {s.u, out, t.k, t.v, s.uvqk, *s.mean, *s.rstd, ws};
}

// Backward of the uvqk stage: d_uvqk [M, N] already holds the gradients of the v, q, k columns; the u columns
// are filled here (du * SiLU').  LN(x) is rebuilt from the saved statistics.  Returns dx and the gradients of
// norm weight, norm bias, weight and bias.
std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor> uvqk_backward(const Tensor &x, const Tensor &nw, const Tensor &nb,
                                                                 const Tensor &w, const Tensor &uvqk,
                                                                 const Tensor &mean, const Tensor &rstd, double eps,
                                                                 int64_t hv, const MaybeTensor &du_, const Tensor &d_uvqk,
                                                                 int64_t dtype) {
  const NoAutocast no_autocast;
  const int64_t M = x.size(0), D = x.size(1);
  const int32_t dt = (int32_t)dtype;
  Launch l(x);
  if (given(du_)) {
    const Tensor du = du_->stride(-1) != 1 ? du_->contiguous() : *du_;
    check(b200_hstu_silu_bwd(du.data_ptr(), du.stride(0), uvqk.data_ptr(), uvqk.stride(0), d_uvqk.data_ptr(),
                             d_uvqk.stride(0), M, (int32_t)hv, dt, l.stream),
          "b200_hstu_silu_bwd");
  } else {
    d_uvqk.narrow(1, 0, hv).zero_();
  }
  Tensor normed = at::empty_like(x);
  check(b200_hstu_layer_norm_fwd(x.data_ptr(), x.stride(0), nw.data_ptr(), nb.data_ptr(), normed.data_ptr(),
                                 normed.stride(0), nullptr, nullptr, M, (int32_t)D, (float)eps, dt, l.stream),
        "b200_hstu_layer_norm_fwd");
  Tensor dw = at::mm(normed.t(), d_uvqk);
  // column sums on the tensor cores: cheaper than a strided reduction over [M, N]
  Tensor db = at::mm(at::ones({1, M}, x.options()), d_uvqk).view(-1);
  Tensor dnormed = of_type(at::mm(d_uvqk, w.t()), x.scalar_type());
  Tensor dx = at::empty_like(x);
  Tensor dnw = empty_like_of({D}, x), dnb = empty_like_of({D}, x);
  const int64_t n = b200_hstu_layer_norm_bwd_workspace_bytes((int32_t)D);
  Tensor partial = bytes(n, x);
  check(b200_hstu_layer_norm_bwd(dnormed.data_ptr(), dnormed.stride(0), x.data_ptr(), x.stride(0), nw.data_ptr(),
                                 static_cast<const float *>(mean.data_ptr()), static_cast<const float *>(rstd.data_ptr()),
                                 dx.data_ptr(), dx.stride(0), dnw.data_ptr(), dnb.data_ptr(), partial.data_ptr(), n, M,
                                 (int32_t)D, dt, l.stream),
        "b200_hstu_layer_norm_bwd");
  return {dx, dnw, dnb, dw, db};
}

// Backward of uvqk_attention_forward.  uvqk (with mean and rstd) not given: it was not kept, the fused kernel
// runs once more.  The attention writes dq, dk, dv into the column blocks of d_uvqk.  Last result: d_bias.
std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor, MaybeTensor> uvqk_attention_backward(
    const Tensor &x, const Tensor &nw, const Tensor &nb, const Tensor &w, const Tensor &b, const MaybeTensor &uvqk_,
    const Tensor &mean_, const Tensor &rstd_, double eps, int64_t H, int64_t A, int64_t V, const Tensor &offsets,
    const MaybeTensor &targets, const MaybeTensor &bias, int64_t max_seq_len, double alpha, int64_t max_attn_len,
    int64_t contextual_seq_len, int64_t impl, int64_t dtype, const MaybeTensor &du, const MaybeTensor &dattn_,
    const MaybeTensor &dk_more, const MaybeTensor &dv_more, const MaybeTensor &planned, bool want_d_bias,
    bool status) {
  const int64_t hv = H * V;
  Tensor uvqk, mean = mean_, rstd = rstd_;
  if (given(uvqk_)) {
    uvqk = *uvqk_;
  } else {
    const Uvqk s = uvqk_launch(x, nw, nb, w, b, eps, hv, dtype, false, std::nullopt, false);
    uvqk = s.uvqk;
    mean = *s.mean;
    rstd = *s.rstd;
  }
  const int64_t M = uvqk.size(0), N = uvqk.size(1);
  Tensor d_uvqk = empty_like_of({M, N}, x);
  const Qkv d = qkv_views(d_uvqk, H, A, V);
  MaybeTensor d_bias;
  if (!given(dattn_)) {
    d_uvqk.narrow(1, hv, N - hv).zero_();
  } else {
    Tensor dattn = *dattn_;
    if (dattn.stride(-1) != 1 || dattn.stride(1) != dattn.size(2) || dattn.stride(0) < dattn.size(1) * dattn.size(2))
      dattn = dattn.contiguous();
    const Qkv t = qkv_views(uvqk, H, A, V);
    if (want_d_bias) d_bias = at::zeros_like(*bias);
    attention_backward(dattn, t.q, t.k, t.v, offsets, targets, std::nullopt, bias, max_seq_len, alpha, max_attn_len,
                       contextual_seq_len, 0, impl, dtype, d.q, d.k, d.v, planned, d_bias, 0.0, std::nullopt, status);
  }
  if (given(dk_more)) d.k.add_(*dk_more);
  if (given(dv_more)) d.v.add_(*dv_more);
  auto [dx, dnw, dnb, dw, db] = uvqk_backward(x, nw, nb, w, uvqk, mean, rstd, eps, hv, du, d_uvqk, dtype);
  return {dx, dnw, dnb, dw, db, d_bias};
}

}  // namespace

PYBIND11_MODULE(_host, m) {
  // the exceptions that the torch functions of the same calls raise (an allocation that fails is caught by its type)
  py::register_local_exception_translator([](std::exception_ptr p) {
    try {
      if (p) std::rethrow_exception(p);
    } catch (const c10::OutOfMemoryError &e) {
      PyErr_SetString(py::module_::import("torch").attr("OutOfMemoryError").ptr(), e.what_without_backtrace());
    } catch (const c10::IndexError &e) {
      PyErr_SetString(PyExc_IndexError, e.what_without_backtrace());
    } catch (const c10::Error &e) {
      PyErr_SetString(PyExc_RuntimeError, e.what_without_backtrace());
    }
  });
  // (as with ctypes, other threads run while launches are queued)
  const auto unlocked = py::call_guard<py::gil_scoped_release>();
  m.def("attention_forward", &attention_forward, unlocked);
  m.def("attention_backward", &attention_backward, unlocked);
  m.def("norm_mul_forward", &norm_mul_forward, unlocked);
  m.def("norm_mul_backward", &norm_mul_backward, unlocked);
  m.def("output_forward", &output_forward, unlocked);
  m.def("output_backward", &output_backward, unlocked);
  m.def("uvqk_supported", &uvqk_supported, unlocked);
  m.def("uvqk_backward", &uvqk_backward, unlocked);
  m.def("uvqk_attention_inference", &uvqk_attention_inference, unlocked);
  m.def("separate_attention_inference", &separate_attention_inference, unlocked);
  m.def("cached_supported", &cached_supported, unlocked);
  m.def("cached_attention", &cached_attention, unlocked);
  m.def("uvqk_attention_forward", &uvqk_attention_forward, unlocked);
  m.def("uvqk_attention_backward", &uvqk_attention_backward, unlocked);
}
