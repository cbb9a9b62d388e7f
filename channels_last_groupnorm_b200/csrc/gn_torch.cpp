// Thin torch-extension binding over the C ABI of libgnb200.so.
//
// Registers torch.ops.gnb200.fwd / bwd with the schemas of the reference's gnop::fwd / gnop::bwd
// (src/gnnhwc/csrc/custom_gn.cpp:10-16, 44-52, 91-94):
//   fwd(Tensor X, Tensor weight, Tensor bias, int G, float eps, int act) -> (Tensor Y, Tensor means, Tensor rstds)
//   bwd(Tensor dy, Tensor X, Tensor weight, Tensor bias, Tensor means, Tensor rstds, int G, int act)
//       -> (Tensor dX, Tensor dweight, Tensor dbias)
// X / dy / Y / dX are logical (N, C, R) tensors, either with strides (R*C, 1, C), i.e. NHWC storage -
// the only layout the reference's ops accept - or contiguous, i.e. NCHW storage, which goes to the
// native channels-first kernels; results have the storage order of X.
// Differences from the reference, all deliberate: the namespace (so both libraries can live in one
// process), means/rstds are fp32 (fp64 for fp64 tensors), every argument is validated, the
// tensor's device is made current, a third op `bwd_f32` returns the parameter gradients as one packed
// [2, C] tensor in the statistics' dtype (the buffer a data-parallel caller all-reduces), and the ops
// carry explicit schemas with a CUDA implementation (the reference registers catch-all functions, which
// cannot be traced).
#include <ATen/Tensor.h>
#include <ATen/core/LegacyTypeDispatch.h>
#include <ATen/core/dispatch/Dispatcher.h>
#include <ATen/cuda/EmptyTensor.h>
#include <ATen/ops/empty.h>
#include <ATen/ops/zeros.h>
#include <ATen/record_function.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/library.h>

#include <vector>

#include "../../include/gnb200.h"
#include "gn_torch.h"

namespace {

constexpr int kF64 = 3;  // binding-internal code: double tensors go to the gnb200_*_f64 entry points

int dtype_code(const at::Tensor& t, const char* what) {
  switch (t.scalar_type()) {
    case at::kFloat: return GNB200_F32;
    case at::kHalf: return GNB200_F16;
    case at::kBFloat16: return GNB200_BF16;
    case at::kDouble: return kF64;
    default:
      TORCH_CHECK(false, "gnb200: ", what, " has dtype ", t.scalar_type(),
                  "; supported: float32, float16, bfloat16, float64");
  }
  return -1;
}

// Storage order of a logical (N, C, R) tensor: channels-last (strides (R*C, 1, C), the reference's
// layout, custom_gn.cpp:24,66-67) or channels-first (contiguous).  Anything else is refused.
enum Layout { kNHWC = 0, kNCHW = 1 };
Layout layout_of(const at::Tensor& t, const char* what) {
  TORCH_CHECK(t.device().is_cuda(), "gnb200: ", what, " must be a CUDA tensor (there is no CPU path)");
  TORCH_CHECK(t.dim() == 3, "gnb200: ", what, " must be a rank-3 (N, C, R) view, got rank ", t.dim());
  if (t.permute({0, 2, 1}).is_contiguous()) return kNHWC;
  TORCH_CHECK(t.is_contiguous(), "gnb200: ", what,
              " must be channels-last (strides (R*C, 1, C) for sizes (N, C, R)) or contiguous channels-first; got sizes ",
              t.sizes(), " strides ", t.strides());
  return kNCHW;
}

void check_param(const at::Tensor& p, const at::Tensor& like, int64_t C, const char* what) {
  TORCH_CHECK(p.device() == like.device(), "gnb200: ", what, " is on ", p.device(), " but the input is on ",
              like.device());
  TORCH_CHECK(p.scalar_type() == like.scalar_type(), "gnb200: ", what, " has dtype ", p.scalar_type(),
              " but the input has ", like.scalar_type());
  TORCH_CHECK(p.dim() == 1 && p.size(0) == C && p.is_contiguous(), "gnb200: ", what,
              " must be a contiguous vector of num_channels=", C, " elements, got sizes ", p.sizes());
}

// statistics are fp32 for fp32 / fp16 / bf16 tensors and fp64 for fp64 tensors
at::ScalarType stats_dtype(int dtype) { return dtype == kF64 ? at::kDouble : at::kFloat; }

void check_stats(const at::Tensor& s, const at::Tensor& like, int dtype, int64_t N, int64_t G, const char* what) {
  TORCH_CHECK(s.device() == like.device() && s.scalar_type() == stats_dtype(dtype) && s.is_contiguous() &&
                  s.dim() == 2 && s.size(0) == N && s.size(1) == G,
              "gnb200: ", what, " must be the contiguous (N, G) tensor returned by gnb200::fwd for this input");
}

void check_status(int rc) { TORCH_CHECK(rc == GNB200_OK, gnb200_last_error(), " (status ", rc, ")"); }

// a fresh tensor of X's logical sizes and storage order
at::Tensor empty_like_layout(const at::Tensor& X, Layout layout) {
  const int64_t N = X.size(0), C = X.size(1), R = X.size(2);
  return layout == kNHWC ? at::empty({N, R, C}, X.options()).permute({0, 2, 1}) : at::empty({N, C, R}, X.options());
}

std::tuple<at::Tensor, at::Tensor, at::Tensor> gnb200_fwd_op(const at::Tensor& X, const at::Tensor& weight,
                                                             const at::Tensor& bias, int64_t G, double eps,
                                                             int64_t act) {
  const Layout layout = layout_of(X, "X");
  const int64_t N = X.size(0), C = X.size(1), R = X.size(2);
  const int dtype = dtype_code(X, "X");
  check_param(weight, X, C, "weight");
  check_param(bias, X, C, "bias");
  TORCH_CHECK(G >= 1 && C % G == 0, "gnb200: num_channels ", C, " is not divisible by num_groups ", G);
  TORCH_CHECK(act >= 0 && act <= 4, "gnb200: activation code ", act, " is not in 0..4");
  c10::cuda::CUDAGuard guard(X.device());
  at::Tensor Y = empty_like_layout(X, layout);
  at::Tensor means = at::empty({N, G}, X.options().dtype(stats_dtype(dtype)));
  at::Tensor rstds = at::empty({N, G}, X.options().dtype(stats_dtype(dtype)));
  if (X.numel() == 0) return {Y, means, rstds};
  auto stream = c10::cuda::getCurrentCUDAStream().stream();
  if (dtype == kF64) {
    check_status(gnb200_fwd_f64(X.const_data_ptr<double>(), weight.const_data_ptr<double>(),
                                bias.const_data_ptr<double>(), N, R, C, G, eps, (int)act,
                                layout == kNHWC ? GNB200_LAYOUT_NHWC : GNB200_LAYOUT_NCHW, Y.mutable_data_ptr<double>(),
                                means.mutable_data_ptr<double>(), rstds.mutable_data_ptr<double>(), stream));
    return {Y, means, rstds};
  }
  const size_t ws_bytes = layout == kNHWC ? gnb200_fwd_workspace_bytes(N, R, C, G, dtype)
                                          : gnb200_fwd_nchw_workspace_bytes(N, R, C, G, dtype);
  at::Tensor ws;  // most forward plans need no scratch
  if (ws_bytes) ws = at::empty({(int64_t)ws_bytes}, X.options().dtype(at::kByte));
  auto fn = layout == kNHWC ? &gnb200_fwd : &gnb200_fwd_nchw;
  check_status(fn(X.const_data_ptr(), weight.const_data_ptr(), bias.const_data_ptr(), N, R, C, G, eps, (int)act, dtype,
                  Y.mutable_data_ptr(), means.mutable_data_ptr<float>(), rstds.mutable_data_ptr<float>(),
                  ws_bytes ? ws.mutable_data_ptr() : nullptr, ws_bytes, stream));
  return {Y, means, rstds};
}

// shared body of bwd / bwd_f32: (dX, packed [dgamma | dbeta], dweight, dbias)
std::tuple<at::Tensor, at::Tensor, at::Tensor, at::Tensor> bwd_impl(const at::Tensor& dy, const at::Tensor& X,
                                                                    const at::Tensor& weight, const at::Tensor& bias,
                                                                    const at::Tensor& means, const at::Tensor& rstds,
                                                                    int64_t G, int64_t act, bool want_typed,
                                                                    c10::ArrayRef<int64_t> peer_ptrs = {}, int64_t rank = 0) {
  const Layout layout = layout_of(X, "X");
  const int64_t N = X.size(0), C = X.size(1), R = X.size(2);
  const int dtype = dtype_code(X, "X");
  TORCH_CHECK(dy.sizes() == X.sizes() && dy.scalar_type() == X.scalar_type() && dy.device() == X.device(),
              "gnb200: dy must match X in sizes, dtype and device");
  TORCH_CHECK(X.numel() == 0 || layout_of(dy, "dy") == layout || C == 1 || R == 1,
              "gnb200: dy must have the storage order of X; got sizes ", dy.sizes(), " strides ", dy.strides());
  check_param(weight, X, C, "weight");
  check_param(bias, X, C, "bias");
  TORCH_CHECK(G >= 1 && C % G == 0, "gnb200: num_channels ", C, " is not divisible by num_groups ", G);
  TORCH_CHECK(act >= 0 && act <= 4, "gnb200: activation code ", act, " is not in 0..4");
  check_stats(means, X, dtype, N, G, "means");
  check_stats(rstds, X, dtype, N, G, "rstds");
  c10::cuda::CUDAGuard guard(X.device());
  at::Tensor dX = empty_like_layout(X, layout);
  // the packed fp32 sums: a result of their own, or - typed gradients - the tail of the scratch allocation
  const bool packed_in_scratch = want_typed && dtype != kF64 && X.numel() != 0;
  at::Tensor dparam, dweight, dbias;
  if (!packed_in_scratch) dparam = at::empty({2, C}, X.options().dtype(stats_dtype(dtype)));
  if (want_typed && dtype != kF64) {
    dweight = at::empty({C}, X.options());
    dbias = at::empty({C}, X.options());
  }
  if (X.numel() == 0) {
    dparam.zero_();
    if (want_typed) {
      dweight = at::zeros({C}, X.options());
      dbias = at::zeros({C}, X.options());
    }
    return {dX, dparam, dweight, dbias};
  }
  auto stream = c10::cuda::getCurrentCUDAStream().stream();
  // data-parallel ranks of one node: the sum over the ranks happens inside the library's kernels,
  // through the ranks' exchange buffers (peer_ptrs[q] = rank q's buffer as mapped into this process)
  const int world = (int)peer_ptrs.size();
  std::vector<const void*> peers(world);
  for (int q = 0; q < world; ++q) peers[q] = reinterpret_cast<const void*>(static_cast<uintptr_t>(peer_ptrs[q]));
  TORCH_CHECK(world == 0 || dtype != kF64, "gnb200: the in-kernel exchange of parameter gradients is for fp32 / fp16 / bf16 tensors");
  if (dtype == kF64) {
    // the packed buffer is the result: its two rows are dgamma and dbeta
    const size_t ws_bytes = gnb200_bwd_f64_workspace_bytes(N, R, C, G);
    at::Tensor ws = at::empty({(int64_t)ws_bytes}, X.options().dtype(at::kByte));
    double* dp = dparam.mutable_data_ptr<double>();
    check_status(gnb200_bwd_f64(dy.const_data_ptr<double>(), X.const_data_ptr<double>(), weight.const_data_ptr<double>(),
                                bias.const_data_ptr<double>(), means.const_data_ptr<double>(),
                                rstds.const_data_ptr<double>(), N, R, C, G, (int)act,
                                layout == kNHWC ? GNB200_LAYOUT_NHWC : GNB200_LAYOUT_NCHW, dX.mutable_data_ptr<double>(),
                                dp, dp + C, ws.mutable_data_ptr(), ws_bytes, stream));
    if (want_typed) {
      dweight = dparam[0];
      dbias = dparam[1];
    }
    return {dX, dparam, dweight, dbias};
  }
  const size_t ws_bytes = layout == kNHWC ? gnb200_bwd_workspace_bytes(N, R, C, G, dtype)
                                          : gnb200_bwd_nchw_workspace_bytes(N, R, C, G, dtype);
  const size_t ws_end = (ws_bytes + 15) & ~(size_t)15;
  at::Tensor ws = at::empty({(int64_t)(ws_end + (packed_in_scratch ? 2 * C * sizeof(float) : 0))}, X.options().dtype(at::kByte));
  float* dp32 = packed_in_scratch ? reinterpret_cast<float*>(ws.mutable_data_ptr<uint8_t>() + ws_end) : dparam.mutable_data_ptr<float>();
  void* dw = want_typed ? dweight.mutable_data_ptr() : nullptr;
  void* db = want_typed ? dbias.mutable_data_ptr() : nullptr;
  if (world > 1 && layout == kNHWC) {
    check_status(gnb200_bwd_peer(dy.const_data_ptr(), X.const_data_ptr(), weight.const_data_ptr(), bias.const_data_ptr(),
                                 means.const_data_ptr<float>(), rstds.const_data_ptr<float>(), N, R, C, G, (int)act, dtype,
                                 dX.mutable_data_ptr(), dp32, dw, db,
                                 ws_bytes ? ws.mutable_data_ptr() : nullptr, ws_bytes, peers.data(), (int)rank, world, stream));
    return {dX, dparam, dweight, dbias};
  }
  auto fn = layout == kNHWC ? &gnb200_bwd : &gnb200_bwd_nchw;
  check_status(fn(dy.const_data_ptr(), X.const_data_ptr(), weight.const_data_ptr(), bias.const_data_ptr(),
                  means.const_data_ptr<float>(), rstds.const_data_ptr<float>(), N, R, C, G, (int)act, dtype,
                  dX.mutable_data_ptr(), dp32, dw, db,
                  ws_bytes ? ws.mutable_data_ptr() : nullptr, ws_bytes, stream));
  if (world > 1)  // channels-first: the exchange follows the backward as a kernel of its own
    check_status(gnb200_allreduce_param_grads(dp32, dw, db, C, dtype, peers.data(), (int)rank,
                                              world, stream));
  return {dX, dparam, dweight, dbias};
}

std::tuple<at::Tensor, at::Tensor, at::Tensor> gnb200_bwd_op(const at::Tensor& dy, const at::Tensor& X,
                                                             const at::Tensor& weight, const at::Tensor& bias,
                                                             const at::Tensor& means, const at::Tensor& rstds,
                                                             int64_t G, int64_t act) {
  auto r = bwd_impl(dy, X, weight, bias, means, rstds, G, act, true);
  return {std::get<0>(r), std::get<2>(r), std::get<3>(r)};
}

std::tuple<at::Tensor, at::Tensor> gnb200_bwd_f32_op(const at::Tensor& dy, const at::Tensor& X,
                                                     const at::Tensor& weight, const at::Tensor& bias,
                                                     const at::Tensor& means, const at::Tensor& rstds, int64_t G,
                                                     int64_t act) {
  auto r = bwd_impl(dy, X, weight, bias, means, rstds, G, act, false);
  return {std::get<0>(r), std::get<1>(r)};
}

// bwd_f32 with the sum of the parameter gradients over the data-parallel ranks of one node done
// inside the kernels (gnb200_bwd_peer): peer_ptrs[q] is the address of rank q's exchange buffer in
// this process, `rank` this process's index in that list.
std::tuple<at::Tensor, at::Tensor> gnb200_bwd_f32_peer_op(const at::Tensor& dy, const at::Tensor& X,
                                                          const at::Tensor& weight, const at::Tensor& bias,
                                                          const at::Tensor& means, const at::Tensor& rstds, int64_t G,
                                                          int64_t act, c10::ArrayRef<int64_t> peer_ptrs, int64_t rank) {
  TORCH_CHECK(peer_ptrs.size() >= 1 && rank >= 0 && rank < (int64_t)peer_ptrs.size(),
              "gnb200: rank ", rank, " is not an index into the ", peer_ptrs.size(), " exchange buffers");
  auto r = bwd_impl(dy, X, weight, bias, means, rstds, G, act, false, peer_ptrs, rank);
  return {std::get<0>(r), std::get<1>(r)};
}

// ------------------------------------------------------------------------------------------------
// group_norm_act: flatten -> fwd -> restore with its autograd node, as one call.  What GN_NHWC_Func
// (gn_nhwc.py) does in Python, view for view and op for op (the inner ops go through the dispatcher, so dispatch
// modes see them), without the interpreter: on small maps a training step is bound by that (the Python node
// alone, with its backward waiting for the interpreter lock in the engine's thread, took most of 150 us).
// ------------------------------------------------------------------------------------------------
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

// the reference's layout rule (custom_gn.py:68): unit channel stride means channels-last
bool is_channels_last(const at::Tensor& t) { return t.stride(1) == 1 || t.size(1) == 1; }

at::Tensor flatten(const at::Tensor& t, bool channels_last) {
  const int64_t n = t.size(0), c = t.size(1), nd = t.dim();
  if (!channels_last) return t.contiguous().reshape({n, c, -1});
  at::DimVector dims = {0};
  for (int64_t d = 2; d < nd; ++d) dims.push_back(d);
  dims.push_back(1);
  return t.permute(dims).contiguous().reshape({n, -1, c}).permute({0, 2, 1});
}

at::Tensor restore(const at::Tensor& flat, at::IntArrayRef shape, bool channels_last) {
  if (!channels_last) return flat.reshape(shape);
  at::DimVector sizes = {shape[0]}, dims = {0, (int64_t)shape.size() - 1};
  for (size_t d = 2; d < shape.size(); ++d) sizes.push_back(shape[d]), dims.push_back((int64_t)d - 1);
  sizes.push_back(shape[1]);
  return flat.permute({0, 2, 1}).reshape(sizes).permute(dims);
}

at::Tensor as_dtype(const at::Tensor& t, at::ScalarType dtype) { return t.scalar_type() == dtype ? t : t.to(dtype); }

std::tuple<at::Tensor, at::Tensor, at::Tensor> call_fwd(const at::Tensor& X, const at::Tensor& w, const at::Tensor& b, int64_t G,
                                                        double eps, int64_t act) {
  static const auto op = c10::Dispatcher::singleton().findSchemaOrThrow("gnb200::fwd", "").typed<decltype(gnb200_fwd_op)>();
  at::AutoDispatchBelowADInplaceOrView guard;
  return op.call(X, w, b, G, eps, act);
}

// ------------------------------------------------------------------------------------------------
// The same without views and inner dispatches, for plain calls.  A small call is bound by the host: of 19.5 us for one
// without gradients about half went into seven view ops, the second dispatch, three allocations and the autograd node that
// nothing needed.  A call is plain when nothing but autograd and CUDA kernels would see its ops (no dispatch mode, functorch
// transform, tracer, lazy negation, profiler) and its tensor has the storage order that the kernels want; every other call
// goes through the ops as before.  The kernels, their arguments and the results' sizes and strides are the same.
// ------------------------------------------------------------------------------------------------
bool only_cuda_sees(std::initializer_list<const at::Tensor*> tensors) {
  static const c10::DispatchKeySet allowed =
      c10::autograd_dispatch_keyset_with_ADInplaceOrView | c10::autocast_dispatch_keyset |
      c10::DispatchKeySet({c10::DispatchKey::BackendSelect, c10::DispatchKey::CUDA, c10::DispatchKey::AutogradCUDA});
  c10::DispatchKeySet ks;
  for (const at::Tensor* t : tensors) ks = ks | t->key_set();
  const auto tls = c10::impl::tls_local_dispatch_key_set();
  ks = (ks | tls.included_) - tls.excluded_;
  return (ks.raw_repr() & ~allowed.raw_repr()) == 0 && !at::hasCallbacks();
}

// Storage of a plain tensor of rank >= 3, by the rules of flatten() and layout_of(); false where it would be copied.
struct Dense {
  bool channels_last;  // by is_channels_last(): decides the strides of results
  Layout layout;
  int64_t N, C, R;
};
bool dense_order(const at::Tensor& t, bool channels_last) {
  if (!channels_last) return t.is_contiguous();
  const auto sizes = t.sizes(), strides = t.strides();
  if (sizes[1] != 1 && strides[1] != 1) return false;
  int64_t want = sizes[1];
  for (int64_t d = t.dim() - 1; d >= 2; --d) {
    if (sizes[d] != 1 && strides[d] != want) return false;
    want *= sizes[d];
  }
  return sizes[0] == 1 || strides[0] == want;
}
bool plain_tensor(const at::Tensor& t, Dense* out) {
  if (t.dim() < 3 || t.numel() == 0 || !t.is_cuda()) return false;
  const auto st = t.scalar_type();
  if (st != at::kFloat && st != at::kHalf && st != at::kBFloat16) return false;
  const bool cl = is_channels_last(t);
  if (!dense_order(t, cl)) return false;
  const int64_t n = t.size(0), c = t.size(1), r = t.numel() / (n * c);
  *out = Dense{cl, cl || r == 1 ? kNHWC : kNCHW, n, c, r};
  return true;
}
// What flatten() gives for a plain tensor: the same storage and version counter, no graph, none of its own dispatches.
at::Tensor flat_alias(const at::Tensor& t, const Dense& d) {
  auto* impl = t.unsafeGetTensorImpl();
  auto flat = impl->shallow_copy_and_detach(impl->version_counter(), /*allow_tensor_metadata_change=*/true);
  const int64_t sizes[] = {d.N, d.C, d.R};
  const int64_t strides[] = {d.R * d.C, d.channels_last ? 1 : d.R, d.channels_last ? d.C : 1};
  flat->set_sizes_and_strides(sizes, strides);
  return at::Tensor(std::move(flat));
}
// uninitialised, with the strides that restore() gives
at::Tensor empty_result(const at::Tensor& like, at::IntArrayRef sizes, const Dense& d) {
  at::DimVector strides(sizes.size());
  int64_t step = d.channels_last ? d.C : 1;
  for (int64_t i = (int64_t)sizes.size() - 1; i >= 2; --i) strides[i] = step, step *= sizes[i];
  strides[1] = d.channels_last ? 1 : step;
  strides[0] = d.channels_last ? step : step * d.C;
  return at::detail::empty_strided_cuda(sizes, strides, like.scalar_type(), like.device());
}
at::Tensor empty_vector(std::initializer_list<int64_t> sizes, at::ScalarType st, const at::Tensor& like) {
  return at::detail::empty_cuda(at::IntArrayRef(sizes.begin(), sizes.size()), st, like.device(), std::nullopt);
}

// The parameters in X's dtype: themselves, or both rounded from fp32 in one launch, or as as_dtype() does it.
void params_like(const at::Tensor& X, const Dense& d, at::Tensor& w, at::Tensor& b) {
  const at::ScalarType st = X.scalar_type();
  auto fp32_vector = [&](const at::Tensor& p) {
    return p.scalar_type() == at::kFloat && p.dim() == 1 && p.size(0) == d.C && p.is_contiguous() && p.device() == X.device();
  };
  if (st == at::kFloat || !fp32_vector(w) || !fp32_vector(b)) {
    w = as_dtype(w, st);
    b = as_dtype(b, st);
    return;
  }
  c10::cuda::CUDAGuard guard(X.device());
  at::Tensor wc = empty_vector({d.C}, st, X), bc = empty_vector({d.C}, st, X);
  check_status(gnb200_cast_params(w.const_data_ptr<float>(), b.const_data_ptr<float>(), d.C, dtype_code(X, "X"), wc.mutable_data_ptr(),
                                  bc.mutable_data_ptr(), c10::cuda::getCurrentCUDAStream().stream()));
  w = wc;
  b = bc;
}

// Y; where `means` is given the statistics are results too, otherwise they share the scratch.
at::Tensor direct_fwd(const at::Tensor& X, const Dense& d, const at::Tensor& weight, const at::Tensor& bias, int64_t G, double eps,
                      int64_t act, at::Tensor* means, at::Tensor* rstds) {
  const int dtype = dtype_code(X, "X");
  check_param(weight, X, d.C, "weight");
  check_param(bias, X, d.C, "bias");
  TORCH_CHECK(G >= 1 && d.C % G == 0, "gnb200: num_channels ", d.C, " is not divisible by num_groups ", G);
  TORCH_CHECK(act >= 0 && act <= 4, "gnb200: activation code ", act, " is not in 0..4");
  c10::cuda::CUDAGuard guard(X.device());
  at::Tensor Y = empty_result(X, X.sizes(), d);
  const size_t ws_bytes = d.layout == kNHWC ? gnb200_fwd_workspace_bytes(d.N, d.R, d.C, G, dtype)
                                            : gnb200_fwd_nchw_workspace_bytes(d.N, d.R, d.C, G, dtype);
  const size_t ws_end = (ws_bytes + 15) & ~(size_t)15, stat_bytes = (size_t)d.N * G * sizeof(float);
  at::Tensor ws;
  float *mean, *rstd;
  if (means) {
    *means = empty_vector({d.N, G}, at::kFloat, X);
    *rstds = empty_vector({d.N, G}, at::kFloat, X);
    mean = means->mutable_data_ptr<float>();
    rstd = rstds->mutable_data_ptr<float>();
    if (ws_bytes) ws = empty_vector({(int64_t)ws_bytes}, at::kByte, X);
  } else {
    ws = empty_vector({(int64_t)(ws_end + 2 * stat_bytes)}, at::kByte, X);
    mean = reinterpret_cast<float*>(ws.mutable_data_ptr<uint8_t>() + ws_end);
    rstd = mean + d.N * G;
  }
  auto fn = d.layout == kNHWC ? &gnb200_fwd : &gnb200_fwd_nchw;
  check_status(fn(X.const_data_ptr(), weight.const_data_ptr(), bias.const_data_ptr(), d.N, d.R, d.C, G, eps, (int)act, dtype,
                  Y.mutable_data_ptr(), mean, rstd, ws_bytes ? ws.mutable_data_ptr() : nullptr, ws_bytes,
                  c10::cuda::getCurrentCUDAStream().stream()));
  return Y;
}

// X: flat.  typed: dgamma, dbeta in X's dtype; otherwise the two rows of one fp32 tensor
void direct_bwd(const at::Tensor& dy, const at::Tensor& X, const Dense& d, const at::Tensor& weight, const at::Tensor& bias,
                const at::Tensor& means, const at::Tensor& rstds, int64_t G, int64_t act, bool typed, at::Tensor* dx,
                at::Tensor* dgamma, at::Tensor* dbeta) {
  const int dtype = dtype_code(X, "X");
  check_param(weight, X, d.C, "weight");
  check_param(bias, X, d.C, "bias");
  check_stats(means, X, dtype, d.N, G, "means");
  check_stats(rstds, X, dtype, d.N, G, "rstds");
  c10::cuda::CUDAGuard guard(X.device());
  *dx = empty_result(X, dy.sizes(), d);
  const size_t ws_bytes = d.layout == kNHWC ? gnb200_bwd_workspace_bytes(d.N, d.R, d.C, G, dtype)
                                            : gnb200_bwd_nchw_workspace_bytes(d.N, d.R, d.C, G, dtype);
  const size_t ws_end = (ws_bytes + 15) & ~(size_t)15;
  at::Tensor ws = empty_vector({(int64_t)(ws_end + (typed ? 2 * d.C * sizeof(float) : 0))}, at::kByte, X), dparam;
  float* dp32;
  if (typed) {
    dp32 = reinterpret_cast<float*>(ws.mutable_data_ptr<uint8_t>() + ws_end);
    *dgamma = empty_vector({d.C}, X.scalar_type(), X);
    *dbeta = empty_vector({d.C}, X.scalar_type(), X);
  } else {
    dparam = empty_vector({2, d.C}, at::kFloat, X);
    dp32 = dparam.mutable_data_ptr<float>();
  }
  auto fn = d.layout == kNHWC ? &gnb200_bwd : &gnb200_bwd_nchw;
  check_status(fn(dy.const_data_ptr(), X.const_data_ptr(), weight.const_data_ptr(), bias.const_data_ptr(),
                  means.const_data_ptr<float>(), rstds.const_data_ptr<float>(), d.N, d.R, d.C, G, (int)act, dtype,
                  dx->mutable_data_ptr(), dp32, typed ? dgamma->mutable_data_ptr() : nullptr,
                  typed ? dbeta->mutable_data_ptr() : nullptr, ws_bytes ? ws.mutable_data_ptr() : nullptr, ws_bytes,
                  c10::cuda::getCurrentCUDAStream().stream()));
  if (!typed) {
    *dgamma = dparam.select(0, 0);
    *dbeta = dparam.select(0, 1);
  }
}

struct GnFunction : torch::autograd::Function<GnFunction> {
  // everything that backward uses is saved through ctx, and it calls dispatcher ops only: compiled autograd may trace it
  static constexpr bool is_traceable = true;

  static at::Tensor forward(AutogradContext* ctx, const at::Tensor& X, const at::Tensor& weight, const at::Tensor& bias,
                            int64_t G, double eps, int64_t act) {
    const bool cl = is_channels_last(X);
    at::Tensor w = weight, b = bias;
    Dense d;
    const bool plain = only_cuda_sees({&X, &w, &b}) && plain_tensor(X, &d);
    ctx->saved_data["arg"] =
        std::vector<int64_t>{G, act, cl ? 1 : 0, (int64_t)weight.scalar_type(), (int64_t)bias.scalar_type(), plain ? 1 : 0};
    ctx->saved_data["shape"] = X.sizes().vec();
    // The flat tensor is saved on either path, not X: hooks and the checks of a checkpoint's recomputation, which may take the
    // other path (a profiler started since), meet the same sizes, and X may be given other data.
    if (plain) {
      params_like(X, d, w, b);
      at::Tensor means, rstds;
      at::Tensor Y = direct_fwd(X, d, w, b, G, eps, act, &means, &rstds);
      ctx->save_for_backward({flat_alias(X, d), w, b, means, rstds});
      return Y;
    }
    w = as_dtype(weight, X.scalar_type());
    b = as_dtype(bias, X.scalar_type());
    const at::Tensor Xf = flatten(X, cl);
    auto [Y, means, rstds] = call_fwd(Xf, w, b, G, eps, act);
    ctx->save_for_backward({Xf, w, b, means, rstds});
    return restore(Y, X.sizes(), cl);
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    static const auto op = c10::Dispatcher::singleton().findSchemaOrThrow("gnb200::bwd", "").typed<decltype(gnb200_bwd_op)>();
    static const auto op32 =
        c10::Dispatcher::singleton().findSchemaOrThrow("gnb200::bwd_f32", "").typed<decltype(gnb200_bwd_f32_op)>();
    const auto saved = ctx->get_saved_variables();
    const auto shape = ctx->saved_data["shape"].toIntVector(), arg = ctx->saved_data["arg"].toIntVector();
    const bool cl = arg[2] != 0;
    const at::ScalarType dtype = saved[0].scalar_type();
    const auto w_dtype = (at::ScalarType)arg[3], b_dtype = (at::ScalarType)arg[4];
    at::Tensor dx, dgamma, dbeta;
    const at::Tensor& g = grads[0];
    Dense d;
    if (arg[5] != 0 && !c10::GradMode::is_enabled() && g.defined() &&
        only_cuda_sees({&g, &saved[0], &saved[1], &saved[2], &saved[3], &saved[4]}) && plain_tensor(saved[0], &d) &&
        dense_order(saved[0], cl) && g.scalar_type() == dtype && g.device() == saved[0].device() &&
        g.sizes() == at::IntArrayRef(shape) && dense_order(g, cl)) {
      d.channels_last = cl;  // (of the flat tensor's strides, one row or channel leaves it open)
      d.layout = cl || d.R == 1 ? kNHWC : kNCHW;
      const bool typed = w_dtype == dtype && b_dtype == dtype;
      direct_bwd(g, saved[0], d, saved[1], saved[2], saved[3], saved[4], arg[0], arg[1], typed, &dx, &dgamma, &dbeta);
      return {dx, as_dtype(dgamma, w_dtype), as_dtype(dbeta, b_dtype), at::Tensor(), at::Tensor(), at::Tensor()};
    }
    // (flat already; a hook may have brought it back in another storage order)
    const at::Tensor Xf = flatten(saved[0], cl);
    const at::Tensor dy = as_dtype(flatten(g, cl), dtype);
    if (w_dtype == dtype && b_dtype == dtype) {
      std::tie(dx, dgamma, dbeta) = op.call(dy, Xf, saved[1], saved[2], saved[3], saved[4], arg[0], arg[1]);
    } else {
      at::Tensor dparam;
      std::tie(dx, dparam) = op32.call(dy, Xf, saved[1], saved[2], saved[3], saved[4], arg[0], arg[1]);
      dgamma = dparam.select(0, 0).to(w_dtype);
      dbeta = dparam.select(0, 1).to(b_dtype);
    }
    return {restore(dx, shape, cl), dgamma, dbeta, at::Tensor(), at::Tensor(), at::Tensor()};
  }
};

at::Tensor group_norm_act_autograd(const at::Tensor& X, const at::Tensor& weight, const at::Tensor& bias, int64_t G, double eps,
                                   int64_t act) {
  return GnFunction::apply(X, weight, bias, G, eps, act);
}

// below autograd (inference mode)
at::Tensor group_norm_act_plain(const at::Tensor& X, const at::Tensor& weight, const at::Tensor& bias, int64_t G, double eps,
                                int64_t act) {
  const bool cl = is_channels_last(X);
  const at::Tensor Y = std::get<0>(call_fwd(flatten(X, cl), as_dtype(weight, X.scalar_type()), as_dtype(bias, X.scalar_type()), G,
                                            eps, act));
  return restore(Y, X.sizes(), cl);
}

}  // namespace

at::Tensor gnb200_ops::group_norm_act_direct(const at::Tensor& X, const at::Tensor& weight, const at::Tensor& bias, int64_t G,
                                             double eps, int64_t act) {
  Dense d;
  if (!only_cuda_sees({&X, &weight, &bias}) || !plain_tensor(X, &d)) return at::Tensor();
  for (const at::Tensor* t : {&X, &weight, &bias})
    if (t->_fw_grad(0).defined()) return at::Tensor();  // dual tensors
  if (c10::GradMode::is_enabled() && (X.requires_grad() || weight.requires_grad() || bias.requires_grad()))
    return GnFunction::apply(X, weight, bias, G, eps, act);
  at::AutoDispatchBelowADInplaceOrView guard;
  at::Tensor w = weight, b = bias;
  params_like(X, d, w, b);
  return direct_fwd(X, d, w, b, G, eps, act, nullptr, nullptr);
}

// Schemas are declared apart from the implementations so that Python can attach fake-tensor
// kernels and an autograd formula to them (channels_last_groupnorm_b200/_compile.py), which is what
// torch.compile needs.  The CPU registration exists only to fail with the message of check_nhwc3
// instead of the dispatcher's.
TORCH_LIBRARY(gnb200, m) {
  m.def("fwd(Tensor X, Tensor weight, Tensor bias, int G, float eps, int act) -> (Tensor, Tensor, Tensor)");
  m.def("bwd(Tensor dy, Tensor X, Tensor weight, Tensor bias, Tensor means, Tensor rstds, int G, int act) -> "
        "(Tensor, Tensor, Tensor)");
  m.def("bwd_f32(Tensor dy, Tensor X, Tensor weight, Tensor bias, Tensor means, Tensor rstds, int G, int act) -> "
        "(Tensor, Tensor)");
  m.def("bwd_f32_peer(Tensor dy, Tensor X, Tensor weight, Tensor bias, Tensor means, Tensor rstds, int G, int act, "
        "int[] peer_ptrs, int rank) -> (Tensor, Tensor)");
  m.def("group_norm_act(Tensor X, Tensor weight, Tensor bias, int G, float eps, int act) -> Tensor");
}

TORCH_LIBRARY_IMPL(gnb200, Autograd, m) { m.impl("group_norm_act", &group_norm_act_autograd); }

TORCH_LIBRARY_IMPL(gnb200, CUDA, m) {
  m.impl("fwd", &gnb200_fwd_op);
  m.impl("bwd", &gnb200_bwd_op);
  m.impl("bwd_f32", &gnb200_bwd_f32_op);
  m.impl("bwd_f32_peer", &gnb200_bwd_f32_peer_op);
  m.impl("group_norm_act", &group_norm_act_plain);
}

TORCH_LIBRARY_IMPL(gnb200, CPU, m) {
  m.impl("fwd", &gnb200_fwd_op);
  m.impl("bwd", &gnb200_bwd_op);
  m.impl("bwd_f32", &gnb200_bwd_f32_op);
}
