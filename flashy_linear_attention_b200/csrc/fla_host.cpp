// Host side of one forward / backward call on torch tensors: checks, output and scratch tensors,
// argument block and the C-ABI call, in one native function each. Python's part of a call is then a
// few attribute reads; doing the same through torch's Python API and ctypes (about 45 stride reads,
// 40 structure fields and four device guards) took longer than the kernels of a small layer: a
// training step of 8 heads x 256 x 64 took 195 us that way, 95 us this way (18 us of kernels).
//
// Both functions return None for calls they do not cover (wrong types, shapes that do not match,
// head dims above 384, running states with head dims above 128): the caller then takes the general path in
// ops.py, which reports the errors and handles the rest. The interpreter lock is given up while they
// work, as ctypes does: an allocation or a full launch queue can block, and other Python threads, that
// drive other streams or GPUs, have to go on meanwhile.
#include <torch/extension.h>

#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>

#include <algorithm>
#include <array>
#include <optional>
#include <string>
#include <vector>

#include "../../include/flashlinear_sm100.h"

namespace {

namespace py = pybind11;
using at::Tensor;
using OptTensor = std::optional<Tensor>;

constexpr int64_t kKernelHeadDim = 128;  // widest head dim of the running-state kernels
constexpr int64_t kWideHeadDim = 384;    // widest head dim one library call covers

// What a TMA tensor map needs: unit innermost stride, 16-byte aligned base and outer strides. The row
// stride counts even where there is one row: the library checks it without looking at the length.
bool addressable(const Tensor& t) {
  if (t.stride(3) != 1 || reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 != 0 ||
      t.stride(2) < (t.size(3) + 7) / 8 * 8 || t.stride(2) % 8 != 0)
    return false;
  for (int d = 0; d < 2; ++d)
    if (t.size(d) > 1 && t.stride(d) % 8 != 0) return false;
  return true;
}

bool usable(const Tensor& t, const Tensor& ref) {
  return t.layout() == at::kStrided && t.dim() == 4 && t.is_cuda() && t.device() == ref.device() &&
         t.scalar_type() == ref.scalar_type() && !t.is_neg();
}

bool same_rows(const Tensor& a, const Tensor& b) {  // batch, heads, tokens
  return a.size(0) == b.size(0) && a.size(1) == b.size(1) && a.size(2) == b.size(2);
}

bool is_state(const OptTensor& s, const Tensor& ref, int64_t bh, int64_t dk, int64_t dv) {
  return !s.has_value() || (s->is_cuda() && s->device() == ref.device() && s->scalar_type() == at::kFloat &&
                            s->is_contiguous() && s->dim() == 3 && s->size(0) == bh && s->size(1) == dk &&
                            s->size(2) == dv);
}

FlaTensor desc(const Tensor& t) {
  FlaTensor d;
  d.ptr = t.data_ptr();
  d.stride_b = t.stride(0);
  d.stride_h = t.stride(1);
  d.stride_n = t.stride(2);
  return d;
}

// View [..., :d] of a fresh tensor whose rows are padded to a multiple of 8 elements.
Tensor padded_empty(const Tensor& like) {
  const int64_t d = like.size(3);
  return at::empty({like.size(0), like.size(1), like.size(2), (d + 7) / 8 * 8}, like.options()).narrow(3, 0, d);
}

// empty_like() of a tensor of these sizes and strides that is not at hand any more.
Tensor empty_like_of(const Tensor& sizes_of, at::IntArrayRef strides) {
  const at::IntArrayRef sizes = sizes_of.sizes();
  // strides without gaps or overlaps are kept as they are: walk the dimensions from the inside out
  int order[4] = {3, 2, 1, 0};
  std::stable_sort(order, order + 4, [&](int a, int b) { return strides[a] < strides[b]; });
  int64_t next = 1;
  bool dense = true;
  for (int d : order) {
    if (sizes[d] == 1) continue;
    dense = dense && strides[d] == next;
    next *= sizes[d];
  }
  if (dense) return at::empty_strided(sizes, strides, sizes_of.options());
  return at::empty_like(at::empty_strided(sizes, strides, sizes_of.options().device(at::kMeta)), sizes_of.options());
}

void check(int rc, const char* name) {
  if (rc != FLA_OK)
    throw std::runtime_error(std::string("flashlinear: ") + name + " returned " + std::to_string(rc) + ": " +
                             fla_sm100_strerror(rc));
}

// The library's pad / unpad kernels work on contiguous tensors of any row length.
bool contiguous_rows(const Tensor& t) {
  return t.is_contiguous() && reinterpret_cast<uintptr_t>(t.data_ptr()) % 4 == 0;
}

// Replaces every tensor the kernels cannot address in place by a copy with padded rows. Contiguous
// tensors of one row length share a launch of the pad kernel.
void kernel_views(Tensor* t, int n, void* stream) {
  constexpr int kMax = 4;
  const void* src[kMax];
  void* dst[kMax];
  Tensor copies[kMax];
  bool done[kMax] = {};
  for (int i = 0; i < n; ++i) {
    if (addressable(t[i])) done[i] = true;
    else copies[i] = padded_empty(t[i]);
    if (!done[i] && !contiguous_rows(t[i])) {
      copies[i].copy_(t[i]);
      done[i] = true;
    }
  }
  for (int i = 0; i < n; ++i) {
    if (done[i]) continue;
    int count = 0;
    for (int j = i; j < n; ++j) {
      if (done[j] || t[j].size(3) != t[i].size(3)) continue;
      src[count] = t[j].data_ptr();
      dst[count++] = copies[j].data_ptr();
      done[j] = true;
    }
    check(fla_sm100_pad_rows_batch(src, dst, count, t[i].numel() / t[i].size(3), static_cast<int>(t[i].size(3)),
                                   static_cast<int>(copies[i].stride(2)), stream),
          "fla_sm100_pad_rows_batch");
  }
  for (int i = 0; i < n; ++i)
    if (copies[i].defined()) t[i] = copies[i];
}

// An output with the layout of empty_like(t) and what the kernel writes to: the output itself, or a
// row-padded scratch tensor that is copied back. keep_padded: the padded tensor IS the output.
struct Output {
  Tensor full, view;
};
Output output_like(const Tensor& t, bool keep_padded, const std::vector<int64_t>* strides) {
  Output o;
  if (keep_padded && t.size(3) % 8 != 0) {
    o.full = o.view = padded_empty(t);
    return o;
  }
  o.full = strides != nullptr ? empty_like_of(t, *strides) : at::empty_like(t);
  o.view = addressable(o.full) ? o.full : padded_empty(o.full);
  return o;
}
// Results from the padded scratch rows into the caller-layout outputs, grouped like kernel_views().
void copy_back(const Output* o, int n, void* stream) {
  constexpr int kMax = 4;
  const void* src[kMax];
  void* dst[kMax];
  bool done[kMax] = {};
  for (int i = 0; i < n; ++i) {
    done[i] = o[i].view.is_same(o[i].full);
    if (!done[i] && !contiguous_rows(o[i].full)) {
      o[i].full.copy_(o[i].view);
      done[i] = true;
    }
  }
  for (int i = 0; i < n; ++i) {
    if (done[i]) continue;
    int count = 0;
    const int64_t d = o[i].full.size(3);
    for (int j = i; j < n; ++j) {
      if (done[j] || o[j].full.size(3) != d) continue;
      src[count] = o[j].view.data_ptr();
      dst[count++] = o[j].full.data_ptr();
      done[j] = true;
    }
    check(fla_sm100_unpad_rows_batch(src, dst, count, o[i].full.numel() / d, static_cast<int>(d),
                                     static_cast<int>(o[i].view.stride(2)), stream),
          "fla_sm100_unpad_rows_batch");
  }
}

bool covered_dims(const Tensor& q, const Tensor& v) {
  if (q.numel() == 0 || v.numel() == 0) return false;
  if (q.size(0) > INT32_MAX || q.size(1) > INT32_MAX || q.size(2) > INT32_MAX) return false;
  const int64_t m = std::max(q.size(3), v.size(3));
  if (q.scalar_type() == at::kBFloat16) return m <= kWideHeadDim;
  return q.scalar_type() == at::kHalf && m <= kKernelHeadDim;
}

void set_sizes(FlaArgs& a, const Tensor& q, const Tensor& v, unsigned debug_flags, uintptr_t status) {
  a = FlaArgs{};
  a.batch = static_cast<int32_t>(q.size(0));
  a.heads = static_cast<int32_t>(q.size(1));
  a.seqlen = static_cast<int32_t>(q.size(2));
  a.dk = static_cast<int32_t>(q.size(3));
  a.dv = static_cast<int32_t>(v.size(3));
  a.dtype = q.scalar_type() == at::kHalf ? FLA_DTYPE_F16 : FLA_DTYPE_BF16;
  a.debug_flags = debug_flags;
  a.status = reinterpret_cast<int32_t*>(status);
}

Tensor scratch(FlaArgs& a, int pass, const Tensor& ref) {
  const size_t need = fla_sm100_workspace_bytes(&a, pass);
  if (need == 0) return Tensor();
  Tensor ws = at::empty({static_cast<int64_t>(need)}, ref.options().dtype(at::kByte));
  a.workspace = ws.data_ptr();
  a.workspace_bytes = need;
  return ws;
}

// views: with state 2, the q, k, v the kernels read where
// one of them had to be repacked, for the backward of the same call.
// state: 0 none; 1 always return the final state, [B, H, dk, dv]; 2 return what the backward of
// these shapes uses (final state and boundary states, each a tensor or None).
struct Forward {
  Tensor out;
  OptTensor s_final, seg_states;
  std::optional<std::array<Tensor, 3>> views;
};
std::optional<Forward> forward(const Tensor& q, const Tensor& k, const Tensor& v, const OptTensor& s_init, int state,
                               unsigned debug_flags, uintptr_t status) {
  if (!usable(q, q) || !usable(k, q) || !usable(v, q) || !covered_dims(q, v) || !same_rows(q, k) ||
      !same_rows(q, v) || q.size(3) != k.size(3))
    return std::nullopt;
  const int64_t bh = q.size(0) * q.size(1), dk = q.size(3), dv = v.size(3);
  const bool wide = dk > kKernelHeadDim || dv > kKernelHeadDim;
  if (wide && (s_init.has_value() || state == 1)) return std::nullopt;
  if (!is_state(s_init, q, bh, dk, dv)) return std::nullopt;
  const c10::cuda::CUDAGuard guard(q.device());
  void* stream = c10::cuda::getCurrentCUDAStream(q.device().index()).stream();
  const Output out = output_like(v, false, nullptr);
  Tensor in[3] = {q, k, v};
  kernel_views(in, 3, stream);
  FlaArgs a;
  set_sizes(a, q, v, debug_flags, status);
  a.stream = stream;
  OptTensor s_final, seg_states;
  if (!wide && (state == 1 || (state == 2 && fla_sm100_bwd_uses_final_state(&a) != 0))) {
    s_final = state == 1 ? at::empty({q.size(0), q.size(1), dk, dv}, q.options().dtype(at::kFloat))
                         : at::empty({bh, dk, dv}, q.options().dtype(at::kFloat));
    if (state == 2) {
      const size_t need = fla_sm100_seg_states_bytes(&a);
      if (need > 0) {
        seg_states = at::empty({static_cast<int64_t>(need)}, q.options().dtype(at::kByte));
        a.seg_states = seg_states->data_ptr();
        a.seg_states_bytes = need;
      }
    }
  }
  a.q = desc(in[0]);
  a.k = desc(in[1]);
  a.v = desc(in[2]);
  a.o = desc(out.view);
  if (s_init.has_value()) a.s_init = s_init->data_ptr<float>();
  if (s_final.has_value()) a.s_final = s_final->data_ptr<float>();
  const Tensor ws = scratch(a, 0, q);
  check(fla_sm100_fwd(&a), "libflashlinear_sm100");
  copy_back(&out, 1, stream);
  Forward res{out.full, s_final, seg_states, std::nullopt};
  if (state == 2 && !(in[0].is_same(q) && in[1].is_same(k) && in[2].is_same(v)))
    res.views = std::array<Tensor, 3>{in[0], in[1], in[2]};
  return res;
}

// strides: those of the three tensors that q, k, v are repacked copies of; the gradients take their layout.
using Strides = std::optional<std::array<std::vector<int64_t>, 3>>;
std::optional<std::array<Tensor, 3>> backward(const Tensor& g, const Tensor& q, const Tensor& k, const Tensor& v,
                                              const OptTensor& s_last, const OptTensor& seg_states, bool keep_padded,
                                              const Strides& strides, unsigned debug_flags, uintptr_t status) {
  Tensor in[4] = {q, k, v, g};
  for (const Tensor& t : in)
    if (!usable(t, q) || !same_rows(t, q)) return std::nullopt;
  if (!covered_dims(q, v) || q.size(3) != k.size(3) || g.size(3) != v.size(3)) return std::nullopt;
  if (strides.has_value())
    for (const auto& s : *strides)
      if (s.size() != 4) return std::nullopt;
  const int64_t bh = q.size(0) * q.size(1), dk = q.size(3), dv = v.size(3);
  if ((dk > kKernelHeadDim || dv > kKernelHeadDim) && s_last.has_value()) return std::nullopt;
  if (!is_state(s_last, g, bh, dk, dv)) return std::nullopt;
  const c10::cuda::CUDAGuard guard(g.device());
  void* stream = c10::cuda::getCurrentCUDAStream(g.device().index()).stream();
  Output out[3];
  for (int i = 0; i < 3; ++i) out[i] = output_like(in[i], keep_padded, strides.has_value() ? &(*strides)[i] : nullptr);
  kernel_views(in, 4, stream);
  FlaArgs a;
  set_sizes(a, q, v, debug_flags, status);
  a.stream = stream;
  a.q = desc(in[0]);
  a.k = desc(in[1]);
  a.v = desc(in[2]);
  a.d_o = desc(in[3]);
  a.d_q = desc(out[0].view);
  a.d_k = desc(out[1].view);
  a.d_v = desc(out[2].view);
  if (s_last.has_value()) a.s_last = s_last->data_ptr<float>();
  if (seg_states.has_value()) {
    a.seg_states = seg_states->data_ptr();
    a.seg_states_bytes = static_cast<size_t>(seg_states->numel() * seg_states->element_size());
  }
  const Tensor ws = scratch(a, 1, g);
  check(fla_sm100_bwd(&a), "libflashlinear_sm100");
  copy_back(out, 3, stream);
  return std::array<Tensor, 3>{out[0].full, out[1].full, out[2].full};
}

// Attention on the Taylor features of raw q, k.
bool taylor_covered(const Tensor& q, const Tensor& k, const Tensor& v) {
  const int64_t d = q.dim() == 4 ? q.size(3) : 0, dv = v.dim() == 4 ? v.size(3) : 0;
  return usable(q, q) && usable(k, q) && usable(v, q) && same_rows(q, k) && same_rows(q, v) && k.size(3) == d &&
         (d == 8 || d == 16) && (dv == 8 || dv == 16 || dv == 32 || dv == 64) && q.scalar_type() == at::kBFloat16 && covered_dims(q, v);
}
std::optional<Tensor> taylor_forward(const Tensor& q, const Tensor& k, const Tensor& v, unsigned debug_flags, uintptr_t status) {
  if (!taylor_covered(q, k, v)) return std::nullopt;
  const c10::cuda::CUDAGuard guard(q.device());
  void* stream = c10::cuda::getCurrentCUDAStream(q.device().index()).stream();
  const Output out = output_like(v, false, nullptr);
  Tensor in[3] = {q, k, v};
  kernel_views(in, 3, stream);
  FlaArgs a;
  set_sizes(a, q, v, debug_flags, status);
  a.stream = stream;
  a.q = desc(in[0]);
  a.k = desc(in[1]);
  a.v = desc(in[2]);
  a.o = desc(out.view);
  check(fla_sm100_taylor_fwd(&a), "fla_sm100_taylor_fwd");
  copy_back(&out, 1, stream);
  return out.full;
}
std::optional<std::array<Tensor, 3>> taylor_backward(const Tensor& g, const Tensor& q, const Tensor& k, const Tensor& v,
                                                     unsigned debug_flags, uintptr_t status) {
  if (!taylor_covered(q, k, v) || !usable(g, q) || !same_rows(g, q) || g.size(3) != v.size(3)) return std::nullopt;
  const c10::cuda::CUDAGuard guard(g.device());
  void* stream = c10::cuda::getCurrentCUDAStream(g.device().index()).stream();
  const Tensor dq = at::empty(q.sizes(), q.options()), dk = at::empty(k.sizes(), k.options());
  const Output dv = output_like(v, false, nullptr);
  Tensor in[4] = {q, k, v, g};
  kernel_views(in, 4, stream);
  FlaArgs a;
  set_sizes(a, q, v, debug_flags, status);
  a.stream = stream;
  a.q = desc(in[0]);
  a.k = desc(in[1]);
  a.v = desc(in[2]);
  a.d_o = desc(in[3]);
  a.d_q = desc(dq);
  a.d_k = desc(dk);
  a.d_v = desc(dv.view);
  check(fla_sm100_taylor_bwd(&a), "fla_sm100_taylor_bwd");
  copy_back(&dv, 1, stream);
  return std::array<Tensor, 3>{dq, dk, dv.full};
}

// The same through features in memory: out and the features of q and k, rows padded to a multiple of 8
// elements; and the gradients from those. (Prepared in Python a training step took 200 us of the host.)
struct FeatureDims {
  int features, padded;
};
std::optional<FeatureDims> feature_dims(const Tensor& q, const Tensor& k, const Tensor& v) {
  FeatureDims f;
  if (!usable(q, q) || !usable(k, q) || !usable(v, q) || q.sizes() != k.sizes() || !same_rows(q, v) ||
      q.scalar_type() != at::kBFloat16 || !covered_dims(q, v) ||
      fla_sm100_taylor_dims(static_cast<int>(q.size(3)), &f.features, &f.padded) != FLA_OK)
    return std::nullopt;
  return f;
}
Tensor aligned_rows(const Tensor& x) {  // what the feature kernels read
  const Tensor c = x.contiguous();
  return reinterpret_cast<uintptr_t>(c.data_ptr()) % 16 == 0 ? c : c.clone();
}
std::optional<std::array<Tensor, 3>> taylor_forward_in_memory(const Tensor& q, const Tensor& k, const Tensor& v,
                                                              unsigned debug_flags, uintptr_t status) {
  const auto dims = feature_dims(q, k, v);
  if (!dims.has_value()) return std::nullopt;
  const c10::cuda::CUDAGuard guard(q.device());
  void* stream = c10::cuda::getCurrentCUDAStream(q.device().index()).stream();
  auto features = [&](const Tensor& x) {
    const Tensor rows = aligned_rows(x);
    const Tensor phi = at::empty({x.size(0), x.size(1), x.size(2), dims->padded}, x.options());
    check(fla_sm100_taylor_features(rows.data_ptr(), phi.data_ptr(), x.numel() / x.size(3), static_cast<int>(x.size(3)), stream),
          "fla_sm100_taylor_features");
    return phi.narrow(3, 0, dims->features);
  };
  const Tensor pq = features(q), pk = features(k);
  const std::optional<Forward> r = forward(pq, pk, v, std::nullopt, 0, debug_flags, status);
  if (!r.has_value()) return std::nullopt;
  return std::array<Tensor, 3>{r->out, pq, pk};
}
std::optional<std::array<Tensor, 3>> taylor_backward_in_memory(const Tensor& g, const Tensor& q, const Tensor& k,
                                                               const Tensor& v, const Tensor& pq, const Tensor& pk,
                                                               unsigned debug_flags, uintptr_t status) {
  const auto dims = feature_dims(q, k, v);
  if (!dims.has_value()) return std::nullopt;
  const auto r = backward(g, pq, pk, v, std::nullopt, std::nullopt, true, std::nullopt, debug_flags, status);
  if (!r.has_value()) return std::nullopt;
  const c10::cuda::CUDAGuard guard(q.device());
  void* stream = c10::cuda::getCurrentCUDAStream(q.device().index()).stream();
  auto raw = [&](const Tensor& dphi, const Tensor& x) {  // (dphi: fresh, its rows padded as those of the features)
    const Tensor rows = aligned_rows(x), dx = at::empty(x.sizes(), x.options());
    check(fla_sm100_taylor_features_bwd(dphi.data_ptr(), rows.data_ptr(), dx.data_ptr(), x.numel() / x.size(3),
                                        static_cast<int>(x.size(3)), stream),
          "fla_sm100_taylor_features_bwd");
    return dx;
  };
  return std::array<Tensor, 3>{raw((*r)[0], q), raw((*r)[1], k), (*r)[2]};
}

// What is saved beside the repacked copy of an input that is not kept itself: an empty tensor that shares
// its version count, for autograd to see that it was changed in place. (An inference tensor has none;
// it is returned itself, and autograd refuses it as it always does.)
Tensor version_of(const Tensor& t) {
  if (t.is_inference()) return t;
  const Tensor version = at::empty({0}, t.options());
  torch::autograd::impl::set_version_counter(version, torch::autograd::impl::version_counter(t));
  return version;
}

}  // namespace

PYBIND11_MODULE(_hostcalls, m) {
  m.attr("abi_version") = FLA_ABI_VERSION;
  m.def("forward", [](const Tensor& q, const Tensor& k, const Tensor& v, const OptTensor& s_init, int state,
                      unsigned debug_flags, uintptr_t status) -> py::object {
    std::optional<Forward> r;
    {
      const py::gil_scoped_release unlocked;
      r = forward(q, k, v, s_init, state, debug_flags, status);
    }
    if (!r.has_value()) return py::none();
    py::object views = py::none();
    if (r->views.has_value()) views = py::make_tuple((*r->views)[0], (*r->views)[1], (*r->views)[2]);
    return py::make_tuple(r->out, r->s_final, r->seg_states, views);
  });
  m.def("version_of", &version_of);
  m.def("taylor_forward", &taylor_forward, py::call_guard<py::gil_scoped_release>());
  m.def("taylor_backward", &taylor_backward, py::call_guard<py::gil_scoped_release>());
  m.def("taylor_forward_in_memory", &taylor_forward_in_memory, py::call_guard<py::gil_scoped_release>());
  m.def("taylor_backward_in_memory", &taylor_backward_in_memory, py::call_guard<py::gil_scoped_release>());
  m.def("backward", [](const Tensor& g, const Tensor& q, const Tensor& k, const Tensor& v, const OptTensor& s_last,
                       const OptTensor& seg_states, bool keep_padded, const Strides& strides, unsigned debug_flags,
                       uintptr_t status) -> py::object {
    std::optional<std::array<Tensor, 3>> r;
    {
      const py::gil_scoped_release unlocked;
      r = backward(g, q, k, v, s_last, seg_states, keep_padded, strides, debug_flags, status);
    }
    if (!r.has_value()) return py::none();
    return py::make_tuple((*r)[0], (*r)[1], (*r)[2]);
  });
}
