// Bindings of the dense-parameter path (fused dense step, DCT compression).
#include <ATen/cuda/CUDAEvent.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <pybind11/stl.h>
#include <torch/extension.h>

#include "cuda/dense_kernels.h"
#include "cuda/mlp_gemm.h"

namespace py = pybind11;
using namespace kb;

namespace {

cudaStream_t cur_stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

void check_launch(const char* what) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) throw std::runtime_error(std::string(what) + ": " + cudaGetErrorString(e));
}

template <typename T>
T* optr(const c10::optional<torch::Tensor>& t) {
  return (t.has_value() && t->defined() && t->numel() > 0) ? reinterpret_cast<T*>(t->data_ptr()) : nullptr;
}

cu::SymHost sym_from(const std::vector<uintptr_t>& bases, int rank) {
  cu::SymHost s{};
  TORCH_CHECK(bases.size() <= static_cast<size_t>(cu::kMaxWorldHost), "too many ranks");
  for (size_t i = 0; i < bases.size(); ++i) s.base[i] = reinterpret_cast<void*>(bases[i]);
  s.rank = rank;
  s.world = static_cast<int>(bases.size());
  return s;
}

// All matrices in as few launches as possible, their bf16 copies (and transposes) in ONE buffer, which is returned
// with the views so that a caller on another stream has one tensor to record.
std::tuple<std::vector<torch::Tensor>, std::vector<torch::Tensor>, torch::Tensor> cast_weights(
    const std::vector<torch::Tensor>& ws, bool transpose) {
  int64_t total = 0;
  auto room = [](int64_t n) { return (n + 63) / 64 * 64; };
  std::vector<torch::Tensor> rows;  // a copy of those that are not stored row by row
  for (const auto& w : ws) rows.push_back(w.contiguous());
  for (const auto& w : rows) {
    TORCH_CHECK(w.is_cuda() && w.scalar_type() == torch::kFloat32 && w.dim() == 2,
                "weights must be 2-D CUDA f32 tensors");
    total += room(w.numel()) * (transpose ? 2 : 1);
  }
  std::vector<torch::Tensor> w16s, wt16s;
  if (ws.empty()) return {w16s, wt16s, torch::Tensor()};
  torch::Tensor buf = torch::empty({total}, ws[0].options().dtype(torch::kBFloat16));
  __nv_bfloat16* base = reinterpret_cast<__nv_bfloat16*>(buf.data_ptr());
  cu::CastBatch batch{};
  int64_t at = 0;
  for (const auto& w : rows) {
    const int N = w.size(0), K = w.size(1);
    w16s.push_back(buf.narrow(0, at, w.numel()).view({N, K}));
    __nv_bfloat16* const w16 = base + at;
    at += room(w.numel());
    __nv_bfloat16* wt16 = nullptr;
    if (transpose) {
      wt16s.push_back(buf.narrow(0, at, w.numel()).view({K, N}));
      wt16 = base + at;
      at += room(w.numel());
    }
    const float* src = w.data_ptr<float>();
    if (N % 8 != 0 || K % 8 != 0 || reinterpret_cast<uintptr_t>(src) % 16 != 0) {
      torch::Tensor spare;
      if (wt16 == nullptr) {
        spare = torch::empty({w.numel()}, buf.options());
        wt16 = reinterpret_cast<__nv_bfloat16*>(spare.data_ptr());
      }
      cu::cast_w_wt(src, N, K, w16, wt16, cur_stream());
      continue;
    }
    const int l = batch.layers++;
    batch.w[l] = src, batch.w16[l] = w16, batch.wt16[l] = wt16, batch.N[l] = N, batch.K[l] = K;
    if (batch.layers == cu::CastBatch::kMax) {
      cu::cast_weights(batch, cur_stream());
      batch.layers = 0;
    }
  }
  if (batch.layers > 0) cu::cast_weights(batch, cur_stream());
  check_launch("cast_weights");
  return {w16s, wt16s, buf};
}

struct StreamEvent {
  at::cuda::CUDAEvent event;
  void Wait() { event.block(c10::cuda::getCurrentCUDAStream()); }
};

// `later` waits for what `earlier` has been given so far.
void join(const c10::cuda::CUDAStream& earlier, const c10::cuda::CUDAStream& later) {
  at::cuda::CUDAEvent e;
  e.record(earlier);
  e.block(later);
}

// The caching allocator keeps `t`'s memory until `stream` has passed this point.
void on_stream(const torch::Tensor& t, const c10::cuda::CUDAStream& stream) {
  c10::cuda::CUDACachingAllocator::recordStream(t.storage().data_ptr(), stream);
}

}  // namespace

void bind_dense(py::module_& m) {
  py::class_<cu::DenseLayout>(m, "DenseLayout")
      .def(py::init<>())
      .def_readwrite("grad", &cu::DenseLayout::grad)
      .def_readwrite("param", &cu::DenseLayout::param)
      .def_readwrite("flag_grad", &cu::DenseLayout::flag_grad)
      .def_readwrite("flag_done", &cu::DenseLayout::flag_done)
      .def_readwrite("coo_cnt", &cu::DenseLayout::coo_cnt)
      .def_readwrite("coo_idx", &cu::DenseLayout::coo_idx)
      .def_readwrite("coo_val", &cu::DenseLayout::coo_val);
  m.attr("DENSE_CHUNK") = cu::kDenseChunk;
  m.attr("DENSE_CTRL_INTS") = cu::kDenseCtrlInts;

  m.def("dense_step",
        [](const std::vector<uintptr_t>& bases, int rank, const cu::DenseLayout& lay, const torch::Tensor& ctrl,
           int64_t n_pad, const c10::optional<torch::Tensor>& s0, const c10::optional<torch::Tensor>& s1,
           const c10::optional<torch::Tensor>& s2, const c10::optional<torch::Tensor>& acc,
           const torch::Tensor& chunk_table, const torch::Tensor& table_steps, const torch::Tensor& table_active,
           const OptimPOD& optim, const torch::Tensor& lr, float grad_scale, bool use_coo, uint32_t spin) {
          TORCH_CHECK(n_pad % (static_cast<int64_t>(bases.size()) * cu::kDenseChunk) == 0,
                      "n_pad must be a multiple of world * 256");
          TORCH_CHECK(chunk_table.numel() == n_pad / cu::kDenseChunk, "chunk_table has the wrong size");
          TORCH_CHECK(!use_coo || optr<float>(acc) != nullptr, "COO mode needs the accumulator");
          TORCH_CHECK(ctrl.is_cuda() && ctrl.scalar_type() == torch::kInt32 && ctrl.numel() >= cu::kDenseCtrlInts,
                      "ctrl must be an int32 CUDA tensor of at least ", cu::kDenseCtrlInts, " elements");
          cu::dense_step(sym_from(bases, rank), lay, reinterpret_cast<cu::DenseCtrl*>(ctrl.data_ptr()), n_pad,
                         optr<float>(s0), optr<float>(s1), optr<float>(s2), optr<float>(acc),
                         chunk_table.data_ptr<int>(), table_steps.data_ptr<int>(), table_active.data_ptr<uint8_t>(),
                         static_cast<int>(table_steps.numel()), optim, lr.data_ptr<float>(), grad_scale,
                         use_coo ? 1 : 0, spin, cur_stream());
          check_launch("dense_step");
        });
  m.def("dense_step_dct",
        [](const std::vector<uintptr_t>& bases, int rank, const cu::DenseLayout& lay, const torch::Tensor& ctrl,
           int64_t n_pad, const c10::optional<torch::Tensor>& s0, const c10::optional<torch::Tensor>& s1,
           const c10::optional<torch::Tensor>& s2, const torch::Tensor& residual, const torch::Tensor& tau, bool add,
           const torch::Tensor& chunk_table, const torch::Tensor& table_steps, const torch::Tensor& table_active,
           const OptimPOD& optim, const torch::Tensor& lr, float grad_scale) {
          TORCH_CHECK(bases.size() == 1 && n_pad % cu::kDenseChunk == 0, "dense_step_dct: one GPU, n_pad a multiple of 256");
          TORCH_CHECK(chunk_table.numel() == n_pad / cu::kDenseChunk && residual.numel() == n_pad &&
                          tau.numel() == table_steps.numel(),
                      "chunk_table, residual or tau has the wrong size");
          TORCH_CHECK(ctrl.is_cuda() && ctrl.scalar_type() == torch::kInt32 && ctrl.numel() >= cu::kDenseCtrlInts,
                      "ctrl must be an int32 CUDA tensor of at least ", cu::kDenseCtrlInts, " elements");
          cu::dense_step_dct(sym_from(bases, rank), lay, reinterpret_cast<cu::DenseCtrl*>(ctrl.data_ptr()), n_pad,
                             optr<float>(s0), optr<float>(s1), optr<float>(s2), residual.data_ptr<float>(),
                             tau.data_ptr<float>(), add, chunk_table.data_ptr<int>(), table_steps.data_ptr<int>(),
                             table_active.data_ptr<uint8_t>(), static_cast<int>(table_steps.numel()), optim,
                             lr.data_ptr<float>(), grad_scale, cur_stream());
          check_launch("dense_step_dct");
        });
  m.def("dct_accumulate", [](const torch::Tensor& grad, const torch::Tensor& residual) {
    TORCH_CHECK(grad.numel() == residual.numel(), "grad and residual differ in size");
    cu::dct_accumulate(grad.data_ptr<float>(), residual.data_ptr<float>(), grad.numel(), cur_stream());
    check_launch("dct_accumulate");
  });
  m.def("dct_select_tau", [](const torch::Tensor& x, int64_t k, const torch::Tensor& hist,
                             const torch::Tensor& prefix_state, const torch::Tensor& tau) {
    TORCH_CHECK(x.is_cuda() && x.scalar_type() == torch::kFloat32 && x.is_contiguous(), "x must be CUDA f32");
    TORCH_CHECK(k >= 1 && k <= x.numel(), "k out of range");
    TORCH_CHECK(hist.numel() >= 1024 && prefix_state.numel() >= 2, "radix scratch too small");
    cu::dct_select_tau(x.data_ptr<float>(), x.numel(), k, reinterpret_cast<uint32_t*>(hist.data_ptr()),
                       reinterpret_cast<uint32_t*>(prefix_state.data_ptr()), tau.data_ptr<float>(), cur_stream());
    check_launch("dct_select_tau");
  });
  m.def("dct_compact", [](const std::vector<uintptr_t>& bases, int rank, const cu::DenseLayout& lay, int64_t n_pad,
                          const torch::Tensor& residual, const torch::Tensor& tau, const torch::Tensor& chunk_table) {
    cu::dct_compact(sym_from(bases, rank), lay, n_pad, residual.data_ptr<float>(), tau.data_ptr<float>(),
                    chunk_table.data_ptr<int>(), cur_stream());
    check_launch("dct_compact");
  });
  m.def("dct_threshold_dense", [](const torch::Tensor& grad, const torch::Tensor& residual, const torch::Tensor& tau,
                                  const torch::Tensor& chunk_table) {
    cu::dct_threshold_dense(grad.data_ptr<float>(), residual.data_ptr<float>(), grad.numel(), tau.data_ptr<float>(),
                            chunk_table.data_ptr<int>(), cur_stream());
    check_launch("dct_threshold_dense");
  });

  // ---------------- tcgen05 Linear layers (bf16 in, fp32 accumulate)
  auto bf = [](const torch::Tensor& t) { return reinterpret_cast<const __nv_bfloat16*>(t.data_ptr()); };
  auto need_bf16 = [](const torch::Tensor& t, const char* name) {
    TORCH_CHECK(t.is_cuda() && t.scalar_type() == torch::kBFloat16 && t.dim() == 2 && t.stride(1) == 1, name,
                " must be a 2-D CUDA bf16 tensor with unit inner stride");
  };
  m.def("linear_forward", [bf, need_bf16](const torch::Tensor& x, const torch::Tensor& w,
                                          const c10::optional<torch::Tensor>& bias, bool relu, const torch::Tensor& y,
                                          const torch::Tensor& status, const c10::optional<torch::Tensor>& mask_out) {
    need_bf16(x, "x");
    need_bf16(w, "w");
    need_bf16(y, "y");
    const int M = x.size(0), K = x.size(1), N = w.size(0);
    TORCH_CHECK(w.size(1) == K && y.size(0) == M && y.size(1) == N, "linear_forward: shape mismatch");
    uint16_t* mp = nullptr;
    int ldm = 0;
    if (mask_out.has_value()) {
      TORCH_CHECK(mask_out->is_cuda() && mask_out->scalar_type() == torch::kInt16 && mask_out->dim() == 2 &&
                      mask_out->stride(1) == 1 && mask_out->size(0) * 16 >= N && mask_out->size(1) >= M,
                  "mask_out must be a CUDA int16 tensor [ceil(N / 16), >= M]");
      mp = reinterpret_cast<uint16_t*>(mask_out->data_ptr());
      ldm = mask_out->stride(0);
    }
    c10::optional<torch::Tensor> b;
    bool late = false;
    if (bias.has_value() && bias->defined()) late = !bias->is_contiguous(), b = bias->contiguous();
    const int rc = cu::linear_forward(bf(x), x.stride(0), bf(w), w.stride(0), optr<float>(b),
                                      reinterpret_cast<__nv_bfloat16*>(y.data_ptr()), y.stride(0), M, N, K, relu, mp, ldm,
                                      status.data_ptr<int>(), late, cur_stream());
    TORCH_CHECK(rc == 0, "linear_forward: cannot encode the TMA descriptors (pitches must be multiples of 8)");
  }, py::arg("x"), py::arg("w"), py::arg("bias"), py::arg("relu"), py::arg("y"), py::arg("status"),
     py::arg("mask_out") = py::none());
  m.def("linear_dgrad", [bf, need_bf16](const torch::Tensor& dy, const torch::Tensor& wt,
                                        const c10::optional<torch::Tensor>& h, const torch::Tensor& dx,
                                        const torch::Tensor& status, const c10::optional<torch::Tensor>& mask,
                                        int zero_cols) {
    need_bf16(dy, "dy");
    need_bf16(wt, "wt");
    need_bf16(dx, "dx");
    const int M = dy.size(0), N = dy.size(1), K = wt.size(0);
    TORCH_CHECK(wt.size(1) == N && dx.size(0) == M && dx.size(1) == K, "linear_dgrad: shape mismatch");
    const __nv_bfloat16* hp = nullptr;
    int ldh = 0;
    if (h.has_value()) {
      need_bf16(*h, "h");
      TORCH_CHECK(h->size(0) == M && h->size(1) == K, "linear_dgrad: mask shape mismatch");
      hp = bf(*h);
      ldh = h->stride(0);
    }
    const uint16_t* mp = nullptr;
    int ldm = 0;
    if (mask.has_value()) {
      TORCH_CHECK(mask->is_cuda() && mask->scalar_type() == torch::kInt16 && mask->dim() == 2 && mask->stride(1) == 1 &&
                      mask->size(0) * 16 >= K && mask->size(1) >= M,
                  "mask must be a CUDA int16 tensor [ceil(K / 16), >= M]");
      mp = reinterpret_cast<const uint16_t*>(mask->data_ptr());
      ldm = mask->stride(0);
    }
    const int rc = cu::linear_dgrad(bf(dy), dy.stride(0), bf(wt), wt.stride(0), hp, ldh, mp, ldm,
                                    reinterpret_cast<__nv_bfloat16*>(dx.data_ptr()), dx.stride(0), M, N, K, zero_cols,
                                    status.data_ptr<int>(), cur_stream());
    TORCH_CHECK(rc == 0, "linear_dgrad: cannot encode the TMA descriptors (pitches must be multiples of 8)");
  }, py::arg("dy"), py::arg("wt"), py::arg("h"), py::arg("dx"), py::arg("status"), py::arg("mask") = py::none(),
     py::arg("zero_cols") = 0);
  m.def("linear_wgrad", [bf, need_bf16](const torch::Tensor& dy, const torch::Tensor& x, const torch::Tensor& dw,
                                        const torch::Tensor& status, const c10::optional<torch::Tensor>& db) {
    need_bf16(dy, "dy");
    need_bf16(x, "x");
    TORCH_CHECK(!db.has_value() || (db->is_cuda() && db->scalar_type() == torch::kFloat32 && db->is_contiguous() &&
                                    db->numel() >= dy.size(1)),
                "db too small");
    TORCH_CHECK(dw.is_cuda() && dw.scalar_type() == torch::kFloat32 && dw.dim() == 2 && dw.stride(1) == 1,
                "dw must be a 2-D CUDA f32 tensor");
    const int M = dy.size(0), N = dy.size(1), K = x.size(1);
    TORCH_CHECK(x.size(0) == M && dw.size(0) == N && dw.size(1) == K, "linear_wgrad: shape mismatch");
    const int rc = cu::linear_wgrad(bf(dy), dy.stride(0), bf(x), x.stride(0), dw.data_ptr<float>(), dw.stride(0),
                                    db.has_value() ? db->data_ptr<float>() : nullptr, M, N, K, status.data_ptr<int>(),
                                    cur_stream());
    TORCH_CHECK(rc == 0, "linear_wgrad: cannot encode the TMA descriptors (pitches must be multiples of 8)");
  }, py::arg("dy"), py::arg("x"), py::arg("dw"), py::arg("status"), py::arg("db") = py::none());
  m.def("gemm_set_tuning", &cu::gemm_set_tuning, py::arg("variant") = 0, py::arg("n_tiles") = 0);
  m.def("colsum_bf16", [bf, need_bf16](const torch::Tensor& dy, const torch::Tensor& db) {
    need_bf16(dy, "dy");
    TORCH_CHECK(db.is_cuda() && db.scalar_type() == torch::kFloat32 && db.numel() >= dy.size(1), "db too small");
    cu::colsum_bf16(bf(dy), dy.stride(0), dy.size(0), dy.size(1), db.data_ptr<float>(), cur_stream());
    check_launch("colsum_bf16");
  });
  m.def("rowdot_forward", [bf, need_bf16](const torch::Tensor& x, const torch::Tensor& w,
                                          const c10::optional<torch::Tensor>& bias, const torch::Tensor& y,
                                          const c10::optional<torch::Tensor>& addend) {
    need_bf16(x, "x");
    TORCH_CHECK(w.is_cuda() && w.scalar_type() == torch::kFloat32 && w.is_contiguous() && w.numel() == x.size(1),
                "w must be a contiguous CUDA f32 vector of K elements");
    TORCH_CHECK(y.scalar_type() == torch::kFloat32 && y.numel() == x.size(0) && (x.stride(0) % 2) == 0, "bad y / pitch");
    TORCH_CHECK(!addend.has_value() || (addend->is_cuda() && addend->scalar_type() == torch::kFloat32 &&
                                        addend->is_contiguous() && addend->numel() == x.size(0)),
                "addend must be a contiguous CUDA f32 vector of M elements");
    cu::rowdot_forward(bf(x), x.stride(0), w.data_ptr<float>(), optr<float>(bias), optr<float>(addend), x.size(0),
                       x.size(1), y.data_ptr<float>(), cur_stream());
    check_launch("rowdot_forward");
  }, py::arg("x"), py::arg("w"), py::arg("bias"), py::arg("y"), py::arg("addend") = py::none());
  m.def("rowdot_backward", [bf, need_bf16](const torch::Tensor& x, const torch::Tensor& w, const torch::Tensor& dy,
                                           bool relu_mask, const c10::optional<torch::Tensor>& dx,
                                           const torch::Tensor& dw, const c10::optional<torch::Tensor>& db) {
    need_bf16(x, "x");
    TORCH_CHECK(dy.is_cuda() && dy.scalar_type() == torch::kFloat32 && dy.is_contiguous() && dy.numel() == x.size(0),
                "dy must be a contiguous CUDA f32 vector of M elements");
    TORCH_CHECK(dw.scalar_type() == torch::kFloat32 && dw.is_contiguous() && dw.numel() == x.size(1), "bad dw");
    __nv_bfloat16* dxp = nullptr;
    int lddx = 0;
    if (dx.has_value()) {
      need_bf16(*dx, "dx");
      TORCH_CHECK(dx->size(0) == x.size(0) && dx->size(1) == x.size(1) && (dx->stride(0) % 2) == 0, "bad dx");
      dxp = reinterpret_cast<__nv_bfloat16*>(dx->data_ptr());
      lddx = dx->stride(0);
    }
    cu::rowdot_backward(bf(x), x.stride(0), w.data_ptr<float>(), dy.data_ptr<float>(), x.size(0), x.size(1), relu_mask,
                        dxp, lddx, dw.data_ptr<float>(), optr<float>(db), cur_stream());
    check_launch("rowdot_backward");
  });
  m.def("head_supported", [](const torch::Tensor& x, const torch::Tensor& w, const c10::optional<torch::Tensor>& dw) {
    return x.is_cuda() && x.scalar_type() == torch::kBFloat16 && x.dim() == 2 && x.stride(1) == 1 && w.is_cuda() &&
           w.scalar_type() == torch::kFloat32 && w.dim() == 2 && w.is_contiguous() && w.size(1) == x.size(1) &&
           cu::head_supported(x.data_ptr(), x.stride(0), w.data_ptr(), x.size(1), w.size(0)) &&
           (!dw.has_value() || (dw->is_cuda() && dw->scalar_type() == torch::kFloat32 && dw->is_contiguous() &&
                                dw->numel() == w.numel() && reinterpret_cast<uintptr_t>(dw->data_ptr()) % 16 == 0));
  }, py::arg("x"), py::arg("w"), py::arg("dw") = py::none());
  m.def("head_forward", [bf](const torch::Tensor& x, const torch::Tensor& w, const torch::Tensor& bias, const torch::Tensor& y) {
    TORCH_CHECK(cu::head_supported(x.data_ptr(), x.stride(0), w.data_ptr(), x.size(1), w.size(0)) && w.size(1) == x.size(1),
                "head_forward: unsupported operands");
    TORCH_CHECK(y.is_cuda() && y.scalar_type() == torch::kFloat32 && y.is_contiguous() &&
                    y.numel() == x.size(0) * w.size(0) && bias.is_cuda() && bias.is_contiguous() &&
                    bias.scalar_type() == torch::kFloat32 && bias.numel() == w.size(0),
                "head_forward: shape mismatch");
    cu::head_forward(bf(x), x.stride(0), w.data_ptr<float>(), bias.data_ptr<float>(), x.size(0), x.size(1), w.size(0),
                     y.data_ptr<float>(), cur_stream());
    check_launch("head_forward");
  });
  m.def("head_backward", [bf](const torch::Tensor& x, const torch::Tensor& w, const torch::Tensor& g, bool relu_mask,
                              const c10::optional<torch::Tensor>& dx, const torch::Tensor& dw, const torch::Tensor& db) {
    TORCH_CHECK(cu::head_supported(x.data_ptr(), x.stride(0), w.data_ptr(), x.size(1), w.size(0)) && w.size(1) == x.size(1),
                "head_backward: unsupported operands");
    TORCH_CHECK(g.is_cuda() && g.scalar_type() == torch::kFloat32 && g.is_contiguous() && g.numel() == x.size(0) * w.size(0),
                "g must be a contiguous CUDA f32 [M, classes]");
    TORCH_CHECK(dw.scalar_type() == torch::kFloat32 && dw.is_contiguous() && dw.numel() == w.numel() &&
                    reinterpret_cast<uintptr_t>(dw.data_ptr()) % 16 == 0 && db.scalar_type() == torch::kFloat32 &&
                    db.is_contiguous() && db.numel() == w.size(0),
                "bad dw / db");
    __nv_bfloat16* dxp = nullptr;
    int lddx = 0;
    if (dx.has_value()) {
      TORCH_CHECK(dx->is_cuda() && dx->scalar_type() == torch::kBFloat16 && dx->dim() == 2 && dx->stride(1) == 1 &&
                      dx->size(0) == x.size(0) && dx->size(1) == x.size(1) && dx->stride(0) % 4 == 0 &&
                      reinterpret_cast<uintptr_t>(dx->data_ptr()) % 8 == 0,
                  "bad dx");
      dxp = reinterpret_cast<__nv_bfloat16*>(dx->data_ptr());
      lddx = dx->stride(0);
    }
    torch::Tensor part;  // on this stream, like the kernels that write and read it
    const size_t floats = cu::head_part_floats(x.size(0), x.size(1), w.size(0));
    if (floats > 0) part = torch::empty({static_cast<int64_t>(floats)}, g.options());
    cu::head_backward(bf(x), x.stride(0), w.data_ptr<float>(), g.data_ptr<float>(), x.size(0), x.size(1), w.size(0),
                      relu_mask, dxp, lddx, dw.data_ptr<float>(), db.data_ptr<float>(),
                      floats > 0 ? part.data_ptr<float>() : nullptr, cur_stream());
    check_launch("head_backward");
  });
  m.def("cast_weights", &cast_weights);
  // The casts on stream `side` beside whatever the current stream does next; `wait` of the event orders a stream behind them.
  py::class_<StreamEvent>(m, "StreamEvent").def("wait", &StreamEvent::Wait);
  m.def("prepare_weights", [](const std::vector<torch::Tensor>& ws, bool transpose, int64_t id, int64_t index, int64_t type) {
    const auto side = c10::cuda::CUDAStream::unpack3(id, index, static_cast<c10::DeviceType>(type));
    const c10::cuda::CUDAGuard device(side.device());
    const auto main = c10::cuda::getCurrentCUDAStream();
    join(main, side);
    auto event = std::make_unique<StreamEvent>();
    std::tuple<std::vector<torch::Tensor>, std::vector<torch::Tensor>, torch::Tensor> cast;
    {
      const c10::cuda::CUDAStreamGuard on(side);
      cast = cast_weights(ws, transpose);
      if (std::get<2>(cast).defined()) on_stream(std::get<2>(cast), main);
      event->event.record(side);
    }
    return py::make_tuple(std::get<0>(cast), std::get<1>(cast), std::move(event));
  });
  // The hidden layers of an MLP, every one Linear + ReLU: returns [x, h1, h2, ...] and, with `masks`, the ReLU bits of the
  // h's (see linear_forward).
  m.def("mlp_hidden_forward", [bf, need_bf16](const torch::Tensor& x, const std::vector<torch::Tensor>& ws,
                                              const std::vector<torch::Tensor>& bs, const torch::Tensor& status, bool masks) {
    need_bf16(x, "x");
    TORCH_CHECK(bs.size() >= ws.size(), "a bias per layer is needed");
    const c10::cuda::CUDAGuard device(x.device());
    std::vector<torch::Tensor> acts{x}, bits;
    const int M = x.size(0);
    for (size_t i = 0; i < ws.size(); ++i) {
      const torch::Tensor h = acts.back(), w = ws[i], bias = bs[i].contiguous();
      need_bf16(w, "w");
      const int N = w.size(0), K = w.size(1);
      TORCH_CHECK(h.size(1) == K && bias.is_cuda() && bias.scalar_type() == torch::kFloat32 && bias.numel() == N,
                  "mlp_hidden_forward: shape mismatch");
      torch::Tensor y = torch::empty({M, N}, x.options());
      torch::Tensor mask;
      if (masks) mask = torch::empty({(N + 15) / 16, (M + 63) / 64 * 64}, x.options().dtype(torch::kInt16));
      const int rc = cu::linear_forward(bf(h), h.stride(0), bf(w), w.stride(0), bias.data_ptr<float>(),
                                        reinterpret_cast<__nv_bfloat16*>(y.data_ptr()), y.stride(0), M, N, K, true,
                                        masks ? reinterpret_cast<uint16_t*>(mask.data_ptr()) : nullptr,
                                        masks ? static_cast<int>(mask.stride(0)) : 0, status.data_ptr<int>(),
                                        !bs[i].is_contiguous(), cur_stream());
      TORCH_CHECK(rc == 0, "linear_forward: cannot encode the TMA descriptors (pitches must be multiples of 8)");
      acts.push_back(y);
      if (masks) bits.push_back(mask);
    }
    return std::make_pair(acts, bits);
  });
  // Their backward.  dh: gradient of acts.back() with its ReLU mask applied.  The chain dh_L -> dh_{L-1} -> ... is serial and
  // runs on the current stream; a layer's weight and bias gradients only need that layer's dh and run on stream `side`,
  // behind it (in a graph capture this becomes a parallel branch).  `input_cols` > 0: only the leading columns of x want a
  // gradient, the rest are zeros.  on_ready(i), if given, is called when everything that writes layer i's gradients is
  // enqueued.  Unless `deferred`, the current stream waits for `side` at the end.  Returns the gradient of x or None.
  m.def("mlp_hidden_backward", [bf, need_bf16](torch::Tensor dh, const std::vector<torch::Tensor>& acts,
                                               const std::vector<torch::Tensor>& masks,
                                               const std::vector<torch::Tensor>& wts, const std::vector<torch::Tensor>& dws,
                                               const std::vector<torch::Tensor>& dbs, const torch::Tensor& status,
                                               bool x_needs_grad, int input_cols, int64_t id, int64_t index, int64_t type,
                                               bool deferred, const py::object& on_ready) -> py::object {
    const int L = static_cast<int>(dws.size());
    need_bf16(dh, "dh");
    TORCH_CHECK(static_cast<int>(acts.size()) == L + 1 && static_cast<int>(masks.size()) >= L &&
                    static_cast<int>(wts.size()) >= L && static_cast<int>(dbs.size()) >= L,
                "mlp_hidden_backward: one tensor per layer is needed");
    const c10::cuda::CUDAGuard device(dh.device());
    const auto main = c10::cuda::getCurrentCUDAStream();
    const auto side = c10::cuda::CUDAStream::unpack3(id, index, static_cast<c10::DeviceType>(type));
    const int M = dh.size(0);
    for (int i = L - 1; i >= 0; --i) {
      at::cuda::CUDAEvent ready;
      ready.record(main);
      const torch::Tensor& h = acts[i];
      const int N = dh.size(1), K = h.size(1);
      torch::Tensor dprev;
      if (i > 0 || x_needs_grad) {
        // the chain first: it is what the rest of the backward pass waits for
        need_bf16(wts[i], "wt");
        TORCH_CHECK(wts[i].size(0) == K && wts[i].size(1) == N, "mlp_hidden_backward: weight shape");
        dprev = torch::empty({M, K}, dh.options());
        const int cols = i == 0 && input_cols > 0 && input_cols < K ? input_cols : K;  // behind them zeros
        // masks[i - 1] holds the ReLU bits of h; the input of the MLP has none
        const uint16_t* mask = i > 0 ? reinterpret_cast<const uint16_t*>(masks[i - 1].data_ptr()) : nullptr;
        const int rc = cu::linear_dgrad(bf(dh), dh.stride(0), bf(wts[i]), wts[i].stride(0), nullptr, 0, mask,
                                        i > 0 ? static_cast<int>(masks[i - 1].stride(0)) : 0,
                                        reinterpret_cast<__nv_bfloat16*>(dprev.data_ptr()), K, M, N, cols, K - cols,
                                        status.data_ptr<int>(), main.stream());
        TORCH_CHECK(rc == 0, "linear_dgrad: cannot encode the TMA descriptors (pitches must be multiples of 8)");
      }
      ready.block(side);
      const torch::Tensor &dw = dws[i], &db = dbs[i];
      TORCH_CHECK(dw.is_cuda() && dw.scalar_type() == torch::kFloat32 && dw.dim() == 2 && dw.stride(1) == 1 &&
                      dw.size(0) == N && dw.size(1) == K && db.is_cuda() && db.scalar_type() == torch::kFloat32 &&
                      db.is_contiguous() && db.numel() == N,
                  "mlp_hidden_backward: gradient buffers must be f32 of the parameters' shapes");
      const int rc = cu::linear_wgrad(bf(dh), dh.stride(0), bf(h), h.stride(0), dw.data_ptr<float>(), dw.stride(0),
                                      db.data_ptr<float>(), M, N, K, status.data_ptr<int>(), side.stream());
      TORCH_CHECK(rc == 0, "linear_wgrad: cannot encode the TMA descriptors (pitches must be multiples of 8)");
      on_stream(dh, side);
      if (deferred) on_stream(h, side);  // nobody waits for this stream before the graph lets go of the layer's input
      if (!on_ready.is_none()) on_ready(i);
      dh = dprev;
    }
    if (!deferred) join(side, main);
    return dh.defined() ? py::cast(dh) : py::none();
  });
}
