// Bindings: router top-k and MoE token permutation.
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>

#include "launch.h"

namespace {

inline cudaStream_t cur_stream() {
  (void)cudaGetLastError();
  mb_count_launch(1);
  return at::cuda::getCurrentCUDAStream().stream();
}
inline void check(int rc, const char* what) {
  if (rc == 0) return;
  char buf[256];
  snprintf(buf, sizeof(buf), "%s failed with code %d (%s)", what, rc,
           rc > 0 && rc < 1000 ? cudaGetErrorString(static_cast<cudaError_t>(rc)) : "launcher");
  throw std::runtime_error(buf);
}

// logits fp32 [T,E] → (weights fp32 [T,K], idx int32 [T,K], probs fp32 [T,E])
// replay: int32 [T, K] recorded choices (rows may be apart), err: the error flag that a choice of no expert raises; see moe.cu
std::vector<at::Tensor> router_topk(const at::Tensor& logits, int64_t K, bool normalize, bool want_probs, const c10::optional<at::Tensor>& replay,
                                    const c10::optional<at::Tensor>& err) {
  c10::cuda::CUDAGuard g(logits.device());
  const int64_t T = logits.size(0), E = logits.size(1);
  auto w = at::empty({T, K}, logits.options());
  auto idx = at::empty({T, K}, logits.options().dtype(at::kInt));
  const int* recorded = replay.has_value() && replay->defined() ? replay->data_ptr<int>() : nullptr;
  TORCH_CHECK(recorded == nullptr || (replay->size(0) == T && replay->size(1) == K && (K == 1 || replay->stride(1) == 1)), "router_topk: replay [T, K]");
  TORCH_CHECK(recorded == nullptr || (replay->device() == logits.device() && err.has_value() && err->device() == logits.device()),
              "router_topk: recorded choices on ", recorded != nullptr ? replay->device() : logits.device(), ", logits on ", logits.device());
  at::Tensor probs;
  if (want_probs) probs = at::empty({T, E}, logits.options());
  check(mb_router_topk(logits.data_ptr<float>(), want_probs ? probs.data_ptr<float>() : nullptr, w.data_ptr<float>(),
                       idx.data_ptr<int>(), T, E, K, normalize, recorded, recorded != nullptr ? replay->stride(0) : 0,
                       recorded != nullptr ? err->data_ptr<int>() : nullptr, cur_stream()),
        "mb_router_topk");
  return {w, idx, probs};
}

// rmsnorm(x (+ residual)) and its top-k experts: x [T, H] bf16 → (sum [T, H] or undefined, normed [T, H], weights fp32 [T, K], idx int32 [T, K])
std::vector<at::Tensor> norm_router(const at::Tensor& x, const c10::optional<at::Tensor>& residual, const at::Tensor& norm_w, double eps, const at::Tensor& W,
                                    int64_t K, bool normalize, bool static_w) {
  c10::cuda::CUDAGuard g(x.device());
  const int64_t T = x.size(0), H = x.size(1), E = W.size(0);
  const bool add = residual.has_value() && residual->defined();
  TORCH_CHECK(x.is_contiguous() && W.is_contiguous() && norm_w.is_contiguous() && W.size(1) == H && norm_w.numel() == H &&
                  (!add || (residual->is_contiguous() && residual->sizes() == x.sizes())),
              "norm_router: x, residual [T, H], norm_w [H], W [E, H], contiguous");
  at::Tensor sum;
  if (add) sum = at::empty_like(x);
  auto normed = at::empty_like(x);
  auto w = at::empty({T, K}, x.options().dtype(at::kFloat));
  auto idx = at::empty({T, K}, x.options().dtype(at::kInt));
  check(mb_norm_router(x.data_ptr(), add ? residual->data_ptr() : nullptr, norm_w.data_ptr(), W.data_ptr(), eps, T, H, E, K, normalize, static_w,
                       add ? sum.data_ptr() : nullptr, normed.data_ptr(), w.data_ptr<float>(), idx.data_ptr<int>(), cur_stream()),
        "mb_norm_router");
  return {sum, normed, w, idx};
}

// idx int32 [n] global expert ids → seg_offsets [E+1], tile_expert [max_rows/pad], row_src [max_rows], dst_row [n]
std::vector<at::Tensor> moe_align(const at::Tensor& idx, int64_t E, int64_t expert_offset, int64_t max_rows,
                                  const c10::optional<at::Tensor>& n_dev, int64_t pad, bool ordered) {
  c10::cuda::CUDAGuard g(idx.device());
  const int64_t n = idx.numel();
  const int* n_ptr = n_dev.has_value() && n_dev->defined() ? n_dev->data_ptr<int>() : nullptr;
  auto opt = idx.options().dtype(at::kInt);
  auto seg = at::empty({E + 1}, opt);
  TORCH_CHECK(pad > 0 && max_rows % pad == 0, "moe_align: max_rows must be a multiple of pad");
  auto tile = at::empty({max_rows / pad}, opt);
  auto row_src = at::empty({max_rows}, opt);
  auto dst_row = at::empty({n}, opt);
  check(mb_moe_align_pad(idx.data_ptr<int>(), n, n_ptr, E, expert_offset, seg.data_ptr<int>(), tile.data_ptr<int>(),
                         row_src.data_ptr<int>(), dst_row.data_ptr<int>(), max_rows, pad, ordered, cur_stream()),
        "mb_moe_align");
  return {seg, tile, row_src, dst_row};
}

void moe_gather(const at::Tensor& x, at::Tensor& x_perm, const at::Tensor& row_src, const at::Tensor& seg, int64_t k) {
  c10::cuda::CUDAGuard g(x.device());
  check(mb_moe_gather(x.data_ptr(), x_perm.data_ptr(), row_src.data_ptr<int>(), seg.data_ptr<int>(), seg.numel() - 1, k, x.size(-1),
                      x_perm.size(0), cur_stream()),
        "mb_moe_gather");
}

void moe_combine(const at::Tensor& y_perm, const c10::optional<at::Tensor>& w, const at::Tensor& dst_row, at::Tensor& out, int64_t k,
                 bool identity_rows) {
  c10::cuda::CUDAGuard g(out.device());
  check(mb_moe_combine(y_perm.data_ptr(), w.has_value() && w->defined() ? w->data_ptr<float>() : nullptr, dst_row.data_ptr<int>(),
                       out.data_ptr(), out.size(0), k, out.size(-1), identity_rows ? 1 : 0, cur_stream()),
        "mb_moe_combine");
}

void moe_combine_bwd(const at::Tensor& dout, const at::Tensor& y_perm, const at::Tensor& w, const at::Tensor& row_src,
                     const at::Tensor& seg, at::Tensor& dy_perm, const c10::optional<at::Tensor>& dw, int64_t k) {
  c10::cuda::CUDAGuard g(dout.device());
  check(mb_moe_combine_bwd(dout.data_ptr(), y_perm.data_ptr(), w.data_ptr<float>(), row_src.data_ptr<int>(), seg.data_ptr<int>(),
                           seg.numel() - 1, dy_perm.data_ptr(), dw.has_value() && dw->defined() ? dw->data_ptr<float>() : nullptr, k,
                           dout.size(-1), dy_perm.size(0), cur_stream()),
        "mb_moe_combine_bwd");
}

// (rmsnorm(sum) · norm_w, sum) with sum = Σ_j w[t, j] · y_perm[dst_row[t, j]] + residual
std::vector<at::Tensor> moe_combine_norm(const at::Tensor& y_perm, const at::Tensor& w, const at::Tensor& dst_row, const at::Tensor& residual,
                                         const at::Tensor& norm_w, int64_t k, double eps) {
  c10::cuda::CUDAGuard g(residual.device());
  const int64_t T = residual.size(0), H = residual.size(1);
  TORCH_CHECK(y_perm.is_contiguous() && w.is_contiguous() && dst_row.is_contiguous() && residual.is_contiguous() && norm_w.is_contiguous() && y_perm.size(1) == H &&
                  norm_w.numel() == H && w.numel() == T * k && dst_row.numel() == T * k,
              "moe_combine_norm: shapes");
  auto y = at::empty_like(residual), sum = at::empty_like(residual);
  check(mb_moe_combine_norm(y_perm.data_ptr(), w.data_ptr<float>(), dst_row.data_ptr<int>(), residual.data_ptr(), norm_w.data_ptr(), y.data_ptr(), sum.data_ptr(), T,
                            k, H, eps, cur_stream()),
        "mb_moe_combine_norm");
  return {y, sum};
}

// h1 [rows, 2F], act_w [rows, F] (dout · W2 → weighted activation), dh1 [rows, 2F], w and dw fp32 [pairs]
void moe_glu_bwd(const at::Tensor& h1, at::Tensor& act_w, at::Tensor& dh1, const at::Tensor& w, const at::Tensor& row_src, const at::Tensor& seg, at::Tensor& dw) {
  c10::cuda::CUDAGuard g(h1.device());
  TORCH_CHECK(h1.is_contiguous() && act_w.is_contiguous() && dh1.is_contiguous() && w.is_contiguous() && dw.is_contiguous() && h1.sizes() == dh1.sizes() &&
                  h1.size(0) == act_w.size(0) && h1.size(1) == 2 * act_w.size(1) && w.numel() == dw.numel(),
              "moe_glu_bwd: h1, dh1 [rows, 2F], act_w [rows, F], w, dw [pairs], contiguous");
  check(mb_moe_glu_bwd(h1.data_ptr(), act_w.data_ptr(), dh1.data_ptr(), w.data_ptr<float>(), row_src.data_ptr<int>(), seg.data_ptr<int>(), seg.numel() - 1,
                       dw.data_ptr<float>(), act_w.size(1), act_w.size(0), cur_stream()),
        "mb_moe_glu_bwd");
}

}  // namespace

void register_moe(pybind11::module& m) {
  m.def("router_topk", &router_topk, py::arg("logits"), py::arg("k"), py::arg("normalize"), py::arg("want_probs"), py::arg("replay") = py::none(),
        py::arg("err") = py::none());
  m.def("norm_router", &norm_router);
  m.def("moe_align", &moe_align, py::arg("idx"), py::arg("E"), py::arg("expert_offset"), py::arg("max_rows"), py::arg("n_dev"),
        py::arg("pad") = 128, py::arg("ordered") = true);
  m.def("moe_gather", &moe_gather);
  m.def("moe_combine", &moe_combine, pybind11::arg("y_perm"), pybind11::arg("w"), pybind11::arg("dst_row"), pybind11::arg("out"),
        pybind11::arg("k"), pybind11::arg("identity_rows") = false);
  m.def("moe_combine_bwd", &moe_combine_bwd);
  m.def("moe_glu_bwd", &moe_glu_bwd);
  m.def("moe_combine_norm", &moe_combine_norm);
}
