// Python bindings of the C++ host side.
#include <torch/csrc/utils/pybind.h>

#include "layer.h"

namespace py = pybind11;
using namespace mintb_host;

static PyObject* g_failure = nullptr;   // the exception class that a CUDA failure raises

// An ops.GradScale.
struct PyScale : ScaleHolder {
  explicit PyScale(py::object o) : obj(o.release().ptr()) {}
  ~PyScale() override {
    if (!Py_IsInitialized()) return;
    py::gil_scoped_acquire gil;
    Py_DECREF(obj);
  }
  double current() override {
    py::gil_scoped_acquire gil;
    py::object s = py::reinterpret_borrow<py::object>(obj).attr("scale");
    return s.is_none() ? 0.0 : s.cast<double>();
  }
  double fix(double amax) override {
    py::gil_scoped_acquire gil;
    return py::reinterpret_borrow<py::object>(obj).attr("fix")(amax).cast<double>();
  }
  PyObject* obj;
};

PYBIND11_MODULE(_mintb_host, m) {
  m.doc() = "C++ host side of mint_plus_b200: launches and autograd nodes over libmintb";
  py::register_exception_translator([](std::exception_ptr p) {
    try {
      if (p) std::rethrow_exception(p);
    } catch (const MintbFailure& e) {
      PyErr_SetString(g_failure ? g_failure : PyExc_RuntimeError, e.what());
    }
  });
  m.def("set_failure_class", [](py::object c) { g_failure = c.release().ptr(); });
  m.def("dev_status", &dev_status);
  m.def("cached_free_bytes", &cached_free_bytes);
  m.def("capture_id", &capture_id);
  auto nogil = py::call_guard<py::gil_scoped_release>();
  m.def("attention",
        [](const Tensor& q0, const Tensor& q1, const Tensor& q2, const Tensor& q3, const Tensor& q4, const Tensor& q5, const Tensor& meta, const OptTensor& cos,
           const OptTensor& sin, double scale, int64_t flags) { return attention({q0, q1, q2, q3, q4, q5}, meta, cos, sin, scale, flags); },
        nogil);
  m.def("attention_ids",
        [](const Tensor& q0, const Tensor& q1, const Tensor& q2, const Tensor& q3, const Tensor& q4, const Tensor& q5, const Tensor& chain_ids, const OptTensor& key_pad,
           const OptTensor& cos, const OptTensor& sin, double scale, int64_t flags) {
          return attention({q0, q1, q2, q3, q4, q5}, Tensor(), cos, sin, scale, flags, chain_ids, key_pad);
        },
        nogil);
  m.def("mask_meta", &mask_meta, nogil);
  m.def("combine", &combine, nogil);
  m.def("linear", &linear, nogil);
  m.def("linear_f32", &linear_f32, nogil);
  m.def("heads_f32", &heads_f32, nogil);
  m.def("add_layernorm", &add_layernorm, nogil);
  m.def("embed", &embed, nogil);
  m.def("masked_ce", &masked_ce, nogil);
  m.def("mlm_corrupt", &mlm_corrupt, nogil);

  py::class_<Operand>(m, "Operand")
      .def(py::init([](const OptTensor& w, double w_scale, double x_scale, double out_scale, py::object holder) {
             Operand o{opt(w), w_scale, x_scale, out_scale};
             if (!holder.is_none()) {
               o.holder = std::make_shared<PyScale>(holder);
               o.grad_scale = o.holder->current();
             }
             return o;
           }),
           py::arg("w"), py::arg("w_scale") = 1.0, py::arg("x_scale") = 1.0, py::arg("out_scale") = 1.0, py::arg("grad_scale") = py::none());
  py::class_<LayerPlan>(m, "LayerPlan")
      .def(py::init([](bool mu, bool fp8, bool sqrt_softmax, int64_t H, int64_t D, double scale, double keep, double add, double eps1, double eps2,
                       const std::vector<OptTensor>& params, int64_t n_self, int64_t n_cross, const Operand& qkv_self, const Operand& qkv_cross, const Operand& out,
                       const Operand& fc1, const Operand& fc2, bool joint, const OptTensor& qkv6, int64_t lora_r, double lora_scaling) {
             LayerPlan p;
             p.lora_r = lora_r; p.lora_scaling = lora_scaling;
             p.mu = mu; p.fp8 = fp8; p.sqrt_softmax = sqrt_softmax; p.H = H; p.D = D; p.scale = scale; p.keep = keep; p.add = add; p.eps1 = eps1; p.eps2 = eps2;
             for (const OptTensor& t : params) p.params.push_back(opt(t));
             p.n_self = n_self; p.n_cross = n_cross; p.qkv_self = qkv_self; p.qkv_cross = qkv_cross; p.out = out; p.fc1 = fc1; p.fc2 = fc2;
             p.joint = joint; p.qkv6 = opt(qkv6);
             p.form();
             return p;
           }),
           py::kw_only(), py::arg("mu"), py::arg("fp8"), py::arg("sqrt_softmax"), py::arg("H"), py::arg("D"), py::arg("scale"), py::arg("keep"), py::arg("add"),
           py::arg("eps1"), py::arg("eps2"), py::arg("params"), py::arg("n_self"), py::arg("n_cross"), py::arg("qkv_self"), py::arg("qkv_cross"), py::arg("out"),
           py::arg("fc1"), py::arg("fc2"), py::arg("joint"), py::arg("qkv6"),
           py::arg("lora_r") = 0, py::arg("lora_scaling") = 1.0)
      .def("state", &LayerPlan::state)
      .def("refreshed", &LayerPlan::refreshed)
      .def("forward",
           [](const LayerPlan& p, const Tensor& x, const OptTensor& xq, int64_t T, int64_t B, const Tensor& meta, const OptTensor& cos, const OptTensor& sin,
              const OptTensor& rows32, const OptTensor& rows64, const OptTensor& inv32, double next_quant) {
             return p.forward(x, xq, Batch{T, B, meta, opt(cos), opt(sin), opt(rows32), opt(rows64), opt(inv32)}, next_quant);
           },
           nogil);
}
