// Looks a dict of torch tensors over in one call.  From Python the same checks took 70 to 90 us for the 148 tensors of GPT-2
// small, more than the kernel over a table of a few million elements does; here they take 4 us.  The one translation unit
// that uses torch's headers; a module of its own, loaded when a table is made on a GPU.
#include <ATen/core/Tensor.h>
#include <c10/core/GradMode.h>
#include <torch/csrc/autograd/python_variable.h>

#include <algorithm>
#include <cstdint>
#include <utility>
#include <vector>

namespace {

namespace py = pybind11;

class TensorList {
 public:
  TensorList(py::list names, std::vector<std::vector<int64_t>> shapes, int device)
      : names_(std::move(names)), shapes_(std::move(shapes)), device_(device) {
    if (names_.size() != shapes_.size()) throw std::invalid_argument("one shape per name");
  }

  // The tensors' addresses as packed 64-bit words, or None if one of them needs a conversion, a broadcast or autograd on the
  // way, or has no memory.  `written`: the caller is about to overwrite them (their version counters move).
  py::object addresses(const py::object& tensors, bool written) const {
    const size_t n = shapes_.size();
    std::vector<uintptr_t> out(n);
    std::vector<py::object> held(n);
    const bool tracked = written && c10::GradMode::is_enabled();
    for (size_t k = 0; k < n; k++) {
      held[k] = tensors[names_[k]];
      PyObject* const o = held[k].ptr();
      if (!THPVariable_Check(o)) return py::none();
      const at::Tensor& t = THPVariable_Unpack(o);
      if (!t.defined() || !t.has_storage() || t.scalar_type() != at::kFloat || t.layout() != at::kStrided || !t.is_cuda() || t.get_device() != device_ || t.is_neg() ||
          t.key_set().has(c10::DispatchKey::Python) || !(t.sizes() == at::IntArrayRef(shapes_[k])) || !t.is_contiguous() || (tracked && t.requires_grad()))
        return py::none();
      // zeros without memory (forward-mode differentiation makes them), and tensors whose storage has been given up
      if (t._is_zerotensor() || t.storage().nbytes() < (size_t(t.storage_offset()) + size_t(t.numel())) * sizeof(float)) return py::none();
      out[k] = reinterpret_cast<uintptr_t>(written ? t.mutable_data_ptr() : const_cast<void*>(t.const_data_ptr()));
    }
    if (written) {
      // names that share memory, wholly or in part, are written one after the other
      std::vector<std::pair<uintptr_t, uintptr_t>> spans;
      spans.reserve(n);
      for (size_t k = 0; k < n; k++)
        if (const size_t bytes = THPVariable_Unpack(held[k].ptr()).nbytes()) spans.emplace_back(out[k], out[k] + bytes);
      std::sort(spans.begin(), spans.end());
      for (size_t k = 1; k < spans.size(); k++)
        if (spans[k].first < spans[k - 1].second) return py::none();
      for (size_t k = 0; k < n; k++) THPVariable_Unpack(held[k].ptr()).unsafeGetTensorImpl()->bump_version();
    }
    return py::bytes(reinterpret_cast<const char*>(out.data()), n * sizeof(uintptr_t));
  }

 private:
  py::list names_;
  std::vector<std::vector<int64_t>> shapes_;
  int device_;
};

}  // namespace

PYBIND11_MODULE(_tensors, m) {
  m.doc() = "sharedtensor_b200: checks and addresses of a dict of torch tensors";
  py::class_<TensorList>(m, "TensorList")
      .def(py::init<py::list, std::vector<std::vector<int64_t>>, int>())
      .def("addresses", &TensorList::addresses);
}
