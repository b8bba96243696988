// Module MakePytorchBackend: same names and argument lists as the reference's pybind/bind.cpp:11-24.
#include <torch/extension.h>

#include "backend_ops.h"
#include "conv_module.h"

namespace py = pybind11;

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  py::class_<Foo>(m, "Foo")
      .def(py::init<>())
      .def("setKey", &Foo::setKey)
      .def("getKey", &Foo::getKey)
      .def("__repr__", [](const Foo &a) { return a.toString(); });
  m.def("AddGPU", &AddGPU);
  m.def("WinoSplit", &WinoSplit);
  m.def("WinoConcat", &WinoConcat);
  m.def("DWM", &DWM);
  m.def("set_dwm_output_block", &set_dwm_output_block);
  m.def("get_dwm_output_block", &get_dwm_output_block);
  m.def("conv_call", &conv_call, py::call_guard<py::gil_scoped_release>());
  py::class_<ConvRunner, c10::intrusive_ptr<ConvRunner>>(m, "ConvRunner")
      .def(py::init<int64_t, std::vector<int64_t>, std::vector<int64_t>, int64_t, int64_t, bool, bool, int64_t, int64_t>())
      .def("forward", &ConvRunner::forward, py::call_guard<py::gil_scoped_release>())
      .def("entries", [](ConvRunner &r) {
        py::list out;
        for (auto &e : r.entries())
          out.append(py::make_tuple(std::get<0>(e), std::get<1>(e), std::get<2>(e), std::get<3>(e), std::get<4>(e), py::bytes(std::get<5>(e))));
        return out;
      });
}
