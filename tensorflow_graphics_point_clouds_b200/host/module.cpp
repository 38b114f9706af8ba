// Module of the host layer: error translation and the bindings of cells.cpp and
// layers.cpp.
#include "host.h"

namespace tfgpc_host {

static PyObject* g_error_class = nullptr;   // _lib.TfgpcError, held for the process

void raise_error(int code, const std::string& message, const std::vector<int32_t>* cells) {
  py::gil_scoped_acquire gil;
  if (!g_error_class) throw std::runtime_error(message);
  py::object err = py::handle(g_error_class)(code, message);
  if (cells) err.attr("num_cells") = py::cast(*cells);
  PyErr_SetObject(g_error_class, err.ptr());
  throw py::error_already_set();
}

void raise_value_error(const std::string& message) { throw py::value_error(message); }

}  // namespace tfgpc_host

PYBIND11_MODULE(_host, m) {
  m.def("set_error_class", [](py::object cls) {
    tfgpc_host::g_error_class = cls.release().ptr();
  });
  tfgpc_host::bind_cells(m);
  tfgpc_host::bind_layers(m);
}
