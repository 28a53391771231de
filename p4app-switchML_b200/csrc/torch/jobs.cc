// lib/torch_switchml_jobs.so: submission of torch tensors and the handle of a job, for parallel/context.py.
//
// A short allreduce is as fast as its submission. In Python, the questions to two tensors, five arguments
// through ctypes and an object with a finaliser took 2.9 us of 7.8 us per job in stream order. The library's
// entry points come in as addresses, because which build of it is loaded is for the caller to say.
#include <ATen/cuda/CUDAContext.h>
#include <torch/extension.h>

#include <algorithm>
#include <string>

namespace {

struct Entry {
  int64_t (*allreduce_async)(void*, void*, uint64_t, int, void*);
  int (*wait)(int64_t, double);
  int (*status)(int64_t);
  int (*stream_wait)(int64_t, void*);
  int (*error)(int64_t, char*, size_t);
  void (*release)(int64_t);
  const char* (*last_error)();
  int (*emu_allreduce)(int, void* const*, void* const*, uint64_t, int, int, int, int, uint64_t, int, int, float, int, int);
};
Entry g_entry;
py::object* g_status = nullptr;  // tuple of JobStatus, and the exception class: live as long as the process
py::object* g_native_error = nullptr;

[[noreturn]] void Raise(const std::string& what) {
  PyErr_SetString(g_native_error->ptr(), what.c_str());
  throw py::error_already_set();
}

py::object Status(int code) {
  if (code < 0) Raise(g_entry.last_error());
  return py::reinterpret_borrow<py::object>(PyTuple_GET_ITEM(g_status->ptr(), code));
}

// A stream object of torch, or a plain handle.
void* StreamHandle(const py::object& stream) {
  if (PyLong_Check(stream.ptr())) return PyLong_AsVoidPtr(stream.ptr());
  const py::object handle = stream.attr("cuda_stream");
  return PyLong_AsVoidPtr(handle.ptr());
}

class Job {
 public:
  Job(int64_t handle, py::object keep) : handle_(handle), keep_(std::move(keep)) {}
  Job(int64_t handle, at::Tensor in, at::Tensor out) : handle_(handle), in_(std::move(in)), out_(std::move(out)) {}
  ~Job() { Release(); }
  py::object Wait(const py::object& timeout_ms) {
    const double limit = timeout_ms.is_none() ? -1.0 : timeout_ms.cast<double>();
    int code;
    {
      py::gil_scoped_release no_gil;
      code = g_entry.wait(handle_, limit);
    }
    return Status(code);
  }
  py::object GetStatus() { return Status(g_entry.status(handle_)); }
  void StreamWait(const py::object& stream) {
    void* s = stream.is_none() ? at::cuda::getCurrentCUDAStream().stream() : StreamHandle(stream);
    int rc;
    {
      py::gil_scoped_release no_gil;  // may have to wait until the job is enqueued
      rc = g_entry.stream_wait(handle_, s);
    }
    if (rc != 0) Raise(g_entry.last_error());
  }
  std::string Error() {
    std::string text(4096, '\0');
    int n = g_entry.error(handle_, text.data(), text.size());
    if (n < 0) Raise(g_entry.last_error());
    if (static_cast<size_t>(n) >= text.size()) {
      text.resize(n + 1);
      n = g_entry.error(handle_, text.data(), text.size());
    }
    text.resize(n);
    return text;
  }
  void Release() {
    if (!handle_) return;
    g_entry.release(handle_);
    handle_ = 0;
    keep_ = py::none();
    in_.reset();
    out_.reset();
  }
  std::string Repr() {
    if (!handle_) return "<switchml Job released>";
    return "<switchml Job handle=" + std::to_string(handle_) + " " + GetStatus().attr("name").cast<std::string>() + ">";
  }

 private:
  int64_t handle_;
  py::object keep_;     // what must outlive the job: these, or
  at::Tensor in_, out_;  // the tensors
};

int Code(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return 0;
    case at::kInt: return 1;
    case at::kBFloat16: return 2;
    case at::kByte: return 3;
    default: return -1;
  }
}

// A job for plain torch tensors, or None when Python has to look at the arguments (other objects, or
// something to complain about).
py::object Submit(const py::object& tensor, const py::object& out, const py::object& stream) {
  if (!THPVariable_Check(tensor.ptr()) || !(out.is_none() || THPVariable_Check(out.ptr()))) return py::none();
  const at::Tensor& in = THPVariable_Unpack(tensor.ptr());
  const bool in_place = out.is_none();
  const at::Tensor& to = in_place ? in : THPVariable_Unpack(out.ptr());
  const int code = Code(in.scalar_type());
  if (code < 0 || !in.is_contiguous() || in.layout() != at::kStrided) return py::none();
  if (!in_place && (to.scalar_type() != in.scalar_type() || to.numel() != in.numel() || to.layout() != at::kStrided || !to.is_contiguous()))
    return py::none();
  void* s = nullptr;
  if (!stream.is_none()) s = StreamHandle(stream);
  else if (in.is_cuda()) s = at::cuda::getCurrentCUDAStream(in.get_device()).stream();
  int64_t handle;
  {
    py::gil_scoped_release no_gil;
    handle = g_entry.allreduce_async(in.data_ptr(), to.data_ptr(), static_cast<uint64_t>(in.numel()), code, s);
  }
  if (handle < 0) Raise(g_entry.last_error());
  return py::cast(new Job(handle, in, in_place ? at::Tensor() : to), py::return_value_policy::take_ownership);
}

// ops/emulation.py: the outputs of an aggregation of several workers on this GPU, or None when Python has to look at the
// arguments. (In Python the questions to the tensors and the call through ctypes took 7 us with two workers and 10 with
// eight, of calls of 25 to 40.)
py::object Emulate(const py::object& inputs, const py::object& outputs, int mode, int algo, int block_numel, int64_t slot_bytes,
                   int slots_per_channel, int channels, double post_scale, int repeats, int exponent_lookahead) {
  constexpr int kMost = 8;
  if (!PyList_CheckExact(inputs.ptr()) || !(outputs.is_none() || PyList_CheckExact(outputs.ptr()))) return py::none();
  const Py_ssize_t n = PyList_GET_SIZE(inputs.ptr());
  if (n < 1 || n > kMost || block_numel < 1 || slot_bytes < 1 || (!outputs.is_none() && PyList_GET_SIZE(outputs.ptr()) != n)) return py::none();
  at::Tensor in[kMost], out[kMost];  // they outlive the call, whatever other threads do to the lists
  void *ins[kMost], *outs[kMost];
  py::list made;
  for (Py_ssize_t r = 0; r < n; r++) {
    PyObject* const i = PyList_GET_ITEM(inputs.ptr(), r);
    PyObject* const o = outputs.is_none() ? nullptr : PyList_GET_ITEM(outputs.ptr(), r);
    if (!THPVariable_Check(i) || (o && !THPVariable_Check(o))) return py::none();
    in[r] = THPVariable_Unpack(i);
    if (!in[r].is_cuda() || in[r].layout() != at::kStrided || !in[r].is_contiguous() || in[r].scalar_type() != in[0].scalar_type() ||
        in[r].numel() != in[0].numel() || Code(in[r].scalar_type()) < 0 || in[r].scalar_type() == at::kByte)
      return py::none();
  }
  for (Py_ssize_t r = 0; r < n; r++) {
    if (outputs.is_none()) {
      out[r] = at::empty_like(in[r]);
      made.append(py::cast(out[r]));
    } else {
      out[r] = THPVariable_Unpack(PyList_GET_ITEM(outputs.ptr(), r));
      // (Python says what is wrong with another one.)
      if (out[r].layout() != at::kStrided || !out[r].is_contiguous() || out[r].device() != in[r].device() ||
          out[r].scalar_type() != in[0].scalar_type() || out[r].numel() < in[0].numel())
        return py::none();
    }
    ins[r] = in[r].data_ptr();
    outs[r] = out[r].data_ptr();
  }
  const int64_t unit = n * static_cast<int64_t>(block_numel > 128 ? block_numel : 128) * 4;
  int64_t slot = std::max(unit, slot_bytes / unit * unit);
  if (algo == 3) slot = std::max(slot, 2 * unit);  // push: receive areas and result areas
  int rc;
  {
    py::gil_scoped_release no_gil;
    rc = g_entry.emu_allreduce(static_cast<int>(n), ins, outs, static_cast<uint64_t>(in[0].numel()), Code(in[0].scalar_type()), mode, algo,
                               block_numel, static_cast<uint64_t>(slot), slots_per_channel, channels, static_cast<float>(post_scale),
                               repeats, exponent_lookahead);
  }
  if (rc != 0) Raise("emulated allreduce failed (" + std::to_string(rc) + "): " + g_entry.last_error());
  return outputs.is_none() ? py::object(made) : outputs;
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  m.def("init", [](const std::vector<uintptr_t>& entry, const py::object& status, const py::object& native_error) {
    TORCH_CHECK(entry.size() * sizeof(uintptr_t) == sizeof(Entry), "one address for each entry point");
    memcpy(&g_entry, entry.data(), sizeof(Entry));
    g_status = new py::object(status);
    g_native_error = new py::object(native_error);
  });
  m.def("submit", &Submit);
  m.def("emulate", &Emulate);
  py::class_<Job>(m, "Job", "Handle of a submitted allreduce (``switchml::Job``).")
      .def(py::init<int64_t, py::object>())
      .def("wait", &Job::Wait, py::arg("timeout_ms") = py::none(),
           "Block until FINISHED or FAILED (``Job::WaitToComplete``); returns the status.")
      .def("status", &Job::GetStatus)
      .def("stream_wait", &Job::StreamWait, py::arg("stream") = py::none(),
           "Order a CUDA stream after the job without waiting on the host (cuda backend).")
      .def("error", &Job::Error)
      .def("release", &Job::Release)
      .def("__repr__", &Job::Repr);
}
