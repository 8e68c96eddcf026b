// Collectives on torch tensors: the checks and conversions of the Python Communicator, once, in C++.  Every function
// answers false for arguments that are not a well-formed pair of contiguous tensors of one dtype on one device; the caller
// then takes its general path, which handles numpy arrays and raw pointers and says what is wrong with the rest.
#include "common.h"

namespace mccl_torch {
namespace {

bool dtypeOf(const Tensor& t, mcclDataType_t* dt) {
  switch (t.scalar_type()) {
    case at::kChar: *dt = mcclInt8; return true;
    case at::kByte: *dt = mcclUint8; return true;
    case at::kInt: *dt = mcclInt32; return true;
    case at::kUInt32: *dt = mcclUint32; return true;
    case at::kLong: *dt = mcclInt64; return true;
    case at::kUInt64: *dt = mcclUint64; return true;
    case at::kHalf: *dt = mcclFloat16; return true;
    case at::kBFloat16: *dt = mcclBfloat16; return true;
    case at::kFloat: *dt = mcclFloat32; return true;
    case at::kDouble: *dt = mcclFloat64; return true;
    default: return false;
  }
}

// send and recv as a call takes them; `num` x the elements of send fit into recv.
bool pair(const py::object& so, const py::object& ro, int64_t num, Tensor* send, Tensor* recv, mcclDataType_t* dt) {
  if (!THPVariable_Check(so.ptr()) || !THPVariable_Check(ro.ptr())) return false;
  *send = THPVariable_Unpack(so.ptr());
  *recv = THPVariable_Unpack(ro.ptr());
  return send->layout() == at::kStrided && recv->layout() == at::kStrided && send->is_contiguous() && recv->is_contiguous() &&
         send->scalar_type() == recv->scalar_type() && send->device() == recv->device() && recv->numel() >= send->numel() * num &&
         dtypeOf(*send, dt);
}

mcclStream_t streamFor(const Tensor& t, std::optional<int64_t> stream) {
  if (stream) return reinterpret_cast<mcclStream_t>(*stream);
  return t.is_cuda() ? streamOf(t) : nullptr;
}

mcclComm_t commOf(int64_t h) { return reinterpret_cast<mcclComm_t>(h); }

int sizeOf(mcclComm_t c) { int n = 1; mcclCommCount(c, &n); return n; }

// The library's status: 0, in progress, or an error the caller raises; -1: not handled here.
int allReduce(int64_t comm, const py::object& so, const py::object& ro, int op, std::optional<int64_t> stream) {
  Tensor send, recv;
  mcclDataType_t dt;
  if (!pair(so, ro, 1, &send, &recv, &dt)) return -1;
  mcclStream_t s = streamFor(send, stream);
  py::gil_scoped_release nogil;
  return mcclAllReduce(commOf(comm), send.data_ptr(), recv.data_ptr(), (size_t)send.numel(), dt, (mcclRedOp_t)op, s);
}

int allGather(int64_t comm, const py::object& so, const py::object& ro, std::optional<int64_t> stream) {
  Tensor send, recv;
  mcclDataType_t dt;
  if (!pair(so, ro, sizeOf(commOf(comm)), &send, &recv, &dt)) return -1;
  mcclStream_t s = streamFor(send, stream);
  py::gil_scoped_release nogil;
  return mcclAllGather(commOf(comm), send.data_ptr(), recv.data_ptr(), (size_t)send.numel(), dt, s);
}

int reduceScatter(int64_t comm, const py::object& so, const py::object& ro, int op, std::optional<int64_t> stream) {
  Tensor send, recv;
  mcclDataType_t dt;
  if (!pair(ro, so, sizeOf(commOf(comm)), &recv, &send, &dt)) return -1;     // send holds one block of recv's size per rank
  mcclStream_t s = streamFor(send, stream);
  py::gil_scoped_release nogil;
  return mcclReduceScatter(commOf(comm), send.data_ptr(), recv.data_ptr(), (size_t)recv.numel(), dt, (mcclRedOp_t)op, s);
}

int allToAll(int64_t comm, const py::object& so, const py::object& ro, std::optional<int64_t> stream) {
  Tensor send, recv;
  mcclDataType_t dt;
  const int n = sizeOf(commOf(comm));
  if (!pair(so, ro, 1, &send, &recv, &dt) || send.numel() % n) return -1;
  mcclStream_t s = streamFor(send, stream);
  py::gil_scoped_release nogil;
  return mcclAllToAll(commOf(comm), send.data_ptr(), recv.data_ptr(), (size_t)(send.numel() / n), dt, s);
}

int broadcast(int64_t comm, const py::object& so, const py::object& ro, int root, std::optional<int64_t> stream) {
  Tensor send, recv;
  mcclDataType_t dt;
  if (!pair(ro, so, 1, &recv, &send, &dt)) return -1;                        // the root sends as many elements as everyone receives
  mcclStream_t s = streamFor(recv, stream);
  py::gil_scoped_release nogil;
  return mcclBroadcast(commOf(comm), send.data_ptr(), recv.data_ptr(), (size_t)recv.numel(), dt, root, s);
}

}  // namespace

void bindComm(py::module_& m) {
  m.def("all_reduce", &allReduce);
  m.def("all_gather", &allGather);
  m.def("reduce_scatter", &reduceScatter);
  m.def("all_to_all", &allToAll);
  m.def("broadcast", &broadcast);
}

}  // namespace mccl_torch
