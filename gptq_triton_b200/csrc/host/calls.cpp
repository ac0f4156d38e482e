// Layer calls from Python without ctypes: checks, output allocation, workspace look-up and the launch of one C-ABI entry point.
//
// A call of the smallest layer is bound by the host: o_proj of a 7B layer for one token took 16.5 us a call, 5.5 of them on the GPU; the rest was
// Python (argument checks, torch.empty, nineteen ctypes conversions).  Every function here serves the plain case and returns None for anything
// else (other types, devices or layouts, tensor subclasses, a missing or small workspace, an active torch-function mode, an error from the library),
// without having done anything; the caller then goes on in Python, which supports or reports it.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/core/Tensor.h>
#include <ATen/ops/empty.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../../include/gptq_b200.h"

namespace {

// entry points of the library that the ctypes binding has loaded
decltype(&gptq_workspace_bytes) workspace_bytes = nullptr;
decltype(&gptq_qmatmul) qmatmul_fn = nullptr;
decltype(&gptq_gateup_silu) gateup_fn = nullptr;
decltype(&gptq_qkv_rope) qkv_fn = nullptr;

// A dense CUDA tensor of the given type on `device` (an empty pointer: not the plain case).
const at::Tensor *plain(PyObject *o, at::ScalarType type, int device) {
	if (!THPVariable_CheckExact(o)) {
		if (!THPVariable_Check(o) || Py_TYPE(o) != reinterpret_cast<PyTypeObject *>(ParameterClass)) return nullptr;
	}
	const at::Tensor &t = THPVariable_Unpack(o);
	const auto keys = t.key_set();
	if (!t.defined() || !t.has_storage() || t.layout() != at::kStrided || keys.has(c10::DispatchKey::Python) || keys.has(c10::DispatchKey::FuncTorchBatched) ||
		keys.has(c10::DispatchKey::FuncTorchGradWrapper) || keys.has(c10::DispatchKey::Functionalize) || !t.is_cuda() || t.scalar_type() != type ||
		(device >= 0 && t.get_device() != device) || !t.is_contiguous() || t.is_conj() || t.is_neg())
		return nullptr;
	return &t;
}
// the same for an operand that may be None; `ok` turns false when it is neither
const at::Tensor *maybe(PyObject *o, at::ScalarType type, int device, bool &ok) {
	if (o == Py_None) return nullptr;
	const at::Tensor *t = plain(o, type, device);
	if (!t) ok = false;
	return t;
}
void *ptr(const at::Tensor *t) { return t ? t->data_ptr() : nullptr; }
const int32_t *words(const at::Tensor *t) { return static_cast<const int32_t *>(ptr(t)); }

// Nothing between this call and the GPU that Python code would have been asked about.
bool quiet() { return !at::impl::torch_function_mode_enabled() && !c10::impl::dispatch_mode_enabled(); }

struct Operands {          // of one packed layer
	const at::Tensor *qweight, *scales, *qzeros;
	int64_t K, N;
	bool load(PyObject *const *a, int device) {
		qweight = plain(a[0], at::kInt, device);
		scales = qweight ? plain(a[1], at::kHalf, device) : nullptr;
		qzeros = scales ? plain(a[2], at::kInt, device) : nullptr;
		if (!qzeros || qweight->dim() != 2) return false;
		K = qweight->size(0) * 8;
		N = qweight->size(1);
		return true;
	}
};

// Rows of x, the workspace of this device and stream, and whether the library has a kernel for the call.
struct Call {
	const at::Tensor *x = nullptr;
	int device = -1;
	int64_t M = 0;
	cudaStream_t stream = nullptr;
	void *ws = nullptr;
	size_t ws_bytes = 0;

	bool input(PyObject *o) {
		x = plain(o, at::kHalf, -1);
		if (!x || x->dim() < 1 || x->numel() == 0) return false;
		device = x->get_device();
		return device == c10::cuda::current_device();
	}
	bool rows(const Operands &w, int64_t groupsize, bool act_order, bool tensor_cores) {
		if (x->size(-1) != w.K || w.K == 0) return false;
		M = x->numel() / w.K;
		if (M > (1 << 20) || w.K > (1 << 24) || w.N > (1 << 24)) return false;
		if (M <= 16) return true;
		const int64_t gs = groupsize == -1 ? w.K : groupsize;          // (the rule of prefill_kernel_available)
		return tensor_cores && !act_order && w.N % 128 == 0 && w.K % 64 == 0 && gs > 0 && gs % 64 == 0 && w.K % gs == 0;
	}
	bool workspace(PyObject *table, int64_t K, int64_t N) {
		stream = c10::cuda::getCurrentCUDAStream(device).stream();
		PyObject *key = Py_BuildValue("(iK)", device, reinterpret_cast<unsigned long long>(stream));
		if (!key) {
			PyErr_Clear();
			return false;
		}
		PyObject *found = PyDict_Check(table) ? PyDict_GetItemWithError(table, key) : nullptr;
		Py_DECREF(key);
		if (!found) {
			PyErr_Clear();
			return false;
		}
		const at::Tensor *t = plain(found, at::kByte, device);
		if (!t) return false;
		ws = t->data_ptr();
		ws_bytes = t->numel();
		return ws_bytes >= workspace_bytes((int)M, (int)K, (int)N);
	}
};

PyObject *none() { Py_RETURN_NONE; }

// Runs f, which returns a new reference or nullptr for "not the plain case"; no C++ exception leaves.
template <typename F>
PyObject *guarded(F &&f) {
	try {
		if (quiet())
			if (PyObject *r = f()) return r;
	} catch (...) {
	}
	PyErr_Clear();
	return none();
}

bool integer(PyObject *o, int64_t &v) {
	if (!PyLong_CheckExact(o)) return false;
	v = PyLong_AsLongLong(o);
	return !(v == -1 && PyErr_Occurred()) && v >= -1 && v <= (1 << 24);
}

at::Tensor like(const Call &c, int64_t N) {
	c10::SmallVector<int64_t, 6> sizes(c.x->sizes().begin(), c.x->sizes().end());
	sizes.back() = N;
	return at::empty(sizes, at::TensorOptions().dtype(at::kHalf).device(c.x->device()));
}

// qmatmul(workspaces, tensor_cores, groupsize, x, qweight, scales, qzeros, bias, perm, residual)
PyObject *qmatmul(PyObject *, PyObject *const *a, Py_ssize_t n) {
	return guarded([&]() -> PyObject * {
		Call c;
		Operands w;
		int64_t gs;
		bool ok = n == 10 && qmatmul_fn && integer(a[2], gs) && c.input(a[3]) && w.load(a + 4, c.device);
		if (!ok) return nullptr;
		const at::Tensor *bias = maybe(a[7], at::kHalf, c.device, ok), *perm = maybe(a[8], at::kInt, c.device, ok), *res = maybe(a[9], at::kHalf, c.device, ok);
		if (!ok || !c.rows(w, gs, perm, a[1] == Py_True) || (res && res->numel() != c.M * w.N) || !c.workspace(a[0], w.K, w.N)) return nullptr;
		at::Tensor y = like(c, w.N);
		if (y.key_set().has(c10::DispatchKey::Python)) return nullptr;
		int rc;
		void *out = y.data_ptr();
		Py_BEGIN_ALLOW_THREADS
		rc = qmatmul_fn(ptr(c.x), words(w.qweight), words(w.qzeros), ptr(w.scales), nullptr, words(perm), ptr(bias), ptr(res), w.N, out, (int)c.M, (int)w.K, (int)w.N, (int)gs,
						w.K, w.N, c.ws, c.ws_bytes, reinterpret_cast<gptq_stream_t>(c.stream));
		Py_END_ALLOW_THREADS
		return rc == GPTQ_OK ? THPVariable_Wrap(std::move(y)) : nullptr;
	});
}

// gateup(workspaces, tensor_cores, groupsize, x, gate qweight, scales, qzeros, up qweight, scales, qzeros, perm)
PyObject *gateup(PyObject *, PyObject *const *a, Py_ssize_t n) {
	return guarded([&]() -> PyObject * {
		Call c;
		Operands g, u;
		int64_t gs;
		bool ok = n == 11 && gateup_fn && integer(a[2], gs) && c.input(a[3]) && g.load(a + 4, c.device) && u.load(a + 7, c.device);
		if (!ok || g.K != u.K || g.N != u.N || !g.scales->sizes().equals(u.scales->sizes()) || !g.qzeros->sizes().equals(u.qzeros->sizes())) return nullptr;
		const at::Tensor *perm = maybe(a[10], at::kInt, c.device, ok);
		if (!ok || !c.rows(g, gs, perm, a[1] == Py_True) || !c.workspace(a[0], g.K, g.N)) return nullptr;
		at::Tensor y = like(c, g.N);
		if (y.key_set().has(c10::DispatchKey::Python)) return nullptr;
		int rc;
		void *out = y.data_ptr();
		Py_BEGIN_ALLOW_THREADS
		rc = gateup_fn(ptr(c.x), words(g.qweight), words(g.qzeros), ptr(g.scales), words(u.qweight), words(u.qzeros), ptr(u.scales), nullptr, words(perm), out, (int)c.M, (int)g.K,
					   (int)g.N, (int)gs, g.K, g.N, c.ws, c.ws_bytes, reinterpret_cast<gptq_stream_t>(c.stream));
		Py_END_ALLOW_THREADS
		return rc == GPTQ_OK ? THPVariable_Wrap(std::move(y)) : nullptr;
	});
}

// qkv(workspaces, tensor_cores, groupsize, x [b, t, K], qweight, scales, qzeros, cos, sin, positions int32 [b * t], heads, head_dim, perm) -> (q, k, v), each [b, heads, t, head_dim]
PyObject *qkv(PyObject *, PyObject *const *a, Py_ssize_t n) {
	return guarded([&]() -> PyObject * {
		Call c;
		Operands w;
		int64_t gs, H, D;
		bool ok = n == 13 && qkv_fn && integer(a[2], gs) && c.input(a[3]) && c.x->dim() == 3 && w.load(a + 4, c.device) && integer(a[10], H) && integer(a[11], D) && H > 0 && D > 0;
		if (!ok) return nullptr;
		const at::Tensor *cos = plain(a[7], at::kHalf, c.device), *sin = plain(a[8], at::kHalf, c.device), *pos = plain(a[9], at::kInt, c.device);
		const at::Tensor *perm = maybe(a[12], at::kInt, c.device, ok);
		if (!ok || !cos || !sin || !pos || cos->dim() != 2 || w.N != 3 * H * D || !c.rows(w, gs, perm, a[1] == Py_True) || pos->numel() != c.M || !c.workspace(a[0], w.K, w.N))
			return nullptr;
		const int64_t b = c.x->size(0), t = c.x->size(1);
		const auto options = at::TensorOptions().dtype(at::kHalf).device(c.x->device());
		at::Tensor q = at::empty({b, t, H, D}, options), k = at::empty({b, H, t, D}, options), v = at::empty({b, H, t, D}, options);
		if ((q.key_set() | k.key_set() | v.key_set()).has(c10::DispatchKey::Python)) return nullptr;
		int rc;
		void *qp = q.data_ptr(), *kp = k.data_ptr(), *vp = v.data_ptr();
		Py_BEGIN_ALLOW_THREADS
		rc = qkv_fn(ptr(c.x), words(w.qweight), words(w.qzeros), ptr(w.scales), nullptr, words(perm), ptr(cos), ptr(sin), words(pos), (int)cos->size(0), qp, H * D, kp, vp, (int)t,
					H * t * D, D, t * D, 0, (int)c.M, (int)w.K, (int)H, (int)D, (int)gs, w.K, c.ws, c.ws_bytes, reinterpret_cast<gptq_stream_t>(c.stream));
		Py_END_ALLOW_THREADS
		if (rc != GPTQ_OK) return nullptr;
		PyObject *qo = THPVariable_Wrap(q.transpose(1, 2)), *ko = THPVariable_Wrap(std::move(k)), *vo = THPVariable_Wrap(std::move(v));
		PyObject *r = qo && ko && vo ? PyTuple_Pack(3, qo, ko, vo) : nullptr;
		Py_XDECREF(qo);
		Py_XDECREF(ko);
		Py_XDECREF(vo);
		return r;
	});
}

// bind(addresses of gptq_workspace_bytes, gptq_qmatmul, gptq_gateup_silu, gptq_qkv_rope)
PyObject *bind(PyObject *, PyObject *const *a, Py_ssize_t n) {
	if (n != 4) {
		PyErr_SetString(PyExc_TypeError, "bind() takes four addresses");
		return nullptr;
	}
	void *p[4];
	for (int i = 0; i < 4; ++i) {
		p[i] = PyLong_AsVoidPtr(a[i]);
		if (PyErr_Occurred()) return nullptr;
	}
	workspace_bytes = reinterpret_cast<decltype(workspace_bytes)>(p[0]);
	qmatmul_fn = reinterpret_cast<decltype(qmatmul_fn)>(p[1]);
	gateup_fn = reinterpret_cast<decltype(gateup_fn)>(p[2]);
	qkv_fn = reinterpret_cast<decltype(qkv_fn)>(p[3]);
	return none();
}

template <typename F>
PyCFunction fast(F f) { return reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(f)); }

PyMethodDef methods[] = {{"bind", fast(bind), METH_FASTCALL, nullptr}, {"qmatmul", fast(qmatmul), METH_FASTCALL, nullptr}, {"gateup", fast(gateup), METH_FASTCALL, nullptr},
						 {"qkv", fast(qkv), METH_FASTCALL, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}   // namespace

PyMODINIT_FUNC PyInit__host() { return PyModule_Create(&module); }
