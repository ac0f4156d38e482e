// Layer calls from Python without ctypes: checks, output allocation, workspace look-up and the launch of one C-ABI entry point.
//
// A call of the smallest layer is bound by the host: o_proj of a 7B layer for one token took 16.5 us a call, 5.5 of them on the GPU; the rest was
// Python (argument checks, torch.empty, nineteen ctypes conversions).  Every function here serves the plain case and returns None for anything
// else (other types, devices or layouts, tensor subclasses, a missing or small workspace, an active torch-function mode, an error code from the library);
// the caller then makes the whole call in Python, which supports or reports it.  What has been launched by then (attend() and a gate product come before
// a code of a later launch) wrote to tensors of its own only.  Exceptions of torch (out of memory, a CUDA error) go to the caller as they are.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/core/Tensor.h>
#include <ATen/core/grad_mode.h>
#include <ATen/ops/add.h>
#include <ATen/ops/cat.h>
#include <ATen/ops/empty.h>
#include <ATen/ops/index_select.h>
#include <ATen/ops/matmul.h>
#include <ATen/ops/mul.h>
#include <ATen/ops/scaled_dot_product_attention.h>
#include <ATen/ops/silu.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../../include/gptq_b200.h"

namespace {

// entry points of the library that the ctypes binding has loaded
decltype(&gptq_workspace_bytes) workspace_bytes = nullptr;
decltype(&gptq_qmatmul) qmatmul_fn = nullptr;
decltype(&gptq_gateup_silu) gateup_fn = nullptr;
decltype(&gptq_qkv_rope) qkv_fn = nullptr;
decltype(&gptq_dequantize) dequantize_fn = nullptr;
decltype(&gptq_attn_prompt_full_scratch_bytes) attend_scratch = nullptr;
decltype(&gptq_attn_prompt_prepare) attend_prepare = nullptr;
decltype(&gptq_attn_prompt) attend_fn = nullptr;

// A CUDA tensor of the given type on `device`, with nothing but data behind it (an empty pointer: not the plain case).
const at::Tensor *strided(PyObject *o, at::ScalarType type, int device) {
	if (!THPVariable_CheckExact(o)) {
		if (!THPVariable_Check(o) || Py_TYPE(o) != reinterpret_cast<PyTypeObject *>(ParameterClass)) return nullptr;
	}
	const at::Tensor &t = THPVariable_Unpack(o);
	const auto keys = t.key_set();
	if (!t.defined() || !t.has_storage() || t.layout() != at::kStrided || keys.has(c10::DispatchKey::Python) || keys.has(c10::DispatchKey::FuncTorchBatched) ||
		keys.has(c10::DispatchKey::FuncTorchGradWrapper) || keys.has(c10::DispatchKey::Functionalize) || !t.is_cuda() || t.scalar_type() != type ||
		(device >= 0 && t.get_device() != device) || t.is_conj() || t.is_neg())
		return nullptr;
	return &t;
}
// ... and contiguous
const at::Tensor *plain(PyObject *o, at::ScalarType type, int device) {
	const at::Tensor *t = strided(o, type, device);
	return t && t->is_contiguous() ? t : nullptr;
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
	at::Tensor held;          // the workspace: another thread may take it out of the table while the library runs without the GIL

	bool input(PyObject *o) {
		x = plain(o, at::kHalf, -1);
		if (!x || x->dim() < 1 || x->numel() == 0) return false;
		device = x->get_device();
		return device == c10::cuda::current_device();
	}
	// ... and, for a prompt, x[:, perm] in a tensor of its own (the tensor-core kernel reads x by TMA: gathered once up front)
	at::Tensor gathered;
	bool gather(const Operands &w, const at::Tensor *&perm) {
		if (M <= 16 || !perm) return true;
		if (perm->dim() != 1 || perm->numel() != w.K) return false;
		gathered = at::index_select(x->view({M, w.K}), 1, *perm);
		perm = nullptr;
		return !gathered.key_set().has(c10::DispatchKey::Python);
	}
	void *rows_ptr() const { return gathered.defined() ? gathered.data_ptr() : x->data_ptr(); }
	bool rows(const Operands &w, int64_t groupsize, bool tensor_cores) {
		if (x->size(-1) != w.K || w.K == 0) return false;
		M = x->numel() / w.K;
		if (M > (1 << 20) || w.K > (1 << 24) || w.N > (1 << 24)) return false;
		const int64_t gs = groupsize == -1 ? w.K : groupsize;          // (the rule of prefill_kernel_available)
		dense = M > 16 && !(tensor_cores && w.N % 128 == 0 && w.K % 64 == 0 && gs > 0 && gs % 64 == 0 && w.K % gs == 0);
		return !dense || dequantize_fn;
	}
	bool dense = false;          // a prompt that no kernel covers: dequantise and multiply
	at::Tensor product(const Operands &w, int64_t groupsize) const {
		at::Tensor full = at::empty({w.K, w.N}, at::TensorOptions().dtype(at::kHalf).device(x->device()));
		if (full.key_set().has(c10::DispatchKey::Python) ||
			dequantize_fn(words(w.qweight), words(w.qzeros), w.scales->data_ptr(), nullptr, full.data_ptr(), (int)w.K, (int)w.N, (int)groupsize, reinterpret_cast<gptq_stream_t>(stream)) !=
				GPTQ_OK)
			return at::Tensor();
		return at::matmul(gathered.defined() ? gathered : x->view({M, w.K}), full);
	}
	at::Tensor shaped(const at::Tensor &y) const {
		c10::SmallVector<int64_t, 6> sizes(x->sizes().begin(), x->sizes().end());
		sizes.back() = y.size(1);
		return y.view(sizes);
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
		held = *t;
		ws = t->data_ptr();
		ws_bytes = t->numel();
		return ws_bytes >= workspace_bytes((int)M, (int)K, (int)N);
	}
};

PyObject *none() { Py_RETURN_NONE; }

// Runs f, which returns a new reference or nullptr for "not the plain case"; a C++ exception becomes the Python one that torch makes of it.
template <typename F>
PyObject *guarded(F &&f) {
	HANDLE_TH_ERRORS
	if (quiet())
		if (PyObject *r = f()) return r;
	PyErr_Clear();
	return none();
	END_HANDLE_TH_ERRORS
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
		if (!ok || !c.rows(w, gs, a[1] == Py_True) || (res && res->numel() != c.M * w.N) || !c.workspace(a[0], w.K, w.N) || !c.gather(w, perm)) return nullptr;
		if (c.dense) {
			at::Tensor y = c.product(w, gs);
			if (!y.defined()) return nullptr;
			if (bias) y = at::add(y, *bias);
			if (res) y = at::add(y, res->view({c.M, w.N}));
			return THPVariable_Wrap(c.shaped(y));
		}
		at::Tensor y = like(c, w.N);
		if (y.key_set().has(c10::DispatchKey::Python)) return nullptr;
		int rc;
		void *out = y.data_ptr();
		Py_BEGIN_ALLOW_THREADS
		rc = qmatmul_fn(c.rows_ptr(), words(w.qweight), words(w.qzeros), ptr(w.scales), nullptr, words(perm), ptr(bias), ptr(res), w.N, out, (int)c.M, (int)w.K, (int)w.N, (int)gs,
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
		if (!ok || !c.rows(g, gs, a[1] == Py_True) || !c.workspace(a[0], g.K, g.N) || !c.gather(g, perm)) return nullptr;
		if (c.dense) {
			const at::Tensor a1 = c.product(g, gs), a2 = c.product(u, gs);
			if (!a1.defined() || !a2.defined()) return nullptr;
			return THPVariable_Wrap(c.shaped(at::mul(at::silu(a1.to(at::kFloat)), a2.to(at::kFloat)).to(at::kHalf)));
		}
		at::Tensor y = like(c, g.N);
		if (y.key_set().has(c10::DispatchKey::Python)) return nullptr;
		int rc;
		void *out = y.data_ptr();
		Py_BEGIN_ALLOW_THREADS
		rc = gateup_fn(c.rows_ptr(), words(g.qweight), words(g.qzeros), ptr(g.scales), words(u.qweight), words(u.qzeros), ptr(u.scales), nullptr, words(perm), out, (int)c.M, (int)g.K,
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
		if (!ok || !cos || !sin || !pos || cos->dim() != 2 || w.N != 3 * H * D || !c.rows(w, gs, a[1] == Py_True) || c.dense || pos->numel() != c.M || !c.workspace(a[0], w.K, w.N) || !c.gather(w, perm))
			return nullptr;
		const int64_t b = c.x->size(0), t = c.x->size(1);
		const auto options = at::TensorOptions().dtype(at::kHalf).device(c.x->device());
		at::Tensor q = at::empty({b, t, H, D}, options), k = at::empty({b, H, t, D}, options), v = at::empty({b, H, t, D}, options);
		if ((q.key_set() | k.key_set() | v.key_set()).has(c10::DispatchKey::Python)) return nullptr;
		int rc;
		void *qp = q.data_ptr(), *kp = k.data_ptr(), *vp = v.data_ptr();
		Py_BEGIN_ALLOW_THREADS
		rc = qkv_fn(c.rows_ptr(), words(w.qweight), words(w.qzeros), ptr(w.scales), nullptr, words(perm), ptr(cos), ptr(sin), words(pos), (int)cos->size(0), qp, H * D, kp, vp, (int)t,
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

// [b, heads, n, 128], rows contiguous, everything on 16 bytes
bool head_rows(const at::Tensor &t, int64_t b, int64_t heads) {
	return t.dim() == 4 && t.size(0) == b && t.size(1) == heads && t.size(3) == 128 && t.stride(3) == 1 && t.stride(2) == 128 && t.stride(0) % 8 == 0 && t.stride(1) % 8 == 0 &&
		   reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0;
}

// Attention of new tokens behind cached ones with an additive mask, up to the output projection:
// attend(workspaces, tensor_cores, groupsize, x [b, t, K], qweight, scales, qzeros, cos, sin, positions [b, t], heads, perm, mask [b, 1, t, S] fp16, past keys, past values)
//   -> (attention output [b, t, heads * 128], keys, values [b, heads, S, 128])
PyObject *attend(PyObject *, PyObject *const *a, Py_ssize_t n) {
	return guarded([&]() -> PyObject * {
		Call c;
		Operands w;
		int64_t gs, H;
		bool ok = n == 15 && attend_fn && integer(a[2], gs) && c.input(a[3]) && c.x->dim() == 3 && w.load(a + 4, c.device) && integer(a[10], H) && H > 0;
		if (!ok) return nullptr;
		const at::Tensor *cos = plain(a[7], at::kHalf, c.device), *sin = plain(a[8], at::kHalf, c.device), *ids = strided(a[9], at::kLong, c.device);
		const at::Tensor *perm = maybe(a[11], at::kInt, c.device, ok), *mask = strided(a[12], at::kHalf, c.device);
		if (!ids) ids = strided(a[9], at::kInt, c.device);
		const at::Tensor *pk = a[13] == Py_None ? nullptr : strided(a[13], at::kHalf, c.device), *pv = a[14] == Py_None ? nullptr : strided(a[14], at::kHalf, c.device);
		if (!ok || !cos || !sin || !ids || !mask || (a[13] != Py_None && !pk) || (a[14] != Py_None && !pv) || !pk != !pv || cos->dim() != 2 || cos->size(1) != 128 || w.N != 384 * H ||
			!c.rows(w, gs, a[1] == Py_True) || c.dense)
			return nullptr;
		const int64_t b = c.x->size(0), t = c.x->size(1), past = pk ? pk->size(2) : 0, S = past + t;
		if (at::GradMode::is_enabled() && (mask->requires_grad() || (pk && (pk->requires_grad() || pv->requires_grad())))) return nullptr;
		if (mask->dim() != 4 || mask->size(0) != b || mask->size(1) != 1 || mask->size(2) != t || mask->size(3) != S || mask->stride(3) != 1 || ids->numel() != c.M || S > (1 << 24)) return nullptr;
		if (pk && (!head_rows(*pk, b, H) || !head_rows(*pv, b, H) || pv->size(2) != past)) return nullptr;
		// Long prompts whose mask rows start on 16 bytes are better off with the library kernel.  Whole block, this kernel / library, us: 32 heads, t = 1000 198 / 169,
		// t = 400 of 5 sequences 312 / 295, t = 200 56 / 65, t = 64 40 / 65, t = 2 behind 100 36 / 80; 16 heads, t = 1200 98 / 105.  Rows off 16 bytes have to be
		// copied for it: t = 701 behind 64 110 / 143, t = 1300 behind 3 223 / 325, t = 2048 behind 1501 551 / 678; masks of the lowest value 117, 236, 577; biases that
		// hide nothing 135, 286, 702.
		// One token over many keys, or a few tokens of many heads: a CTA per head and 64 queries has little to do per key, the library kernel splits the keys. GPU time, us:
		// one token, 32 heads, 257 keys 32 / 33, 513 43 / 32, 1002 59 / 38, 4002 173 / 63, 16 sequences of 81 keys 45 / 55, of 256 82 / 65; 3 tokens, 4 sequences of 64 heads,
		// 258 keys 84 / 87, 1004 145 / 139, 4004 410 / 380; 2 tokens, 4 sequences of 32 heads, 1003 keys 83 / 88.
		const bool library = t == 1 ? S > 256 || b * H * S > 40000 : t <= 128 && b * H > 160 && S > 192;
		// A prompt in portions behind a long cache of many heads has little mask to copy: 200 behind 3001, 2 sequences of 64 heads 455 / 425, 140 behind 2001, 8 of 32 476 / 456;
		// 512 behind 2001, 2 of 32 308 / 305, 3 of 32 440 / 507.
		const bool off = t > 128 && !(b * H >= 64 && S >= 8 * t) && (mask->stride(2) % 8 != 0 || reinterpret_cast<uintptr_t>(mask->data_ptr()) % 16 != 0);
		if (!off && !library && b * H * t * S > (8 << 20)) return nullptr;
		if (!c.workspace(a[0], w.K, w.N) || !c.gather(w, perm)) return nullptr;
		const at::Tensor pos = ids->reshape({-1}).to(at::kInt).contiguous();
		const auto options = at::TensorOptions().dtype(at::kHalf).device(c.x->device());
		const int shared = b == 1 || mask->stride(0) == 0, mask_b = shared ? 1 : (int)b;
		const bool tiles = !library && (past > 0 || S > 128);          // (a launch less where there is next to nothing to skip)
		const size_t need = tiles ? attend_scratch(mask_b, (int)b, (int)H, (int)t, (int)S) : 0;
		const int64_t rows = library ? t : S;          // (the library route concatenates: rows written between the cached ones are copied at half the speed)
		at::Tensor q = at::empty({b, t, H, 128}, options), k = at::empty({b, H, rows, 128}, options), v = at::empty({b, H, rows, 128}, options), out;
		if (!library) out = at::empty({b, t, H * 128}, options);
		at::Tensor flags = at::empty({(int64_t)need}, options.dtype(at::kByte));
		if ((q.key_set() | k.key_set() | v.key_set() | flags.key_set() | pos.key_set()).has(c10::DispatchKey::Python)) return nullptr;
		int rc;
		void *qp = q.data_ptr(), *kp = k.data_ptr(), *vp = v.data_ptr(), *op = library ? nullptr : out.data_ptr(), *fp = tiles ? flags.data_ptr() : nullptr;
		const size_t skip = library ? 0 : (size_t)past * 128 * 2;
		const auto st = reinterpret_cast<gptq_stream_t>(c.stream);
		Py_BEGIN_ALLOW_THREADS
		rc = GPTQ_OK;
		if (tiles)
			rc = attend_prepare(ptr(mask), mask->stride(0), mask->stride(2), mask_b, (int)b, (int)H, (int)t, (int)S, ptr(pk), pk ? pk->stride(0) : 0, pk ? pk->stride(1) : 0, ptr(pv),
								pv ? pv->stride(0) : 0, pv ? pv->stride(1) : 0, (int)past, kp, vp, fp, need, st);
		if (rc == GPTQ_OK)
			rc = qkv_fn(c.rows_ptr(), words(w.qweight), words(w.qzeros), ptr(w.scales), nullptr, words(perm), ptr(cos), ptr(sin), words(&pos), (int)cos->size(0), qp, H * 128,
						static_cast<char *>(kp) + skip, static_cast<char *>(vp) + skip, (int)t, H * rows * 128, 128, rows * 128, 0, (int)c.M, (int)w.K, (int)H, 128, (int)gs, w.K, c.ws,
						c.ws_bytes, st);
		if (rc == GPTQ_OK && !library)
			rc = attend_fn(qp, t * H * 128, H * 128, 128, kp, vp, ptr(mask), mask->stride(0), mask->stride(2), mask_b, (int)b, (int)H, (int)t, (int)S, 0.08838834764831845f, op, fp, need, st);
		Py_END_ALLOW_THREADS
		if (rc != GPTQ_OK) return nullptr;
		if (library) {
			if (past) k = at::cat({*pk, k}, 2), v = at::cat({*pv, v}, 2);
			out = at::scaled_dot_product_attention(q.transpose(1, 2), k, v, *mask).transpose(1, 2).reshape({b, t, H * 128});
		}
		PyObject *oo = THPVariable_Wrap(std::move(out)), *ko = THPVariable_Wrap(std::move(k)), *vo = THPVariable_Wrap(std::move(v));
		PyObject *r = oo && ko && vo ? PyTuple_Pack(3, oo, ko, vo) : nullptr;
		Py_XDECREF(oo);
		Py_XDECREF(ko);
		Py_XDECREF(vo);
		return r;
	});
}

// bind(addresses of gptq_workspace_bytes, gptq_qmatmul, gptq_gateup_silu, gptq_qkv_rope, gptq_attn_prompt_full_scratch_bytes, _prepare, gptq_attn_prompt,
// gptq_dequantize)
PyObject *bind(PyObject *, PyObject *const *a, Py_ssize_t n) {
	if (n != 8) {
		PyErr_SetString(PyExc_TypeError, "bind() takes eight addresses");
		return nullptr;
	}
	void *p[8];
	for (int i = 0; i < 8; ++i) {
		p[i] = PyLong_AsVoidPtr(a[i]);
		if (PyErr_Occurred()) return nullptr;
	}
	workspace_bytes = reinterpret_cast<decltype(workspace_bytes)>(p[0]);
	qmatmul_fn = reinterpret_cast<decltype(qmatmul_fn)>(p[1]);
	gateup_fn = reinterpret_cast<decltype(gateup_fn)>(p[2]);
	qkv_fn = reinterpret_cast<decltype(qkv_fn)>(p[3]);
	attend_scratch = reinterpret_cast<decltype(attend_scratch)>(p[4]);
	attend_prepare = reinterpret_cast<decltype(attend_prepare)>(p[5]);
	attend_fn = reinterpret_cast<decltype(attend_fn)>(p[6]);
	dequantize_fn = reinterpret_cast<decltype(dequantize_fn)>(p[7]);
	return none();
}

template <typename F>
PyCFunction fast(F f) { return reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(f)); }

PyMethodDef methods[] = {{"bind", fast(bind), METH_FASTCALL, nullptr}, {"qmatmul", fast(qmatmul), METH_FASTCALL, nullptr}, {"gateup", fast(gateup), METH_FASTCALL, nullptr},
						 {"qkv", fast(qkv), METH_FASTCALL, nullptr}, {"attend", fast(attend), METH_FASTCALL, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}   // namespace

PyMODINIT_FUNC PyInit__host() {
	PyObject *m = PyModule_Create(&module);
	if (m && PyModule_AddStringConstant(m, "torch_version", GPTQ_TORCH_VERSION) != 0) Py_CLEAR(m);          // of the torch that it was compiled against
	return m;
}
