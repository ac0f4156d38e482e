"""ctypes binding of libgptq_b200.so (declared in include/gptq_b200.h).

There is no fallback: if the library is missing or a kernel cannot run, an exception is
raised.  The library is built in-tree by `python -m gptq_triton_b200.build`.  (The extension
module of host() is another way into the same library, and can be missing.)
"""
from __future__ import annotations

import ctypes
import functools
import os
import warnings
from ctypes import c_char_p, c_int, c_int64, c_size_t, c_void_p
from pathlib import Path
from typing import Dict, Optional, Tuple

import torch

_PKG = Path(__file__).resolve().parent
LIB_PATH = _PKG / 'libgptq_b200.so'

_lib: Optional[ctypes.CDLL] = None
_host = None          # extension module csrc/host/calls.cpp, bound to the library, or what stands for it (see host())

_P = c_void_p
_SIGNATURES = {
	'gptq_version': (c_int, []),
	'gptq_error_string': (c_char_p, [c_int]),
	'gptq_last_cuda_error': (c_int, []),
	'gptq_workspace_bytes': (c_size_t, [c_int, c_int, c_int]),
	'gptq_qmatmul': (c_int, [_P, _P, _P, _P, _P, _P, _P, _P, c_int64, _P, c_int, c_int, c_int, c_int, c_int64, c_int64, _P, c_size_t, _P]),
	'gptq_gateup_silu': (c_int, [_P, _P, _P, _P, _P, _P, _P, _P, _P, _P, c_int, c_int, c_int, c_int, c_int64, c_int64, _P, c_size_t, _P]),
	'gptq_qkv_rope': (c_int, [_P, _P, _P, _P, _P, _P, _P, _P, _P, c_int, _P, c_int64, _P, _P, c_int, c_int64, c_int64, c_int64, c_int64,
							  c_int, c_int, c_int, c_int, c_int, c_int64, _P, c_size_t, _P]),
	'gptq_qmatmul_sumsq': (c_int, [_P, _P, _P, _P, _P, _P, _P, _P, c_int64, _P, c_int, c_int, c_int, c_int, c_int64, c_int64, _P, c_size_t, _P, _P]),
	'gptq_gateup_silu_rms': (c_int, [_P, _P, _P, _P, _P, _P, _P, _P, _P, _P, c_int, c_int, c_int, c_int, c_int64, c_int64, _P, c_size_t, _P,
									 _P, _P, c_int, ctypes.c_float]),
	'gptq_qkv_rope_rms': (c_int, [_P, _P, _P, _P, _P, _P, _P, _P, _P, c_int, _P, c_int64, _P, _P, c_int, c_int64, c_int64, c_int64, c_int64,
								  c_int, c_int, c_int, c_int, c_int, c_int64, _P, c_size_t, _P, _P, _P, c_int, ctypes.c_float]),
	'gptq_ar_partial_bytes': (c_size_t, [c_int]),
	'gptq_ar_flag_bytes': (c_size_t, [c_int]),
	'gptq_qmatmul_ar': (c_int, [_P, _P, _P, _P, _P, _P, _P, _P, c_int64, _P, c_int, c_int, c_int, c_int, c_int64, c_int64, _P, c_size_t, _P, _P,
								c_int, c_int, _P, _P]),
	'gptq_peer_alloc': (c_int, [c_size_t, ctypes.POINTER(c_void_p)]),
	'gptq_peer_free': (c_int, [_P]),
	'gptq_peer_export': (c_int, [_P, _P]),
	'gptq_peer_open': (c_int, [_P, ctypes.POINTER(c_void_p)]),
	'gptq_peer_close': (c_int, [_P]),
	'gptq_unpack_qweight': (c_int, [_P, _P, c_int, c_int, _P]),
	'gptq_unpack_qzeros': (c_int, [_P, _P, c_int, c_int, _P]),
	'gptq_dequantize': (c_int, [_P, _P, _P, _P, _P, c_int, c_int, c_int, _P]),
	'gptq_act_order_rows': (c_int, [_P, _P, _P, c_int, c_int, _P]),
	'gptq_attn_workspace_bytes': (c_size_t, [c_int, c_int]),
	'gptq_qkv_attn_supported': (c_int, [c_int, c_int, c_int, c_int]),
	'gptq_qkv_attn_decode': (c_int, [_P, _P, _P, _P, _P, _P, _P, c_int, _P, _P, c_int64, _P, c_int, c_int, c_int, c_int, ctypes.c_float, _P, _P, c_int,
									 ctypes.c_float, _P, c_size_t, _P]),
	'gptq_qkv_attn_oproj_scratch_bytes': (c_size_t, [c_int, c_int]),
	'gptq_qkv_attn_oproj_decode': (c_int, [_P, _P, _P, _P, _P, _P, _P, c_int, _P, _P, c_int64, c_int, c_int, c_int, c_int, ctypes.c_float, _P, _P, c_int,
										   ctypes.c_float, _P, _P, _P, c_int, c_int, _P, _P, _P, _P, _P, c_size_t, _P, c_size_t, _P]),
	'gptq_qkv_attn_oproj_decode_ar': (c_int, [_P, _P, _P, _P, _P, _P, _P, c_int, _P, _P, c_int64, c_int, c_int, c_int, c_int, ctypes.c_float, _P, _P, c_int,
											  ctypes.c_float, _P, _P, _P, c_int, c_int, _P, _P, _P, _P, _P, c_size_t, _P, c_size_t, _P, c_int, c_int, _P, _P]),
	'gptq_attn_decode': (c_int, [_P, c_int64, _P, _P, c_int64, c_int64, _P, _P, c_int64, c_int, c_int, c_int, c_int, ctypes.c_float, _P, c_size_t, _P]),
	'gptq_rmsnorm': (c_int, [_P, c_int64, _P, _P, c_int64, c_int, c_int, ctypes.c_float, _P]),
	'gptq_embed_rmsnorm': (c_int, [_P, c_int64, c_int64, _P, _P, _P, c_int64, _P, c_int64, c_int, c_int, ctypes.c_float, _P]),
	'gptq_qmatmul_noalloc': (c_int, [_P, _P, _P, _P, _P, _P, _P, c_int64, _P, c_int, c_int, c_int, c_int, c_int64, c_int64, _P]),
	'gptq_noalloc_scratch_bytes': (c_size_t, [c_int, c_int, c_int, c_int]),
	'gptq_noalloc_status': (c_int, [c_int]),
	'gptq_attn_prompt_scratch_bytes': (c_size_t, [c_int, c_int, c_int]),
	'gptq_attn_prompt_full_scratch_bytes': (c_size_t, [c_int, c_int, c_int, c_int, c_int]),
	'gptq_attn_prompt_prepare': (c_int, [_P, c_int64, c_int64, c_int, c_int, c_int, c_int, c_int, _P, c_int64, c_int64, _P, c_int64, c_int64, c_int, _P, _P, _P, c_size_t, _P]),
	'gptq_attn_prompt': (c_int, [_P, c_int64, c_int64, c_int64, _P, _P, _P, c_int64, c_int64, c_int, c_int, c_int, c_int, c_int, ctypes.c_float, _P, _P, c_size_t, _P]),
	'gptq_chain_supported': (c_int, [c_int, c_int, c_int, c_int, c_int]),
	'gptq_chain_desc_bytes': (c_size_t, [c_int]),
	'gptq_chain_scratch_bytes': (c_size_t, [c_int, c_int, c_int, c_int, c_int]),
	'gptq_chain_build': (c_int, [_P, c_int, c_int, c_int, _P]),
	'gptq_decode_chain': (c_int, [_P, c_int, c_int, c_int, c_int, c_int, c_int, _P, _P, _P, _P, _P, c_int, c_int64, c_int64, ctypes.c_float,
							  _P, _P, _P, c_size_t, _P]),
	'gptq_lm_head_workspace_bytes': (c_size_t, [c_int]),
	'gptq_lm_head_argmax': (c_int, [_P, _P, _P, _P, c_int, c_int, c_int, ctypes.c_float, _P, _P, _P, _P, c_size_t, _P]),
}
# Entry points outside the header's stable surface (tuning hooks); bound when present.
_OPTIONAL = {
	'gptq_debug_force_splitk': (None, [c_int]),
	'gptq_debug_max_stages': (None, [c_int]),
	'gptq_debug_max_stages2': (None, [c_int]),
	'gptq_debug_set_pdl': (None, [c_int]),
	'gptq_debug_qa_stages': (None, [c_int]),
	'gptq_debug_soft_max_splits': (None, [c_int]),
	'gptq_debug_allow_narrow': (None, [c_int]),
	'gptq_debug_tc_force': (None, [c_int]),
	'gptq_debug_dec_min_rows': (None, [c_int]),
	'gptq_debug_tc_splitk': (None, [c_int]),
	'gptq_debug_chain_stages': (None, [c_int]),
}


def exported_symbols():
	"""Names that include/gptq_b200.h declares."""
	return list(_SIGNATURES)


def lib() -> ctypes.CDLL:
	global _lib
	if _lib is None:
		if not LIB_PATH.exists():
			raise ImportError(
				f'{LIB_PATH} is missing: build it with `python -m gptq_triton_b200.build` '
				'(needs nvcc with sm_100a support). There is no CPU or Triton fallback.')
		l = ctypes.CDLL(str(LIB_PATH))
		for name, (res, args) in _SIGNATURES.items():
			fn = getattr(l, name)
			fn.restype = res
			fn.argtypes = args
		for name, (res, args) in _OPTIONAL.items():
			if hasattr(l, name):
				fn = getattr(l, name)
				fn.restype = res
				fn.argtypes = args
		if os.environ.get('GPTQ_B200_STAGES') and hasattr(l, 'gptq_debug_max_stages'):
			l.gptq_debug_max_stages(int(os.environ['GPTQ_B200_STAGES']))      # ring depth of the decode kernel (A/B measurements)
		if os.environ.get('GPTQ_B200_PDL', '1') == '0' and hasattr(l, 'gptq_debug_set_pdl'):
			l.gptq_debug_set_pdl(0)      # opt out of programmatic dependent launch (A/B measurements)
		_lib = l
	return _lib


class _Ctypes:
	"""In the place of the extension module: serves nothing, so every call goes through ctypes."""
	qmatmul = gateup = qkv = attend = staticmethod(lambda *a: None)


def host():
	"""Layer calls in native code; each returns None when the call is not the plain case.  Without the module, or with one that was built
	against another torch, the layers run through ctypes (several microseconds more per call)."""
	global _host
	if _host is None:
		try:
			l = lib()
		except ImportError:
			return _Ctypes          # (said by whatever needs the library)
		try:
			from . import _host as module
			built = getattr(module, 'torch_version', 'unknown')
			if built != str(torch.__version__):
				raise ImportError(f'built against torch {built}, this is {torch.__version__}')
		except ImportError as e:
			warnings.warn(f'{_PKG / "_host.so"} is not used ({e}): layer calls take several microseconds more; build it with `python -m gptq_triton_b200.build`.', RuntimeWarning)
			_host = _Ctypes
			return _host
		address = lambda name: ctypes.cast(getattr(l, name), c_void_p).value
		module.bind(*map(address, ('gptq_workspace_bytes', 'gptq_qmatmul', 'gptq_gateup_silu', 'gptq_qkv_rope', 'gptq_attn_prompt_full_scratch_bytes',
									 'gptq_attn_prompt_prepare', 'gptq_attn_prompt', 'gptq_dequantize')))
		_host = module
	return _host


class GptqB200Error(RuntimeError):
	pass


def check(code: int, what: str):
	if code != 0:
		l = lib()
		msg = l.gptq_error_string(code).decode()
		extra = f' (cudaError {l.gptq_last_cuda_error()})' if code == -5 else ''
		err = ValueError if code in (-1, -2, -4) else GptqB200Error
		raise err(f'{what}: {msg}{extra}')


# Addresses and streams go to ctypes as plain integers and the stream is asked for without building a Stream object.
def ptr(t: Optional[torch.Tensor]):
	return None if t is None else t.data_ptr()


def stream_ptr(device) -> int:
	return _raw_stream(torch.cuda.current_device() if device.index is None else device.index)


def _raw_stream(index: int) -> int:
	return torch.cuda.current_stream(index).cuda_stream


_raw_stream = getattr(torch._C, '_cuda_getCurrentRawStream', _raw_stream)


def require_cuda(*tensors):
	for t in tensors:
		if t is not None and not t.is_cuda:
			raise GptqB200Error('gptq_triton_b200 runs on CUDA tensors only; there is no CPU path')


# One zero-initialised scratch buffer per (device, stream): split-K partial sums and the
# arrival counters that the kernels leave zeroed after each launch.
_workspaces: Dict[Tuple[int, int], torch.Tensor] = {}


@functools.lru_cache(maxsize=4096)
def _workspace_bytes(M: int, K: int, N: int) -> int:          # (depends on the sizes alone)
	return lib().gptq_workspace_bytes(M, K, N)


def workspace(device: torch.device, M: int, K: int, N: int, min_bytes: int = 0) -> torch.Tensor:
	need = max(_workspace_bytes(M, K, N), min_bytes)
	index = device.index if device.index is not None else torch.cuda.current_device()
	key = (index, _raw_stream(index))
	ws = _workspaces.get(key)
	if ws is None or ws.numel() < need:
		if ws is not None:
			_retired.append(ws)     # a captured CUDA graph may still point at it
		ws = torch.zeros(max(need, 1 << 20), dtype=torch.uint8, device=device)
		_workspaces[key] = ws
	return ws


_retired = []
_status_buffers = []      # scratch areas of other kernels whose status word sits at the same offset (bytes 16380..16383)


def register_status_buffer(buf: torch.Tensor):
	"""Includes the status word of `buf` (a kernel's scratch area, first 16 KiB = control words) in kernel_status()."""
	import weakref
	_status_buffers.append(weakref.ref(buf))


def kernel_status(device=None) -> int:
	"""OR of the status words that the decode kernels keep in their workspaces (0 = healthy;
	1 = a TMA / bulk load never completed within the bounded wait; 2 = shared memory misaligned;
	3 = a wait inside the tensor-core kernel ran out; 4 = position outside the rotary table / cache, or token outside the vocabulary;
	5 = a peer never arrived in the fused tensor-parallel all-reduce; 6 = a split-K partial sum never arrived;
	7 = a grid barrier of the persistent decode-step kernel timed out)."""
	st = 0
	for (dev, _), ws in _workspaces.items():
		if device is None or dev == (device.index if isinstance(device, torch.device) else device):
			st |= int(ws[16384 - 4:16384].view(torch.int32).item())
	for ref in _status_buffers:
		buf = ref()
		if buf is not None and (device is None or buf.device.index == (device.index if isinstance(device, torch.device) else device)):
			st |= int(buf[16384 - 4:16384].view(torch.int32).item())
	return st


def clear_kernel_status():
	"""Resets the status words (after the cause of a non-zero status has been dealt with) and, with them, the whole control area of every
	scratch buffer: arrival counters, hand-over flags and barriers, which a launch that gave up leaves behind and which the next one would
	take for its own.  Buffers that only captured graphs still use are among them.  Waits for the devices, since the buffers belong to
	several streams."""
	buffers = [*_workspaces.values(), *_retired, *(buf for buf in (ref() for ref in _status_buffers) if buf is not None)]
	devices = {buf.device for buf in buffers if buf.is_cuda}
	for device in devices:
		torch.cuda.synchronize(device)
	for buf in buffers:
		buf[:16384].zero_()
	for device in devices:
		torch.cuda.synchronize(device)
