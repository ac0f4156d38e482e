"""Layer calls through the extension module against the same calls through ctypes: the same bits for everything that either takes, the same
errors for what is refused."""
import pytest
import torch

import gptq_triton_b200 as G
from gptq_triton_b200 import _lib, synth

pytestmark = pytest.mark.gpu


class _Declines:
	"""Stands for the extension module and serves nothing."""
	qmatmul = gateup = qkv = staticmethod(lambda *a: None)


def _both(monkeypatch, call):
	"""call() through the extension module (which must serve it) and through ctypes."""
	served = []
	host = _lib.host()

	class Counts:
		pass
	for name in ('qmatmul', 'gateup', 'qkv'):
		setattr(Counts, name, staticmethod(lambda *a, f=getattr(host, name): served.append(f(*a)) or served[-1]))
	with monkeypatch.context() as m:
		m.setattr(_lib, '_host', Counts)
		new = call()
	with monkeypatch.context() as m:
		m.setattr(_lib, '_host', _Declines)
		old = call()
	return new, old, served


def _layer(K, N, gs, bias=False, act=False, seed=1):
	t = synth.quant_tensors(K, N, gs, seed=seed, bias=bias)
	layer = G.QuantLinear(4, gs, K, N, bias)
	layer.qweight, layer.qzeros, layer.scales = t['qweight'], t['qzeros'], t['scales']
	if bias:
		layer.bias = t['bias']
	layer = layer.cuda()
	if act:
		g = K if gs == -1 else gs
		layer.set_g_idx((torch.arange(K, dtype=torch.int32) // g)[torch.randperm(K, generator=torch.Generator().manual_seed(seed))])
	return layer


@pytest.mark.parametrize('M,K,N,gs,bias,act', [(1, 256, 128, 128, False, False), (7, 512, 256, -1, True, False), (16, 1024, 384, 128, True, True), (17, 512, 256, 64, False, False),
												(40, 1024, 256, 128, True, False), (3, 96, 40, 32, False, False),
												(40, 1024, 256, 128, False, True), (40, 256, 72, 32, True, False), (20, 256, 128, 32, False, True)])
@pytest.mark.parametrize('residual', [False, True])
def test_linear(monkeypatch, M, K, N, gs, bias, act, residual):
	layer = _layer(K, N, gs, bias, act)
	x = torch.randn(1, M, K, device='cuda').half()
	r = torch.randn(1, M, N, device='cuda').half() if residual else None
	layer(x, residual=r)          # (the workspace is there)
	new, old, served = _both(monkeypatch, lambda: layer(x, residual=r))
	assert served[0] is not None and new.shape == old.shape and torch.equal(new, old)


@pytest.mark.parametrize('M', [1, 16, 33])
@pytest.mark.parametrize('gs,act', [(128, False), (32, False), (128, True)])
def test_mlp_and_qkv(monkeypatch, M, gs, act):
	H, I = 256, 384
	gate, up = (_layer(H, I, gs, act=act, seed=s) for s in (1, 3))
	up.set_g_idx(gate.g_idx)
	mlp = G.QuantLlamaMLP(gate, _layer(I, H, gs, act=act, seed=2), up)
	x = torch.randn(1, M, H, device='cuda').half()
	attn = G.QuantLlamaAttention(G.LlamaConfig(hidden_size=H, num_attention_heads=2), _layer(H, 3 * H, 128, seed=4), _layer(H, H, 128, seed=5), None)
	mlp(x), attn(x)
	new, old, served = _both(monkeypatch, lambda: mlp(x))
	assert len(served) == 2 and None not in served and torch.equal(new, old)
	new, old, served = _both(monkeypatch, lambda: attn(x, use_cache=True))
	assert len(served) == 2 and not any(s is None for s in served)
	assert torch.equal(new[0], old[0]) and all(torch.equal(a, b) and a.stride() == b.stride() for a, b in zip(new[2], old[2]))


def test_what_is_not_the_plain_case(monkeypatch):
	"""Declined by the extension module, and served or refused as before: other layouts, types and devices, tensor subclasses, a torch-function
	mode, a batch dimension of vmap; a missing workspace, other streams and graph capture work."""
	layer = _layer(256, 128, 128)
	x = torch.randn(2, 256, device='cuda').half()
	y = layer(x)
	wide = torch.randn(2, 300, device='cuda').half()
	with pytest.raises(AssertionError):
		layer(wide[:, :256])
	with pytest.raises(AssertionError):
		layer(wide)
	with pytest.raises(TypeError):
		layer(x.float())
	with pytest.raises(G._lib.GptqB200Error):
		layer(x.cpu())
	with pytest.raises(RuntimeError):
		torch.func.vmap(layer)(x)
	assert layer(x[:0]).shape == (0, 128)

	class Sub(torch.Tensor):
		pass
	assert torch.equal(layer(x.as_subclass(Sub)), y)

	class Mode(torch.overrides.TorchFunctionMode):
		seen = []

		def __torch_function__(self, f, types, args=(), kwargs=None):
			self.seen.append(f)
			return f(*args, **(kwargs or {}))
	with Mode():
		assert torch.equal(layer(x), y)
	assert torch.empty in Mode.seen          # the mode saw the allocation, as before
	with monkeypatch.context() as m:
		m.setattr(_lib, '_workspaces', {})
		assert torch.equal(layer(x), y) and len(_lib._workspaces) == 1
	side = torch.cuda.Stream()
	side.wait_stream(torch.cuda.current_stream())
	with torch.cuda.stream(side):
		a, b = layer(x), layer(x)
	side.synchronize()
	assert torch.equal(a, y) and torch.equal(b, y)
	graph = torch.cuda.CUDAGraph()
	with torch.cuda.graph(graph):
		z = layer(x)
	z.zero_()
	graph.replay()
	assert torch.equal(z, y)
	p = x.clone().requires_grad_()
	assert not layer(p).requires_grad


def test_workspace_outlives_the_call(monkeypatch):
	"""The library runs without the GIL, so another thread may replace the workspace meanwhile: the call keeps the one it was given.  A callback
	stands for the library here and launches nothing."""
	import ctypes
	import gc
	layer = _layer(256, 128, 128)
	x = torch.randn(2, 256, device='cuda').half()
	layer(x)
	l, host = _lib.lib(), _lib.host()
	names = ('gptq_workspace_bytes', 'gptq_qmatmul', 'gptq_gateup_silu', 'gptq_qkv_rope', 'gptq_attn_prompt_full_scratch_bytes', 'gptq_attn_prompt_prepare', 'gptq_attn_prompt', 'gptq_dequantize')
	addresses = [ctypes.cast(getattr(l, n), ctypes.c_void_p).value for n in names]
	table = {(0, torch.cuda.current_stream().cuda_stream): torch.zeros(64 << 20, dtype=torch.uint8, device='cuda')}
	freed = []

	def replaced(*a):
		gc.collect()
		before = torch.cuda.memory_allocated()
		table.clear()
		freed.append(before - torch.cuda.memory_allocated())
		return 0
	callback = ctypes.CFUNCTYPE(ctypes.c_int, *_lib._SIGNATURES['gptq_qmatmul'][1])(replaced)
	monkeypatch.setattr(_lib, '_workspaces', table)
	try:
		host.bind(*(ctypes.cast(callback, ctypes.c_void_p).value if n == 'gptq_qmatmul' else a for n, a in zip(names, addresses)))
		assert layer(x) is not None
	finally:
		host.bind(*addresses)
	assert freed == [0] and not table


def test_an_exception_of_torch_reaches_the_caller(monkeypatch):
	"""Out of memory inside a native call is raised there and then; the call is not made a second time in Python."""
	layer = _layer(128, 8192, 128)
	x = torch.randn(1 << 16, 128, device='cuda').half()
	layer(x)          # (the workspace is there; the output took 1 GB)
	torch.cuda.empty_cache()
	again = []
	monkeypatch.setattr(_lib, 'require_cuda', lambda *a: again.append(a))
	total = torch.cuda.get_device_properties(0).total_memory
	try:
		torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (256 << 20)) / total)
		with pytest.raises(torch.OutOfMemoryError):
			layer(x)
	finally:
		torch.cuda.set_per_process_memory_fraction(1.0)
	assert not again and layer(x).shape == (1 << 16, 8192)


@pytest.mark.parametrize('M', [1, 16, 33])
def test_qkv_of_an_act_order_layer(monkeypatch, M):
	"""The QKV call with a permutation: gathered in the workspace up to 16 rows, in a tensor of its own above."""
	H = 256
	attn = G.QuantLlamaAttention(G.LlamaConfig(hidden_size=H, num_attention_heads=2), _layer(H, 3 * H, 128, act=True, seed=4), _layer(H, H, 128, seed=5), None)
	x = torch.randn(1, M, H, device='cuda').half()
	attn(x)
	new, old, served = _both(monkeypatch, lambda: attn(x, use_cache=True))
	assert len(served) == 2 and not any(s is None for s in served)
	assert torch.equal(new[0], old[0]) and all(torch.equal(a, b) and a.stride() == b.stride() for a, b in zip(new[2], old[2]))
