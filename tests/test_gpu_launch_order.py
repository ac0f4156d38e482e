"""Order of dependent launches: attention over a static cache directly behind the projections that fill it.

`attn_decode` and `qkv_attn_decode` read old cache rows ahead of their wait for the kernel in front, so nothing that still stores such rows
may be running by then.  Every sequence is captured into a graph (no host between the launches), the cache holds NaN before each replay,
and the results have to be those of the same calls with dependent launch off, bit for bit.
"""
import pytest
import torch

from oracle import gptq_oracle as O

pytestmark = pytest.mark.gpu

H, D, S, GS = 2, 128, 512, 128


@pytest.fixture(scope='module')
def G():
	import gptq_triton_b200 as g
	from gptq_triton_b200 import build
	build.build()
	return g


def weights(K, seed):
	from gptq_triton_b200 import synth
	w = synth.quant_tensors(K, 3 * H * D, GS, seed)
	return w['qweight'].cuda(), w['scales'].cuda(), w['qzeros'].cuda()


# rows of the launches that fill the cache: more than 16 run on the prompt kernel, 7 to 16 on the decode kernel that keeps weights in tensor
# memory, fewer on the other one; single rows come last (the part of the cache that attn_decode reads late; qkv_attn_decode reads none late)
ORDERS = [(rows, reader) for rows in ([20], [100], [300], [24, 8], [16], [5], [64, 7, 1]) for reader in ('attn_decode', 'attn_decode at once', 'qkv_attn_decode')
		  if rows[-1] > 1 or reader != 'qkv_attn_decode']


@pytest.mark.parametrize('rows,reader', ORDERS)
@pytest.mark.parametrize('K', [1024, 4096])
def test_attention_behind_the_projections_that_fill_the_cache(G, K, rows, reader):
	from gptq_triton_b200 import _lib
	from gptq_triton_b200.fused_attention import attn_decode, qkv_attn_decode
	w = weights(K, 5)
	cos, sin = (t.cuda() for t in O.rope_tables(D, S))
	t = sum(rows)
	kc, vc = (torch.empty((1, H, S, D), dtype=torch.float16, device='cuda') for _ in range(2))
	x = torch.empty((1, t + 1, K), dtype=torch.float16, device='cuda')
	cuts = [sum(rows[:i]) for i in range(len(rows) + 1)]
	xs = [x[:, a:b] for a, b in zip(cuts, cuts[1:])]
	pos = [torch.arange(a, b, dtype=torch.int32, device='cuda').unsqueeze(0) for a, b in zip(cuts, cuts[1:] + [t + 1])]
	new = torch.tensor([[t]], dtype=torch.int32, device='cuda')
	last = pos[-2][:, -1:].clone() if reader == 'attn_decode at once' else new

	def steps():
		for i, part in enumerate(xs):
			q, _, _ = G.qkv_rope(GS, part, *w, cos, sin, pos[i], H, D, kv_cache=(kc, vc))
		if reader == 'qkv_attn_decode':
			return qkv_attn_decode(GS, x[:, t:], *w, cos, sin, new.view(1), kc, vc, H)
		if reader == 'attn_decode':
			q, _, _ = G.qkv_rope(GS, x[:, t:], *w, cos, sin, new, H, D, kv_cache=(kc, vc))
		else:
			q = q[:, :, -1:]
		return attn_decode(q, kc, vc, last, t + 1)

	def fill(seed):
		x.copy_(torch.randn(x.shape, generator=torch.Generator(device='cuda').manual_seed(seed), device='cuda'))
		kc.fill_(float('nan'))
		vc.fill_(float('nan'))

	seeds = range(1, 13)
	want = []
	try:
		_lib.lib().gptq_debug_set_pdl(0)
		for seed in seeds:
			fill(seed)
			want.append(steps().clone())
	finally:
		_lib.lib().gptq_debug_set_pdl(1)
	assert all(bool(torch.isfinite(y).all()) for y in want)
	stream = torch.cuda.Stream()
	stream.wait_stream(torch.cuda.current_stream())
	with torch.cuda.stream(stream):
		steps()          # workspaces of this stream
		graph = torch.cuda.CUDAGraph()
		with torch.cuda.graph(graph, stream=stream):
			y = steps()
		for seed, ref in zip(seeds, want):
			fill(seed)
			graph.replay()
			assert torch.equal(y, ref), seed
	torch.cuda.synchronize()
	assert _lib.kernel_status() == 0
