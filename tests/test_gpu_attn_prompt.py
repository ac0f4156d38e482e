"""Attention of a prompt behind cached tokens with an additive mask: the kernels against 64 bits, and the calls of the attention block that run on
them against the path that they replace."""

import pytest
import torch

import gptq_triton_b200 as G
from gptq_triton_b200 import _lib, synth

pytestmark = pytest.mark.gpu
INF = float('inf')


def _mask(kind, b, t, S, gen):
	past = S - t
	hidden = torch.triu(torch.ones((t, S), dtype=torch.bool, device='cuda'), diagonal=past + 1)
	m = torch.zeros((b, 1, t, S), device='cuda', dtype=torch.float16)
	if kind == 'shared':
		return m[:1].masked_fill(hidden, -INF).expand(b, 1, t, S)
	if kind == 'lowest':
		return m.masked_fill(hidden, torch.finfo(torch.float16).min)
	if kind == 'random':
		return torch.randn((b, 1, t, S), generator=gen, device='cuda').half()
	if kind == 'padded':          # every sequence hides a different number of leading keys, and its first queries see nothing at all
		for i in range(b):
			m[i, :, :, :(i * 37) % S] = -INF
			m[i, :, :min(i, t)] = -INF
		return m.masked_fill(hidden, -INF)
	wide = torch.zeros((b, 1, t, S + 5), device='cuda', dtype=torch.float16)          # rows that start anywhere
	wide[..., 3:S + 3] = m.masked_fill(hidden, -INF)
	return wide[..., 3:S + 3]


@pytest.mark.parametrize('kind', ['shared', 'lowest', 'random', 'padded', 'wide'])
@pytest.mark.parametrize('b,H,t,past', [(1, 2, 1, 5), (3, 2, 7, 0), (2, 3, 64, 64), (1, 2, 65, 63), (3, 2, 130, 1), (2, 1, 63, 200), (1, 2, 300, 128)])
def test_kernels(kind, b, H, t, past):
	gen = torch.Generator(device='cuda').manual_seed(t)
	S, D = t + past, 128
	rnd = lambda *shape: torch.randn(shape, generator=gen, device='cuda').half()
	q, new_k, new_v, mask = rnd(b, t, H, D), rnd(b, H, t, D), rnd(b, H, t, D), _mask(kind, b, t, S, gen)
	old_k, old_v = rnd(b, H, past + 3, D)[:, :, :past], rnd(b, past, H, D).transpose(1, 2).contiguous()
	k, v = (torch.full((b, H, S, D), float('nan'), dtype=torch.float16, device='cuda') for _ in range(2))
	k[:, :, past:], v[:, :, past:] = new_k, new_v
	mask_b = 1 if mask.stride(0) == 0 else b
	need = _lib.lib().gptq_attn_prompt_scratch_bytes(mask_b, t, S)
	flags = torch.full((need + 64,), 7, dtype=torch.uint8, device='cuda')
	P, st = _lib.ptr, _lib.stream_ptr(q.device)
	where = (P(mask), mask.stride(0), mask.stride(2), mask_b, b, H, t, S)
	assert _lib.lib().gptq_attn_prompt_prepare(*where, P(old_k), *old_k.stride()[:2], P(old_v), *old_v.stride()[:2], past, P(k), P(v), P(flags), need, st) == 0
	whole_k, whole_v = torch.cat([old_k, new_k], 2), torch.cat([old_v, new_v], 2)
	assert torch.equal(k, whole_k) and torch.equal(v, whole_v) and bool((flags[:need] < 3).all()) and bool((flags[need:] == 7).all())
	outs = []
	for scratch, size in ((flags, need), (None, 0)):
		out = torch.full((b, t, H * D), float('nan'), dtype=torch.float16, device='cuda')
		rc = _lib.lib().gptq_attn_prompt(P(q), t * H * D, H * D, D, P(k), P(v), *where[:4], b, H, t, S, D ** -0.5, P(out), P(scratch), size, st)
		assert rc == 0
		outs.append(out.view(b, t, H, D).transpose(1, 2))
	s = q.transpose(1, 2).double() @ whole_k.double().transpose(2, 3) * D ** -0.5 + mask.double()
	ref = torch.softmax(s, -1).nan_to_num(0.0) @ whole_v.double()          # a query that sees nothing: zeros
	# weights and result are rounded to fp16 (2^-11 of at most max |v| each); the rest is fp32
	bound = 1.1 * 2.0 ** -10 * float(whole_v.abs().max())
	for out in outs:
		assert float((out.double() - ref).abs().max()) <= bound


def test_what_the_mask_holds():
	"""A row of infinities or NaN makes its own query NaN, nothing else; refused sizes and alignments come back as errors."""
	b, H, t, S, D = 1, 2, 70, 134, 128
	q, k, v = (torch.randn(b, n, H, D, device='cuda').half() for n in (t, S, S))
	k, v = k.transpose(1, 2).contiguous(), v.transpose(1, 2).contiguous()
	mask = torch.zeros((b, 1, t, S), device='cuda', dtype=torch.float16)
	mask[0, 0, 3], mask[0, 0, 68] = INF, float('nan')
	out = torch.empty((b, t, H * D), dtype=torch.float16, device='cuda')
	P, st = _lib.ptr, _lib.stream_ptr(q.device)
	f = _lib.lib().gptq_attn_prompt
	assert f(P(q), t * H * D, H * D, D, P(k), P(v), P(mask), t * S, S, 1, b, H, t, S, D ** -0.5, P(out), None, 0, st) == 0
	bad = out.isnan().all(-1)[0]
	assert bad[3] and bad[68] and int(out.isnan().any(-1).sum()) == 2
	assert f(None, 0, 0, 0, P(k), P(v), P(mask), t * S, S, 1, b, H, t, S, 1.0, P(out), None, 0, st) == -1
	assert f(P(q), t * H * D, H * D, D, P(k), P(v), P(mask), t * S, S, 2, b, H, t, S, 1.0, P(out), None, 0, st) == -1
	assert f(P(q), t * H * D, H * D + 4, D, P(k), P(v), P(mask), t * S, S, 1, b, H, t, S, 1.0, P(out), None, 0, st) == -4


@pytest.mark.parametrize('b,t,past,kind,served', [(1, 1, 40, 'shared', True), (2, 9, 0, 'shared', True), (1, 140, 61, 'lowest', True), (2, 33, 96, 'padded', True), (1, 201, 64, 'wide', True),
												  (1, 2040, 8, 'shared', True), (1, 2048, 8, 'shared', False), (1, 3000, 0, 'shared', False), (1, 3001, 0, 'shared', True), (2, 33, 96, 'float32', False),
												  (2, 33, 96, 'bool', False), (1, 33, 0, 'grad', False), (1, 33, 30, 'transposed past', False)])
def test_calls_of_the_block(monkeypatch, b, t, past, kind, served):
	H, K = 2, 256
	def layer(N, seed):
		d = synth.quant_tensors(K, N, 128, seed)
		q = G.QuantLinear(4, 128, K, N, False)
		q.qweight, q.qzeros, q.scales = d['qweight'], d['qzeros'], d['scales']
		return q
	attn = G.QuantLlamaAttention(G.LlamaConfig(hidden_size=K, num_attention_heads=H, max_position_embeddings=4096), layer(3 * K, 1), layer(K, 2), None).cuda()
	gen = torch.Generator(device='cuda').manual_seed(5)
	x = torch.randn((b, t, K), generator=gen, device='cuda').half()
	kv = tuple(torch.randn((b, H, past, 128), generator=gen, device='cuda').half() for _ in range(2)) if past else None
	mask = _mask(kind if kind in ('shared', 'lowest', 'padded', 'wide') else 'shared', b, t, past + t, gen)
	if kind == 'float32':
		mask = mask.float()
	elif kind == 'bool':
		mask = mask == 0
	elif kind == 'grad':
		mask = mask.clone().requires_grad_()
	elif kind == 'transposed past':
		kv = tuple(p.transpose(1, 2).contiguous().transpose(1, 2) for p in kv)
	host, seen = _lib.host(), []

	class Counts:
		qmatmul, gateup, qkv = host.qmatmul, host.gateup, host.qkv
		attend = staticmethod(lambda *a: seen.append(host.attend(*a)) or seen[-1])

	class Declines(Counts):
		attend = staticmethod(lambda *a: None)

	def call(module):
		with monkeypatch.context() as m:
			m.setattr(_lib, '_host', module)
			return attn(x, attention_mask=mask, past_key_value=kv, use_cache=True)
	call(Declines)          # (the workspace is there)
	new, old = call(Counts), call(Declines)
	assert len(seen) == 1 and (seen[0] is not None) == served
	assert new[1] is None and all(torch.equal(a, c) and a.stride() == c.stride() for a, c in zip(new[2], old[2]))
	if served:
		scale = float(old[0].float().abs().max())
		assert float((new[0].float() - old[0].float()).abs().max()) <= 2e-3 * scale          # two roundings of the softmax weights
	else:
		assert torch.equal(new[0].nan_to_num(7.0), old[0].nan_to_num(7.0))
	assert attn(x, attention_mask=mask, past_key_value=kv)[2] is None
	with pytest.raises(ValueError):
		attn(x, attention_mask=torch.zeros((b, 1, t, past + t + 1), device='cuda').half(), past_key_value=kv)


def _attend(q, k, v, mask, scale, full):
	"""Output of the kernels [b, H, t, D] for q [b, t, H, D], whole k and v [b, H, S, D], and the classes of the tiles."""
	(b, t, H, D), S = q.shape, k.shape[2]
	mask_b = 1 if mask.stride(0) == 0 else b
	l, P, st = _lib.lib(), _lib.ptr, _lib.stream_ptr(q.device)
	classes = l.gptq_attn_prompt_scratch_bytes(mask_b, t, S)
	need = l.gptq_attn_prompt_full_scratch_bytes(mask_b, b, H, t, S) if full else classes
	scratch = torch.full((need + 64,), 0x5A, dtype=torch.uint8, device='cuda')
	where = (P(mask), mask.stride(0), mask.stride(2), mask_b, b, H, t, S)
	assert l.gptq_attn_prompt_prepare(*where, None, 0, 0, None, 0, 0, 0, P(k), P(v), P(scratch), need, st) == 0
	out = torch.full((b, t, H * D), float('nan'), dtype=torch.float16, device='cuda')
	assert l.gptq_attn_prompt(P(q), t * H * D, H * D, D, P(k), P(v), *where[:4], b, H, t, S, scale, P(out), P(scratch), need, st) == 0
	assert bool((scratch[need:] == 0x5A).all())
	return out.view(b, t, H, D).transpose(1, 2), scratch[:classes]


@pytest.mark.parametrize('b,H,t,past', [(1, 2, 70, 0), (2, 3, 130, 70), (1, 2, 300, 129), (3, 1, 64, 577), (1, 1, 9, 8700)])
@pytest.mark.parametrize('kind', ['lowest', 'both', 'ten thousand', 'blind rows', 'bias', 'strong'])
def test_masks_of_finite_values(kind, b, H, t, past):
	"""Masks as `transformers` builds them (the lowest fp16 value, its sum with itself, -10000), biases that hide nothing, and scores so large that
	keys behind -9000 do count: with the full scratch, with the classes only, and against 64 bits."""
	gen = torch.Generator(device='cuda').manual_seed(t + past)
	S, D, low = t + past, 128, torch.finfo(torch.float16).min
	rnd = lambda *shape: torch.randn(shape, generator=gen, device='cuda').half()
	q, k, v = rnd(b, t, H, D), rnd(b, H, S, D), rnd(b, H, S, D)
	hidden = torch.triu(torch.ones((t, S), dtype=torch.bool, device='cuda'), diagonal=past + 1)
	mask = torch.zeros((b, 1, t, S), device='cuda', dtype=torch.float16).masked_fill(hidden, {'ten thousand': -1e4, 'strong': -9e3}.get(kind, low))
	if kind in ('both', 'blind rows'):
		for i in range(b):
			mask[i, :, :, :(i + 1) * 37 % S] += low          # -inf where both
	if kind == 'blind rows':
		mask[:, :, t // 2:t // 2 + 3] = low
	if kind == 'bias':
		mask = rnd(b, 1, t, S) * 3
	if kind == 'strong':          # whole heads' scores of up to +-20000, the visible ones at most zero
		q[..., :], k[..., :] = 0, 0
		q[..., 0] = 60.0
		k[:, :, :past + t // 2, 0] = -0.25 * torch.rand((b, H, past + t // 2), generator=gen, device='cuda').half()
		k[:, :, past + t // 2:, 0] = 4000.0 * torch.rand((b, H, t - t // 2), generator=gen, device='cuda').half()
	scale = 0.09
	s = q.transpose(1, 2).double() @ k.double().transpose(2, 3) * torch.tensor(scale, dtype=torch.float32).double().item() + mask.double()
	blind = (s.amax(-1) < -3e4)
	ref = torch.softmax(s, -1).nan_to_num(0.0) @ v.double()
	# fp16 weights and result, and logits that are rounded in fp32: by 2^-9 at 65504, by 2^-11 at 20000, which is twice as much of a weight
	bound = (1.1 * 2.0 ** -10 + torch.where(blind, 2.0 ** -8, 2.0 ** -10 if kind == 'strong' else 0.0)) * float(v.abs().max())
	outs = [_attend(q, k, v, mask, scale, full) for full in (True, False)]
	for out, _ in outs:
		assert bool(((out.double() - ref).abs() <= bound[..., None]).all())
	if kind in ('lowest', 'ten thousand', 'strong') and t > 128:
		assert int((outs[0][1] == 3).sum()) > 0 and int((outs[1][1] == 3).sum()) == 0          # tiles that only the full scratch knows to be low


def test_low_tiles_with_values_that_are_not_finite():
	"""A query or key of infinities or NaN keeps the low tiles in: what a query sees of it does not depend on the scratch."""
	b, H, t, D, low = 1, 2, 200, 128, torch.finfo(torch.float16).min
	gen = torch.Generator(device='cuda').manual_seed(1)
	q, k, v = (torch.randn(shape, generator=gen, device='cuda').half() for shape in ((b, t, H, D), (b, H, t, D), (b, H, t, D)))
	mask = torch.zeros((b, 1, t, t), device='cuda', dtype=torch.float16).masked_fill(torch.triu(torch.ones((t, t), dtype=torch.bool, device='cuda'), diagonal=1), low)
	q[0, 5, 0], k[0, 1, 190, 3] = float('nan'), INF
	full, part = (_attend(q, k, v, mask, D ** -0.5, f)[0] for f in (True, False))
	assert torch.equal(full.isnan(), part.isnan()) and bool(full[0, 0, 5].isnan().all()) and bool(full[0, 1, :190].isnan().any())
	assert torch.allclose(full.nan_to_num(0), part.nan_to_num(0), atol=2e-3)


def test_low_tiles_change_no_bit():
	"""Left out or computed: the same bits (with a key whose norm keeps the tiles in, and which no query sees)."""
	b, H, t, D, low = 1, 2, 333, 128, torch.finfo(torch.float16).min
	gen = torch.Generator(device='cuda').manual_seed(2)
	q, k, v = (torch.randn(shape, generator=gen, device='cuda').half() for shape in ((b, t, H, D), (b, H, t, D), (b, H, t, D)))
	mask = torch.zeros((b, 1, t, t), device='cuda', dtype=torch.float16).masked_fill(torch.triu(torch.ones((t, t), dtype=torch.bool, device='cuda'), diagonal=1), low)
	left_out = _attend(q, k, v, mask, D ** -0.5, True)[0]
	k[:, :, t - 1] = 0
	k[:, :, t - 1, 0] = 6e4
	q[:, :t - 1, :, 0] = 0          # its score is zero for all queries in front, but the bound does not know
	without = _attend(q, k.index_copy(2, torch.tensor([t - 1], device='cuda'), torch.zeros_like(k[:, :, :1])), v, mask, D ** -0.5, True)[0]
	computed = _attend(q, k, v, mask, D ** -0.5, True)[0]
	assert torch.equal(computed[:, :, :t - 1], without[:, :, :t - 1]) and bool(torch.isfinite(left_out).all())


def _layer(K, N, seed, gs=128, act=False):
	d = synth.quant_tensors(K, N, gs, seed)
	layer = G.QuantLinear(4, gs, K, N, False)
	layer.qweight, layer.qzeros, layer.scales = d['qweight'], d['qzeros'], d['scales']
	layer = layer.cuda()
	if act:
		layer.set_g_idx((torch.arange(K, dtype=torch.int32) // gs)[torch.randperm(K, generator=torch.Generator().manual_seed(seed))])
	return layer


def _block(H, K=256, gs=128, act=False):
	attn = G.QuantLlamaAttention(G.LlamaConfig(hidden_size=H * 128, num_attention_heads=H, max_position_embeddings=4096), _layer(H * 128, 3 * H * 128, 1, gs, act), _layer(H * 128, H * 128, 2), None)
	return attn.cuda()


def _both(monkeypatch, call):
	"""call() as it is and with the native attention declined; what the native attention returned."""
	host, seen = _lib.host(), []

	class Counts:
		qmatmul, gateup, qkv = host.qmatmul, host.gateup, host.qkv
		attend = staticmethod(lambda *a: seen.append(host.attend(*a)) or seen[-1])

	class Declines(Counts):
		attend = staticmethod(lambda *a: None)
	outs = []
	for module in (Declines, Counts, Declines):          # (the first for the workspace)
		with monkeypatch.context() as m:
			m.setattr(_lib, '_host', module)
			outs.append(call())
	return outs[1], outs[2], seen[0]


@pytest.mark.parametrize('H,b,t,past,library', [(2, 1, 1, 255, False), (2, 1, 1, 256, True), (2, 3, 1, 2000, True), (2, 79, 1, 252, False), (2, 80, 1, 252, True), (2, 80, 3, 220, False),
												(2, 81, 3, 190, True), (2, 81, 3, 189, False), (2, 81, 128, 65, True), (2, 81, 129, 64, False)])
@pytest.mark.parametrize('kind', ['shared', 'padded'])
def test_one_token_and_many_heads(monkeypatch, kind, H, b, t, past, library):
	"""Both sides of the lines beyond which the library's attention is the faster one: there the block gives its bits, as
	without the native call."""
	attn = _block(H)
	gen = torch.Generator(device='cuda').manual_seed(past)
	x = torch.randn((b, t, H * 128), generator=gen, device='cuda').half()
	kv = tuple(torch.randn((b, H, past, 128), generator=gen, device='cuda').half() for _ in range(2))
	mask = _mask(kind, b, t, t + past, gen)
	new, old, seen = _both(monkeypatch, lambda: attn(x, attention_mask=mask, past_key_value=kv, use_cache=True))
	assert seen is not None and all(torch.equal(a, c) and a.stride() == c.stride() for a, c in zip(new[2], old[2])) and new[0].shape == old[0].shape
	same = torch.equal(new[0].nan_to_num(7.0), old[0].nan_to_num(7.0))
	if library:
		assert same
	else:
		assert float((new[0].float() - old[0].float()).abs().max()) <= 2e-3 * float(old[0].float().abs().max())


@pytest.mark.parametrize('b,past,served', [(32, 902, True), (32, 904, False), (31, 904, True)])
def test_portions_behind_a_long_cache(monkeypatch, b, past, served):
	"""Mask rows off 16 bytes: 64 heads and more with eight times as many keys as queries are declined, as they were before there was a kernel."""
	H, t = 2, 129
	attn = _block(H)
	gen = torch.Generator(device='cuda').manual_seed(past)
	x = torch.randn((b, t, H * 128), generator=gen, device='cuda').half()
	kv = tuple(torch.randn((b, H, past, 128), generator=gen, device='cuda').half() for _ in range(2))
	mask = _mask('wide', b, t, t + past, gen)
	new, old, seen = _both(monkeypatch, lambda: attn(x, attention_mask=mask, past_key_value=kv, use_cache=True))
	assert (seen is not None) == served and all(torch.equal(a, c) for a, c in zip(new[2], old[2]))
	assert float((new[0].float() - old[0].float()).abs().max()) <= (2e-3 * float(old[0].float().abs().max()) if served else 0.0)


@pytest.mark.parametrize('t,past,act,gs,ids', [(1, 2000, False, 128, None), (9, 31, True, 128, None), (40, 31, True, 128, torch.int64), (33, 96, False, 128, torch.int32), (16, 0, True, 64, torch.int64)])
def test_native_attention_of_other_layers_and_positions(monkeypatch, t, past, act, gs, ids):
	"""Act-order projections (gathered in the workspace up to 16 rows, ahead of the call above), given positions that are not a range, one query
	behind 2000 keys: keys, values and outputs of the Python form; on a side stream and in a captured graph the same bits."""
	b, H = 2, 2
	attn = _block(H, gs=gs, act=act)
	gen = torch.Generator(device='cuda').manual_seed(t)
	x = torch.randn((b, t, H * 128), generator=gen, device='cuda').half()
	kv = tuple(torch.randn((b, H, past, 128), generator=gen, device='cuda').half() for _ in range(2)) if past else None
	mask = _mask('padded', b, t, t + past, gen)
	pos = None if ids is None else torch.randint(0, 3000, (b, t), generator=gen, device='cuda').to(ids)
	call = lambda: attn(x, attention_mask=mask, position_ids=pos, past_key_value=kv, use_cache=True)
	new, old, seen = _both(monkeypatch, call)
	assert seen is not None and all(torch.equal(a, c) for a, c in zip(new[2], old[2]))
	assert float((new[0].nan_to_num(7.0).float() - old[0].nan_to_num(7.0).float()).abs().max()) <= 2e-3 * float(old[0].nan_to_num(0.0).float().abs().max())
	side = torch.cuda.Stream()
	side.wait_stream(torch.cuda.current_stream())
	with torch.cuda.stream(side):
		call()          # (workspace of this stream)
		again = call()
		graph = torch.cuda.CUDAGraph()
		with torch.cuda.graph(graph, stream=side):
			captured = call()
		for y in (captured[0], *captured[2]):
			y.zero_()
		graph.replay()
	side.synchronize()
	for got in (again, captured):
		assert torch.equal(got[0].nan_to_num(7.0), new[0].nan_to_num(7.0)) and all(torch.equal(a, c) for a, c in zip(got[2], new[2]))


@pytest.mark.parametrize('case', ['groups of 32', 'no workspace', 'no tensor cores'])
def test_native_attention_declines(monkeypatch, case):
	"""... what it has no kernel or no workspace for; the block gives the results of the Python form."""
	from gptq_triton_b200 import quant_linear
	attn = _block(2, gs=32 if case == 'groups of 32' else 128)
	x = torch.randn((1, 40, 256), device='cuda').half()
	mask = _mask('padded', 1, 40, 40, None)
	if case == 'no workspace':
		monkeypatch.setattr(_lib, '_workspaces', {})
	if case == 'no tensor cores':
		monkeypatch.setattr(quant_linear, 'USE_TENSOR_CORE_KERNEL', False)
	seen, host = [], _lib.host()

	class Counts:
		qmatmul, gateup, qkv = host.qmatmul, host.gateup, host.qkv
		attend = staticmethod(lambda *a: seen.append(host.attend(*a)))
	monkeypatch.setattr(_lib, '_host', Counts)
	got = attn(x, attention_mask=mask, use_cache=True)
	ref = attn(x, attention_mask=mask, use_cache=True, output_attentions=True)
	assert seen == [None] and all(torch.equal(a, c) for a, c in zip(got[2], ref[2]))
	assert float((got[0].nan_to_num(0).float() - ref[0].nan_to_num(0).float()).abs().max()) <= 4e-3 * float(ref[0].nan_to_num(0).float().abs().max())
