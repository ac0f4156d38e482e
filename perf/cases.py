"""Timed cases of the framework: quantised layers as a module tree calls them, attention with the tuples of past keys that
HF-style generation passes around, and whole requests through the engines, from one row to the longest prompts.

Sizes are those of the LLaMA 7B and 65B architectures, of their tensor-parallel shards and of the models that bench.py builds.
Layers get the value distributions of the benchmark configurations (uniform 4-bit weights and zeros, scales U(0.002, 0.02),
activations N(0, 1)).  Models get random weights of a trained model's size; their output head follows the embedding, so that the
greedy choice is as clear as a trained model's mostly is.
"""
import math

import torch
import torch.nn as nn
import torch.nn.functional as F

import gptq_triton_b200 as G

DEV = 'cuda'


def listed():
	return [
		# o_proj of a 7B layer for one token: the smallest call a module tree makes
		{'name': 'linear_1', 'kind': 'linear', 'm': 1, 'k': 4096, 'n': 4096, 'g': 128, 'act': False, 'bias': False},
		# down_proj of an act-order checkpoint in a batch of a few sequences
		{'name': 'linear_6_act', 'kind': 'linear', 'm': 6, 'k': 11008, 'n': 4096, 'g': 128, 'act': True, 'bias': False},
		# fused QKV for a batch of 40 sequences, or a prompt of a line
		{'name': 'linear_40', 'kind': 'linear', 'm': 40, 'k': 4096, 'n': 12288, 'g': 128, 'act': False, 'bias': False},
		# the benchmark's stand-alone layer: 512 rows, with a bias
		{'name': 'linear_512', 'kind': 'linear', 'm': 512, 'k': 4096, 'n': 4096, 'g': 128, 'act': False, 'bias': True},
		# fused MLP, sixteen sequences, one scale per column
		{'name': 'mlp_16', 'kind': 'mlp', 'm': 16, 'hidden': 4096, 'inter': 11008, 'g': -1, 'act': False},
		# fused MLP of a 65B layer for a paragraph of odd length
		{'name': 'mlp_203', 'kind': 'mlp', 'm': 203, 'hidden': 8192, 'inter': 22016, 'g': 128, 'act': False},
		# fused MLP, a whole context of 2048 tokens
		{'name': 'mlp_2048', 'kind': 'mlp', 'm': 2048, 'hidden': 4096, 'inter': 11008, 'g': 128, 'act': False},
		# attention block as HF-style generation calls it: a prompt behind cached tokens, additive mask
		{'name': 'attention_701', 'kind': 'attention', 'b': 1, 't': 701, 'past': 64, 'hidden': 4096, 'g': 128},
		# one request to a 7B model: 2048 tokens of prompt, 48 generated (batch 1, the headline configuration)
		{'name': 'generate_7b', 'kind': 'llama', 'b': 1, 't': 2048, 'steps': 48, 'layers': 32, 'hidden': 4096, 'inter': 11008, 'g': 128},
		# sixteen requests at once, short prompts
		{'name': 'generate_batch', 'kind': 'llama', 'b': 16, 't': 97, 'steps': 32, 'layers': 8, 'hidden': 8192, 'inter': 22016, 'g': 128},
		# one request to a latent-attention model
		{'name': 'befalix', 'kind': 'befalix', 'b': 1, 't': 1500, 'steps': 32, 'layers': 8, 'hidden': 2048, 'inter': 5504},
		# a trace replayed through the differential-attention and state-space model: logits of every step
		{'name': 'lifinex', 'kind': 'lifinex', 'b': 1, 't': 1200, 'steps': 24, 'layers': 4, 'hidden': 2048, 'inter': 5504},
	]


def _log(rng, lo, hi):
	return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
	kind = rng.choice(['linear'] * 6 + ['mlp'] * 5 + ['attention'] * 2 + ['llama'] * 3 + ['befalix', 'lifinex'])
	g = rng.choice([128, 128, 128, 128, -1, -1, 64, 32])
	if kind == 'linear':
		return {'kind': kind, 'm': _log(rng, 1, 2048), 'k': 128 * _log(rng, 8, 172), 'n': 128 * _log(rng, 8, 192), 'g': g, 'act': rng.random() < 0.25, 'bias': rng.random() < 0.25}
	if kind == 'mlp':
		return {'kind': kind, 'm': _log(rng, 1, 2048), 'hidden': 128 * _log(rng, 8, 64), 'inter': 128 * _log(rng, 16, 172), 'g': g, 'act': rng.random() < 0.2}
	if kind == 'attention':
		b = rng.choice([1, 1, 1, 2, 5])
		t = _log(rng, 1, 2048 // b)
		return {'kind': kind, 'b': b, 't': t, 'past': rng.choice([0, 0, _log(rng, 1, 1500)]), 'hidden': rng.choice([2048, 4096, 5120, 8192]), 'g': rng.choice([128, 128, -1])}
	hidden = rng.choice([2048, 4096])
	inter, layers = {2048: (5504, rng.randint(2, 8)), 4096: (11008, rng.randint(1, 4))}[hidden]
	if kind == 'llama':
		b = rng.choice([1, 1, 1, 2, 4, 7, 12, 16, 32])
		if b == 1 and rng.random() < 0.5:
			hidden, inter, layers = 4096, 11008, rng.randint(6, 24)
		return {'kind': kind, 'b': b, 't': _log(rng, 8, 2048 // b), 'steps': rng.randint(8, 40), 'layers': layers, 'hidden': hidden, 'inter': inter,
				'g': rng.choice([128, 128, -1])}
	if kind == 'befalix':
		b = rng.choice([1, 1, 2, 5])
		return {'kind': kind, 'b': b, 't': _log(rng, 16, 2048 // b), 'steps': rng.randint(8, 32), 'layers': layers, 'hidden': hidden, 'inter': inter}
	return {'kind': kind, 'b': 1, 't': _log(rng, 16, 1600), 'steps': rng.randint(8, 24), 'layers': rng.choice([2, 4]), 'hidden': hidden, 'inter': inter}


# ---- inputs ----------------------------------------------------------------------------------------------------------------
def _gen(seed):
	return torch.Generator(device=DEV).manual_seed(seed)


def _words(shape, gen):
	return torch.randint(-2 ** 31, 2 ** 31, shape, generator=gen, device=DEV, dtype=torch.int64).to(torch.int32)


def _groups(k, g):
	return 1 if g == -1 else k // g


def _packed(k, n, g, gen):
	"""A layer's tensors with the benchmark configurations' distributions."""
	scales = torch.empty((_groups(k, g), n), device=DEV).uniform_(0.002, 0.02, generator=gen).half()
	return {'qweight': _words((k // 8, n), gen), 'qzeros': _words((_groups(k, g), n // 8), gen), 'scales': scales}


def _act_order(k, g, gen):
	gs = k if g == -1 else g
	return (torch.arange(k, device=DEV, dtype=torch.int32) // gs)[torch.randperm(k, generator=gen, device=DEV)]


def _layer(w, g, g_idx=None, bias=None):
	k, n = w['qweight'].shape[0] * 8, w['qweight'].shape[1]
	with torch.device('meta'):
		layer = G.QuantLinear(4, g, k, n, bias is not None)
	state = dict(w, **({} if bias is None else {'bias': bias}))
	for name, t in state.items():
		layer._buffers[name] = t
	if g_idx is not None:
		layer.set_g_idx(g_idx)
	return layer


def _linear_inputs(c, seed):
	gen = _gen(seed)
	w = _packed(c['k'], c['n'], c['g'], gen)
	g_idx = _act_order(c['k'], c['g'], gen) if c['act'] else None
	bias = torch.randn(c['n'], generator=gen, device=DEV).half() if c['bias'] else None
	return w, g_idx, bias, torch.randn((1, c['m'], c['k']), generator=gen, device=DEV).half()


def _mlp_inputs(c, seed):
	gen = _gen(seed)
	h, i, g = c['hidden'], c['inter'], c['g']
	ws = [_packed(h, i, g, gen), _packed(h, i, g, gen), _packed(i, h, g, gen)]
	idx = _act_order(h, g, gen) if c['act'] else None
	idx_down = _act_order(i, g, gen) if c['act'] else None
	# zero points are uniform, so a row of weights has a mean; activations behind a norm keep gate and up near unit variance
	x = torch.randn((1, c['m'], h), generator=gen, device=DEV) / (0.07 * math.sqrt(h))
	return ws, idx, idx_down, x.half()


def _model_layer(k, n, g, gen):
	"""Weights of a trained model's size: standard deviation 0.02 around zero (zero points 7 and 8: codes are uniform)."""
	scales = (0.02 / 4.6) * torch.empty((_groups(k, g), n), device=DEV).uniform_(0.8, 1.2, generator=gen)
	return {'qweight': _words((k // 8, n), gen), 'qzeros': (_words((_groups(k, g), n // 8), gen) & 0x11111111) + 0x66666666, 'scales': scales.half()}


def _attention_inputs(c, seed):
	gen = _gen(seed)
	h, b, t, p = c['hidden'], c['b'], c['t'], c['past']
	qkv, o = _model_layer(h, 3 * h, c['g'], gen), _model_layer(h, h, c['g'], gen)
	x = torch.randn((b, t, h), generator=gen, device=DEV).half()
	past = [torch.randn((b, h // 128, p, 128), generator=gen, device=DEV).half() for _ in range(2)] if p else None
	pos = torch.arange(p, p + t, device=DEV).unsqueeze(0).expand(b, t)
	mask = torch.triu(torch.full((t, p + t), float('-inf'), device=DEV, dtype=torch.float16), diagonal=p + 1)[None, None].expand(b, 1, t, p + t) if t > 1 else None
	return qkv, o, x, past, pos, mask


VOCAB = 32000


def _llama_inputs(c, seed):
	gen = _gen(seed)
	h, i, g = c['hidden'], c['inter'], c['g']
	layers = []
	for _ in range(c['layers']):
		norm = lambda: (1.0 + 0.1 * torch.randn(h, generator=gen, device=DEV)).half()
		layers.append({'qkv': _model_layer(h, 3 * h, g, gen), 'o': _model_layer(h, h, g, gen), 'gate': _model_layer(h, i, g, gen), 'up': _model_layer(h, i, g, gen),
					   'down': _model_layer(i, h, g, gen), 'ln1': norm(), 'ln2': norm()})
	# the stream keeps the token's own direction among what the layers add
	embed = 1.3 * math.sqrt(c['layers']) * torch.randn((VOCAB, h), generator=gen, device=DEV)
	head = 0.02 * F.normalize(embed, dim=-1).roll(1, 0) * math.sqrt(h)
	norm = (1.0 + 0.1 * torch.randn(h, generator=gen, device=DEV)).half()
	tokens = torch.randint(0, VOCAB, (c['b'], c['t']), generator=gen, device=DEV)
	return layers, embed.half(), head.half(), norm, tokens


def _befalix_config(c):
	H = c['hidden'] // 128
	layer = {'type': 'latent_attention', 'mlp': {'kind': 'dense', 'ff': c['inter']},
			 'mixer': {'heads': H, 'dim': 128, 'rot_dim': 64, 'vdim': 128, 'kv_rank': 512, 'scale': 192 ** -0.5, 'rot': {'base': 10000.0, 'dims': 64}}}
	return {'vocab': VOCAB, 'width': c['hidden'], 'norm': {'eps': 1e-6}, 'residual_mult': 1.0, 'logit_scale': 1.0, 'layers': [layer] * c['layers']}


def _lifinex_config(c):
	ff, hid = {'kind': 'dense', 'ff': c['inter']}, c['hidden']
	H = hid // 128
	att = {'type': 'attention', 'mlp': ff, 'mixer': {'heads': H, 'kv_heads': H // 4, 'dim': 64, 'vdim': 128, 'scale': 0.125, 'softcap': 25.0, 'diff': 0.4}}
	ssm = {'type': 'mamba2', 'mlp': ff, 'mixer': {'heads': hid // 32, 'vdim': 64, 'state': 128, 'groups': 8, 'conv': 4, 'norm_groups': 8}}
	layers, loop = {4: ([ssm, att, ssm], (1, 2, 2)), 2: ([att, ssm], (0, 1, 1))}[c['layers']]
	return {'vocab': VOCAB, 'width': hid, 'layers': layers, 'norm': {'eps': 1e-6}, 'max_positions': 2048, 'token_side': {'dim': 256}, 'loop': dict(zip(('start', 'stop', 'times'), loop))}


def _dense_tensors(shapes, seed):
	"""bf16 checkpoint tensors that keep activations near unit variance."""
	gen, out = _gen(seed), {}
	for name, shape in shapes.items():
		t, short = torch.randn(shape, generator=gen, device=DEV), name.split('.', 1)[-1]
		if short == 'mix.dt_bias':
			t = t - 3.0
		elif short == 'mix.A_log':
			t = 0.5 * t + 0.5
		elif name == 'final.norm.b' or short in ('norm1.b', 'norm2.b', 'mix.conv.b', 'mix.lq1', 'mix.lk1', 'mix.lq2', 'mix.lk2'):
			t = 0.1 * t
		elif short in ('ls1', 'ls2'):
			t = 0.3 + 0.03 * t
		elif name.startswith('side.') or short in ('mix.q.norm', 'mix.k.norm', 'mix.norm', 'mix.D', 'side.norm', 'mix.dkv.norm'):
			t = 1.0 + 0.1 * t if len(shape) == 1 else t
		elif len(shape) == 1:
			t = (1.0 if 'final.norm.b' in shapes else 0.0) + 0.1 * t
		elif name not in ('embed', 'pos', 'loop.step'):
			t = t * shape[1] ** -0.5
		out[name] = t.bfloat16()
	return out


def _dense_inputs(c, seed):
	d = (_befalix_config if c['kind'] == 'befalix' else _lifinex_config)(c)
	config = (G.BefalixConfig if c['kind'] == 'befalix' else G.LifinexConfig).from_dict(d)
	tokens = torch.randint(0, VOCAB, (c['b'], c['t'] + c['steps']), generator=_gen(seed + 1), device=DEV)
	return d, config, _dense_tensors(config.tensor_shapes(), seed), tokens


# ---- what a program keeps, and one pass ------------------------------------------------------------------------------------

def prepare(case, seed):
	c, kind = case, case['kind']
	if kind == 'linear':
		w, g_idx, bias, x = _linear_inputs(c, seed)
		return {'case': c, 'layer': _layer(w, c['g'], g_idx, bias), 'x': x}
	if kind == 'mlp':
		(gate, up, down), idx, idx_down, x = _mlp_inputs(c, seed)
		return {'case': c, 'mlp': G.QuantLlamaMLP(_layer(gate, c['g'], idx), _layer(down, c['g'], idx_down), _layer(up, c['g'], idx)), 'x': x}
	if kind == 'attention':
		qkv, o, x, past, pos, mask = _attention_inputs(c, seed)
		config = G.LlamaConfig(hidden_size=c['hidden'], num_attention_heads=c['hidden'] // 128)
		attn = G.QuantLlamaAttention(config, _layer(qkv, c['g']), _layer(o, c['g']), None)
		return {'case': c, 'attn': attn, 'x': x, 'past': None if past is None else tuple(past), 'pos': pos, 'mask': mask}
	if kind == 'llama':
		layers, embed, head, norm, tokens = _llama_inputs(c, seed)
		config = G.LlamaConfig(hidden_size=c['hidden'], intermediate_size=c['inter'], num_hidden_layers=c['layers'], num_attention_heads=c['hidden'] // 128, vocab_size=VOCAB)
		with torch.device('meta'):
			model = G.LlamaForCausalLM(config)
		half = lambda t: nn.Parameter(t, requires_grad=False)
		model.model.embed_tokens.weight, model.lm_head.weight, model.model.norm.weight = half(embed), half(head), half(norm)
		for layer, w in zip(model.model.layers, layers):
			layer.self_attn = G.QuantLlamaAttention(config, _layer(w['qkv'], c['g']), _layer(w['o'], c['g']), None)
			layer.mlp = G.QuantLlamaMLP(_layer(w['gate'], c['g']), _layer(w['down'], c['g']), _layer(w['up'], c['g']))
			layer.input_layernorm.weight, layer.post_attention_layernorm.weight = half(w['ln1']), half(w['ln2'])
		return {'case': c, 'engine': G.make_engine(model, c['b'], c['t'] + c['steps']), 'tokens': tokens}
	_, config, tensors, tokens = _dense_inputs(c, seed)
	model = (G.BefalixForCausalLM if kind == 'befalix' else G.LifinexForCausalLM)(config, tensors)
	return {'case': c, 'engine': G.make_engine(model, c['b'], c['t'] + c['steps']), 'tokens': tokens}


@torch.no_grad()
def run(state):
	c, kind = state['case'], state['case']['kind']
	if kind == 'linear':
		return state['layer'](state['x'])
	if kind == 'mlp':
		return state['mlp'](state['x'])
	if kind == 'attention':
		y, _, (k, v) = state['attn'](state['x'], attention_mask=state['mask'], position_ids=state['pos'], past_key_value=state['past'], use_cache=True)
		return [y, k, v]
	engine, tokens, t = state['engine'], state['tokens'], c['t']
	if kind == 'lifinex':
		engine.reset()
		return [engine.feed(tokens[:, :t])] + [engine.feed(tokens[:, i:i + 1]) for i in range(t, t + c['steps'])]
	new = engine.generate(tokens[:, :t], c['steps'])
	return [new, engine.logits]


# ---- what a pass cannot do without -----------------------------------------------------------------------------------------
def _packed_bytes(k, n, g):
	return k * n / 2 + _groups(k, g) * n * 2.5


def work(case):
	c, kind = case, case['kind']
	if kind == 'linear':
		return {'bytes': _packed_bytes(c['k'], c['n'], c['g']) + (4 * c['k'] if c['act'] else 0) + 2 * c['m'] * (c['k'] + c['n']) + (2 * c['n'] if c['bias'] else 0), 'flops': 2.0 * c['m'] * c['k'] * c['n']}
	if kind == 'mlp':
		h, i = c['hidden'], c['inter']
		return {'bytes': 2 * _packed_bytes(h, i, c['g']) + _packed_bytes(i, h, c['g']) + 4 * c['m'] * h, 'flops': 6.0 * c['m'] * h * i}
	h, b, t = c['hidden'], c['b'], c['t']
	if kind == 'attention':
		seen = b * (t * c['past'] + t * (t + 1) / 2)          # pairs of a query and a key that it sees
		return {'bytes': _packed_bytes(h, 4 * h, c['g']) + 4 * b * t * h + 4 * b * c['past'] * h + 4 * b * (c['past'] + t) * h, 'flops': 8.0 * b * t * h * h + 4.0 * seen * h}
	steps = c['steps'] if kind == 'lifinex' else c['steps'] - 1          # the first token comes from the prompt
	rows, seen = b * (t + steps), b * (t + steps) * (t + steps + 1) / 2
	ctx = sum(range(t + 1, t + steps + 1)) * b          # cached positions that the steps read
	if kind == 'llama':
		layer = _packed_bytes(h, 4 * h, c['g']) + 2 * _packed_bytes(h, c['inter'], c['g']) + _packed_bytes(c['inter'], h, c['g'])
		flops = c['layers'] * (2.0 * rows * (4 * h * h + 3 * h * c['inter']) + 4.0 * seen * h) + 2.0 * b * (steps + 1) * h * VOCAB
		return {'bytes': (steps + 1) * (c['layers'] * layer + 2 * h * VOCAB) + c['layers'] * 4 * h * (ctx + rows), 'flops': flops}
	if kind == 'befalix':
		H = h // 128
		mat = h * (H * 192 + 576 + H) + 512 * H * 256 + h * H * 128 + 3 * h * c['inter']
		flops = c['layers'] * (2.0 * rows * mat + 2.0 * seen * H * 320) + 2.0 * b * (steps + 1) * h * VOCAB
		return {'bytes': (steps + 1) * 2 * (c['layers'] * mat + h * VOCAB) + c['layers'] * 1152 * (ctx + rows), 'flops': flops}
	H, runs = h // 128, c['layers']
	inner, chan = 2 * h, 2 * h + 2048
	att = h * (H * 128 + H // 4 * 256) + h * h
	ssm = h * (inner + chan + h // 32) + inner * h
	mat = runs / 2 * (att + ssm) + runs * (3 * h * c['inter'] + 512 * h) + (1 + (2 if runs == 4 else 1)) * h * h
	flops = 2.0 * rows * mat + runs / 2 * (2.0 * seen * H * 2 * 192 + 4.0 * rows * inner * 128) + 2.0 * b * (steps + 1) * h * VOCAB
	return {'bytes': (steps + 1) * 2 * (mat + h * VOCAB) + runs / 2 * (H // 4 * 512 * (ctx + rows) + steps * 8 * inner * 128), 'flops': flops}


def tolerance(case):
	# about four times the error against 64 bits: rounding of the fp16 output, of fp16 weights above 16 rows, of fp16 or bf16 streams
	return {'linear': {'rel': 1.2e-3, 'max': 0.02}, 'mlp': {'rel': 3e-3, 'max': 0.05}, 'attention': {'rel': 3.2e-3, 'max': 0.05}, 'llama': {'rel': 1.3e-2, 'max': 0.2},
			'befalix': {'rel': 1.3e-2, 'max': 0.2}, 'lifinex': {'rel': 1.7e-2, 'max': 0.3}}[case['kind']]


# ---- the same in 64 bits ---------------------------------------------------------------------------------------------------
def _weights64(w, g, g_idx=None):
	"""(q - z - 1) * s as float64 [k, n]."""
	shift = torch.arange(0, 32, 4, device=DEV, dtype=torch.int32)
	q = ((w['qweight'][:, None, :] >> shift[None, :, None]) & 15).flatten(0, 1)
	z = ((w['qzeros'][:, :, None] >> shift) & 15).flatten(1)
	k = q.shape[0]
	group = (g_idx if g_idx is not None else torch.arange(k, device=DEV) // (k if g == -1 else g)).long()
	return (q - z[group] - 1).double() * w['scales'].double()[group]


def _silu(v):
	return v / (1 + torch.exp(-v))


def _rms(x, eps=1e-6):
	return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _rope(x, pos):
	"""x [..., t, 128], rotate-half."""
	ang = pos.double()[:, None] * 10000.0 ** (-torch.arange(0, 128, 2, device=DEV).double() / 128)[None]
	cos, sin = torch.cat([ang.cos()] * 2, -1), torch.cat([ang.sin()] * 2, -1)
	return x * cos + torch.cat([-x[..., 64:], x[..., :64]], -1) * sin


def _causal(q, k, v, scale, cap=None):
	"""q [t, d] at the last t of k's positions."""
	s = q @ k.T * scale
	if cap is not None:
		s = cap * torch.tanh(s / cap)
	t, n = s.shape
	s.masked_fill_(torch.arange(n, device=DEV)[None, :] > torch.arange(n - t, n, device=DEV)[:, None], -math.inf)
	return torch.softmax(s, -1) @ v


def _attend(q, k, v, scale):
	"""[b, h, t, d] against [b, h, n, d]."""
	out = torch.empty_like(q)
	for b in range(q.shape[0]):
		for h in range(q.shape[1]):
			out[b, h] = _causal(q[b, h], k[b, h], v[b, h], scale)
	return out


def _llama_logits(inputs, g, tokens, last):
	"""Logits of the last positions of tokens [b, t]."""
	layers, embed, head, norm, _ = inputs
	b, t = tokens.shape
	h = embed.shape[1]
	x = embed[tokens].double()
	for w in layers:
		y = _rms(x) * w['ln1'].double() @ _weights64(w['qkv'], g)
		q, k, v = y.view(b, t, 3, h // 128, 128).permute(2, 0, 3, 1, 4)
		pos = torch.arange(t, device=DEV)
		y = _attend(_rope(q, pos), _rope(k, pos), v, 128 ** -0.5).transpose(1, 2).reshape(b, t, h)
		x = x + y @ _weights64(w['o'], g)
		y = _rms(x) * w['ln2'].double()
		y = _silu(y @ _weights64(w['gate'], g)) * (y @ _weights64(w['up'], g))
		x = x + y @ _weights64(w['down'], g)
	return _rms(x[:, -last:]) * norm.double() @ head.double().T


def _layer_norm(x, w, b, eps=1e-6):
	d = x - x.mean(-1, keepdim=True)
	return d / torch.sqrt((d * d).mean(-1, keepdim=True) + eps) * w + b


def _interleaved(x, pos):
	n = x.shape[-1]
	ang = pos.double()[:, None] * 10000.0 ** (-torch.arange(0, n, 2, device=DEV).double() / n)[None]
	u, v = x[..., 0::2], x[..., 1::2]
	return torch.stack([u * ang.cos() - v * ang.sin(), v * ang.cos() + u * ang.sin()], -1).flatten(-2)


def _befalix_logits(d, W, tokens, last):
	H = d['width'] // 128
	W = {k: v.double() for k, v in W.items()}
	out = []
	for seq in tokens:
		x, pos = W['embed'][seq], torch.arange(len(seq), device=DEV)
		for i in range(len(d['layers'])):
			w = lambda name: W[f'l{i}.{name}']
			y = x @ w('mix.dkv').T
			latent, key_rot = _rms(y[:, :512]) * w('mix.dkv.norm'), _interleaved(y[:, 512:], pos)
			q, gate = (x @ w('mix.q').T).view(-1, H, 192), torch.sigmoid(x @ w('mix.g').T)
			heads = []
			for n in range(H):
				k = torch.cat([latent @ w('mix.uk')[128 * n:128 * n + 128].T, key_rot], -1)
				qn = torch.cat([q[:, n, :128], _interleaved(q[:, n, 128:], pos)], -1)
				heads.append(_causal(qn, k, latent @ w('mix.uv')[128 * n:128 * n + 128].T, 192 ** -0.5) * gate[:, n:n + 1])
			x = x + _layer_norm(torch.cat(heads, -1) @ w('mix.o').T, w('norm1'), w('norm1.b')) * w('ls1')
			y = (_silu(x @ w('mlp.gate').T) * (x @ w('mlp.up').T)) @ w('mlp.down').T
			x = x + _layer_norm(y, w('norm2'), w('norm2.b')) * w('ls2')
		out.append(_layer_norm(x[-last:], W['final.norm'], W['final.norm.b']) @ W['embed'].T)
	return torch.stack(out)


def _gelu(z):
	return 0.5 * z * (1 + torch.tanh(math.sqrt(2 / math.pi) * (z + 0.044715 * z ** 3)))


def _lifinex_mixer(h, w, kind, m):
	t = h.shape[0]
	if kind == 'attention':
		H, R, lam = m['heads'], m['kv_heads'], torch.exp((w('mix.lq1') * w('mix.lk1')).sum()) - torch.exp((w('mix.lq2') * w('mix.lk2')).sum()) + m['diff']
		q, k = _rms((h @ w('mix.q').T).view(t, H, 2, 64)) * w('mix.q.norm'), _rms((h @ w('mix.k').T).view(t, R, 2, 64)) * w('mix.k.norm')
		v, out = (h @ w('mix.v').T).view(t, R, 128), []
		for n in range(H):
			r = n // (H // R)
			a, b = (_causal(q[:, n, j], k[:, r, j], v[:, r], m['scale'], m['softcap']) for j in range(2))
			out.append(_rms(a - lam * b) * (1 - m['diff']))
		return torch.cat(out, -1) @ w('mix.o').T
	H, P, N, R = m['heads'], m['vdim'], m['state'], m['groups']
	z, u, dt = (h @ w('mix.in').T).split([H * P, H * P + 2 * R * N, H], -1)
	u = F.pad(u, (0, 0, 3, 0))
	u = _silu(sum(u[i:i + t] * w('mix.conv')[:, i] for i in range(4)) + w('mix.conv.b'))
	x, B, C = u[:, :H * P].view(t, H, P), u[:, H * P:H * P + R * N].view(t, R, N).repeat_interleave(H // R, 1), u[:, H * P + R * N:].view(t, R, N).repeat_interleave(H // R, 1)
	dt = F.softplus(dt + w('mix.dt_bias'))
	decay, S, y = torch.exp(-torch.exp(w('mix.A_log')) * dt), torch.zeros((H, N, P), dtype=torch.float64, device=DEV), []
	for i in range(t):
		S = decay[i][:, None, None] * S + (dt[i][:, None] * B[i])[:, :, None] * x[i][:, None, :]
		y.append(torch.bmm(C[i][:, None, :], S)[:, 0])
	y = (torch.stack(y) + w('mix.D')[:, None] * x).reshape(t, H * P) * _silu(z)
	return (_rms(y.view(t, m['norm_groups'], -1)).reshape(t, -1) * w('mix.norm')) @ w('mix.o').T


def _lifinex_logits(d, config, W, seq, last):
	W = {k: v.double() for k, v in W.items()}
	x = x0 = W['embed'][seq] + W['pos'][:len(seq)]
	for i, entry in config.runs():
		w, layer = (lambda name: W[f'l{i}.{name}']), d['layers'][i]
		if entry is not None:
			x = torch.cat([x, x0], -1) @ W['loop.in'].T + W['loop.step'][entry]
		x = x + _lifinex_mixer(_rms(x) * (1 + w('norm1')), w, layer['type'], layer['mixer'])
		h = _rms(x) * (1 + w('norm2'))
		x = x + (_gelu(h @ w('mlp.gate').T) * (h @ w('mlp.up').T)) @ w('mlp.down').T
		e = W['side.embed'][seq][:, 256 * i:256 * i + 256]
		x = x + _rms((_gelu(x @ w('side.gate').T) * e) @ w('side.proj').T) * w('side.norm')
	return _rms(x[-last:]) * (1 + W['final.norm']) @ W['head'].T


@torch.no_grad()
def exact(case, seed):
	c, kind = case, case['kind']
	if kind == 'linear':
		w, g_idx, bias, x = _linear_inputs(c, seed)
		y = x.double() @ _weights64(w, c['g'], g_idx)
		return y if bias is None else y + bias.double()
	if kind == 'mlp':
		(gate, up, down), idx, idx_down, x = _mlp_inputs(c, seed)
		x = x.double()
		return (_silu(x @ _weights64(gate, c['g'], idx)) * (x @ _weights64(up, c['g'], idx))) @ _weights64(down, c['g'], idx_down)
	if kind == 'attention':
		qkv, o, x, past, pos, _ = _attention_inputs(c, seed)
		b, t, h = x.shape
		q, k, v = (x.double() @ _weights64(qkv, c['g'])).view(b, t, 3, h // 128, 128).permute(2, 0, 3, 1, 4)
		q, k = _rope(q, pos[0]), _rope(k, pos[0])
		if past is not None:
			k, v = torch.cat([past[0].double(), k], 2), torch.cat([past[1].double(), v], 2)
		y = _attend(q, k, v, 128 ** -0.5).transpose(1, 2).reshape(b, t, h) @ _weights64(o, c['g'])
		return [y, k, v]
	steps, b = c['steps'], c['b']
	if kind == 'llama':
		inputs = _llama_inputs(c, seed)
		tokens, logits = inputs[4], lambda seq: _llama_logits(inputs, c['g'], seq, steps)
		guess = (tokens[:, -1:] + 1 + torch.arange(steps, device=DEV)) % VOCAB
	else:
		d, config, W, tokens = _dense_inputs(c, seed)
		if kind == 'lifinex':
			y = _lifinex_logits(d, config, W, tokens[0], steps + 1)
			return [y[None, None, i] for i in range(steps + 1)]
		tokens, logits = tokens[:, :c['t']], lambda seq: _befalix_logits(d, W, seq, steps)
		guess = tokens[:, -1:].expand(b, steps)
	for _ in range(steps):          # the greedy continuation of a guessed one, until it is its own
		y = logits(torch.cat([tokens, guess[:, :-1]], 1))
		new = y.argmax(-1)
		if torch.equal(new, guess):
			break
		guess = new
	return [guess, y[:, -1:]]
