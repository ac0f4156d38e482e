"""CPU tests of the host-side layer: packer/quantiser against the oracle, module surgery,
state-dict compatibility with the reference checkpoint layout, checkpoint round trip."""
import json

import numpy as np
import pytest
import torch

import gptq_triton_b200 as G
from gptq_triton_b200 import loader, quantize
from gptq_triton_b200.llama import LlamaConfig
from oracle import gptq_oracle as O

SMALL = LlamaConfig(hidden_size=256, intermediate_size=512, num_hidden_layers=2, num_attention_heads=2, vocab_size=128, max_position_embeddings=64)


@pytest.mark.parametrize('gs', [128, -1, 32])
def test_rtn_quantiser_and_packer_match_oracle(gs):
	torch.manual_seed(0)
	W = torch.randn(64, 256) * 0.02
	qw, qz, sc = quantize.quantize_linear_weight(W, gs)
	fq, s, z = O.rtn_quantize(W, gs)
	a, b, c = O.pack_linear(fq, s, z, gs)
	assert torch.equal(qw, a) and torch.equal(qz, b) and torch.equal(sc, c)


def test_packer_matches_reference_fixture(golden_dir):
	d = dict(np.load(golden_dir / 'pack_a.npz'))
	gs = int(d['groupsize'])
	fq = torch.from_numpy(d['fakequant'])
	# quantising the fake-quantised weights again reproduces the reference's integers
	qw, qz, sc = quantize.quantize_linear_weight(fq, gs)
	assert np.array_equal(O.unpack_qweight(qw), O.unpack_qweight(d['qweight']))


def test_quantlinear_contract():
	with pytest.raises(NotImplementedError):
		G.QuantLinear(3, 128, 256, 256, False)
	with pytest.raises(AssertionError):
		G.QuantLinear(4, 128, 256, 252, False)
	m = G.QuantLinear(4, -1, 256, 64, True)
	assert m.groupsize == 256 and m.qweight.shape == (32, 64) and m.qzeros.shape == (1, 8) and m.scales.shape == (1, 64)
	assert m.qweight.dtype == torch.int32 and m.scales.dtype == torch.float16 and m.bias.shape == (64,)
	assert set(m.state_dict()) == {'qweight', 'qzeros', 'scales', 'bias'}
	m2 = G.QuantLinear(4, 128, 256, 64, False)
	assert set(m2.state_dict()) == {'qweight', 'qzeros', 'scales'}
	sd = dict(m2.state_dict())
	sd['g_idx'] = torch.arange(256, dtype=torch.int32) // 128
	m2.load_state_dict(sd)
	assert 'g_idx' in m2.state_dict()


def test_module_surgery_and_checkpoint_round_trip(tmp_path):
	model = loader._empty_model(SMALL, 4, 128)
	names = [n for n, m in model.named_modules() if isinstance(m, G.QuantLinear)]
	assert len(names) == 7 * SMALL.num_hidden_layers and 'lm_head' not in names
	assert isinstance(model.lm_head, torch.nn.Linear)
	gen = torch.Generator().manual_seed(1)
	for n, m in model.named_modules():
		if isinstance(m, G.QuantLinear):
			qw, qz, sc = quantize.quantize_linear_weight(torch.randn((m.outfeatures, m.infeatures), generator=gen) * 0.02, 128)
			m.qweight.copy_(qw); m.qzeros.copy_(qz); m.scales.copy_(sc)
	for prm in model.parameters():
		prm.data.normal_(0, 0.02, generator=gen)
	keys = set(model.state_dict())
	assert 'model.layers.0.self_attn.q_proj.qweight' in keys and 'model.layers.1.mlp.down_proj.scales' in keys
	assert 'model.embed_tokens.weight' in keys and 'lm_head.weight' in keys and 'model.norm.weight' in keys
	loader.save_quant(model, tmp_path, 128)
	assert json.load(open(tmp_path / 'quant_config.json')) == {'wbits': 4, 'groupsize': 128}
	loaded = G.load_quant(str(tmp_path), warmup_autotune=False, device=None)
	layer = loaded.model.layers[0]
	assert isinstance(layer.self_attn, G.QuantLlamaAttention) and isinstance(layer.mlp, G.QuantLlamaMLP)
	qkv = layer.self_attn.qkv_proj
	assert qkv.outfeatures == 3 * SMALL.hidden_size and qkv.qweight.shape == (SMALL.hidden_size // 8, 3 * SMALL.hidden_size)
	src = model.model.layers[0].self_attn
	assert torch.equal(qkv.qweight, torch.cat([src.q_proj.qweight, src.k_proj.qweight, src.v_proj.qweight], dim=1))
	assert torch.equal(qkv.qzeros, torch.cat([src.q_proj.qzeros, src.k_proj.qzeros, src.v_proj.qzeros], dim=1))
	assert torch.equal(layer.mlp.gate_proj_qweight, model.model.layers[0].mlp.gate_proj.qweight)
	assert torch.equal(loaded.lm_head.weight, model.lm_head.weight)
	assert loaded.seqlen == 2048
	unfused = G.load_quant(str(tmp_path), warmup_autotune=False, device=None, fuse_mlp=False)
	assert not isinstance(unfused.model.layers[0].mlp, G.QuantLlamaMLP)
	with pytest.raises(FileNotFoundError):
		(tmp_path / 'model.safetensors').unlink()
		G.load_quant(str(tmp_path), warmup_autotune=False, device=None)


@pytest.mark.parametrize('safetensors', [True, False])
def test_checkpoint_with_rotary_inv_freq_keys_loads(tmp_path, safetensors):
	"""Checkpoints written under the transformers versions the reference names carry
	`self_attn.rotary_emb.inv_freq` per layer; they must load, in both file formats, and any OTHER
	unexpected key of a safetensors file must still be refused."""
	model = loader._empty_model(SMALL, 4, 128)
	gen = torch.Generator().manual_seed(2)
	for n, m in model.named_modules():
		if isinstance(m, G.QuantLinear):
			qw, qz, sc = quantize.quantize_linear_weight(torch.randn((m.outfeatures, m.infeatures), generator=gen) * 0.02, 128)
			m.qweight.copy_(qw); m.qzeros.copy_(qz); m.scales.copy_(sc)
	for prm in model.parameters():
		prm.data.normal_(0, 0.02, generator=gen)
	loader.save_quant(model, tmp_path, 128, safetensors=safetensors)
	head_dim = SMALL.hidden_size // SMALL.num_attention_heads
	extra = {f'model.layers.{i}.self_attn.rotary_emb.inv_freq': 1.0 / (10000.0 ** (torch.arange(0, head_dim, 2).float() / head_dim))
			 for i in range(SMALL.num_hidden_layers)}
	if safetensors:
		from safetensors.torch import load_file, save_file
		sd = load_file(str(tmp_path / 'model.safetensors'))
		save_file({**sd, **extra}, str(tmp_path / 'model.safetensors'))
	else:
		sd = torch.load(tmp_path / 'model.pt')
		torch.save({**sd, **extra}, tmp_path / 'model.pt')
	loaded = G.load_quant(str(tmp_path), warmup_autotune=False, device=None)
	assert torch.equal(loaded.model.layers[1].self_attn.o_proj.qweight, model.model.layers[1].self_attn.o_proj.qweight)
	if safetensors:
		save_file({**sd, **extra, 'model.layers.0.bogus.weight': torch.zeros(1)}, str(tmp_path / 'model.safetensors'))
		with pytest.raises(RuntimeError):
			G.load_quant(str(tmp_path), warmup_autotune=False, device=None)


def test_decode_engine_refuses_to_step_past_its_cache():
	"""Host-side guard: step() raises before a position beyond the static cache could reach a kernel
	(checked without a GPU by calling the guard on a bare object)."""
	from gptq_triton_b200.llama import DecodeEngine
	e = DecodeEngine.__new__(DecodeEngine)
	e.next_pos, e.max_seq = 8, 8
	with pytest.raises(RuntimeError, match='is full'):
		e.step()


def test_make_fused_mlp_returns_module():
	model = loader._empty_model(SMALL, 4, 128)
	mlp = model.model.layers[0].mlp
	fused = G.make_fused_mlp(mlp)
	assert isinstance(fused, G.QuantLlamaMLP) and fused.infeatures == 256 and fused.outfeatures == 256
	assert G.make_fused_mlp(torch.nn.Linear(4, 4)).__class__ is torch.nn.Linear


def test_bench_reference_arm_prints_one_json_line():
	"""`bench.py --impl reference` (the CPU port of the reference path) runs without a GPU and prints the contract's
	JSON line with its own cpu_baseline and e2e records."""
	import subprocess, sys
	from pathlib import Path
	root = Path(__file__).resolve().parent.parent
	r = subprocess.run([sys.executable, str(root / 'bench.py'), '--impl', 'reference', '--steps', '1', '--warmup', '0'], capture_output=True, text=True, timeout=600)
	assert r.returncode == 0, r.stderr[-2000:]
	line = json.loads(r.stdout.strip().splitlines()[-1])
	assert line['impl'] == 'reference' and line['unit'] == 'tokens/s' and line['value'] > 0
	assert line['cpu_baseline']['kind'] == 'port' and line['cpu_baseline']['cores'] >= 1 and line['cpu_baseline']['factor'] == 32
	assert line['e2e'] == {'value': line['value'], 'unit': 'tokens/s', 'h2d_bytes_per_step': 0, 'd2h_bytes_per_step': 0}


@pytest.mark.parametrize('b,t,S', [(1, 200, 265), (3, 200, 265), (1, 256, 264), (2, 3, 5), (1, 128, 401), (2, 33, 2001), (1, 129, 401)])
def test_aligned_mask_has_the_same_values(b, t, S):
	"""Rows of a large additive mask start on 16 bytes afterwards; values, shape and the sharing over the batch stay; small masks, masks of
	up to 128 queries (for which the copy does not pay) and masks of truth values are passed on."""
	from gptq_triton_b200.fused_attention import aligned_mask
	mask = torch.randn(1, 1, t, S).half().expand(b, 1, t, S)
	out = aligned_mask(mask)
	assert out.shape == mask.shape and torch.equal(out, mask)
	if t <= 128 or t * S < 1 << 15:
		assert out is mask
	else:
		assert out.stride(-1) == 1 and out.stride(-2) % 8 == 0 and (b == 1 or out.stride(0) == 0)
	own = torch.randn(b, 1, t, S).half().transpose(-1, -2).contiguous().transpose(-1, -2)          # columns first, one per sequence
	assert torch.equal(aligned_mask(own), own)
	assert aligned_mask(None) is None and aligned_mask(mask > 0) .dtype == torch.bool


def test_projections_that_store_many_cache_rows_do_not_start_their_successor_early():
	"""Attention reads old cache rows ahead of its wait for the kernel in front.  By the source: the prompt projection waits before
	its first copy and never triggers, the decode projections trigger for one token per sequence only, dec_kernel not before its own wait."""
	from gptq_triton_b200.build import CSRC
	prompt = (CSRC / 'qmm_tc_kernel.inl').read_text()
	assert 'pdl_trigger();' not in prompt and prompt.count('pdl_wait();') == 1
	assert prompt.index('pdl_wait();') < min(prompt.index(call) for call in ('tma_load_2d(', 'tc_bulk_load('))
	for name, count in (('qmm_dec.cu', 1), ('qmm_skinny.cuh', 2)):
		text = (CSRC / name).read_text()
		lines = [line for line in text.splitlines() if 'pdl_trigger();' in line]
		assert len(lines) == count and sum('tokens_per_batch == 1' in line for line in lines) == 1          # the other one: gather_x_kernel
		if name == 'qmm_dec.cu':
			assert text.index('pdl_wait();') < text.index('pdl_trigger();')


@pytest.mark.parametrize('what', ['missing', 'other torch', 'old'])
def test_without_the_extension_module_calls_go_through_ctypes(monkeypatch, what):
	"""The module is another way into the library, not a part of it: missing, or built against another torch, it is left out with one warning."""
	import sys
	import types
	from gptq_triton_b200 import _lib, build
	build.build()
	monkeypatch.setattr(_lib, '_host', None)
	monkeypatch.setattr(_lib, '_lib', None)
	module = None if what == 'missing' else types.SimpleNamespace(torch_version='1.0', bind=lambda *a: pytest.fail('bound')) if what == 'other torch' else types.SimpleNamespace()
	monkeypatch.setitem(sys.modules, 'gptq_triton_b200._host', module)
	if module is not None:
		monkeypatch.setattr(G, '_host', module, raising=False)
	else:
		monkeypatch.delattr(G, '_host', raising=False)
	assert _lib.lib().gptq_version() >= 100
	with pytest.warns(RuntimeWarning, match='_host.so is not used'):
		host = _lib.host()
	assert all(getattr(host, f)() is None for f in ('qmatmul', 'gateup', 'qkv', 'attend')) and _lib.host() is host
	with pytest.raises(_lib.GptqB200Error):          # (the error that such a call had before)
		G.triton_matmul4(128, torch.zeros(1, 256, dtype=torch.float16), torch.zeros(32, 256, dtype=torch.int32), torch.zeros(2, 256, dtype=torch.float16), torch.zeros(2, 32, dtype=torch.int32))


def test_cpu_tensors_are_refused_without_the_library(monkeypatch, tmp_path):
	"""... with the message that says why, which needs no library."""
	from gptq_triton_b200 import _lib
	monkeypatch.setattr(_lib, '_host', None)
	monkeypatch.setattr(_lib, '_lib', None)
	monkeypatch.setattr(_lib, 'LIB_PATH', tmp_path / 'none.so')
	with pytest.raises(_lib.GptqB200Error, match='CUDA tensors only'):
		G.triton_matmul4(128, torch.zeros(1, 256, dtype=torch.float16), torch.zeros(32, 256, dtype=torch.int32), torch.zeros(2, 256, dtype=torch.float16), torch.zeros(2, 32, dtype=torch.int32))
	with pytest.raises(ImportError):
		_lib.lib()


def test_build_goes_on_without_the_extension_module(monkeypatch):
	"""g++ or the headers of Python missing: the libraries are built, the module is left out with a warning, unless it was asked for by name."""
	from gptq_triton_b200 import build
	built = []

	def one(target, verbose):
		if target == 'host':
			raise RuntimeError('g++ failed building _host.so')
		built.append(target)
	monkeypatch.setattr(build, '_build_one', one)
	with pytest.warns(RuntimeWarning, match='_host.so was not built'):
		assert build.build(force=True) == build.LIB
	assert built == ['gptq', 'dense']
	with pytest.raises(RuntimeError):
		build.build(force=True, only=['host'])


def test_dense_ring_kernel_gives_up_as_a_whole_warp():
	"""A wait that runs out has to be known to every lane: the MMAs behind it are the warp's, and lane 0 reports.  By the source."""
	from gptq_triton_b200.build import CSRC
	text = (CSRC / 'dense' / 'dense_skinny.cu').read_text()
	waits = [line for line in text.splitlines() if 'mbar_wait_bounded(' in line or 'mbar_try_wait(' in line]
	assert waits and all('__all_sync(0xffffffffu, mbar_' in line for line in waits)
	kernel = text[text.index('dense_ring_kernel('):]
	kernel = kernel[:kernel.index('\n}\n')]
	given_up = kernel[kernel.index('!rg_wait('):]
	assert given_up.index('left = 0;') < given_up.index('load();') < given_up.index('if (!ok)') < given_up.index('atomicExch(p.status')


def test_gain_and_shift_are_read_with_y_only():
	"""Rows without a y have no gain or shift; whatever the two pointers hold then is not to be read ahead of the wait either.  By the source."""
	from gptq_triton_b200.build import CSRC
	text = (CSRC / 'dense' / 'dense.cuh').read_text()
	weights = text[text.index('struct RowWeights'):]
	weights = weights[:weights.index('\n};')]
	reads = [line for line in weights.splitlines() if 'p.gain' in line or 'p.shift' in line]
	assert len(reads) == 2 and all('p.y ? p.' in line for line in reads)


def test_clear_kernel_status_clears_the_whole_control_area(monkeypatch):
	"""Arrival counters and hand-over flags of a launch that gave up go with its status, in retired workspaces too (a captured graph may
	still use one); what lies behind the first 16 KB stays."""
	from gptq_triton_b200 import _lib
	buffers = [torch.full((20000,), 1, dtype=torch.uint8) for _ in range(3)]
	monkeypatch.setattr(_lib, '_workspaces', {(0, 0): buffers[0]})
	monkeypatch.setattr(_lib, '_retired', [buffers[1]])
	monkeypatch.setattr(_lib, '_status_buffers', [])
	_lib.register_status_buffer(buffers[2])
	assert _lib.kernel_status() != 0
	_lib.clear_kernel_status()
	assert _lib.kernel_status() == 0
	for buf in buffers:
		assert not buf[:16384].any() and buf[16384:].all()
