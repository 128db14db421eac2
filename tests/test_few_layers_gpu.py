"""A model's layers launched from one native call (csrc/few_layers.cu) against the same kernels launched part by part: the same bits."""
import dataclasses
import gc
import weakref

import pytest
import torch

import bitnet_c_b200 as bn
from bitnet_c_b200.cache import PAGE
from bitnet_c_b200.csrc import ops
from bitnet_c_b200.engine import Model
from bitnet_c_b200.engine.batch import pack_step
from bitnet_c_b200.weights import random_parameters

pytestmark = pytest.mark.gpu


def _config(width, heads, kv, dim, ff, layers, tied):
    return {"architectures": ["LlamaForCausalLM"], "model_type": "llama", "hidden_size": width, "intermediate_size": ff, "num_hidden_layers": layers,
            "num_attention_heads": heads, "num_key_value_heads": kv, "head_dim": dim, "vocab_size": 512, "max_position_embeddings": 4096,
            "rope_theta": 10000.0, "rms_norm_eps": 1e-5, "tie_word_embeddings": tied, "hidden_act": "silu"}


def _logits(model, prompts, wants, steps):
    room = sum(-(-(len(p) + steps + 1) // 64) * 64 for p in prompts)
    cache = model.new_cache(max_tokens=room, max_seqs=len(prompts))
    slots = [cache.open() for _ in prompts]
    out = [model.step(cache, [bn.SeqStep(s, p, w) for s, p, w in zip(slots, prompts, wants)])]
    for i in range(steps):
        out.append(model.step(cache, [bn.SeqStep(s, [(7 * i + s) % 512], [0]) for s in slots]))
    return out


@pytest.mark.parametrize("size", [(64, 4, 2, 16, 176, 2, False), (2048, 32, 8, 64, 8192, 2, True), (512, 4, 4, 128, 1536, 3, False)])
@pytest.mark.parametrize("lengths", [[1], [12], [64], [3, 1, 20], [1] * 17, [5] * 12])
def test_same_bits(size, lengths):
    model = Model.from_random(_config(*size), seed=3, matrix_std=size[0] ** -0.5)
    assert model.few_layers is not None
    g = torch.Generator().manual_seed(len(lengths))
    prompts = [torch.randint(0, 512, (n,), generator=g).tolist() for n in lengths]
    for wants in ([[n - 1] for n in lengths], [list(range(n)) for n in lengths]):  # the last rows, or all of them (the final norm is then fused)
        native = _logits(model, prompts, wants, 3)
        few, model.few_layers = model.few_layers, None
        parts = _logits(model, prompts, wants, 3)
        model.few_layers = few
        assert all(torch.equal(a, b) for a, b in zip(native, parts))


def test_what_stays_with_the_parts():
    cfg = _config(64, 4, 2, 16, 176, 2, False)
    assert Model.from_random(cfg, dtype="float32").few_layers is None
    wide = Model.from_random(dict(cfg, head_dim=144), seed=1)  # no tcgen05 attention for prompts
    assert wide.few_layers is None
    model = Model.from_random(cfg, seed=1)
    cache = model.new_cache(max_tokens=128, max_seqs=1)
    slot = cache.open()
    ran = []
    run, model.few_layers.run = model.few_layers.run, lambda *a: ran.append(a) or run(*a)
    model.step(cache, [bn.SeqStep(slot, list(range(65)), [64])])  # more rows than the products of few rows take
    assert not ran
    model.step(cache, [bn.SeqStep(slot, [1], [0])])
    assert len(ran) == 1


@pytest.fixture
def native_calls(monkeypatch):
    """The native call's structures, as often as it is made."""
    made, run = [], ops.few_layers
    monkeypatch.setattr(ops, "few_layers", lambda step, launches: (made.append(step), run(step, launches))[1])
    return made


@pytest.mark.parametrize("other", [dict(head_dim=32), dict(num_key_value_heads=1), dict(num_key_value_heads=4), "float32"])
@pytest.mark.parametrize("tokens", [1, 20])
def test_a_cache_that_does_not_fit_is_refused(native_calls, other, tokens):
    """A cache of another head size, number of heads or type: the parts' error, and the native call is not made."""
    cfg = _config(64, 4, 2, 16, 176, 2, False)
    model = Model.from_random(cfg, seed=1)
    owner = Model.from_random(cfg, seed=1, dtype="float32") if other == "float32" else Model.from_random(dict(cfg, **other), seed=1)
    cache = owner.new_cache(max_tokens=128, max_seqs=1)
    slot = cache.open()
    with pytest.raises(ops.KernelError):
        model.step(cache, [bn.SeqStep(slot, list(range(tokens)), [0])])
    assert not native_calls
    assert cache.length(slot) == 0
    fitting = model.new_cache(max_tokens=128, max_seqs=1)
    model.step(fitting, [bn.SeqStep(fitting.open(), list(range(tokens)), [0])])
    assert len(native_calls) == 1


def test_a_weight_set_anew_is_looked_at(native_calls):
    """Weights of another type or layout than those bound are what the parts make of them, not bits read as bfloat16."""
    model = Model.from_random(_config(64, 4, 2, 16, 176, 2, False), seed=3, matrix_std=0.125)
    few = model.few_layers
    for part, name in ((model.blocks[1].ffn, "w_down"), (model.blocks[0].mixer, "w_qkv"), (model.blocks[1].mixer, "w_o")):
        old = getattr(part, name)
        setattr(part, name, old.float())
        native = _logits(model, [[5, 9, 11]], [[2]], 2)
        model.few_layers = None
        parts = _logits(model, [[5, 9, 11]], [[2]], 2)
        model.few_layers = few
        assert all(torch.equal(a, b) for a, b in zip(native, parts))
        setattr(part, name, old)
    assert not native_calls
    _logits(model, [[5, 9, 11]], [[2]], 2)
    assert len(native_calls) == 3


def test_a_dropped_model_is_gone():
    """Nothing of a model refers back to it: its weights are free when the last reference goes, not when the collector runs."""
    model = Model.from_random(_config(64, 4, 2, 16, 176, 2, False), seed=1)
    assert model.few_layers is not None
    gone = weakref.ref(model)
    gc.disable()
    try:
        del model
        assert gone() is None
    finally:
        gc.enable()


def _step_of(model, cache, slots, tokens, group):
    """One token for every sequence; ``group``: with the work list that a recorded step of these lengths would have."""
    lengths = [cache.length(s) for s in slots]
    seqs = [bn.SeqStep(s, [t], [0]) for s, t in zip(slots, tokens)]
    ctx = pack_step(seqs, lengths, model.device)
    if group:
        ctx.decode_item_group, items = ops.decode_items([n // PAGE + 1 for n in lengths], model.decode_blocks_per_sequence(),
                                                        group=None if group < 0 else group)
        ctx.decode_items = torch.tensor(items, dtype=torch.int32, device=model.device)
    for s in slots:
        cache.reserve(s, 1)
    cache.sync()
    logits = model.forward(cache, ctx)
    for s in slots:
        cache.advance(s, 1)
    return logits


@pytest.mark.parametrize("group", [-1, 1, 2, 3, 0])  # -1: the group that the batch itself asks for; 0: no list
def test_unequal_lengths_same_bits(native_calls, group):
    """Steps of a batch of unequal lengths, with a work list and without one."""
    model = Model.from_random(_config(256, 16, 16, 16, 704, 2, False), seed=5, matrix_std=0.06)
    lengths = [900, 70, 130, 10, 65, 64, 63, 200, 5, 77]
    g = torch.Generator().manual_seed(1)
    prompts = [torch.randint(0, 512, (n,), generator=g).tolist() for n in lengths]
    out = {}
    for few in (model.few_layers, None):
        model.few_layers = few
        cache = model.new_cache(max_tokens=sum(-(-(n + 4) // 64) * 64 for n in lengths), max_seqs=len(lengths))
        slots = [cache.open() for _ in lengths]
        for s, p in zip(slots, prompts):
            model.step(cache, [bn.SeqStep(s, p, ())])
        del native_calls[:]
        out[few] = [_step_of(model, cache, slots, [(7 * i + s) % 512 for s in range(len(slots))], group) for i in range(3)]
        assert len(native_calls) == (3 if few is not None else 0)
        assert all(bool(c.items) == bool(group) for c in native_calls)
    a, b = out.values()
    assert all(torch.equal(x, y) for x, y in zip(a, b))


@pytest.mark.parametrize("forced", [0, 12])  # 12: more blocks a sequence than one cluster has, merged through global memory
@pytest.mark.parametrize("window", [0, 100])
def test_split_sequences_and_windows_same_bits(native_calls, monkeypatch, forced, window):
    """Long sequences, whose pages several blocks share, and layers that see the last ``window`` keys only."""
    base = Model.from_random(_config(64, 4, 2, 16, 176, 2, False), seed=3, matrix_std=0.125)
    blocks = tuple(dataclasses.replace(b, mixer=dataclasses.replace(b.mixer, window=window)) for b in base.spec.blocks)
    model = Model(dataclasses.replace(base.spec, blocks=blocks), arch=base.arch, config=base.config)
    model.bind({path: t for path, _name, t in random_parameters(model.spec, base.arch.tensor_name, 3, model.dtype, 0.125, 0.1, model.device)})
    few = model.few_layers
    assert few is not None
    monkeypatch.setattr(ops, "_FORCE_SPLITS", forced)
    g = torch.Generator().manual_seed(1)
    pieces = [torch.randint(0, 512, (n,), generator=g).tolist() for n in (1500, 40, 64)]  # the last two: prompts of few tokens behind a long one
    out = {}
    for f in (few, None):
        model.few_layers = f
        cache = model.new_cache(max_tokens=1664, max_seqs=1)
        slot = cache.open()
        del native_calls[:]
        got = [model.step(cache, [bn.SeqStep(slot, p, [len(p) - 1])]) for p in pieces]
        got += [model.step(cache, [bn.SeqStep(slot, [i], [0])]) for i in range(3)]
        out[f] = got
        assert len(native_calls) == (5 if f is not None else 0)
        assert all(c.window == window for c in native_calls) and all(c.n_splits > 1 for c in native_calls[2:])
    a, b = out.values()
    assert all(torch.equal(x, y) for x, y in zip(a, b))
