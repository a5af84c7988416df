"""The layer loop of plain decoders in native code (csrc/plain_layers.cu) against the parts' own forward, to the bit: both make
the same launches."""
import pytest
import torch

import util

pytestmark = pytest.mark.gpu

BASE = dict(architectures=["LlamaForCausalLM"], model_type="llama", hidden_size=256, num_hidden_layers=3, num_attention_heads=4,
            num_key_value_heads=2, head_dim=64, intermediate_size=448, vocab_size=515, rope_theta=10000.0, rms_norm_eps=1e-5,
            tie_word_embeddings=False, max_position_embeddings=4096, hidden_act="silu", bos_token_id=1, eos_token_id=2)
MODELS = {"grouped": BASE, "wide heads": dict(BASE, head_dim=128, num_key_value_heads=4),
          "scaled": dict(BASE, tie_word_embeddings=True, rope_scaling=dict(rope_type="llama3", factor=8.0, low_freq_factor=1.0,
                                                                           high_freq_factor=4.0, original_max_position_embeddings=512))}


def build(cfg, std=0.1):
    """A model of random weights on the device, in bfloat16."""
    from lmsf_b200.config.registry import resolve_architecture
    from lmsf_b200 import models  # noqa: F401
    from lmsf_b200.parts.decoder import DecoderModel
    from lmsf_b200.weights.loader import collect_requirements
    cfg, dev = dict(cfg), torch.device("cuda:0")
    arch = resolve_architecture(cfg)
    g = torch.Generator(device=dev).manual_seed(5)
    model = DecoderModel(arch.build_spec(arch.parse_config(cfg)))
    per_part, parts = {}, {}
    for part, logical, wspec, names in collect_requirements(model):
        sizes = [wspec.concrete(i) for i in range(len(wspec.shapes))]
        shape = (sum(s[0] for s in sizes), *sizes[0][1:])
        t = torch.randn(shape, generator=g, device=dev) * std + (1.0 if "norm" in names[0] else 0.0)
        per_part.setdefault(id(part), {})[logical] = t.to(torch.bfloat16)
        parts[id(part)] = part
    for pid, tensors in per_part.items():
        parts[pid].set_weights(tensors)
    model.prepare(torch.bfloat16, dev)
    return model


def watch(monkeypatch):
    """Notes for every step that is not a replay whether the native loop took it."""
    from lmsf_b200.parts import plain_layers
    taken, inner = [], plain_layers.run

    def noted(*a):
        r = inner(*a)
        taken.append(r is not None)
        return r

    monkeypatch.setattr(plain_layers, "run", noted)
    return taken


def life(model, cfg, native, monkeypatch, block_size=16):
    """The logits of seven steps: prompts, portions, few rows, many prompts, and a decode batch eager, captured and replayed."""
    from lmsf_b200.engine.model_runner import ModelRunner, StepEntry
    from lmsf_b200.parts import plain_layers
    ids = [util.random_ids(n, cfg["vocab_size"], 7 + n) for n in (300, 41, 17, 1)]
    monkeypatch.setattr(plain_layers, "USE_NATIVE_LAYERS", native)
    runner = ModelRunner(model, torch.bfloat16, torch.device("cuda:0"), block_size, num_blocks=[4800 // block_size], max_num_seqs=64, max_model_len=1024)
    mgr = runner.make_cache_manager()
    out = []
    step = lambda entries: out.append(runner.step(entries, mgr).clone())
    for i in range(24):
        mgr.add(i)
    step([StepEntry(0, ids[0][:160], [159, 3]), StepEntry(1, ids[1], [40])])                   # prompts
    step([StepEntry(0, ids[0][160:], [139]), StepEntry(1, [5], [0]), StepEntry(2, ids[2], [16])])   # a later portion, a single token
    step([StepEntry(2, ids[1][:9], [8])])                                                      # few rows
    step([StepEntry(i, ids[0][:150], [0]) for i in range(3, 24)])
    for k in range(3):                                                                         # a decode batch: eager, captured, replayed
        step([StepEntry(i, [11 + i + k], [0]) for i in range(3, 24)])
    return out


def same_bits(model, cfg, monkeypatch, block_size=16):
    taken = watch(monkeypatch)
    a = life(model, cfg, True, monkeypatch, block_size)
    assert taken == [True, True, False, True, True, True]          # the last: the capture
    taken.clear()
    b = life(model, cfg, False, monkeypatch, block_size)
    assert not any(taken)
    for x, y in zip(a, b):
        assert torch.isfinite(x).all() and torch.equal(x, y)
    taken.clear()
    return taken


@pytest.mark.parametrize("name", list(MODELS))
def test_same_bits_as_the_parts(name, monkeypatch):
    """Prompts whole and in portions, prompts beside requests that decode, a decode batch above 16, and 16 rows and fewer, which stay with
    the parts; a model whose second layer is not plain (a window) stays with them whole."""
    cfg = MODELS[name]
    model = build(cfg)
    taken = same_bits(model, cfg, monkeypatch)
    # one layer that is not plain
    model.blocks[1]._mixer.window = 50
    life(model, cfg, True, monkeypatch)
    assert not any(taken)
    model.blocks[1]._mixer.window = None


@pytest.mark.parametrize("act", ["silu", "gelu_pytorch_tanh"])
def test_same_bits_with_the_gated_kernel(act, monkeypatch):
    """As many tiles of features as the device has pairs of SMs, the last one not whole: the steps of 201 and 3,150 rows take gate, up and
    activation in one kernel, in the loop and in the parts, the others do not."""
    from lmsf_b200 import kernels
    from lmsf_b200.parts import linear
    cfg = dict(BASE, hidden_act=act, intermediate_size=kernels.sm_count("cuda:0") // 2 * 128 - 72)
    chosen, inner = [], linear.gated_in_one
    monkeypatch.setattr(linear, "gated_in_one", lambda rows, *a: (lambda r: (chosen.append((rows, r)), r)[1])(inner(rows, *a)))
    same_bits(build(cfg), cfg, monkeypatch)
    assert {rows for rows, r in chosen if r} == {201, 3150} and {rows for rows, r in chosen if not r} == {158, 24}      # 21 decoding requests are padded to 24
    # asked once a step by the loop and once a layer by the parts
    assert [chosen.count((rows, True)) for rows in (201, 3150)] == [1 + cfg["num_hidden_layers"]] * 2


@pytest.mark.parametrize("what", ["norms in float32", "interleaved", "half rotated", "heads in threes", "pages of 8", "pages of 64", "swish"])
def test_same_bits_over_what_a_plain_layer_may_be(what, monkeypatch):
    cfg = dict(BASE)
    if what == "heads in threes":
        cfg.update(num_attention_heads=6)
    if what == "swish":
        cfg.update(hidden_act="swish")
    model = build(cfg)
    for b in model.blocks:
        if what == "norms in float32":
            for n in (b.mixer_norm, b.ffn_norm):
                n.set_weights({"weight": n.weight.float() + 1e-3})
        pe = b._mixer.position_encoding
        if what == "interleaved":
            pe.is_neox = False
        if what == "half rotated":
            pe.rot_dim, pe.inv_freq = pe.rot_dim // 2, pe.inv_freq[::2].contiguous()
    same_bits(model, cfg, monkeypatch, {"pages of 8": 8, "pages of 64": 64}.get(what, 16))


def test_requests_of_very_unequal_length_stay_with_the_parts(monkeypatch):
    """A decode batch whose mean context is a quarter of its longest and less is split per request, from a list that a kernel of the step
    makes: the parts' own way, in eager steps and in graphs."""
    from lmsf_b200.engine.model_runner import ModelRunner, StepEntry
    taken = watch(monkeypatch)
    runner = ModelRunner(build(BASE), torch.bfloat16, torch.device("cuda:0"), 16, num_blocks=[300], max_num_seqs=64, max_model_len=1024)
    mgr = runner.make_cache_manager()
    for i in range(20):
        mgr.add(i)
    runner.step([StepEntry(i, util.random_ids(900 if i == 7 else 20, BASE["vocab_size"], i), [0]) for i in range(20)], mgr)
    assert taken == [True]
    for k in range(3):
        out = runner.step([StepEntry(i, [3 + i + k], [0]) for i in range(20)], mgr)
    assert taken == [True, False, False] and torch.isfinite(out).all()
    # the same beside a portion
    mgr.add(20)
    runner.step([StepEntry(i, [5 + i], [0]) for i in range(20)] + [StepEntry(20, util.random_ids(50, BASE["vocab_size"], 1), [0])], mgr)
    assert taken == [True, False, False, False]


def test_caches_of_another_geometry_are_refused():
    """Pages of fewer heads or of another size than the step's tables say are refused by the kernels' faces, as without the native loop:
    it looks at them before it hands their addresses on."""
    from lmsf_b200 import kernels
    from lmsf_b200.engine.model_runner import ModelRunner, StepEntry
    dev = torch.device("cuda:0")
    model = build(BASE)
    runner = ModelRunner(model, torch.bfloat16, dev, 16, num_blocks=[40], max_num_seqs=4, max_model_len=256)
    mgr = runner.make_cache_manager()
    mgr.add(0)
    good = [c.kv for c in runner.storage.layer_caches]
    for shape in ((41, 2, 1, 16, 64), (41, 2, 2, 8, 64), (41, 1, 2, 16, 64)):
        for c in runner.storage.layer_caches:
            c.kv = torch.zeros(shape, dtype=torch.bfloat16, device=dev)
        with pytest.raises(kernels.KernelError, match="cache of shape"):
            runner.step([StepEntry(0, util.random_ids(40, BASE["vocab_size"], 1), [39])], mgr)
    for c, kv in zip(runner.storage.layer_caches, good):
        c.kv = kv
    assert torch.isfinite(runner.step([StepEntry(0, util.random_ids(40, BASE["vocab_size"], 1), [39])], mgr)).all()


def test_unaligned_weights_are_multiplied_by_the_parts(monkeypatch):
    """A gate and up matrix at an odd address, in a step whose rows the gated kernel would take: the same logits as from an aligned one but
    for the rounding of gate and up in one layer of three (2^-8 of the value each; the bound is five times that)."""
    from lmsf_b200.engine.model_runner import ModelRunner, StepEntry
    from lmsf_b200.parts import linear, plain_layers
    dev = torch.device("cuda:0")
    model = build(BASE)
    monkeypatch.setattr(linear, "gated_in_one", lambda *a: True)
    runner = ModelRunner(model, torch.bfloat16, dev, 16, num_blocks=[40], max_num_seqs=4, max_model_len=256)
    mgr, ids, out, taken = runner.make_cache_manager(), util.random_ids(100, BASE["vocab_size"], 1), [], []
    inner = plain_layers.run
    monkeypatch.setattr(plain_layers, "run", lambda *a: (lambda r: (taken.append(r is not None), r)[1])(inner(*a)))
    ff = model.blocks[1].feed_forward
    for i, odd in enumerate((0, 1)):
        w = torch.empty(ff.gate_up.numel() + odd, dtype=torch.bfloat16, device=dev)[odd:].view(ff.gate_up.shape)
        w.copy_(ff.gate_up)
        ff.set_weights({"gate_up": w})
        mgr.add(i)
        out.append(runner.step([StepEntry(i, ids, list(range(100)))], mgr).double())
    assert taken == [True, False]
    assert (out[0] - out[1]).norm() <= 0.02 * out[0].norm()
