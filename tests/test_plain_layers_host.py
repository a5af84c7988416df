"""When the layer loop in native code (csrc/plain_layers.cu) takes a step, and when it leaves it to the parts, whose kernels' faces
then take it or refuse it.  The native call is a stand-in here: nothing is launched and no GPU is needed."""
import ctypes
import types

import pytest
import torch

from lmsf_b200 import kernels
from lmsf_b200 import models  # noqa: F401
from lmsf_b200.config.registry import resolve_architecture
from lmsf_b200.parts import linear, plain_layers
from lmsf_b200.parts.base import CacheGroupView, LayerCache, StepContext
from lmsf_b200.parts.decoder import DecoderModel
from lmsf_b200.weights.loader import collect_requirements

CFG = dict(architectures=["LlamaForCausalLM"], model_type="llama", hidden_size=128, num_hidden_layers=2, num_attention_heads=4,
           num_key_value_heads=2, head_dim=64, intermediate_size=256, vocab_size=50, rope_theta=10000.0, rms_norm_eps=1e-5,
           tie_word_embeddings=False, max_position_embeddings=512, hidden_act="silu", bos_token_id=1, eos_token_id=2)
BLOCK, PAGES, TOKENS = 16, 9, 40


def i32(*v):
    return torch.tensor(v, dtype=torch.int32)


@pytest.fixture
def step(monkeypatch):
    """(model, context, caches, embedding rows, calls of the stand-in) of one prompt of 40 tokens beside a request that decodes."""
    arch = resolve_architecture(dict(CFG))
    model = DecoderModel(arch.build_spec(arch.parse_config(dict(CFG))))
    per_part, parts = {}, {}
    for part, logical, wspec, _ in collect_requirements(model):
        sizes = [wspec.concrete(i) for i in range(len(wspec.shapes))]
        per_part.setdefault(id(part), {})[logical] = torch.zeros((sum(s[0] for s in sizes), *sizes[0][1:]), dtype=torch.bfloat16)
        parts[id(part)] = part
    for pid, tensors in per_part.items():
        parts[pid].set_weights(tensors)
    model.prepare(torch.bfloat16, torch.device("cpu"))
    n = TOKENS + 1
    ctx = StepContext(n_tokens=n, n_seqs=2, dtype=torch.bfloat16, device=torch.device("cpu"), token_ids=torch.zeros(n, dtype=torch.int32),
                      positions=torch.arange(n, dtype=torch.int32), token_seq=torch.zeros(n, dtype=torch.int32), cu_q=i32(0, TOKENS, n),
                      ctx_len=i32(TOKENS, 30), state_slot=i32(0, 1),
                      groups=[CacheGroupView(torch.zeros((2, 3), dtype=torch.int32), BLOCK)], q_lens=[TOKENS, 1], ctx_lens=[TOKENS, 30],
                      state_slots=[0, 1], error_flag=i32(0), decode_seq_ids=i32(1), n_decode_seqs=1, q_tile_seq=i32(0), q_tile_q0=i32(0),
                      n_q_tiles=1, q_tile128_seq=i32(0), q_tile128_q0=i32(0), n_q_tiles128=1)
    caches = [LayerCache(kv=torch.zeros((PAGES, 2, 2, BLOCK, 64), dtype=torch.bfloat16), group=0) for _ in range(2)]
    x = torch.zeros((n, 128), dtype=torch.bfloat16)
    taken = []

    def run(step_ref, layers, rc):
        s = ctypes.cast(step_ref, ctypes.POINTER(plain_layers._Step)).contents
        taken.append({name: getattr(s, name) for name, _ in s._fields_})
        return 9

    monkeypatch.setattr(plain_layers, "_usable", lambda device: True)
    monkeypatch.setattr(plain_layers, "_entry_points", lambda head_dim: {})
    monkeypatch.setattr(plain_layers, "_library_product", lambda: (1, 2, 3))
    monkeypatch.setattr(plain_layers, "load_library", lambda source, defines=(): types.SimpleNamespace(lmsf_plain_layers_run=run))
    monkeypatch.setattr(plain_layers.attention, "planned_splits", lambda *a: (1, 4))
    monkeypatch.setattr(torch.cuda, "current_blas_handle", lambda: 0)
    monkeypatch.setattr(kernels, "_stream", lambda: 0)
    monkeypatch.setattr(kernels, "sm_count", lambda device: 148)
    monkeypatch.setattr(kernels, "_ptr", lambda t: None if t is None else t.data_ptr())
    return types.SimpleNamespace(model=model, ctx=ctx, caches=caches, x=x, taken=taken, fits=lambda: plain_layers.run(model, ctx, caches, x) is not None)


def test_a_plain_step_is_taken(step):
    assert step.fits() and len(step.taken) == 1
    s = step.taken[0]
    assert (s["tokens"], s["hidden"], s["n_decode"], s["n_tiles"], s["n_seqs"], s["splits"]) == (41, 128, 1, 1, 2, 1)
    assert s["page_stride"] == 2 * 2 * BLOCK * 64 and s["n_pages"] == PAGES and s["block_size"] == BLOCK


@pytest.mark.parametrize("shape", [(PAGES, 2, 2, BLOCK // 2, 64), (PAGES, 2, 4, BLOCK, 64), (PAGES, 2, 2, BLOCK, 32), (PAGES, 1, 2, BLOCK, 64),
                                   (PAGES, 2, 2, BLOCK * 2, 32)])
def test_caches_of_another_geometry_are_left_to_the_parts(step, shape):
    """All caches alike, but not what the heads and the pages of the step say: rope_cache_write and the attention refuse them."""
    for c in step.caches:
        c.kv = torch.zeros(shape, dtype=torch.bfloat16)
    assert not step.fits() and not step.taken


def test_caches_at_an_odd_address_are_left_to_the_parts(step):
    n = step.caches[0].kv.numel()
    step.caches[1].kv = torch.zeros(n + 1, dtype=torch.bfloat16)[1:].view(step.caches[0].kv.shape)
    assert not step.fits() and not step.taken


TABLES = ["positions", "token_seq", "cu_q", "ctx_len", "block_table", "decode_seq_ids", "q_tile128_seq", "q_tile128_q0", "error_flag"]


@pytest.mark.parametrize("name,how", [(n, h) for n in TABLES for h in ("int64", "another device")] + [(n, "strided") for n in TABLES[:5]])
def test_tables_of_another_kind_are_left_to_the_parts(step, name, how):
    """What the kernels' faces refuse (`kernels._i32`): tables that are not 32-bit, not contiguous or not on the step's device."""
    owner = step.ctx.groups[0] if name == "block_table" else step.ctx
    t = getattr(owner, name)
    if how == "int64":
        t = t.long()
    elif how == "strided":
        t = torch.stack([t, t], -1)[..., 0]
    else:
        t = t.to("meta")
    setattr(owner, name, t)
    assert not step.fits() and not step.taken


def test_a_block_table_of_other_requests_is_left_to_the_parts(step):
    """attention_decode sizes its scratch by the table's rows."""
    step.ctx.groups[0].block_table = torch.zeros((5, 3), dtype=torch.int32)
    assert not step.fits() and not step.taken


def test_frequencies_elsewhere_are_left_to_the_parts(step):
    pe = step.model.blocks[1]._mixer.position_encoding
    pe.inv_freq = pe.inv_freq.to("meta")
    assert not step.fits() and not step.taken


def test_an_unaligned_gate_and_up_matrix_is_left_to_the_parts(step, monkeypatch):
    """A contiguous matrix at an odd address: the gated kernel would refuse it in the middle of the layers, the parts multiply with the
    library there.  Without the gated kernel the loop takes it as the library does."""
    ff = step.model.blocks[1].feed_forward
    w = ff.gate_up
    ff.set_weights({"gate_up": torch.zeros(w.numel() + 1, dtype=w.dtype)[1:].view(w.shape)})
    monkeypatch.setattr(linear, "gated_in_one", lambda *a: True)
    assert not step.fits() and not step.taken
    monkeypatch.setattr(linear, "gated_in_one", lambda *a: False)
    assert step.fits() and step.taken[0]["gu"] is not None


def test_a_step_without_an_error_word_does_not_take_the_gated_kernel_here(step, monkeypatch):
    """The kernel reports a wait that ran out; its face falls back on the device's own word, which the loop would not."""
    step.ctx.error_flag = None
    monkeypatch.setattr(linear, "gated_in_one", lambda *a: True)
    assert not step.fits() and not step.taken
    monkeypatch.setattr(linear, "gated_in_one", lambda *a: False)
    assert step.fits()


def test_the_build_of_the_attention_is_the_parts_own(monkeypatch):
    """A pipeline depth set between two steps names another build of the decode attention, for the loop as for the parts."""
    monkeypatch.setattr(plain_layers, "_addresses", {})
    monkeypatch.setattr(plain_layers, "_address", lambda source, name, defines=(): (source, defines))
    for depth in (None, 2, None):
        monkeypatch.setattr(kernels, "MMA_KV_STAGES", depth)
        for head_dim in (64, 128):
            assert plain_layers._entry_points(head_dim)["decode"] == ("attention_mma.cu", kernels._mma_defines(head_dim))
            assert plain_layers._entry_points(head_dim)["prefill"] == ("attention_tc.cu", (f"LMSF_HEAD_DIM={head_dim}",))


@pytest.mark.parametrize("part,name,shape,dtype", [("_mixer", "qkv_bias", (512,), torch.bfloat16), ("_mixer", "o_bias", (128,), torch.bfloat16),
                                                   ("_mixer", "_sinks", (4,), torch.float32), ("_mixer", "_hb32", (4,), torch.float32),
                                                   ("feed_forward", "gate_up_bias", (512,), torch.bfloat16),
                                                   ("feed_forward", "down_bias", (128,), torch.bfloat16)])
def test_biases_that_a_part_was_given_keep_the_parts_own_way(step, part, name, shape, dtype):
    """A part adds the biases that it holds, whether its parameters spoke of them or not."""
    getattr(step.model.blocks[1], part).set_weights({name: torch.zeros(shape, dtype=dtype)})
    assert not step.fits() and not step.taken


def test_another_library_for_products_keeps_the_parts_own_way(step):
    """torch.mm follows a program's choice of library, the loop calls cuBLAS."""
    before = torch.backends.cuda.preferred_blas_library()
    try:
        torch.backends.cuda.preferred_blas_library("cublaslt")
        assert not step.fits() and not step.taken
    finally:
        torch.backends.cuda.preferred_blas_library(before)
    assert step.fits()


def test_the_library_is_the_one_that_torch_brings(monkeypatch):
    """It is looked up by torch's own version, and a program is told when it is not there."""
    monkeypatch.setattr(plain_layers, "_cublas", None)
    assert len(plain_layers._library_product()) == 3
    monkeypatch.setattr(plain_layers, "_cublas", None)
    monkeypatch.setattr(torch.version, "cuda", "99.1")
    with pytest.warns(RuntimeWarning, match="libcublas.so.99"):
        assert plain_layers._library_product() is None
