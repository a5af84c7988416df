"""The layers of a plain pre-norm decoder in one native call (csrc/plain_layers.cu).

Steps with more rows than the weight-streaming products take (prompts, mixed steps, decode batches above 16) launch eight to ten
kernels a layer: four of them products of the library, or three and the gated kernel, and two attentions where prompts run beside
requests that decode.  Made one by one from Python they cost the host 15 to 20 us each, more than the device needs for them while
the rows are few.  Where every layer is the plain arrangement (RMSNorm, paged attention with a rotation and without anything a design may add,
RMSNorm, gated feed-forward; bfloat16; no biases) the loop over them runs in native code, with the same kernels and the same
arguments.  Anything else keeps the parts' own `forward`.  Whether a model is plain, and where its weights lie, is read anew at
every step: parts may be changed or given other weights between steps.
"""
from __future__ import annotations

import ctypes
import os
import warnings
from ctypes import c_float, c_int, c_longlong, c_void_p
from typing import List, Optional, Tuple

import torch

from .. import kernels
from ..csrc.build import load_library
from ..utils import tracing
from . import attention, linear
from .attention import PagedAttention
from .base import LayerCache, StepContext
from .block import PreNormBlock
from .mlp import GatedMLP
from .norm import RMSNorm
from .rope import RotaryEmbedding

USE_NATIVE_LAYERS = True


class _Step(ctypes.Structure):
    _fields_ = ([(n, c_void_p) for n in ("norm", "rope", "act", "decode", "prefill", "gated", "gemm", "get_mode", "set_mode", "handle", "stream",
                                         "x", "y", "res", "h", "qkv", "att", "gu", "m", "positions", "token_seq", "block_table", "cu_q",
                                         "ctx_len", "decode_seq_ids", "tile_seq", "tile_q0", "error_flag", "scratch")]
                + [("page_stride", c_longlong), ("n_pages", c_longlong)]
                + [(n, c_int) for n in ("tokens", "hidden", "n_q_heads", "n_kv_heads", "head_dim", "ff", "max_blocks", "block_size",
                                        "n_decode", "n_tiles", "act_code", "n_layers", "n_seqs", "splits", "warps", "pad")])


class _Layer(ctypes.Structure):
    _fields_ = ([(n, c_void_p) for n in ("norm1", "qkv", "o", "norm2", "gate_up", "down", "cache", "inv_freq")]
                + [(n, c_int) for n in ("norm1_dtype", "norm2_dtype", "rot_dim", "is_neox")]
                + [(n, c_float) for n in ("eps1", "eps2", "scale")] + [("pad", c_int)])


_STAGES = {2: ("rmsnorm.cu", "lmsf_rmsnorm"), 3: ("rope_cache.cu", "lmsf_rope_cache"), 4: ("attention_mma.cu", "lmsf_attention_mma"),
           5: ("attention_tc.cu", "lmsf_attention_tc"), 6: ("activation.cu", "lmsf_activation"), 7: ("gemm_gated_tc.cu", "lmsf_gemm_gated_tc")}
_cublas = None


def _library_product():
    """(cublasGemmEx, cublasGetMathMode, cublasSetMathMode) of the library that torch has loaded, or None (said once)."""
    global _cublas
    if _cublas is None:
        name = f"libcublas.so.{(torch.version.cuda or '0').split('.')[0]}"
        try:
            lib = ctypes.CDLL(name, mode=os.RTLD_NOLOAD | os.RTLD_NOW)
            _cublas = tuple(ctypes.cast(getattr(lib, n), c_void_p).value for n in ("cublasGemmEx", "cublasGetMathMode", "cublasSetMathMode"))
        except (OSError, AttributeError) as e:
            warnings.warn(f"torch's cuBLAS was not found as {name} ({e}); steps of many rows are launched from Python, short prompts take "
                          f"twice as long", RuntimeWarning, stacklevel=2)
            _cublas = ()
    return _cublas or None


def _products_are_cublas() -> bool:
    """Whether torch.mm goes to the library that the loop calls (a program may prefer cublasLt for its products)."""
    return torch.backends.cuda.preferred_blas_library() in (torch._C._BlasBackend.Default, torch._C._BlasBackend.Cublas)


def _address(source: str, name: str, defines=()) -> int:
    lib = load_library(source, defines)
    return ctypes.cast(getattr(lib, name), c_void_p).value


_addresses = {}


def _entry_points(head_dim: int):
    defines = kernels._mma_defines(head_dim)              # names the build: a pipeline depth may have been set since the last step
    a = _addresses.get(defines)
    if a is None:
        a = _addresses[defines] = dict(
            norm=_address("rmsnorm.cu", "lmsf_add_rmsnorm"), rope=_address("rope_cache.cu", "lmsf_rope_cache_write"),
            act=_address("activation.cu", "lmsf_gated_act"), gated=_address("gemm_gated_tc.cu", "lmsf_gemm_gated_tc"),
            decode=_address("attention_mma.cu", "lmsf_attention_decode_width", defines),
            prefill=_address("attention_tc.cu", "lmsf_attention_prefill_tc", defines[:1]))
        f = load_library("plain_layers.cu").lmsf_plain_layers_run
        f.restype, f.argtypes = c_int, [c_void_p, c_void_p, c_void_p]
    return a


def plain_attention(m) -> bool:
    """Whether an attention part is the plain one: rotated queries and keys, a softmax over all keys, nothing beside it (neither
    declared nor handed over by `set_weights`: the part's own way looks at the tensors)."""
    pe = m.position_encoding
    return (type(m) is PagedAttention and type(pe) is RotaryEmbedding and pe.mult == 1.0 and m.own_kv and not (
        m.qk_filter_taps or m.values_are_keys or m.head_gate or m.value_gate or m.qk_norm or m.value_norm or m.has_bias or m.has_out_bias
        or m.window or m.chunk or m.softcap or m.sigmoid_weights or m.has_head_bias or m.unit_sink or m.learned_sink) and all(
        t is None for t in (m.qkv_bias, m.o_bias, m._hb32, m._sinks)))


def _plain_block(b) -> bool:
    if type(b) is not PreNormBlock:
        return False
    n1, n2, ff = b.mixer_norm, b.ffn_norm, b.feed_forward
    return (type(n1) is RMSNorm and type(n2) is RMSNorm and not n1.has_layer_scale and not n2.has_layer_scale and type(ff) is GatedMLP
            and not ff.has_bias and ff.gate_up_bias is None and ff.down_bias is None and ff.activation in kernels.ACT_CODES and plain_attention(b._mixer))


def _matrix(w: Optional[torch.Tensor], rows: int, cols: int, device: torch.device) -> int:
    """The address of a contiguous bfloat16 matrix of this shape on the device, or 0."""
    if w is None or w.dtype != torch.bfloat16 or w.device != device or w.shape != (rows, cols) or not w.is_contiguous():
        return 0
    return w.data_ptr()


def _vector(w: Optional[torch.Tensor], n: int, device: torch.device) -> Tuple[int, int]:
    if w is None or w.device != device or w.shape != (n,) or not w.is_contiguous() or w.dtype not in (torch.bfloat16, torch.float32):
        return 0, 0
    return w.data_ptr(), kernels.dtype_code(w.dtype)


def _usable(device: torch.device) -> bool:
    return device.type == "cuda"


def _tables_fit(ctx: StepContext, block_table: torch.Tensor, device: torch.device) -> bool:
    """Whether the step's tables are what the kernels' faces ask for (`kernels._i32`): they go to the native loop as addresses, and
    nothing behind it can look at them."""
    tables = [ctx.positions, ctx.token_seq, ctx.cu_q, ctx.ctx_len, block_table]
    if ctx.error_flag is not None:
        tables.append(ctx.error_flag)
    if ctx.n_decode_seqs and ctx.n_decode_seqs != ctx.n_seqs:
        tables.append(ctx.decode_seq_ids)
    if ctx.n_q_tiles:
        tables += [ctx.q_tile128_seq, ctx.q_tile128_q0]
    return block_table.dim() == 2 and block_table.shape[0] == ctx.n_seqs and all(
        t is not None and t.dtype == torch.int32 and t.device == device and t.is_contiguous() for t in tables)


def _cache_fits(kv: Optional[torch.Tensor], shape: Tuple[int, ...], device: torch.device) -> bool:
    """Whether a layer's pages are [pages, 2, kv heads, block size, head size] as the step's heads and tables say."""
    return (kv is not None and kv.dtype == torch.bfloat16 and kv.device == device and tuple(kv.shape) == shape and kv.is_contiguous()
            and kv.data_ptr() % 16 == 0)


def run(model, ctx: StepContext, caches: List[LayerCache], x: torch.Tensor) -> Optional[Tuple[torch.Tensor, torch.Tensor]]:
    """(pending branch, residual stream) behind the last layer, or None where the parts have to run themselves.  x: the embedding."""
    if not (USE_NATIVE_LAYERS and ctx.dtype == torch.bfloat16 and ctx.n_tokens > kernels.SKINNY_MAX_M and attention.USE_TC_PREFILL
            and linear.USE_SKINNY and not tracing.ENABLED and model.layer_hook is None and not ctx.extras.get("force_generic_attention")
            and not torch.backends.cuda.matmul.allow_bf16_reduced_precision_reduction and _products_are_cublas()):
        return None
    calls, blocks = model.calls, model.blocks
    first = blocks[calls[0].layer] if calls else None
    if first is None or not _plain_block(first):
        return None
    m0, T, D = first._mixer, ctx.n_tokens, first.mixer_norm.hidden_size
    nh, nkv, hd, ff = m0.num_heads, m0.num_kv_heads, m0.head_dim, first.feed_forward.intermediate_size
    act, group_index, kv0 = first.feed_forward.activation, caches[0].group, caches[0].kv
    device = x.device
    if hd not in (64, 128) or kv0 is None or x.dtype != torch.bfloat16 or not x.is_contiguous() or x.shape != (T, D) or \
            not _usable(device) or _library_product() is None:
        return None
    # What the kernels' faces refuse is left to the parts, which say so
    group = ctx.groups[group_index]
    pages = (kv0.shape[0], 2, nkv, group.block_size, hd)
    if not _tables_fit(ctx, group.block_table, device):
        return None
    if ctx.n_decode_seqs:
        visible, mean_visible = attention.decode_lengths(ctx)
        if attention.splits_per_request(ctx, visible, mean_visible):
            return None                     # a list of work items that a kernel of the step makes: the parts' own way
    q_size, kv_size = nh * hd, nkv * hd
    layers = (_Layer * len(calls))()
    for j, call in enumerate(calls):
        b, c = blocks[call.layer], caches[j]
        if call.entry is not None or call.cache_of is not None or not c.owner or c.group != group_index or c.extra or (j and not _plain_block(b)):
            return None
        m, f, n1, n2 = b._mixer, b.feed_forward, b.mixer_norm, b.ffn_norm
        inv = m.position_encoding.inv_freq
        if (m.num_heads, m.num_kv_heads, m.head_dim, m.hidden_size, f.intermediate_size, f.activation) != (nh, nkv, hd, D, ff, act) or \
                not _cache_fits(c.kv, pages, device) or inv is None or inv.dtype != torch.float32 or inv.device != device or \
                inv.numel() * 2 != m.position_encoding.rot_dim:
            return None
        l = layers[j]
        l.qkv, l.o = _matrix(m.qkv, q_size + 2 * kv_size, D, device), _matrix(m.o, D, q_size, device)
        l.gate_up, l.down = _matrix(f.gate_up, 2 * ff, D, device), _matrix(f.down, D, ff, device)
        l.norm1, l.norm1_dtype = _vector(n1.weight, D, device)
        l.norm2, l.norm2_dtype = _vector(n2.weight, D, device)
        if not (l.qkv and l.o and l.gate_up and l.down and l.norm1 and l.norm2):
            return None
        l.cache, l.inv_freq, l.rot_dim, l.is_neox = c.kv.data_ptr(), inv.data_ptr(), m.position_encoding.rot_dim, int(m.position_encoding.is_neox)
        l.eps1, l.eps2, l.scale = n1.eps, n2.eps, m.scale
    gated = linear.gated_in_one(T, D, ff, device)
    if gated and (ctx.error_flag is None or any(l.gate_up % 16 for l in layers)):
        # The parts' own way: they choose per layer (the gated kernel wants 16-byte alignment, the library does not), and report a wait
        # that ran out in the device's error word where the step names none
        return None
    # The buffers: the pending branch, the normed rows and the residual stream stay; q, k, v and the heads' outputs share their place
    # with what the feed-forward holds, which is not needed at the same time.
    up = lambda n: (n + 255) // 256 * 256
    row, gu_bytes = up(T * D * 2), 0 if gated else up(T * 2 * ff * 2)
    both = max(up(T * (q_size + 2 * kv_size) * 2) + up(T * q_size * 2), gu_bytes + up(T * ff * 2))
    space = torch.empty(row + both, dtype=torch.uint8, device=device)
    y, res = torch.empty_like(x), torch.empty((T, D), dtype=torch.float32, device=device)
    s = _Step(**_entry_points(hd))
    s.gemm, s.get_mode, s.set_mode = _library_product()
    s.handle, s.stream = torch.cuda.current_blas_handle(), kernels._stream()
    at = space.data_ptr()
    s.x, s.y, s.res, s.h = x.data_ptr(), y.data_ptr(), res.data_ptr(), at
    s.qkv, s.att = at + row, at + row + up(T * (q_size + 2 * kv_size) * 2)
    s.gu, s.m = None if gated else at + row, at + row + gu_bytes
    s.positions, s.token_seq, s.block_table = ctx.positions.data_ptr(), ctx.token_seq.data_ptr(), group.block_table.data_ptr()
    s.cu_q, s.ctx_len = ctx.cu_q.data_ptr(), ctx.ctx_len.data_ptr()
    s.max_blocks, s.block_size, s.page_stride, s.n_pages = group.block_table.shape[1], group.block_size, kv0.stride(0), kv0.shape[0]
    s.error_flag = ctx.error_flag.data_ptr() if ctx.error_flag is not None else None
    if ctx.n_decode_seqs:
        s.decode_seq_ids = None if ctx.n_decode_seqs == ctx.n_seqs else ctx.decode_seq_ids.data_ptr()
        s.splits, s.warps = attention.planned_splits(ctx, nh, nkv, hd, visible, mean_visible)
        scratch = attention.decode_scratch(ctx, nh, s.splits, hd)
        s.scratch = scratch.data_ptr() if scratch is not None else None
    if ctx.n_q_tiles:
        s.tile_seq, s.tile_q0 = ctx.q_tile128_seq.data_ptr(), ctx.q_tile128_q0.data_ptr()
    s.n_decode, s.n_tiles = ctx.n_decode_seqs, ctx.n_q_tiles128 if ctx.n_q_tiles else 0
    s.tokens, s.hidden, s.n_q_heads, s.n_kv_heads, s.head_dim, s.ff = T, D, nh, nkv, hd, ff
    s.act_code, s.n_layers, s.n_seqs = kernels.ACT_CODES[act], len(calls), ctx.n_seqs
    rc = c_int(0)
    n = load_library("plain_layers.cu").lmsf_plain_layers_run(ctypes.byref(s), layers, ctypes.byref(rc))
    if n < 0:
        source, prefix = _STAGES.get(-n, (None, None))
        if source is None:
            raise kernels.KernelError(f"the library's product failed ({rc.value})")
        kernels._check(rc.value, source, prefix, kernels._mma_defines(hd) if -n == 4 else kernels._mma_defines(hd)[:1] if -n == 5 else ())
    kernels.add_launches(n)
    return y, res
