"""All layers of a plain pre-norm decoder in one native call (``csrc/prenorm_layers.cu``): the launches that
``PreNormBlock``, ``PagedAttention`` and ``GatedMLP`` would make one by one for a step with prompt portions, in the same order and
with the same operands.  Issued from Python such a step is bound by the host up to about a thousand tokens.

Which models: every block pre-norm with RMS norms, attention without options beside a rotation table and a window, a silu
feed-forward, bfloat16 throughout, all layers of one geometry, nothing done to the stream between them.  Which steps: more
rows than the streaming products take, and at least one request that brings more than one token (steps of decode tokens
alone are graphs), with ``torch.mm`` left at its own defaults.  Sizes and pointers are read anew for every step; nothing is kept from one to the next."""

from __future__ import annotations

import ctypes
import os
from ctypes import c_float, c_int, c_void_p

import torch

from .. import kernels
from .attention import PORTION_ROWS, PagedAttention
from .block import PreNormBlock
from .feedforward import GatedMLP
from .norms import RMSNorm

_LAYER_POINTERS = ("norm1", "qkv_w", "o_w", "norm2", "gate_up_w", "down_w", "kpool", "vpool")
_STEP_POINTERS = ("gemm_ex", "handle", "gemm_silu", "attn_small", "attn_tc", "attn_mma", "residual", "delta", "normed", "qkv", "attn_out",
                  "mixer_out", "gate_up", "hidden", "ff_out", "cos_t", "sin_t", "positions", "slot_mapping", "block_table", "q_start",
                  "ctx_before", "work_req", "work_pair0", "scratch")
_STEP_INTS = ("n", "width", "n_heads", "n_kv_heads", "hd", "inter", "page_size", "table_stride", "n_requests", "n_pages", "window",
              "n_work", "n_splits", "split_keys", "rotate_q", "n_sms", "mma_rows")


class _Layer(ctypes.Structure):
    _fields_ = ([(n, c_void_p) for n in _LAYER_POINTERS] + [("eps1", c_float), ("eps2", c_float)]
                + [("gain1_dtype", c_int), ("gain2_dtype", c_int)])


class _Step(ctypes.Structure):
    _fields_ = [(n, c_void_p) for n in _STEP_POINTERS] + [(n, c_int) for n in _STEP_INTS] + [("scale", c_float)]


_gemm_ex: int | None = None


def _library_product() -> int:
    """The address of the matrix product that ``torch.mm`` calls for bfloat16 operands (0: not found).  It gets PyTorch's own
    handle, so it has to come from the library that PyTorch has loaded: a library of the same name that only lies on the path
    is not opened, nor one of another major version than PyTorch was built for."""
    global _gemm_ex
    if _gemm_ex is None:
        try:
            major = (torch.version.cuda or "").split(".")[0]
            if major != "12":              # the types of the call (parts of the library's interface) are those of version 12
                raise OSError("PyTorch is built for another version of the library")
            lib = ctypes.CDLL("libcublas.so.12", mode=os.RTLD_NOLOAD | os.RTLD_NOW)
            _gemm_ex = ctypes.cast(lib.cublasGemmEx, c_void_p).value or 0
        except (OSError, AttributeError):
            _gemm_ex = 0
    return _gemm_ex


def _torch_product_is_plain() -> bool:
    """Whether ``torch.mm`` would call that very product with the handle's standing settings.  A program can ask for full-precision
    partial sums, another library or tuned kernels, and ``torch.mm`` looks at all three on every call."""
    return (torch.backends.cuda.matmul.allow_bf16_reduced_precision_reduction is True and not torch.cuda.tunable.is_enabled()
            and torch.backends.cuda.preferred_blas_library() == torch._C._BlasBackend.Cublas)


def _address(fn) -> int:
    return ctypes.cast(fn, c_void_p).value


def _geometry(block, rt):
    """What all layers have to share, or None for a block that is not of the plain kind."""
    if type(block) is not PreNormBlock or block.feedforward is None:
        return None
    a, f = block.mixer, block.feedforward
    if type(a) is not PagedAttention or type(f) is not GatedMLP or type(block.mixer_norm) is not RMSNorm or type(block.ff_norm) is not RMSNorm:
        return None
    s = a.spec
    weights = (a.qkv, a.o, f.gate_up, f.down)
    if not (a.plain and f.plain_silu and s.head_dim in kernels.MMA_HEAD_DIMS and getattr(a.position, "score_bias", None) is None
            and a.position.rotary_tables() is not None and s.n_heads // s.n_kv_heads <= 16
            and all(w.bias is None and w.weight.dtype is torch.bfloat16 for w in weights)):
        return None
    return (s.hidden, s.n_heads, s.n_kv_heads, s.head_dim, s.window, a.scale, f.spec.intermediate, id(a.position.rotary_tables()[0]))


class NativeLayers:
    def __init__(self, blocks, views, rt):
        self.blocks, self.views, self.rt = blocks, views, rt

    @classmethod
    def of(cls, model, views):
        """For a decoder whose cache is bound; None where the parts have to run one by one."""
        rt = model.rt
        blocks = [model.layers[e.layer] for e in model.spec.schedule]
        if rt.act_dtype is not torch.bfloat16 or not blocks:
            return None
        shapes = [_geometry(b, rt) for b in blocks]
        if shapes[0] is None or any(s != shapes[0] for s in shapes):
            return None
        if any(v.kind != "kv" or not v.write or v.group != views[0].group or v.k.shape != views[0].k.shape
               or not v.k.is_contiguous() or not v.v.is_contiguous() for v in views[:len(blocks)]):
            return None
        sizes = (c_int(), c_int())
        kernels.core().ie_prenorm_layers_sizes(*(ctypes.addressof(x) for x in sizes))
        assert (sizes[0].value, sizes[1].value) == (ctypes.sizeof(_Layer), ctypes.sizeof(_Step)), "prenorm_layers.cu has another layout"
        return cls(blocks, list(views[:len(blocks)]), rt)

    def takes(self, ctx) -> bool:
        return ctx.n_tokens > kernels.STREAM_BEST_ROWS and ctx.max_q_len > 1 and "graph" not in ctx.host and _torch_product_is_plain() \
            and _library_product() != 0

    def forward(self, residual: torch.Tensor, pending, ctx):
        """``(residual, delta)`` after the last layer, as its block would return them."""
        ws, bf, ptr = self.rt.ws, torch.bfloat16, kernels._ptr
        a, f = self.blocks[0].mixer, self.blocks[0].feedforward
        s, n, group = a.spec, ctx.n_tokens, a.spec.n_heads // a.spec.n_kv_heads
        kv = ctx.kv[self.views[0].group]
        inter = f.spec.intermediate
        st = _Step()
        qkv = ws.take("attn_qkv", (n, a.q_width + 2 * a.k_width), bf)
        ff_out = ws.take("ff_out", (n, s.hidden), bf)
        cos, sin = a.position.rotary_tables()
        st.gemm_ex, st.handle = _library_product(), torch.cuda.current_blas_handle()
        st.residual, st.delta, st.normed = ptr(residual), ptr(pending), ptr(ws.take("normed", tuple(residual.shape), bf))
        st.qkv, st.attn_out = ptr(qkv), ptr(ws.take("attn_out", (n, a.out_width), bf))
        st.mixer_out, st.ff_out = ptr(ws.take("mixer_out", (n, s.hidden), bf)), ptr(ff_out)
        st.hidden = ptr(ws.take("ff_hidden", (n, inter), bf))
        if f.gate_up_on_tcgen05(n, s.hidden):
            st.gemm_silu = _address(kernels.tcgen05_library().ie_gemm_tcgen05_act)
        else:
            st.gate_up = ptr(ws.take("ff_gate_up", (n, 2 * inter), bf))
        st.cos_t, st.sin_t, st.positions = ptr(cos), ptr(sin), ptr(ctx.positions)
        st.slot_mapping, st.block_table, st.q_start, st.ctx_before = (ptr(t) for t in (kv.slot_mapping, kv.block_table, ctx.q_start, ctx.ctx_before))
        st.rotate_q = 0 if a._portions_only_on_tcgen05(ctx) else 1
        # the requests of at most 16 rows on the split-key kernel, the others on tiles, as PagedAttention deals them out
        n_small, keys = a.small_requests(ctx, False)
        if n_small:
            st.n_splits, st.split_keys = a.split_keys(n_small, keys, False)
            st.scratch = ptr(a._decode_scratch(ctx, st.n_splits))
            st.attn_small = _address(kernels.attention_mma_library(s.head_dim).ie_attention_decode)
        if n_small < ctx.n_requests:
            on_tc = a.portions_on_tcgen05(ctx)
            st.mma_rows = PORTION_ROWS
            work_req, work_pair0, st.n_work = ctx.attention_work(group, 128 if on_tc else PORTION_ROWS, 16 if n_small else 0)
            st.work_req, st.work_pair0 = ptr(work_req), ptr(work_pair0)
            if on_tc:
                st.attn_tc = _address(kernels.attention_tcgen05_library().ie_attention_tcgen05)
            else:
                st.attn_mma = _address(kernels.attention_mma_library(s.head_dim).ie_attention_prefill)
        st.n, st.width, st.n_heads, st.n_kv_heads, st.hd, st.inter = n, s.hidden, s.n_heads, s.n_kv_heads, s.head_dim, inter
        st.page_size, st.table_stride, st.n_requests = ctx.page_size, kv.block_table.stride(0), ctx.n_requests
        st.n_pages, st.window, st.n_sms, st.scale = self.views[0].k.shape[0], int(s.window or 0), kernels.sm_count(), a.scale
        table = (_Layer * len(self.blocks))()
        for row, b, v in zip(table, self.blocks, self.views):
            n1, n2 = b.mixer_norm, b.ff_norm
            row.norm1, row.qkv_w, row.o_w = n1.gain.data_ptr(), b.mixer.qkv.weight.data_ptr(), b.mixer.o.weight.data_ptr()
            row.norm2, row.gate_up_w, row.down_w = n2.gain.data_ptr(), b.feedforward.gate_up.weight.data_ptr(), b.feedforward.down.weight.data_ptr()
            row.kpool, row.vpool, row.eps1, row.eps2 = v.k.data_ptr(), v.v.data_ptr(), n1.eps, n2.eps
            row.gain1_dtype, row.gain2_dtype = kernels.dtype_code(n1.gain.dtype), kernels.dtype_code(n2.gain.dtype)
        kernels.prenorm_layers(ctypes.addressof(table), len(self.blocks), ctypes.addressof(st))
        return residual, ff_out
