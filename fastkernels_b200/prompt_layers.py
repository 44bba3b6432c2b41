"""A decoder layer of a Llama / Qwen3 prompt portion in one native call.

LlamaModel.forward offers its layers to a `PromptRun` one by one: it launches what the layer
would launch (fk_llama_prompt_layers) when calling it as a module would do nothing else, and
returns None when it might: a hooked, compiled or replaced module, class or operator, a tensor
that one of the operators would convert or refuse, tensor parallelism, gradients.  Nothing is kept
between calls.
"""
from __future__ import annotations

import struct

import torch
from torch.nn.modules import module as _module

from fastkernels_b200 import _lib, ops
from fastkernels_b200.candidate.L1.flash_attn_prefill import FlashAttnPrefill
from fastkernels_b200.candidate.L1.flashinfer_prefill import TRTLLMPrefill
from fastkernels_b200.candidate.L1.rms_norm import RMSNorm
from fastkernels_b200.candidate.L1.rotary_emb import RotaryEmbedding
from fastkernels_b200.candidate.L1.silu_and_mul import SiluAndMul
from fastkernels_b200.candidate.L2.attention import LlamaAttention
from fastkernels_b200.candidate.L2.attention_impl import Attention
from fastkernels_b200.candidate.L2.llama_mlp import LlamaMLP
from fastkernels_b200.candidate.L2.parallel_linear import (MergedColumnParallelLinear,
                                                            QKVParallelLinear, RowParallelLinear)
from fastkernels_b200.candidate.L3.llama_decoder import LlamaDecoderLayer
from fastkernels_b200.comm import get_tp_comm
from fastkernels_b200.infra.context import get_context
from fastkernels_b200.infra.tp import _tp_size

BF16 = torch.bfloat16
_PREFILL = {"NHD": FlashAttnPrefill, "HND": TRTLLMPrefill}

# what the layers run, as it is defined here
_DEFINED = [(c, "forward", c.__dict__["forward"]) for c in
            (LlamaDecoderLayer, LlamaAttention, LlamaMLP, RMSNorm, QKVParallelLinear,
             MergedColumnParallelLinear, RowParallelLinear, SiluAndMul, FlashAttnPrefill,
             TRTLLMPrefill)]
_DEFINED += [(c, n, c.__dict__[n]) for c, n in
             ((LlamaDecoderLayer, "add_norm"), (RMSNorm, "forward_cuda"), (Attention, "attend"),
              (LlamaMLP, "_stock"), (RotaryEmbedding, "activation_cache"))]
_DEFINED += [(ops, n, getattr(ops, n)) for n in
             ("rmsnorm", "fused_add_rmsnorm", "gemm_bf16", "qkv_rope_store", "prefill_attn",
              "gemm_silu_mul", "gemm_silu_mul_fusable", "gemm_act_mul_many",
              "gemm_act_mul_many_fits", "silu_and_mul")]
_OWN = {"forward", "attend", "add_norm", "forward_cuda", "_stock", "activation_cache"}


def _plain(module, kind) -> bool:
    """Calling the module runs what its class defines and nothing else."""
    d = module.__dict__
    return type(module) is kind and not (
        d["_forward_hooks"] or d["_forward_pre_hooks"] or d["_backward_hooks"]
        or d["_backward_pre_hooks"] or d.get("_compiled_call_impl") is not None
        or not _OWN.isdisjoint(d))


class _NotPlain(Exception):
    pass


def _linear(module, kind, rows, cols, device):
    """(weight, bias) addresses of a projection to `rows` columns."""
    if not _plain(module, kind):
        raise _NotPlain
    p = module._parameters
    w, b = p.get("weight"), p.get("bias")
    if w is None or w.dtype is not BF16 or w.device != device or w.shape != (rows, cols) or \
            not w.is_contiguous():
        raise _NotPlain
    if b is None:
        return w.data_ptr(), 0
    if b.dtype is not BF16 or b.device != device or b.shape != (rows,) or not b.is_contiguous():
        raise _NotPlain
    return w.data_ptr(), b.data_ptr()


def _norm(module, cols, device):
    if not _plain(module, RMSNorm):
        raise _NotPlain
    w = module._parameters.get("weight")
    if w is None or not module.elementwise_affine or w.dtype is not BF16 or w.device != device or \
            w.shape != (cols,) or not w.is_contiguous():
        raise _NotPlain
    return w.data_ptr()


def _pack_layer(layer, rope, hidden, device):
    """The sizes of a layer, and the fields of its struct fk_llama_layer."""
    if not _plain(layer, LlamaDecoderLayer):
        raise _NotPlain
    sub = layer._modules
    att, mlp, norm1, norm2 = (sub.get(n) for n in ("self_attn", "mlp", "input_layernorm",
                                                   "post_attention_layernorm"))
    if not (_plain(att, LlamaAttention) and _plain(mlp, LlamaMLP) and att.fused and mlp.fused_act):
        raise _NotPlain
    s = att._modules
    cache, act = s.get("attn"), mlp._modules.get("act_fn")
    if s.get("rotary_emb") is not rope or not _plain(cache, Attention) or \
            not _plain(act, SiluAndMul):
        raise _NotPlain
    hq, hkv, d, layout = att.num_heads, att.num_kv_heads, att.head_dim, cache.kv_layout
    kc, vc = cache.k_cache, cache.v_cache
    prefill = cache._modules.get("prefill_op")
    if (cache.num_heads, cache.num_kv_heads, cache.head_size) != (hq, hkv, d) or \
            not _plain(prefill, _PREFILL[layout]) or kc.dim() != 4 or kc.dtype is not BF16 or \
            vc.dtype is not BF16 or kc.device != device or vc.device != device or \
            kc.shape != vc.shape or not (kc.is_contiguous() and vc.is_contiguous()):
        raise _NotPlain
    if layout == "HND":
        blocks, heads, page, dim = kc.shape
    else:
        blocks, page, heads, dim = kc.shape
    if (heads, dim) != (hkv, d) or kc.numel() == 0 or prefill.num_kv_heads != hkv or \
            (prefill.num_heads if layout == "NHD" else prefill.num_qo_heads) != hq:
        raise _NotPlain
    if prefill._status is None:
        prefill._status = ops.new_status(device)
    gate_up = mlp._modules.get("gate_up_proj")
    ff = gate_up._parameters["weight"].shape[0] // 2
    qk = [0, 0]
    for i, n in enumerate(("q_norm", "k_norm")):
        if s.get(n) is not None:
            qk[i] = _norm(s[n], d, device)
        elif getattr(att, n, None) is not None:
            raise _NotPlain
    o, down = s.get("o_proj"), mlp._modules.get("down_proj")
    for m in (o, down):
        if m.__dict__.get("tp_size") != 1:
            raise _NotPlain
    return (hq, hkv, d, ff, layout, blocks, page, kc.stride(0)), (
        _norm(norm1, hidden, device),
        *_linear(s.get("qkv_proj"), QKVParallelLinear, (hq + 2 * hkv) * d, hidden, device), *qk,
        *_linear(o, RowParallelLinear, hidden, hq * d, device), _norm(norm2, hidden, device),
        *_linear(gate_up, MergedColumnParallelLinear, 2 * ff, hidden, device),
        *_linear(down, RowParallelLinear, hidden, ff, device),
        kc.data_ptr(), vc.data_ptr(), prefill._status.data_ptr(),
        norm1.eps, att.rms_norm_eps, norm2.eps, cache.scale)


def _plain_int32(t) -> bool:
    return type(t) is torch.Tensor and t.dtype is torch.int32 and t.is_cuda


class PromptRun:
    """One forward of a prompt portion.  `begin` returns None where no layer can go this way."""

    @classmethod
    def begin(cls, rope, hidden, positions):
        ctx = get_context()
        if type(hidden) is not torch.Tensor or not hidden.is_cuda or hidden.dim() != 2 or \
                hidden.shape[0] == 0 or torch.is_grad_enabled() or \
                torch.compiler.is_compiling() or not getattr(ctx, "is_prefill", False) or \
                getattr(ctx, "is_mixed", False) or getattr(ctx, "is_tree_verify", False) or \
                _tp_size() != 1 or get_tp_comm() is not None or _module._has_any_global_hook():
            return None
        table, cu_q, cu_k = ctx.block_tables, ctx.cu_seqlens_q, ctx.cu_seqlens_k
        if type(positions) is not torch.Tensor or not positions.is_cuda or \
                positions.dtype is not torch.int64 or not positions.is_contiguous() or \
                not _plain_int32(table) or table.dim() != 2 or table.stride(1) != 1 or \
                type(rope) is not RotaryEmbedding or not _OWN.isdisjoint(rope.__dict__) or \
                not all(_plain_int32(t) and t.is_contiguous()
                        for t in (ctx.slot_mapping, cu_q, cu_k)) or \
                cu_q.numel() != cu_k.numel() or \
                any(c.__dict__.get(n) is not f for c, n, f in _DEFINED):
            return None
        self = cls()
        self.rope, self.positions, self.ctx = rope, positions, ctx
        self.shape, self.device = hidden.shape, hidden.device
        self.sizes = None
        return self

    def _start(self, sizes) -> None:
        """Scratch that the layers share, and what of struct fk_llama_prompt is the same for all."""
        (m, width), device, ctx = self.shape, self.device, self.ctx
        hq, hkv, d, ff, layout, blocks, page, kv_stride = self.sizes = sizes
        # the MLP's forms in one launch; else the projection and the activation are two calls
        few = ops.gemm_silu_mul_fusable(m, 2 * ff, width)
        self.many = not few and m > ops.MANY_ROWS and (2 * ff) % 16 == 0 and width % 64 == 0
        self.fits = few or self.many
        if not self.fits:
            return
        self.scratch = [torch.empty((m, cols), dtype=BF16, device=device)
                        for cols in ((hq + 2 * hkv) * d, hq * d, ff)]
        cos_sin, ws = self.rope.activation_cache(BF16, device), ops.gemm_workspace(device)
        self.hold = cos_sin, ws
        table, cu_q = ctx.block_tables, ctx.cu_seqlens_q
        self.tail = struct.pack(
            "11Q15q", *(t.data_ptr() for t in self.scratch), self.positions.data_ptr(),
            cos_sin.data_ptr(), ctx.slot_mapping.data_ptr(), cu_q.data_ptr(),
            ctx.cu_seqlens_k.data_ptr(), table.data_ptr(), ws.data_ptr(),
            ops.default_status(device).data_ptr(), ws.numel() * ws.element_size(), m, width, ff,
            cos_sin.shape[0], blocks, page, kv_stride, int(layout == "HND"), table.stride(0),
            cu_q.numel() - 1, int(ctx.max_seqlen_q), hq, hkv, d)

    def layer(self, layer, hidden, residual):
        """(output, residual) as layer(positions, hidden, residual) returns them, or None."""
        for t in (hidden,) if residual is None else (hidden, residual):
            if type(t) is not torch.Tensor or t.dtype is not BF16 or t.shape != self.shape or \
                    t.device != self.device or not t.is_contiguous():
                return None
        try:
            sizes, fields = _pack_layer(layer, self.rope, self.shape[1], self.device)
        except (_NotPlain, AttributeError, KeyError):
            return None
        if self.sizes is None:
            self._start(sizes)
        if not self.fits or sizes != self.sizes or \
                (self.many and (fields[8] % 16 or fields[9] % 16)):      # gate_up and its bias
            return None
        first = residual is None
        if first:
            hidden, residual = torch.empty_like(hidden), hidden
        # objects that live until the call returns: it reads both structs between its launches, with
        # the interpreter's lock released, and a pointer made of a temporary holds nothing
        fields = struct.pack("15Q4d", *fields)
        prompt = struct.pack("2Q", residual.data_ptr(), hidden.data_ptr()) + self.tail
        _lib.check(_lib.lib.fk_llama_prompt_layers(fields, 1, int(first), prompt, ops._stream()),
                   "fk_llama_prompt_layers")
        return hidden, residual
