"""SwiGLU MLP: gate_up_proj -> SiluAndMul -> down_proj.
Drop-in for LlamaMLP (fastkernels/tasks/baseline/L2/llama_mlp.py:16-38)."""
from __future__ import annotations

import torch
import torch.nn as nn
from torch.nn.modules import module as _module

from fastkernels_b200 import _lib, ops
from fastkernels_b200.candidate.L1.silu_and_mul import SiluAndMul
from fastkernels_b200.candidate.L2.parallel_linear import (MergedColumnParallelLinear,
                                                            RowParallelLinear)
from fastkernels_b200.candidate import share_classes


class LlamaMLP(nn.Module):
    def __init__(self, config, quant_config: dict | None = None,
                 hidden_size: int | None = None, intermediate_size: int | None = None,
                 reduce_results: bool = True):
        super().__init__()
        h = hidden_size if hidden_size is not None else config.hidden_size
        i = intermediate_size if intermediate_size is not None else config.intermediate_size
        self.gate_up_proj = MergedColumnParallelLinear(h, [i] * 2, quant_config=quant_config)
        self.down_proj = RowParallelLinear(i, h, quant_config=quant_config,
                                           reduce_results=reduce_results)
        self.down_proj.comm_slot = 1
        self.act_fn = SiluAndMul()
        # build-only switch (not a reference argument): run gate_up + SiLU as one kernel
        self.fused_act = True

    def _stock(self, gu) -> bool:
        """Calling the projection and the activation as modules would run what they define and
        nothing else: no hooks, no replaced forward."""
        return type(gu) is MergedColumnParallelLinear and type(self.act_fn) is SiluAndMul and \
            not _module._has_any_global_hook() and \
            not any(m._forward_hooks or m._forward_pre_hooks or m._backward_hooks or
                    m._backward_pre_hooks or "forward" in m.__dict__ for m in (gu, self.act_fn))

    def forward(self, x):
        gu = self.gate_up_proj
        if (self.fused_act and x.dim() == 2 and x.is_cuda and x.dtype == torch.bfloat16
                and not torch.compiler.is_compiling()):
            # gate/up projection and SiLU-and-multiply in one launch (same rounding
            # points as the two ops)
            if ops.gemm_silu_mul_fusable(x.shape[0], gu.weight.shape[0], x.shape[1]):
                return self.down_proj(ops.gemm_silu_mul(x, gu.weight, gu.bias))
            # prompts: no module call is passed by that a program has hooked or replaced
            if ops.gemm_act_mul_many_fits(x, gu.weight, gu.bias) and self._stock(gu):
                return self.down_proj(ops.gemm_act_mul_many(x, gu.weight, _lib.ACT_SILU, gu.bias))
        return self.down_proj(self.act_fn(gu(x)))


share_classes(globals())
