"""LayerNorm on the library's kernels (csrc/norm.cu) for half-precision CUDA activations.

``LayerNorm`` is a drop-in ``nn.LayerNorm`` (same parameters, same state-dict keys); inputs the kernels do not cover
(CPU, fp32, a normalised dimension above 2048 or not a multiple of 8, no affine parameters) take the torch path. The
models' transformer blocks normalise a ``[tokens, d_model]`` matrix twice each; forward and backward are one pass over
that matrix here; the backward kernel leaves partial weight / bias gradients, which a second small kernel adds. The autograd
function around them is C++ (csrc/torch_norm.cpp).
"""
from __future__ import annotations

import torch
import torch.nn as nn
import torch.nn.functional as F

from .. import native as N
from . import gemm as G

MAX_D = 2048


def supported(x: torch.Tensor, normalized_shape, weight) -> bool:
    d = x.shape[-1] if x.dim() else 0
    return (x.is_cuda and x.dtype in (torch.bfloat16, torch.float16) and weight is not None and weight.dtype == x.dtype
            and len(normalized_shape) == 1 and normalized_shape[0] == d and d % 8 == 0 and 8 <= d <= MAX_D and x.numel() > 0)


def layer_norm(x, normalized_shape, weight, bias, eps=1e-5):
    """``F.layer_norm`` that runs on the library's kernels where they apply."""
    if supported(x, tuple(normalized_shape), weight) and (bias is None or bias.dtype == x.dtype):
        return N.torch_module().layer_norm(x, weight, bias, G.Workspace.of(x).status, eps, G.DEFAULT_WAIT_NS)
    return F.layer_norm(x, normalized_shape, weight, bias, eps)


class LayerNorm(nn.LayerNorm):
    """``nn.LayerNorm`` whose forward and backward run on csrc/norm.cu for bf16 / fp16 CUDA inputs."""

    def forward(self, x):
        return layer_norm(x, self.normalized_shape, self.weight, self.bias, self.eps)
