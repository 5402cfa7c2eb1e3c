"""The `linear` operator: one opaque op per fused EXL3 group with every row-count branch, dtype cast, pad and trim
inside, as the reference's cuda/src/sglang_exl3/runtime/ops.py:62-137 (0xSero/trellis-serve) does for its engines.

Same schema as the reference's custom op (ops.py:133):

    linear(Tensor x, Tensor[] trellis, Tensor[] suh, Tensor[] svh, Tensor[] dense, Tensor[] sliced, int sliced_min_rows,
           Tensor[] marlin_w, int[] marlin_ends, int[] codebooks, int[] out_widths) -> Tensor

registered as `torch.ops.exl3_b200.linear` (native: csrc/exl3_torch.cpp), with a fake (meta) implementation so tracing
compilers see only shapes.
`marlin_w` carries the output of `kernels.linear.prepare`: [packed, suh_cat, svh_cat]; `marlin_ends` its shard ends.
`trellis`, `suh`, `svh` (the stored tensors) are optional here: the resident layout alone serves every path.
`dense` may hold resident decoded fp16 weights per matrix; `sliced` is accepted for schema compatibility and unused.

Dispatch (there is a single backend, so the reference's ladder, ops.py:79-95, collapses to two paths):

  few rows                  fused decode kernel (up to 64: weights streamed once)
  many rows                 many-row path: the fused tcgen05 kernel (`kernels.linear.run_tc`: weights decoded once per
                            512 rows into the tensor-core operand); when resident decoded weights are passed in `dense`,
                            `dense_group` instead (batched input rotation, library fp16 GEMM on the resident weight,
                            output rotation), which is the reference's many-row sequence

x may have any leading dims; a last dim narrower than the stored (128-padded) k reads as zero-padded (ops.py:98-99) and
stored output columns beyond the true `out_widths` are dropped (ops.py:122-124), up to 64 rows without a copy for either.  fp16 / bf16 go through as they are;
any other dtype is computed in fp16 and cast back.
"""
from __future__ import annotations

import os
import sys
import types

import torch

from .. import _lib as _native_lib
from ..kernels import linear as lin

_ops = _native_lib.native()
_lib = torch.library.Library("exl3_b200", "FRAGMENT")       # must stay alive at module scope


class _Module(types.ModuleType):
    """Measurement knobs, module attributes that live in the native operator.

    DENSE_ROWS: row count from which the many-row path is taken; 0 = decide per call with `prefers_decode`.  PREFILL: "tc" = fused tcgen05 kernel; "library" = decode to fp16 + library GEMM (the reference's sequence), for
    comparisons."""

    @property
    def DENSE_ROWS(self) -> int:
        return _ops.knob(0, -1)

    @DENSE_ROWS.setter
    def DENSE_ROWS(self, rows: int) -> None:
        _ops.knob(0, int(rows))

    @property
    def PREFILL(self) -> str:
        return "library" if _ops.knob(1, -1) else "tc"

    @PREFILL.setter
    def PREFILL(self, path: str) -> None:
        _ops.knob(1, int(path == "library"))


sys.modules[__name__].__class__ = _Module
_ops.knob(0, int(os.environ.get("EXL3_B200_DENSE_ROWS", "0")))
_ops.knob(1, int(os.environ.get("EXL3_B200_PREFILL", "tc") == "library"))


def prefers_decode(rows: int, k: int, n_total: int, sms: int = 148) -> bool:
    """Whether a call goes through the decode kernel: up to 64 rows, one pass over the weights.  The sizes and the device's multiprocessor
    count `sms` are part of the interface; the rule does not look at them today."""
    return bool(_native_lib.load().exl3_prefers_decode(rows, k, n_total, sms))


def dense_group(x: torch.Tensor, packed: torch.Tensor, suh_cat: torch.Tensor, svh_cat: torch.Tensor, shard_ends: list[int],
                codebook: int, out: torch.Tensor, weights: list[torch.Tensor] | None = None) -> torch.Tensor:
    """Many-row (prefill) path of a fused group, the reference's `dense_group` (ops.py:36-59): ONE batched input
    rotation for all matrices, per matrix the decoded fp16 weight (resident `weights[i]`, or decoded now from the
    resident layout) times the rotated rows in an fp16 GEMM with fp32 accumulation, and an output rotation written
    straight into the matrix's column span of `out` in out's dtype."""
    rows = x.shape[0]
    xh = lin.had_in_group(x, suh_cat)
    bounds = [0, *shard_ends, svh_cat.shape[0]]
    for i, (a, b) in enumerate(zip(bounds[:-1], bounds[1:])):
        w = weights[i] if weights is not None else lin.reconstruct_packed(packed[a // 128:b // 128], codebook)
        y = torch.mm(xh[i * rows:(i + 1) * rows], w)
        del w
        lin.had_out_into(y, svh_cat[a:b], out, a)
    return out


def _dense_linear(h: torch.Tensor, dense: list[torch.Tensor], marlin_w: list[torch.Tensor], marlin_ends: list[int], codebook: int) -> torch.Tensor:
    """The branch of `linear` for resident decoded weights (`dense`) and for the library sequence."""
    packed, suh_cat, svh_cat = marlin_w
    y = torch.empty((h.shape[0], packed.shape[0] * 128), dtype=h.dtype, device=h.device)
    return dense_group(h, packed, suh_cat, svh_cat, list(marlin_ends), codebook, y, list(dense) if dense else None)


def _linear_fake(x, trellis, suh, svh, dense, sliced, sliced_min_rows, marlin_w, marlin_ends, codebooks, out_widths):
    return x.new_empty((*x.shape[:-1], sum(out_widths)))


_lib.define("dense_linear(Tensor h, Tensor[] dense, Tensor[] marlin_w, int[] marlin_ends, int codebook) -> Tensor")
_lib.impl("dense_linear", _dense_linear, "CUDA")
torch.library.register_fake("exl3_b200::linear", _linear_fake, lib=_lib)

_operator = torch.ops.exl3_b200.linear
_direct = _native_lib.direct().linear


def linear(*args, **kwargs):
    """`torch.ops.exl3_b200.linear`.  Plain eager calls (positional CUDA tensors, no gradients, no mode, tracer or profiler watching)
    skip the dispatcher, which is two thirds of the host time of a small call; everything else goes through it."""
    if not kwargs and not torch.compiler.is_compiling():
        y = _direct(*args)
        if y is not None:
            return y
    return _operator(*args, **kwargs)


linear.default = _operator.default
