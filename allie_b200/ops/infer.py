"""Bindings of the native inference schedule (``csrc/infer.cu``): one forward pass over a packed batch
whose last positions are the only outputs, and of the kernel that lays its results out for the host."""
from __future__ import annotations

import ctypes
from ctypes import c_float, c_int, c_longlong, c_void_p

import torch

from . import _lib
from ._lib import ptr, stream_ptr


class InferLayer(ctypes.Structure):
    """``AbInferLayer``."""
    _fields_ = [(n, c_void_p) for n in ("ln1_w", "ln1_b", "ln2_w", "ln2_b", "qkv_w", "qkv_b", "o_w", "o_b",
                                        "fc_w", "fc_b", "pr_w", "pr_b")]


class Infer(ctypes.Structure):
    """``AbInfer``."""
    _fields_ = ([(n, c_int) for n in ("n_layer", "d", "H", "hd", "F", "V", "rms")] + [("eps", c_float)]
                + [(n, c_void_p) for n in ("wte", "wpe", "ctrl", "lnf_w", "lnf_b", "wte_bf16", "wv", "bv", "wt", "bt")]
                + [(n, c_int) for n in ("n", "M", "T")]
                + [(n, c_void_p) for n in ("ids", "pos", "row0", "last", "x", "ln", "qkv", "att", "act", "x_last",
                                           "att_last", "h", "logits", "value", "time", "kc", "vc")]
                + [("kv_layer", c_longlong), ("S", c_int), ("max_ctas", c_int), ("status", c_void_p)])


def infer_last(args: Infer, layers) -> None:
    rc = _lib.cuda().ab_infer_last(ctypes.byref(args), layers, stream_ptr())
    if rc < 0:
        raise RuntimeError(f"ab_infer_last failed with code {rc} (n={args.n} M={args.M} T={args.T})")
    _lib.count_launches(rc)


def results_to_host(logits: torch.Tensor, value: torch.Tensor | None,
                    time: torch.Tensor | None) -> tuple[torch.Tensor, torch.Tensor, torch.Tensor]:
    """bf16 logits [n, V] and fp32 value and time [n] (zeros without them) as fp32 on the host, in one
    copy.  The status word comes along: raises if a wait of a kernel ran out before (what was computed
    behind such a kernel is not to be used)."""
    n, V = logits.shape
    assert logits.dtype == torch.bfloat16 and logits.is_contiguous()
    for t in (value, time):
        assert t is None or (t.dtype == torch.float32 and t.is_contiguous())
    out = torch.empty(n * (V + 2) + 1, dtype=torch.float32, device=logits.device)
    rc = _lib.cuda().ab_result_rows(ptr(logits), ptr(value), ptr(time), c_int(n), c_int(V), ptr(out),
                                    ptr(_lib.status_word()), stream_ptr())
    if rc != 0:
        raise RuntimeError(f"ab_result_rows failed with code {rc}")
    _lib.count_launches(1)
    host = out.cpu()
    _lib.raise_on_status(int(host.numpy()[-1:].view("int32")[0]))
    row = V + 2
    return host.as_strided((n, V), (row, 1)), host.as_strided((n,), (row,), V), host.as_strided((n,), (row,), V + 1)
