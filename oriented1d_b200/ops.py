"""torch-facing wrappers of the C ABI: tensors in, tensors out.

torch is used for device memory (its caching allocator owns every buffer) and for the
current stream; all arithmetic happens in libo1d.so, reached through csrc/o1d_torch.cpp (checks,
allocation, stream and call in native code).  There is no CPU path: every
function raises on a non-CUDA tensor, as the reference's extension does
(CHECK_CUDA, models/dwoconv1d/kernels/kernels.cu:11).
"""
from __future__ import annotations

import numpy as np
import torch

from . import _lib
from ._lib import ext, lib, check

# kernels launched by one call of each entry point (used by the benchmark's launch count)
KERNELS_PER_CALL = {"fprop": 1, "dgrad": 1, "wgrad": 2, "transpose": 1}

_DTYPES = {torch.float32: _lib.F32, torch.bfloat16: _lib.BF16}


def offsets(theta, K: int):
    """Rasterised tap offsets (dh, dw), int8 arrays [C, K], from fp32 angles
    (reference rule: models/dwoconv1d_reference/kernels/kernels.cpp:37,43-44)."""
    th = np.ascontiguousarray(np.asarray(theta, dtype=np.float32).reshape(-1))
    C = th.shape[0]
    dh = np.empty((C, K), np.int8)
    dw = np.empty((C, K), np.int8)
    check(lib.o1d_offsets(th.ctypes.data, C, K, dh.ctypes.data, dw.ctypes.data), "o1d_offsets")
    return dh, dw


class Plan:
    """Per-layer tap table (orientation classes) on the host plus one copy per device."""

    def __init__(self, theta, K: int):
        th = torch.as_tensor(theta).detach().to(device="cpu", dtype=torch.float32).reshape(-1).contiguous()
        self.C, self.K = int(th.numel()), int(K)
        nbytes = lib.o1d_plan_bytes(self.C, self.K)
        if nbytes == 0:
            raise ValueError("o1d_plan_bytes: invalid C or K")
        self.host = torch.zeros(nbytes, dtype=torch.uint8)
        check(lib.o1d_plan_build(th.data_ptr(), self.C, self.K, self.host.data_ptr()), "o1d_plan_build")
        self.num_classes = lib.o1d_plan_num_classes(self.host.data_ptr())
        self._dev: dict[torch.device, torch.Tensor] = {}

    def on(self, device: torch.device) -> torch.Tensor:
        d = self._dev.get(device)
        if d is None:
            d = self.host.to(device)
            self._dev[device] = d
        return d

    def pointers(self, t: torch.Tensor):
        """Addresses of the two copies for a call on t's device ((0, 0) when t is not on one: the
        call then reports what is wrong with its arguments).  Taken from the tensors at each call:
        a copy of a plan has tensors of its own, and an address kept beside them would still name
        the original's."""
        if not t.is_cuda:
            return 0, 0
        return self.host.data_ptr(), self.on(t.device).data_ptr()


def fprop(x, w, bias, plan: Plan, stride: int = 1, nhwc: bool = False, add_identity: bool = False,
          gelu_input: bool = False):
    """y = oriented conv of x.  x: [N,C,H,W] (or [N,H,W,C] if nhwc), contiguous.  gelu_input: x is a
    pre-activation tensor and exact GELU is applied as it is loaded, y = conv(GELU(x))."""
    return ext.fprop(x, w, bias, plan.C, plan.K, *plan.pointers(x), stride, bool(nhwc), bool(add_identity), bool(gelu_input))


def dgrad(dy, w, plan: Plan, H: int, W: int, stride: int = 1, nhwc: bool = False,
          add_identity: bool = False, pre=None):
    """dx [.., H, W ..] from dy [.., ceil(H/s), ceil(W/s) ..].  pre (shape of dx): the forward pass was
    conv(GELU(pre)); the result is then the gradient with respect to pre (times GELU'(pre))."""
    return ext.dgrad(dy, w, plan.C, plan.K, *plan.pointers(dy), H, W, stride, bool(nhwc), bool(add_identity), pre)


def wgrad(dy, x, plan: Plan, stride: int = 1, nhwc: bool = False, with_bias: bool = False,
          gelu_input: bool = False, out_dtype: torch.dtype = torch.float32):
    """(dw [C,1,1,K], db [C] or None) in `out_dtype`.  Deterministic.  gelu_input: x is the pre-activation
    tensor of a forward pass conv(GELU(x))."""
    bf16 = out_dtype == torch.bfloat16
    dw, db = ext.wgrad(dy, x, plan.C, plan.K, *plan.pointers(x), stride, bool(nhwc), bool(with_bias), bool(gelu_input), bf16)
    if not bf16 and out_dtype != torch.float32:
        dw, db = dw.to(out_dtype), None if db is None else db.to(out_dtype)
    return dw, db


def nhwc_to_nchw(x):
    """[N,H,W,C] -> [N,C,H,W], contiguous (reference: kernels.cu:56-61)."""
    return ext.transpose(x, False)


def nchw_to_nhwc(x):
    """[N,C,H,W] -> [N,H,W,C], contiguous (reference: kernels.cu:63-68)."""
    return ext.transpose(x, True)


def layer_norm_cl(x, weight, bias, eps: float = 1e-6, gelu: bool = False):
    """LayerNorm over the last (contiguous) axis, optionally fused with exact GELU.  Forward
    only (no autograd): for inference and for callers that handle gradients themselves."""
    return ext.layer_norm_cl(x, weight, bias, float(eps), bool(gelu))


def layer_norm_cl_supported(x, gelu: bool = False, backward: bool = False) -> bool:
    """Can layer_norm_cl (and, with backward=True, layer_norm_cl_bwd) take this tensor?"""
    if not (x.is_cuda and x.dtype in (torch.float32, torch.bfloat16)):
        return False
    C, ve = x.shape[-1], (4 if x.dtype == torch.float32 else 8)
    if backward:
        return C % ve == 0 and C // ve <= 128
    return C % ve == 0 and C <= 1024


def layer_norm_cl_bwd(x, dy, weight, eps: float = 1e-6, bias=None, gelu: bool = False):
    """Gradients of layer_norm_cl: dx in x's dtype, dweight and dbias in fp32.  With gelu=True the
    forward call ended in exact GELU and `bias` is needed again.  The statistics are recomputed
    from x; dweight / dbias are summed in a fixed order."""
    return ext.layer_norm_cl_bwd(x, dy, weight, float(eps), bias, bool(gelu), False)


class LayerNormCL:
    """Channels-last LayerNorm with this library's kernels on both passes (F.layer_norm and its
    autograd backward in the reference, models/convnext.py:28-56).  The node lives in native code."""

    @staticmethod
    def apply(x, weight, bias, eps, gelu=False):
        return ext.layer_norm_train(x, weight, bias, float(eps), bool(gelu))


def colsum(x):
    """Sum over all but the last (contiguous) axis, in fp32 and in a fixed order: [..., C] -> [C]."""
    return ext.colsum(x, False)


class LinearCL:
    """F.linear on channels-last activations whose bias gradient is this library's column sum
    (autograd's own is a generic reduction that runs at a fifth of the memory rate on these
    shapes); the two matrix products stay with the GEMM library, as in nn.Linear."""

    @staticmethod
    def apply(x, weight, bias):
        return torch.nn.functional.linear(x, weight) if bias is None else ext.linear_train(x, weight, bias)


def linear_cl(module, x):
    """module(x) for an nn.Linear; on CUDA with gradients enabled the bias gradient runs here."""
    C = module.out_features
    if (x.is_cuda and torch.is_grad_enabled() and module.bias is not None and x.dtype == module.weight.dtype
            and x.dtype in (torch.float32, torch.bfloat16) and C % (4 if x.dtype == torch.float32 else 8) == 0):
        return LinearCL.apply(x, module.weight, module.bias)
    return module(x)


def pointwise_in(x, weight, bias):
    """Channels-last ``Linear`` over the few channels of an NCHW image: x [N,Cin,H,W] (Cin <= 4),
    weight [Cout,Cin], bias [Cout] or None -> [N,H,W,Cout] (models/convnext.py:143,170-176 in one
    pass).  Forward only."""
    return ext.pointwise_in(x, weight, bias)


def uses_tiled(plan: Plan, N: int, H: int, W: int, stride: int, nhwc: bool, dtype: torch.dtype) -> bool:
    """Would this request run on one of the TMA-staged families (tiled, direct, segments; True) or on the
    general kernels (False)?"""
    code = _DTYPES.get(dtype)
    if code is None:
        return False
    return bool(lib.o1d_uses_tiled(plan.host.data_ptr(), N, H, W, plan.C, plan.K, stride, int(nhwc), code))


def gelu_uses_tiled(plan: Plan, N: int, H: int, W: int, dtype: torch.dtype) -> bool:
    """Would conv(GELU(x)) with the GELU applied on load (NHWC, stride 1) run on the tiled kernels (True)
    or the general ones (False)?  No other family applies an activation."""
    code = _DTYPES.get(dtype)
    if code is None:
        return False
    return bool(lib.o1d_gelu_uses_tiled(plan.host.data_ptr(), N, H, W, plan.C, plan.K, code))


def set_route(route) -> None:
    """Testing aid.  False/0: automatic choice; True/1: general kernels only; 2: prefer the
    tiled kernels; 3: prefer the direct kernels; 4: the whole-line kernels; 5: the walker kernels
    (these two serve square fp32 NHWC stage maps only and fall through elsewhere); 6: the segment
    kernels, on 7x7 maps too."""
    check(lib.o1d_set_route(int(route)), "o1d_set_route")


ROUTE_NAMES = {-1: "none", 0: "general", 1: "tiled", 2: "direct", 3: "plane7", 4: "lines", 5: "walk", 6: "segments"}


def last_route() -> str:
    """Kernel family that served this thread's last fprop / dgrad / wgrad call."""
    return ROUTE_NAMES[lib.o1d_last_route()]


def device_status(device=None, clear: bool = False) -> int:
    """Device-side failure flag (0 = healthy).  Synchronises the device.  ``clear`` resets it."""
    import ctypes
    flag = ctypes.c_int(0)
    with torch.cuda.device(device if device is not None else torch.cuda.current_device()):
        if clear:
            check(lib.o1d_device_status_clear(ctypes.byref(flag)), "o1d_device_status_clear")
        else:
            check(lib.o1d_device_status(ctypes.byref(flag)), "o1d_device_status")
    return flag.value
