"""Drop-in for the reference's operator module.

Mirrors ``models/dwoconv1d/dwoconv1d.py`` (and ``models/dwoconv1d_specialized/
dwoconv1d_specialized.py``, whose public surface is identical): the same
``DepthwiseOrientedConv1d(nn.Conv2d)`` constructor, ``forward`` / ``forward_safe``,
autograd contract and state-dict layout (``weight [C,1,1,K]``, ``bias [C]``,
``theta [C]`` or ``[C,1]``), so ``models/convnext.py`` can import it under the name
``dwoconv1d`` or ``dwoconv1d_specialized`` (see ``oriented1d_b200/compat``).

What differs underneath:

* kernels are prebuilt (``libo1d.so``); nothing is compiled in the constructor
  (reference: dwoconv1d.py:144-152 JIT-compiles one module per template tuple);
* NHWC inputs are convolved in place — no nhwc_to_nchw / nchw_to_nhwc round trips
  (reference: dwoconv1d.py:25-26,36-37,50-51,58-59);
* bias add and the ``w + resid`` identity tap are fused into the kernels
  (reference: dwoconv1d.py:22-23,34-35) and ``db`` comes out of the weight-gradient
  kernel (reference: dwoconv1d.py:66-67);
* any H x W is handled natively, so ``forward_safe`` does not pad to powers of two
  (reference: dwoconv1d.py:154-187); results are identical because the padding is zeros;
* float32 and bfloat16 activations (the reference is float32 only, dwoconv1d.py:144-146).
"""
from __future__ import annotations

import torch
import torch.nn as nn

from . import ops

__all__ = ["DepthwiseOrientedConv1d", "get_dwoconv1d_kernel", "oriented_dwconv1d_get_module_from_params"]


def _via_nhwc(x, plan, stride) -> bool:
    """Does an NCHW tensor go through its NHWC form?  Where that form has a fast path: converting it on
    the way in and out (two 128-bit transposes) costs far less than the general NCHW kernels, and the
    NHWC copy is what is kept for backward.  The reference does the opposite: it converts NHWC inputs
    to NCHW around NCHW-only kernels (dwoconv1d.py:25-26,36-37)."""
    if not x.is_cuda or x.dim() != 4:
        return False
    N, C, H, W = x.shape
    return (ops.uses_tiled(plan, N, H, W, stride, True, x.dtype)
            and not ops.uses_tiled(plan, N, H, W, stride, False, x.dtype))


class DepthwiseOrientedConv1d(nn.Conv2d):
    """Oriented 1D depthwise convolution (reference: dwoconv1d.py:92-198).

    ``angle`` is a scalar or a per-channel list in radians.  The kernels use
    ``pad = kernel_size // 2`` regardless of ``padding`` (reference: dwoconv1d.py:133,
    144-146); ``padding`` only lands in ``nn.Conv2d.padding``.
    """

    def __init__(self, in_channels, out_channels, kernel_size=3, *, groups=1, stride=1, padding=1,
                 bias=True, angle=0, nhwc=False, resid=False, arbitrary_size=False):
        super().__init__(in_channels, out_channels, (1, kernel_size), groups=groups, stride=stride,
                         padding=(0, padding), bias=bias)
        assert (isinstance(kernel_size, int) and in_channels == out_channels
                and groups == in_channels and kernel_size % 2 == 1)
        assert self.stride[0] == self.stride[1]

        if isinstance(angle, (float, int)):
            angle = torch.zeros((in_channels, 1)) + angle
        # same construction as the reference (dwoconv1d.py:128-131): python floats -> fp32
        self.theta = torch.nn.Parameter(torch.as_tensor(angle, dtype=torch.float32).clone()
                                        if isinstance(angle, torch.Tensor)
                                        else torch.tensor(angle, dtype=torch.float32))
        self.nhwc = nhwc
        self.add_identity = bool(resid)
        # Set by a caller whose input is a pre-activation tensor: forward then computes
        # conv(GELU(x)) with the GELU applied inside the kernels (the reference runs F.gelu as a
        # separate pass in front of its second block conv, models/convnext.py:389-391).  Not a
        # constructor argument: the reference's signature is kept as it is.  True: always inside
        # the kernels; "auto": inside the kernels where that saves time (large maps, which the
        # tiled kernels serve anyway), as a separate F.gelu pass elsewhere (small maps, where
        # the kernel families without activation-on-load are the faster ones).
        self.gelu_input = False
        # kept for parity with the reference attribute (dwoconv1d.py:136-141); the kernels
        # add the identity tap themselves and never read this tensor
        if resid:
            delta = torch.zeros_like(self.weight)
            delta[:, :, :, kernel_size // 2] = 1
            self.resid = delta
        else:
            self.resid = None
        # fp32 angles as constructed: rasterisation must not see a theta rounded by
        # .bfloat16()/.half() (bf16(pi/2) would move the end taps of a vertical line)
        self._angles_fp32 = self.theta.detach().clone().reshape(-1)
        self._plan = None
        self._plan_key = None
        self._plan_src = None
        if arbitrary_size:
            self.forward = self.forward_safe

    # -- plan cache -------------------------------------------------------------------
    def _get_plan(self) -> ops.Plan:
        th = self.theta
        # the key holds the tensor that backs the parameter: a new tensor swapped in through
        # `theta.data = ...` can then never reuse the old one's address while the plan lives
        key = (th._version, th.data_ptr(), th.dtype)
        if self._plan is None or key != self._plan_key or self._plan_src is not th.data.untyped_storage():
            self._plan_src = th.data.untyped_storage()
            if th.dtype == torch.float32:
                angles = th.detach().reshape(-1)
            else:
                kept = self._angles_fp32.to(th.device)
                same = torch.equal(kept.to(th.dtype), th.detach().reshape(-1))
                angles = kept if same else th.detach().reshape(-1).float()
            self._plan = ops.Plan(angles, self.kernel_size[1])
            self._plan_key = key
        return self._plan

    def _gelu_in_kernel(self, x) -> bool:
        """The "auto" rule: activation on load only on maps of 28x28 and larger that the tiled
        kernels, the only fast ones with an activation, can serve.  What it buys is memory (the GELU output is never stored, one 4*dim
        activation less per block kept for backward), not time: the tiled kernels are bound by
        instruction issue, so the erf costs more there than the memory pass it removes (B200,
        ConvNeXt-B-1D++ training step, batch 64: 60.3 ms unfused, 63.5 ms with this rule, 74.1 ms
        with the activation forced into every stage)."""
        if self.gelu_input != "auto":
            return bool(self.gelu_input)
        if not (x.is_cuda and x.dim() == 4 and self.nhwc and self.stride[0] == 1):
            return False
        N, H, W, _ = x.shape
        return H * W >= 28 * 28 and ops.gelu_uses_tiled(self._get_plan(), N, H, W, x.dtype)

    def _apply_op(self, x):
        gelu = self._gelu_in_kernel(x)
        if self.gelu_input and not gelu:
            x = torch.nn.functional.gelu(x)
        plan, stride = self._get_plan(), self.stride[0]
        via = not self.nhwc and not gelu and _via_nhwc(x, plan, stride)
        if torch.is_grad_enabled():          # the autograd node (reference: dwoconv1d.py:18-69) lives in native code
            return ops.ext.conv(x, self.weight, self.theta, self.bias, plan.host, plan.on(x.device), plan.C, plan.K, stride,
                                self.nhwc, via, self.add_identity, gelu)
        if via:
            return ops.nhwc_to_nchw(ops.fprop(ops.nchw_to_nhwc(x), self.weight, self.bias, plan, stride, True,
                                              self.add_identity))
        return ops.fprop(x, self.weight, self.bias, plan, stride, self.nhwc, self.add_identity, gelu)

    def forward_safe(self, x):
        """Any H x W; output extents ceil(H/stride) x ceil(W/stride) (dwoconv1d.py:154-187)."""
        return self._apply_op(x)

    def forward(self, x):
        h, w = (x.shape[1], x.shape[2]) if self.nhwc else (x.shape[2], x.shape[3])
        if h % self.stride[0] or w % self.stride[0]:
            # reference: TORCH_CHECK in kernels.cu:19-20
            raise RuntimeError("Invalid input size: H,W not divisible by stride")
        return self._apply_op(x)


# --------------------------------------------------------------------------------------
# The 5-callable "extension module" surface of the reference loader
# (dwoconv1d_kernel.py:30-35,76-90): fprop(x,w,theta), dgrad(dy,w,theta),
# wgrad(dy,x,theta), nhwc_to_nchw(x), nchw_to_nhwc(x) on contiguous NCHW tensors with
# (K, stride, pad) fixed at creation.  Kept so either implementation can be swapped
# under the reference's autograd function.
# --------------------------------------------------------------------------------------
class _KernelModule:
    def __init__(self, kernel_size: int, stride: int, pad: int):
        if pad != kernel_size // 2:
            raise ValueError("pad must equal kernel_size // 2")
        self.K, self.stride = int(kernel_size), int(stride)
        self._plans: dict = {}

    def _plan(self, theta) -> ops.Plan:
        """Plan of these angles.  A cache entry keeps the storage of the tensor it was built from
        alive, so the allocator cannot hand that address to a later tensor with other angles;
        a hit therefore means the same memory at the same version, i.e. the same values."""
        key = (theta.data_ptr(), theta._version, theta.numel())
        hit = self._plans.get(key)
        if hit is not None:
            return hit[1]
        if len(self._plans) > 64:
            self._plans.clear()
        p = ops.Plan(theta, self.K)
        self._plans[key] = (theta.detach().untyped_storage(), p)
        return p

    def fprop(self, x, w, theta):
        if x.shape[2] % self.stride or x.shape[3] % self.stride:
            raise RuntimeError("Invalid input size: H,W not divisible by stride")
        return ops.fprop(x, w, None, self._plan(theta), self.stride, False, False)

    def dgrad(self, dy, w, theta):
        return ops.dgrad(dy, w, self._plan(theta), dy.shape[2] * self.stride, dy.shape[3] * self.stride,
                         self.stride, False, False)

    def wgrad(self, dy, x, theta):
        return ops.wgrad(dy, x, self._plan(theta), self.stride, False, False)[0]

    nhwc_to_nchw = staticmethod(ops.nhwc_to_nchw)
    nchw_to_nhwc = staticmethod(ops.nchw_to_nhwc)


_modules: dict = {}


def get_dwoconv1d_kernel(ftype, kernel_size, stride, pad, Sb=None, verbose=False):
    """Same call as the reference loader (dwoconv1d_kernel.py:76-90); ``Sb`` (tap
    chunking for shared-memory size) has no meaning here and is ignored."""
    if ftype != "float":
        raise ValueError("ftype must be 'float'")
    key = (int(kernel_size), int(stride), int(pad))
    if key not in _modules:
        _modules[key] = _KernelModule(*key)
    return _modules[key]


def oriented_dwconv1d_get_module_from_params(ftype, kernel_size, stride, pad, Sb=None):
    """5-tuple as in dwoconv1d.py:72-80."""
    m = get_dwoconv1d_kernel(ftype, kernel_size, stride, pad, Sb=Sb)
    return (m.fprop, m.dgrad, m.wgrad, m.nhwc_to_nchw, m.nchw_to_nhwc)
