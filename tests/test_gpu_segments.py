"""Segment kernels (csrc/o1d_seg.cuh): sizes around the edges of their blocks, lanes and tiles, against
the general kernels on the same device inputs."""
import math

import pytest
import torch

import oriented1d_b200 as o1d
from tests.util import angle_list

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _plan(mode, C, K):
    return o1d.Plan([math.pi * int(mode[3:]) / 8] * C if mode.startswith("one") else angle_list(mode, C), K)


# N, H, W, C, K, angles: one pixel, one row, blocks of 14 / 28 positions and 3 x 8 / 14 x diagonal blocks with and
# without remainder, several images per item, a last item with fewer, channels that do not fill a chunk, pairs of
# channels on two lines, maps cut along either axis
SHAPES = [(1, 1, 1, 16, 31, "one2"), (3, 1, 29, 16, 31, "one1"), (2, 30, 1, 8, 15, "one6"), (5, 13, 15, 64, 31, "model"),
          (4, 14, 28, 24, 27, "one7"), (2, 29, 27, 64, 31, "model+"), (17, 10, 9, 40, 7, "model"), (2, 57, 56, 32, 31, "one5"),
          (1, 56, 57, 96, 31, "model"), (2, 61, 120, 48, 31, "model+"), (1, 130, 35, 64, 13, "model"), (1, 210, 333, 16, 31, "one3"),
          (1, 99, 301, 16, 31, "one6"), (1, 300, 301, 8, 31, "one4")]


# buffers refilled many times while the warps are at different items: lines of unequal cost in one chunk, two
# buffers and four, whole images and cut ones
SHAPES += [(2500, 28, 14, 32, 31, "model+"), (900, 32, 33, 16, 31, "model"), (24, 150, 150, 48, 31, "model+")]
# more chunks than a third of the CTAs: a CTA goes from one cut of the map, and size of the buffers, to another
SHAPES += [(2, 30, 61, 2048, 31, "model"), (3, 28, 100, 1536, 31, "model")]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16], ids=["f32", "bf16"])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_segments_equal_general(shape, dtype):
    got = check_against_general(*shape, dtype, route=6)
    assert got == ("segments", "segments")


# where the segment kernels come first, where behind another family, and where before the general kernels only
# (forward, weight gradient)
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16], ids=["f32", "bf16"])
@pytest.mark.parametrize("shape,families", [
    ((3, 9, 9, 64, 31, "model"), ("segments", "segments")), ((3, 8, 9, 64, 31, "model"), ("segments", "segments")),
    ((3, 8, 8, 128, 31, "model"), ("segments", "direct")), ((1, 7, 8, 128, 31, "model"), ("segments", "direct")),
    ((513, 6, 6, 64, 31, "model"), ("direct", "direct")), ((256, 5, 5, 128, 15, "model"), ("direct", "direct")),
    ((511, 6, 6, 64, 31, "model"), ("direct/segments", "direct")),           # fp32 / bf16
    ((1024, 1, 1, 32, 31, "one2"), ("direct", "direct")), ((3, 7, 7, 64, 31, "model"), ("plane7", "plane7")),
    ((600, 6, 6, 72, 31, "model"), ("direct/segments", "direct/segments")),  # channels that the bf16 direct kernels refuse
    ((296, 56, 56, 32, 31, "model"), ("tiled", "tiled")), ((295, 56, 56, 32, 31, "model"), ("segments", "segments")),
    ((170, 56, 56, 56, 31, "model"), ("tiled", "tiled")), ((200, 56, 56, 48, 31, "model"), ("segments", "segments")),
    ((240, 28, 28, 40, 31, "model"), ("segments", "segments")), ((300, 40, 60, 32, 31, "model"), ("segments", "segments")),
], ids=lambda s: "x".join(map(str, s)) if isinstance(s, tuple) and len(s) == 6 else "")
def test_place_among_the_families(shape, families, dtype):
    got = check_against_general(*shape, dtype, route=0)
    assert got == tuple(f.split("/")[-1 if dtype == torch.bfloat16 else 0] for f in families)


def check_against_general(N, H, W, C, K, mode, dtype, route):
    """Forward, input gradient and weight gradient of both; the families that served forward and weight gradient."""
    g = torch.Generator(device=DEV).manual_seed(H * W + C)
    x = torch.randn((N, H, W, C), generator=g, device=DEV).to(dtype)
    dy = torch.randn((N, H, W, C), generator=g, device=DEV).to(dtype)
    w = 0.1 * torch.randn((C, 1, 1, K), generator=g, device=DEV)
    bias = torch.randn((C,), generator=g, device=DEV)
    plan = _plan(mode, C, K)

    def run(route):
        try:
            o1d.ops.set_route(route)
            out = (o1d.fprop(x, w, bias, plan, 1, True, True),)
            names = o1d.ops.last_route()
            out += (o1d.dgrad(dy, w, plan, H, W, 1, True),)
            assert o1d.ops.last_route() == names
            out += o1d.wgrad(dy, x, plan, 1, True, True)
            return out, (names, o1d.ops.last_route())
        finally:
            o1d.ops.set_route(0)

    ref, _ = run(1)
    got, names = run(route)
    assert o1d.ops.device_status() == 0
    for a, b in zip(got[:2], ref[:2]):
        a, b = a.float(), b.float()
        if dtype == torch.float32:
            assert float((a - b).abs().max()) <= 1e-5 * float(b.abs().max())
        else:                                    # both round an fp32 sum: at most one bf16 ulp apart
            assert float(((a - b).abs() / b.abs().clamp_min(1e-2)).max()) <= 2 ** -7
    for a, b in zip(got[2:], ref[2:]):
        assert float((a - b).abs().max()) <= 1e-4 * float(b.abs().max())
    again = run(route)[0]
    assert all(torch.equal(a, b) for a, b in zip(got, again))        # same bits again
    return names


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16], ids=["f32", "bf16"])
@pytest.mark.parametrize("shape", [(5, 13, 15, 64, 31, "model"), (2, 29, 27, 40, 15, "model+"), (1, 56, 57, 96, 31, "model"),
                                   (2, 30, 61, 2048, 31, "model")], ids=lambda s: "x".join(map(str, s)))
def test_parameters_read_and_written_as_bf16(shape, dtype):
    """bf16 weights and biases go to the kernels as they are stored: the bits of a call with the same values in
    fp32, and gradients that are its fp32 ones rounded."""
    from oriented1d_b200 import _lib
    N, H, W, C, K, mode = shape
    g = torch.Generator(device=DEV).manual_seed(C)
    x, dy = (torch.randn((N, H, W, C), generator=g, device=DEV).to(dtype) for _ in range(2))
    w = (0.1 * torch.randn((C, 1, 1, K), generator=g, device=DEV)).to(torch.bfloat16)
    bias = torch.randn((C,), generator=g, device=DEV).to(torch.bfloat16)
    plan = _plan(mode, C, K)
    want = (o1d.fprop(x, w.float(), bias.float(), plan, 1, True, True), o1d.dgrad(dy, w.float(), plan, H, W, 1, True))
    want += tuple(t.to(torch.bfloat16) for t in o1d.wgrad(dy, x, plan, 1, True, True))
    # through the C ABI, which does not convert: these requests are served as they are
    y, dx = torch.empty_like(x), torch.empty_like(x)
    dw, db = torch.empty_like(w), torch.empty_like(bias)
    host, dev = plan.pointers(x)
    code, flag, st = (_lib.F32 if dtype == torch.float32 else _lib.BF16), 4, torch.cuda.current_stream().cuda_stream
    size = _lib.lib.o1d_wgrad_workspace_bytes(N, H, W, C, K, 1, _lib.NHWC, code)
    ws = torch.empty(size, dtype=torch.uint8, device=DEV)
    sizes = (N, H, W, C, K, 1, _lib.NHWC, code)
    calls = (lambda: _lib.lib.o1d_fprop(x.data_ptr(), w.data_ptr(), bias.data_ptr(), host, dev, y.data_ptr(), *sizes, _lib.FLAG_IDENTITY | flag, st),
             lambda: _lib.lib.o1d_dgrad(dy.data_ptr(), w.data_ptr(), host, dev, dx.data_ptr(), *sizes, flag, st),
             lambda: _lib.lib.o1d_wgrad_act(dy.data_ptr(), x.data_ptr(), host, dev, dw.data_ptr(), db.data_ptr(), ws.data_ptr(), size, *sizes, flag, st))
    for call in calls:
        _lib.check(call(), "segments with bf16 parameters")
        assert o1d.ops.last_route() == "segments"
    assert o1d.ops.device_status() == 0
    assert all(torch.equal(a, b) for a, b in zip((y, dx, dw, db), want))
    # and through the wrappers
    got = (o1d.fprop(x, w, bias, plan, 1, True, True), o1d.dgrad(dy, w, plan, H, W, 1, True))
    got += o1d.wgrad(dy, x, plan, 1, True, True, out_dtype=torch.bfloat16)
    assert all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("shape,served", [((600, 6, 6, 64, 31, "model"), True), ((3, 8, 8, 64, 31, "model"), True), ((296, 56, 56, 32, 31, "model"), True),
                                          ((3, 7, 7, 72, 31, "model"), False), ((3, 6, 6, 64, 31, "random"), False)],
                         ids=lambda s: "x".join(map(str, s)) if isinstance(s, tuple) else "")
def test_bf16_parameters_where_another_family_comes_first(shape, served):
    """A caller that cannot convert its parameters is served wherever the segment kernels take the layer; one
    that can is told where to."""
    from oriented1d_b200 import _lib
    N, H, W, C, K, mode = shape
    torch.manual_seed(C)
    x, dy = (torch.randn((N, H, W, C), device=DEV).to(torch.bfloat16) for _ in range(2))
    w = (0.1 * torch.randn((C, 1, 1, K), device=DEV)).to(torch.bfloat16)
    plan = _plan(mode, C, K)
    host, dev = plan.pointers(x)
    sizes, st = (N, H, W, C, K, 1, _lib.NHWC, _lib.BF16), torch.cuda.current_stream().cuda_stream
    size = _lib.lib.o1d_wgrad_workspace_bytes(*sizes)
    ws = torch.empty(size, dtype=torch.uint8, device=DEV)
    y, dw = torch.empty_like(x), torch.empty_like(w)

    def wgrad(flags):
        return _lib.lib.o1d_wgrad_act(dy.data_ptr(), x.data_ptr(), host, dev, dw.data_ptr(), None, ws.data_ptr(), size, *sizes, flags, st)

    rc = _lib.lib.o1d_fprop(x.data_ptr(), w.data_ptr(), None, host, dev, y.data_ptr(), *sizes, 4, st), wgrad(4)
    assert rc == ((0, 0) if served else (2, 2)) and wgrad(4 | 8) == 2
    if served:
        assert float((y.float() - o1d.fprop(x, w, None, plan, 1, True).float()).abs().max()) <= 2 ** -7 * float(y.float().abs().max())
        a, b = dw.float(), o1d.wgrad(dy, x, plan, 1, True)[0]
        assert float((a - b).abs().max()) <= 2 ** -8 * float(b.abs().max())
        assert o1d.ops.device_status() == 0


def test_nchw_module_of_odd_channel_groups():
    """An NCHW bf16 layer whose channels do not fill groups of 32 bytes: the segment kernels behind two
    layout steps, with the results of the general NCHW kernels."""
    N, C, H, W, K = 3, 40, 20, 30, 31
    m = o1d.DepthwiseOrientedConv1d(C, C, K, groups=C, padding=K // 2, angle=[float(a) for a in angle_list("model", C)]).to(DEV, torch.bfloat16)
    with torch.no_grad():
        m.weight.mul_(0.3)
    x, dy = (torch.randn((N, C, H, W), device=DEV).to(torch.bfloat16) for _ in range(2))

    def run(conv):
        y = conv(x)
        return (y, o1d.ops.last_route()) + torch.autograd.grad(y, (xr, m.weight, m.bias), dy)

    xr = x.requires_grad_(True)
    y, name, dx, dw, db = run(m)
    assert name == "segments" and o1d.ops.device_status() == 0
    try:
        o1d.ops.set_route(1)
        ry, rname, rdx, rdw, rdb = run(m)
    finally:
        o1d.ops.set_route(0)
    assert rname == "general"
    for a, b in ((y, ry), (dx, rdx), (dw, rdw), (db, rdb)):      # each rounds an fp32 sum: at most one bf16 ulp apart
        a, b = a.detach().float(), b.detach().float()
        assert float(((a - b).abs() / b.abs().clamp_min(1e-2 * float(b.abs().max()))).max()) <= 2 ** -7


# bf16 sums have the bits of the family that the shape would otherwise take (2: tiled, 3: direct)
@pytest.mark.parametrize("shape,family", [((2, 56, 56, 96, 31), 2), ((8, 28, 28, 96, 31), 2), ((64, 28, 28, 96, 31), 2), ((3, 28, 28, 192, 31), 3),
                                          ((33, 14, 14, 384, 31), 3), ((5, 24, 24, 192, 31), 2), ((1, 13, 29, 32, 15), 3)],
                         ids=lambda s: "x".join(map(str, s)) if isinstance(s, tuple) else str(s))
def test_bits_of_the_family_replaced(shape, family):
    N, H, W, C, K = shape
    torch.manual_seed(H * C)
    x = torch.randn((N, H, W, C), device=DEV).to(torch.bfloat16)
    w, bias = 0.1 * torch.randn((C, 1, 1, K), device=DEV), torch.randn((C,), device=DEV)
    plan = _plan("model", C, K)

    def run(route):
        try:
            o1d.ops.set_route(route)
            return o1d.fprop(x, w, bias, plan, 1, True, True), o1d.dgrad(x, w, plan, H, W, 1, True)
        finally:
            o1d.ops.set_route(0)

    got, other = run(0), run(5 - family)
    assert all(torch.equal(a, b) for a, b in zip(got, run(family)))
    # the other order shows: a few sums in a hundred thousand round to the other side
    assert H * W < 400 or not all(torch.equal(a, b) for a, b in zip(got, other))


# maps of which the direct kernels' tile holds two images, but not of a batch of one
@pytest.mark.parametrize("H,W,C,K,mode", [(8, 8, 1536, 31, "one1"), (14, 14, 1536, 15, "one1"), (16, 16, 768, 15, "one2"), (14, 14, 64, 7, "model")])
def test_an_image_does_not_depend_on_its_batch(H, W, C, K, mode):
    torch.manual_seed(H * C)
    x = torch.randn((33, H, W, C), device=DEV).to(torch.bfloat16)
    w, bias = 0.1 * torch.randn((C, 1, 1, K), device=DEV), torch.randn((C,), device=DEV)
    plan = _plan(mode, C, K)

    def run(t):
        out = o1d.fprop(t, w, bias, plan, 1, True, True), o1d.dgrad(t, w, plan, H, W, 1, True)
        assert o1d.ops.last_route() == "segments"
        return out

    whole = run(x)
    for i in (0, 7, 32):
        assert all(torch.equal(a[i:i + 1], b) for a, b in zip(whole, run(x[i:i + 1].contiguous())))
