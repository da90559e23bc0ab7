"""INT8 convolutions on the direct kernel, and 1x1 layers that the rule leaves to the GEMM kernel on single CTAs, bit for bit against the
GEMM kernel on pairs of CTAs: whole outputs, the last block of 16 channels and its padding too, on both sides of each line of the rules
between the kernels and of the epilogue's division, every result type."""
import pytest
import torch

import refutil as R

pytestmark = pytest.mark.gpu

DIRECT = [      # n, ic, oc, h, w, k, stride
    # 1x1: planes that no tile width divides, ragged channels, one and several tiles per CTA
    (32, 64, 256, 56, 56, 1, 1), (7, 96, 240, 31, 30, 1, 1), (20, 200, 600, 30, 30, 1, 1), (40, 32, 16, 1, 9, 1, 1), (9, 48, 80, 7, 7, 1, 1),
    (2, 1040, 1000, 1, 1, 1, 1),
    # 3x3: counts of column blocks that four does not divide, pairs, split K loops
    (3, 64, 16, 14, 14, 3, 1), (3, 64, 40, 14, 14, 3, 1), (2, 96, 80, 20, 17, 3, 1), (2, 64, 144, 14, 14, 3, 2), (1, 512, 272, 14, 14, 3, 1),
    (8, 256, 256, 14, 14, 3, 1), (24, 64, 64, 28, 28, 3, 1), (30, 96, 192, 60, 60, 3, 1), (64, 128, 256, 56, 56, 3, 2), (16, 128, 128, 56, 56, 3, 1),
    (20, 48, 48, 100, 100, 3, 1), (3, 62, 640, 99, 99, 3, 1),
    # around the lines of the sharing rule
    (16, 256, 1024, 14, 14, 1, 1), (42, 298, 128, 24, 24, 1, 1), (39, 119, 528, 14, 14, 1, 1), (3, 528, 192, 101, 107, 1, 1), (21, 656, 848, 15, 14, 1, 1),
    (18, 592, 305, 46, 49, 1, 1), (5, 176, 1439, 41, 41, 3, 1), (4, 128, 640, 41, 41, 3, 1), (5, 64, 16, 61, 52, 3, 1),
]
# the GEMM kernel is the faster one: resident filters of several channel groups
GEMM = [(9, 144, 32, 72, 114, 1, 1), (49, 149, 16, 41, 66, 1, 1), (12, 144, 16, 92, 92, 1, 1), (50, 432, 16, 41, 41, 1, 1), (5, 704, 30, 32, 32, 1, 1),
        (1, 144, 48, 15, 13, 1, 1)]


@pytest.mark.parametrize("shape", DIRECT + GEMM, ids=str)
@pytest.mark.parametrize("types,total", [("u8f32u8f32", False), ("u8f32u8f32", True), ("u8f32s8f32", False), ("u8f32f32f32", False)])
def test_whole_outputs(pkg, shape, types, total, monkeypatch):
    import gpuutil as G
    n, ic, oc, h, w, k, stride = shape
    case = R.ConvCase("whole", n, ic, oc, h, w, kh=k, kw=k, pad=k // 2, stride=stride, types=types, algo="1x1" if k == 1 else "direct",
                      relu=types == "u8f32u8f32", bias=True, sum=total, oscale=2.0 if k == 1 else 8.0)
    E = G.package()
    g = torch.Generator(device="cuda").manual_seed(n * 1000 + ic)
    x = torch.randint(0, 256, (n, (ic + 15) // 16, h, w, 16), generator=g, device="cuda", dtype=torch.uint8)
    got = {}
    for pairs in (False, True):
        if pairs:
            monkeypatch.setenv("ELB_I8_CTA2", "1")
        d = G.make_desc(case)
        assert d.setup() == 0, E.last_error()
        assert (d.launched_kernel == "conv_halo") == (not pairs and shape in DIRECT)
        gw = torch.Generator(device="cuda").manual_seed(7)
        wt = torch.randn(d.sizes.weights, generator=gw, device="cuda") * 0.1
        b = torch.randn(d.sizes.bias, generator=gw, device="cuda")
        y = torch.arange(d.byte_sizes.output, device="cuda").remainder(251).to(torch.uint8)      # (the residual, where it is added)
        assert d.prepare(wt, b) == 0 and d.enqueue(y, x) == 0, E.last_error()
        torch.cuda.synchronize()
        assert d.device_status() == 0
        got[pairs] = y
        d.close()
    assert torch.equal(got[False], got[True])
