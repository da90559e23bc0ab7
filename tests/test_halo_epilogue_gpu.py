"""INT8 direct convolutions whose epilogue warps share each tile (a quarter of the column blocks per group): counts of blocks that
four does not divide, one and several tiles per CTA, pairs, split K loops and tiles below the sharing rule, bit for bit against the
GEMM kernel on pairs of CTAs, which none of this touches."""
import pytest
import torch

import refutil as R

pytestmark = pytest.mark.gpu

SHAPES = [      # n, ic, oc, h, w, k, stride
    (3, 64, 16, 14, 14, 3, 1), (3, 64, 40, 14, 14, 3, 1), (2, 96, 80, 20, 17, 3, 1), (2, 64, 144, 14, 14, 3, 2), (1, 512, 272, 14, 14, 3, 1),
    (8, 256, 256, 14, 14, 3, 1), (16, 256, 1024, 14, 14, 1, 1), (24, 64, 64, 28, 28, 3, 1), (30, 96, 192, 60, 60, 3, 1),
    (64, 128, 256, 56, 56, 3, 2), (16, 128, 128, 56, 56, 3, 1), (20, 48, 48, 100, 100, 3, 1), (3, 62, 640, 99, 99, 3, 1),
]


@pytest.mark.parametrize("shape", SHAPES, ids=str)
@pytest.mark.parametrize("types,total", [("u8f32u8f32", False), ("u8f32u8f32", True), ("u8f32s8f32", False)])
def test_shared_tiles(pkg, shape, types, total, monkeypatch):
    import gpuutil as G
    n, ic, oc, h, w, k, stride = shape
    case = R.ConvCase("spread", n, ic, oc, h, w, kh=k, kw=k, pad=k // 2, stride=stride, types=types, algo="1x1" if k == 1 else "direct",
                      relu=types == "u8f32u8f32", bias=True, sum=total, oscale=8.0)
    E = G.package()
    g = torch.Generator(device="cuda").manual_seed(hash(shape) & 0xFFFF)
    x = torch.randint(0, 256, (n, (ic + 15) // 16, h, w, 16), generator=g, device="cuda", dtype=torch.uint8)
    got = {}
    for pairs in (False, True):
        if pairs:
            monkeypatch.setenv("ELB_I8_CTA2", "1")
        d = G.make_desc(case)
        assert d.setup() == 0, E.last_error()
        assert (d.launched_kernel == "conv_halo") == (not pairs)
        gw = torch.Generator(device="cuda").manual_seed(7)
        wt = torch.randn(d.sizes.weights, generator=gw, device="cuda") * 0.1
        b = torch.randn(d.sizes.bias, generator=gw, device="cuda")
        y = torch.arange(d.byte_sizes.output, device="cuda").remainder(251).to(torch.uint8)      # (the residual, where it is added)
        assert d.prepare(wt, b) == 0 and d.enqueue(y, x) == 0, E.last_error()
        torch.cuda.synchronize()
        assert d.device_status() == 0
        got[pairs] = y.view(n, (oc + 15) // 16, -1)[:, :oc // 16]      # (channels that are padding are not compared)
        d.close()
    assert torch.equal(got[False], got[True])
