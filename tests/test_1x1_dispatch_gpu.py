"""Plain INT8 1x1 layers on the direct kernel, which most of them now take, against the GEMM kernel on pairs of CTAs: planes that no
tile width divides, tiles across images, many tiles per CTA, one and several channel tiles, every result type, bit for bit."""
import pytest
import torch

import refutil as R

pytestmark = pytest.mark.gpu

SHAPES = [(32, 64, 256, 56, 56), (5, 128, 128, 45, 94), (7, 96, 240, 31, 30), (3, 32, 112, 112, 111), (20, 200, 600, 30, 30), (53, 16, 32, 55, 55),
          (2, 3, 64, 30, 30), (1, 16, 16, 17, 17), (40, 32, 16, 1, 9), (9, 48, 80, 7, 7), (2, 1040, 1000, 1, 1)]


@pytest.mark.parametrize("shape", SHAPES, ids=str)
@pytest.mark.parametrize("types,total", [("u8f32u8f32", False), ("u8f32u8f32", True), ("u8f32s8f32", False), ("u8f32f32f32", False)])
def test_direct_equals_gemm(pkg, shape, types, total, monkeypatch):
    import gpuutil as G
    n, ic, oc, h, w = shape
    case = R.ConvCase("disp", n, ic, oc, h, w, kh=1, kw=1, pad=0, types=types, algo="1x1", relu=total, bias=True, sum=total, oscale=2.0)
    E = G.package()
    g = torch.Generator(device="cuda").manual_seed(n * 1000 + ic)
    x = torch.randint(0, 256, (n, (ic + 15) // 16, h, w, 16), generator=g, device="cuda", dtype=torch.uint8)
    wt = bias = None
    got = {}
    for gemm in (False, True):
        if gemm:
            monkeypatch.setenv("ELB_I8_CTA2", "1")
        d = G.make_desc(case)
        assert d.setup() == 0, E.last_error()
        assert d.launched_kernel == ("i8_gemm_umma" if gemm else "conv_halo")
        if wt is None:
            wt = torch.randn(d.sizes.weights, generator=g, device="cuda") * 0.1
            bias = torch.randn(d.sizes.bias, generator=g, device="cuda")
        y = torch.arange(d.byte_sizes.output, device="cuda").remainder(251).to(torch.uint8)
        assert d.prepare(wt, bias) == 0 and d.enqueue(y, x) == 0, E.last_error()
        torch.cuda.synchronize()
        assert d.device_status() == 0
        got[gemm] = y.view(n, (oc + 15) // 16, -1)[:, :oc // 16]      # (channels that are padding are not compared)
        d.close()
    assert torch.equal(got[False], got[True])
