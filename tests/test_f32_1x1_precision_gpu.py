"""Plain fp32 1x1 layers of few input channels on the direct kernel: its error against a 64-bit convolution, bounded and against
that of the GEMM kernel which it replaced there, with mixed and all-positive inputs, the residual and the clamp."""
import pytest
import torch

import refutil as R

pytestmark = pytest.mark.gpu

SHAPES = [(16, 64, 256, 56, 56), (5, 64, 403, 94, 45), (8, 32, 112, 112, 111), (16, 16, 64, 112, 112), (7, 160, 700, 20, 20),
          (64, 64, 256, 28, 28), (64, 512, 2048, 7, 7)]
# layers with a residual whose wide tiles are slower here: they stay on the GEMM kernel
WIDE_SUM = [(24, 32, 742, 25, 25), (14, 144, 1392, 32, 32), (4, 130, 256, 90, 90)]


def _case(shape, total):
    n, ic, oc, h, w = shape
    return R.ConvCase("disp", n, ic, oc, h, w, kh=1, kw=1, pad=0, types="fp32", algo="1x1", relu=total, bias=True, sum=total)


@pytest.mark.parametrize("shape", SHAPES, ids=str)
@pytest.mark.parametrize("total", [False, True], ids=["plain", "sum"])
@pytest.mark.parametrize("positive", [False, True], ids=["mixed", "positive"])
def test_error_against_the_gemm_kernel(pkg, shape, total, positive, monkeypatch):
    import gpuutil as G
    n, ic, oc, h, w = shape
    E = G.package()
    g = torch.Generator(device="cuda").manual_seed(ic)
    ocp = (oc + 15) // 16 * 16
    x = torch.rand((n, ic // 16, h, w, 16), generator=g, device="cuda") * 2 - 1
    wt = torch.randn((oc, ic), generator=g, device="cuda") * (2.0 / ic) ** 0.5
    if positive:
        x, wt = x.abs(), wt.abs()
    full = torch.zeros((ocp, ic), device="cuda")
    full[:oc] = wt
    bias = torch.randn(ocp, generator=g, device="cuda") * 0.1
    y0 = torch.rand((n, ocp // 16, h, w, 16), generator=g, device="cuda")
    want = torch.einsum("nbhwi,obi->nohw", x.double(), full.double().view(ocp, ic // 16, 16)) + bias.double().view(1, -1, 1, 1)
    if total:
        want = (want + y0.double().permute(0, 1, 4, 2, 3).reshape(n, ocp, h, w)).clamp_min(0)
    error = {}
    for kernel in ("conv_halo", "f32_direct_umma"):
        if kernel == "f32_direct_umma":      # the GEMM kernel behind a gather of its operand: products, order and sums are the same as on the tensor itself
            monkeypatch.setenv("ELB_F32_NO_FLAT", "1")
        d = G.make_desc(_case(shape, total))
        assert d.setup() == 0 and d.launched_kernel == kernel, E.last_error()
        buf = torch.zeros(d.sizes.weights, device="cuda")
        blocked = full.view(ocp // 16, 16, ic // 16, 16).permute(0, 2, 3, 1).reshape(-1)
        buf[:blocked.numel()] = blocked
        y = y0.clone()
        assert d.prepare(buf, bias) == 0 and d.enqueue(y, x) == 0, E.last_error()
        torch.cuda.synchronize()
        assert d.device_status() == 0
        got = y.double().permute(0, 1, 4, 2, 3).reshape(n, ocp, h, w)
        error[kernel] = ((got - want)[:, :oc].norm() / want[:, :oc].norm()).item()
        d.close()
    # 3xTF32: products exact to 2^-22; each of the up to 3 * ic / 8 additions to the accumulator cuts 1.9e-8 of the result off where
    # signs are mixed.  Positive sums only grow: at most 2^-23 of a running sum that is half of the result on average.
    assert error["conv_halo"] <= 2.4e-7 + (2.0 ** -24 if positive else 1.9e-8) * 3 * ic / 8
    # (from the same sums up to what differs in the last place of the few values: one per cent)
    assert error["conv_halo"] <= 1.01 * error["f32_direct_umma"]


@pytest.mark.parametrize("shape", WIDE_SUM, ids=str)
def test_wide_tiles_with_a_residual(pkg, shape):
    import gpuutil as G
    for total, kernel in ((True, "f32_direct_umma"), (False, "conv_halo")):
        d = G.make_desc(_case(shape, total))
        assert d.setup() == 0 and d.launched_kernel == kernel, G.package().last_error()
        d.close()
