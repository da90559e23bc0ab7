"""Plain fp32 1x1 layers of few input channels on the direct kernel: against a 64-bit convolution, with the residual and the clamp."""
import pytest
import torch

import refutil as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(16, 64, 256, 56, 56), (5, 64, 403, 94, 45), (8, 32, 112, 112, 111), (16, 16, 64, 112, 112), (7, 160, 700, 20, 20),
                                   (64, 64, 256, 28, 28)], ids=str)
@pytest.mark.parametrize("total", [False, True], ids=["plain", "sum"])
def test_error_against_64_bits(pkg, shape, total):
    import gpuutil as G
    n, ic, oc, h, w = shape
    case = R.ConvCase("disp", n, ic, oc, h, w, kh=1, kw=1, pad=0, types="fp32", algo="1x1", relu=total, bias=True, sum=total)
    E = G.package()
    g = torch.Generator(device="cuda").manual_seed(ic)
    ocp = (oc + 15) // 16 * 16
    x = torch.rand((n, ic // 16, h, w, 16), generator=g, device="cuda") * 2 - 1
    wt = torch.randn((oc, ic), generator=g, device="cuda") * (2.0 / ic) ** 0.5
    full = torch.zeros((ocp, ic), device="cuda")
    full[:oc] = wt
    d = G.make_desc(case)
    assert d.setup() == 0 and d.launched_kernel == "conv_halo", E.last_error()
    buf = torch.zeros(d.sizes.weights, device="cuda")
    blocked = full.view(ocp // 16, 16, ic // 16, 16).permute(0, 2, 3, 1).reshape(-1)
    buf[:blocked.numel()] = blocked
    bias = torch.randn(ocp, generator=g, device="cuda") * 0.1
    y = torch.rand((n, ocp // 16, h, w, 16), generator=g, device="cuda")
    want = torch.einsum("nbhwi,obi->nohw", x.double(), full.double().view(ocp, ic // 16, 16)) + bias.double().view(1, -1, 1, 1)
    if total:
        want = (want + y.double().permute(0, 1, 4, 2, 3).reshape(n, ocp, h, w)).clamp_min(0)
    assert d.prepare(buf, bias) == 0 and d.enqueue(y, x) == 0, E.last_error()
    torch.cuda.synchronize()
    assert d.device_status() == 0
    got = y.double().permute(0, 1, 4, 2, 3).reshape(n, ocp, h, w)
    # 3xTF32: products exact to 2^-22; each of the up to 3 * ic / 8 additions to the accumulator cuts 1.9e-8 of the result off
    assert ((got - want)[:, :oc].norm() / want[:, :oc].norm()).item() <= 2.4e-7 + 1.9e-8 * 3 * ic / 8
    d.close()
