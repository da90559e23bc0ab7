"""INT8 stacks whose subsample is folded into the next layer's loads: bit for bit the chain of a layer, the subsample kernel and the
next layer, on planes that the step does not divide, tiles across images, pairs of CTAs."""
import ctypes

import pytest
import torch

import refutil as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,chans,hw,step", [
    (8, (16, 64, 128), (223, 225), 2), (16, (32, 128, 256), (57, 55), 2), (6, (16, 64, 128), (334, 100), 3), (64, (32, 256, 512), (27, 28), 2),
    (24, (16, 128, 160), (63, 61), 4),
], ids=str)
def test_folded_subsample_equals_the_kernel(pkg, n, chans, hw, step):
    import gpuutil as G
    E = G.package()
    a, b, c = chans
    h, w = hw
    sh, sw = (h + step - 1) // step, (w + step - 1) // step
    cases = [R.ConvCase("fold_a", n, a, b, h, w, types="u8f32u8f32", algo="direct", relu=True, bias=True, iscale=0.02, oscale=0.05),
             R.ConvCase("fold_b", n, b, c, sh, sw, types="u8f32u8f32", algo="direct", relu=True, bias=True, iscale=0.05, oscale=0.1)]
    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randint(0, 256, (n, a // 16, h, w, 16), generator=g, device="cuda", dtype=torch.uint8)
    single = [G.make_desc(k) for k in cases]
    weights = []
    for d in single:
        assert d.setup() == 0, E.last_error()
        wt = torch.randn(d.sizes.weights, generator=g, device="cuda") * 0.05
        bias = torch.randn(d.sizes.bias, generator=g, device="cuda") * 0.1
        assert d.prepare(wt, bias) == 0
        weights.append((wt, bias))
    mid = torch.empty((n, b // 16, h, w, 16), dtype=torch.uint8, device="cuda")
    small = torch.empty((n, b // 16, sh, sw, 16), dtype=torch.uint8, device="cuda")
    want = torch.empty((n, c // 16, sh, sw, 16), dtype=torch.uint8, device="cuda")
    assert single[0].enqueue(mid, x) == 0
    assert E.subsample(small, mid, n, b, h, w, step, step) == 0
    assert single[1].enqueue(want, small) == 0
    # what was refused before stays refused
    assert not single[1].input_step_supported() and single[1].enqueue_strided(want, mid, h, w, step) != 0
    st = E.ConvStack([G.make_desc(k) for k in cases], [step, 1])
    for k, (wt, bias) in enumerate(weights):
        assert st.prepare(k, wt, bias) == 0
    got = torch.zeros_like(want)
    before = st.launch_count()
    assert st.enqueue(got, x, torch.cuda.current_stream().cuda_stream) == 0, E.last_error()
    torch.cuda.synchronize()
    layers = 0
    for k in range(2):
        info = E.ElbConvInfo()
        assert E.lib.elb_conv_info(st.layer_plan(k), ctypes.byref(info)) == 0
        layers += info.launches_per_call
    assert st.launch_count() - before == layers      # no subsample kernel
    assert torch.equal(got, want)
    st.close()
    for d in single:
        d.close()
