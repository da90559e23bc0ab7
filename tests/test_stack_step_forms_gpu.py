"""INT8 stacks whose subsample is folded into the next layer's loads: bit for bit the chain of a layer, the subsample kernel and the
next layer, with one channel block, ragged channels, 5x5 and 7x7 filters, zero points and every result type."""
import ctypes

import pytest
import torch

import refutil as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,chans,hw,step,k,kind", [
    # one channel block (two taps per K step), ragged channels, other filters, a zero point (shift by position), other results
    (9, (16, 16, 256), (61, 43), 2, 3, ""), (40, (16, 24, 200), (90, 87), 2, 3, ""), (7, (16, 41, 72), (49, 67), 3, 5, ""), (3, (16, 64, 128), (57, 57), 2, 7, ""),
    (40, (16, 64, 128), (81, 79), 2, 3, "zero point"), (4, (16, 96, 176), (35, 33), 2, 5, "zero point"), (40, (16, 80, 144), (81, 79), 2, 3, "s8"),
    (40, (16, 80, 144), (81, 79), 2, 3, "f32"),
], ids=str)
def test_folded_subsample_forms(pkg, n, chans, hw, step, k, kind):
    import gpuutil as G
    E = G.package()
    a, b, c = chans
    h, w = hw
    sh, sw = (h + step - 1) // step, (w + step - 1) // step
    cases = [R.ConvCase("fold_a", n, a, b, h, w, types="u8f32u8f32", algo="direct", relu=True, bias=True, iscale=0.02, oscale=0.05),
             R.ConvCase("fold_b", n, b, c, sh, sw, kh=k, kw=k, pad=k // 2, types={"s8": "u8f32s8f32", "f32": "u8f32f32f32"}.get(kind, "u8f32u8f32"),
                        algo="direct", relu=kind != "s8", bias=True, iscale=0.05, iz=30.0 if kind == "zero point" else 0.0, oscale=0.1)]
    channels = [(x + 15) // 16 for x in chans]      # in blocks
    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randint(0, 256, (n, channels[0], h, w, 16), generator=g, device="cuda", dtype=torch.uint8)
    single = [G.make_desc(i) for i in cases]
    weights = []
    for d in single:
        assert d.setup() == 0, E.last_error()
        wt = torch.randn(d.sizes.weights, generator=g, device="cuda") * 0.05
        bias = torch.randn(d.sizes.bias, generator=g, device="cuda") * 0.1
        assert d.prepare(wt, bias) == 0
        weights.append((wt, bias))
    mid = torch.empty((n, channels[1], h, w, 16), dtype=torch.uint8, device="cuda")
    small = torch.empty((n, channels[1], sh, sw, 16), dtype=torch.uint8, device="cuda")
    want = torch.empty((n, channels[2], sh, sw, 16), dtype=torch.float32 if kind == "f32" else torch.uint8, device="cuda")
    assert single[0].enqueue(mid, x) == 0
    assert E.subsample(small, mid, n, 16 * channels[1], h, w, step, step) == 0
    assert single[1].enqueue(want, small) == 0
    # what was refused before stays refused
    assert not single[1].input_step_supported() and single[1].enqueue_strided(want, mid, h, w, step) != 0
    st = E.ConvStack([G.make_desc(i) for i in cases], [step, 1])
    for i, (wt, bias) in enumerate(weights):
        assert st.prepare(i, wt, bias) == 0
    got = torch.zeros_like(want)
    before = st.launch_count()
    assert st.enqueue(got, x, torch.cuda.current_stream().cuda_stream) == 0, E.last_error()
    torch.cuda.synchronize()
    layers = 0
    for i in range(2):
        info = E.ElbConvInfo()
        assert E.lib.elb_conv_info(st.layer_plan(i), ctypes.byref(info)) == 0
        layers += info.launches_per_call
    assert st.launch_count() - before == layers      # no subsample kernel
    assert torch.equal(got, want)
    st.close()
    for d in single:
        d.close()
