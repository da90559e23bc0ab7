"""nhwc tensors read and written by the Winograd transform kernels themselves: bit for bit what the same plan makes of the
blocked tensors, and what a tensor off the kernels' alignment (which is converted first) gives."""
import dataclasses

import numpy as np
import pytest

import refutil as R

pytestmark = pytest.mark.gpu


def _case(types, tile, n, ic, oc, ih, iw, **kw):
    kw.setdefault("relu", True)
    return R.ConvCase(f"nhwc_{types}_{tile}_{ic}_{oc}_{ih}x{iw}", n, ic, oc, ih, iw, types=types, algo="wino", tile=tile, bias=True, **kw)


CASES = [      # whole groups of four channels but not of sixteen, ragged planes, one image and tile blocks across images
    _case("fp32", 6, 8, 100, 196, 23, 21),
    _case("fp32", 6, 3, 484, 260, 13, 9, sum=True),
    _case("fp32", 4, 4, 260, 132, 11, 17),
    _case("u8f32f32f32", 6, 3, 36, 20, 19, 22, relu=False),
    _case("u8f32f32f32", 4, 2, 148, 12, 9, 30),
    _case("u8f32u8f32", 6, 2, 64, 44, 14, 7, oscale=2.0),
    _case("u8f32s8f32", 4, 2, 20, 68, 8, 8, oscale=0.1, sum=True),
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: c.name)
def test_nhwc_equals_blocked(pkg, case, monkeypatch):
    monkeypatch.setenv("ELB_WINO_CTA2", "1")      # (keeps the fp32 layers on the transform kernels)
    import torch
    import gpuutil as G
    E = G.package()
    t = R.make_tensors(case)
    if case.types != "fp32":
        case = R.calibrate_tinput(case, t)
    blocked, d0 = G.run_gpu(case, t)
    d0.close()
    want = R.act_to_user(blocked, case.oc, "nhwc")
    plain = dataclasses.replace(case, ifmt="nhwc", ofmt="nhwc")
    u = R.user_tensors(plain, t)
    got, d = G.run_gpu(plain, u)
    assert d.kernel.startswith("wino") and d.launched_kernel == d.kernel and d.launch_count() == 3      # no conversions
    assert np.array_equal(got, want)
    # one element off: converted first, with the same result
    x = torch.empty(u["input"].size + 1, dtype=torch.from_numpy(u["input"]).dtype, device="cuda")
    x[1:] = torch.from_numpy(u["input"]).cuda().flatten()
    y = torch.empty(want.size + 1, dtype=torch.from_numpy(want).dtype, device="cuda")
    y[1:] = torch.from_numpy(u["residual"]).cuda().flatten() if case.sum else 0
    assert d.enqueue(y.data_ptr() + y.element_size(), x.data_ptr() + x.element_size(), None, None, None) == 0, E.last_error()
    torch.cuda.synchronize()
    assert d.launch_count() == 3 + 5 + (1 if case.sum else 0)
    assert np.array_equal(y[1:].cpu().numpy().reshape(want.shape), want)
    d.close()


def test_nhwc_channels_that_are_no_groups_of_four_are_converted(pkg, monkeypatch):
    monkeypatch.setenv("ELB_WINO_CTA2", "1")
    import gpuutil as G
    case = _case("fp32", 6, 4, 482, 130, 18, 18)
    t = R.make_tensors(case)
    blocked, d0 = G.run_gpu(case, t)
    d0.close()
    plain = dataclasses.replace(case, ifmt="nhwc", ofmt="nhwc")
    got, d = G.run_gpu(plain, R.user_tensors(plain, t))
    assert d.launch_count() == 5 and np.array_equal(got, R.act_to_user(blocked, case.oc, "nhwc"))
    d.close()


@pytest.mark.parametrize("chunks", [2, 3])
@pytest.mark.parametrize("case", CASES, ids=lambda c: c.name)
def test_image_ranges(pkg, case, chunks, monkeypatch):
    """Host tensors cut into ranges of images: the kernels find each range in the nhwc tensors by the caller's pitch (channel counts that
    are no multiple of 16), as the blocked tensor's result in one range."""
    monkeypatch.setenv("ELB_WINO_CTA2", "1")
    import gpuutil as G
    t = R.make_tensors(case)
    if case.types != "fp32":
        case = R.calibrate_tinput(case, t)
    blocked, d0 = G.run_gpu(case, t)
    d0.close()
    plain = dataclasses.replace(case, ifmt="nhwc", ofmt="nhwc")
    monkeypatch.setenv("ELB_HOST_CHUNKS", str(chunks))
    got, d = G.run_gpu(plain, R.user_tensors(plain, t), host_buffers=True)
    assert d.launch_count() == 3 * min(chunks, case.n) and d.device_status() == 0      # no conversions
    d.close()
    assert np.array_equal(got, R.act_to_user(blocked, case.oc, "nhwc"))
