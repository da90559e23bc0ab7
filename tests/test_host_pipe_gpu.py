"""Pageable host tensors of more than a megabyte (pinned slots and helper threads), and the layout converters' word
widths, at their edges."""
import os
import threading

import numpy as np
import pytest

import refutil as R

pytestmark = pytest.mark.gpu

CASES = [
    R.ConvCase("pipe_i8_sum", 9, 64, 64, 56, 56, kh=1, kw=1, pad=0, types="u8f32u8f32", algo="1x1", relu=True, bias=True, sum=True,
               sscale=0.5, oscale=0.3),
    R.ConvCase("pipe_i8_ragged", 7, 40, 24, 61, 67, types="u8f32u8f32", algo="direct", relu=True, bias=True, oscale=0.3),
    R.ConvCase("pipe_f32_big_images", 2, 48, 32, 90, 75, types="fp32", algo="direct", relu=True, bias=True),
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: c.name)
def test_pageable_tensors(pkg, case):
    import gpuutil as G
    t = R.make_tensors(case)
    got, d = G.run_gpu(case, t, host_buffers=True, repeat=3)
    if case.types == "fp32":
        assert R.rel_l2(got, R.oracle_direct_f64(case, t)) <= 1e-5
    else:
        assert np.array_equal(got, R.oracle_int8_conv(case, t))
    d.close()


def _threads():
    return len(os.listdir("/proc/self/task"))


@pytest.mark.parametrize("case", CASES, ids=lambda c: c.name)
def test_helpers_come_with_use_and_go_with_the_plan(pkg, case):
    """Pinned slots and helper threads are made for a plan that has moved 192 MB the plain way, not for one that runs
    once; another plan may use them meanwhile, and the last plan gives them back."""
    import gpuutil as G
    E = G.package()
    t = R.make_tensors(case)
    want = R.oracle_direct_f64(case, t) if case.types == "fp32" else R.oracle_int8_conv(case, t)
    out = np.zeros(R.out_shape(case), case.out_dtype)

    def run(d):
        out[...] = t["residual"] if case.sum else 0
        assert E.elx_conv(d, out, t["input"], t["weights"], t["bias"]) == E.ELX_OK, E.last_error()
        assert R.rel_l2(out, want) <= 1e-5 if case.types == "fp32" else np.array_equal(out, want)

    def plan():
        d = G.make_desc(case)
        assert d.setup() == E.ELD_OK
        run(d)
        return d

    plan().close()                                  # (the driver starts threads of its own with the first call)
    before = _threads()
    d = plan()
    assert _threads() == before
    for _ in range((192 << 20) // (t["input"].nbytes + out.nbytes) + 2):
        run(d)
    assert _threads() > before or os.cpu_count() < 4
    other = plan()
    d.close()
    run(other)
    other.close()
    assert _threads() == before


def test_pageable_tensors_from_two_threads(pkg):
    import gpuutil as G
    E = G.package()
    case = CASES[1]
    t = R.make_tensors(case)
    want = R.oracle_int8_conv(case, t)
    bad = []

    def work():
        d = G.make_desc(case)
        out = np.zeros(R.out_shape(case), case.out_dtype)
        ok = d.setup() == E.ELD_OK
        for _ in range(5):
            out[...] = 0
            ok = ok and E.elx_conv(d, out, t["input"], t["weights"], t["bias"]) == E.ELX_OK and np.array_equal(out, want)
        d.close()
        if not ok:
            bad.append(E.last_error())

    th = [threading.Thread(target=work) for _ in range(2)]
    for x in th:
        x.start()
    for x in th:
        x.join()
    assert not bad


@pytest.mark.parametrize("dtype", [np.uint8, np.float32])
@pytest.mark.parametrize("n,c,h,w", [(2, 16, 8, 8), (1, 20, 5, 13), (3, 33, 7, 7), (2, 48, 1, 129), (1, 100, 16, 65)])
def test_activation_converters(pkg, dtype, n, c, h, w):
    import torch
    import gpuutil as G
    E = G.package()
    rng = np.random.default_rng(R.seed_for("conv", f"{n}{c}{h}{w}"))
    x = rng.integers(0, 256, (n, c, h, w)).astype(dtype)
    blocked = R.to_nChw16c(x)
    for fmt, plain in ((E.nchw, x), (E.nhwc, np.ascontiguousarray(x.transpose(0, 2, 3, 1)))):
        a = torch.from_numpy(plain).cuda()
        b = torch.full(blocked.shape, 77, dtype=a.dtype, device="cuda")
        assert E.reorder(b, E.nChw16c, a, fmt, n, c, h, w) == 0
        back = torch.full(plain.shape, 77, dtype=a.dtype, device="cuda")
        assert E.reorder(back, fmt, b, E.nChw16c, n, c, h, w) == 0
        torch.cuda.synchronize()
        assert np.array_equal(b.cpu().numpy(), blocked) and np.array_equal(back.cpu().numpy(), plain)
