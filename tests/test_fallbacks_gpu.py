"""Layers that the direct convolution kernel does not take, on the kernels that serve them instead, and 1x1 layers with
padding.  INT8 bit-exact (accumulators and outputs), fp32 against 64 bits."""
import numpy as np
import pytest

import refutil as R

pytestmark = pytest.mark.gpu


def _c(name, n, ic, oc, ih, iw, k, types="u8f32u8f32", **kw):
    kw.setdefault("algo", "direct")
    if types != "fp32":
        kw.setdefault("oscale", 0.3)
    return R.ConvCase(name, n, ic, oc, ih, iw, kh=k, kw=k, types=types, relu=True, bias=True, **kw)


def _run(case, launched, launches):
    import gpuutil as G
    t = R.make_tensors(case)
    if case.types == "fp32":
        got, d = G.run_gpu(case, t)
        # (up to 1.9e-8 of the result is cut off with each MMA that adds to an accumulator: four per tap and channel block in
        # the GEMM behind an im2col tensor; the direct kernel has one or three, fewer where the K loop is split)
        additions = 4 * case.kh * case.kw * ((case.ic + 15) // 16)
        assert R.rel_l2(got, R.oracle_direct_f64(case, t)) <= max(1e-5, 2.2e-8 * additions)
    else:
        want, want_acc = R.oracle_int8_conv(case, t, want_acc=True)
        got, d, acc = G.run_gpu(case, t, want_acc=True)
        assert np.array_equal(acc, want_acc) and np.array_equal(got, want)
    assert d.launched_kernel == launched and d.launch_count() == launches and d.device_status() == 0
    d.close()


@pytest.mark.parametrize("case", [
    _c("f32_k11", 1, 40, 24, 23, 21, 11, types="fp32", pad=5, sum=True),
    _c("f32_1x1_p1", 3, 64, 40, 9, 7, 1, types="fp32", pad=1),
    _c("f32_s3", 2, 48, 40, 19, 17, 3, types="fp32", stride=3),
], ids=lambda c: c.name)
def test_fp32_filters_beyond_the_direct_kernel(pkg, case):
    """An im2col tensor, the GEMM over several taps, and the epilogue kernel."""
    _run(case, "f32_direct_umma", 3)


def test_int8_filter_beyond_the_direct_kernel(pkg):
    _run(_c("i8_k11_1024", 1, 1024, 32, 12, 12, 11, pad=5, oscale=3.0), "i8_conv_umma", 1)


@pytest.mark.parametrize("case", [
    _c("i8_box_3x3", 1, 48, 40, 13, 9, 3),
    _c("i8_box_3x3_s2_sum", 1, 64, 272, 15, 11, 3, stride=2, sum=True, sscale=0.5),
    _c("i8_box_5x5_zero_point", 1, 32, 24, 9, 9, 5, pad=2, iz=128.0),
    _c("i8_box_7x7_s2_rgb", 1, 3, 64, 20, 22, 7, pad=3, stride=2),
], ids=lambda c: c.name)
def test_int8_one_copy_per_tap(pkg, case, monkeypatch):
    """The implicit GEMM with one tiled copy per tap (on one CTA: fewer than four pixel tiles), which the switch keeps."""
    monkeypatch.setenv("ELB_I8_CTA2", "1")
    _run(case, "i8_conv_umma", 1)


@pytest.mark.parametrize("case", [
    _c("i8_1x1_p1", 2, 64, 40, 9, 7, 1, pad=1),
    _c("i8_1x1_p1_zero_point", 3, 48, 24, 7, 7, 1, pad=1, iz=100.0),
    _c("i8_1x1_p2_s2", 2, 160, 272, 9, 12, 1, pad=2, stride=2),
    _c("f32_1x1_p1_s2_sum", 2, 48, 200, 12, 13, 1, types="fp32", pad=1, stride=2, sum=True),
    _c("f32_k9", 2, 32, 48, 15, 13, 9, types="fp32", pad=4),
    _c("i8_k9_s2", 2, 48, 40, 19, 17, 9, pad=4, stride=2),
], ids=lambda c: c.name)
def test_padded_1x1_and_wide_filters_on_the_direct_kernel(pkg, case):
    _run(case, "conv_halo", 1)
