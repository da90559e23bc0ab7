"""The quantising input transform of the INT8 Winograd path around the bound that chooses its kernel (scaled values below 2^15: pairs
of channels; below 2^22: one channel at a time; beyond: the general conversion): the transform-domain accumulators against the
restatement, bit for bit, on planes of border tiles only, mixed and wide ones."""
import dataclasses

import numpy as np
import pytest

import refutil as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rep", [0.02, 4.5, 4.7, 500.0, 700.0])      # 255 * 5.28125^2 * rep: 142, 32006, 33428, 3.6e6, 5.0e6
@pytest.mark.parametrize("shape", [(1, 16, 16, 3, 5), (2, 48, 32, 9, 35), (1, 144, 16, 20, 66)], ids=str)
@pytest.mark.parametrize("fmt", ["", "nhwc"])
def test_accumulators_around_the_bound(pkg, rep, shape, fmt):
    import gpuutil as G
    n, ic, oc, h, w = shape
    case = R.ConvCase("u8_in", n, ic, oc, h, w, types="u8f32f32f32", algo="wino", tile=6, iscale=0.05, tscale=0.05 / rep, tz=100.0 if rep < 1 else 3.0)
    t = R.make_tensors(case)
    want, dumps = R.oracle_int8_wino(case, t, dumps=True)
    plain = dataclasses.replace(case, ifmt=fmt)
    got, d, acc = G.run_gpu(plain, R.user_tensors(plain, t), want_acc=True, acc_shape=(36, R.wino_tiles(case), R.alignup(oc)))
    assert d.kernel == "wino_i8_umma" and d.device_status() == 0
    d.close()
    assert np.array_equal(acc, dumps["acc"])
    assert R.rel_l2(got, want) <= 1e-5


# Three columns of three rows each, whose border corner quantises to another 8-bit value at 4.5 V + 3 when one product and the
# sum behind it are rounded once (an fma) instead of twice
ROUND_TWICE = [(137, 126, 171, 233, 101, 32, 85, 104, 176), (163, 208, 211, 216, 106, 74, 47, 8, 126), (227, 20, 19, 5, 22, 80, 141, 111, 130),
               (163, 166, 165, 173, 185, 40, 4, 246, 9), (43, 157, 146, 182, 132, 37, 104, 145, 123), (55, 11, 13, 210, 104, 23, 82, 155, 175),
               (47, 207, 241, 205, 104, 59, 136, 6, 80), (135, 208, 169, 208, 136, 66, 2, 76, 147)]


@pytest.mark.parametrize("fmt", ["", "nhwc"])
def test_border_corners_round_twice(pkg, fmt):
    """V[0][5] and V[5][0] of border tiles, whose products and sums the reference rounds one by one: inputs for which an fma in their
    place gives another 8-bit value, in tiles (1, 0) and (0, 1) of a plane of 3 x 3 tiles."""
    import gpuutil as G
    case = R.ConvCase("u8_corner", 1, 64, 16, 9, 9, types="u8f32f32f32", algo="wino", tile=6, iscale=0.05, tscale=0.05 / 4.5, tz=3.0)
    t = R.make_tensors(case)
    planes = np.moveaxis(t["input"].reshape(4, 9, 9, 16), 3, 1).reshape(64, 9, 9).copy()      # (channel, row, column)
    for at, rows, cols in ((0, (3, 5, 7), (0, 2, 4)), (32, (0, 2, 4), (3, 5, 7))):
        for k, px in enumerate(ROUND_TWICE):
            planes[at + k][np.ix_(rows, cols)] = np.reshape(px, (3, 3))
    t["input"] = np.ascontiguousarray(np.moveaxis(planes.reshape(4, 16, 9, 9), 1, 3)).reshape(t["input"].shape)
    want, dumps = R.oracle_int8_wino(case, t, dumps=True)
    plain = dataclasses.replace(case, ifmt=fmt)
    got, d, acc = G.run_gpu(plain, R.user_tensors(plain, t), want_acc=True, acc_shape=(36, R.wino_tiles(case), R.alignup(case.oc)))
    d.close()
    assert np.array_equal(acc, dumps["acc"])
    assert R.rel_l2(got, want) <= 1e-5
