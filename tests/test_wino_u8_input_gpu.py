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
