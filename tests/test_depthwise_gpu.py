"""GPU parity of the INT8 depthwise 3x3 kernel against the CPU restatement, through the C-ABI.

Bit-exact: u8 / s8 outputs and the raw int32 accumulators.  The cases cover both strides, pads 0
and 1, the reference's split of a u8 output row into floored 4-pixel groups and nearest-rounded
remainders (chunk length T = flatting.t), its wrap-around packing when a floored value leaves
[0, 255], a non-zero input zero point, ragged widths and channel counts beyond one block.
"""
import dataclasses

import numpy as np
import pytest

import refutil as R

pytestmark = pytest.mark.gpu


def _dw(name, n, c, ih, iw, T, **kw):
    kw.setdefault("types", "u8f32u8f32")
    kw.setdefault("relu", True)
    kw.setdefault("bias", True)
    return R.ConvCase(name, n, c, c, ih, iw, g=c, algo="direct", knobs=dict(flt_t=T) if T else {}, **kw)


CASES = [
    _dw("dw_s1_t14", 2, 32, 28, 28, 14),
    _dw("dw_s1_t7_ragged", 2, 48, 23, 19, 7),
    _dw("dw_s1_t28_mobilenet_1", 2, 32, 112, 112, 28),
    _dw("dw_s2_t28_mobilenet_2", 2, 64, 112, 112, 28, stride=2, pad=0),
    _dw("dw_s2_t7", 2, 64, 28, 28, 7, stride=2),
    _dw("dw_s2_p1_odd", 1, 32, 15, 17, 5, stride=2),
    _dw("dw_s1_pad0", 1, 32, 14, 14, 6, pad=0),
    _dw("dw_s1_s8", 2, 32, 28, 28, 14, types="u8f32s8f32", relu=False),
    _dw("dw_s1_u8_norelu", 1, 32, 28, 28, 14, relu=False),
    _dw("dw_s1_overflow", 1, 32, 20, 12, 6, oscale=0.003),
    _dw("dw_s1_overflow_norelu", 1, 32, 20, 12, 6, oscale=0.003, relu=False),
    _dw("dw_s1_iz", 1, 32, 14, 14, 5, iz=3.0),
    _dw("dw_s1_t_default", 1, 32, 9, 9, 0),
    _dw("dw_s1_t3", 1, 32, 9, 10, 3),
    _dw("dw_s1_1024ch_7x7", 2, 1024, 7, 7, 7),
    _dw("dw_s1_tall_strip", 1, 16, 67, 8, 8),
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: c.name)
def test_depthwise_bit_exact(pkg, case):
    import gpuutil as G
    t = R.make_tensors(case)
    want, want_acc = R.oracle_int8_depthwise(case, t, want_acc=True)
    got, d, acc = G.run_gpu(case, t, want_acc=True)
    try:
        assert d.kernel == "i8_depthwise"
        cb = case.oc // 16
        assert np.array_equal(acc[:, :cb], want_acc[:, :cb]), "int32 accumulators differ"
        bad = int((got[:, :cb] != want[:, :cb]).sum())
        assert bad == 0, f"{bad} of {want[:, :cb].size} output bytes differ"
    finally:
        d.close()


# Without an accumulator dump the layers run on the kernel whose epilogue works on the FMA pipe (stride 1 and 2): strips
# of 2 and more rows, pairs of chunk remainders (T % 4 and the last chunk's up to 2, with even and odd chunk counts, or 3),
# groups with values above 255, both signs of the output, images narrower than a window.
FAST_CASES = CASES + [
    _dw("dw_fast_pairs_odd", 2, 32, 30, 42, 14),
    _dw("dw_fast_pairs_last_only", 1, 48, 9, 30, 8),
    _dw("dw_fast_rest3", 1, 32, 11, 21, 7),
    _dw("dw_fast_narrow", 2, 32, 5, 3, 0),
    _dw("dw_fast_s2_s8", 2, 48, 31, 33, 5, stride=2, types="u8f32s8f32"),
    _dw("dw_fast_s2_rows", 8, 64, 57, 40, 20, stride=2),
    _dw("dw_fast_many", 8, 256, 14, 14, 0),
]


@pytest.mark.parametrize("case", FAST_CASES, ids=lambda c: c.name)
def test_depthwise_without_dump(pkg, case):
    import gpuutil as G
    t = R.make_tensors(case)
    want = R.oracle_int8_depthwise(case, t)
    got, d = G.run_gpu(case, t)
    d.close()
    cb = case.oc // 16
    bad = int((got[:, :cb] != want[:, :cb]).sum())
    assert bad == 0, f"{bad} of {want[:, :cb].size} output bytes differ"


def test_depthwise_host_buffers_and_repeat(pkg):
    """The drop-in call with host memory, twice (weights are only read on the first call)."""
    import gpuutil as G
    case = _dw("dw_host", 2, 32, 28, 28, 14)
    t = R.make_tensors(case)
    want = R.oracle_int8_depthwise(case, t)
    got, d = G.run_gpu(case, t, host_buffers=True, repeat=2)
    try:
        assert np.array_equal(got, want)
    finally:
        d.close()


def test_depthwise_is_a_convolution(pkg):
    """Independent of the restatement: accumulators equal a plain integer depthwise convolution
    computed with numpy on the quantised weights the test data was built from."""
    import gpuutil as G
    case = _dw("dw_prop", 2, 32, 20, 20, 4, stride=2)
    t = R.make_tensors(case)
    _, d, acc = G.run_gpu(case, t, want_acc=True)
    d.close()
    x = R.from_nChw16c(t["input"], case.ic).astype(np.int64)
    q = t["q"].astype(np.int64)[:, 0]                       # [c][kh][kw]
    xp = np.pad(x, ((0, 0), (0, 0), (1, 1), (1, 1)))
    ref = np.zeros((case.n, case.oc, case.oh, case.ow), np.int64)
    for kh in range(3):
        for kw in range(3):
            ref += xp[:, :, kh:kh + 2 * case.oh:2, kw:kw + 2 * case.ow:2] * q[None, :, kh, kw, None, None]
    assert np.array_equal(R.from_nChw16c(acc, case.oc), ref)


@pytest.mark.parametrize("case", [
    _dw("dw_rej_s2_t1", 1, 32, 14, 14, 0, stride=2),          # T defaults to 1: reference double-counts
    _dw("dw_rej_s2_tr1", 1, 32, 14, 14, 6, stride=2),         # ow = 7, T = 6 -> remainder chunk of 1
], ids=lambda c: c.name)
def test_depthwise_rejects_undefined_chunkings(pkg, case):
    import gpuutil as G
    d = G.make_desc(case)
    assert d.setup() == pkg.ELD_UNIMPLEMENTED
    assert "one-pixel chunk" in pkg.last_error()
    d.close()


@pytest.mark.parametrize("stride", [1, 2])
def test_depthwise_between_its_neighbours(pkg, stride):
    """The kernel may start under the one before it: directly behind the layer that writes its input, and directly behind
    one that still reads the tensor it writes."""
    import torch
    import gpuutil as G
    E = G.package()
    before = R.ConvCase("dwn_before", 16, 32, 64, 56, 56, kh=1, kw=1, pad=0, types="u8f32u8f32", algo="1x1", relu=True, bias=True, oscale=0.5)
    dw = _dw("dwn", 16, 64, 56, 56, 14, stride=stride)
    after = R.ConvCase("dwn_after", 16, 64, 32, dw.oh, dw.ow, types="u8f32u8f32", algo="direct", relu=True, bias=True, oscale=0.5)
    tens = [R.make_tensors(c) for c in (before, dw, after)]
    descs = []
    for c, t in zip((before, dw, after), tens):
        d = G.make_desc(c)
        assert d.setup() == E.ELD_OK, E.last_error()
        assert d.prepare(torch.from_numpy(t["weights"]).cuda(), torch.from_numpy(t["bias"]).cuda()) == 0
        descs.append(d)
    rng = np.random.default_rng(R.seed_for("dwn", str(stride)))
    images = [rng.integers(0, 256, tens[0]["input"].shape, dtype=np.uint8) for _ in range(2)]
    plain = rng.integers(0, 256, tens[1]["input"].shape, dtype=np.uint8)      # a depthwise input of no producer

    def chain(x):
        return R.oracle_int8_conv(after, dict(tens[2], input=R.oracle_int8_depthwise(dw, dict(tens[1], input=x))))

    want = [chain(R.oracle_int8_conv(before, dict(tens[0], input=x))) for x in images]
    want_plain = chain(plain)
    xs = [torch.from_numpy(x).cuda() for x in images]
    xp = torch.from_numpy(plain).cuda()
    b1 = torch.zeros(R.out_shape(before), dtype=torch.uint8, device="cuda")
    b2 = torch.zeros(R.out_shape(dw), dtype=torch.uint8, device="cuda")
    ys = [[torch.zeros(R.out_shape(after), dtype=torch.uint8, device="cuda") for _ in range(2)] for _ in range(10)]
    s = torch.cuda.current_stream().cuda_stream
    for k, (y, z) in enumerate(ys):
        for d, o, i in ((descs[0], b1, xs[k % 2]), (descs[1], b2, b1), (descs[2], y, b2), (descs[1], b2, xp), (descs[2], z, b2)):
            assert d.enqueue(o, i, stream=s) == 0, E.last_error()
    torch.cuda.synchronize()
    for k, (y, z) in enumerate(ys):
        assert np.array_equal(y.cpu().numpy(), want[k % 2]) and np.array_equal(z.cpu().numpy(), want_plain), k
    for d in descs:
        d.close()
