"""The halo-tiled kernel (conv_halo.cu) at the edges of its tiles, channel groups and weight-stage forms, against
the C restatement: INT8 bit-exact (accumulators and outputs), fp32 to the direct path's tolerance."""
import ctypes
import dataclasses

import numpy as np
import pytest

import refutil as R

pytestmark = pytest.mark.gpu


def _c(name, n, ic, oc, ih, iw, types="u8f32u8f32", **kw):
    kw.setdefault("relu", True)
    kw.setdefault("bias", True)
    kw.setdefault("algo", "direct")
    if types != "fp32":
        kw.setdefault("oscale", 0.3)
    return R.ConvCase(name, n, ic, oc, ih, iw, types=types, **kw)


SHAPES = [                                            # n, ic, oc, ih, iw, extra
    (1, 16, 16, 16, 8, {}),                           # exactly one tile, one chunk per group
    (2, 32, 24, 17, 9, {}),                           # one row and one column over a tile
    (5, 96, 48, 7, 7, {}),                            # six blocks, tiles across several small images
    (3, 64, 64, 14, 14, {}),                          # weights resident, four accumulators
    (2, 144, 80, 15, 15, {}),                         # nine blocks: a padded group
    (4, 128, 256, 14, 13, {}),                        # 256-wide tiles
    (3, 256, 272, 9, 9, {}),                          # two groups, two channel tiles
    (2, 64, 32, 21, 10, dict(stride=2)),              # four parity planes, odd extents
    (1, 32, 48, 12, 12, dict(kh=5, kw=5, pad=2)),
    (2, 16, 32, 20, 20, dict(kh=7, kw=7, pad=3, stride=2)),
    (36, 128, 256, 14, 14, {}),                       # pairs of CTAs
    (37, 64, 256, 28, 28, dict(stride=2)),            # pairs, parity planes; an odd number of row tiles
    (3, 96, 300, 17, 19, dict(stride=2)),             # stride 2, taps as weight stages: six, four and two blocks per group
    (2, 64, 260, 12, 30, dict(stride=2)),
    (2, 32, 272, 15, 15, dict(stride=2)),
    (2, 64, 260, 16, 15, dict(stride=2, pad=0)),
    (3, 160, 272, 9, 9, dict(kh=1, kw=1, pad=0, stride=2)),
    (3, 160, 272, 13, 9, dict(stride=2, sum=True, sscale=0.5)),
    (1, 512, 64, 14, 14, {}),                         # a tile's K loop shared by the CTAs of a cluster
    (2, 1024, 256, 7, 7, dict(kh=1, kw=1, pad=0, algo="1x1")),
    (1, 304, 40, 9, 9, dict(kh=1, kw=1, pad=0, algo="1x1")),
    (2, 48, 64, 9, 11, dict(kh=1, kw=1, pad=0, stride=2)),
]


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s[:5])) + "".join(f"_{k}{v}" for k, v in s[5].items()))
@pytest.mark.parametrize("types", ["u8f32u8f32", "fp32"])
def test_halo_matches_oracle(pkg, shape, types):
    import gpuutil as G
    n, ic, oc, ih, iw, kw = shape
    case = _c("halo", n, ic, oc, ih, iw, types=types, **kw)
    t = R.make_tensors(case)
    if types == "fp32":
        got, d = G.run_gpu(case, t)
        assert d.launch_count() == 1 and d.device_status() == 0
        assert d.launched_kernel == "conv_halo"
        assert R.rel_l2(got, R.oracle_direct_f64(case, t)) <= 1e-5
    else:
        want, want_acc = R.oracle_int8_conv(case, t, want_acc=True)
        got, d, acc = G.run_gpu(case, t, want_acc=True)
        assert d.launch_count() == 1 and d.device_status() == 0
        assert d.launched_kernel == ("i8_gemm_umma" if shape[:3] == (1, 304, 40) else "conv_halo")      # (a 1x1 layer the GEMM kernel keeps)
        assert np.array_equal(acc, want_acc) and np.array_equal(got, want)
    d.close()


@pytest.mark.parametrize("shape", [(1, 64, 64, 17, 20), (2, 96, 40, 9, 9), (1, 512, 512, 14, 14)], ids=str)
@pytest.mark.parametrize("tile", [6, 4])
@pytest.mark.parametrize("total", [False, True])
def test_winograd_request_on_the_direct_kernel(pkg, shape, tile, total):
    """fp32 Winograd requests the plan serves with the direct kernel: one launch, the Winograd result."""
    import gpuutil as G
    n, ic, oc, ih, iw = shape
    case = R.ConvCase("halo_wino", n, ic, oc, ih, iw, types="fp32", algo="wino", tile=tile, relu=True, bias=True, sum=total)
    t = R.make_tensors(case)
    got, d = G.run_gpu(case, t)
    assert d.kernel == "wino_f32_umma" and d.launched_kernel == "conv_halo" and d.launch_count() == 1 and d.device_status() == 0
    assert R.rel_l2(got, R.oracle_wino_f32(case, t)) <= 1e-5
    d.close()


@pytest.mark.parametrize("shape", [(1, 32, 48, 28, 31), (2, 64, 64, 56, 56), (1, 96, 112, 40, 31), (24, 64, 128, 28, 28), (4, 128, 128, 28, 27),
                                   (1, 144, 64, 60, 60), (1, 256, 256, 14, 14)], ids=str)
def test_winograd_request_is_no_less_precise_than_the_transform_kernels(pkg, shape):
    """Whatever kernel a plan chooses, its error against 64 bits is at most that of the three transform kernels.
    F(4x4,3x3): the allocation-free entry point always runs those.  F(2x2,3x3): their error as it was measured, 1.9e-8 of the
    result for each MMA that adds into an accumulator (4 or 6 per channel block) and 5 to 7 times that for the transforms."""
    import torch
    import gpuutil as G
    E = G.package()
    n, ic, oc, ih, iw = shape
    case = R.ConvCase("halo_precision", n, ic, oc, ih, iw, types="fp32", algo="wino", tile=6, bias=True)
    t = R.make_tensors(case)
    want = R.oracle_direct_f64(case, t)
    desc = G.make_desc(case)._c_desc()
    x, w, b = (torch.from_numpy(t[k]).cuda() for k in ("input", "weights", "bias"))
    y = torch.zeros(R.out_shape(case), device="cuda")
    rc = E.lib.elb_wino_f32_conv_noalloc(ctypes.byref(desc), y.data_ptr(), x.data_ptr(), w.data_ptr(), b.data_ptr(), None)
    assert rc == 0, E.last_error()
    torch.cuda.synchronize()
    limit = R.rel_l2(y.cpu().numpy(), want)
    got, d6 = G.run_gpu(case, t)
    assert R.rel_l2(got, want) <= 1.02 * limit
    got, d4 = G.run_gpu(dataclasses.replace(case, tile=4), t)
    assert R.rel_l2(got, want) <= 2.2e-8 * ((4 if oc <= 128 else 6) * ((ic + 15) // 16) + 7)
    d6.close()
    d4.close()


def test_winograd_request_keeps_infinities(pkg):
    """The Winograd path's ReLU is a plain maximum with zero: an infinite sum stays infinite."""
    import gpuutil as G
    case = R.ConvCase("halo_inf", 1, 512, 512, 14, 14, types="fp32", algo="wino", tile=6, relu=True, bias=True)
    t = R.make_tensors(case)
    t["bias"] = t["bias"].copy()
    t["bias"][[3, 500]], t["bias"][4] = np.inf, -np.inf
    got, d = G.run_gpu(case, t)
    assert d.launch_count() == 1
    got = R.from_nChw16c(got, 512)
    assert np.isposinf(got[:, [3, 500]]).all() and (got[:, 4] == 0).all() and np.isfinite(np.delete(got, [3, 500], 1)).all()
    d.close()


def test_direct_kernel_reads_its_input_with_a_step(pkg):
    import torch
    import gpuutil as G
    E = G.package()
    case = R.ConvCase("halo_step", 2, 64, 48, 11, 10, types="fp32", algo="wino", tile=6, relu=True, bias=True)
    t = R.make_tensors(case)
    want = R.oracle_wino_f32(case, t)
    d = G.make_desc(case)
    assert d.setup() == E.ELD_OK and d.input_step_supported()
    assert d.prepare(torch.from_numpy(t["weights"]).cuda(), torch.from_numpy(t["bias"]).cuda()) == 0
    big = np.full((2, 4, 21, 20, 16), 7.0, np.float32)
    big[:, :, ::2, ::2] = t["input"]
    out = torch.zeros(R.out_shape(case), device="cuda")
    assert d.enqueue_strided(out, torch.from_numpy(big).cuda(), 21, 20, 2) == 0, E.last_error()
    torch.cuda.synchronize()
    assert d.launch_count() == 1 and R.rel_l2(out.cpu().numpy(), want) <= 1e-5
    d.close()


ALIGN_CASES = [
    R.ConvCase("al_direct", 2, 48, 40, 13, 11, stride=2, types="fp32", algo="direct", relu=True, bias=True, sum=True),
    R.ConvCase("al_split", 1, 256, 64, 14, 14, types="fp32", algo="direct", bias=True),
    R.ConvCase("al_wino", 16, 64, 64, 24, 24, types="fp32", algo="wino", tile=6, relu=True, bias=True),
    R.ConvCase("al_small_ic", 2, 3, 40, 19, 21, types="fp32", algo="wino", tile=6, relu=True, bias=True),
    R.ConvCase("al_small_ic_image", 2, 3, 40, 19, 20, types="fp32", algo="wino", tile=6, bias=True, ifmt="nchw"),
    R.ConvCase("al_rgb", 2, 3, 64, 19, 40, types="fp32", algo="wino", tile=6, relu=True, bias=True, ifmt="nchw"),
    R.ConvCase("al_u8_f32", 2, 64, 40, 13, 11, types="u8f32f32f32", algo="direct", relu=True, bias=True),
]


@pytest.mark.parametrize("case", ALIGN_CASES, ids=lambda c: c.name)
def test_tensors_sixteen_bytes_into_an_allocation(pkg, case):
    """16-byte alignment is all that the library asks of a tensor; 32-byte stores need a look at the address."""
    import torch
    import gpuutil as G
    E = G.package()
    blocked = dataclasses.replace(case, ifmt="")
    t = R.make_tensors(blocked)
    oracle = R.oracle_int8_conv if case.types != "fp32" else R.oracle_wino_f32 if case.algo == "wino" else R.oracle_direct_f64
    want = oracle(blocked, t)
    t = R.user_tensors(case, t)
    first = t["residual"] if case.sum else np.zeros(R.out_shape(case), case.out_dtype)

    def shifted(a):
        raw = torch.full((a.nbytes + 4096 + 16,), 0xA5, dtype=torch.uint8, device="cuda")
        raw[16:16 + a.nbytes] = torch.from_numpy(np.ascontiguousarray(a).view(np.uint8).reshape(-1)).cuda()
        return raw, raw.data_ptr() + 16

    d = G.make_desc(case)
    assert d.setup() == E.ELD_OK, E.last_error()
    x, x_ptr = shifted(t["input"])
    y, y_ptr = shifted(first)
    assert x_ptr % 32 == 16 and y_ptr % 32 == 16
    assert E.elx_conv(d, y_ptr, x_ptr, torch.from_numpy(t["weights"]).cuda(), torch.from_numpy(t["bias"]).cuda()) == E.ELX_OK, E.last_error()
    raw = y.cpu().numpy()
    got = raw[16:16 + first.nbytes].view(case.out_dtype).reshape(first.shape)
    assert (raw[:16] == 0xA5).all() and (raw[16 + first.nbytes:] == 0xA5).all() and d.device_status() == 0
    if case.types == "fp32":
        assert R.rel_l2(got, want) <= 1e-5
    else:
        assert np.array_equal(got, want)
    d.close()


@pytest.mark.parametrize("case", [
    _c("turns_i8_s2", 3, 64, 48, 15, 13, stride=2),
    _c("turns_i8_small_images", 5, 32, 32, 7, 7),
    _c("turns_f32", 3, 32, 48, 9, 20, types="fp32"),
], ids=lambda c: c.name)
def test_inputs_taking_turns(pkg, case):
    """A plan keeps its tensor maps per image count, not per address: every call reads the tensor it is given."""
    import torch
    import gpuutil as G
    E = G.package()
    sets = [R.make_tensors(dataclasses.replace(case, name=f"{case.name}{k}")) for k in range(4)]
    w, b = (torch.from_numpy(sets[0][k]).cuda() for k in ("weights", "bias"))
    d = G.make_desc(case)
    assert d.setup() == E.ELD_OK and d.prepare(w, b) == 0
    xs = [torch.from_numpy(t["input"]).cuda() for t in sets]
    oracle = R.oracle_direct_f64 if case.types == "fp32" else R.oracle_int8_conv
    wants = [oracle(case, dict(sets[0], input=t["input"])) for t in sets]
    ys = [torch.zeros(R.out_shape(case), dtype=torch.from_numpy(wants[0]).dtype, device="cuda") for _ in range(12)]
    for k, y in enumerate(ys):
        assert d.enqueue(y, xs[(5 * k) % 4], stream=torch.cuda.current_stream().cuda_stream) == 0, E.last_error()
    torch.cuda.synchronize()
    for k, y in enumerate(ys):
        want = wants[(5 * k) % 4]
        assert (R.rel_l2(y.cpu().numpy(), want) <= 1e-5) if case.types == "fp32" else np.array_equal(y.cpu().numpy(), want)
    d.close()
