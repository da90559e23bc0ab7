"""Performance cases of the convolution library: what its users run, through the public entry points of
the package (``eld_conv_t``, ``elx_conv``, ``eld_conv_t.enqueue``, ``ConvStack``).

A case is a dict of plain values.  ``kind`` names the path:

  i8_conv    INT8 u8s8 convolution, 1x1 or KxK, stride 1 or 2 (ResNet-style layers, requantised)
  i8_dw      INT8 depthwise 3x3 (MobileNet-style layers)
  i8_wino    INT8 Winograd 3x3
  f32_wino   FP32 Winograd 3x3
  f32_conv   FP32 direct convolution, 1x1 or KxK
  vgg_f32    the 13 convolutions of VGG-16 as one stack, FP32 Winograd
  vgg_i8     the same stack with INT8 direct convolutions, u8 between the layers

``call`` says how the user calls it: "stream" enqueues on the current stream with device tensors, "sync" is
``elx_conv`` on device tensors (returns when the result is there), "host" is ``elx_conv`` on numpy arrays
or, for the stacks, ``ConvStack.execute`` on pinned host tensors.
"""
import importlib
import math

import numpy as np
import torch

E = importlib.import_module("deep-learning-math-kernel-research_b200")


def _conv(name, kind, n, ic, oc, h, w, k=3, stride=1, **more):
    c = dict(name=name, kind=kind, n=n, ic=ic, oc=oc, h=h, w=w, k=k, stride=stride, relu=True, sum=False,
             out="f32" if kind.startswith("f32") else "u8", tile=6, layout="nChw16c", call="stream")
    c.update(more)
    return c


def listed():
    return [
        # one image through a ResNet-50 res4 reduce layer, waited for: what a latency-bound server pays per call
        _conv("i8_1x1_one_image", "i8_conv", 1, 1024, 256, 14, 14, k=1, call="sync"),
        # one image through a VGG-16 conv5 layer, waited for
        _conv("f32_wino_one_image", "f32_wino", 1, 512, 512, 14, 14, call="sync"),
        # the same ResNet-50 layer at a training-sized batch, inside a stream of other work
        _conv("i8_1x1_batch", "i8_conv", 64, 1024, 256, 14, 14, k=1),
        # downsampling 3x3 with a residual added in place (the shortcut's tensor is the output tensor)
        _conv("i8_3x3_s2_sum", "i8_conv", 64, 128, 256, 56, 56, stride=2, sum=True),
        # MobileNet-v1 depthwise layer
        _conv("i8_depthwise", "i8_dw", 64, 128, 128, 56, 56),
        # INT8 Winograd, fp32 result, the largest single layer of the benchmark in operations
        _conv("i8_wino", "i8_wino", 128, 512, 512, 28, 28, out="f32", relu=False),
        # FP32 Winograd, VGG-16 conv3_2
        _conv("f32_wino_batch", "f32_wino", 64, 256, 256, 56, 56),
        # FP32 downsampling 3x3 without Winograd
        _conv("f32_3x3_s2", "f32_conv", 64, 128, 256, 56, 56, stride=2),
        # a caller with plain channels-last tensors and ragged sizes
        _conv("f32_nhwc_ragged", "f32_wino", 8, 96, 200, 45, 27, layout="nhwc", tile=0),
        # a caller of the CPU library who keeps numpy arrays and switches to this one
        _conv("i8_1x1_host", "i8_conv", 64, 1024, 256, 14, 14, k=1, call="host"),
        # the whole VGG-16 stack on the device, and fed from pinned host memory in batches
        dict(name="vgg_f32", kind="vgg_f32", n=64, images=64, call="stream"),
        dict(name="vgg_i8_host", kind="vgg_i8", n=64, images=256, call="host"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _channels(rng, lo, hi):
    """Mostly multiples of 16, as networks have them; one in four is not."""
    c = _log_int(rng, lo, hi)
    return c if rng.random() < 0.25 else max(16, c // 16 * 16)


def _draw_once(rng):
    kind = rng.choice(["i8_conv", "i8_conv", "i8_conv", "i8_dw", "i8_wino", "f32_wino", "f32_wino", "f32_conv", "f32_conv",
                       "vgg_f32", "vgg_i8"])
    if kind.startswith("vgg"):
        n = _log_int(rng, 1, 64)
        call = rng.choice(["stream", "host"])
        return dict(kind=kind, n=n, images=n * (rng.randint(1, 3) if call == "host" else 1), call=call)
    c = _conv("", kind, _log_int(rng, 1, 128), _channels(rng, 16, 1024), _channels(rng, 16, 1024), _log_int(rng, 7, 224), 0)
    del c["name"]
    c["w"] = c["h"] if rng.random() < 0.7 else max(7, min(224, int(c["h"] * rng.uniform(0.6, 1.7))))
    c["relu"] = rng.random() < 0.8
    c["call"] = rng.choice(["stream", "stream", "stream", "sync", "sync", "host"])
    if kind == "i8_dw":
        c["oc"] = c["ic"]
        c["stride"] = rng.choice([1, 1, 2])
        c["out"] = rng.choice(["u8", "u8", "u8", "s8"])
        return c
    if kind in ("i8_conv", "f32_conv"):
        c["k"] = rng.choice([1, 1, 3, 3, 5, 7])
        c["stride"] = rng.choice([1, 1, 2])
        c["sum"] = rng.random() < 0.25
        if c["k"] == 7:      # the first layer of an image network
            c["ic"], c["stride"], c["layout"], c["sum"] = 3, 2, "nchw", False
    else:
        c["tile"] = rng.choice([6, 6, 6, 4])
    if kind == "i8_conv":
        c["out"] = rng.choice(["u8", "u8", "s8", "f32"])
    if kind == "i8_wino":
        c["out"] = "f32"
    if c["layout"] == "nChw16c" and rng.random() < 0.2:
        c["layout"] = rng.choice(["nchw", "nhwc"])
    return c


def draw(rng):
    top = [work(c) for c in listed()]
    most_bytes, most_flops = 3e8, max(w["flops"] for w in top) / 4
    while True:
        c = _draw_once(rng)
        w = work(c)
        fits = w["bytes"] <= (most_bytes if c["call"] != "host" else 1e8) and w["flops"] <= most_flops
        if c["kind"].startswith("vgg") or fits:
            return c


# ---------------------------------------------------------------------------------------- geometry
def _up(v):
    return (v + 15) // 16 * 16


def _pad(c):
    return c["k"] // 2


def _out_hw(c):
    p = _pad(c)
    return tuple((v + 2 * p - c["k"]) // c["stride"] + 1 for v in (c["h"], c["w"]))


VGG16 = [(3, 64, 224, 1), (64, 64, 224, 2), (64, 128, 112, 1), (128, 128, 112, 2), (128, 256, 56, 1), (256, 256, 56, 1),
         (256, 256, 56, 2), (256, 512, 28, 1), (512, 512, 28, 1), (512, 512, 28, 2), (512, 512, 14, 1), (512, 512, 14, 1),
         (512, 512, 14, 1)]      # input channels, output channels, plane edge, subsample behind the layer


def work(case):
    """Bytes: input, weights and result once (int8: one byte per weight).  Operations: those of the algorithm
    the case asks for, i.e. F(4x4,3x3) needs a quarter of the direct convolution's and F(2x2,3x3) 4/9."""
    c = case
    if c["kind"].startswith("vgg"):
        el, flops, bytes_ = (4, 0, 0) if c["kind"] == "vgg_f32" else (1, 0, 0)
        for k, (ic, oc, hw, step) in enumerate(VGG16):
            saved = 4 if c["kind"] == "vgg_f32" and k > 0 else 1
            flops += 2 * c["images"] * ic * oc * hw * hw * 9 // saved
            bytes_ += ic * oc * 9 * el
        bytes_ += c["images"] * (3 * 224 * 224 + 512 * 14 * 14) * el
        return {"bytes": bytes_, "flops": flops}
    oh, ow = _out_hw(c)
    eb = 4 if c["kind"].startswith("f32") else 1
    ob = 4 if c["out"] == "f32" else 1
    icg = 1 if c["kind"] == "i8_dw" else c["ic"]
    n_in = c["n"] * c["ic"] * c["h"] * c["w"]
    n_out = c["n"] * c["oc"] * oh * ow
    flops = 2 * n_out * icg * c["k"] ** 2
    if c["kind"].endswith("wino"):
        flops = flops * 4 // 9 if c["tile"] == 4 else flops // 4
    return {"bytes": n_in * eb + c["oc"] * icg * c["k"] ** 2 * eb + n_out * ob * (2 if c["sum"] else 1), "flops": flops}


def tolerance(case):
    if case["kind"] == "vgg_f32":
        return {"rel": 3e-5}          # 13 chained fp32 layers
    if case["kind"].startswith("f32"):
        return {"rel": 1e-5}          # fp32 sums in another order
    if case["kind"] == "i8_wino":
        return {"rel": 2e-6}          # exact integer sums, fp32 output transform
    if case.get("out") == "f32":
        return {"rel": 1e-6}          # exact integer sum, one fp32 multiply-add
    return "exact"                    # whole numbers


# ---------------------------------------------------------------------------------------- inputs
def _rng(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _activations(c, ch, h, w, values):
    """values: function(shape) -> device tensor; returned in the case's layout, padding channels zero."""
    if c["layout"] == "nchw":
        return values((c["n"], ch, h, w))
    if c["layout"] == "nhwc":
        return values((c["n"], h, w, ch))
    x = values((c["n"], _up(ch) // 16, h, w, 16))
    if ch % 16:
        x[:, -1, :, :, ch % 16:] = 0
    return x


def _blocked_weights(w, size):
    """[o][i][kh][kw] -> OIhw16i16o in a buffer of the size the descriptor asks for."""
    o, i, kh, kw = w.shape
    full = torch.zeros((_up(o), _up(i), kh, kw), device=w.device)
    full[:o, :i] = w
    full = full.view(_up(o) // 16, 16, _up(i) // 16, 16, kh, kw).permute(0, 2, 4, 5, 3, 1).reshape(-1)
    buf = torch.zeros(size, device=w.device)
    buf[:full.numel()] = full
    return buf


def _s8_weights(g, oc, icg, k):
    """s8 uniform codes times a scale per output channel uniform[0.001, 0.01]."""
    q = torch.randint(-127, 128, (oc, icg, k, k), generator=g, device="cuda").float()
    q.view(oc, -1)[:, 0] = 127.0
    return q * (0.001 + 0.009 * torch.rand((oc, 1, 1, 1), generator=g, device="cuda"))


class _State:
    pass


def _check(rc, what):
    if rc != 0:
        raise RuntimeError(f"{what} rc={rc}: {E.last_error()}")


def _prepare_conv(c, seed):
    g = _rng(seed)
    s = _State()
    int8, dw = c["kind"].startswith("i8"), c["kind"] == "i8_dw"
    oh, ow = _out_hw(c)
    d = s.d = E.eld_conv_t()
    d.dims.n, d.dims.g, d.dims.ic, d.dims.oc = c["n"], c["ic"] if dw else 1, c["ic"], c["oc"]
    d.dims.ih, d.dims.iw, d.dims.oh, d.dims.ow, d.dims.kh, d.dims.kw = c["h"], c["w"], oh, ow, c["k"], c["k"]
    d.pads.l = d.pads.r = d.pads.t = d.pads.b = _pad(c)
    d.strides.h = d.strides.w = c["stride"]
    d.with_relu, d.with_bias, d.with_ip_sum = c["relu"], True, c["sum"]
    fmt = {"nChw16c": E.nChw16c, "nchw": E.nchw, "nhwc": E.nhwc}[c["layout"]]
    d.formats.input = d.formats.output = fmt
    d.formats.weights = E.goihw if dw else E.OIhw16i16o
    icg = 1 if dw else c["ic"]
    if c["kind"].endswith("wino"):
        d.algorithm, d.tile_size = E.CONV_WINOGRAD, c["tile"]
    else:
        d.algorithm = E.CONV_DIRECT_1X1 if c["k"] == 1 else E.CONV_DIRECT
    if int8:
        d.data_type.input = E.u8
        d.data_type.output = {"u8": E.u8, "s8": E.s8, "f32": E.f32}[c["out"]]
        sd = math.sqrt(icg * c["k"] ** 2) * 0.05 * 147 * 0.4     # of the result: codes 0..255, weights about +-0.4
        d.input_quant.scale, d.input_quant.z = 0.05, 0.0
        d.output_quant.scale, d.output_quant.z = sd * 3 / 128, 0.0
        d.sum_quant.scale, d.sum_quant.z = 1.0, 0.0
        if c["kind"] == "i8_wino":                               # |transformed input| mostly below 8 * 255
            d.wino_tinput_quant.scale, d.wino_tinput_quant.z = 0.05 * 8, 128.0
        d.sampling_kind = E.CALIBRATED
        if dw:
            d.flatting.t = 14 if ow % 14 == 0 else ow
    _check(d.setup(), "setup")

    def values(shape):
        if int8:
            return torch.randint(0, 256, shape, generator=g, device="cuda", dtype=torch.uint8)
        return torch.rand(shape, generator=g, device="cuda").mul_(2.0).sub_(1.0)

    s.x = _activations(c, c["ic"], c["h"], c["w"], values)
    w = _s8_weights(g, c["oc"], icg, c["k"]) if int8 else \
        torch.randn((c["oc"], icg, c["k"], c["k"]), generator=g, device="cuda") * math.sqrt(2.0 / (icg * c["k"] ** 2))
    if dw:
        s.w = torch.zeros(d.sizes.weights, device="cuda")
        s.w[:w.numel()] = w.reshape(-1)
    else:
        s.w = _blocked_weights(w, d.sizes.weights)
    s.b = torch.zeros(d.sizes.bias, device="cuda")
    s.b[:c["oc"]] = torch.rand(c["oc"], generator=g, device="cuda") * 0.2 - 0.1
    dt = {"u8": torch.uint8, "s8": torch.int8, "f32": torch.float32}[c["out"]]

    def residual(shape):
        if not c["sum"]:
            return torch.zeros(shape, dtype=dt, device="cuda")
        if dt == torch.float32:
            return torch.rand(shape, generator=g, device="cuda")
        return torch.randint(0, 128, shape, generator=g, device="cuda", dtype=dt)

    s.y = _activations(c, c["oc"], oh, ow, residual)
    torch.cuda.synchronize()
    _check(d.prepare(s.w, s.b), "prepare")
    if c["call"] == "host":
        s.x, s.w, s.b, s.y = (t.cpu().numpy() for t in (s.x, s.w, s.b, s.y))
    return s


def _prepare_vgg(c, seed):
    g = _rng(seed)
    s = _State()
    s.images = c["images"]
    int8 = c["kind"] == "vgg_i8"
    descs = []
    for k, (ic, oc, hw, _) in enumerate(VGG16):
        d = E.eld_conv_t()
        d.dims.n, d.dims.ic, d.dims.oc, d.dims.kh, d.dims.kw = c["n"], ic, oc, 3, 3
        d.dims.ih = d.dims.iw = d.dims.oh = d.dims.ow = hw
        d.with_relu = d.with_bias = True
        d.formats.input = E.nchw if k == 0 else E.nChw16c
        if int8:
            # images in 1/255 steps; He-initialised layers keep the second moment, so one scale serves all others
            d.data_type.input = d.data_type.output = E.u8
            d.input_quant.scale, d.output_quant.scale = (1.0 if k == 0 else 4.0) / 255.0, 4.0 / 255.0
            d.input_quant.z = d.output_quant.z = 0.0
            d.algorithm, d.sampling_kind = E.CONV_DIRECT, E.CALIBRATED
        else:
            d.algorithm, d.tile_size = E.CONV_WINOGRAD, 6
        descs.append(d)
    s.st = E.ConvStack(descs, [step for *_, step in VGG16])
    for k, (ic, oc, _, _) in enumerate(VGG16):
        w = torch.randn((oc, ic, 3, 3), generator=g, device="cuda") * math.sqrt(2.0 / (9 * ic))
        b = torch.rand(_up(oc), generator=g, device="cuda") * 0.2 - 0.1
        w = _blocked_weights(w, _up(oc) * _up(ic) * 9 + 64)      # (the library reads 64 elements of slack)
        torch.cuda.synchronize()
        _check(s.st.prepare(k, w, b), "prepare")
    shape = (c["images"], 3, 224, 224)
    if int8:
        s.x = torch.randint(0, 256, shape, generator=g, device="cuda", dtype=torch.uint8)
    else:
        s.x = torch.rand(shape, generator=g, device="cuda").mul_(2.0).sub_(1.0)
    s.y = torch.zeros((c["images"], 32, 14, 14, 16), dtype=s.x.dtype, device="cuda")
    if c["call"] == "host":
        s.x, s.y = s.x.cpu().pin_memory(), s.y.cpu().pin_memory()
    return s


def prepare(case, seed):
    s = (_prepare_vgg if case["kind"].startswith("vgg") else _prepare_conv)(case, seed)
    s.call = case["call"]
    s.stack = case["kind"].startswith("vgg")
    return s


def run(state):
    s = state
    if s.stack:
        if s.call == "host":
            rc = s.st.execute(s.y, s.x, s.images)
        else:
            rc = s.st.enqueue(s.y, s.x, torch.cuda.current_stream().cuda_stream)
    elif s.call == "stream":
        rc = s.d.enqueue(s.y, s.x, stream=torch.cuda.current_stream().cuda_stream)
    else:
        rc = E.elx_conv(s.d, s.y, s.x, s.w, s.b)
    _check(rc, "run")
    return s.y
