"""Performance cases: what a user of this framework has it do, through its public entry points.

Two kinds of use are covered.

* Whole networks on host data (``excalibur_b200.host``): a pipeline is created once from a model file and then called
  with one batch of host images after the other; a pass ends when the results are back in host memory.  The networks
  are the benchmark configurations (ResNet-18-, MobileNetV2- and YOLOv5s-style) and one of the shipped
  architectures (a DB text detector), from single images to the benchmark's batches.
* Single operations on device tensors (``excalibur_b200.capi``, the C ABI): a host program that keeps its activations
  on the GPU and calls convolution, depthwise convolution and pooling itself, on its own stream.

``listed()`` are the fixed cases, ``draw(rng)`` gives others of the same ranges.
"""
import functools
import math
import types

import numpy as np
import torch

from excalibur_b200 import capi, host, model_zoo, models

NETS = {
    # builder, int8 variant exists, largest input value (graphs with an Input normalisation take 0..255 images), and per
    # image at size x size: FLOP (2 x MAC), output floats that scale with the area, output floats that do not; weights
    "resnet18": dict(build=models.resnet18, hi=1.0, size=224, flops=3.628e9, out_area=0, out_fixed=1000, weights=11678912),
    "mobilenetv2": dict(build=models.mobilenet_v2, hi=1.0, size=224, flops=0.6016e9, out_area=0, out_fixed=1000, weights=3469760),
    "yolov5s": dict(build=models.yolov5s, hi=1.0, size=640, flops=16.434e9, out_area=255 * 8400, out_fixed=0, weights=7215616),
    "det_db_resnet18": dict(build=model_zoo.det_db_resnet18, hi=255.0, size=640, flops=53.772e9, out_area=640 * 640, out_fixed=0,
                            weights=12189792),
}


def listed():
    return [
        # the headline configuration: int8 classifier, offline throughput, page-locked batches
        _net("resnet18_int8_b256", "resnet18", True, 256, 224, 224, "pinned"),
        # one image at a time from ordinary (pageable) memory: a request in a service, latency counts
        _net("resnet18_int8_b1", "resnet18", True, 1, 224, 224, "pageable"),
        # the fp16 configuration at its batch
        _net("resnet18_fp16_b64", "resnet18", False, 64, 224, 224, "pinned"),
        # a caller that holds fp16 images already (pipeline<unsigned short>), a batch that is no power of two
        _net("resnet18_int8_f16in_b100", "resnet18", True, 100, 224, 224, "pinned", "f16"),
        # depthwise-separable classifier: memory-bound kernels and pointwise GEMMs
        _net("mobilenetv2_int8_b256", "mobilenetv2", True, 256, 224, 224, "pinned"),
        # a small batch of images of an odd size, as they come out of a crop
        _net("mobilenetv2_fp16_b9_odd", "mobilenetv2", False, 9, 197, 179, "pageable"),
        # detector with three dense heads: results are larger than the input
        _net("yolov5s_fp16_b32", "yolov5s", False, 32, 640, 640, "pinned"),
        # text detector on a few landscape pages: normalisation, up-sampling, transposed convolutions
        _net("det_db_fp16_b4", "det_db_resnet18", False, 4, 480, 736, "pinned"),
        # the smallest convolution of the configurations: one 64-channel 56 x 56 image, 3x3 + ReLU
        dict(name="conv_fp16_b1", kind="conv", dtype="f16", batch=1, h=56, w=56, cin=64, cout=64, k=3, stride=1, residual=False),
        # the second convolution of a residual block: int8 in, fp16 skip, fp16 and int8 out
        dict(name="conv_int8_res_b256", kind="conv", dtype="i8", batch=256, h=28, w=28, cin=128, cout=128, k=3, stride=1,
             residual=True),
        # depthwise layer of an inverted-residual block
        dict(name="dwconv_fp16_b256", kind="dwconv", dtype="f16", batch=256, h=56, w=56, c=144, stride=1),
        # spatial pooling of a feature pyramid, odd map
        dict(name="maxpool5_fp16_b24", kind="pool", type="max", batch=24, h=45, w=39, c=256, k=5, stride=1),
    ]


def _net(name, net, int8, batch, h, w, memory, values="f32"):
    return dict(name=name, kind="net", net=net, int8=int8, batch=batch, h=h, w=w, memory=memory, input=values)


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(("net", "net", "net", "net", "conv", "conv", "dwconv", "pool"))
    if kind == "net":
        net = rng.choice(("resnet18", "resnet18", "mobilenetv2", "mobilenetv2", "yolov5s", "det_db_resnet18"))
        if net in ("resnet18", "mobilenetv2"):
            case = _net("", net, rng.random() < 0.5, _log(rng, 1, 256), rng.randint(96, 224), rng.randint(96, 224), "")
            if rng.random() < 0.5:
                case["h"] = case["w"] = 224
            if rng.random() < 0.25:                       # fp16 images; their rows are whole 8-byte groups
                case["input"], case["w"] = "f16", case["w"] // 4 * 4
        else:       # these graphs add up-sampled maps to larger ones: sides are multiples of 32
            case = _net("", net, False, _log(rng, 1, 32 if net == "yolov5s" else 8), 32 * rng.randint(10, 20), 32 * rng.randint(10, 20), "")
        case["memory"] = rng.choice(("pinned", "pageable")) if case["batch"] <= 16 else "pinned"
    elif kind == "conv":
        dtype = rng.choice(("f16", "i8"))
        step = 16 if dtype == "f16" else 32               # channels as the plans lay them out
        k = rng.choice((1, 3, 3))
        case = dict(kind="conv", dtype=dtype, batch=_log(rng, 1, 256), h=rng.randint(7, 80), w=rng.randint(7, 80),
                    cin=step * rng.randint(1, 512 // step), cout=8 * rng.randint(2, 64), k=k, stride=rng.choice((1, 1, 2)), residual=False)
        case["residual"] = case["stride"] == 1 and rng.random() < 0.4
        while _elems(case) * 4 > 1 << 30 or work(case)["flops"] > 2e11:
            case["batch"] = case["batch"] // 2
    elif kind == "dwconv":
        case = dict(kind="dwconv", dtype=rng.choice(("f16", "f16", "i8")), batch=_log(rng, 1, 256), h=rng.randint(7, 112), w=rng.randint(7, 112),
                    c=8 * _log(rng, 2, 120), stride=rng.choice((1, 1, 2)))
        while _elems(case) * 4 > 1 << 30:
            case["batch"] = case["batch"] // 2
    else:
        k, stride = rng.choice(((3, 2), (2, 2), (5, 1), (0, 1)))     # 0: the whole map
        case = dict(kind="pool", type="avg" if k == 0 else rng.choice(("max", "max", "avg")), batch=_log(rng, 1, 256), h=rng.randint(7, 112),
                    w=rng.randint(7, 112), c=8 * _log(rng, 2, 64), k=k, stride=stride)
        while _elems(case) * 4 > 1 << 30:
            case["batch"] = case["batch"] // 2
    case.pop("name", None)
    return case


def _elems(case):
    """Elements of the larger of an operation's input and output."""
    return case["batch"] * case["h"] * case["w"] * max(case.get("c", 0), case.get("cin", 0), case.get("cout", 0))


@functools.lru_cache(maxsize=None)
def _model(net, int8):
    """The model file a program has in hand: graph description and weights.  int8 scales come from a max-abs calibration
    pass of seeded images through the framework's own floating-point pipeline."""
    n = NETS[net]
    g, info = n["build"]()
    if int8:
        p = host.Pipeline(g.phai_text(), g.racy_bytes(), 0, fusion=False)
        images = np.random.default_rng(77).uniform(0, n["hi"], (4, 3, n["size"], n["size"])).astype(np.float32)
        scales = models.calibrate(p, info["conv_inputs"], images)
        p.close()
        g, info = n["build"](act_scales=scales)
    return g.phai_text(), g.racy_bytes(), info.get("outputs") or [info["output"]]


def prepare(case, seed):
    return {"net": _prepare_net, "conv": _prepare_conv, "dwconv": _prepare_dwconv, "pool": _prepare_pool}[case["kind"]](case, seed)


def run(state):
    return state.run()


def _prepare_net(case, seed):
    phai, racy, outputs = _model(case["net"], case["int8"])
    N, H, W = case["batch"], case["h"], case["w"]
    gen = torch.Generator("cuda").manual_seed(seed)
    x = torch.rand((N, 3, H, W), generator=gen, device="cuda").mul_(NETS[case["net"]]["hi"])
    f16 = case["input"] == "f16"
    x = (x.half() if f16 else x).cpu()
    pinned = case["memory"] == "pinned"
    if pinned:
        x = x.pin_memory()
    a = x.numpy()
    pipe = (host.PipelineF16 if f16 else host.Pipeline)(phai, racy, 0)
    s = types.SimpleNamespace(pipe=pipe, x=x)
    if f16:
        def call():
            pipe.forward_ptr(x.data_ptr(), N, 3, H, W)
            return {n: pipe.get(n) for n in outputs}
    elif pinned:        # large batches: results are read where the pipeline put them
        def call():
            pipe.forward_ptr(x.data_ptr(), N, 3, H, W)
            return {n: _view(pipe, n) for n in outputs}
    else:
        def call():
            return pipe.forward(a)
    s.run = call
    return s


def _view(pipe, name):
    """A result in the pipeline's own host memory, which lives as long as the pipeline does."""
    t = torch.from_numpy(pipe.output_view(name))
    t.pipe = pipe
    return t


def _activations(shape, gen, dtype):
    """Activations behind a ReLU, as the layers meet them; int8: quantised to the whole range."""
    x = torch.randn(shape, generator=gen, device="cuda").clamp_(0, 4)
    return (x * (127.0 / 4)).round_().to(torch.int8) if dtype == "i8" else x.half()


def _prepare_conv(case, seed):
    N, H, W, cin, cout, k, stride = (case[n] for n in ("batch", "h", "w", "cin", "cout", "k", "stride"))
    r = np.random.default_rng(seed)
    gen = torch.Generator("cuda").manual_seed(seed)
    ctx = capi.Context(0)
    w = (r.standard_normal((cout, cin, k, k), np.float32) * np.float32(math.sqrt(2.0 / (cin * k * k))))
    b = r.standard_normal(cout).astype(np.float32) * np.float32(0.1)
    i8 = case["dtype"] == "i8"
    res = case["residual"]
    d = capi.make_conv_desc(N, H, W, cin, cout, k, stride, k // 2, capi.EXB_I8 if i8 else capi.EXB_F16,
                            capi.EXB_I8 if i8 and not res else capi.EXB_F16, capi.EXB_I8 if i8 and res else -1, res=res, act=capi.ACT_RELU,
                            out_scale=127.0 / 6, out2_scale=127.0 / 6)
    if i8:
        wq, ws = models.quantize_weights(w)
        packed = capi.ConvWeights(ctx, d, wq, b, ws, 127.0 / 4)
    else:
        packed = capi.ConvWeights(ctx, d, w, b)
    x = _activations((N, H, W, cin), gen, case["dtype"])
    oh, ow = capi.conv_out_dims(d)
    skip = _activations((N, oh, ow, cout), gen, "f16") if res else None

    def call():
        y, y2 = capi.conv2d(ctx, d, x, packed, residual=skip)
        return [y] if y2 is None else [y, y2]
    return types.SimpleNamespace(ctx=ctx, packed=packed, run=call)


def _prepare_dwconv(case, seed):
    N, H, W, c, stride = (case[n] for n in ("batch", "h", "w", "c", "stride"))
    r = np.random.default_rng(seed)
    gen = torch.Generator("cuda").manual_seed(seed)
    ctx = capi.Context(0)
    w = r.standard_normal((c, 3, 3)).astype(np.float32) * np.float32(math.sqrt(2.0 / 9))
    b = r.standard_normal(c).astype(np.float32) * np.float32(0.1)
    # fp16 maps, or fp16 in and int8 out: the layer in front of an int8 projection
    d = capi.make_dw_desc(N, H, W, c, 3, stride, 1, capi.EXB_F16, capi.EXB_I8 if case["dtype"] == "i8" else capi.EXB_F16, capi.ACT_RELU6,
                          out_scale=127.0 / 6)
    packed = capi.DwWeights(ctx, d, w, b)
    x = _activations((N, H, W, c), gen, "f16")
    return types.SimpleNamespace(ctx=ctx, packed=packed, run=lambda: capi.dwconv2d(ctx, d, x, packed))


def _prepare_pool(case, seed):
    N, H, W, c, k, stride = (case[n] for n in ("batch", "h", "w", "c", "k", "stride"))
    gen = torch.Generator("cuda").manual_seed(seed)
    ctx = capi.Context(0)
    d = capi.make_pool_desc(N, H, W, c, 0 if case["type"] == "max" else 1, k or 1, stride, (k - 1) // 2 if k else 0, global_pool=k == 0)
    x = _activations((N, H, W, c), gen, "f16")
    return types.SimpleNamespace(ctx=ctx, run=lambda: capi.pool2d(ctx, d, x)[0])


def work(case):
    N, H, W = case["batch"], case["h"], case["w"]
    if case["kind"] == "net":
        n = NETS[case["net"]]
        area = H * W / n["size"] ** 2
        b = 2 if case["input"] == "f16" else 4
        return {"bytes": N * (3 * H * W + n["out_area"] * area + n["out_fixed"]) * b + n["weights"] * (1 if case["int8"] else 2),
                "flops": N * n["flops"] * area}
    k, s = case["k"] if case["kind"] != "dwconv" else 3, case["stride"]
    pad = (k - 1) // 2
    oh, ow = ((H + 2 * pad - k) // s + 1, (W + 2 * pad - k) // s + 1) if k else (1, 1)
    if case["kind"] == "conv":
        e = 1 if case["dtype"] == "i8" else 2
        per_out = (2 + 2 + e % 2 if case["residual"] else e)      # fp16 skip, fp16 result (and its int8 copy), or one result
        return {"bytes": N * H * W * case["cin"] * e + N * oh * ow * case["cout"] * per_out + case["cout"] * case["cin"] * k * k * e,
                "flops": 2.0 * N * oh * ow * case["cout"] * case["cin"] * k * k}
    c = case["c"]
    if case["kind"] == "dwconv":
        return {"bytes": N * c * (H * W * 2 + oh * ow * (1 if case["dtype"] == "i8" else 2)) + c * 9 * 4, "flops": 2.0 * N * c * oh * ow * 9}
    return {"bytes": N * c * (H * W + oh * ow) * 2, "flops": float(N * c * (oh * ow * k * k if k else H * W))}


def tolerance(case):
    if case["kind"] == "net":
        # fp16 (int8) activations rounded after each of some twenty layers
        return {"rel": 2e-2, "max": 0.3} if case["int8"] else {"rel": 5e-3, "max": 0.1}
    if case["kind"] == "pool" and case["type"] == "max":
        return "exact"
    # 32-bit sums, results rounded once to fp16 (2^-11); int8 results may differ where a value lies at a rounding tie
    return {"rel": 5e-4, "max": 4e-3, "differ": 1e-3}
