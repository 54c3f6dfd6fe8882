"""Timed workloads of the convolution library: what programs that use it have it do.

Every case goes through the public entry points of ``theano_b200.shim``:

* ``call``:  what one Theano op does in ``perform``: NCHW numpy arrays in, numpy arrays out.
* ``layer``: one convolution layer on channels-last tensors that stay in HBM, forward alone
  (bias and ReLU in the epilogue) or forward + gradInputs + gradWeights.
* ``stack``: forward pass of the VGG-16 stack (bias, ReLU and pooling in the epilogues) with the
  feature maps of every layer as its result, issued call by call or replayed as a captured graph.
* ``block``: backward pass of a pooled convolution block, from the pooled gradient to the
  gradients of filters, bias and input.
* ``step``:  one training step of all ResNet-50 convolutions: filter packing, forward pass and
  backward pass with the filter gradients in one flat float32 buffer, replayed as a graph.

Layer shapes are those of ``theano_b200.workloads`` and of the test matrix, or generic ones.
"""
import math

import numpy as np
import torch

from theano_b200 import hostlogic, shim
from theano_b200 import workloads as WL

DTYPES = {"f32": (np.float32, torch.float32, 4), "f16": (np.float16, torch.float16, 2)}


def _layer(kind, name, dtype, N, C, K, H, W, k=3, s=1, d=1, g=1, pad="half", train=True, **more):
    return dict(kind=kind, name=name, dtype=dtype, N=N, C=C, K=K, H=H, W=W, k=k, s=s, d=d, g=g, pad=pad,
                train=train, **more)


def listed():
    return [
        # the smallest call: a Theano function's forward convolution of a 16-image batch
        _layer("call", "call_fwd_small", "f32", 16, 3, 64, 32, 32, train=False),
        # a small training function with ragged channel counts and 'valid' borders: all three ops
        _layer("call", "call_train_ragged", "f32", 100, 20, 50, 12, 12, k=5, pad="valid"),
        # an ordinary training layer whose arrays (26 MB each) live on the host
        _layer("call", "call_train_large", "f32", 64, 128, 128, 28, 28),
        # a training layer at a small batch: launches and host work count
        _layer("layer", "layer_f16_small", "f16", 8, 64, 64, 28, 28),
        # the single-layer benchmark: 3x3, 256 channels at 14x14, batch 128
        _layer("layer", "layer_f32_3x3_256", "f32", 128, 256, 256, 14, 14),
        # a down-sampling layer of the geometry sweep
        _layer("layer", "layer_f32_stride2", "f32", 256, 64, 128, 56, 56, s=2),
        # the grouped layer of the geometry sweep
        _layer("layer", "layer_f32_groups32", "f32", 256, 256, 256, 28, 28, g=32),
        # odd sizes all over: channels off every tile, images that are not square
        _layer("layer", "layer_f16_ragged", "f16", 37, 100, 75, 27, 33, k=5),
        # serving one image: the whole stack as one graph replay
        dict(kind="stack", name="stack_f32_one_image", dtype="f32", N=1, H=224, graph=True),
        # the VGG-16 benchmark: 64 images, calls issued one by one
        dict(kind="stack", name="stack_f32_batch64", dtype="f32", N=64, H=224, graph=False),
        # backward pass of a pooled block of that network on resident activations
        dict(kind="block", name="block_f32_backward", dtype="f32", N=64, C=64, K=128, H=112),
        # the headline benchmark: the training step of the 53 ResNet-50 convolutions
        dict(kind="step", name="step_f16_batch256", dtype="f16", N=256),
    ]


# ---- drawn cases -----------------------------------------------------------------------------
def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _channels(rng, lo, hi):
    """Multiples of 16 as often as odd counts."""
    c = _log(rng, lo, hi)
    return max(16, c // 16 * 16) if c >= 16 and rng.random() < 0.5 else c


def _draw_layer(rng, kind):
    dtype = rng.choice(["f32", "f16"])
    k = rng.choice([1, 3, 3, 3, 5, 7])
    s, d = rng.choice([1, 1, 1, 2]), rng.choice([1, 1, 1, 2]) if k > 1 else 1
    pad = rng.choice(["half", "half", "valid", "full", "asym"]) if k > 1 else rng.choice(["half", "valid"])
    H = max(_log(rng, 6, 120), (k - 1) * d + 1)
    W = H if rng.random() < 0.6 else max(_log(rng, 6, 120), (k - 1) * d + 1)
    g = 1
    if rng.random() < 0.15:                 # whole 16-byte pieces per group, which the device layout asks for
        g = rng.choice([2, 4, 8, 32])
        C, K = g * 8 * _log(rng, 1, 8), g * 8 * _log(rng, 1, 8)
    else:
        C, K = _channels(rng, 1, 1024), _channels(rng, 4, 1024)
    N = _log(rng, 1, 256)
    case = _layer(kind, "", dtype, N, C, K, H, W, k, s, d, g, pad, train=rng.random() < 0.7)
    del case["name"]
    most_bytes, most_flops = (1e8, 2e11) if kind == "call" else (2e9, 1e12)
    while True:                             # fewer images, then fewer channels, until the pass is affordable
        w = work(case)
        if w["bytes"] <= most_bytes and w["flops"] <= most_flops:
            return case
        if case["N"] > 1:
            case["N"] = (case["N"] + 1) // 2
        elif g == 1:
            case["C"], case["K"] = (case["C"] + 1) // 2, (case["K"] + 1) // 2
        else:
            case["H"], case["W"] = max(8, case["H"] // 2), max(8, case["W"] // 2)


def draw(rng):
    kind = rng.choices(["call", "layer", "stack", "block", "step"], [25, 40, 15, 10, 10])[0]
    if kind in ("call", "layer"):
        return _draw_layer(rng, kind)
    if kind == "stack":
        H = 32 * rng.randint(1, 7)
        N = _log(rng, 1, max(1, min(128, 64 * 224 * 224 // (H * H))))
        return dict(kind="stack", dtype=rng.choice(["f32", "f16"]), N=N, H=H, graph=rng.random() < 0.5)
    if kind == "block":
        H = 2 * _log(rng, 5, 56)
        N = _log(rng, 1, max(1, min(128, 64 * 112 * 112 // (H * H))))
        return dict(kind="block", dtype=rng.choice(["f32", "f16"]), N=N, C=_channels(rng, 16, 256),
                    K=_channels(rng, 16, 256), H=H)
    dtype = rng.choice(["f16", "f16", "f32"])
    return dict(kind="step", dtype=dtype, N=_log(rng, 2, 192 if dtype == "f16" else 64))


# ---- geometry --------------------------------------------------------------------------------
def _border(case):
    return ((1, 2), (2, 1)) if case["pad"] == "asym" else case["pad"]


def _kwargs(case):
    return dict(border_mode=_border(case), subsample=(case["s"],) * 2, filter_dilation=(case["d"],) * 2,
                num_groups=case["g"], filter_flip=True)


def _shapes(case):
    """(x, w, y) shapes of a 'call' or 'layer' case."""
    xs = (case["N"], case["C"], case["H"], case["W"])
    ws = (case["K"], case["C"] // case["g"], case["k"], case["k"])
    kw = _kwargs(case)
    ys, _ = hostlogic.forward_shape(xs, ws, kw["border_mode"], kw["subsample"], kw["filter_dilation"], case["g"])
    return xs, ws, ys


def _stack_layers(case):
    """The layers of the VGG-16 stack on H x H images, one dict per layer instance."""
    return [dict(lay, H=lay["H"] * case["H"] // 224) for lay in WL.VGG16 for _ in range(lay["n"])]


def work(case):
    es = DTYPES[case["dtype"]][2]
    if case["kind"] in ("call", "layer"):
        xs, ws, ys = _shapes(case)
        x, w, y = (math.prod(v) for v in (xs, ws, ys))
        passes = 3 if case["train"] else 1
        return {"bytes": es * (x + w + y) * (2 if case["train"] else 1),
                "flops": passes * hostlogic.conv_flops(xs, ws, ys)}
    if case["kind"] == "stack":
        layers = _stack_layers(case)
        n, h = case["N"], case["H"]
        maps = sum(l["K"] * (l["H"] // (2 if l["pool"] else 1)) ** 2 for l in layers)
        return {"bytes": es * (n * 3 * h * h + n * maps + sum(l["K"] * (l["C"] * 9 + 1) for l in layers)),
                "flops": sum(WL.flops(l, n) for l in layers)}
    if case["kind"] == "block":
        n, c, k, h = case["N"], case["C"], case["K"], case["H"]
        # x and dx, y, pooled output and its gradient, filters and their gradient, bias gradient
        return {"bytes": es * (2 * n * c * h * h + n * k * h * h + 2 * n * k * (h // 2) ** 2 + 2 * 9 * c * k + k),
                "flops": 2 * 2 * n * k * c * 9 * h * h}
    layers = WL.resnet50_network()
    total = 0
    for lay in layers:
        x, w, y = (math.prod(v) for v in WL.shapes(lay, case["N"]))
        total += es * (2 * x + w + 2 * y) + 4 * w
    return {"bytes": total, "flops": 3 * sum(WL.flops(l, case["N"]) for l in layers)}


def tolerance(case):
    """float32 multiplies in TF32 (10 mantissa bits), float16 results are rounded to 10 bits; both
    accumulate in float32.  The stack passes its rounding errors through thirteen layers."""
    return {"rel": 5e-3 if case["kind"] == "stack" else 1e-3}


# ---- inputs ----------------------------------------------------------------------------------
class _Maker(object):
    """Seeded tensors on the GPU and the framework's view of them."""

    def __init__(self, case, seed):
        self.ctx = shim.get_context(0)
        self.np_dtype, self.dtype, self.es = DTYPES[case["dtype"]]
        self.gen = torch.Generator(device="cuda")
        self.gen.manual_seed(seed)
        self.keep = []                      # storage of the device tensors handed out

    def normal(self, shape, scale=1.0, dtype=None):
        t = torch.empty(shape, dtype=dtype or self.dtype, device="cuda")
        return t.normal_(0.0, scale, generator=self.gen)

    def image(self, shape, scale=None, storage=None):
        """(channels-last storage, DeviceTensor) of an NCHW shape: N(0, scale^2) with zeros in the pad
        channels, or, without a scale, an output buffer."""
        n, c, h, w = shape
        cp = self.ctx.padded_channels(c, self.np_dtype)
        t = torch.zeros((n, h, w, cp), dtype=self.dtype, device="cuda") if storage is None else storage.view(n, h, w, cp)
        if scale is not None:
            t.normal_(0.0, scale, generator=self.gen)
            t[..., c:] = 0
        return t, self.wrap(t, shape, "nhwc")

    def wrap(self, t, shape, layout="nchw", np_dtype=None):
        self.keep.append(t)
        return shim.DeviceTensor(self.ctx, shape, np_dtype or self.np_dtype, layout, _ptr=t.data_ptr())

    def filters(self, shape):
        t = self.normal(shape, math.sqrt(2.0 / (shape[1] * shape[2] * shape[3])))
        self.ctx.filters_changed(t.data_ptr())      # this memory may have held the filters of another program
        return t, self.wrap(t, shape)

    def dy_scale(self):
        return 0.1 if self.dtype == torch.float16 else 1.0


def prepare(case, seed):
    m = _Maker(case, seed)
    state = {"call": _prepare_call, "layer": _prepare_layer, "stack": _prepare_stack, "block": _prepare_block,
             "step": _prepare_step}[case["kind"]](case, m)
    state.update(case=case, kind=case["kind"], ctx=m.ctx, keep=m.keep)
    torch.cuda.synchronize()
    return state


def _prepare_call(case, m):
    xs, ws, ys = _shapes(case)
    host = lambda t: t.cpu().numpy()  # noqa: E731
    st = dict(x=host(m.normal(xs)), w=host(m.filters(ws)[0]), kw=_kwargs(case), bias=None)
    if case["train"]:
        st["dy"] = host(m.normal(ys, m.dy_scale()))
    else:
        st["bias"] = host(m.normal((ws[0],), 0.1))
    return st


def _prepare_layer(case, m):
    xs, ws, ys = _shapes(case)
    st = dict(x=m.image(xs, 1.0)[1], w=m.filters(ws)[1], kw=_kwargs(case), hw=xs[2:], bias=None, out={})
    st["out"]["y"], st["y"] = m.image(ys)
    if case["train"]:
        st["dy"] = m.image(ys, m.dy_scale())[1]
        st["out"]["dx"], st["dx"] = m.image(xs)
        st["out"]["dw"] = torch.zeros(ws, dtype=m.dtype, device="cuda")
        st["dw"] = m.wrap(st["out"]["dw"], ws)
    else:
        st["bias"] = m.wrap(m.normal((ws[0],), 0.1), (1, ws[0], 1, 1))
    return st


def _prepare_stack(case, m):
    """The network a serving program keeps: filters packed once, activation buffers, and for `graph`
    the captured pass."""
    n = case["N"]
    x, cur = m.image((n, 3, case["H"], case["H"]))
    x.uniform_(0.0, 1.0, generator=m.gen)
    x[..., 3:] = 0
    layers, descs, ptrs, outs = [], [], [], []
    for lay in _stack_layers(case):
        ws = (lay["K"], lay["C"], 3, 3)
        w = m.filters(ws)[1]
        b = m.wrap(m.normal((lay["K"],), 0.05), (1, lay["K"], 1, 1))
        h = lay["H"] // 2 if lay["pool"] else lay["H"]
        outs.append(m.image((n, lay["K"], h, h)))
        y = outs[-1][1]
        full = m.image((n, lay["K"], lay["H"], lay["H"]))[1] if lay["pool"] else None
        layers.append(dict(x=cur, w=w, b=b, y=y, pool=lay["pool"], full=full, fused=lay["pool"]))
        descs.append(shim.layer_desc(cur.shape, ws, border_mode=(1, 1), dtype=m.np_dtype))
        ptrs.append(w.ptr)
        cur = y
    torch.cuda.synchronize()
    m.ctx.prepack(descs, ptrs, 1)
    for lay in layers:                      # where the epilogue cannot pool, pooling is a call of its own
        try:
            _stack_layer(lay)
        except shim.B200Error:
            lay["fused"] = False
            _stack_layer(lay)
    m.ctx.sync()
    graph = m.ctx.capture(lambda: [_stack_layer(lay) for lay in layers]) if case["graph"] else None
    return dict(layers=layers, graph=graph, out=[t for t, _ in outs])


def _stack_layer(lay):
    pool_after = lay["pool"] and not lay["fused"]
    shim.device_conv2d(lay["x"], lay["w"], border_mode=(1, 1), bias=lay["b"], relu=True, pool=lay["fused"],
                       out=lay["full"] if pool_after else lay["y"])
    if pool_after:
        shim.device_maxpool2x2(lay["full"], out=lay["y"])


def _prepare_block(case, m):
    """What the backward pass finds: the input, the rectified activations of the forward pass, their
    2x2 maxima and the gradient of those."""
    n, c, k, h = case["N"], case["C"], case["K"], case["H"]
    st = dict(out={}, h=h)
    st["x"] = m.image((n, c, h, h), 1.0)[1]
    y, st["y"] = m.image((n, k, h, h), 1.0)
    y.clamp_(min=0)
    p, st["p"] = m.image((n, k, h // 2, h // 2))
    p.copy_(y.view(n, h // 2, 2, h // 2, 2, y.shape[3]).amax(dim=(2, 4)))
    st["gp"] = m.image((n, k, h // 2, h // 2), m.dy_scale())[1]
    st["w"] = m.filters((k, c, 3, 3))[1]
    st["gy"], st["mask"] = m.image((n, k, h, h))[1], m.image((n, k, h, h))[1]
    st["out"]["dx"], st["dx"] = m.image((n, c, h, h))
    st["out"]["dw"] = torch.zeros((k, c, 3, 3), dtype=m.dtype, device="cuda")
    st["dw"] = m.wrap(st["out"]["dw"], (k, c, 3, 3))
    return st


def _prepare_step(case, m):
    """Per layer its own x, y, dy, dx in HBM, all filter gradients in one flat float32 buffer (what a
    data-parallel program all-reduces), the step captured as one graph."""
    net = WL.resnet50_network()
    shapes = [WL.shapes(lay, case["N"]) for lay in net]

    def flat(which, scale=None):
        """One storage for a tensor of every layer and the layers' views of it."""
        sizes = [v[0] * v[2] * v[3] * m.ctx.padded_channels(v[1], m.np_dtype) for v in (s[which] for s in shapes)]
        buf = torch.zeros(sum(sizes), dtype=m.dtype, device="cuda")
        return buf, [m.image(s[which], scale, part)[1] for s, part in zip(shapes, buf.split(sizes))]

    _, X = flat(0, 1.0)
    _, DY = flat(2, m.dy_scale())
    y, Y = flat(2)
    dx, DX = flat(0)
    W = [m.filters(s[1])[1] for s in shapes]
    sizes = [math.prod(s[1]) for s in shapes]
    dw = torch.zeros(sum(sizes), dtype=torch.float32, device="cuda")
    DW = [m.wrap(part, s[1], np_dtype=np.float32) for s, part in zip(shapes, dw.split(sizes))]
    kw = [WL.conv_kwargs(lay) for lay in net]
    descs = [shim.layer_desc(s[0], s[1], dtype=m.np_dtype, **k) for s, k in zip(shapes, kw)]
    ptrs = [w.ptr for w in W]
    ctx = m.ctx

    def step():
        ctx.prepack(descs, ptrs)
        for i in range(len(net)):
            shim.device_conv2d(X[i], W[i], out=Y[i], **kw[i])
        for i in reversed(range(len(net))):
            shim.device_grad_weights(X[i], DY[i], shapes[i][1][2:], out=DW[i], **kw[i])
            shim.device_grad_inputs(W[i], DY[i], shapes[i][0][2:], out=DX[i], **kw[i])

    torch.cuda.synchronize()
    step()                                  # kernels are chosen and the memory pool is warm before the capture
    ctx.sync()
    return dict(graph=ctx.capture(step), out={"y": y, "dx": dx, "dw": dw})


# ---- one pass --------------------------------------------------------------------------------
def run(state):
    return {"call": _run_call, "layer": _run_layer, "stack": _run_stack, "block": _run_block,
            "step": _run_step}[state["kind"]](state)


def _run_call(st):
    x, w, kw = st["x"], st["w"], st["kw"]
    if "dy" not in st:
        return shim.conv2d_forward(x, w, bias=st["bias"], relu=True, **kw)
    y = shim.conv2d_forward(x, w, **kw)
    dw = shim.conv2d_grad_weights(x, st["dy"], w.shape[2:], **kw)
    dx = shim.conv2d_grad_inputs(w, st["dy"], x.shape[2:], **kw)
    return {"y": y, "dw": dw, "dx": dx}


def _run_layer(st):
    kw = st["kw"]
    if "dy" not in st:
        shim.device_conv2d(st["x"], st["w"], bias=st["bias"], relu=True, out=st["y"], **kw)
        return st["out"]
    shim.device_conv2d(st["x"], st["w"], out=st["y"], **kw)
    shim.device_grad_weights(st["x"], st["dy"], st["w"].shape[2:], out=st["dw"], **kw)
    shim.device_grad_inputs(st["w"], st["dy"], st["hw"], out=st["dx"], **kw)
    return st["out"]


def _run_stack(st):
    if st["graph"] is not None:
        st["graph"].launch()
    else:
        for lay in st["layers"]:
            _stack_layer(lay)
    return st["out"]


def _run_block(st):
    gy = shim.device_maxpool2x2_grad(st["y"], st["p"], st["gp"], out=st["gy"])
    mask = shim.device_elementwise("sgn", st["y"], out=st["mask"])
    gz = shim.device_elementwise("mul", gy, mask, out=gy)
    db = shim.device_channel_sum(gz)
    shim.device_grad_weights(st["x"], gz, (3, 3), border_mode=(1, 1), out=st["dw"])
    shim.device_grad_inputs(st["w"], gz, (st["h"], st["h"]), border_mode=(1, 1), out=st["dx"])
    return dict(st["out"], db=db)


def _run_step(st):
    st["graph"].launch()
    return st["out"]
