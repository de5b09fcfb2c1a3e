"""What this framework is timed on: whole training steps, evaluation, single layers and the extension calls, through the
entry points that a user's program calls.

Five kinds of work:
  train   ``Trainer.step``: a pinned host batch in, one integer training step, the logits back (the training loop proper);
  module  ``TiNet.forward`` + ``TiNet.backward`` on a batch that is on the GPU: the layer-by-layer API of the reference's
          own training loop, every layer updating its weights in its backward;
  eval    ``TiNet.forward`` with ``TRAINING`` off: validation and inference;
  conv / linear   one ``TiConv2d`` / ``TiLinear``: forward, backward and update of a single layer;
  compat  the calls that the reference's unmodified Python makes into its four extension modules for one
          convolution + pooling block and a classifier.
Everything is integer arithmetic with keyed random bits, so results are the same bit for bit whatever computes them.
"""
import torch

from niti_b200 import ti_torch, ti_vgg
from niti_b200.compat import cutlassconv_cuda, int8mm_cuda, int8pool_cuda
from niti_b200.trainer import Trainer

# networks of the framework's table of layer lists (ti_vgg.cifar_cfg): the reference's depths 7, 8 and 9, and two more
NETS = {"vgg7": 7, "vgg8": 8, "vgg9": 9, "vgg9_wide": "vgg9_wide", "vgg13": "vgg13"}
MEAN = (0.49139968, 0.48215827, 0.44653124)
STD = (0.24703233, 0.24348505, 0.26158768)
ROUNDINGS = ("nearest", "stochastic")


def listed():
    return [
        # the training loop: the default benchmark; one GPU's share of a global batch of 256 on eight GPUs; the largest
        # batch that the framework's configurations name
        {"name": "train vgg7 b128", "kind": "train", "net": "vgg7", "batch": 128},
        {"name": "train vgg9_wide b32", "kind": "train", "net": "vgg9_wide", "batch": 32},
        {"name": "train vgg13 b1024", "kind": "train", "net": "vgg13", "batch": 1024},
        # a program written against the reference's modules: the reference's default batch, and the last batch of an
        # epoch of 50000 images in batches of 128
        {"name": "module vgg7 b256", "kind": "module", "net": "vgg7", "batch": 256, "rounding": "nearest"},
        {"name": "module vgg9 b80", "kind": "module", "net": "vgg9", "batch": 80, "rounding": "stochastic"},
        # classifying one image as it arrives, and a validation pass
        {"name": "eval vgg7 b1", "kind": "eval", "net": "vgg7", "batch": 1},
        {"name": "eval vgg8 b500", "kind": "eval", "net": "vgg8", "batch": 500},
        # single layers: the benchmark's convolution; a ragged one; the largest of the benchmark's sweep; the classifier on
        # an odd batch; a large square matrix product
        {"name": "conv 128x32x32 128-128", "kind": "conv", "batch": 128, "h": 32, "w": 32, "cin": 128, "cout": 128,
         "rounding": "stochastic"},
        {"name": "conv 37x15x13 48-80", "kind": "conv", "batch": 37, "h": 15, "w": 13, "cin": 48, "cout": 80,
         "rounding": "nearest"},
        {"name": "linear 77x8192x10", "kind": "linear", "batch": 77, "cin": 8192, "cout": 10, "rounding": "nearest"},
        {"name": "linear 4096x4096x4096", "kind": "linear", "batch": 4096, "cin": 4096, "cout": 4096, "rounding": "nearest"},
        # the reference's own Python over the extension modules, one block of its network at batch 128
        {"name": "compat 128x16x16 256-256", "kind": "compat", "batch": 128, "h": 16, "w": 16, "cin": 256, "cout": 256},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def _draw(rng):
    kind = rng.choice(("train", "train", "module", "eval", "conv", "conv", "linear", "compat"))
    if kind in ("train", "module", "eval"):
        # batches from a handful (one for evaluation) to the largest configuration, rarely a power of two
        case = {"kind": kind, "net": rng.choice(sorted(NETS)), "batch": _log_int(rng, 1 if kind == "eval" else 4, 1024)}
        if kind == "module":
            case["rounding"] = rng.choice(ROUNDINGS)
        return case
    if kind == "conv":
        # 3x3 layers on the maps of 32x32 networks and between them; channel counts that need no padding in the reference
        return {"kind": kind, "batch": _log_int(rng, 4, 512), "h": rng.randint(4, 32), "w": rng.randint(4, 32),
                "cin": 16 * _log_int(rng, 1, 32), "cout": 16 * _log_int(rng, 1, 32), "rounding": rng.choice(ROUNDINGS)}
    if kind == "linear":
        # classifiers of 10 to 100 classes, or wide layers
        cout = rng.randint(10, 100) if rng.random() < 0.5 else 16 * _log_int(rng, 8, 256)
        return {"kind": kind, "batch": _log_int(rng, 8, 8192), "cin": 16 * _log_int(rng, 16, 512), "cout": cout,
                "rounding": rng.choice(ROUNDINGS)}
    # the reference's weight gradient takes the batch as channels, in multiples of 16; its pools are 2x2 on even maps
    hw = rng.choice((4, 8, 16, 32))
    return {"kind": kind, "batch": 16 * _log_int(rng, 1, 16), "h": hw, "w": hw, "cin": 16 * _log_int(rng, 1, 32),
            "cout": 16 * _log_int(rng, 1, 32)}


def draw(rng):
    most = max(work(c)["flops"] for c in listed())
    while True:
        case = _draw(rng)
        if work(case)["flops"] <= most:
            return case


# ---------------------------------------------------------------------------------------------------- inputs
def _bytes(gen, shape, lo=-127):
    return torch.randint(lo, 128, shape, dtype=torch.int8, device="cuda", generator=gen)


def _images(gen, batch):
    """8-bit images, scaled and normalised as the reference's loader does, and labels."""
    u8 = torch.randint(0, 256, (batch, 3, 32, 32), device="cuda", generator=gen).float()
    mean, std = (torch.tensor(v, device="cuda").view(1, 3, 1, 1) for v in (MEAN, STD))
    return ((u8 / 255.0 - mean) / std).contiguous(), torch.randint(0, 10, (batch,), device="cuda", generator=gen)


def _settings(case, seed):
    ti_torch.GRAD_BITWIDTH, ti_torch.TRAINING, ti_torch.SAMPLE_OFFSET = 5, case["kind"] != "eval", 0
    method = ti_torch.StoShift if case.get("rounding") == "stochastic" else ti_torch.RoundShift
    ti_torch.ACT_ROUND_METHOD = ti_torch.ERROR_ROUND_METHOD = method
    ti_torch.set_seed(seed, "cuda")


def _with_host_seed(seed, make):
    """make() with the host generator that the weight initialisation draws from set to the seed."""
    with torch.random.fork_rng(devices=[]):
        torch.manual_seed(seed)
        return make()


def prepare(case, seed):
    _settings(case, seed)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind, batch = case["kind"], case["batch"]
    s = {"kind": kind}
    if kind in ("train", "module", "eval"):
        s["model"] = _with_host_seed(seed, lambda: ti_vgg.TiVGG_cifar(NETS[case["net"]]))
        s["x"], s["t"] = _images(gen, batch)
        s["layers"] = s["model"].weighted_layers()
        if kind == "train":
            # a loop that is under way: batch in pinned memory, the trainer past its first (uncaptured) steps
            s["x"], s["t"] = s["x"].cpu().pin_memory(), s["t"].cpu().pin_memory()
            s["trainer"] = Trainer(s["model"], batch, "cuda:0", seed=seed)
            for _ in range(3):
                s["trainer"].step(s["x"], s["t"])
            s["trainer"].sync()
        return s
    cin, cout = case["cin"], case["cout"]
    if kind == "compat":
        h, w = case["h"], case["w"]
        f = (h // 2) * (w // 2) * cout                 # features behind the pool
        y = _bytes(gen, (batch, h, w, cout)).clamp_(min=0)
        err = _bytes(gen, (batch, h, w, cout))
        wt = _bytes(gen, (cout, 3, 3, cin))
        x = _bytes(gen, (batch, h, w, cin))
        p = int8pool_cuda.int8_pool(y, 2, 2, 0)
        s.update(x=x, w=wt, y=y, p16=p.half(), dy16=_bytes(gen, tuple(p.shape)).half(), y16=y.half(), err=err,
                 # the operands as the reference's Python arranges them: flipped filters, batch innermost
                 w_flip=torch.flip(wt, [1, 2]).transpose(0, 3).contiguous(), x_t=x.transpose(0, 3).contiguous(),
                 err_t=err.transpose(0, 3).contiguous(), feat=_bytes(gen, (batch, f)), fc=_bytes(gen, (f, 12)),
                 fc_err=_bytes(gen, (batch, 12)), fc_t=_bytes(gen, (12, f)), fc_err_t=_bytes(gen, (12, batch)))
        return s
    exp = torch.full((), -7, dtype=torch.int32, device="cuda")
    if kind == "conv":
        s["layer"] = _with_host_seed(seed, lambda: ti_torch.TiConv2d(cin, cout))
        shape_in, shape_out = (batch, case["h"], case["w"], cin), (batch, case["h"], case["w"], cout)
    else:
        s["layer"] = _with_host_seed(seed, lambda: ti_torch.TiLinear(cin, cout))
        shape_in, shape_out = (batch, cin), (batch, cout)
    s["x"], s["err"] = (_bytes(gen, shape_in), exp), (_bytes(gen, shape_out), exp)
    return s


# ---------------------------------------------------------------------------------------------------- one pass
def run(s):
    kind = s["kind"]
    if kind == "train":
        r = s["trainer"].step(s["x"], s["t"])
        return [r.out, r.exp, [l.weight for l in s["layers"]]]
    if kind == "module":
        out, exp = s["model"](s["x"])
        s["model"].backward(s["t"])
        ti_torch.advance_seed("cuda")
        return [out, exp, [l.weight for l in s["layers"]]]
    if kind == "eval":
        return list(s["model"](s["x"]))
    if kind == "compat":
        return [cutlassconv_cuda.sp_conv_optimized(s["x"], s["w"], 1, 1),
                int8pool_cuda.int8_pool(s["y"], 2, 2, 0),
                int8mm_cuda.int8_mm(s["feat"], s["fc"]),
                int8mm_cuda.int8_mm(s["fc_err"], s["fc_t"]),
                int8mm_cuda.int8_mm(s["fc_err_t"], s["feat"]),
                int8pool_cuda.int8_pool_backward(s["p16"], s["dy16"], s["y16"], 2, 2, 0),
                cutlassconv_cuda.sp_conv_optimized(s["err"], s["w_flip"], 1, 1),
                cutlassconv_cuda.sp_conv_optimized(s["x_t"], s["err_t"], 1, 1)]
    layer = s["layer"]
    y, y_exp = layer.forward(s["x"])
    e, e_exp = layer.backward(s["err"])
    return [y, y_exp, e, e_exp, layer.grad_int32acc, layer.weight]


# ---------------------------------------------------------------------------------------------------- what it cannot do without
def _net_work(case):
    """(weights, multiply-adds of the forward products, those of the first layer) of one image."""
    cfg = ti_vgg.cifar_cfg[NETS[case["net"]]]
    cin, hw, weights, macs, first = 3, 32, 0, 0, 0
    for c in cfg:
        if c == "M":
            hw //= 2
            continue
        weights += 9 * cin * c
        macs += hw * hw * 9 * cin * c
        first = first or macs
        cin = c
    f = cin * hw * hw
    return weights + 10 * f, macs + 10 * f, first


def work(case):
    kind, b = case["kind"], case["batch"]
    if kind in ("train", "module", "eval"):
        weights, macs, first = _net_work(case)
        if kind == "eval":
            return {"bytes": 4 * 3072 * b + weights + 10 * b, "flops": 2 * b * macs}
        # forward, error (not past the first layer) and weight gradient; images and labels in, weights read and written
        return {"bytes": (4 * 3072 + 8) * b + 2 * weights + 10 * b, "flops": 2 * b * (3 * macs - first)}
    cin, cout = case["cin"], case["cout"]
    if kind == "compat":
        px = b * case["h"] * case["w"]
        f = case["h"] * case["w"] // 4 * cout
        conv = 3 * px * 9 * cin * cout
        fc = 3 * b * f * 12
        # int8 operands and int32 results of the products; int8 pooling forward, fp16 in and out backward
        moved = (px * cin + 9 * cin * cout + 4 * px * cout) + (px * cout + 9 * cin * cout + 4 * px * cin)
        moved += px * (cin + cout) + 4 * 9 * cin * cout + px * cout * 5 // 4 + 2 * (px * cout * 5 // 4 + px * cout)
        moved += (b * f + 12 * f + 48 * b) + (12 * b + 12 * f + 4 * b * f) + (12 * b + b * f + 48 * f)
        return {"bytes": moved, "flops": 2 * (conv + fc)}
    rows, per = (b * case["h"] * case["w"], 9) if kind == "conv" else (b, 1)
    # activations and errors in, outputs and errors out, weights read and written, the int32 gradient out
    return {"bytes": 2 * rows * (cin + cout) + 6 * per * cin * cout, "flops": 6 * rows * per * cin * cout}


def tolerance(case):
    return "exact"
