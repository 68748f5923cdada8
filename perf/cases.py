"""Work that users of this framework have it do, as cases that can be timed and compared.

Two kinds of program use it.  One loads a ``.one`` model into a ``Net`` for a fixed batch and runs
inference after inference: device-resident input, ``run`` and ``sync`` (a batch server), or one call from
host memory to host memory (an interactive client).  The other keeps the graph itself and calls the Conv,
Gemm and MatMul operators through the drop-in libraries on tensors of its own.

The models are the synthetic ones of ``onenew_b200.models`` with the weights of one fixed seed (a program
loads the same file each time), built as a user gets them from the constructor: no tile search, default
folding, CUDA graph on.  The inputs are drawn from the seed.
"""
import functools

import torch

from onenew_b200 import abi, models, net, ops, quant

WORKSPACE = 1 << 30    # scratch of one Net: enough for the largest stem of the ranges below
CUDA = "cuda"


def listed():
    return [
        # --- operators of a host that keeps its own graph (drop-in eval, fp32 in and out, tf32 products)
        # the single-operator configuration: one 3x3 conv of a residual block on one image
        {"name": "conv_64x56x56_b1", "kind": "conv", "n": 1, "c": 64, "h": 56, "w": 56, "oc": 64, "k": 3, "s": 1, "p": 1, "act": "relu"},
        # the classifier of ResNet-50 on a full batch
        {"name": "gemm_256x2048x1000", "kind": "gemm", "m": 256, "k": 2048, "n": 1000},
        # attention scores of a transformer block: both operands are activations
        {"name": "matmul_24x197x64x197", "kind": "matmul", "b": 24, "m": 197, "k": 64, "n": 197, "shared": False},
        # --- ResNet-50
        # one photo from host memory to host memory: the interactive client
        {"name": "resnet50_f16_b1_host", "kind": "resnet50", "prec": "f16", "batch": 1, "image": 224, "host": True},
        # what each of eight GPUs gets of a batch of 256
        {"name": "resnet50_f16_b32", "kind": "resnet50", "prec": "f16", "batch": 32, "image": 224, "host": False},
        # the throughput benchmark
        {"name": "resnet50_f16_b256", "kind": "resnet50", "prec": "f16", "batch": 256, "image": 224, "host": False},
        # the library's default precision, a batch that is no round number and smaller images
        {"name": "resnet50_tf32_b61_i192", "kind": "resnet50", "prec": "tf32", "batch": 61, "image": 192, "host": False},
        # --- ViT-Tiny/16
        {"name": "vit_tf32_b1", "kind": "vit", "prec": "tf32", "batch": 1, "image": 224, "dim": 192, "host": False},
        {"name": "vit_tf32_b256", "kind": "vit", "prec": "tf32", "batch": 256, "image": 224, "dim": 192, "host": False},
        # --- the int8 backbone of a detector: one video frame, and a batch of them
        {"name": "yolo_int8_b1", "kind": "yolo", "prec": "tf32", "batch": 1, "image": 640, "host": False},
        {"name": "yolo_int8_b64", "kind": "yolo", "prec": "tf32", "batch": 64, "image": 640, "host": False},
    ]


def _log(rng, lo, hi):
    """A whole number from lo to hi, spread over its logarithm."""
    return max(lo, min(hi, round(lo * (hi / lo) ** rng.random())))


def draw(rng):
    kind = rng.choice(["op", "op", "resnet50", "resnet50", "vit", "yolo"])
    if kind == "op":
        kind = rng.choice(["conv", "conv", "gemm", "matmul"])
    if kind == "conv":
        k = rng.choice([1, 3, 3, 5, 7])
        h = _log(rng, max(7, k), 112)
        case = {"kind": "conv", "n": _log(rng, 1, 32), "c": rng.choice([3, 16, 24, 32, 64, 96, 128, 256, 512]), "h": h, "w": rng.choice([h, h, _log(rng, max(7, k), 112)]),
                "oc": _log(rng, 8, 512), "k": k, "s": rng.choice([1, 1, 2]), "p": k // 2, "act": rng.choice(["relu", "relu", "silu", "none"])}
        while case["n"] > 1 and _conv_flops(case) > 6e10:
            case["n"] //= 2
        while case["c"] > 64 and _conv_flops(case) > 6e10:
            case["c"] //= 2
        return case
    if kind == "gemm":
        return {"kind": "gemm", "m": _log(rng, 1, 1024), "k": _log(rng, 64, 4096), "n": _log(rng, 10, 4096)}
    if kind == "matmul":
        shared = rng.random() < 0.5    # a linear layer, or a product of two activations
        return {"kind": "matmul", "b": _log(rng, 1, 96), "m": _log(rng, 16, 257), "k": _log(rng, 32, 768), "n": _log(rng, 32, 768), "shared": shared}
    host = rng.random() < 0.25
    if kind == "resnet50":
        image = rng.choice([128, 160, 192, 224, 256, rng.randrange(96, 257)])
        return {"kind": kind, "prec": rng.choice(["f16", "f16", "tf32"]), "batch": _log(rng, 1, min(128, 128 * 224 * 224 // image ** 2)), "image": image, "host": host}
    if kind == "vit":
        dim = rng.choice([192, 192, 384])
        return {"kind": kind, "prec": "tf32", "batch": _log(rng, 1, 192 if dim == 192 else 64), "image": 16 * rng.randrange(6, 16), "dim": dim, "host": host}
    image = 32 * rng.randrange(10, 21)
    return {"kind": "yolo", "prec": "tf32", "batch": _log(rng, 1, 48), "image": image, "host": host}


# ------------------------------------------------------------------------------------------ inputs
@functools.lru_cache(maxsize=4)
def _model_file(kind, image, dim):
    """The model as a program finds it on disk."""
    if kind == "resnet50":
        return models.build_resnet50(image=image).tobytes()
    if kind == "vit":
        return models.build_vit(image=image, dim=dim, heads=dim // 64, mlp=4 * dim).tobytes()
    fp32 = models.build_yolo_backbone(models.yolo_backbone_weights(), image=image).tobytes()
    return quant.quantize_model(fp32, _yolo_scales())


@functools.lru_cache(maxsize=1)
def _yolo_scales():
    """Activation scales of the backbone: calibrated once, whatever size it is run at later."""
    fp32 = models.build_yolo_backbone(models.yolo_backbone_weights(), image=320).tobytes()
    return quant.calibrate_mse(fp32, models.yolo_input(4, image=320))


class _DeviceArray:
    """A Net's own device buffer, for torch to look at; the tensor keeps this object, and so the Net, alive."""

    def __init__(self, owner, is_output):
        self.owner = owner
        shape = (owner.outputs if is_output else owner.inputs)[0][1]
        self.__cuda_array_interface__ = {"data": (owner.io_ptr(is_output), False), "shape": tuple(shape), "typestr": "<f4", "version": 3}


def _images(case, gen):
    x = torch.rand((case["batch"], 3, case["image"], case["image"]), generator=gen, device=CUDA)
    if case["kind"] == "resnet50":
        mean = torch.tensor(models.IMAGENET_MEAN, device=CUDA).view(1, 3, 1, 1)
        std = torch.tensor(models.IMAGENET_STD, device=CUDA).view(1, 3, 1, 1)
        x = (x - mean) / std
    return x


def prepare(case, seed):
    gen = torch.Generator(device=CUDA).manual_seed(seed)
    if case["kind"] == "conv":
        x = torch.rand((case["n"], case["c"], case["h"], case["w"]), generator=gen, device=CUDA) * 2 - 1
        w = torch.randn((case["oc"], case["c"], case["k"], case["k"]), generator=gen, device=CUDA) * 0.05
        b = torch.randn((case["oc"],), generator=gen, device=CUDA) * 0.01
        lut = torch.from_numpy(net.activation_table("silu")).to(CUDA) if case["act"] == "silu" else None
        act = {"none": abi.NOT_ACT, "relu": abi.RELU, "silu": abi.SILU}[case["act"]]
        return {"kind": "conv", "x": x, "w": w, "b": b, "strides": (case["s"],) * 2, "pads": (case["p"],) * 4, "act": act, "lut": lut}
    if case["kind"] == "gemm":
        a = torch.randn((case["m"], case["k"]), generator=gen, device=CUDA)
        w = torch.randn((case["n"], case["k"]), generator=gen, device=CUDA) * 0.05
        b = torch.randn((case["n"],), generator=gen, device=CUDA) * 0.01
        return {"kind": "gemm", "a": a, "w": w, "b": b}
    if case["kind"] == "matmul":
        a = torch.randn((case["b"], case["m"], case["k"]), generator=gen, device=CUDA)
        shape = (case["k"], case["n"]) if case["shared"] else (case["b"], case["k"], case["n"])
        return {"kind": "matmul", "a": a, "b": torch.randn(shape, generator=gen, device=CUDA) * 0.05}
    n = net.Net(_model_file(case["kind"], case["image"], case.get("dim", 0)), batch=case["batch"], precision=case["prec"], workspace_bytes=WORKSPACE)
    x = _images(case, gen)
    if case["host"]:
        return {"kind": "host", "net": n, "x": x.cpu().pin_memory(), "y": torch.empty(n.outputs[0][1], dtype=torch.float32).pin_memory()}
    torch.as_tensor(_DeviceArray(n, False), device=CUDA).copy_(x)
    torch.cuda.synchronize()
    return {"kind": "device", "net": n, "y": torch.as_tensor(_DeviceArray(n, True), device=CUDA)}


# ------------------------------------------------------------------------------------------ one pass
def run(state):
    kind = state["kind"]
    if kind == "conv":
        return ops.conv(state["x"], state["w"], state["b"], state["strides"], state["pads"], state["act"], lut=state["lut"])
    if kind == "gemm":
        return ops.gemm(state["a"], state["w"], state["b"])
    if kind == "matmul":
        return ops.matmul(state["a"], state["b"])
    if kind == "host":
        state["net"].run_host(state["x"], state["y"])
        return state["y"]
    state["net"].run()
    state["net"].sync()      # the output may be read, and a stalled or out-of-range inference is reported here
    return state["y"]


# ------------------------------------------------------------------------------------------ work
def _out(size, k, s, p):
    return (size + 2 * p - k) // s + 1


def _conv_flops(c):
    return 2.0 * c["n"] * c["oc"] * c["c"] * c["k"] ** 2 * _out(c["h"], c["k"], c["s"], c["p"]) * _out(c["w"], c["k"], c["s"], c["p"])


def _resnet50_work(image, es):
    """(flops of one image, weight bytes)"""
    flops, weights = 0.0, 0

    def conv(cin, cout, k, s, p, size):
        nonlocal flops, weights
        size = _out(size, k, s, p)
        flops += 2.0 * cin * cout * k * k * size * size
        weights += cin * cout * k * k
        return size

    size = _out(conv(3, 64, 7, 2, 3, image), 3, 2, 1)
    cin = 64
    for stage, blocks in enumerate((3, 4, 6, 3)):
        mid = 64 << stage
        for blk in range(blocks):
            s = 2 if blk == 0 and stage else 1
            conv(cin, mid, 1, 1, 0, size)
            after = conv(mid, mid, 3, s, 1, size)
            conv(mid, 4 * mid, 1, 1, 0, after)
            if blk == 0:
                conv(cin, 4 * mid, 1, s, 0, size)
            size, cin = after, 4 * mid
    return flops + 2.0 * 1000 * cin, (weights + 1000 * cin) * es


def _vit_work(image, dim):
    t = (image // 16) ** 2 + 1
    block = 4 * dim * dim + 8 * dim * dim
    flops = 2.0 * (t - 1) * 768 * dim + 12 * (2.0 * t * block + 4.0 * t * t * dim) + 2.0 * 1000 * dim
    return flops, 4 * (12 * block + 768 * dim + 1000 * dim + t * dim)


def _yolo_work(image):
    """(flops of one image, weight bytes, output values of one image)"""
    flops, weights, hw = 0.0, 0, image
    for ci, co, k, s, p in models.YOLO_STACK:
        hw = _out(hw, k, s, p)
        flops += 2.0 * co * hw * hw * ci * k * k
        weights += co * ci * k * k
    return flops, weights, models.YOLO_STACK[-1][1] * hw * hw


def work(case):
    """Inputs and weights read once, outputs written once; what lies between two layers need not leave the chip."""
    if case["kind"] == "conv":
        y = case["n"] * case["oc"] * _out(case["h"], case["k"], case["s"], case["p"]) * _out(case["w"], case["k"], case["s"], case["p"])
        x = case["n"] * case["c"] * case["h"] * case["w"]
        return {"bytes": 4.0 * (x + y + case["oc"] * (case["c"] * case["k"] ** 2 + 1)), "flops": _conv_flops(case)}
    if case["kind"] == "gemm":
        m, k, n = case["m"], case["k"], case["n"]
        return {"bytes": 4.0 * (m * k + n * k + n + m * n), "flops": 2.0 * m * n * k}
    if case["kind"] == "matmul":
        b, m, k, n = case["b"], case["m"], case["k"], case["n"]
        return {"bytes": 4.0 * (b * m * k + (1 if case["shared"] else b) * k * n + b * m * n), "flops": 2.0 * b * m * n * k}
    images = 4.0 * case["batch"] * 3 * case["image"] ** 2
    if case["kind"] == "resnet50":
        flops, weights = _resnet50_work(case["image"], 2 if case["prec"] == "f16" else 4)
        return {"bytes": images + weights + 4.0 * case["batch"] * 1000, "flops": case["batch"] * flops}
    if case["kind"] == "vit":
        flops, weights = _vit_work(case["image"], case["dim"])
        return {"bytes": images + weights + 4.0 * case["batch"] * 1000, "flops": case["batch"] * flops}
    flops, weights, out = _yolo_work(case["image"])
    return {"bytes": images + weights + 4.0 * case["batch"] * out, "flops": case["batch"] * flops}


def tolerance(case):
    if case["kind"] == "yolo":
        return "exact"               # int32 sums, and every float step of the reference in its own order
    if case["kind"] in ("conv", "gemm", "matmul"):
        return {"rel": 1e-3}         # products of 10-bit mantissas, fp32 sums
    return {"rel": 5e-3}             # the same through some fifty layers, each rounding its activations
