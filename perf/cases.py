"""The work that users of this package have it do, as measurable cases.

Every case goes through the public module (`GN_NHWC`) the way a model calls it: `infer` is one call under
`torch.no_grad()`, `train` is one call plus the gradients of the input, weight and bias through autograd.
Sizes are those of the repository's benchmark configurations; `draw` gives further ones of the same ranges,
odd and ragged sizes among them.
"""
import torch

from channels_last_groupnorm_b200 import GN_NHWC

DTYPES = {"float32": torch.float32, "float16": torch.float16, "bfloat16": torch.bfloat16}
BYTES = {"float32": 4, "float16": 2, "bfloat16": 2}


def _case(mode, n, c, h, w, groups, act, dtype, eps=1e-5, layout="channels_last", param_dtype=None, dist="normal", scale=1.0):
    return {"mode": mode, "n": n, "c": c, "h": h, "w": w, "groups": groups, "act": act, "dtype": dtype, "eps": eps,
            "layout": layout, "param_dtype": param_dtype or dtype, "dist": dist, "scale": scale}


def _named(name, *args, **kw):
    return dict(_case(*args, **kw), name=name)


def listed():
    return [
        # Diffusion U-Net blocks, one image, half precision, SiLU after the norm: dozens of such calls per denoising
        # step.  The innermost level is the smallest call there is (latency and launches), the outermost the largest.
        _named("unet_1280x8_infer", "infer", 1, 1280, 8, 8, 32, "silu", "float16"),
        _named("unet_320x64_infer", "infer", 1, 320, 64, 64, 32, "silu", "float16"),
        # Image decoder at 1024 pixels: activations grow from 34 MB to 268 MB per tensor while the batch is one.
        _named("vae_512x128_infer", "infer", 1, 512, 128, 128, 32, "silu", "float16", eps=1e-6, scale=2.0),
        _named("vae_256x512_infer", "infer", 1, 256, 512, 512, 32, "silu", "float16", eps=1e-6, scale=2.0),
        # ... and the same decoder being trained or fine-tuned; the last level is the largest tensor of all.
        _named("vae_512x256_train", "train", 1, 512, 256, 256, 32, "silu", "float16", eps=1e-6, scale=2.0),
        _named("vae_128x1024_train", "train", 1, 128, 1024, 1024, 32, "silu", "float16", eps=1e-6, scale=2.0),
        # Batched training in bf16: the whole batch on one GPU, ...
        _named("train_64x256x64", "train", 64, 256, 64, 64, 32, "gelu", "bfloat16"),
        # ... and one rank's eighth of it with fp32 master parameters, as under autocast.
        _named("train_8x256x64_fp32_params", "train", 8, 256, 64, 64, 32, "gelu", "bfloat16", param_dtype="float32"),
        # Small fp32 training step without an activation.
        _named("fp32_2x128x32_train", "train", 2, 128, 32, 32, 32, "identity", "float32"),
        # Odd spatial size and five channels per group: vectors of four straddle the groups.
        _named("odd_3x40x17x33_train", "train", 3, 40, 17, 33, 8, "relu", "float32", dist="uniform3"),
        # Last stage of a classifier: many channels, 7 x 7 pixels.
        _named("wide_16x2048x7_train", "train", 16, 2048, 7, 7, 32, "gelu_tanh", "bfloat16", dist="uniform3"),
        # A model that kept its activations channels-first.
        _named("channels_first_512x256_train", "train", 1, 512, 256, 256, 32, "silu", "float16", eps=1e-6,
               layout="channels_first", scale=2.0),
    ]


#: a drawn case moves at most this much, about half of the largest listed one
MOST_BYTES = 7e8


def _between(rng, lo, hi):
    """A whole number spread evenly over the logarithm of [lo, hi]."""
    return min(hi, max(lo, int(round(lo * (hi / lo) ** rng.random()))))


def _drawn(rng):
    family = rng.choice(["unet", "decoder", "batch", "edge"])
    first = rng.random() < 0.12
    layout = "channels_first" if first else "channels_last"
    if family == "unet":  # one or a few images, narrow to wide channels, SiLU
        c = rng.choice([320, 640, 960, 1280, 1920, 2560])
        h = _between(rng, 8, 96)
        return _case("infer", rng.choice([1, 1, 2, 4]), c, h, max(4, h + rng.choice([0, 0, 0, -3, 1, 8])), 32, "silu",
                     rng.choice(["float16", "float16", "bfloat16"]), layout=layout)
    if family == "decoder":  # large images, few of them
        c = rng.choice([128, 256, 512])
        h = _between(rng, 64, 1024)
        return _case(rng.choice(["infer", "train"]), rng.choice([1, 1, 1, 2, 3]), c, h, _between(rng, 64, 1024), 32, "silu",
                     rng.choice(["float16", "float16", "bfloat16", "float32"]), eps=1e-6, layout=layout, scale=2.0)
    if family == "batch":  # training batches of feature maps
        c = rng.choice([64, 96, 128, 192, 256, 384, 512, 1024, 2048])
        h = _between(rng, 7, 96)
        dtype = rng.choice(["bfloat16", "bfloat16", "float16", "float32"])
        return _case("train", _between(rng, 4, 64), c, h, h, rng.choice([32, 32, 16, 8, 1]),
                     rng.choice(["gelu", "gelu_tanh", "silu", "identity"]), dtype, layout=layout,
                     param_dtype=rng.choice([dtype, "float32"]))
    # everything else that is legal: few or odd channels, one channel per group, long thin images
    groups = rng.choice([1, 3, 4, 8, 30, 64])
    per = rng.choice([1, 4, 5, 7, 12, 16, 32]) if groups < 64 else rng.choice([1, 2, 4])
    dtype = rng.choice(["float32", "float32", "bfloat16", "float16"])
    return _case(rng.choice(["infer", "train", "train"]), _between(rng, 1, 24), groups * per, _between(rng, 5, 320), _between(rng, 5, 320), groups,
                 rng.choice(["gelu_tanh", "relu", "silu", "gelu", "identity"]), dtype, layout=layout, dist="uniform3")


def draw(rng):
    while True:
        case = _drawn(rng)
        # The gradient of a ReLU jumps where its argument crosses zero: over many elements two correct sums that
        # differ in the last bit put one of them on different sides, which no tolerance can tell from a mistake.
        if case["act"] == "relu" and case["mode"] == "train" and case["n"] * case["c"] * case["h"] * case["w"] > 1e5:
            case["act"] = "silu"
        if 1e5 <= work(case)["bytes"] <= MOST_BYTES:
            return case


def prepare(case, seed):
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev).manual_seed(seed)
    n, c, h, w = case["n"], case["c"], case["h"], case["w"]
    dtype = DTYPES[case["dtype"]]

    def activations(dist, scale):
        shape = (n, h, w, c) if case["layout"] == "channels_last" else (n, c, h, w)
        if dist == "uniform3":
            t = torch.rand(shape, device=dev, generator=gen, dtype=dtype).mul_(6.0).sub_(3.0)
        else:
            t = torch.randn(shape, device=dev, generator=gen, dtype=dtype).mul_(scale)
        return t.permute(0, 3, 1, 2) if case["layout"] == "channels_last" else t

    module = GN_NHWC(case["groups"], c, activation=case["act"], eps=case["eps"], device=dev, dtype=DTYPES[case["param_dtype"]])
    with torch.no_grad():
        module.weight.uniform_(0.5, 1.5, generator=gen)
        module.bias.normal_(0.0, 0.1, generator=gen)
    state = {"module": module, "x": activations(case["dist"], case["scale"]), "dy": None}
    if case["mode"] == "train":
        state["x"].requires_grad_(True)
        state["dy"] = activations("normal", 1.0)
    return state


def run(state):
    module, x = state["module"], state["x"]
    if state["dy"] is None:
        with torch.no_grad():
            return module(x)
    y = module(x)
    dx, dweight, dbias = torch.autograd.grad(y, (x, module.weight, module.bias), state["dy"])
    return y.detach(), dx, dweight, dbias


def work(case):
    elements = case["n"] * case["c"] * case["h"] * case["w"]
    params = case["c"] * BYTES[case["param_dtype"]]
    if case["mode"] == "infer":  # x in, y out; two sums and one affine map per element
        return {"bytes": 2 * elements * BYTES[case["dtype"]] + 2 * params, "flops": 6 * elements}
    # forward, then x and dy in, dx out; two more sums, the derivative's product and dx
    return {"bytes": 5 * elements * BYTES[case["dtype"]] + 6 * params, "flops": 16 * elements}


def tolerance(case):
    # Relative error of every output against the same call in fp64, over the listed and some fifty drawn cases:
    # fp32 up to 3e-7 (longer sums are given more room), fp16 up to 1.3e-3, bf16 up to 3.7e-3; the largest single
    # difference is 9e-7, 0.024 and 0.045 (a 16-bit activation derivative near a zero crossing).
    limits = {"float32": {"rel": 5e-6, "max": 1e-4}, "float16": {"rel": 4e-3, "max": 0.1}, "bfloat16": {"rel": 1.5e-2, "max": 0.2}}
    return limits[case["dtype"]]
