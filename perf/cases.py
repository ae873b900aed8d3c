"""Performance cases of the public operators: what users of the package call, over the range of sizes they call it with.

A case is a dict of plain values. `op` is an operator of morphocore_b200.functional (dilation, erosion, smorph, opening,
sigma_layer; "smorph_scm" is smorph with a beta) or "stack", the four-layer model of workloads.CFG5_LAYERS built from
morphocore_b200.nn. `train` runs forward and backward (gradients of the input, as in a hidden layer, and of every
parameter), otherwise the call runs under no_grad, as at inference. Options that draw random numbers inside the call
(weight dropout, weight noise) are left out: their outputs differ from pass to pass.
"""
import math

import torch

import morphocore_b200.functional as F
import morphocore_b200.nn as Mnn
import workloads as WL

DTYPES = {"float32": torch.float32, "float64": torch.float64, "bfloat16": torch.bfloat16, "float16": torch.float16}
SMOOTH = ("smorph", "smorph_scm")


def _case(name, op, merge, B, Ci, Co, H, W, kH, kW, train, dtype="float32", padding="replicate", alpha=0.0, spread=0.0):
    c = dict(op=op, merge=merge, B=B, Ci=Ci, Co=Co, H=H, W=W, kH=kH, kW=kW, train=train, dtype=dtype, padding=padding, alpha=alpha, spread=spread)
    return dict(c, name=name) if name else c


def listed():
    return [
        # One grey image through one structuring element: the smallest call, all latency.
        _case("one_image_infer", "dilation", "identity", 1, 1, 1, 64, 64, 5, 5, False),
        # First layer of a small network on a batch of RGB crops (benchmark configuration 1).
        _case("rgb_max_infer", "dilation", "max", 8, 3, 16, 128, 128, 3, 3, False),
        # Smooth layer of a classifier on small feature maps, one learned alpha per pair.
        _case("smorph_28_train", "smorph", "sum", 8, 8, 16, 28, 28, 3, 3, True, alpha=1.0, spread=0.25),
        # Erosion with winning channel on odd image sizes (rows that are not 16-byte aligned), zero border.
        _case("ragged_max_train", "erosion", "max", 5, 12, 20, 75, 101, 3, 3, True, padding="zero"),
        # Mixed-precision training: half-precision storage, a middle layer's feature maps.
        _case("bf16_mean_train", "erosion", "mean", 16, 32, 64, 56, 56, 3, 3, True, dtype="bfloat16"),
        # Learnable blend of dilation and erosion on middle-sized maps.
        _case("sigma_sum_train", "sigma_layer", "sum", 8, 16, 16, 96, 96, 5, 5, True),
        # Per-channel opening of larger images, as in background removal; nothing outside the image.
        _case("opening_infer", "opening", "identity", 16, 8, 8, 240, 320, 7, 7, False, padding="geodesic"),
        # The four-layer model on one image: latency of a deployed model.
        _case("stack_infer_1", "stack", "sum", 1, 3, 64, 224, 224, 0, 0, False),
        # Training of one wide erosion layer (benchmark configuration 2).
        _case("erosion_sum_train", "erosion", "sum", 32, 16, 32, 256, 256, 5, 5, True),
        # Training of one smooth layer with a large structuring element (benchmark configuration 3).
        _case("smorph_7x7_train", "smorph", "mean", 16, 32, 32, 128, 128, 7, 7, True, alpha=2.0),
        # Double precision, per-channel, large structuring element (benchmark configuration 4).
        _case("f64_11x11_train", "dilation", "identity", 8, 64, 64, 512, 512, 11, 11, True, dtype="float64"),
        # One training pass of the four-layer model on the 32 images each of eight GPUs gets (benchmark configuration 5).
        _case("stack_train_32", "stack", "sum", 32, 3, 64, 224, 224, 0, 0, True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _side(rng, lo, hi):
    n = _log(rng, lo, hi)
    return n if rng.random() < 0.5 else max(8, n // 8 * 8)  # half of the images have sides that are multiples of 8


def _draw_one(rng):
    op = rng.choices(("dilation", "erosion", "smorph", "smorph_scm", "opening", "sigma_layer", "stack"), (5, 5, 6, 1, 2, 2, 2))[0]
    train = rng.random() < 0.65
    B, H = _log(rng, 1, 32), _side(rng, 14, 512)
    W = H if rng.random() < 0.4 else max(14, min(512, _side(rng, max(14, H * 0.6), H * 1.7)))
    if op == "stack":
        return _case(None, op, "sum", min(B, 16), 3, 64, min(H, 256), min(W, 256), 0, 0, train)
    merges = {"smorph": ((6, 3, 1, 0, 2)), "opening": (1, 0, 0, 0, 4), "smorph_scm": (1, 0, 0, 0, 0)}.get(op, (4, 2, 2, 1, 2))
    merge = rng.choices(("sum", "mean", "max", "min", "identity"), merges)[0]
    Ci, Co = _log(rng, 1, 64), _log(rng, 1, 64)
    if merge == "identity":
        Co = Ci
    kH, kW = rng.choices(((3, 3), (5, 5), (7, 7), (9, 9), (11, 11), (3, 5), (5, 3), (1, 7)), (9, 6, 3, 1, 1, 0.5, 0.5, 0.5))[0]
    dtype = rng.choices(("float32", "float64", "bfloat16", "float16"), (8, 2, 1.5, 0.5))[0]
    padding = "replicate" if op in SMOOTH else rng.choices(("replicate", "zero", "geodesic", "constant"), (4, 2, 2, 1))[0]
    alpha, spread = (rng.choice(WL.CFG3_ALPHAS), rng.choice((0.0, 0.25))) if op in SMOOTH else (0.0, 0.0)
    return _case(None, op, merge, B, Ci, Co, H, W, kH, kW, train, dtype, padding, alpha, spread)


def draw(rng):
    """One more case: image sides of 14 to 512, 1 to 64 channels, 1 to 32 images, structuring elements of 3 x 3 to 11 x 11,
    every merge, border and type, sizes spread over their logarithm; at most 20 G taps (40 for the stack) and 150 M elements a tensor."""
    while True:
        c = _draw_one(rng)
        elements = c["B"] * c["H"] * c["W"] * max(c["Ci"], c["Co"])
        if _taps(c) <= (40e9 if c["op"] == "stack" else 20e9) and elements <= 150e6:
            return c


def _taps(c):
    if c["op"] == "stack":
        return sum(WL.taps(c["B"], co, ci, c["H"], c["W"], k, k) for (_, ci, co, k, _, _) in WL.CFG5_LAYERS)
    n = WL.taps(c["B"], c["Co"], c["Ci"], c["H"], c["W"], c["kH"], c["kW"], c["merge"] == "identity")
    if c["op"] == "opening":
        n += WL.taps(c["B"], c["Co"], c["Co"], c["H"], c["W"], c["kH"], c["kW"], True)
    return 2 * n if c["op"] == "sigma_layer" else n


def _stack():
    layers = []
    for kind, ci, co, k, merge, alpha in WL.CFG5_LAYERS:
        if kind == "smorph":
            layers.append(Mnn.SMorph(ci, co, k, merge, init_alpha=alpha))
        else:
            layers.append((Mnn.Dilation if kind == "dilation" else Mnn.Erosion)(ci, co, k, merge))
    return torch.nn.Sequential(*layers).cuda()


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    B, Ci, Co, H, W = (case[k] for k in ("B", "Ci", "Co", "H", "W"))
    dtype, train = DTYPES[case["dtype"]], case["train"]

    def normal(*shape, scale=1.0):
        work = torch.float64 if dtype == torch.float64 else torch.float32
        return (torch.randn(shape, generator=g, device="cuda", dtype=work) * scale).to(dtype)

    s = {"case": case}
    if case["op"] == "stack":
        s["model"] = _stack()
        with torch.no_grad():
            for layer in s["model"]:
                layer.weight.copy_(normal(*layer.weight.shape, scale=0.1))
        s["x"] = torch.rand((B, 3, H, W), generator=g, device="cuda")
        s["target"] = normal(B, Co, H, W)
        return s
    wide = torch.float64 if dtype == torch.float64 else torch.float32
    pair = 1 if case["merge"] == "identity" else Ci
    # Images (or rectified activations) in [0, 1) for the hard operators, normalised activations for the smooth ones.
    s["x"] = normal(B, Ci, H, W) if case["op"] in SMOOTH else torch.rand((B, Ci, H, W), generator=g, device="cuda", dtype=wide).to(dtype)
    s["w"] = normal(Co, pair, case["kH"], case["kW"], scale=0.05 if case["op"] in SMOOTH else 0.1)
    inputs = ["x", "w"]
    if case["op"] == "opening":
        s["w2"] = normal(Co, 1, case["kH"], case["kW"], scale=0.1)
        inputs.append("w2")
    if case["op"] in SMOOTH or case["op"] == "sigma_layer":
        s["alpha"] = (normal(Co, pair, scale=case["spread"]) + case["alpha"]).to(dtype)
        inputs.append("alpha")
    if case["op"] == "smorph_scm":
        s["beta"] = (normal(Co, scale=0.25) + 1.0).to(dtype)
        inputs.append("beta")
    if train:
        s["gy"] = normal(B, Co, H, W)
        s["grads"] = [s[k].requires_grad_(True) for k in inputs]
    return s


def _call(s, c):
    merge, padding = c["merge"], c["padding"]
    value = 0.5 if padding == "constant" else 0.0
    if c["op"] == "smorph":
        return F.smorph(s["x"], s["w"], s["alpha"], channel_merge_mode=merge)
    if c["op"] == "smorph_scm":
        return F.smorph(s["x"], s["w"], s["alpha"], s["beta"])
    if c["op"] == "opening":
        return F.opening(s["x"], s["w"], s["w2"], merge, padding, padding_value=value)
    if c["op"] == "sigma_layer":
        return F.sigma_layer(s["x"], s["w"], s["alpha"], merge, padding, padding_value=value)
    return (F.dilation if c["op"] == "dilation" else F.erosion)(s["x"], s["w"], merge, padding, padding_value=value)


def run(state):
    c = state["case"]
    if c["op"] == "stack":
        model = state["model"]
        if not c["train"]:
            with torch.no_grad():
                return model(state["x"])
        model.zero_grad()
        y = model(state["x"])
        loss = torch.nn.functional.mse_loss(y, state["target"])
        loss.backward()
        return [y.detach(), loss.detach()] + [p.grad for p in model.parameters()]
    if not c["train"]:
        with torch.no_grad():
            return _call(state, c)
    for t in state["grads"]:
        t.grad = None
    y = _call(state, c)
    y.backward(state["gy"])
    return [y.detach()] + [t.grad for t in state["grads"]]


def work(case):
    """Bytes: every input read once, every output written once. Operations: an add and a comparison per tap for the hard
    operators and the same again for the winners of the backward pass where a merge keeps no index (with an index: two
    adds per output); for the smooth ones three multiply-adds per tap forward (exponential factor, sum, weighted sum) and
    ten operations per tap backward."""
    B, H, W = case["B"], case["H"], case["W"]
    size = {"float32": 4, "float64": 8}.get(case["dtype"], 2)
    taps, train = _taps(case), case["train"]
    if case["op"] == "stack":
        smooth = sum(WL.taps(B, co, ci, H, W, k, k) for (kind, ci, co, k, _, _) in WL.CFG5_LAYERS if kind == "smorph")
        first = WL.taps(B, 64, 3, H, W, 3, 3)
        flops = 6 * smooth + 2 * (taps - smooth) + (10 * smooth + 2 * first if train else 0)
        params = sum(co * ci * k * k for (_, ci, co, k, _, _) in WL.CFG5_LAYERS)
        return {"bytes": 4 * (B * H * W * (3 + 64) + params * (2 if train else 1)), "flops": flops}
    Ci, Co = case["Ci"], case["Co"]
    params = Co * (1 if case["merge"] == "identity" else Ci) * case["kH"] * case["kW"]
    moved = B * H * W * (Ci + Co) + params
    if case["op"] in SMOOTH:
        flops = taps * (16 if train else 6)
    else:
        winner = case["merge"] in ("max", "min")
        flops = 2 * taps + (0 if not train else 2 * B * H * W * Co if winner else 2 * taps)
    return {"bytes": size * moved * (2 if train else 1), "flops": flops}


def tolerance(case):
    """Relative errors another correct implementation of the same precision shows.

    Hard operators: values are sums of exact extrema, gradients are sums in another order. Smooth ones: an exponential's
    relative error is multiplied by |alpha| times its exponent's size in the gradients. Where a soft extremum feeds a
    MAX / MIN (the merges of smorph, layer 3 of the stack, an opening's second stage behind a sum of channels) candidates
    closer than rounding swap places and a whole gradient moves with them: about 1e-5 of the pixels, 5e-3 in the 2-norm."""
    winner = case["merge"] in ("max", "min")
    swaps = case["train"] and (case["op"] == "stack" or case["op"] in SMOOTH and winner or case["op"] == "opening" and case["merge"] in ("sum", "mean"))
    if case["dtype"] in ("bfloat16", "float16"):
        return {"rel": 1e-2 if case["dtype"] == "bfloat16" else 5e-3, "max": 0.99 if swaps else 0.2}
    if case["dtype"] == "float64":
        return {"rel": 5e-3, "max": 0.99} if swaps else {"rel": 1e-11 if case["op"] in SMOOTH else 1e-12}
    if swaps:
        return {"rel": 5e-3, "max": 0.99}
    if case["op"] in SMOOTH or case["op"] == "stack":
        return {"rel": min(1e-4, 2e-5 * (1.0 + abs(case["alpha"]))) if case["op"] in SMOOTH else 3e-5}
    return {"rel": 1e-5}
