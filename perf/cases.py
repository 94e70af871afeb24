"""The work whose speed counts: what a user of the distance nets has the library do.

`listed()` names the cases, `draw(rng)` gives further ones of the same ranges, `prepare(case, seed)` builds
what a program holds before the call, `run(state)` is one pass through the public entry points, `work(case)`
is what the pass cannot do without and `tolerance(case)` how far another correct implementation may be off.

Kinds of case:
  layer    forward and backward of one distance layer (`norm_dist` and autograd), p = inf or finite
  conv     forward and backward of a `NormDistConv` module, one spatial position per output pixel
  bound    lower / upper bounds of one layer (`inf_dist_bound`)
  infer    logits of a trained distance MLP in eval mode
  robust   robustness evaluation of one batch: certification, then a few steps of the PGD attack
  train    one optimisation step of a net: forward with the eps box, loss, backward, AdamW
"""
import math

import torch

import linfdist_b200 as L
from linfdist_b200.train_step import DataParallelStep, MarginLoss, cross_entropy, hinge

INF = float("inf")
UNIT = 1024          # hidden widths of the nets count units of 1024 neurons


def listed():
    return [
        # One image at a time through a small trained MNIST net: latency and launches are all there is.
        {"name": "infer_mnist_one", "kind": "infer", "batch": 1, "din": 784, "depth": 4, "width": 1, "classes": 10},
        # First layer of an MNIST net: images in [0, 1), the benchmark's headline layer.
        {"name": "layer_mnist", "kind": "layer", "batch": 512, "din": 784, "dout": 5120, "group": 1, "p": "inf", "x": "uniform"},
        # A hidden layer of the wide nets on activations as spread out as the weights.
        {"name": "layer_wide", "kind": "layer", "batch": 512, "din": 5120, "dout": 5120, "group": 1, "p": "inf", "x": "normal"},
        # A layer of somebody's own net: no size is a multiple of anything.
        {"name": "layer_ragged", "kind": "layer", "batch": 203, "din": 1027, "dout": 1333, "group": 1, "p": "inf", "x": "normal"},
        # The L_p layer where the annealing starts.
        {"name": "layer_p8", "kind": "layer", "batch": 512, "din": 5120, "dout": 5120, "group": 1, "p": 8.0, "x": "normal"},
        # The L_p layer somewhere along the annealing, where p is no integer, on CIFAR images.
        {"name": "layer_anneal", "kind": "layer", "batch": 256, "din": 3072, "dout": 5120, "group": 1, "p": 23.7, "x": "uniform"},
        # A 3 x 3 convolution of distance neurons on feature maps.
        {"name": "conv_3x3", "kind": "conv", "batch": 64, "cin": 64, "cout": 128, "side": 16, "group": 1, "p": "inf"},
        # Interval bounds of the first CIFAR layer with grouped channels.
        {"name": "bound_groups", "kind": "bound", "batch": 512, "din": 3072, "dout": 5120, "group": 4, "eps": 8 / 255},
        # Evaluation of one CIFAR batch: certified radius 8/255 and a short PGD attack.
        {"name": "robust_cifar", "kind": "robust", "batch": 512, "side": 32, "depth": 5, "width": 5, "classes": 10,
         "eps": 8 / 255, "pgd": 2},
        # Training at p = inf, the last phase of every schedule: CIFAR net, 512 images.
        {"name": "train_cifar", "kind": "train", "batch": 512, "side": 32, "depth": 5, "width": 5, "classes": 10,
         "head": 0, "p": "inf", "eps": 8 / 255},
        # Training at p = 8, the first phase of every schedule.
        {"name": "train_cifar_p8", "kind": "train", "batch": 512, "side": 32, "depth": 5, "width": 5, "classes": 10,
         "head": 0, "p": 8.0, "eps": 8 / 255},
        # Training of the net with an MLP head on TinyImageNet shapes, 200 classes.
        {"name": "train_tiny", "kind": "train", "batch": 256, "side": 64, "depth": 5, "width": 5, "classes": 200,
         "head": 512, "p": "inf", "eps": 1 / 255},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, lo, hi):
    """A size spread over its logarithm; one half are multiples of 16, as most people choose them."""
    n = _log(rng, lo, hi)
    return max(lo, n // 16 * 16) if rng.random() < 0.5 else n


def _power(rng):
    """inf, an integer where schedules stand still, or any p on the way from 8 to 1000."""
    r = rng.random()
    return "inf" if r < 0.5 else rng.choice([8.0, 16.0, 64.0]) if r < 0.7 else round(math.exp(rng.uniform(math.log(8.0), math.log(1000.0))), 3)


def draw(rng):
    kind = rng.choice(["layer", "layer", "layer", "layer", "conv", "bound", "infer", "robust", "train", "train"])
    if kind == "layer":
        group = rng.choice([1, 1, 1, 1, 2, 4])
        p = _power(rng)
        return {"kind": kind, "batch": _size(rng, 8, 1024 if p == "inf" else 512), "din": group * _size(rng, 64, 5120 // group),
                "dout": group * _size(rng, 10, 5120 // group), "group": group, "p": p, "x": rng.choice(["uniform", "normal"])}
    if kind == "conv":
        return {"kind": kind, "batch": _size(rng, 4, 64), "cin": 4 * _log(rng, 4, 16), "cout": 4 * _log(rng, 8, 32),
                "side": rng.randint(6, 16), "group": rng.choice([1, 1, 2]), "p": _power(rng)}
    if kind == "bound":
        group = rng.choice([1, 1, 4])
        return {"kind": kind, "batch": _size(rng, 8, 1024), "din": group * _size(rng, 64, 5120 // group),
                "dout": group * _size(rng, 10, 5120 // group), "group": group, "eps": rng.choice([1 / 255, 8 / 255, 0.1])}
    if kind == "infer":
        return {"kind": kind, "batch": _log(rng, 1, 256), "din": rng.choice([784, 3072]), "depth": rng.randint(2, 5),
                "width": rng.randint(1, 4), "classes": 10}
    if kind == "robust":
        return {"kind": kind, "batch": _size(rng, 32, 512), "side": 32, "depth": rng.randint(3, 5), "width": rng.randint(1, 5),
                "classes": 10, "eps": rng.choice([2 / 255, 8 / 255]), "pgd": rng.randint(1, 3)}
    head, p = rng.choice([0, 0, 512]), _power(rng)
    return {"kind": kind, "batch": _size(rng, 64, 512 if p == "inf" else 224), "side": rng.choice([28, 32]) if head == 0 else 32,
            "depth": rng.randint(3, 5), "width": rng.randint(1, 5), "classes": 10 if head == 0 else 200, "head": head,
            "p": p, "eps": rng.choice([1 / 255, 8 / 255])}


def _p(case):
    return INF if case["p"] == "inf" else float(case["p"])


def _randn(gen, *shape):
    return torch.randn(*shape, generator=gen, device="cuda")


def _rand(gen, *shape):
    return torch.rand(*shape, generator=gen, device="cuda")


def _channels(case):
    return 1 if case["side"] == 28 else 3


def _net(case, seed):
    """A net on the GPU, with weights as training leaves them.  The layers' own initialisation sets one entry of
    every row to -10, so that each layer starts as the identity; the l_inf weight decay shrinks the largest entry
    of a row alone, until these entries have come down among the largest of the others."""
    torch.manual_seed(seed)
    shape = case["din"] if "din" in case else (_channels(case), case["side"], case["side"])
    with torch.device("cuda"):
        if case.get("head"):
            feature = L.MLPFeature(case["depth"], case["width"], shape)
            net = L.Model(feature, L.Predictor(feature.out_features, case["head"], case["classes"]), case["eps"])
        else:
            net = L.Model(L.MLP(case["depth"], case["width"], shape, num_classes=case["classes"]), L.BoundFinalIdentity(), case.get("eps", 0.0))
        with torch.no_grad():
            for m in net.modules():
                if isinstance(m, L.NormDist):
                    low = m.weight == -10.0
                    m.weight.copy_(torch.where(low, -3.0 - 2.0 * torch.rand_like(m.weight), m.weight))
    return net


@torch.no_grad()
def _settle(net, images):
    """Gives the mean-shift layers the statistics that a trained net has: one training-mode pass that takes
    the batch means over as they are."""
    norms = [m for m in net.modules() if isinstance(m, L.MeanNorm)]
    saved = [m.momentum for m in norms]
    for m in norms:
        m.momentum = 1.0
    L.set_p_norm(net, INF)
    net.train()
    net(images)
    for m, s in zip(norms, saved):
        m.momentum = s


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    if kind == "layer":
        B, CI, CO = case["batch"], case["din"], case["dout"]
        x = (_rand if case["x"] == "uniform" else _randn)(gen, B, CI, 1)
        return {"kind": kind, "x": x.requires_grad_(), "w": _randn(gen, CO, CI // case["group"]).requires_grad_(),
                "g": _randn(gen, B, CO, 1), "group": case["group"], "p": _p(case)}
    if kind == "conv":
        torch.manual_seed(seed)
        with torch.device("cuda"):
            layer = L.NormDistConv(case["cin"], case["cout"], 3, padding=1, group=case["group"], p=_p(case), bias=True)
        n = case["side"]
        return {"kind": kind, "layer": layer, "x": _randn(gen, case["batch"], case["cin"], n, n).requires_grad_(),
                "g": _randn(gen, case["batch"], case["cout"], n, n)}
    if kind == "bound":
        B, CI, CO = case["batch"], case["din"], case["dout"]
        x = _rand(gen, B, CI, 1)
        return {"kind": kind, "lower": (x - case["eps"]).clamp(0, 1), "upper": (x + case["eps"]).clamp(0, 1),
                "w": _randn(gen, CO, CI // case["group"]), "group": case["group"]}
    if kind == "infer":
        net = _net(case, seed)
        _settle(net, _rand(gen, 64, case["din"]))
        net.eval()
        return {"kind": kind, "net": net, "x": _rand(gen, case["batch"], case["din"])}
    shape = (case["batch"], _channels(case), case["side"], case["side"])
    images, labels = _rand(gen, *shape), torch.randint(0, case["classes"], (case["batch"],), generator=gen, device="cuda")
    net = _net(case, seed)
    if kind == "robust":
        _settle(net, images)
        net.eval()
        one, zero = torch.ones((), device="cuda"), torch.zeros((), device="cuda")
        attack = L.AttackPGD(net, case["eps"], case["eps"] / 4, case["pgd"], one, zero, random_start=False)
        return {"kind": kind, "net": net, "x": images, "t": labels, "eps": case["eps"], "one": one, "zero": zero, "attack": attack}
    L.set_p_norm(net, _p(case))
    net.train()
    opt = L.AdamW(net, lr=0.02, betas=(0.9, 0.99), eps=1e-10, weight_decay=5e-3)
    loss = MarginLoss(cross_entropy() if case.get("head") else hinge(), 0.75)
    return {"kind": kind, "net": net, "step": DataParallelStep(net, opt), "opt": opt, "loss": loss, "x": images, "t": labels}


def run(state):
    kind = state["kind"]
    if kind == "layer":
        state["x"].grad = state["w"].grad = None
        y = L.norm_dist(state["x"], state["w"], state["group"], state["p"])
        y.backward(state["g"])
        return y.detach(), state["x"].grad, state["w"].grad
    if kind == "conv":
        state["x"].grad = None
        state["layer"].zero_grad(set_to_none=True)
        y = state["layer"](state["x"])[0]
        y.backward(state["g"])
        return [y.detach(), state["x"].grad] + [q.grad for q in state["layer"].parameters()]
    if kind == "bound":
        return L.inf_dist_bound(state["lower"], state["upper"], state["w"], state["group"])
    if kind == "infer":
        with torch.no_grad():
            return state["net"](state["x"])
    if kind == "robust":
        certified, margins = L.certify(state["net"], state["x"], state["t"], state["eps"], state["one"], state["zero"])
        return certified, margins, state["attack"].find(state["x"], state["t"])
    outputs, worst = state["step"](state["x"], targets=state["t"])
    loss = state["loss"](outputs, worst, state["t"])
    state["opt"].zero_grad(set_to_none=True)
    loss.backward()
    state["step"].finish_step()
    state["step"].synchronize()      # the stream waits for the updated weights; the host does not
    params = list(state["net"].parameters())
    return [loss.detach(), outputs.detach()] + [q.grad for q in params] + [q.detach() for q in params]


def _layer_work(batch, ci, co, group, p, backward=True):
    """Bytes and operations of one distance layer: every input read once, every output written once; a term is
    a subtraction and a maximum (p = inf), or a subtraction, the power and an addition."""
    ci_g = ci // group
    terms = batch * co * ci_g
    acts, weights, outs = batch * ci, co * ci_g, batch * co
    nbytes = 4 * (acts + weights + outs)
    power = math.ceil(math.log2(p)) if not math.isinf(p) else 0
    flops = 2 * terms if math.isinf(p) else (2 + power) * terms
    if backward:
        nbytes += 4 * (outs + acts + weights)
        flops += 2 * outs if math.isinf(p) else (4 + power) * terms
    return nbytes, flops


def _widths(case):
    hidden = UNIT * case["width"]
    first = case["din"] if "din" in case else _channels(case) * case["side"] ** 2
    if case.get("head"):
        return [first] + [hidden] * case["depth"]
    return [first] + [hidden] * (case["depth"] - 1) + [case["classes"]]


def work(case):
    kind = case["kind"]
    if kind == "layer":
        nbytes, flops = _layer_work(case["batch"], case["din"], case["dout"], case["group"], _p(case))
    elif kind == "conv":
        pixels = case["batch"] * case["side"] ** 2
        _, flops = _layer_work(pixels, 9 * case["cin"], case["cout"], case["group"], _p(case))
        nbytes = 4 * (2 * pixels * (case["cin"] + case["cout"]) + 2 * case["cout"] * 9 * case["cin"] // case["group"])
    elif kind == "bound":
        terms = case["batch"] * case["dout"] * case["din"] // case["group"]
        nbytes = 4 * (2 * case["batch"] * (case["din"] + case["dout"]) + case["dout"] * case["din"] // case["group"])
        flops = 4 * terms                       # two differences, a maximum and a minimum
    else:
        widths, batch = _widths(case), case["batch"]
        layers = list(zip(widths, widths[1:]))
        params = sum(a * b for a, b in layers)
        if kind == "infer":
            nbytes = 4 * (batch * (widths[0] + widths[-1]) + params)
            flops = 2 * batch * params
        elif kind == "robust":
            passes = 1 + case["pgd"]
            nbytes = 4 * passes * params + 4 * batch * (2 * widths[0] + 2 * widths[-1])
            flops = batch * params * (4 + 2 * case["pgd"])
        else:
            p = _p(case)
            flops = sum(_layer_work(batch, a, b, 1, p)[1] for a, b in layers)
            head = case["head"] * (widths[-1] + case["classes"]) if case["head"] else 0
            flops += 6 * batch * head + 10 * (params + head)
            # weights read by the forward; weights and both moments read and written by the update, gradients returned
            nbytes = 4 * (params + head) * (1 + 7) + 4 * batch * (widths[0] + widths[-1])
            if not math.isinf(p):
                nbytes += 4 * params            # the backward reads the weights once more
    return {"bytes": float(nbytes), "flops": float(flops)}


def tolerance(case):
    """About four times what was measured: layers against the same sums in 64 bits (9e-7 + 2.8e-8 * p at finite
    p: the rounding of a term is raised to the power p), nets against the same step with the batch means summed
    in another order (two steps; where an arg-max changes, a whole gradient entry moves)."""
    kind = case["kind"]
    if kind == "bound":
        return "exact"
    if kind == "infer":
        return {"rel": 1e-6}
    if kind == "robust":
        return {"rel": 1e-5}
    p = _p(case)
    if kind == "train":
        return {"rel": 1.5e-3 if not math.isinf(p) else 8e-2 if case["head"] else 2e-3}
    return {"rel": 2e-6 if math.isinf(p) else 4e-6 + 1.2e-7 * p}
