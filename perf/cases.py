"""What a user has this package do, as cases that can be timed and checked.

A case is a list of gradient tensors (`shapes`), a compression setting and one of the package's
entry points (`kind`):

  train      `TrainStep(model, loss, optimizer, aggregator)(x, y)`: a whole recorded training step
  step       `optimizer_step(optimizer, aggregator)` on gradients that backward has just accumulated
             onto the residuals; `recorded` replays it from a CUDA graph, as launch-bound programs do
  aggregate  `aggregator.aggregate(gradients)`, for programs that bring an optimizer of their own
  rankk      `RankKReducer.reduce(...)` of the research harness
  topk       `TopKReducer.reduce(...)` of the research harness

Accumulating the fresh gradients is part of a pass where the entry point overwrites its inputs with
the residual: without it a second pass would compress an ever smaller rest. Inputs are low-rank
plus noise, as gradients of a layer are. Tensors live in a few flat buffers, each on a 512-byte
boundary as the allocator would place it, so that results can be handed over whole.

All figures are for one GPU.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from powersgd_b200 import Config, PowerSGD, optimizer_step

ALIGN = 128  # floats between the starts of neighbouring tensors
HARNESS_SEED = 714
COMPRESSION = 1 / 244  # of the top-k reducer


# ---- the cases -------------------------------------------------------------------------------
def listed():
    return [
        # the smallest program: two-layer perceptron, one compressed matrix at rank 1, step replayed
        dict(name="train-mlp", kind="train", sizes="784 256 10", batch=64, rank=1, iters=2, rate=10.0, lr=0.1, momentum=0.9),
        # the headline model's gradients: 21 matrices in 12 shape groups, 41 vectors; eager loop ...
        dict(name="step-resnet18", kind="step", shapes="resnet18", rank=2, iters=2, rate=2.0, lr=0.1, momentum=0.9, nesterov=True, decay=1e-4),
        # ... and the same step replayed from a graph, as in training at full speed
        dict(name="recorded-step-resnet18", kind="step", shapes="resnet18", rank=2, iters=2, rate=2.0, lr=0.1, momentum=0.9, nesterov=True, decay=1e-4, recorded=True),
        # the first hundred steps of a run (`start_compressing_after_num_steps`): nothing compressed
        dict(name="step-uncompressed-resnet18", kind="step", shapes="resnet18", rank=2, iters=2, rate=2.0, lr=0.1, momentum=0.9, nesterov=True, decay=1e-4, warmup=True),
        # compression alone: small square matrices, half an iteration
        dict(name="aggregate-4x1024x1024", kind="aggregate", shapes="4*1024x1024", rank=8, iters=1, rate=2.0),
        # compression alone: more than the L2 cache holds
        dict(name="aggregate-4x4096x4096", kind="aggregate", shapes="4*4096x4096", rank=4, iters=2, rate=2.0),
        # an embedding's gradient, very tall, at the largest rank of the compression benchmark
        dict(name="aggregate-50257x1024", kind="aggregate", shapes="50257x1024", rank=16, iters=2, rate=2.0),
        # odd sizes, odd rank, an odd number of half-iterations, a vector beside the matrices
        dict(name="aggregate-odd", kind="aggregate", shapes="3*1001x777 2*515x2049 333", rank=3, iters=3, rate=2.0),
        # recurrent language model: rows of 650 floats, tied 33278-word embedding, plain SGD
        dict(name="step-lstm", kind="step", shapes="lstm", rank=4, iters=1, rate=2.0, lr=1.25, momentum=0.0),
        # the largest: 355 M parameters
        dict(name="step-gpt2-medium", kind="step", shapes="gpt2-medium", rank=4, iters=2, rate=10.0, lr=0.01, momentum=0.9),
        # the research harness: warm-started rank-k reducer and per-tensor top-k
        dict(name="rankk-resnet18", kind="rankk", shapes="resnet18", rank=2),
        dict(name="topk-resnet18", kind="topk", shapes="resnet18"),
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _random_shapes(rng, cap):
    """One to five groups of equal matrices, wide, tall and square, multiples of 16 and odd sizes."""
    words, left = [], cap
    for _ in range(rng.randint(1, 5)):
        n, m = _log(rng, 24, 24000), _log(rng, 24, 5000)
        if rng.random() < 0.5:
            n, m = -(-n // 16) * 16, -(-m // 16) * 16
        count = rng.randint(1, 4)
        while count > 1 and count * n * m > left:
            count -= 1
        if count * n * m > left:
            continue
        left -= count * n * m
        words.append(f"{count}*{n}x{m}")
    if not words:
        words.append("2*640x%d" % rng.randint(200, 900))
    if rng.random() < 0.5:
        words.append(str(_log(rng, 8, 4000)))
    return " ".join(words)


def draw(rng):
    kind = rng.choice(["aggregate"] * 4 + ["step"] * 5 + ["rankk"] * 2 + ["topk", "train"])
    rank = rng.choice([1, 2, 2, 3, 4, 4, 5, 8, 11, 16])
    if kind == "train":
        sizes = [_log(rng, 40, 3000), _log(rng, 40, 3000), rng.randint(2, 100)]
        return dict(kind=kind, sizes=" ".join(map(str, sizes)), batch=_log(rng, 8, 256), rank=min(rank, 4), iters=rng.randint(1, 2),
                    rate=2.0, lr=0.05, momentum=rng.choice([0.0, 0.9]))
    shapes = _random_shapes(rng, _log(rng, 100_000, 64_000_000))
    if kind == "topk":
        return dict(kind=kind, shapes=shapes)
    if kind == "rankk":
        return dict(kind=kind, shapes=shapes, rank=rank)
    iters = rng.choice([1, 2, 2, 3]) if rank <= 8 else rng.choice([1, 2])
    case = dict(kind=kind, shapes=shapes, rank=rank, iters=iters, rate=2.0)
    if kind == "step":
        momentum = rng.choice([0.0, 0.9, 0.9])
        case.update(lr=0.05, momentum=momentum, nesterov=bool(momentum) and rng.random() < 0.5, decay=rng.choice([0.0, 1e-4]))
        if rng.random() < 0.2:
            case.update(warmup=True)
        elif iters == 2 and rng.random() < 0.5:
            case.update(recorded=True)
    return case


# ---- shapes and buffers ------------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _shapes(text):
    if text in ("resnet18", "lstm", "gpt2-medium"):
        from powersgd_b200.models import GPT2, GPT2Config, ResNet18, wikitext2_lstm

        with torch.device("meta"):
            model = {"resnet18": ResNet18, "lstm": wikitext2_lstm, "gpt2-medium": lambda: GPT2(GPT2Config.medium())}[text]()
        return [tuple(p.shape) for p in model.parameters()]
    out = []
    for word in text.split():
        count, _, dims = word.rpartition("*")
        out += [tuple(int(d) for d in dims.split("x"))] * int(count or 1)
    return out


def _offsets(shapes):
    at, cursor = [], 0
    for s in shapes:
        at.append(cursor)
        cursor += -(-math.prod(s) // ALIGN) * ALIGN
    return at, cursor


def _views(flat, shapes):
    at, _ = _offsets(shapes)
    return [flat[a : a + math.prod(s)].view(s) for a, s in zip(at, shapes)]


def _flat(shapes, dtype=torch.float32):
    return torch.zeros(_offsets(shapes)[1], device="cuda", dtype=dtype)


def _fill(flat, shapes, gen, scale):
    """Rank 8 plus noise a tenth as large for what has two dimensions, noise for the rest."""
    for view in _views(flat, shapes):
        if view.dim() < 2:
            view.copy_(torch.randn(view.shape, generator=gen, device="cuda") * scale)
            continue
        mat = view.view(view.shape[0], -1)
        left = torch.randn(mat.shape[0], 8, generator=gen, device="cuda")
        right = torch.randn(8, mat.shape[1], generator=gen, device="cuda")
        mat.copy_(torch.randn(mat.shape, generator=gen, device="cuda"))
        torch.addmm(mat, left, right, beta=0.1 * scale, alpha=scale, out=mat)


def _inputs(case, seed):
    """Flat buffers of a case, from the seed alone: residual (small), fresh gradient, parameters, momentum."""
    shapes = _shapes(case["shapes"])
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    fresh, resid = _flat(shapes), _flat(shapes)
    _fill(fresh, shapes, gen, 0.01)
    if case["kind"] in ("rankk", "topk"):
        return shapes, dict(fresh=fresh)
    if not case.get("warmup"):  # nothing is left over while nothing is compressed
        mask = _mask(shapes, case)
        for view, keep in zip(_views(resid, shapes), mask):
            if keep:
                view.copy_(torch.randn(view.shape, generator=gen, device="cuda") * 0.001)
    bufs = dict(fresh=fresh, resid=resid)
    if case["kind"] == "step":
        param, mom = _flat(shapes), _flat(shapes)
        for view, v in zip(_views(param, shapes), _views(mom, shapes)):
            view.copy_(torch.randn(view.shape, generator=gen, device="cuda") * 0.05)
            v.copy_(torch.randn(view.shape, generator=gen, device="cuda") * 0.01)
        bufs.update(param=param, mom=mom)
    return shapes, bufs


def _mask(shapes, case):
    """Which tensors are compressed: floats per average number of floats sent, above the rate."""
    return [math.prod(s) / (0.5 * case["iters"] * min(case["rank"], *s, 1 << 30) * sum(s)) > case["rate"] for s in shapes]


def _config(case):
    return Config(rank=case["rank"], min_compression_rate=case["rate"], num_iters_per_step=case["iters"],
                  start_compressing_after_num_steps=(1 << 30) if case.get("warmup") else 0)


# ---- prepare and run ---------------------------------------------------------------------------
def _mlp(case, seed):
    a, b, c = (int(s) for s in case["sizes"].split())
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    randn = lambda *s: torch.randn(*s, generator=gen, device="cuda")  # noqa: E731
    weights = [randn(b, a) / math.sqrt(a), 0.1 * randn(b), randn(c, b) / math.sqrt(b), 0.1 * randn(c)]
    x = randn(case["batch"], a)
    y = torch.randint(0, c, (case["batch"],), generator=gen, device="cuda")
    return weights, x, y


TRAIN_BEFORE = 4  # steps in `prepare`: two eager ones, then one for each parity that gets a graph


def _prepare_train(case, seed):
    from powersgd_b200.engine import TrainStep
    from powersgd_b200.models.mlp import MLP

    weights, x, y = _mlp(case, seed)
    model = MLP(*(int(s) for s in case["sizes"].split())).cuda()
    with torch.no_grad():
        for p, w in zip(model.parameters(), weights):
            p.copy_(w)
    optimizer = torch.optim.SGD(model.parameters(), lr=case["lr"], momentum=case["momentum"])
    step = TrainStep(model, torch.nn.functional.cross_entropy, optimizer, PowerSGD(list(model.parameters()), _config(case)))
    for _ in range(TRAIN_BEFORE):
        step(x, y)
    return dict(kind="train", step=step, x=x, y=y, params=list(model.parameters()), optimizer=optimizer)


def prepare(case, seed):
    if case["kind"] == "train":
        return _prepare_train(case, seed)
    shapes, bufs = _inputs(case, seed)
    state = dict(kind=case["kind"], bufs=bufs)
    if case["kind"] in ("rankk", "topk"):
        from powersgd_b200.paper.reducers import RankKReducer, TopKReducer

        state["send"] = _views(bufs["fresh"], shapes)
        bufs["out"], bufs["memory"] = _flat(shapes), _flat(shapes)
        state["out"], state["memory"] = _views(bufs["out"], shapes), _views(bufs["memory"], shapes)
        if case["kind"] == "rankk":
            state["reducer"] = RankKReducer(HARNESS_SEED, bufs["fresh"].device, reuse_query=True, rank=case["rank"])
        else:
            state["reducer"] = TopKReducer(HARNESS_SEED, bufs["fresh"].device, compression=COMPRESSION)
        return state
    state["fresh"], state["grads"] = _views(bufs["fresh"], shapes), _views(bufs["resid"], shapes)
    if case["kind"] == "aggregate":
        state["aggregator"] = PowerSGD(state["grads"], _config(case))
        return state
    params = [torch.nn.Parameter(v) for v in _views(bufs["param"], shapes)]
    for p, g in zip(params, state["grads"]):
        p.grad = g
    optimizer = torch.optim.SGD(params, lr=case["lr"], momentum=case["momentum"], nesterov=case.get("nesterov", False),
                                weight_decay=case.get("decay", 0.0))
    if case["momentum"]:
        for p, v in zip(params, _views(bufs["mom"], shapes)):
            optimizer.state[p]["momentum_buffer"] = v
    state.update(optimizer=optimizer, aggregator=PowerSGD(params, _config(case)))
    if case.get("recorded"):
        # one eager step first, as a recording program does; an even number of half-iterations per
        # step leaves the same side next, so one graph serves every step
        _step(state)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            _step(state)
        state["graph"] = graph
    return state


def _step(state):
    torch._foreach_add_(state["grads"], state["fresh"])  # what backward does with the fresh gradients
    optimizer_step(state["optimizer"], state["aggregator"])


def run(state):
    kind = state["kind"]
    if kind == "train":
        loss = state["step"](state["x"], state["y"])
        moms = [s["momentum_buffer"] for s in state["optimizer"].state.values() if s.get("momentum_buffer") is not None]
        return [loss, state["params"], state["params"][0].grad, moms]
    if kind in ("rankk", "topk"):
        state["reducer"].reduce(state["send"], state["out"], state["memory"])
        return [state["bufs"]["out"], state["bufs"]["memory"]]
    if kind == "aggregate":
        torch._foreach_add_(state["grads"], state["fresh"])
        return [state["aggregator"].aggregate(state["grads"]), state["bufs"]["resid"]]
    if "graph" in state:
        state["graph"].replay()
    else:
        _step(state)
    return [state["bufs"]["param"], state["bufs"]["mom"], state["bufs"]["resid"]]


# ---- what a pass cannot do without ---------------------------------------------------------------
def work(case):
    if case["kind"] == "train":
        a, b, c = (int(s) for s in case["sizes"].split())
        n, batch = a * b + b + b * c + c, case["batch"]
        # parameters and residual read and written (momentum too), inputs read; three products
        return {"bytes": 4.0 * (n * (2 + 2 * bool(case["momentum"])) + 2 * a * b + batch * a),
                "flops": 6.0 * batch * (a * b + b * c) + a * b * case["rank"] * 4.0 * case["iters"]}
    shapes = _shapes(case["shapes"])
    total = sum(math.prod(s) for s in shapes)
    if case["kind"] == "topk":
        return {"bytes": 12.0 * total, "flops": 0.0}
    if case["kind"] == "rankk":
        mats = sum(math.prod(s) for s in shapes if len(s) > 1)
        return {"bytes": 4.0 * (3 * mats + 2 * (total - mats)), "flops": 6.0 * mats * case["rank"]}
    mats = sum(math.prod(s) for s, k in zip(shapes, _mask(shapes, case)) if k and not case.get("warmup"))
    # fresh gradient read, residual read and written (zeroed where nothing is left over); then the
    # update written, or parameters and momentum read and written
    per = 4 if case["kind"] == "aggregate" else 5 + 2 * bool(case["momentum"])
    return {"bytes": 4.0 * (per * mats + (per - 1) * (total - mats)), "flops": mats * 4.0 * case["rank"] * case["iters"]}


def tolerance(case):
    """Single precision throughout: sums of up to 50 000 products, a rank-r basis between them. Against
    64 bits the present kernels are 1e-7 to 5e-6 off; above rank 8, where the basis also spans noise
    directions of nearly equal size and the residual is the small difference, up to 5e-5."""
    if case["kind"] == "topk":
        return "exact"  # values are selected and copied, not computed
    return {"rel": 2e-4 if case["rank"] > 8 else 2e-5}


# ---- the same in 64 bits, without the package ------------------------------------------------------
def _basis(x):
    """Orthonormal columns spanning `x` (one joint norm for a whole group at rank 1)."""
    if x.shape[-1] == 1:
        return x / x.norm().clamp(min=1e-16)
    return torch.linalg.qr(x)[0]


class _Exact:
    """Warm-started power iteration with error feedback on the compressed tensors of a case."""

    def __init__(self, case, shapes):
        self.iters, self.steps = case["iters"], 0
        self.keep = _mask(shapes, case)
        self.groups = {}
        for i, (s, k) in enumerate(zip(shapes, self.keep)):
            if k:
                self.groups.setdefault((s[0], math.prod(s[1:])), []).append(i)
        gen = torch.Generator(device="cuda").manual_seed(0)
        draw_one = lambda b, rows, r: torch.randn(b, rows, r, generator=gen, device="cuda").double()  # noqa: E731
        rank = lambda nm: min(case["rank"], *nm)  # noqa: E731
        self.p = {nm: draw_one(len(i), nm[0], rank(nm)) for nm, i in self.groups.items()}
        self.q = {nm: draw_one(len(i), nm[1], rank(nm)) for nm, i in self.groups.items()}

    def __call__(self, grads):
        """Updates of the compressed tensors, by index; `grads` keep what is left over."""
        updates = {}
        for nm, members in self.groups.items():
            m = torch.stack([grads[i].reshape(nm) for i in members])
            total = torch.zeros_like(m)
            for t in range(self.iters):
                if (self.steps * self.iters + t) % 2 == 0:
                    self.p[nm] = _basis(self.p[nm])
                    self.q[nm] = m.transpose(1, 2) @ self.p[nm]
                else:
                    self.q[nm] = _basis(self.q[nm])
                    self.p[nm] = m @ self.q[nm]
                product = self.p[nm] @ self.q[nm].transpose(1, 2)
                total += product
                m -= product
            for j, i in enumerate(members):
                grads[i].copy_(m[j].reshape(grads[i].shape))
                updates[i] = total[j].reshape(grads[i].shape)
        self.steps += 1
        return updates


def _sgd(case, p, v, g):
    g = g + case.get("decay", 0.0) * p
    if case["momentum"]:
        v.mul_(case["momentum"]).add_(g)
        g = g + case["momentum"] * v if case.get("nesterov") else v
    p.sub_(case["lr"] * g)


def _exact_train(case, seed):
    weights, x, y = _mlp(case, seed)
    params = [w.double() for w in weights]
    shapes = [tuple(p.shape) for p in params]
    moms, resid = [torch.zeros_like(p) for p in params], [torch.zeros_like(p) for p in params]
    compress, x = _Exact(case, shapes), x.double()
    for _ in range(TRAIN_BEFORE + 1):
        leaves = [p.clone().requires_grad_(True) for p in params]
        hidden = torch.relu(x @ leaves[0].t() + leaves[1])
        loss = torch.nn.functional.cross_entropy(hidden @ leaves[2].t() + leaves[3], y)
        for r, g in zip(resid, torch.autograd.grad(loss, leaves)):
            r.add_(g)
        updates = compress(resid)
        for i, (p, v) in enumerate(zip(params, moms)):
            _sgd(case, p, v, updates[i] if i in updates else resid[i].clone())
            if i not in updates:
                resid[i].zero_()
    return [loss.detach(), params, resid[0], moms if case["momentum"] else []]


def exact(case, seed):
    if case["kind"] == "train":
        return _exact_train(case, seed)
    shapes, bufs = _inputs(case, seed)
    wide = {k: b.double() for k, b in bufs.items()}
    views = {k: _views(b, shapes) for k, b in wide.items()}
    if case["kind"] in ("rankk", "topk"):
        out, memory = _flat(shapes, torch.float64), _flat(shapes, torch.float64)
        stream = np.random.RandomState(HARNESS_SEED)
        for x, o, mem in zip(views["fresh"], _views(out, shapes), _views(memory, shapes)):
            if case["kind"] == "topk":
                k = max(1, int(0.5 * COMPRESSION * x.numel()))
                at = x.reshape(-1).abs().topk(k).indices
                o.view(-1)[at] = x.reshape(-1)[at]
                mem.copy_(x - o)
            elif x.dim() < 2:
                o.copy_(x)
            else:
                m = x.reshape(x.shape[0], -1)
                torch.manual_seed(int(stream.randint(1_000_000_000)))
                q = torch.randn(m.shape[1], min(*m.shape, case["rank"]), device="cuda").double()
                p = _basis(m @ q)
                o.view(m.shape).copy_(p @ (p.t() @ m))
                mem.copy_(x - o)
        return [out, memory]
    grads, fresh = views["resid"], views["fresh"]
    compress = _Exact(case, shapes)
    if case["kind"] == "aggregate":
        for g, f in zip(grads, fresh):
            g.add_(f)
        updates = compress(grads)
        outs = [updates[i] if i in updates else grads[i].clone() for i in range(len(shapes))]
        for i, g in enumerate(grads):
            if i not in updates:
                g.zero_()
        return [outs, wide["resid"]]
    for _ in range(2 if case.get("recorded") else 1):
        for g, f in zip(grads, fresh):
            g.add_(f)
        updates = {} if case.get("warmup") else compress(grads)
        for i, (p, v) in enumerate(zip(views["param"], views["mom"])):
            _sgd(case, p, v, updates[i] if i in updates else grads[i].clone())
            if i not in updates:
                grads[i].zero_()
    return [wide["param"], wide["mom"], wide["resid"]]
