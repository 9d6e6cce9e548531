"""Workloads that represent what users of heavyball_b200 run, for timing and output comparison.

Two families, each called through public entry points only:

* one or several ``optimizer.step()`` calls of an optimizer class in the middle of a run (state exists, gradients are
  handed over as a backward pass would), on the parameter shapes of the configurations in ``bench.py`` and of
  ``benchmarks/bench_optimizer_step.py``, and on odd small shapes;
* the model-side ops, forward and backward under bf16 autocast: the head with its cross-entropy and a transformer block.

Kinds: ``adamw``, ``muon``, ``soap``, ``psgd``, ``head``, ``block``.  :func:`exact` restates each of them in 64-bit torch.
"""

from __future__ import annotations

import math

import torch
import torch.nn.functional as F

import heavyball_b200 as hb
from heavyball_b200.models.gpt import Block, GPTConfig
from heavyball_b200.ops import nn as hbnn

DEV = "cuda"

# ---------------------------------------------------------------------------------------- the cases


def listed():
    return [
        # the parameters of GPT-2 small that Muon leaves to AdamW: embeddings, biases and norms (those of two layers; 39.5 M)
        {"name": "adamw-gpt2-rest", "kind": "adamw", "dtype": "float32", "ecc": False,
         "shapes": "50304x768,1024x768," + ",".join(["768,768,2304,768,768,768,3072,768"] * 2) + ",768,768"},
        # AdamW(ecc, mars, caution) over the default workload of the optimizer-step benchmark, 2048 x 2048 matrices
        {"name": "adamw-ecc-8x2048", "kind": "adamw", "shapes": ",".join(["2048x2048"] * 8), "dtype": "float32", "ecc": True},
        # bf16 parameters and gradients of odd sizes (fine-tuning adapters, small heads): ragged ends, unaligned starts
        {"name": "adamw-bf16-ragged", "kind": "adamw", "dtype": "bfloat16", "ecc": False,
         "shapes": "1000x333,333,77x4099,1,129x65,5,1025,3001x1023"},
        # Muon on small odd matrices: one bucket per shape, launches and latency
        {"name": "muon-ragged", "kind": "muon", "shapes": "333x1000,333x1000,200x77,130x130,520x264", "dtype": "float32", "ecc": False},
        # Muon on the 48 block matrices of GPT-2 small (the flagship configuration)
        {"name": "muon-gpt2", "kind": "muon", "dtype": "float32", "ecc": False,
         "shapes": ",".join(["2304x768,768x768,3072x768,768x3072"] * 12)},
        # one layer of the Llama-3-8B configuration: Muon with error-corrected bf16 parameters and state, MARS, caution
        {"name": "muon-llama8b-layer", "kind": "muon", "dtype": "bfloat16", "ecc": True,
         "shapes": "4096x4096,1024x4096,1024x4096,4096x4096,14336x4096,14336x4096,4096x14336"},
        # one layer of the Llama-1.3B SOAP configuration over a whole refresh period (ten steps, one refresh)
        {"name": "soap-llama1.3b-layer", "kind": "soap", "freq": 10, "max_dim": 4096,
         "shapes": "2048x2048,2048x2048,2048x2048,2048x2048,5504x2048,5504x2048,2048x5504"},
        # SOAP at its default refresh period (two steps, one refresh) on eight 1024 x 1024 matrices
        {"name": "soap-8x1024", "kind": "soap", "freq": 2, "max_dim": 2048, "shapes": ",".join(["1024x1024"] * 8)},
        # two layers of the GPT-350M PSGDKron configuration, a step between two fits (nine of ten)
        {"name": "psgd-gpt350m", "kind": "psgd", "fit": False,
         "shapes": ",".join(["3072x1024,1024x1024,4096x1024,1024x4096"] * 2)},
        # the first thousand steps of PSGDKron's default schedule fit the preconditioner every time
        {"name": "psgd-fit-8x1024", "kind": "psgd", "fit": True, "shapes": ",".join(["1024x1024"] * 8)},
        # the head of GPT-2 small with its cross-entropy at the training batch, forward and backward
        {"name": "gpt2-head", "kind": "head", "tokens": 16384, "d": 768, "vocab": 50257, "ignored": 0.0},
        # one transformer block of GPT-2 small at its training batch, forward and backward
        {"name": "gpt2-block", "kind": "block", "batch": 16, "seq": 1024, "d": 768, "heads": 12},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["adamw", "adamw", "muon", "muon", "soap", "psgd", "head", "block"])
    if kind == "adamw":
        total, shapes = _log_int(rng, 2_000, 40_000_000), []
        n = rng.randint(1, 20)
        for _ in range(n):
            size = max(1, int(total / n * rng.uniform(0.1, 1.9)))
            cols = min(size, rng.choice([1, 7, 64, 333, 768, 1024, 2048]))
            shapes.append(f"{max(1, size // cols)}x{cols}" if cols > 1 else str(size))
        ecc = rng.random() < 0.4
        return {"kind": "adamw", "shapes": ",".join(shapes), "dtype": "float32" if ecc else rng.choice(["float32", "bfloat16"]), "ecc": ecc}
    if kind == "muon":
        shapes = []
        for _ in range(rng.randint(1, 3)):
            r, c = _log_int(rng, 96, 3072), _log_int(rng, 96, 3072)
            if rng.random() < 0.6:
                r, c = max(64, r // 64 * 64), max(64, c // 64 * 64)
            shapes += [f"{r}x{c}"] * rng.randint(1, 6)
        ecc = rng.random() < 0.3
        return {"kind": "muon", "shapes": ",".join(shapes), "dtype": "bfloat16" if ecc else "float32", "ecc": ecc}
    if kind in ("soap", "psgd"):
        r, c = _log_int(rng, 130, 2048), _log_int(rng, 130, 2048)
        if rng.random() < 0.7:
            r, c = max(128, r // 128 * 128), max(128, c // 128 * 128)
        shapes = ",".join([f"{r}x{c}"] * rng.randint(1, 6))
        if kind == "soap":
            return {"kind": "soap", "freq": rng.choice([2, 10]), "max_dim": 2048, "shapes": shapes}
        return {"kind": "psgd", "fit": rng.random() < 0.5, "shapes": shapes}
    if kind == "head":
        return {"kind": "head", "tokens": _log_int(rng, 128, 16384), "d": rng.choice([256, 768, 1024]),
                "vocab": _log_int(rng, 1000, 50257), "ignored": round(rng.uniform(0, 0.2), 3)}
    heads = rng.choice([4, 8, 12, 16])
    return {"kind": "block", "batch": rng.randint(1, 16), "seq": _log_int(rng, 64, 1024), "d": 64 * heads, "heads": heads}


# ---------------------------------------------------------------------------------------- inputs


def _shapes(case):
    return [tuple(int(v) for v in s.split("x")) for s in case["shapes"].split(",")]


def _gen(seed, salt=0):
    return torch.Generator(DEV).manual_seed(int(seed) * 1009 + salt)


def _randn(shape, gen, std=1.0, dtype=torch.float32):
    return (torch.randn(shape, generator=gen, device=DEV) * std).to(dtype)


def _optimizer_inputs(case, seed):
    """(parameters, gradients of each step): weights of std 0.02; gradients of std 1e-3."""
    gen, dtype = _gen(seed), getattr(torch, case.get("dtype", "float32"))
    shapes = _shapes(case)
    params = [_randn(s, gen, 0.02, dtype) for s in shapes]
    grads = [[_randn(s, gen, 1e-3, dtype) for s in shapes] for _ in range(3)]
    return params, grads


def _orthogonal(n, gen):
    """A dense orthogonal matrix in 64 bits: a product of three reflections."""
    q = torch.eye(n, dtype=torch.float64, device=DEV)
    for _ in range(3):
        v = torch.randn(n, 1, dtype=torch.float64, generator=gen, device=DEV)
        v /= v.norm()
        q = q - 2 * (q @ v) @ v.mT
    return q


def _soap_checkpoint(case, seed):
    """Mid-run state: eigenbases, statistics they track (eigenvalues over two decades, basis a few percent off), moments."""
    gen, out = _gen(seed, 1), []
    for shape in _shapes(case):
        Q, GG = [], []
        for n in shape:
            if n > case["max_dim"]:
                Q.append(None), GG.append(None)
                continue
            q = _orthogonal(n, gen)
            lam = torch.logspace(2, 0, n, dtype=torch.float64, device=DEV).sqrt()
            s = torch.randn(n, n, dtype=torch.float64, generator=gen, device=DEV) * (0.03 / math.sqrt(n))
            s = torch.triu(s, 1)
            m = torch.eye(n, dtype=torch.float64, device=DEV) + s + s.mT
            gg = q @ (lam[:, None] * m * lam[None, :]) @ q.mT
            Q.append(q.float()), GG.append(((gg + gg.mT) / 2).float())
        exp_avg = _randn(shape, gen, 3e-4)
        exp_avg_sq = _randn(shape, gen, 1e-3).square() * 0.5 + 5e-7
        out.append({"exp_avg": exp_avg, "exp_avg_sq": exp_avg_sq, "Q": Q, "GG": GG})
    return out


def _psgd_checkpoint(case, seed):
    """Mid-run Kronecker factors: upper triangular, diagonally dominant; the lower bounds of their fit."""
    gen, out = _gen(seed, 1), []
    for shape in _shapes(case):
        factors = []
        for n in shape:
            q = torch.triu(_randn((n, n), gen, 0.3 / math.sqrt(n)), 1)
            factors.append(q + torch.diag(1.0 + 0.5 * torch.rand(n, generator=gen, device=DEV)))
        out.append({"Q": factors, "lb": [float(10 * n) for n in shape]})
    return out


def _load(opt, per_param):
    """Puts slot values into the optimizer through its checkpoint, as resuming a run does."""
    sd = opt.state_dict()
    for i, values in enumerate(per_param):
        for st in sd["state"][i].values():
            if not isinstance(st, dict):
                continue
            for key in list(st):
                for slot, make in values.items():
                    if key.rsplit("_", 1)[0].endswith(slot):
                        st[key] = make(st[key])
    opt.load_state_dict(sd)


def _state_tensors(opt, params):
    """Every floating or integer state tensor of the parameters, in a fixed order.  Not the residual of an error-corrected
    weight: after an orthogonalisation in bf16 products it is noise (any change in the order of a sum redraws it)."""
    found = []

    def walk(v):
        if isinstance(v, torch.Tensor):
            if v.ndim and v.numel() > 2:
                found.append(v)
        elif isinstance(v, dict):
            for k in sorted(v, key=str):
                if k != "param::ecc":
                    walk(v[k])
        elif isinstance(v, (list, tuple)):
            for x in v:
                walk(x)

    for p in params:
        walk(opt.state[p])
    return found


def _build(case, params):
    kind = case["kind"]
    if kind == "adamw":
        return hb.AdamW(params, lr=3e-4, weight_decay=0.01, **(dict(ecc="bf16+8", mars=True, caution=True) if case["ecc"] else {}))
    if kind == "muon":
        return hb.Muon(params, lr=0.02, **(dict(ecc="bf16+8", param_ecc="bf16+8", mars=True, caution=True) if case["ecc"] else {}))
    if kind == "soap":
        return hb.SOAP(params, lr=3e-3, betas=(0.95, 0.95), shampoo_beta=0.95, precondition_frequency=case["freq"],
                       max_precond_dim=case["max_dim"])  # fmt: skip
    return hb.PSGDKron(params, max_size_triangular=8192, ecc="bf16+8", preconditioner_update_probability=1.0 if case["fit"] else 0.0)


def _step(opt, params, grads):
    for p, g in zip(params, grads):
        p.grad = g
    opt.step()


def _triu_line(q):
    n = q.shape[-1]
    i = torch.triu_indices(n, n, device=q.device)
    return q[i[0], i[1]]


def prepare(case, seed):
    torch.manual_seed(seed)
    kind = case["kind"]
    if kind == "head":
        h, w, targets = _head_inputs(case, seed)
        return {"kind": kind, "vocab": case["vocab"], "h": h.requires_grad_(), "w": w.requires_grad_(), "targets": targets}
    if kind == "block":
        x, pending, gx, gm, weights = _block_inputs(case, seed)
        blk = Block(GPTConfig(n_layer=1, n_head=case["heads"], d_model=case["d"])).to(DEV)
        with torch.no_grad():
            for p, w in zip(blk.parameters(), weights):
                p.copy_(w)
        return {"kind": kind, "blk": blk, "params": list(blk.parameters()), "x": x.requires_grad_(),
                "pending": pending.requires_grad_(), "gx": gx, "gm": gm}  # fmt: skip
    values, grads = _optimizer_inputs(case, seed)
    params = [torch.nn.Parameter(v) for v in values]
    opt = _build(case, params)
    _step(opt, params, [g.clone() for g in grads[0]])
    if kind == "soap":
        fill = lambda new: (lambda old: [None if o is None else n.view(o.shape) for o, n in zip(old, new)])  # noqa: E731
        _load(opt, [{"_exp_avg": lambda o, c=c: c["exp_avg"].view(o.shape), "_exp_avg_sq": lambda o, c=c: c["exp_avg_sq"].view(o.shape),
                     "_Q": fill(c["Q"]), "_GG": fill(c["GG"])} for c in _soap_checkpoint(case, seed)])  # fmt: skip
    if kind == "psgd":
        _load(opt, [{"_Q": lambda old, c=c: [(o[0], _triu_line(q).view(o[1].shape)) for o, q in zip(old, c["Q"])],
                     "_running_lower_bound": lambda old, c=c: [torch.full_like(o, v) for o, v in zip(old, c["lb"])]}
                    for c in _psgd_checkpoint(case, seed)])  # fmt: skip
        with torch.no_grad():  # the weights that belong to this checkpoint
            for p, v in zip(params, _optimizer_inputs(case, seed)[0]):
                p.copy_(v)
    _step(opt, params, [g.clone() for g in grads[1]])
    # first-order state is updated in place; matrix statistics may move to other buffers, so they are looked up after a pass
    held = _state_tensors(opt, params) if kind in ("adamw", "muon") else None
    return {"kind": kind, "opt": opt, "params": params, "held": held, "grads": grads[2], "steps": case.get("freq", 1)}


def run(state):
    kind = state["kind"]
    if kind == "head":
        h, w = state["h"], state["w"]
        with torch.autocast("cuda", dtype=torch.bfloat16):
            loss = hbnn.linear_cross_entropy(h, w, state["targets"], state["vocab"])
        return [loss.detach(), *torch.autograd.grad(loss, (h, w))]
    if kind == "block":
        with torch.autocast("cuda", dtype=torch.bfloat16):
            x, m = state["blk"](state["x"], state["pending"])
        grads = torch.autograd.grad((x, m), (state["x"], state["pending"], *state["params"]), (state["gx"], state["gm"]))
        return [x.detach(), m.detach(), *grads]
    for _ in range(state["steps"]):
        _step(state["opt"], state["params"], state["grads"])
    held = state["held"] if state["held"] is not None else _state_tensors(state["opt"], state["params"])
    weights = [p.detach() for p in state["params"]]
    return weights + held[max(0, len(weights) + len(held) - 64) :]  # at most 64: all weights, the state of the last of them


# ---------------------------------------------------------------------------------------- model-side inputs


def _head_inputs(case, seed):
    gen = _gen(seed)
    rows = -(-case["vocab"] // 64) * 64  # the models store a multiple of 64 rows; the extra ones are zero
    h = _randn((case["tokens"], case["d"]), gen, 1.0, torch.bfloat16)
    w = _randn((rows, case["d"]), gen, 0.02)
    w[case["vocab"] :].zero_()
    targets = torch.randint(0, case["vocab"], (case["tokens"],), generator=gen, device=DEV)
    drop = torch.rand(case["tokens"], generator=gen, device=DEV) < case["ignored"]
    return h, w, torch.where(drop, torch.full_like(targets, -100), targets)


def _block_inputs(case, seed):
    gen, d = _gen(seed), case["d"]
    shape = (case["batch"], case["seq"], d)
    x, pending = _randn(shape, gen), _randn(shape, gen, 0.1, torch.bfloat16)
    gx, gm = _randn(shape, gen, 1e-3), _randn(shape, gen, 1e-3, torch.bfloat16)
    # ln1 weight, bias; qkv; proj; ln2; fc; out: in the order of Block.parameters()
    weights = [1 + _randn((d,), gen, 0.02), _randn((d,), gen, 0.02), _randn((3 * d, d), gen, 0.02), _randn((3 * d,), gen, 0.02),
               _randn((d, d), gen, 0.02), _randn((d,), gen, 0.02), 1 + _randn((d,), gen, 0.02), _randn((d,), gen, 0.02),
               _randn((4 * d, d), gen, 0.02), _randn((4 * d,), gen, 0.02), _randn((d, 4 * d), gen, 0.02), _randn((d,), gen, 0.02)]  # fmt: skip
    return x, pending, gx, gm, weights


# ---------------------------------------------------------------------------------------- work and tolerances


def work(case):
    kind = case["kind"]
    if kind == "head":
        t, d, v = case["tokens"], case["d"], case["vocab"]
        # h and the fp32 weight in, both gradients out; the logits are a temporary of the present method
        return {"bytes": 4 * t * d + 8 * v * d + 8 * t, "flops": 6 * t * d * v}
    if kind == "block":
        b, s, d = case["batch"], case["seq"], case["d"]
        t = b * s
        # x, pending, both outputs, both incoming and both outgoing gradients; weights in, their gradients out
        return {"bytes": t * d * (4 + 2 + 4 + 2 + 4 + 2 + 4 + 2) + 2 * 4 * 12 * d * d,
                "flops": 3 * 2 * t * 12 * d * d + (2 + 5) * b * s * s * d}  # causal attention: half of the square
    n = sum(math.prod(s) for s in _shapes(case))
    if kind == "adamw":
        p = 2 if case["dtype"] == "bfloat16" else 4
        # parameter in and out, gradient in, two moments in and out (and MARS' old gradient, all three in 16 + 8 bits)
        return {"bytes": n * (3 * p + (3 * 2 * 3 if case["ecc"] else 2 * 2 * 4)), "flops": 15 * n}
    if kind == "muon":
        flops = 0
        for s in _shapes(case):
            m, k = min(s), max(s)
            flops += 5 * (m * m * k + m**3 + 2 * m * m * k)  # Gram and polynomial are symmetric: half of the square
        per = (3 + 3 + 2 + 6 + 6) if case["ecc"] else (4 + 4 + 4 + 8)
        return {"bytes": n * per, "flops": flops}
    sides = [[d for d in s if d <= case.get("max_dim", 1 << 30)] for s in _shapes(case)]
    factor = sum(d * d for s in sides for d in s)
    if kind == "soap":
        project = sum(2 * 2 * math.prod(s) * d for s, ds in zip(_shapes(case), sides) for d in ds)
        stats = sum(math.prod(s) * d for s, ds in zip(_shapes(case), sides) for d in ds)
        # refresh: power iteration, QR, rotation of the first moment
        refresh = sum(2 * d**3 + 4 / 3 * d**3 + 2 * d**3 + 2 * math.prod(s) * d for s, ds in zip(_shapes(case), sides) for d in ds)
        steps = case["freq"]
        return {"bytes": steps * (28 * n + 12 * factor) + 8 * factor, "flops": steps * (project + stats) + refresh}
    apply = sum(2 * math.prod(s) * d for s, ds in zip(_shapes(case), sides) for d in ds)
    if not case["fit"]:
        return {"bytes": n * (12 + 6) + 2 * factor, "flops": apply}
    # both outer products per side (symmetric), A = Q_l G Q_r^T and V Q^-1 (triangular), triu(.) Q, and Q^T Q
    fit = sum(2 * math.prod(s) * d + 2 * math.prod(s) * d + d**3 / 3 + d**3 / 3 for s, ds in zip(_shapes(case), sides) for d in ds)
    return {"bytes": n * (12 + 6) + 4 * factor, "flops": apply + fit}


def tolerance(case):
    kind = case["kind"]
    if kind == "adamw":
        if case["dtype"] == "bfloat16":
            return {"rel": 4e-3, "max": 0.05}
        # moments are kept in 16 + 8 bits and rounded stochastically: a last-bit change of a value moves whole units
        return {"rel": 2e-3, "max": 0.05, "differ": 0.01} if case["ecc"] else {"rel": 2e-6, "max": 2e-4}
    if kind == "muon":
        return {"rel": 4e-3, "max": 0.1, "differ": 0.01} if case["ecc"] else {"rel": 2e-3, "max": 0.05}
    if kind == "soap":
        return {"rel": 1e-4, "max": 0.05}
    if kind == "psgd":
        return {"rel": 2e-3, "max": 0.05, "differ": 0.01}
    return {"rel": 1e-2, "max": 0.5}


# ---------------------------------------------------------------------------------------- 64-bit restatement


def _debias(beta, step):
    return 1 - (1 - beta) / (1 - beta**step) if step > 0 else 0.0


def _mars(g, old):
    a = -0.9 * 0.0025 / (1 - 0.0025)
    return g * (1 - a) + old * a


def _cautious(u, g):
    keep = torch.signbit(g) == torch.signbit(u)
    return u * keep * (u.numel() / max(1, int(keep.sum())))


def _exact_adamw(case, seed):
    values, grads = _optimizer_inputs(case, seed)
    out, states = [], []
    for i, p in enumerate(values):
        p = p.double()
        m, v, old = (torch.zeros_like(p) for _ in range(3))
        for step in (1, 2, 3):
            raw = g = grads[step - 1][i].double()
            if case["ecc"]:
                g = _mars(g, raw if step == 1 else old)
                old = raw
            b1, b2 = _debias(0.9, step), _debias(0.99, step)
            m, v = m * b1 + g * (1 - b1), v * b2 + g * g * (1 - b2)
            u = m / v.sqrt().clamp_min(1e-8)
            if case["ecc"]:
                u = _cautious(u, g)
            p = p * (1 - 0.01 * 3e-4) - 3e-4 * u
        out.append(p)
        # the order of _state_tensors: slots by name, residuals behind their primaries; tensors of one or two elements left out
        slots = [old, None, m, None, v, None] if case["ecc"] else [m, v]
        states += slots if p.numel() > 2 else []
    return out + states[max(0, len(out) + len(states) - 64) :]


def _newton_schulz(x):
    tall = x.shape[0] > x.shape[1]
    x = x / x.norm().clamp_min(1e-7)
    x = x.mT if tall else x
    for a, b, c in ((4.0848, -6.8946, 2.9270), (3.9505, -6.3029, 2.6377), (3.7418, -5.5913, 2.3037), (2.8769, -3.1427, 1.2046),
                    (2.8366, -3.0525, 1.2012)):  # fmt: skip
        s = x @ x.mT
        x = a * x + (b * s + c * (s @ s)) @ x
    return x.mT if tall else x


def _exact_muon(case, seed):
    values, grads = _optimizer_inputs(case, seed)
    out, states = [], []
    for i, p in enumerate(values):
        p = p.double()
        m, old = torch.zeros_like(p), torch.zeros_like(p)
        for step in (1, 2, 3):
            raw = g = grads[step - 1][i].double()
            if case["ecc"]:
                g = _mars(g, raw if step == 1 else old)
                old = raw
            m = m * 0.9 + g * 0.1
            u = _newton_schulz(g + m) * max(1.0, p.shape[0] / p.shape[1]) ** 0.5
            if case["ecc"]:
                u = _cautious(u, raw)
            p = p - 0.02 * u
        out.append(p)
        states += [old, None, m, None] if case["ecc"] else [m]
    return out + states[max(0, len(out) + len(states) - 64) :]


def _exact_soap(case, seed):
    values, grads = _optimizer_inputs(case, seed)
    out, states = [], []
    for i, (p, c) in enumerate(zip(values, _soap_checkpoint(case, seed))):
        p, m, v = p.double(), c["exp_avg"].double(), c["exp_avg_sq"].double()
        Q = [None if q is None else q.double() for q in c["Q"]]
        GG = [None if q is None else q.double() for q in c["GG"]]
        fired = 1 / case["freq"]  # after the initialising step
        for step in range(2, 3 + case["freq"]):
            before, fired = fired, fired + 1 / case["freq"]
            u = grads[1 if step == 2 else 2][i].double()
            x = u if Q[0] is None else Q[0].mT @ u
            x = x if Q[1] is None else x @ Q[1]
            b1 = b2 = _debias(0.95, step - 1)
            m, v = m * b1 + x * (1 - b1), v * b2 + x * x * (1 - b2)
            n = m / v.sqrt().clamp_min(1e-8)
            n = n if Q[0] is None else Q[0] @ n
            n = n if Q[1] is None else n @ Q[1].mT
            p = p * (1 - 0.01 * 3e-3) - 3e-3 * n
            w = 1 - _debias(0.95, step)
            GG = [None if gg is None else gg + (o - gg) * w for gg, o in zip(GG, (u @ u.mT, u.mT @ u))]
            if int(fired) > int(before):
                new = [None if q is None else _refresh(gg, q) for gg, q in zip(GG, Q)]
                m = m if Q[0] is None else new[0].mT @ (Q[0] @ m)
                m = m if Q[1] is None else (m @ Q[1].mT) @ new[1]
                Q = new
        out.append(p)
        one = lambda xs: [x[None] for x in xs if x is not None]  # noqa: E731
        states += [*one(GG), *one(Q), m[None], v[None]]
    return out + states


def _refresh(gg, q):
    power = gg @ q
    order = torch.argsort((q * power).sum(0), descending=True)
    basis, r = torch.linalg.qr(power[:, order])
    basis = basis * torch.sign(torch.diagonal(r))
    out = torch.empty_like(basis)
    out[:, order] = basis
    return out


def _exact_psgd(case, seed):
    if case["fit"]:
        return None  # the fit draws its own probe vectors on the device
    values, grads = _optimizer_inputs(case, seed)
    out, states = [], []
    for i, (p, c) in enumerate(zip(values, _psgd_checkpoint(case, seed))):
        p = p.double()
        m = torch.zeros_like(p)
        left, right = (q.double().mT @ q.double() for q in c["Q"])
        for step in (1, 2, 3):
            b1 = _debias(0.9, step)
            m = m * b1 + grads[step - 1][i].double() * (1 - b1)
            if step > 1:  # the weights are those of the checkpoint that is loaded after the first step
                x = (left @ m @ right) / 1.5
                u = (0.9 * torch.tanh(x) + 0.1 * torch.sign(x) * torch.log1p(x.abs())) * 1.5  # trust-region clip
                p = p - 1e-3 * u.clamp(-2, 2)
        out.append(p)
        states += [m, None, _triu_line(c["Q"][0])[None], _triu_line(c["Q"][1])[None]]
    return out + states[max(0, len(out) + len(states) - 64) :]


def _exact_head(case, seed):
    h, w, targets = _head_inputs(case, seed)
    h64, w64 = h.double().requires_grad_(), w.to(torch.bfloat16).double().requires_grad_()
    loss = F.cross_entropy(F.linear(h64, w64[: case["vocab"]]), targets, ignore_index=-100)
    return [loss.detach(), *torch.autograd.grad(loss, (h64, w64))]


def _exact_block(case, seed):
    x, pending, gx, gm, weights = _block_inputs(case, seed)
    x, pending, *w = [t.double().requires_grad_() for t in (x, pending, *weights)]
    b, s, d = case["batch"], case["seq"], case["d"]
    outs, grads = [], [torch.zeros_like(t) for t in w]
    for i in range(b):  # sequence by sequence: the attention matrix in 64 bits is large
        xi, pi = x.detach()[i].requires_grad_(), pending.detach()[i].requires_grad_()
        s1 = xi + pi
        q, k, v = F.linear(F.layer_norm(s1, (d,), w[0], w[1], 1e-5), w[2], w[3]).view(s, 3, case["heads"], -1).permute(1, 2, 0, 3)
        att = (q @ k.mT / math.sqrt(d // case["heads"])).masked_fill(torch.ones(s, s, dtype=torch.bool, device=DEV).triu(1), float("-inf"))
        s2 = s1 + F.linear((att.softmax(-1) @ v).transpose(0, 1).reshape(s, d), w[4], w[5])
        mlp = F.linear(F.gelu(F.linear(F.layer_norm(s2, (d,), w[6], w[7], 1e-5), w[8], w[9]), approximate="tanh"), w[10], w[11])
        got = torch.autograd.grad((s2, mlp), (xi, pi, *w), (gx[i].double(), gm[i].double()))
        outs.append((s2.detach(), mlp.detach(), got[0], got[1]))
        for acc, g in zip(grads, got[2:]):
            acc += g
    xs, ms, dx, dp = (torch.stack(t) for t in zip(*outs))
    return [xs, ms, dx, dp, *grads]


def exact(case, seed):
    kind = case["kind"]
    return {"adamw": _exact_adamw, "muon": _exact_muon, "soap": _exact_soap, "psgd": _exact_psgd, "head": _exact_head,
            "block": _exact_block}[kind](case, seed)  # fmt: skip
