"""The library's work as its users have it do, as a set of measurable cases.

`listed()` holds fixed cases, `draw()` gives further ones of the same ranges. A case is a dict of plain
values; `prepare` makes what a program has in hand before the call (device tensors and a plan), `run` is
one pass through the public entry points, `work` says what the pass cannot do without, and `exact`
computes its result in 64 bits with plain torch.

Four kinds of work:

* "transpose": one B = alpha * perm(A) + beta * B, through a kept `Plan` or through `transpose()`;
* "batch": many small transpositions in one launch (`Batch`), replayed as a CUDA graph;
* "contract": a tensor contraction staged through transpositions (`ttgt.contract`);
* "train": one training step (forward, loss, backward, Adam) of the schedule selector's network.

Shapes are in the library's column-major convention (dimension 0 has stride 1); lists are written as
comma-separated text.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from ttc_b200 import Plan, transpose
from ttc_b200.batched import Batch
from ttc_b200.cost_model import MLP
from ttc_b200.ttgt import contract, plan_contraction
from ttc_b200.workloads import batched_cases

DTYPE = {"s": torch.float32, "d": torch.float64, "c": torch.complex64, "z": torch.complex128}
BYTES = {"s": 4, "d": 8, "c": 8, "z": 16}
MAX_BYTES = 850_000_000  # the largest listed case's traffic; drawn cases stay below it


# ------------------------------------------------------------------------------------------------
def _t(name, perm, size, dtype, alpha=1.0, beta=0.0, alpha_im=0.0, lda="", ldb="", call="plan"):
    return {"name": name, "kind": "transpose", "perm": perm, "size": size, "dtype": dtype, "alpha": alpha,
            "alpha_im": alpha_im, "beta": beta, "lda": lda, "ldb": ldb, "call": call}


def listed():
    return [
        # the smallest calls of TTC's own test list: launch and host latency, ragged on every side
        _t("small_call", "2,1,0", "33,17,9", "s", 1.1, 0.0, call="function"),
        # an ordinary odd-sized matrix of a few MB: fits L2, a few tiles per SM
        _t("matrix_odd_8MB", "1,0", "1023,1025", "d", 1.0, 0.0),
        # complex rank 4 of 16 MB, updating B in place, short shared stride-1 dimension
        _t("complex_rank4_16MB", "0,3,1,2", "12,43,51,79", "c", 1.1, 1.2),
        # TTC's README example (147 MB moved)
        _t("readme", "1,0,2", "1000,768,16", "s", 1.0, 1.0),
        # four of the 200 MiB benchmark sweep: a thin matrix with an odd stride-1 extent, runs that are
        # short on both sides, rank 6 in fp64 with an update of B, and a shared stride-1 dimension
        _t("sweep_thin_matrix", "1,0", "27,1941807", "s", 1.5, -0.5),
        _t("sweep_short_runs", "2,1,0", "10,25,209715", "s", 1.0, 0.0),
        _t("sweep_rank6", "5,4,0,2,1,3", "7,11,16,38,5,112", "d", 1.5, -0.5),
        _t("sweep_rows", "0,1,3,2", "254,16,215,30", "d", 1.0, 0.0),
        # precision cast of a padded sub-tensor, complex alpha: the largest case
        _t("strided_cast_zc", "3,1,0,2", "96,80,72,64", "zc", 0.5, 0.0, alpha_im=0.25, lda="104,80,76,64"),
        # a thousand uneven small transpositions (log-normal sizes around 64 Ki elements) in one launch
        {"name": "batch_1024", "kind": "batch", "count": 1024, "median": 65536, "lo": 1024, "hi": 1 << 20, "dtype": "s",
         "alpha": 1.0, "beta": 0.0, "shapes": 7},
        # a four-index contraction over two modes, as coupled-cluster codes run them
        {"name": "contraction", "kind": "contract", "a": "aebf", "b": "dfce", "c": "abcd",
         "extents": "a=26,b=22,c=25,d=24,e=21,f=27", "dtype": "s", "alpha": 1.0, "beta": 0.0},
        # a training step of the schedule selector at its training batch size
        {"name": "selector_training", "kind": "train", "rows": 2048, "features": 96, "hidden": 128, "lr": 2e-3},
    ]


# ------------------------------------------------------------------------------------------------
def _csv(values):
    return ",".join(str(int(v)) for v in values)


def _ints(text):
    return [int(x) for x in text.split(",")] if text else None


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _draw_size(rng, rank, n):
    """`rank` extents with a product near n, spread unevenly; half the time one of them in [7, 31]."""
    w = [rng.uniform(0.15, 1.0) for _ in range(rank)]
    size = [0] * rank
    free = list(range(rank))
    if rank > 1 and n >= 4096 and rng.random() < 0.5:
        d = rng.randrange(rank)
        size[d] = rng.randint(7, 31)
        free.remove(d)
        n = n / size[d]
    total = sum(w[i] for i in free)
    for i in free:
        size[i] = max(2, round(n ** (w[i] / total)))
    big = max(free, key=lambda i: size[i])
    rest = math.prod(size[i] for i in free if i != big)
    size[big] = max(2, round(n / rest))
    return size


def draw(rng):
    kind = rng.choices(["transpose", "batch", "contract", "train"], [0.76, 0.1, 0.07, 0.07])[0]
    if kind == "batch":
        dtype, beta, median = rng.choice("ssd"), rng.choice([0.0, 0.0, -0.5]), round(_log_uniform(rng, 4096, 65536))
        per = BYTES[dtype] * (3 if beta else 2)  # the sizes' mean is about 1.6 medians
        most = min(1024, int(0.8 * MAX_BYTES / (1.6 * median * per)))
        return {"kind": "batch", "count": round(_log_uniform(rng, 64, most)), "median": median, "lo": 1024, "hi": 1 << 20,
                "dtype": dtype, "alpha": 1.0, "beta": beta, "shapes": rng.randrange(1 << 20)}
    if kind == "contract":
        modes = list("abcd")
        rng.shuffle(modes)
        a, b = list("ab") + ["e", "f"], list("cd") + ["e", "f"]
        rng.shuffle(a)
        rng.shuffle(b)
        ext = {m: round(_log_uniform(rng, 8, 32)) for m in "abcdef"}
        return {"kind": "contract", "a": "".join(a), "b": "".join(b), "c": "".join(modes),
                "extents": ",".join(f"{m}={v}" for m, v in ext.items()), "dtype": rng.choice("sd"), "alpha": 1.0,
                "beta": rng.choice([0.0, -0.5])}
    if kind == "train":
        return {"kind": "train", "rows": round(_log_uniform(rng, 256, 4096)), "features": rng.randint(8, 128), "hidden": 128,
                "lr": 2e-3}
    dtype = rng.choices(["s", "d", "c", "z", "sd", "ds", "cz", "zc"], [8, 8, 2, 2, 1, 1, 1, 1])[0]
    beta = rng.choice([0.0, 0.0, -0.5, 1.2])
    per = BYTES[dtype[0]] + BYTES[dtype[-1]] * (2 if beta else 1)
    size = _draw_size(rng, rng.randint(2, 6), _log_uniform(rng, 1024, 0.95 * MAX_BYTES / per / 1.3))
    perm = list(range(len(size)))
    while perm == list(range(len(size))):
        rng.shuffle(perm)
    lda = ldb = None
    if rng.random() < 0.15:  # sub-tensors of padded arrays
        lda = [s + rng.choice([0, 0, 1, 4, 8]) for s in size[:-1]] + [size[-1]]
        ldb = [size[p] + rng.choice([0, 0, 1, 4]) for p in perm[:-1]] + [size[perm[-1]]]
        if math.prod(lda) > 1.5 * math.prod(size) or math.prod(ldb) > 1.5 * math.prod(size):
            lda = ldb = None
    c = _t("", _csv(perm), _csv(size), dtype, rng.choice([1.0, 1.0, 1.5]), beta, lda=_csv(lda or []), ldb=_csv(ldb or []),
           call=rng.choice(["plan", "function"]))
    del c["name"]
    return c


# ------------------------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _uniform(n, letter, g):
    """n values uniform in [-1, 1] (complex: real and imaginary parts)."""
    real = torch.float32 if letter in "sc" else torch.float64
    m = 2 * n if letter in "cz" else n
    x = torch.rand(m, dtype=real, device="cuda", generator=g).mul_(2).sub_(1)
    return torch.view_as_complex(x.view(n, 2)) if letter in "cz" else x


def _transpose_inputs(case, seed):
    perm, size = _ints(case["perm"]), _ints(case["size"])
    lda, ldb = _ints(case["lda"]), _ints(case["ldb"])
    na = math.prod((lda or size)[:-1]) * size[-1]
    nb = math.prod((ldb or [size[p] for p in perm])[:-1]) * size[perm[-1]]
    g = _gen(seed)
    return perm, size, lda, ldb, _uniform(na, case["dtype"][0], g), _uniform(nb, case["dtype"][-1], g)


def _alpha(case):
    return complex(case["alpha"], case["alpha_im"]) if case.get("alpha_im") else case["alpha"]


def _batch_inputs(case, seed):
    """The problems' shapes, and their A and B buffers as pieces of two arrays (256-byte aligned)."""
    shapes = batched_cases(seed=case["shapes"], count=case["count"], median=case["median"], lo=case["lo"], hi=case["hi"])
    align = 256 // BYTES[case["dtype"]]
    ns = [math.prod(c["size"]) for c in shapes]
    at, off = 0, []
    for n in ns:
        off.append(at)
        at += -(-n // align) * align
    g = _gen(seed)
    return shapes, ns, off, _uniform(at, case["dtype"], g), _uniform(at, case["dtype"], g)


def _extents(case):
    return {p[0]: int(p[2:]) for p in case["extents"].split(",")}


def _contract_inputs(case, seed):
    ext = _extents(case)
    g = _gen(seed)
    A, B, C = (_uniform(math.prod(ext[m] for m in case[k]), case["dtype"], g) for k in "abc")
    return ext, A, B, C


def _train_inputs(case, seed):
    """Normalised features, targets, and a network some way into its training (weights, moments)."""
    n, k, h = case["rows"], case["features"], case["hidden"]
    g = _gen(seed)

    def normal(*shape, scale=1.0):
        return torch.randn(*shape, device="cuda", generator=g) * scale

    X, y = normal(n, k), normal(n, 1)
    params = [normal(k, h, scale=math.sqrt(2.0 / k)), normal(h, scale=0.05), normal(h, h, scale=math.sqrt(2.0 / h)),
              normal(h, scale=0.05), normal(h, 1, scale=0.3 * math.sqrt(2.0 / h)), normal(1, scale=0.05)]
    m = [normal(*p.shape, scale=0.01) for p in params]
    v = [normal(*p.shape, scale=0.02).square_().add_(1e-4) for p in params]
    return X, y, params, m, v


TRAIN_STEPS_BEFORE = 100


def prepare(case, seed):
    kind = case["kind"]
    if kind == "transpose":
        perm, size, lda, ldb, A, B = _transpose_inputs(case, seed)
        plan = Plan(perm, size, case["dtype"], case["beta"] != 0, lda, ldb) if case["call"] == "plan" else None
        return {"kind": kind, "plan": plan, "A": A, "B": B, "perm": perm, "size": size, "lda": lda, "ldb": ldb,
                "alpha": _alpha(case), "beta": case["beta"]}
    if kind == "batch":
        shapes, ns, off, A, B = _batch_inputs(case, seed)
        plans = [Plan(c["perm"], c["size"], case["dtype"], case["beta"] != 0) for c in shapes]
        batch = Batch(plans, [A[o:o + n] for o, n in zip(off, ns)], [B[o:o + n] for o, n in zip(off, ns)],
                      alpha=case["alpha"], beta=case["beta"])
        return {"kind": kind, "batch": batch, "A": A, "B": B}
    if kind == "contract":
        ext, A, B, C = _contract_inputs(case, seed)
        return {"kind": kind, "case": case, "ext": ext, "A": A, "B": B, "C": C}
    X, y, params, m, v = _train_inputs(case, seed)
    net = MLP(case["features"], case["hidden"])
    net.params, net.m, net.v, net.t = params, m, v, TRAIN_STEPS_BEFORE
    return {"kind": kind, "net": net, "X": X, "y": y, "lr": case["lr"]}


def run(state):
    kind = state["kind"]
    if kind == "transpose":
        if state["plan"] is not None:
            state["plan"](state["A"], state["B"], state["alpha"], state["beta"])
        else:
            transpose(state["A"], state["B"], state["perm"], state["size"], state["alpha"], state["beta"], state["lda"],
                      state["ldb"])
        return state["B"]
    if kind == "batch":
        state["batch"].launch(graph=True)
        return state["B"]
    if kind == "contract":
        c = state["case"]
        return contract(state["A"], c["a"], state["B"], c["b"], state["C"], c["c"], state["ext"], c["alpha"], c["beta"])
    net = state["net"]
    out, cache = net.forward(state["X"])
    loss, d = net.loss_grad(out, state["y"])
    grads = net.backward(d, cache)
    net.step(grads, state["lr"])
    return {"loss": loss, "grads": grads, "params": net.params, "m": net.m, "v": net.v}


# ------------------------------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind == "transpose":
        per = BYTES[case["dtype"][0]] + BYTES[case["dtype"][-1]] * (2 if case["beta"] else 1)
        return {"bytes": math.prod(_ints(case["size"])) * per, "flops": 0}
    if kind == "batch":
        shapes = batched_cases(seed=case["shapes"], count=case["count"], median=case["median"], lo=case["lo"],
                               hi=case["hi"])
        n = sum(math.prod(c["size"]) for c in shapes)
        return {"bytes": n * BYTES[case["dtype"]] * (3 if case["beta"] else 2), "flops": 0}
    if kind == "contract":
        ext = _extents(case)
        n = sum(math.prod(ext[m] for m in case[k]) for k in "abc")
        nc = math.prod(ext[m] for m in case["c"])
        every = math.prod(ext[m] for m in set(case["a"] + case["b"]))
        return {"bytes": (n + (nc if case["beta"] else 0)) * BYTES[case["dtype"]], "flops": 2 * every}
    n, k, h = case["rows"], case["features"], case["hidden"]
    params = k * h + h + h * h + h + h + 1
    # features and targets read; parameters and moments read and written, gradients written
    return {"bytes": 4 * (n * (k + 1) + 7 * params), "flops": 2 * n * (3 * h * h + 2 * k * h + 3 * h)}


# ------------------------------------------------------------------------------------------------
def _wide(x):
    return x.to(torch.complex128 if x.is_complex() else torch.float64)


def _permuted(A, perm, size, lda=None):
    """The column-major tensor A (a flat buffer) with its dimensions reordered, as a dense flat tensor."""
    r = len(size)
    ld = lda or size
    strides = [math.prod(ld[:i]) for i in range(r)]
    x = torch.as_strided(A, [size[p] for p in reversed(perm)], [strides[p] for p in reversed(perm)])
    return x.contiguous().reshape(-1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "transpose":
        perm, size, lda, ldb, A, B = _transpose_inputs(case, seed)
        out = _wide(B)
        del B
        pb = [size[p] for p in perm]
        ld = ldb or pb
        strides = [math.prod(ld[:j]) for j in range(len(pb))]
        view = torch.as_strided(out, pb[::-1], strides[::-1])
        x = _wide(_permuted(A, perm, size, lda)).mul_(_alpha(case)).view(pb[::-1])
        if case["beta"]:
            x += view * case["beta"]
        view.copy_(x)
        return out
    if kind == "batch":
        shapes, ns, off, A, B = _batch_inputs(case, seed)
        out = _wide(B)
        for c, n, o in zip(shapes, ns, off):
            x = _wide(_permuted(A[o:o + n], c["perm"], c["size"])) * case["alpha"]
            out[o:o + n] = x + out[o:o + n] * case["beta"] if case["beta"] else x
        return out
    if kind == "contract":
        ext, A, B, C = _contract_inputs(case, seed)
        p = plan_contraction(case["a"], case["b"], case["c"])
        n = lambda s: math.prod(ext[m] for m in s)  # noqa: E731
        M, K, N = n(p["free_a"]), n(p["contracted"]), n(p["free_b"])
        am = _wide(_permuted(A, p["perm_a"], [ext[m] for m in case["a"]])).view(K, M)
        bm = _wide(_permuted(B, p["perm_b"], [ext[m] for m in case["b"]])).view(N, K)
        cm = torch.matmul(bm, am).reshape(-1)
        out = _permuted(cm, p["perm_c"], [ext[m] for m in p["c_mat"]]) * case["alpha"]
        return out + _wide(C) * case["beta"] if case["beta"] else out
    X, y, params, m, v = _train_inputs(case, seed)
    X, y = X.double(), y.double()
    W1, b1, W2, b2, W3, b3 = (p.double() for p in params)
    h1 = (X @ W1 + b1).clamp_min(0)
    h2 = (h1 @ W2 + b2).clamp_min(0)
    out = h2 @ W3 + b3
    d = 2 * (out - y) / out.numel()
    d2 = (d @ W3.T) * (h2 > 0)
    d1 = (d2 @ W2.T) * (h1 > 0)
    grads = [X.T @ d1, d1.sum(0), h1.T @ d2, d2.sum(0), h2.T @ d, d.sum(0)]
    t = TRAIN_STEPS_BEFORE + 1
    ms = [0.9 * a.double() + 0.1 * g for a, g in zip(m, grads)]
    vs = [0.999 * a.double() + 0.001 * g * g for a, g in zip(v, grads)]
    ps = [p.double() - case["lr"] * (a / (1 - 0.9 ** t)) / ((b / (1 - 0.999 ** t)).sqrt() + 1e-8)
          for p, a, b in zip(params, ms, vs)]
    return {"loss": ((out - y) ** 2).mean().reshape(1), "grads": grads, "params": ps, "m": ms, "v": vs}
