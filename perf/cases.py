"""The framework's work as a user's program has it do: sizes, inputs and calls for timing.

Four entry points are covered, all with operands on the GPU:

* ``ttm``    one call of ``ttmpy.ttm(q, A, B)``: float and double, the default (exact) arithmetic,
             the FP32-accurate tensor-core path ("auto") and the int8-slice path for double
             ("ozaki"); orders 2 to 5, any mode, any layout, m from 1 to 512;
* ``batch``  a ``BatchPlan`` of random problems (``workloads.problems``), replayed as a CUDA graph;
* ``tucker`` a ``ChainPlan`` projecting every mode of a tensor, replayed as a CUDA graph;
* ``ttms``   one call of ``ttmpy.ttms(q, A, Bs)``: every mode but one, as in an alternating
             least-squares sweep.

``listed()`` are the cases themselves, ``draw(rng)`` gives another of the same ranges.
``prepare`` makes what the program holds before the call (tensors from the seed, plans), ``run``
is one pass and ``exact`` the same result in 64 bits from plain torch.
"""
from __future__ import annotations

import math

import torch

from ttm_b200 import ttmpy, workloads
from ttm_b200.plans import BatchPlan, ChainPlan

DTYPES = {"f32": torch.float32, "f64": torch.float64}


def _ttm(name, dtype, na, q, m, pia, precision="default", b_cm=False):
    case = {"kind": "ttm", "dtype": dtype, "precision": precision, "q": q, "m": m, "b_cm": b_cm, "p": len(na)}
    case.update({f"n{r + 1}": n for r, n in enumerate(na)})
    case["layout"] = "".join(str(r) for r in pia)
    if name:
        case["name"] = name
    return case


def listed():
    return [
        # The smallest call: a tensor of the size that unit tests and inner loops of small
        # decompositions use, double as the reference's Python module; launch and host latency.
        _ttm("point_f64", "f64", [12, 10, 9], 2, 6, [3, 2, 1]),
        # Tensor times vector on a tensor of the layout/mode sweep: reads A once.
        _ttm("vector_f32", "f32", [512, 256, 512], 2, 1, [1, 2, 3]),
        # A few output rows and extents that no vector width divides.
        _ttm("few_rows_odd_f32", "f32", [401, 263, 509], 2, 7, [1, 2, 3]),
        # The last mode of a C-ordered array (contiguous fibres), low rank, double.
        _ttm("last_mode_f64", "f64", [260, 300, 384], 3, 16, [3, 2, 1]),
        # A middle mode of an order-5 tensor of the sweep in exact single precision.
        _ttm("order5_f32", "f32", [32, 32, 64, 32, 32], 3, 64, [5, 4, 3, 2, 1], b_cm=True),
        # Exact double precision, the reference's only type in Python; odd extents.
        _ttm("odd_f64", "f64", [150, 171, 333], 2, 100, [3, 2, 1]),
        # FP32-accurate tensor-core arithmetic, a factor of ordinary rank.
        _ttm("rank96_auto", "f32", [300, 420, 500], 2, 96, [1, 2, 3], "auto"),
        # The precision-study contraction (256 columns on every mode), its last mode cut to 64.
        _ttm("square256_auto", "f32", [256, 256, 256, 64], 2, 256, [1, 2, 3, 4], "auto", b_cm=True),
        # Double through int8 tensor-core slices.
        _ttm("ozaki_f64", "f64", [256, 256, 256], 2, 128, [3, 2, 1], "ozaki"),
        # Many independent products of every shape at once.
        {"name": "batch512", "kind": "batch", "count": 512, "draw_seed": 1, "precision": "auto"},
        # Core tensor of a Tucker decomposition: 32 columns on each of four modes of 192.
        {"name": "tucker192", "kind": "tucker", "dtype": "f32", "precision": "auto", "p": 4, "n": 192, "m": 32},
        # One step of an alternating sweep in double: all modes but the first projected to rank 20.
        {"name": "sweep_step_f64", "kind": "ttms", "dtype": "f64", "p": 3, "n1": 200, "n2": 180, "n3": 160, "m": 20, "q": 1,
         "order": "optimal"},
    ]


def draw(rng):
    kind = rng.choices(["ttm", "batch", "tucker", "ttms"], [14, 1, 1, 2])[0]
    log_uniform = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))  # noqa: E731
    if kind == "batch":
        precision = rng.choice(["auto", "default"])
        return {"kind": "batch", "count": log_uniform(16, 400 if precision == "auto" else 120),
                "draw_seed": rng.randrange(1, 10 ** 6), "precision": precision}
    if kind == "tucker":
        p = rng.choice([3, 4])
        n = log_uniform(24, 400 if p == 3 else 140)
        return {"kind": "tucker", "dtype": "f32", "precision": "auto", "p": p, "n": n, "m": min(n, log_uniform(8, 48))}
    if kind == "ttms":
        n = [log_uniform(20, 320) for _ in range(3)]
        return {"kind": "ttms", "dtype": rng.choice(["f32", "f64"]), "p": 3, "n1": n[0], "n2": n[1], "n3": n[2],
                "m": min(min(n), log_uniform(4, 64)), "q": rng.randrange(1, 4),
                "order": rng.choice(["forward", "backward", "optimal"])}
    dtype, precision = rng.choice([("f32", "default"), ("f64", "default"), ("f32", "auto"), ("f64", "ozaki")])
    p = rng.randrange(2, 6)
    target = rng.uniform(9, 26 if precision != "ozaki" else 24) * math.log(2)
    m = log_uniform(1, 512)
    parts = [0.3 + rng.random() for _ in range(p)]
    na = [max(2, int(round(math.exp(target * w / sum(parts))))) for w in parts]
    q = rng.randrange(1, p + 1)
    # a result is at most 2^27 elements, a product in exact arithmetic at most 2^35 operations
    n_a = math.prod(na)
    m = max(1, min(m, (1 << 27) * na[q - 1] // n_a, m if precision == "auto" else (1 << 34) // n_a))
    pia = list(range(1, p + 1))
    how = rng.randrange(3)
    if how == 0:
        pia.reverse()
    elif how == 1:
        rng.shuffle(pia)
    return _ttm(None, dtype, na, q, m, pia, precision, rng.random() < 0.5)


def _extents(case):
    return [case[f"n{r + 1}"] for r in range(case["p"])]


def _strided(gen, shape, pia, dtype):
    """N(0,1) entries in a dense tensor of the given extents whose modes lie in memory in the order pia."""
    x = torch.randn([shape[r - 1] for r in reversed(pia)], generator=gen, device="cuda", dtype=dtype)
    order = [r - 1 for r in reversed(pia)]
    return x.permute([order.index(r) for r in range(len(shape))])


def _size(pr):
    return math.prod(pr["na"]) // pr["na"][pr["q"] - 1] * pr["m"]


def _places(probs):
    """Offsets of a batch's results in one buffer, each on a 256-byte boundary, and the buffer's length."""
    at, total = [], 0
    for pr in probs:
        at.append(total)
        total += -(-_size(pr) // 64) * 64
    return at, total


def _factor(gen, n, m, dtype):
    """An n x m matrix of orthonormal columns, transposed: the projection of a mode of extent n."""
    u = torch.linalg.qr(torch.randn(n, m, generator=gen, device="cuda", dtype=torch.float64))[0]
    return u.t().contiguous().to(dtype)


def _inputs(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    kind = case["kind"]
    if kind == "ttm":
        dt = DTYPES[case["dtype"]]
        na, m, n_q = _extents(case), case["m"], _extents(case)[case["q"] - 1]
        A = _strided(gen, na, [int(c) for c in case["layout"]], dt)
        B = torch.randn(n_q, m, generator=gen, device="cuda", dtype=dt).t() if case["b_cm"] else \
            torch.randn(m, n_q, generator=gen, device="cuda", dtype=dt)
        return A, B
    if kind == "batch":
        out = []
        for pr in workloads.problems(case["count"], case["draw_seed"]):
            A = _strided(gen, pr["na"], pr["pia"], torch.float32)
            out.append(dict(pr, A=A, B=torch.randn(pr["m"], pr["na"][pr["q"] - 1], generator=gen, device="cuda")))
        return out
    dt = DTYPES[case["dtype"]]
    if kind == "tucker":
        n, p = case["n"], case["p"]
        return torch.randn([n] * p, generator=gen, device="cuda", dtype=dt), [_factor(gen, n, case["m"], dt) for _ in range(p)]
    na = _extents(case)
    A = torch.randn(na, generator=gen, device="cuda", dtype=dt)
    return A, [_factor(gen, n, case["m"], dt) for r, n in enumerate(na) if r != case["q"] - 1]


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("ttm", "ttms"):
        A, B = _inputs(case, seed)
        return {"case": case, "A": A, "B": B}
    if kind == "batch":
        probs = _inputs(case, seed)
        at, total = _places(probs)
        C = torch.zeros(total, device="cuda")
        for pr, o in zip(probs, at):
            pr["C"] = C[o:o + _size(pr)]
        return {"case": case, "plan": BatchPlan(probs, precision=case["precision"]), "C": C}
    A, Bs = _inputs(case, seed)
    p, m = case["p"], case["m"]
    C = torch.empty([m] * p, device="cuda", dtype=A.dtype)
    # a C-ordered tensor in memory is a first-order one with its modes reversed
    plan = ChainPlan(A, [case["n"]] * p, list(range(p, 0, -1)), list(range(1, p + 1)), Bs, C, precision=case["precision"])
    return {"case": case, "plan": plan, "C": C}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "ttm":
        return ttmpy.ttm(case["q"], state["A"], state["B"], precision=case["precision"])
    if kind == "ttms":
        return ttmpy.ttms(case["q"], state["A"], state["B"], order=case["order"])
    state["plan"].run_graph()
    return state["C"]


def work(case):
    kind = case["kind"]
    if kind == "batch":
        probs = workloads.problems(case["count"], case["draw_seed"])
        return {"bytes": sum(workloads.io_bytes(pr) for pr in probs), "flops": sum(workloads.flops(pr) for pr in probs)}
    es = 4 if case["dtype"] == "f32" else 8
    if kind == "ttm":
        na = _extents(case)
        n_a, n_q, m = math.prod(na), na[case["q"] - 1], case["m"]
        return {"bytes": es * (n_a + n_a // n_q * m + m * n_q), "flops": 2.0 * m * n_a}
    if kind == "tucker":
        modes, na = range(case["p"]), [case["n"]] * case["p"]
    else:
        na = _extents(case)
        modes = [r for r in range(case["p"]) if r != case["q"] - 1]
        # the cheapest order of the products is what the path cannot do without
        modes = sorted(modes, key=lambda r: 1.0 / na[r] - 1.0 / case["m"])
    ext, flops, nbytes = list(na), 0.0, math.prod(na)
    for r in modes:
        flops += 2.0 * case["m"] * math.prod(ext)
        nbytes += case["m"] * ext[r]
        ext[r] = case["m"]
    return {"bytes": es * (nbytes + math.prod(ext)), "flops": flops}


def _product(A, B, mode):
    """A x_mode B in double (mode zero-based)."""
    return torch.movedim(torch.tensordot(A.double(), B.double(), dims=([mode], [1])), -1, mode)


def exact(case, seed):
    kind = case["kind"]
    data = _inputs(case, seed)
    if kind == "ttm":
        return _product(*data, case["q"] - 1)
    if kind == "batch":
        at, total = _places(data)
        C = torch.zeros(total, device="cuda", dtype=torch.float64)
        for pr, o in zip(data, at):
            c = _product(pr["A"], pr["B"], pr["q"] - 1)
            C[o:o + c.numel()] = c.permute([r - 1 for r in reversed(pr["pia"])]).reshape(-1)
        return C
    A, Bs = data
    A = A.double()
    modes = range(case["p"]) if kind == "tucker" else [r for r in range(case["p"]) if r != case["q"] - 1]
    for r, B in zip(modes, Bs):
        A = _product(A, B, r)
    return A
