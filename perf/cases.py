"""The measured cases: what a program that uses this library has it do.

A case is a dict of plain values.  Kinds:
  run    one uhs.run of a program (T sweeps, both grids on the GPU): the
         twelve star and box shapes in FP64 (the default float-pair path) and
         FP32, and one-sided programs on the generic kernel
  batch  one replay of a uhs.Batch of many small programs

Sizes are interior extents, slowest axis first, with a halo of the program's
radius around them.  They are the library's own configurations (cfg1 to cfg4
of uxxxxxxxxh_gb300/workloads.py, the 8192^2 / T = 4 runs of the reference
harness, the mixed batch suites) and odd extents between them.
"""
import math
import random

import torch

import uxxxxxxxxh_gb300 as uhs

DTYPES = {"f64": (uhs.UHS_F64, torch.float64), "f32": (uhs.UHS_F32, torch.float32)}
ARITHS = {"auto": uhs.UHS_ARITH_AUTO, "exact": uhs.UHS_ARITH_EXACT}


def _run(name, shape, size, T, dtype="f64", coefs="random", arith="auto", data="uniform"):
    return {"name": name, "kind": "run", "shape": shape, "size": size, "T": T, "dtype": dtype, "coefs": coefs,
            "arith": arith, "data": data}


def listed():
    return [
        # the smallest calls: launches and latency are the time
        _run("2d1r_star_f64_256sq", "2d1r_star", "256x256", 100),
        _run("3d1r_star_f32_64cube", "3d1r_star", "64x64x64", 20, dtype="f32"),
        # a mid-sized grid of odd extents
        _run("3d2r_star_f64_odd", "3d2r_star", "97x131x203", 20),
        # cfg1: 2D heat-like sweep
        _run("cfg1_2d1r_star_f64_4096sq", "2d1r_star", "4096x4096", 100),
        # cfg2, the workload the headline number is quoted on, in both types
        _run("cfg2_3d1r_star_f64_512cube", "3d1r_star", "512x512x512", 50, data="signed"),
        _run("cfg2_3d1r_star_f32_512cube", "3d1r_star", "512x512x512", 50, dtype="f32", data="signed"),
        # cfg4's program in calls of 20 steps, as the precision study scores it
        _run("cfg4_3d2r_star_f64_512cube", "3d2r_star", "512x512x512", 20, data="smooth"),
        # cfg3: a 343-point Gaussian, which factors into 1D passes
        _run("cfg3_3d3r_box_f64_256cube", "3d3r_box", "256x256x256", 10, coefs="gauss"),
        # a box of general coefficients, term by term, odd extents
        _run("3d2r_box_f64_ragged", "3d2r_box", "191x255x321", 10),
        # the reference harness: 8192^2, T = 4
        _run("2d2r_star_f64_8192sq_T4", "2d2r_star", "8192x8192", 4),
        # many small programs of mixed shape and type advanced together
        {"name": "batch_24_small", "kind": "batch", "grids": 24, "T": 20, "side2": 512, "side3": 64, "program": 7},
        # a one-sided (upwind) program: outside the templated shapes
        _run("3d_upwind2_f64_256cube", "3d_upwind2", "256x256x256", 4),
    ]


SHAPES = [f"{rank}d{r}r_{kind}" for rank in (2, 3) for r in (1, 2, 3) for kind in ("star", "box")]
MOST_FLOPS = 2 * 7 * 512 ** 3 * 50  # no drawn case costs more than the largest listed one
MOST_BYTES = 16 * 512 ** 3 * 50


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    while True:
        kind = rng.random()
        if kind < 0.1:
            return {"kind": "batch", "grids": rng.randint(8, 32), "T": rng.choice([4, 10, 20]),
                    "side2": _log_int(rng, 256, 1024), "side3": _log_int(rng, 32, 128),
                    "program": rng.randrange(1 << 20)}
        if kind < 0.2:
            shape = rng.choice(["2d_upwind1", "2d_upwind2", "3d_upwind1", "3d_upwind2"])
            arith = rng.choice(["auto", "auto", "exact"])
            coefs = "random"
        else:
            shape, arith = rng.choice(SHAPES), "auto"
            coefs = "gauss" if "box" in shape and rng.random() < 0.5 else "random"
        lo, hi = (256, 8192) if shape[0] == "2" else (48, 512)
        size = "x".join(str(_log_int(rng, lo, hi)) for _ in range(int(shape[0])))
        c = {"kind": "run", "shape": shape, "size": size, "T": rng.choice([4, 10, 20, 50, 100]),
             "dtype": rng.choice(["f64", "f64", "f32"]), "coefs": coefs, "arith": arith,
             "data": rng.choice(["uniform", "signed", "smooth"])}
        w = work(c)
        if w["flops"] <= MOST_FLOPS and w["bytes"] <= MOST_BYTES:
            return c


# ---- programs ----------------------------------------------------------
def _offsets(shape):
    rank = int(shape[0])
    if "upwind" in shape:
        # one-sided differences of the given width along each axis, and the centre
        n = int(shape[-1])
        offs = [(0, 0, 0)]
        for ax in range(3 - rank, 3):
            for d in range(1, n + 1):
                o = [0, 0, 0]
                o[ax] = -d
                offs.append(tuple(o))
        return rank, n, offs
    r = int(shape[2])
    return rank, r, uhs.offsets_for(rank, r, shape.split("_")[1])


def _coefs(offs, how, rng):
    """Weights that sum to 1 (averages, so fields stay bounded however often a run is repeated)."""
    if how == "gauss":
        w = [math.exp(-(z * z + y * y + x * x) / (2 * 1.5 ** 2)) for z, y, x in offs]
    else:
        w = [0.05 + rng.random() for _ in offs]
    s = sum(w)
    return [v / s for v in w]


def _program(shape, size, T, dtype, coefs, rng):
    rank, r, offs = _offsets(shape)
    return uhs.make_stencil(shape, rank, [int(v) for v in size.split("x")], r, offs, _coefs(offs, coefs, rng),
                            iterations=T, dtype=DTYPES[dtype][0])


def _field(st, dtype, data, gen):
    """A grid's initial values, halo included."""
    shape = st.shape
    a = torch.rand(shape, dtype=torch.float64, device="cuda", generator=gen)
    if data == "signed":  # U[-1, 1)
        a.mul_(2.0).sub_(1.0)
    elif data == "smooth":  # a smooth field with a little noise on it
        a.mul_(1e-3)
        wave = None
        for k, n in enumerate(shape):
            t = torch.arange(n, dtype=torch.float64, device="cuda") * (2 * math.pi / n)
            t = (torch.cos(t) if k == 1 else torch.sin(t)).reshape([-1 if i == k else 1 for i in range(len(shape))])
            wave = t if wave is None else wave * t
        a.add_(wave)
    return a.to(DTYPES[dtype][1])


def _grids(st, dtype, data, gen):
    a = _field(st, dtype, data, gen)
    return a, a.clone()  # both grids hold the same halo


def _batch_specs(case):
    """The batch's programs, drawn from the case's own program seed."""
    rng = random.Random(case["program"])
    out = []
    for _ in range(case["grids"]):
        shape = rng.choice(SHAPES)
        lo, hi = (64, case["side2"]) if shape[0] == "2" else (16, case["side3"])
        size = "x".join(str(_log_int(rng, lo, hi)) for _ in range(int(shape[0])))
        out.append((shape, size, rng.choice(["f64", "f32"])))
    return out


def _build(case, seed):
    """The case's programs and grids: [(stencil, dtype, a, b)]."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    rng = random.Random(seed)
    specs = (_batch_specs(case) if case["kind"] == "batch" else [(case["shape"], case["size"], case["dtype"])])
    out = []
    for shape, size, dtype in specs:
        st = _program(shape, size, case["T"], dtype, case.get("coefs", "random"), rng)
        out.append((st, dtype, *_grids(st, dtype, case.get("data", "uniform"), gen)))
    return out


# ---- what is measured --------------------------------------------------
def prepare(case, seed):
    parts = _build(case, seed)
    if case["kind"] == "batch":
        a, b = [p[2] for p in parts], [p[3] for p in parts]
        torch.cuda.synchronize()  # the batch's set-up reads the grids on a stream of its own
        return {"batch": uhs.Batch([p[0] for p in parts], a, b), "a": a, "b": b}
    st, _, a, b = parts[0]
    return {"st": st, "a": a, "b": b, "params": uhs.RunParams(arith=ARITHS[case["arith"]])}


def run(state):
    """T sweeps; the result is in a, step T - 1 in b."""
    if "batch" in state:
        state["batch"].run()
    else:
        uhs.run(state["st"], state["a"], state["b"], state["params"])
    return {"a": state["a"], "b": state["b"]}


def _terms(shape, coefs):
    rank, r, offs = _offsets(shape)
    return rank * (2 * r + 1) if coefs == "gauss" and "box" in shape else len(offs)


def work(case):
    """Each sweep reads and writes every cell once and takes a multiply and an add per term (a Gaussian box: per
    term of its 1D passes)."""
    specs = (_batch_specs(case) if case["kind"] == "batch" else [(case["shape"], case["size"], case["dtype"])])
    nbytes = flops = 0
    for shape, size, dtype in specs:
        n = math.prod(int(v) for v in size.split("x")) * case["T"]
        nbytes += n * (16 if dtype == "f64" else 8)
        flops += 2 * n * _terms(shape, case.get("coefs", "random"))
    return {"bytes": nbytes, "flops": flops}


def _sweeps(st, a, b):
    """T sweeps in FP64: (a, b) as the library leaves them."""
    a, b = a.double().reshape(st.sizes), b.double().reshape(st.sizes)
    dom = tuple(slice(lo, hi) for lo, hi in zip(st.lb, st.ub))
    for _ in range(st.iterations // 2):
        for src, dst in ((a, b), (b, a)):
            acc = torch.zeros_like(src[dom])
            for dz, dy, dx, c in st.terms:
                acc.add_(src[tuple(slice(lo + d, hi + d) for lo, hi, d in zip(st.lb, st.ub, (dz, dy, dx)))], alpha=c)
            dst[dom] = acc
    return a.reshape(st.shape), b.reshape(st.shape)


def exact(case, seed):
    done = [_sweeps(st, a, b) for st, _, a, b in _build(case, seed)]
    if case["kind"] == "batch":
        return {"a": [d[0] for d in done], "b": [d[1] for d in done]}
    return {"a": done[0][0], "b": done[0][1]}
