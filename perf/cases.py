"""The calls whose speed this framework is measured by, and their 64-bit values.

A case is one use of a public entry point at one size:

* ``scft``: a solver advanced by ``iterations`` SCFT iterations (``ScftSolver.update``) from
  where it stands, with the free energy, the partition functions and every field read back, as a
  program does that watches its run or hands the fields on.
* ``batch``: the same for several independent blends of different grids in one ``ScftBatch``.
* ``adjoint``: densities and ln Q of a chain through ``DifferentiableChain`` and the gradients of
  a loss of both (forward and backward).
* ``fft``: ``B200FFT.scaledFFTPair`` on host arrays, the reference's transform plugin.

Fields are seeded random noise on a periodic pattern, as the runs of ``workloads.py`` start.
Mixed-precision runs (FP32 sweeps) hand their results on as float32, FP64 runs as float64.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from polyswift_plusplus_b200 import B200FFT, ScftBatch, ScftSolver
from polyswift_plusplus_b200 import _abi as A
from polyswift_plusplus_b200.adjoint import DifferentiableChain
from polyswift_plusplus_b200.config import Block, Interaction, Polymer, ScftConfig, Updater

CELL = 0.0625  # grid spacing in Rg of the 128^3 and 256^3 workloads


def _scft(name, model, grid, precision, ns, updater="steepestDescent", iterations=1, depth=0, f=0.35, chin=25.0,
          homo=0.0, cell=CELL):
    return {"name": name, "kind": "scft", "model": model, "nx": grid[0], "ny": grid[1], "nz": grid[2],
            "precision": precision, "ns": ns, "updater": updater, "iterations": iterations, "depth": depth, "f": f,
            "chin": chin, "homo": homo, "cell": cell}


def listed():
    return [
        # The smallest melts: a unit cell of a branched polymer, many of which a phase-diagram scan runs.
        _scft("star16_fp64", "star", (16, 16, 16), "fp64", 100, iterations=4, f=0.3, chin=15.0, cell=0.2),
        # The plain FP64 method on the reference's usual unit cell.
        _scft("diblock32_fp64", "diblock", (32, 32, 32), "fp64", 100, iterations=4, f=0.3, chin=20.0, cell=0.125),
        # A two-dimensional run (one cell in z): cylinders and lamellae in the plane.
        _scft("film128_fp64", "diblock", (128, 128, 1), "fp64", 100, iterations=4, f=0.4, chin=18.0),
        # A box whose sides differ (a unit cell that is not cubic), with odd step counts per block.
        _scft("slab_mixed", "blend", (64, 96, 48), "mixed", 100, iterations=2, f=0.37, chin=20.0, homo=0.1),
        # An ordinary FP64 melt.
        _scft("diblock64_fp64", "diblock", (64, 64, 64), "fp64", 128, iterations=1, f=0.5, chin=18.0),
        # A blend of the batched workload's largest size on its own, Anderson mixing.
        _scft("blend96_mixed", "blend", (96, 96, 96), "mixed", 100, "andersonMixing", depth=10, f=0.3, chin=22.0,
              homo=0.15, cell=0.125),
        # The benchmark's melt: mixed precision, Anderson mixing of depth 10, 200 contour steps.
        _scft("diblock128_mixed", "diblock", (128, 128, 128), "mixed", 200, "andersonMixing", depth=10),
        # The same melt on the FP64 path (reference accuracy, and the end of an escalated run).
        _scft("diblock128_fp64", "diblock", (128, 128, 128), "fp64", 200),
        # The largest grid: an ABC triblock.
        _scft("triblock256_mixed", "triblock", (256, 256, 256), "mixed", 100, f=0.3, chin=30.0),
        # Blends of uneven size advanced together, as the batched workload draws them.
        {"name": "batch_blends", "kind": "batch", "sizes": "32,96,48,64,32,48,96,64,32,48,64,48", "precision": "mixed",
         "ns": 100, "depth": 10, "iterations": 1, "f": 0.31, "chin": 19.0, "homo": 0.1},
        # Gradients through a whole forward and conjugate sweep (cell optimisation, inverse design).
        {"name": "adjoint64", "kind": "adjoint", "n": 64, "ns": 128, "f": 0.4, "chin": 18.0},
        # The transform plugin called by a host program.
        {"name": "fft_pair128", "kind": "fft", "nx": 128, "ny": 128, "nz": 128},
    ]


def draw(rng):
    """One more call from the ranges above: grids 12 to 128 a side, cubic, flat or uneven."""
    pick = rng.random()
    ns = rng.randrange(40, 161)
    f = rng.randrange(20, 81) / 100.0
    fs = max(5, min(ns - 5, round(f * ns))) / ns  # whole numbers of steps per block
    chin = round(rng.uniform(12.0, 30.0), 3)
    if pick < 0.1:
        return {"kind": "fft", "nx": rng.choice((16, 24, 32, 64, 96, 128)), "ny": rng.choice((16, 32, 48, 64, 96)),
                "nz": rng.choice((16, 32, 48, 64, 96, 128))}
    if pick < 0.25:
        return {"kind": "adjoint", "n": rng.choice((16, 24, 32, 48, 64)), "ns": ns, "f": fs, "chin": chin}
    if pick < 0.35:
        sizes = [rng.choice((24, 32, 48, 64)) for _ in range(rng.randrange(3, 9))]
        return {"kind": "batch", "sizes": ",".join(map(str, sizes)), "precision": rng.choice(("fp64", "mixed")),
                "ns": ns, "depth": rng.randrange(2, 12), "iterations": 1, "f": fs, "chin": chin,
                "homo": rng.randrange(0, 21) / 100.0}
    shape = rng.random()
    if shape < 0.6:
        n = rng.choice((12, 16, 24, 32, 48, 64, 96, 128))
        grid = (n, n, n)
    elif shape < 0.75:
        n = rng.choice((16, 32, 64, 128))
        grid = (n, n, 1)
    else:
        grid = tuple(rng.choice((16, 24, 32, 48, 64, 96)) for _ in range(3))
    model = rng.choice(("diblock", "blend", "triblock", "star"))
    updater = rng.choice(("steepestDescent", "andersonMixing"))
    small = grid[0] * grid[1] * grid[2] <= 32 ** 3
    c = _scft("", model, grid, rng.choice(("fp64", "mixed")), ns, updater, iterations=rng.randrange(2, 6) if small else 1,
              depth=rng.randrange(2, 13) if updater == "andersonMixing" else 0,
              f=0.3 if model in ("star", "triblock") else fs, chin=chin,
              homo=rng.randrange(1, 21) / 100.0 if model == "blend" else 0.0)
    if model in ("star", "triblock"):
        c["ns"] = 10 * (ns // 10)  # 0.3, 0.3 and 0.4 of it are whole
    elif model == "blend":
        c["ns"], c["f"] = 2 * (ns // 2), max(6, round(f * (ns // 2)) * 2) / (2 * (ns // 2))
    del c["name"]
    return c


# ---------------------------------------------------------------------------
# The models.
# ---------------------------------------------------------------------------
def _chain(name, fields, fracs, ds, length=100, volfrac=1.0, star=False):
    names = ["%s_%s%d" % (name, x, i) for i, x in enumerate(fields)]
    blocks = []
    for i, x in enumerate(fields):
        if star:
            head, tail = ["freeEnd"], [b for b in names if b != names[i]]
        else:
            head = [names[i - 1]] if i else ["freeEnd"]
            tail = [names[i + 1]] if i + 1 < len(fields) else ["freeEnd"]
        blocks.append(Block(names[i], x, ds, fracs[i], head, tail, force_block_steps=True))
    return Polymer(name=name, volfrac=volfrac, length=length, blocks=blocks)


def _model(model, ns, f, homo):
    """(fields, polymers, pairs and their share of chiN) of a named model."""
    ds = 1.0 / ns
    if model == "diblock" or (model == "blend" and homo <= 0.0):
        return ["A", "B"], [_chain("ab", "AB", (f, 1.0 - f), ds)], [("A", "B", 1.0)]
    if model == "blend":
        return ["A", "B"], [_chain("ab", "AB", (f, 1.0 - f), ds, volfrac=1.0 - homo),
                            _chain("a", "A", (1.0,), ds, length=50, volfrac=homo)], [("A", "B", 1.0)]
    pairs = [("A", "B", 1.0), ("B", "C", 1.0), ("A", "C", 1.5 if model == "triblock" else 1.0)]
    fracs = (f, 0.7 - f, 0.3) if model == "triblock" else (f, f, 1.0 - 2.0 * f)
    return ["A", "B", "C"], [_chain("abc", "ABC", fracs, ds, star=(model == "star"))], pairs


def _config(model, grid, precision, ns, updater, depth, f, chin, homo, cell):
    fields, polymers, pairs = _model(model, ns, f, homo)
    lambdas = (0.1, 0.05) if len(fields) == 2 else (0.05, 0.025)
    upd = Updater(kind="steepestDescent", relaxlambdas=lambdas)
    if updater == "andersonMixing":
        upd = Updater(kind="andersonMixing", relaxlambdas=lambdas, anderson_depth=depth, anderson_mix=0.5,
                      anderson_start=10)
    return ScftConfig(n=grid, cell=(cell, cell, cell), fields=fields, polymers=polymers,
                      interactions=[Interaction(a + b, s * chin / 100, [a, b]) for a, b, s in pairs], updater=upd,
                      seed=38383, precision=precision)


def _case_config(c):
    return _config(c["model"], (c["nx"], c["ny"], c["nz"]), c["precision"], c["ns"], c["updater"], c["depth"], c["f"],
                   c["chin"], c["homo"], c["cell"])


def _batch_configs(c):
    """One blend per size: composition, chiN and homopolymer fraction step through the instances."""
    out = []
    for i, n in enumerate(int(s) for s in c["sizes"].split(",")):
        ns = 2 * (c["ns"] // 2)
        k = max(6, min(ns - 6, 2 * (round(c["f"] * ns / 2) + i % 4)))
        out.append(_config("blend", (n, n, n), c["precision"], ns, "andersonMixing", c["depth"], k / ns,
                           c["chin"] + 0.7 * i, round(c["homo"] * (1.0 + 0.05 * i), 6), 4.0 / 32))
    return out


def _pattern(grid, nf):
    """Opposite waves for the fields: along x for two of them, a third along y."""
    ax = [torch.arange(n, dtype=torch.float64, device="cuda") * (2 * math.pi / n) for n in grid]
    x, y, _ = torch.meshgrid(*ax, indexing="ij")
    waves = [torch.cos(2 * x if grid[0] > 48 else x), -torch.cos(2 * x if grid[0] > 48 else x), torch.cos(y)]
    return torch.stack([w.reshape(-1) for w in waves[:nf]])


def _fields(grid, nf, seed, amp=0.1):
    g = torch.Generator(device="cuda").manual_seed(int(seed) % (1 << 62))
    u = torch.rand((nf, grid[0] * grid[1] * grid[2]), generator=g, dtype=torch.float64, device="cuda")
    return _pattern(grid, nf) + 2 * amp * (u - 0.5)


# ---------------------------------------------------------------------------
# prepare and run.
# ---------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind == "scft":
        cfg = _case_config(case)
        s = ScftSolver(cfg)
        _set(s, _fields(cfg.n, len(cfg.fields), seed))
        return {"kind": kind, "solver": s, "iterations": case["iterations"], "out": _buffers(cfg)}
    if kind == "batch":
        cfgs = _batch_configs(case)
        b = ScftBatch(cfgs)
        for k, cfg in enumerate(cfgs):
            _set(b.instance(k), _fields(cfg.n, len(cfg.fields), seed * 101 + k))
        return {"kind": kind, "batch": b, "iterations": case["iterations"], "out": [_buffers(c) for c in cfgs]}
    if kind == "adjoint":
        cfg = _config("diblock", (case["n"],) * 3, "fp64", case["ns"], "steepestDescent", 0, case["f"], case["chin"],
                      0.0, 6.0 / 64)
        w = _fields(cfg.n, 2, seed)
        return {"kind": kind, "chain": DifferentiableChain(cfg), "w": w, "target": _target(cfg.n)}
    grid = (case["nx"], case["ny"], case["nz"])
    data, kdata = _fft_inputs(grid, seed)
    return {"kind": kind, "fft": B200FFT(grid), "data": data, "kdata": kdata}


def _set(solver, w):
    torch.cuda.synchronize()  # the solver copies on a stream of its own
    for i in range(len(w)):
        solver.set_field(A.PS_FIELD_W, i, w[i])


def _buffers(cfg):
    nf, N = len(cfg.fields), cfg.n_total
    return {"w": torch.empty((nf, N), dtype=torch.float64, device="cuda"),
            "phi": torch.empty((nf, N), dtype=torch.float64, device="cuda"),
            "p": torch.empty(N, dtype=torch.float64, device="cuda")}


def _target(grid):
    z = torch.arange(grid[2], dtype=torch.float64, device="cuda") * (2 * math.pi / grid[2])
    return (0.5 + 0.4 * torch.cos(z)).repeat(grid[0] * grid[1])


def _fft_inputs(grid, seed):
    """A propagator slice and the operator exp(-ds k^2) / N it is multiplied by, on the host."""
    g = torch.Generator().manual_seed(int(seed) % (1 << 62))
    data = torch.rand(grid, generator=g, dtype=torch.float64) + 0.5
    return data.reshape(-1).numpy(), np.ascontiguousarray(_kernel(grid, CELL, 0.01, "cpu").numpy().reshape(-1))


def _read(solver, cfg, out):
    for i in range(len(cfg.fields)):
        solver.get_field(A.PS_FIELD_W, i, out=out["w"][i])
        solver.get_field(A.PS_FIELD_PHI, i, out=out["phi"][i])
    solver.get_field(A.PS_FIELD_PRES, 0, out=out["p"])
    s = solver.scalars()
    kind = torch.float32 if cfg.precision == "mixed" else torch.float64
    sc = torch.tensor([s["free_energy"], s["free_energy_nodis"], s["dh_norm"]] + list(s["q"]), dtype=kind)
    return {"w": out["w"].to(kind), "phi": out["phi"].to(kind), "p": out["p"].to(kind), "scalars": sc}


def run(state):
    kind = state["kind"]
    if kind == "scft":
        state["solver"].update(state["iterations"])
        return _read(state["solver"], state["solver"].cfg, state["out"])
    if kind == "batch":
        b = state["batch"]
        b.update(state["iterations"])
        return [_read(b.instance(i), c, state["out"][i]) for i, c in enumerate(b.cfgs)]
    if kind == "adjoint":
        w = state["w"].clone().requires_grad_(True)
        chain = state["chain"]
        box = torch.tensor(chain.box0, dtype=torch.float64, requires_grad=True)
        ds = torch.tensor(chain.ds0, dtype=torch.float64, requires_grad=True)
        phi, lnq = chain(w, box, ds)
        loss = ((phi[0] - state["target"]) ** 2).sum() + 10.0 * lnq
        loss.backward()
        return {"phi": phi.detach(), "lnq": lnq.detach(), "dw": w.grad, "dbox": box.grad, "dds": ds.grad}
    return state["fft"].scaledFFTPair(state["data"], state["kdata"])


# ---------------------------------------------------------------------------
# What a pass cannot do without.
# ---------------------------------------------------------------------------
def _steps(cfg):
    """Propagator steps of one iteration (a homopolymer's two sweeps are one) and chains."""
    n = 0
    for p in cfg.polymers:
        alpha = p.length / cfg.polymers[0].length
        one = sum(int(math.floor(alpha * b.lengthfrac / b.ds + 0.5)) for b in p.blocks)
        n += one if len(p.blocks) == 1 else 2 * one
    return n


def _iteration_work(cfg):
    N, nf = cfg.n_total, len(cfg.fields)
    size = 4 if cfg.precision == "mixed" else 8
    steps = _steps(cfg)
    fft = 2.5 * N * math.log2(N)
    # every propagator slice is written and read once (the contour sums pair the first slice of one
    # sweep with the last of the other), and every field is read and written once
    return 2.0 * steps * N * size + 8.0 * N * (4 * nf + 2), steps * (2 * fft + 4.0 * N)


def work(case):
    kind = case["kind"]
    if kind in ("scft", "batch"):
        cfgs = [_case_config(case)] if kind == "scft" else _batch_configs(case)
        both = [_iteration_work(c) for c in cfgs]
        return {"bytes": case["iterations"] * sum(b for b, _ in both), "flops": case["iterations"] * sum(f for _, f in both)}
    if kind == "adjoint":
        N = case["n"] ** 3
        # forward, its recomputation from checkpoints and the adjoint sweeps: the slices of two
        # sweeps written and read, each adjoint step two transform pairs
        return {"bytes": 4.0 * case["ns"] * 2 * N * 8, "flops": 2 * case["ns"] * 3 * (5.0 * N * math.log2(N) + 4 * N)}
    N = case["nx"] * case["ny"] * case["nz"]
    return {"bytes": 24.0 * N, "flops": 5.0 * N * math.log2(N) + N}


# ---------------------------------------------------------------------------
# The same values in 64 bits, from torch alone.
# ---------------------------------------------------------------------------
def _kernel(grid, cell, ds, device):
    """exp(-ds k^2) / N on the full grid."""
    k2 = torch.zeros(grid, dtype=torch.float64, device=device)
    for d in range(3):
        k = 2 * math.pi * torch.fft.fftfreq(grid[d], d=cell, dtype=torch.float64, device=device)
        k2 = k2 + (k * k).reshape([-1 if a == d else 1 for a in range(3)])
    return torch.exp(-ds * k2) / (grid[0] * grid[1] * grid[2])


def _sweep(q, w, steps, ds, half):
    """The slices of one block from start q: q <- e IFFT(half FFT(e q)), e = exp(-ds w / 2)."""
    e = torch.exp(-0.5 * ds * w)
    out = [q]
    for _ in range(steps):
        q = e * torch.fft.irfftn(half * torch.fft.rfftn(e * q), s=q.shape)
        out.append(q)
    return out


def _contour(qs, qts, ds):
    """The contour sum of q(n) qt(M - n): Simpson with the factor 0.33333, a trapezoid on the last
    interval where the number of points is even."""
    num = len(qs)
    at = lambda n: qs[n] * qts[num - 1 - n]  # noqa: E731
    acc = torch.zeros_like(qs[0])
    for n in range(0, num - 3 if num % 2 == 0 else num - 2, 2):
        acc = acc + 0.33333 * ds * (at(n) + 4.0 * at(n + 1) + at(n + 2))
    if num % 2 == 0:
        acc = acc + 0.5 * ds * (at(num - 2) + at(num - 1))
    return acc


def _exact_chain(fields, steps, star, w, ds, half, one):
    """(Q, density of each block) of a linear chain or an arm star from the field w of each block."""
    nb = len(steps)
    if star:
        outward = [_sweep(one, w[f], steps[b], ds, half) for b, f in enumerate(fields)]
        inward = []
        for b in range(nb):
            q = one
            for c in range(nb):
                if c != b:
                    q = q * outward[c][-1]
            inward.append(_sweep(q, w[fields[b]], steps[b], ds, half))
    else:
        outward, q = [], one
        for b in range(nb):
            outward.append(_sweep(q, w[fields[b]], steps[b], ds, half))
            q = outward[-1][-1]
        inward, q = [None] * nb, one
        for b in reversed(range(nb)):
            inward[b] = _sweep(q, w[fields[b]], steps[b], ds, half)
            q = inward[b][-1]
    big_q = (outward[0][0] * inward[0][-1]).mean()
    return big_q, [_contour(outward[b], inward[b], ds) / big_q for b in range(nb)]


def _exact_iterations(cfg, w, iterations):
    """Fields, densities, pressure and scalars after the iterations (steepest descent)."""
    grid, nf = cfg.n, len(cfg.fields)
    half = _kernel(grid, cfg.cell[0], cfg.polymers[0].blocks[0].ds, "cuda") * (grid[0] * grid[1] * grid[2])
    half = half[:, :, : grid[2] // 2 + 1]
    w = [x.reshape(grid) for x in w]
    one = torch.ones(grid, dtype=torch.float64, device="cuda")
    p = torch.zeros_like(one)
    pairs = [(cfg.fields.index(t.scfields[0]), cfg.fields.index(t.scfields[1]), t.chi * cfg.polymers[0].length)
             for t in cfg.interactions]
    avg = [0.0] * nf
    for poly in cfg.polymers:
        for b in poly.blocks:
            avg[cfg.fields.index(b.scfield)] += poly.volfrac * b.lengthfrac
    l0, l1 = cfg.updater.relaxlambdas
    for _ in range(iterations):
        phi = [torch.zeros_like(one) for _ in range(nf)]
        qs, ends = [], 0.0
        for poly in cfg.polymers:
            alpha = poly.length / cfg.polymers[0].length
            fields = [cfg.fields.index(b.scfield) for b in poly.blocks]
            steps = [int(math.floor(alpha * b.lengthfrac / b.ds + 0.5)) for b in poly.blocks]
            star = len(poly.blocks) > 2 and "freeEnd" in poly.blocks[1].headjoined
            q, dens = _exact_chain(fields, steps, star, w, poly.blocks[0].ds, half, one)
            for f, d in zip(fields, dens):
                phi[f] = phi[f] + (poly.volfrac / alpha) * d
            qs.append(float(q))
            ends -= poly.volfrac * math.log(float(q)) / alpha
        dh = []
        for i in range(nf):
            d = p - w[i]
            for a, b, c in pairs:
                if i in (a, b):
                    o = b if i == a else a
                    d = d + c * (phi[o] - avg[o])
            dh.append(d)
        w = [w[i] + l0 * (dh[i] - l1 * sum(dh[j] for j in range(nf) if j != i)) for i in range(nf)]
        p = sum(w)
        if nf == 3:
            for a, b, c in pairs:
                n = 3 - a - b
                p = p + c * (phi[n] - avg[n])
        p = p / nf
        p = p - p.mean()
        fe = -sum((phi[i] * w[i]).mean() for i in range(nf))
        nodis = ends + fe + sum(c * (phi[a] * phi[b]).mean() for a, b, c in pairs)
        full = nodis - sum(c * avg[a] * avg[b] for a, b, c in pairs)
        norm = math.sqrt(float(sum((d * d).sum() for d in dh)) / one.numel())
    return {"w": torch.stack([x.reshape(-1) for x in w]), "phi": torch.stack([x.reshape(-1) for x in phi]),
            "p": p.reshape(-1), "scalars": torch.tensor([float(full), float(nodis), norm] + qs, dtype=torch.float64)}


def exact(case, seed):
    kind = case["kind"]
    if kind == "scft":
        cfg = _case_config(case)
        return _exact_iterations(cfg, _fields(cfg.n, len(cfg.fields), seed), case["iterations"])
    if kind == "batch":
        return [_exact_iterations(c, _fields(c.n, len(c.fields), seed * 101 + k), case["iterations"])
                for k, c in enumerate(_batch_configs(case))]
    if kind == "adjoint":
        n, ns = case["n"], case["ns"]
        grid, N = (n, n, n), n ** 3
        w = _fields(grid, 2, seed).requires_grad_(True)
        box = torch.tensor([n * (6.0 / 64)] * 3, dtype=torch.float64, requires_grad=True)
        steps = [int(math.floor(case["f"] * ns + 0.5)), int(math.floor((1.0 - case["f"]) * ns + 0.5))]
        ds = torch.full((2,), 1.0 / ns, dtype=torch.float64, requires_grad=True)
        k2 = 0.0
        for d in range(3):
            i = torch.fft.fftfreq(n, dtype=torch.float64, device="cuda") * n
            if d == 2:
                i = i[: n // 2 + 1]
            k = 2 * math.pi * i / box[d].to("cuda")
            k2 = k2 + (k * k).reshape([-1 if a == d else 1 for a in range(3)])
        dsc = ds.to("cuda")
        half = [torch.exp(-dsc[b] * k2) for b in range(2)]
        one = torch.ones(grid, dtype=torch.float64, device="cuda")
        v = [w[b].reshape(grid) for b in range(2)]
        out0 = _sweep(one, v[0], steps[0], dsc[0], half[0])
        out1 = _sweep(out0[-1], v[1], steps[1], dsc[1], half[1])
        in1 = _sweep(one, v[1], steps[1], dsc[1], half[1])
        in0 = _sweep(in1[-1], v[0], steps[0], dsc[0], half[0])
        q = (out0[0] * in0[-1]).mean()
        phi = torch.stack([_contour(out0, in0, dsc[0]).reshape(N), _contour(out1, in1, dsc[1]).reshape(N)]) / q
        lnq = torch.log(q)
        (((phi[0] - _target(grid)) ** 2).sum() + 10.0 * lnq).backward()
        return {"phi": phi.detach(), "lnq": lnq.detach(), "dw": w.grad, "dbox": box.grad, "dds": ds.grad}
    grid = (case["nx"], case["ny"], case["nz"])
    data, kdata = _fft_inputs(grid, seed)
    x = torch.from_numpy(data).reshape(grid)
    # unnormalised transforms both ways
    y = torch.fft.ifftn(torch.from_numpy(kdata).reshape(grid) * torch.fft.fftn(x), norm="forward")
    return y.real.reshape(-1).contiguous().numpy()
