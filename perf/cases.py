"""The workloads the stencil library's speed is judged by: what a program that uses it calls, through
the public entry points of kernels_gb300, over the sizes, types and options in earnest use.

A case is a dict: `kind` says which calls it makes (below), the rest sizes and options.

  run     a PRK run as a driver makes it: kg.run (iterations + 1 applications, each followed by
          in += 1), then the norm the driver checks. depth 1, 2, 4 or 8 applications per launch, or
          "whole" for every timed application in one launch
  dropin  one trip of a reference driver whose operator was replaced: starR/gridR(n, tile, in, out),
          then in += 1
  apply   one fused application: out += S(in) and in_next = in + 1 (kg.apply)
  batch   independent grids advanced together by a kg.Batch the program keeps
  host    a run from host arrays, copies included, as the CPU drivers hold them (kg.run_host)
  nstream, transpose   one iteration of the two neighbouring PRK kernels

Fields: "prk" is the field of a PRK run k0 applications in, in = i + j + k0 and out = 2 k0 inside (k0
from the seed); "real" is uniform in [0, 1), for programs that use the operators on measured or
computed data.
"""
from __future__ import annotations

import math
import random

import torch

import kernels_gb300 as kg

PATTERN = {"star": kg.STAR, "grid": kg.GRID}
DTYPE = {"fp64": kg.FP64, "fp32c": kg.FP32C}


def listed() -> list[dict]:
    return [
        # the reference's continuous-integration run: 10 iterations of a small grid, where launches
        # and host work count
        dict(name="ci_run", kind="run", pattern="star", r=2, n=200, iterations=10, depth=1, dtype="fp64"),
        # a trip of a reference driver at its default test size, its operator swapped for ours
        dict(name="dropin_small", kind="dropin", pattern="star", r=2, n=1000, dtype="fp64", field="prk"),
        # the same at a large odd order with a wide stencil
        dict(name="dropin_odd", kind="dropin", pattern="grid", r=4, n=8191, dtype="fp64", field="prk"),
        # the headline: one fused application of star R=2 on the large grid
        dict(name="fused_star2", kind="apply", pattern="star", r=2, n=16384, dtype="fp64", field="prk"),
        # the other stencil of that configuration
        dict(name="fused_grid2", kind="apply", pattern="grid", r=2, n=16384, dtype="fp64", field="prk"),
        # a field of real numbers, where no tile is whole
        dict(name="fused_real", kind="apply", pattern="star", r=3, n=8192, dtype="fp64", field="real"),
        # the compensated single-precision form on an order no tensor map takes
        dict(name="fused_fp32c_odd", kind="apply", pattern="grid", r=3, n=8189, dtype="fp32c", field="prk"),
        # the radius sweep: a whole run of a wide stencil
        dict(name="sweep_grid5", kind="run", pattern="grid", r=5, n=16384, iterations=20, depth="whole", dtype="fp64"),
        # the large configuration's stencil in the compensated form, several applications per launch
        dict(name="large_fp32c", kind="run", pattern="star", r=4, n=32768, iterations=48, depth=8, dtype="fp32c"),
        # many independent grids of uneven order, radius and pattern
        dict(name="batch", kind="batch", count=32, n_lo=128, n_hi=2048, iterations=20, depth="whole", dtype="fp64", pick=11),
        # a run from host arrays: copies in, 101 applications, copies back, norm
        dict(name="host_run", kind="host", pattern="star", r=2, n=8192, iterations=100, dtype="fp64"),
        # the triad on the same bandwidth roofline
        dict(name="nstream", kind="nstream", length=1 << 27),
    ]


def _log(rng: random.Random, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random) -> dict:
    kind = rng.choice(["run", "run", "dropin", "dropin", "apply", "apply", "apply", "batch", "host", "nstream", "transpose"])
    pattern, r = rng.choice(["star", "grid"]), rng.randint(1, 5)
    dtype = rng.choice(["fp64", "fp64", "fp32c"])
    if kind == "run":
        return dict(kind=kind, pattern=pattern, r=r, n=_log(rng, 200, 12000), iterations=rng.randint(5, 20),
                    depth=rng.choice([1, 2, 4, 8, "whole"]), dtype=dtype)
    if kind in ("dropin", "apply"):
        return dict(kind=kind, pattern=pattern, r=r, n=_log(rng, 500, 16384), dtype=dtype,
                    field=rng.choice(["prk", "prk", "prk", "real"]))
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(4, 32), n_lo=128, n_hi=_log(rng, 512, 2048),
                    iterations=rng.randint(5, 20), depth=rng.choice([1, 8, "whole"]), dtype=dtype,
                    pick=rng.randint(0, 1 << 30))
    if kind == "host":
        return dict(kind=kind, pattern=pattern, r=r, n=_log(rng, 500, 6000), iterations=rng.randint(10, 100), dtype=dtype)
    if kind == "nstream":
        return dict(kind=kind, length=_log(rng, 1 << 16, 1 << 27))
    return dict(kind=kind, n=_log(rng, 256, 12000))


# ---- inputs -----------------------------------------------------------------------------------


def _grids(case: dict) -> list[tuple[int, int, int]]:
    """(pattern, radius, n) of each grid of a batch: n log-uniform, R in 1..4, star or grid."""
    rng = random.Random(case["pick"])
    return [(rng.randint(0, 1), rng.randint(1, 4), _log(rng, case["n_lo"], case["n_hi"])) for _ in range(case["count"])]


def _start(seed: int) -> int:
    return random.Random(seed).randint(0, 1000)


def _field(n: int, r: int, dtype: int, field: str, seed: int, device: str):
    """in and out of a grid before the call."""
    tdt = torch.float64 if dtype == kg.FP64 else torch.float32
    out = torch.zeros((n, n) if dtype == kg.FP64 else (n, n, 2), dtype=tdt, device=device)
    inner = out[r:n - r, r:n - r] if dtype == kg.FP64 else out[r:n - r, r:n - r, 0]
    if field == "real":
        gen = torch.Generator(device=device)
        gen.manual_seed(seed)
        in_ = torch.rand((n, n), dtype=tdt, device=device, generator=gen)
        inner.copy_(torch.rand((n - 2 * r, n - 2 * r), dtype=tdt, device=device, generator=gen))
    else:
        k0 = _start(seed)
        i = torch.arange(n, dtype=tdt, device=device)
        in_ = i[:, None] + (i + k0)[None, :]
        inner.fill_(2.0 * k0)
    return in_, out


def _vectors(case: dict, seed: int):
    """A, B, C of the triad k0 iterations in (A = 0, B = C = 2, scalar 3 at the start)."""
    k0, length = _start(seed), case["length"]
    return (torch.full((length,), 8.0 * k0, dtype=torch.float64, device="cuda"),
            torch.full((length,), 2.0, dtype=torch.float64, device="cuda"),
            torch.full((length,), 2.0, dtype=torch.float64, device="cuda"))


def _matrices(case: dict, seed: int):
    """A and B of the transpose: A[j][i] = order j + i plus the iterations so far, B their sum."""
    n, k0 = case["n"], _start(seed)
    a = torch.arange(n * n, dtype=torch.float64, device="cuda").reshape(n, n)
    b = (a.t() * float(k0) + k0 * (k0 - 1) / 2.0).contiguous()
    return a + float(k0), b


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    if kind == "nstream":
        return {"case": case, "v": _vectors(case, seed)}
    if kind == "transpose":
        return {"case": case, "v": _matrices(case, seed)}
    dtype = DTYPE[case["dtype"]]
    if kind == "batch":
        grids = []
        for k, (p, r, n) in enumerate(_grids(case)):
            in_a, out = _field(n, r, dtype, "prk", seed + k, "cuda")
            grids.append((p, r, in_a, torch.empty_like(in_a), out))
        whole = case["depth"] == "whole"
        return {"case": case, "grids": grids,
                "batch": kg.Batch(grids, depth=None if whole else case["depth"], whole=whole)}
    r, n = case["r"], case["n"]
    in_a, out = _field(n, r, dtype, case.get("field", "prk"), seed, "cuda")
    if kind == "host":
        pin = {"device": "cpu", "pin_memory": True}
        h_in, h_out = torch.empty(in_a.shape, dtype=in_a.dtype, **pin), torch.empty(out.shape, dtype=out.dtype, **pin)
        h_in.copy_(in_a)
        h_out.copy_(out)
        return {"case": case, "in": h_in, "out": h_out, "final": torch.empty(in_a.shape, dtype=in_a.dtype, **pin)}
    state = {"case": case, "in": in_a, "out": out}
    if kind == "dropin":
        state["op"] = getattr(kg, f"{case['pattern']}{r}")
    else:
        state["other"] = torch.empty_like(in_a)
    return state


def run(state: dict):
    case = state["case"]
    kind = case["kind"]
    if kind == "run":
        whole = case["depth"] == "whole"
        res = kg.run(PATTERN[case["pattern"]], case["r"], case["iterations"], state["in"], state["other"], state["out"],
                     depth=1 if whole else case["depth"], whole=whole)
        if res.final_in is not state["in"]:
            state["in"], state["other"] = state["other"], state["in"]
        return {"in": state["in"], "out": state["out"], "norm": kg.norm(case["r"], state["out"])}
    if kind == "dropin":
        state["op"](case["n"], 32, state["in"], state["out"])
        kg.add(state["in"])
        return {"in": state["in"], "out": state["out"]}
    if kind == "apply":
        kg.apply(PATTERN[case["pattern"]], case["r"], state["in"], state["out"], state["other"])
        state["in"], state["other"] = state["other"], state["in"]
        return {"in": state["in"], "out": state["out"]}
    if kind == "batch":
        b = state["batch"]
        b.run(case["iterations"], graph=True)
        return {"in": [b.final_in(k) for k in range(case["count"])], "out": [g[4] for g in state["grids"]]}
    if kind == "host":
        res = kg.run_host(PATTERN[case["pattern"]], case["r"], case["iterations"], state["in"], state["out"], state["final"])
        state["in"], state["final"] = state["final"], state["in"]
        return {"in": state["in"], "out": state["out"], "norm": res["norm"]}
    if kind == "nstream":
        a, b, c = state["v"]
        kg.nstream(a, b, c, 3.0)
        return {"A": a}
    a, b = state["v"]
    kg.transpose(a, b)
    return {"A": a, "B": b}


# ---- work and exact results -------------------------------------------------------------------


def _work(pattern: str, r: int, n: int, apps: int, dtype: str) -> tuple[float, float]:
    size = 4 * r + 1 if pattern == "star" else (2 * r + 1) ** 2
    inner = float(n - 2 * r) ** 2
    return (16.0 if dtype == "fp64" else 8.0) * n * n + 16.0 * inner, (2.0 * size + 1.0) * inner * apps


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "nstream":
        return {"bytes": 32.0 * case["length"], "flops": 2.0 * case["length"]}
    if kind == "transpose":
        return {"bytes": 32.0 * case["n"] ** 2, "flops": 2.0 * case["n"] ** 2}
    apps = case.get("iterations", 0) + 1
    grids = [(("star", "grid")[p], r, n) for p, r, n in _grids(case)] if kind == "batch" else \
        [(case["pattern"], case["r"], case["n"])]
    each = [_work(p, r, n, apps, case["dtype"]) for p, r, n in grids]
    return {"bytes": sum(b for b, _ in each), "flops": sum(f for _, f in each)}


def _taps(pattern: str, r: int) -> list[tuple[int, int, float]]:
    """(row offset, column offset, weight) of the positive half of a PRK stencil, whose other half is
    its point mirror with the sign turned: the weight matrix of the reference's generator."""
    taps = []
    for dr in range(0, r + 1):
        for dc in range(-r, r + 1):
            if dr == 0 and dc <= 0:
                continue
            m = max(abs(dr), abs(dc))
            if pattern == "star":
                if dr == 0 or dc == 0:
                    taps.append((dr, dc, 1.0 / (2 * m * r)))
            elif abs(dr) == abs(dc):
                if dr == dc:
                    taps.append((dr, dc, 1.0 / (4 * m * r)))
            else:
                w = 1.0 / (4 * m * (2 * m - 1) * r)
                taps.append((dr, dc, w if (dr if dr == m else dc) > 0 else -w))
    return taps


def _exact_grid(pattern: str, r: int, in_: torch.Tensor, out: torch.Tensor, apps: int):
    """in and out after `apps` applications in 64 bits. The weights sum to zero, so every application
    of a run adds the same S."""
    n = in_.shape[0]
    x = in_.double()
    m = n - 2 * r
    s = torch.zeros((m, m), dtype=torch.float64, device=x.device)
    for dr, dc, w in _taps(pattern, r):
        s += (x[r + dr:r + dr + m, r + dc:r + dc + m] - x[r - dr:r - dr + m, r - dc:r - dc + m]).mul_(w)
    s *= float(apps)
    end = in_.add_(float(apps)) if in_.dtype == torch.float64 else (x + float(apps)).float()
    if out.dim() == 2:
        out[r:n - r, r:n - r] += s
        return end, out
    s += out[r:n - r, r:n - r, 0].double() + out[r:n - r, r:n - r, 1].double()
    hi = s.float()  # the pair (hi, lo) whose sum is the value
    out[r:n - r, r:n - r, 0] = hi
    out[r:n - r, r:n - r, 1] = (s - hi.double()).float()
    return end, out


def _norm(r: int, out: torch.Tensor) -> float:
    n = out.shape[0]
    v = out if out.dim() == 2 else out[..., 0].double() + out[..., 1].double()
    return float(v[r:n - r, r:n - r].abs().sum()) / float(n - 2 * r) ** 2


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind == "nstream":
        a, b, c = _vectors(case, seed)
        return {"A": a + b + 3.0 * c}
    if kind == "transpose":
        a, b = _matrices(case, seed)
        b += a.t()
        return {"A": a + 1.0, "B": b}
    dtype = DTYPE[case["dtype"]]
    apps = case.get("iterations", 0) + 1
    if kind == "batch":
        ends, outs = [], []
        for k, (p, r, n) in enumerate(_grids(case)):
            end, out = _exact_grid(("star", "grid")[p], r, *_field(n, r, dtype, "prk", seed + k, "cuda"), apps)
            ends.append(end)
            outs.append(out)
        return {"in": ends, "out": outs}
    r = case["r"]
    end, out = _exact_grid(case["pattern"], r, *_field(case["n"], r, dtype, case.get("field", "prk"), seed, "cuda"), apps)
    if kind in ("run", "host"):
        return {"in": end, "out": out, "norm": _norm(r, out)}
    return {"in": end, "out": out}
