"""Kernels launched while the stream's previous kernel still runs (launch_chained): by source, each waits
(chain_wait), and none takes a __restrict__ pointer, through which a load may be moved above the wait; on
the GPU, many launches in a row on odd orders give what the same launches give one at a time."""
import re
from pathlib import Path

import numpy as np
import pytest

import kernels_gb300 as kg
from oracle import prk_oracle as po

CSRC = Path(kg.__file__).resolve().parent / "csrc"


def chained_kernels():
    """(name, parameter list, body) of every kernel that some launch_chained call names."""
    text = "\n".join(p.read_text() for p in sorted(CSRC.glob("*.cu*")))
    calls = " ".join(re.findall(r"launch_chained\(([^;]*?);", text))
    found = {}
    for m in re.finditer(r"__global__[^{;]*?\b(k_\w+)\(([^{;]*)\)\s*\{(.*?)\n\}", text, re.S):
        if re.search(rf"\b{m.group(1)}\b", calls):
            found[m.group(1)] = (m.group(2), m.group(3))
    return found


def test_chained_kernels_by_source():
    found = chained_kernels()
    assert set(found) == {"k_stencil_tile", "k_stencil_plain", "k_add", "k_norm_partial", "k_norm_final"}
    for name, (params, body) in found.items():
        assert "__restrict__" not in params, name
        assert "chain_wait()" in body, name


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [kg.FP64, kg.FP32C])
@pytest.mark.parametrize("pattern,r", [(kg.STAR, 1), (kg.STAR, 2), (kg.GRID, 1), (kg.GRID, 3), (kg.STAR, 5)])
@pytest.mark.parametrize("n", [333, 1001])
def test_launches_in_a_row(cuda, pattern, r, n, dtype):
    """40 applications, one per launch, on the plain-staged kernels: each reads what the one before wrote."""
    apps = 40
    rng = np.random.default_rng(n + r)
    tdt = cuda.float64 if dtype == kg.FP64 else cuda.float32
    a = cuda.from_numpy(rng.uniform(-50.0, 50.0, (n, n))).to(tdt)
    o = cuda.from_numpy(rng.uniform(-1.0, 1.0, (n, n) if dtype == kg.FP64 else (n, n, 2))).to(tdt)

    def run(wait):
        bufs, out = [a.cuda(), cuda.empty((n, n), dtype=tdt, device="cuda")], o.cuda()
        for k in range(apps):
            kg.apply(pattern, r, bufs[k & 1], out, bufs[(k + 1) & 1])
            if wait:
                cuda.cuda.synchronize()
        cuda.cuda.synchronize()
        return bufs[apps & 1].cpu().numpy(), out.cpu().numpy()

    got_in, got = run(False)
    want_in, want = run(True)
    assert np.array_equal(got_in, want_in) and np.array_equal(got, want)
    if dtype == kg.FP64:
        ref_in, ref = a.numpy().copy(), o.numpy().copy()
        for _ in range(apps):
            po.apply(pattern, r, ref_in, ref)
            ref_in += 1.0
        assert np.array_equal(got_in, ref_in) and np.array_equal(got.view(np.uint64), ref.view(np.uint64))
