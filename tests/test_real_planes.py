"""The shared-memory plane of products that FP64 tiles of real values use (star R=3..5, grid R=2..5): by
source, the tile loads' mbarrier, over which the plane lies, is ended before the tile is evaluated; on the
GPU, 64-row tiles and row slabs give the oracle's bits."""
import re
from pathlib import Path

import numpy as np
import pytest

import kernels_gb300 as kg
from oracle import prk_oracle as po

STRICT = [(kg.STAR, 3), (kg.STAR, 4), (kg.STAR, 5), (kg.GRID, 2), (kg.GRID, 3), (kg.GRID, 4), (kg.GRID, 5)]


def test_barrier_ends_before_its_memory_is_reused():
    text = (Path(kg.__file__).resolve().parent / "csrc" / "stencil_tile.cuh").read_text()
    body = text[re.search(r"\bk_stencil_tile\(const __grid_constant__", text).start():]
    body = body[:body.index("\n}")]
    wait = body.index("__syncthreads_and(mbar_wait_bounded(bar, 0))")
    assert wait < body.index("mbar_inval(bar)") < body.index("process_tile<")


@pytest.fixture(scope="module")
def case():
    n, apps = 180, 9
    rng = np.random.default_rng(2)
    a, o = rng.standard_normal((n, n)) * 10.0, rng.standard_normal((n, n))
    return n, apps, a, o


@pytest.mark.gpu
@pytest.mark.parametrize("pattern,r", STRICT)
def test_tall_tiles_and_slabs(cuda, case, pattern, r):
    n, apps, a, o = case
    want_in, want = a.copy(), o.copy()
    for _ in range(apps):
        po.apply(pattern, r, want_in, want)
        want_in += 1.0
    for depth in (1, 2, 4, 8):
        in_a, out = cuda.from_numpy(a.copy()).cuda(), cuda.from_numpy(o.copy()).cuda()
        res = kg.run(pattern, r, apps - 1, in_a, cuda.empty_like(in_a), out, depth=depth, tall=True)
        assert np.array_equal(out.cpu().numpy(), want), depth
        assert np.array_equal(res.final_in.cpu().numpy(), want_in), depth
    got, got_in = o.copy(), a.copy()
    for b, e in ((0, 45), (45, 101), (101, n)):
        lo, hi = max(0, b - r), min(n, e + r)
        in_, out = cuda.from_numpy(a[lo:hi].copy()).cuda(), cuda.from_numpy(o[lo:hi].copy()).cuda()
        nxt = cuda.empty_like(in_)
        kg.slab_run(pattern, r, n, apps, b, e, in_, nxt, out)
        got[b:e], got_in[b:e] = out.cpu().numpy()[b - lo:e - lo], nxt.cpu().numpy()[b - lo:e - lo]
    assert np.array_equal(got, want) and np.array_equal(got_in, want_in)
