"""The 64-bit fixed-point chain of the strict FP64 stencils (star R=3..5, grid R=2..5) against the
oracle, bit for bit, where it changes form: values around powers of two (the rounding position differs
from point to point), windows of 126 to 129 values, of either sign, next to zero (the 96-bit form),
with a smallest value too small for 64 bits, and windows that climb through zero inside one launch; at
the grid's edges, on 64-row tiles, odd orders, row slabs and batches."""
import numpy as np
import pytest

import kernels_gb300 as kg
from oracle import prk_oracle as po

pytestmark = pytest.mark.gpu

STRICT = [(kg.STAR, 3), (kg.STAR, 4), (kg.STAR, 5), (kg.GRID, 2), (kg.GRID, 3), (kg.GRID, 4), (kg.GRID, 5)]
N = 140  # 5 x 3 tiles, ragged on both sides

WINDOWS = {
    "below_2_10": (1024 - 120, 1024), "around_2_10": (1024 - 60, 1024 + 60), "around_3_2_9": (1536 - 50, 1536 + 50),
    "around_2_18": (2 ** 18 - 64, 2 ** 18 + 63), "up_to_2_19": (2 ** 19 - 127, 2 ** 19), "negative": (-4160, -4040),
    "negative_2_19": (-(2 ** 19) + 1, -(2 ** 19) + 120), "from_one": (1, 128), "from_three": (3, 130),
    "from_100": (100, 227), "range_128": (900, 1028), "range_129": (900, 1029), "ends_at_minus_one": (-127, 0),
    "constant": (777, 778),
}


def same(x, y):
    return np.array_equal(np.ascontiguousarray(x).view(np.uint64), np.ascontiguousarray(y).view(np.uint64))


def fields(n, lo, hi, seed):
    rng = np.random.default_rng(seed)
    a = rng.integers(lo, hi, (n, n)).astype(np.float64)
    return a, rng.standard_normal((n, n)) * 50.0


def dev(torch, a):
    return torch.from_numpy(a.copy()).cuda()


@pytest.mark.parametrize("pattern,r", STRICT)
@pytest.mark.parametrize("window", sorted(WINDOWS))
def test_windows_one_application(cuda, pattern, r, window):
    for n in (N, N + 1):  # the TMA tiles and the plain-staged ones
        a, o = fields(n, *WINDOWS[window], seed=17 * r + pattern)
        want = o.copy()
        po.apply(pattern, r, a, want)
        in_, out = dev(cuda, a), dev(cuda, o)
        nxt = cuda.empty_like(in_)
        kg.apply(pattern, r, in_, out, nxt)
        assert same(out.cpu().numpy(), want) and same(nxt.cpu().numpy(), a + 1.0)
        out = dev(cuda, o)
        kg.apply(pattern, r, in_, out)
        assert same(out.cpu().numpy(), want)


@pytest.mark.parametrize("pattern,r", STRICT)
@pytest.mark.parametrize("lo,hi", [(-150, -70), (-60, -10), (-3, 40), (1000, 1060), (2 ** 16 - 90, 2 ** 16 - 20)])
def test_windows_that_climb(cuda, pattern, r, lo, hi):
    """170 applications in one launch (every form of the window, rebuilt as the values climb past its
    tables), and the same through launches of eight on 32- and 64-row tiles."""
    apps = 170
    for n in (N, N + 1):
        a, o = fields(n, lo, hi, seed=r + 7 * pattern)
        want_in, want = a.copy(), o.copy()
        for _ in range(apps + 1):
            po.apply(pattern, r, want_in, want)
            want_in += 1.0
        for kw in ({"whole": True}, {"depth": 8}, {"depth": 8, "tall": True}):
            if n != N and "tall" in kw:
                continue
            in_a, out = dev(cuda, a), dev(cuda, o)
            res = kg.run(pattern, r, apps, in_a, cuda.empty_like(in_a), out, **kw)
            assert same(out.cpu().numpy(), want), (n, kw)
            assert same(res.final_in.cpu().numpy(), want_in), (n, kw)


@pytest.mark.parametrize("pattern,r", STRICT)
def test_slabs_and_batches(cuda, pattern, r):
    n, apps = N, 5
    a, o = fields(n, 1000, 1100, seed=3 * r)
    want_in, want = a.copy(), o.copy()
    for _ in range(apps):
        po.apply(pattern, r, want_in, want)
        want_in += 1.0
    got, got_in = o.copy(), a.copy()
    for b, e in ((0, 37), (37, 101), (101, n)):
        lo, hi = max(0, b - r), min(n, e + r)
        in_, out = dev(cuda, a[lo:hi]), dev(cuda, o[lo:hi])
        nxt = cuda.empty_like(in_)
        kg.slab_run(pattern, r, n, apps, b, e, in_, nxt, out)
        got[b:e], got_in[b:e] = out.cpu().numpy()[b - lo:e - lo], nxt.cpu().numpy()[b - lo:e - lo]
    assert same(got, want) and same(got_in, want_in)
    in_a, out = dev(cuda, a), dev(cuda, o)
    batch = kg.Batch([(pattern, r, in_a, cuda.empty_like(in_a), out)], whole=True)
    batch.run(apps - 1)
    assert same(out.cpu().numpy(), want) and same(batch.final_in(0).cpu().numpy(), want_in)
