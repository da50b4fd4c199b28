"""FP32C on whole-number tiles of small range (the integer route) and just off it: values 127 to 129 from
the tile's middle, one value that is not whole, magnitudes up to and past 2^21, more applications than
one FP32 sum or the whole route takes, on TMA tiles, plain-staged tiles, 64-row tiles, slabs, batches and
in the operator form. The result is compared with the exact sum of the taps."""
import numpy as np
import pytest

import kernels_gb300 as kg
from oracle import prk_oracle as po

pytestmark = pytest.mark.gpu

ALL = [(p, r) for p in (kg.STAR, kg.GRID) for r in range(1, 6)]


def exact(pattern, r, a, apps):
    """apps * S(a) in extended precision on the interior (the weights sum to zero, so in += 1 changes no
    application's sum), and apps * sum |w d| over the pairs of taps d."""
    n = a.shape[0]
    x = a.astype(np.longdouble)
    s = np.zeros((n - 2 * r, n - 2 * r), np.longdouble)
    m = np.zeros_like(s)
    for dc, dr, w in po.taps(pattern, r):
        if w > 0:
            den = np.longdouble(round(1.0 / w))
            d = x[r + dr:n - r + dr, r + dc:n - r + dc] - x[r - dr:n - r - dr, r - dc:n - r - dc]
            s += d / den
            m += np.abs(d) / den
    return s * apps, m * apps


def check(pattern, r, a, out0, got, apps, whole=True):
    """Every point of a tile on the route, against the exact sum. Grid R=5's route takes values within 128
    of the tile's middle only: the tile that holds a[0, 0], past that range, keeps the group sums, whose
    lazily renormalised out is not what is checked here."""
    s, m = exact(pattern, r, a, apps)
    n = a.shape[0]
    if (pattern, r) == (kg.GRID, 5) and whole and abs(float(a[0, 0]) - float(a[1, 1])) > 64:
        s, got = s.copy(), got.copy()
        k = (slice(r, 64), slice(r, 128))
        got[k] = 0.0
        got[k][..., 0] = out0[k]
        s[:64 - r, :128 - r] = 0.0
    inner = (slice(r, n - r), slice(r, n - r))
    want = out0[inner].astype(np.longdouble) + s
    err = np.abs(got[..., 0][inner].astype(np.longdouble) + got[..., 1][inner].astype(np.longdouble) - want)
    # two-float sums and products: 2^-44 of the terms' magnitude; a difference of values that are not
    # whole, and the sums of a group's, round to 24 bits first, once per tap of an application
    bound = (m + np.abs(out0[inner])) * np.longdouble(2.0 ** -44) + (0 if whole else m * np.longdouble(2.0 ** -20))
    assert (err <= bound).all(), float((err / bound).max())


def run_all(cuda, pattern, r, a, apps, whole=True):
    n = a.shape[0]
    rng = np.random.default_rng(r)
    out0 = rng.integers(-50, 50, (n, n)).astype(np.float32)
    out_h = np.zeros((n, n, 2), np.float32)
    out_h[..., 0] = out0

    def fresh():
        return cuda.from_numpy(a.copy()).cuda(), cuda.from_numpy(out_h.copy()).cuda()

    final = a.astype(np.float64) + apps
    forms = [{"depth": 8}, {"whole": True}] + ([{"depth": 4, "tall": True}] if n % 4 == 0 else [])
    for kw in forms:
        in_a, out = fresh()
        res = kg.run(pattern, r, apps - 1, in_a, cuda.empty_like(in_a), out, **kw)
        check(pattern, r, a, out0, out.cpu().numpy(), apps, whole)
        if whole:
            assert np.array_equal(res.final_in.cpu().numpy().astype(np.float64), final), kw
    in_a, out = fresh()
    batch = kg.Batch([(pattern, r, in_a, cuda.empty_like(in_a), out)], whole=True)
    batch.run(apps - 1)
    check(pattern, r, a, out0, out.cpu().numpy(), apps, whole)
    for nxt in (False, True):  # one application, the operator form and the fused form
        in_, out = fresh()
        kg.apply(pattern, r, in_, out, cuda.empty_like(in_) if nxt else None)
        check(pattern, r, a, out0, out.cpu().numpy(), 1, whole)


@pytest.mark.parametrize("pattern,r", ALL)
@pytest.mark.parametrize("n", [180, 149])
@pytest.mark.parametrize("base,spread", [(0, 127), (1000, 128), (-500, 129), (2 ** 21 - 200, 120), (2 ** 21 + 50, 120),
                                         (-(2 ** 20), 40)])
def test_whole_fields(cuda, pattern, r, n, base, spread):
    rng = np.random.default_rng(11 * r + pattern)
    a = (base + rng.integers(-spread // 2, spread // 2 + 1, (n, n))).astype(np.float32)
    a[n // 2, n // 2] = base + spread // 2
    a[0, 0] = base - spread // 2 - spread  # one tile at the edge of the range or past it
    run_all(cuda, pattern, r, a, 18)


@pytest.mark.parametrize("pattern,r", ALL)
@pytest.mark.parametrize("n", [180, 149])
def test_one_value_off(cuda, pattern, r, n):
    """A tile with one value that is not whole takes the group sums, its neighbours the integer route."""
    ii, jj = np.meshgrid(np.arange(n), np.arange(n), indexing="ij")
    a = (ii + jj).astype(np.float32)
    a[40, 70] += 0.5
    run_all(cuda, pattern, r, a, 10, whole=False)


@pytest.mark.parametrize("pattern,r", [(kg.GRID, 5), (kg.GRID, 4), (kg.STAR, 5)])
def test_more_applications_than_one_sum_takes(cuda, pattern, r):
    """Launches of more applications than one FP32 sum takes, up to those the route takes (462 for grid
    R=5), on a field that keeps every tile in range; and one application more, which grid R=5 runs on the
    group sums (the form's 1e-6 bound)."""
    n = 100
    rng = np.random.default_rng(3)
    a = (700 + rng.integers(-60, 61, (n, n))).astype(np.float32)
    out0 = np.zeros((n, n), np.float32)
    for apps in (130, 462, 463):
        in_, out = cuda.from_numpy(a.copy()).cuda(), cuda.zeros((n, n, 2), device="cuda")
        in_b = cuda.empty_like(in_)
        kg.slab_run(pattern, r, n, apps, 0, n, in_, in_b, out)
        got = out.cpu().numpy()
        if apps <= 462:
            check(pattern, r, a, out0, got, apps)
        else:
            s, m = exact(pattern, r, a, apps)
            inner = (slice(r, n - r), slice(r, n - r))
            assert (np.abs(got[..., 0][inner].astype(np.longdouble) + got[..., 1][inner] - s) <= 1e-6 * m).all()
        assert np.array_equal(in_b.cpu().numpy(), a + np.float32(apps))


@pytest.mark.parametrize("pattern,r", ALL)
@pytest.mark.parametrize("n", [180, 149])
@pytest.mark.parametrize("base", [64, -100000])
def test_small_value_among_whole_ones(cuda, pattern, r, n, base):
    """A value of 2^-20 whose difference from the tile's middle rounds to a whole number: the tile keeps the
    group sums, in += 1 keeps the value (its sums with 1..6 are exact in FP32), and the points around it,
    in a block of zeros, get its taps."""
    a = np.full((n, n), base, np.float32)
    a[4:28, 8:32] = 0.0
    a[16, 20] = 2.0 ** -20
    zeros, apps = np.zeros((n, n), np.float32), 6

    def fresh():
        return cuda.from_numpy(a.copy()).cuda(), cuda.zeros((n, n, 2), device="cuda")

    in_a, out = fresh()
    res = kg.run(pattern, r, apps - 1, in_a, cuda.empty_like(in_a), out, whole=True)
    check(pattern, r, a, zeros, out.cpu().numpy(), apps, whole=False)
    assert np.array_equal(res.final_in.cpu().numpy().astype(np.float64), a.astype(np.float64) + apps)
    in_a, out = fresh()
    kg.Batch([(pattern, r, in_a, cuda.empty_like(in_a), out)], whole=True).run(apps - 1)
    check(pattern, r, a, zeros, out.cpu().numpy(), apps, whole=False)
    for nxt in (False, True):
        in_, out = fresh()
        nx = cuda.empty_like(in_) if nxt else None
        kg.apply(pattern, r, in_, out, nx)
        check(pattern, r, a, zeros, out.cpu().numpy(), 1, whole=False)
        assert nx is None or np.array_equal(nx.cpu().numpy().astype(np.float64), a.astype(np.float64) + 1)
