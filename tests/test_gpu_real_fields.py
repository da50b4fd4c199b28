"""FP64 on real-valued tiles (products shared between taps or fused into the adds) against the oracle, bit
for bit: random reals of small and large magnitudes, signed zeros, values at the ends of the exponent
range the path takes and past them (the plain chain), infinities and NaNs, one application and several,
on TMA, plain-staged and batched tiles and in the operator form."""
import numpy as np
import pytest

import kernels_gb300 as kg
from oracle import prk_oracle as po

pytestmark = pytest.mark.gpu

ALL = [(p, r) for p in (kg.STAR, kg.GRID) for r in range(1, 6)]
NAN = 0x7FF8000000000000


def fields(n):
    rng = np.random.default_rng(n)
    f = {"unit": rng.random((n, n)), "signed": rng.standard_normal((n, n)) * 1e3}
    z = rng.standard_normal((n, n))
    z[rng.random((n, n)) < 0.3] = 0.0
    z[rng.random((n, n)) < 0.3] = -0.0
    f["zeros"] = z
    f["wide"] = rng.standard_normal((n, n)) * 2.0 ** rng.integers(-60, 60, (n, n)).astype(np.float64)
    for name, e in (("lowest", -895), ("below", -897), ("highest", 876), ("above", 878)):
        v = rng.standard_normal((n, n))
        v[n // 3, n // 3] = np.ldexp(1.0 + rng.random(), e)  # the ends of the range: 2^-895 and 2^877
        f[name] = v
    t = rng.standard_normal((n, n))
    t[::7, ::5] = 5e-324
    t[1::9, 2::5] = -3e-310
    f["subnormal"] = t
    i = rng.standard_normal((n, n))
    i[20, 30], i[50, 60], i[70, 8] = np.inf, -np.inf, np.nan
    f["specials"] = i
    return f


def same(got, want):
    """Equal bits; where the oracle has a NaN, a NaN."""
    g, w = np.ascontiguousarray(got).view(np.uint64), np.ascontiguousarray(want).view(np.uint64)
    nan = np.isnan(want)
    return np.array_equal(np.isnan(got), nan) and np.array_equal(g[~nan], w[~nan])


@pytest.mark.parametrize("pattern,r", ALL)
@pytest.mark.parametrize("n", [140, 141])
def test_bit_exact(cuda, pattern, r, n):
    rng = np.random.default_rng(5)
    o = rng.standard_normal((n, n))
    o[::3] = -0.0
    for name, a in fields(n).items():
        with np.errstate(all="ignore"):
            want1, a1 = o.copy(), a + 1.0
            po.apply(pattern, r, a, want1)
            want3, a3 = want1.copy(), a1.copy()
            for _ in range(3):
                po.apply(pattern, r, a3, want3)
                a3 += 1.0
        in_, out = cuda.from_numpy(a.copy()).cuda(), cuda.from_numpy(o.copy()).cuda()
        nxt = cuda.empty_like(in_)
        kg.apply(pattern, r, in_, out, nxt)
        assert same(out.cpu().numpy(), want1) and same(nxt.cpu().numpy(), a1), name
        out = cuda.from_numpy(o.copy()).cuda()
        kg.apply(pattern, r, in_, out)
        assert same(out.cpu().numpy(), want1), name
        for form in ("steps", "batch"):
            out = cuda.from_numpy(o.copy()).cuda()
            if form == "steps":
                kg.apply_steps(pattern, r, 4, in_, out, nxt)
            else:
                batch = kg.Batch([(pattern, r, in_.clone(), nxt, out)], whole=True)
                batch.run(3)
                nxt = batch.final_in(0)
            assert same(out.cpu().numpy(), want3) and same(nxt.cpu().numpy(), a3), (name, form)
