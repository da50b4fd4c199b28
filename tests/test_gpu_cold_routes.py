"""The speed of FP64 routes that few fields take: the plain chain on tiles that hold a subnormal, against its
binary64 operations at the measured rate (two neighbouring points share products, so it beats one product and
one add per tap), and the 96-bit form on values about zero."""
import statistics

import pytest

import kernels_gb300 as kg

pytestmark = pytest.mark.gpu


def median(torch, call):
    """Median seconds of nine timings of three calls."""
    ts = []
    for _ in range(9):
        e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        e[0].record()
        for _ in range(3):
            call()
        e[1].record()
        torch.cuda.synchronize()
        ts.append(e[0].elapsed_time(e[1]) / 3e3)
    return statistics.median(ts)


def test_plain_chain_shares_products(cuda):
    n, r = 4096, 5
    in_a, in_b, out = kg.alloc(n)
    kg.init(in_a, out)
    in_a.copy_(cuda.rand_like(in_a))
    in_a[::16, ::16] = 1e-310
    ops = 2 * (2 * r + 1) ** 2 - 2 * (2 * r + 1)  # 110 taps, a product and an add each
    at_rate = ops * (n - 2 * r) ** 2 / kg.probe_dadd()
    # 1.03 of it with a product per tap, 0.92 with the shared ones
    assert median(cuda, lambda: kg.apply(kg.GRID, r, in_a, out, in_b)) <= 0.97 * at_rate


@pytest.mark.parametrize("pattern,r,most", [(kg.STAR, 3, 1.75), (kg.GRID, 2, 2.0)])
def test_values_about_zero(cuda, pattern, r, most):
    """The 96-bit form, which windows that hold zero take, on 64-row tiles, against the 64-bit form on a PRK
    field: 1.62 (star R=3) and 1.84 times as long per application; 1.89 and 2.19 as a loop over the taps."""
    n = 4096
    in_a, in_b, out = kg.alloc(n)
    kg.init(in_a, out)
    in_a += 8192.0
    narrow = median(cuda, lambda: kg.apply_steps(pattern, r, 2, in_a, out, in_b)) / 2
    in_a.copy_(cuda.randint(-50, 51, (n, n), device="cuda"))
    about_zero = min(kg.run(pattern, r, 8, in_a, in_b, out, depth=4, tall=True).elapsed_s for _ in range(9)) / 8
    assert about_zero <= most * narrow, about_zero / narrow
