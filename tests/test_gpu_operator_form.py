"""The operator form (out += S(in), no in_next: starR/gridR and kg.apply without in_next) on the tile
kernels: FP64 bit for bit the strict-order oracle on whole-number and real fields, FP32C within the
error of its sums of the same FP32 differences, at the edges of tiles, on odd orders and off a
16-byte boundary; `in` and the frame of `out` untouched; the first call of a process inside a stream
capture."""
import subprocess
import sys

import numpy as np
import pytest

import kernels_gb300 as kg
from oracle import prk_oracle as po

pytestmark = pytest.mark.gpu

ALL = [(p, r) for p in (kg.STAR, kg.GRID) for r in range(1, 6)]


def field(n, kind, seed=5):
    rng = np.random.default_rng(seed)
    if kind == "prk":
        ii, jj = np.meshgrid(np.arange(n), np.arange(n), indexing="ij")
        return (ii + jj + 3.0), np.full((n, n), 6.0)
    if kind == "mixed":  # the left third whole numbers, the rest real: neighbouring tiles take different routes
        a = rng.uniform(-100.0, 100.0, (n, n))
        a[:, :n // 3] = np.floor(a[:, :n // 3]) + 0.0
        return a, rng.uniform(-1.0, 1.0, (n, n))
    return rng.uniform(-1.0, 1.0, (n, n)), rng.uniform(-1.0, 1.0, (n, n))


def device(torch, host, shift):
    """A device copy of `host` starting `shift` elements past a 16-byte boundary."""
    flat = torch.empty(host.size + shift, dtype=torch.from_numpy(host).dtype, device="cuda")
    view = flat[shift:].view(*host.shape)
    view.copy_(torch.from_numpy(host))
    return view


@pytest.mark.parametrize("pattern,r", ALL)
@pytest.mark.parametrize("kind", ["prk", "mixed", "real"])
@pytest.mark.parametrize("n,shift", [(11, 0), (16, 0), (63, 0), (64, 0), (66, 1), (97, 0), (200, 0), (333, 1)])
def test_fp64_bit_exact(cuda, pattern, r, kind, n, shift):
    in_h, out_h = field(n, kind)
    in_d, out_d = device(cuda, in_h, shift), device(cuda, out_h, shift)
    kg.apply(pattern, r, in_d, out_d)
    po.apply(pattern, r, in_h, out_h)
    assert np.array_equal(out_d.cpu().numpy().view(np.uint64), out_h.view(np.uint64))
    assert np.array_equal(in_d.cpu().numpy().view(np.uint64), in_h.view(np.uint64))


@pytest.mark.parametrize("pattern,r", ALL)
@pytest.mark.parametrize("kind", ["prk", "real"])
@pytest.mark.parametrize("n,shift", [(11, 0), (64, 0), (129, 0), (132, 2), (260, 0)])
def test_fp32c(cuda, pattern, r, kind, n, shift):
    in_h, hi = field(n, kind)
    in_h = in_h.astype(np.float32)
    out_h = np.zeros((n, n, 2), np.float32)
    out_h[..., 0] = hi
    in_d, out_d = device(cuda, in_h, shift), device(cuda, out_h, shift)
    kg.apply(pattern, r, in_d, out_d)
    got = out_d.cpu().numpy()
    # the sum over the taps' FP32 differences in binary64; the kernel's products (each within 2^-46 of
    # |w d| <= 2, at most 55) and two-float sums stay within 1e-12 of it
    ref = out_h[..., 0].astype(np.float64)
    inner = slice(r, n - r)
    for dc, dr, w in po.taps(pattern, r):
        if w > 0:
            up = in_h[r + dr:n - r + dr, r + dc:n - r + dc]
            dn = in_h[r - dr:n - r - dr, r - dc:n - r - dc]
            ref[inner, inner] += w * (up - dn).astype(np.float64)
    assert np.abs(got[..., 0].astype(np.float64) + got[..., 1] - ref).max() <= 1e-12
    assert np.array_equal(got[:r].view(np.uint32), out_h[:r].view(np.uint32))
    assert np.array_equal(in_d.cpu().numpy(), in_h)


def test_tma_required_still_refuses_the_operator_form(cuda):
    in_a, _, out = kg.alloc(64, kg.FP64)
    kg.init(in_a, out)
    prev = kg.set_kernel(kg.KERNEL_TMA)
    try:
        with pytest.raises(kg.PrkError):
            kg.star2(64, 32, in_a, out)
    finally:
        kg.set_kernel(prev)


FIRST_CALL = """
import torch, kernels_gb300 as kg
n = 200
in_ = torch.arange(n, dtype=torch.float64, device="cuda")[:, None] + torch.arange(n, dtype=torch.float64, device="cuda")
out = torch.zeros((n, n), dtype=torch.float64, device="cuda")
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g):
    kg.star2(n, 32, in_, out)
    kg.add(in_)
for _ in range(3):
    g.replay()
torch.cuda.synchronize()
assert (out[2:-2, 2:-2] == 6.0).all() and float(in_[0, 0]) == 3.0
kg.status()
print("captured")
"""


def test_first_call_inside_a_capture(cuda):
    """A process whose first library call is the operator form inside a graph capture."""
    res = subprocess.run([sys.executable, "-c", FIRST_CALL], capture_output=True, text=True, timeout=300,
                         cwd=str(__import__("pathlib").Path(__file__).resolve().parents[1]))
    assert res.returncode == 0 and "captured" in res.stdout, res.stderr[-2000:]
