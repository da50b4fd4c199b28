"""in += 1 (kg.add) at every offset from a 16-byte boundary, with fewer elements than a vector, whole
vectors with remainders and more vectors than one trip of the grid: every element the rounded sum."""
import pytest

import kernels_gb300 as kg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 31, 64, 65, 201, 1700, 2305])
@pytest.mark.parametrize("shift", [0, 1, 2, 3])
@pytest.mark.parametrize("dtype", [kg.FP64, kg.FP32C])
def test_add_every_element(cuda, n, shift, dtype):
    tdt = cuda.float64 if dtype == kg.FP64 else cuda.float32
    cuda.manual_seed(n + shift)
    flat = cuda.rand(n * n + 8, dtype=tdt, device="cuda") * 64.0 - 32.0
    flat[::3] = cuda.floor(flat[::3])
    want = flat.clone()
    want[shift:shift + n * n] += 1.0
    kg.add(flat[shift:shift + n * n].view(n, n))
    assert cuda.equal(flat, want)
