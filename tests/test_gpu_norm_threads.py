"""Norms of several threads at the same time, each on a stream of its own and over a field of its own:
every one gets its own field's value, whole grids and row slabs alike, with more threads than the library
has places for partial sums."""
import threading

import pytest

import kernels_gb300 as kg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads,n,calls", [(4, 2000, 300), (4, 300, 300), (80, 500, 20)])
@pytest.mark.parametrize("dtype", [kg.FP64, kg.FP32C])
def test_concurrent_norms(cuda, threads, n, calls, dtype):
    r = 2
    tdt = cuda.float64 if dtype == kg.FP64 else cuda.float32
    shape = (n, n) if dtype == kg.FP64 else (n, n, 2)
    outs = [cuda.full(shape, float(k + 1), dtype=tdt, device="cuda") for k in range(threads)]
    inner = n - 2 * r
    want = [(k + 1.0) * (1 if dtype == kg.FP64 else 2) for k in range(threads)]
    cuda.cuda.synchronize()
    wrong, start = [], threading.Barrier(threads)

    def work(k):
        try:
            s = cuda.cuda.Stream()
            start.wait()
            for _ in range(calls):
                got = kg.norm(r, outs[k], stream=s)
                slab = kg.slab_norm(r, n, 0, n, outs[k], stream=s) / inner ** 2
                if abs(got - want[k]) > 1e-12 * want[k] or abs(slab - want[k]) > 1e-12 * want[k]:
                    wrong.append((k, got, slab))
        except Exception as e:  # reported by the assertion below
            wrong.append((k, e))

    ts = [threading.Thread(target=work, args=(k,)) for k in range(threads)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not wrong, wrong[:4]
