"""Runs beside other streams' work: a call waits for its own kernels only, and another thread's stream
capture goes on through it."""
import threading

import pytest

import kernels_gb300 as kg

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def calls(cuda):
    """The synchronous calls, each made once so that their buffers exist."""
    in_a, in_b, out = kg.alloc(256)
    kg.init(in_a, out)
    batch = kg.Batch([(kg.STAR, 2, in_a, in_b, out)])
    stream = cuda.cuda.Stream()
    host = [cuda.zeros((256, 256), dtype=cuda.float64) for _ in range(3)]

    def batch_run():
        with cuda.cuda.stream(stream):
            batch.run(4)

    c = {"batch": batch_run, "host": lambda: kg.run_host(kg.STAR, 2, 4, *host), "status": kg.status,
         "run": lambda: kg.run(kg.STAR, 2, 4, in_a, in_b, out, stream=stream),
         "norm": lambda: kg.norm(2, out, stream=stream)}
    for f in c.values():
        f()
    cuda.cuda.synchronize()
    return c


@pytest.mark.parametrize("name", ["batch", "host", "status", "run", "norm"])
@pytest.mark.parametrize("mode", ["thread_local", "relaxed"])
def test_beside_a_capture(cuda, calls, name, mode):
    started, done, result = threading.Event(), threading.Event(), {}

    def capture():
        try:
            x, st = cuda.zeros(16, device="cuda"), cuda.cuda.Stream()
            cuda.cuda.synchronize()
            g = cuda.cuda.CUDAGraph()
            with cuda.cuda.graph(g, stream=st, capture_error_mode=mode):
                x.add_(1)
                started.set()
                done.wait(60)
                x.add_(1)
            g.replay()
            cuda.cuda.synchronize()
            result["x"] = float(x[0])
        except Exception as e:  # reported by the assertion below
            result["x"] = e
        started.set()

    th = threading.Thread(target=capture)
    th.start()
    try:
        assert started.wait(60)
        calls[name]()
    finally:
        done.set()
        th.join()
    assert result["x"] == 2.0


@pytest.mark.parametrize("name", ["batch", "host", "run", "norm"])
def test_beside_a_busy_stream(cuda, calls, name):
    other, end = cuda.cuda.Stream(), cuda.cuda.Event()
    cuda.cuda.synchronize()
    with cuda.cuda.stream(other):
        cuda.cuda._sleep(2 * 10 ** 9)  # about a second
        end.record()
    calls[name]()
    busy = not end.query()
    cuda.cuda.synchronize()
    assert busy
