"""A context's stream is not ordered with the default stream, so what a context
copies or clears has to go to its own stream: a kernel must not read what a
copy on the default stream may still be filling."""
import os
import re
import threading
import time

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "logo-tsp-solver_gb300", "csrc")


@pytest.mark.parametrize("name", ["capi.cu", "capi_batch.cu", "capi_server.cu"])
def test_no_copy_on_the_default_stream(name):
    """These files launch on non-blocking streams of their own; a copy or clear
    without a stream would be unordered with every launch."""
    text = open(os.path.join(CSRC, name)).read()
    text = re.sub(r"//[^\n]*", "", text)
    assert "cudaStreamNonBlocking" in text
    found = re.findall(r"\b(cudaMemcpy|cudaMemset|cudaMemcpy2D|cudaMemcpyToSymbol)\s*\(", text)
    assert found == []


@pytest.mark.gpu
def test_contexts_made_while_the_default_stream_is_busy(lg, inst, oracle_mod):
    torch = pytest.importorskip("torch")
    stop = threading.Event()

    def keep_busy():
        torch.cuda.set_device(0)
        while not stop.is_set():
            done = torch.cuda.Event()
            for _ in range(4):
                torch.cuda._sleep(1_000_000)  # about half a millisecond each
            done.record()
            while not done.query():
                time.sleep(0.0002)

    t = threading.Thread(target=keep_busy)
    t.start()
    try:
        for k, n in enumerate((40, 500, 3000, 7000)):
            xy = inst.uniform_f32(n, 50 + n, 1.0e4 * 3 ** k)
            r = inst.random_tour(n, 51 + n)
            with lg.Solver(xy) as s:
                assert s.optimize_step(r) == oracle_mod.best_move(xy, r)
                s.set_search(lg.SEARCH_NEIGHBOUR)
                got, _ = s.optimize(r, max_moves=3)
            with lg.Solver(xy) as s:
                s.set_search(lg.SEARCH_NEIGHBOUR)
                assert (got == s.optimize(r, max_moves=3)[0]).all()
    finally:
        stop.set()
        t.join()
