"""The host path of QuantizedLinear (csrc/native.cpp): threads, CUDA graphs, the buffers it keeps per stream."""
import threading
import time

import pytest
import torch

from tilus_b200 import QuantizedLinear, float16
from tilus_b200 import dtypes as D

pytestmark = pytest.mark.gpu


def _layer(n, k, seed=0, dt=D.int4b):
    layer = QuantizedLinear(float16, dt, 128, k, n).cuda()
    layer.load_and_quantize(torch.randn(n, k, generator=torch.Generator().manual_seed(seed)))
    return layer


def _rows(m, k, seed):
    return torch.randn(m, k, generator=torch.Generator().manual_seed(seed)).half()


def _close(got, want):
    return float((got.float().cpu() - want.float().cpu()).abs().max()) <= 2e-3 * float(want.float().abs().max())


def test_other_threads_run_while_a_host_call_waits_for_the_gpu():
    """A result in pageable memory is copied by a call that waits for everything queued before it (here 0.3 s of
    idling on the GPU): the other threads of the process go on meanwhile."""
    layer = _layer(512, 1024)
    x, out = _rows(40, 1024, 1), torch.zeros(40, 512, dtype=torch.float16)  # pageable
    layer.forward_host(x, out)
    torch.cuda.synchronize()
    want = out.clone()
    ticks, stop = [], threading.Event()

    def tick():
        while not stop.is_set():
            ticks.append(time.perf_counter())
            time.sleep(0.001)

    worker = threading.Thread(target=tick)
    worker.start()
    try:
        torch.cuda._sleep(int(0.3 * 1.9e9))
        t0 = time.perf_counter()
        layer.forward_host(x, out)
        t1 = time.perf_counter()
    finally:
        stop.set()
        worker.join()
    torch.cuda.synchronize()
    assert torch.equal(out, want)
    assert t1 - t0 > 0.1  # the call did wait
    assert sum(t0 < t < t1 for t in ticks) >= 10


def test_host_calls_of_several_threads_on_one_stream():
    """Threads that share a stream share its staging buffers; every call gets its own rows' results."""
    k, n = 1024, 512
    layer = _layer(n, k)
    cases = []
    for i, m in enumerate((1, 5, 40, 100)):
        x = _rows(m, k, 10 + i)
        x = x.pin_memory() if i % 2 else x
        out = torch.zeros(m, n, dtype=torch.float16)
        cases.append((x, out.pin_memory() if i != 1 else out, layer(x.cuda()).cpu()))
    torch.cuda.synchronize()

    def work(x, out):
        for _ in range(50):
            layer.forward_host(x, out)

    threads = [threading.Thread(target=work, args=c[:2]) for c in cases]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    for x, out, want in cases:
        assert _close(out, want)
