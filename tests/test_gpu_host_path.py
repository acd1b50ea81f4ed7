"""The host path of QuantizedLinear (csrc/native.cpp): threads, CUDA graphs, the buffers it keeps per stream."""
import threading
import time

import pytest
import torch

from tilus_b200 import QuantizedLinear, _lib, float16, ops
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


def test_decode_calls_of_two_threads_do_not_overtake_each_other():
    """A fetching decode call starts before the kernel in front of it has ended only if that kernel has let go of the
    staging buffer; whose thread queued it does not matter.  One thread's calls fetch (pinned in and out), the
    other's do not (pageable result)."""
    k, n = 8192, 4096
    layer = _layer(n, k)
    cases = []
    for i, m in enumerate((2, 12)):
        x = _rows(m, k, 20 + i).pin_memory()
        outs = [torch.zeros(m, n, dtype=torch.float16) for _ in range(8)]
        cases.append((x, [o.pin_memory() for o in outs] if i == 0 else outs, layer(x.cuda()).cpu()))
    torch.cuda.synchronize()
    start = threading.Barrier(2)

    def work(x, outs):
        start.wait()
        for _ in range(25):
            for o in outs:
                layer.forward_host(x, o)

    threads = [threading.Thread(target=work, args=c[:2]) for c in cases]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    for x, outs, want in cases:
        for o in outs:
            assert _close(o, want)


def test_a_capture_between_two_eager_host_calls_leaves_their_order_alone():
    """What a graph captured has not run: the next eager call still waits for the one before the capture."""
    k, n = 8192, 4096
    layer = _layer(n, k)
    slow, fast = _rows(12, k, 1).pin_memory(), _rows(2, k, 2).pin_memory()
    wide = torch.zeros(12, n + 4, dtype=torch.float16).pin_memory()  # rows not 16 bytes apart: not written directly
    out_slow, out_fast = wide[:, :n], torch.zeros(2, n, dtype=torch.float16).pin_memory()
    want_slow, want_fast = layer(slow.cuda()).cpu(), layer(fast.cuda()).cpu()
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        layer.forward_host(slow, out_slow)
        layer.forward_host(fast, out_fast)
        stream.synchronize()
        for _ in range(5):
            graph = torch.cuda.CUDAGraph()
            out_slow.zero_()
            out_fast.zero_()
            torch.cuda._sleep(2_000_000)
            layer.forward_host(slow, out_slow)
            graph.capture_begin(capture_error_mode="thread_local")  # (torch.cuda.graph would synchronise first)
            layer.forward_host(fast, out_fast)
            graph.capture_end()
            layer.forward_host(fast, out_fast)
            stream.synchronize()
            assert _close(out_slow, want_slow) and _close(out_fast, want_fast)


def _fill_free_memory(stream, sizes):
    """Tensors that take over whatever blocks of these sizes the allocator has free for the stream."""
    with torch.cuda.stream(stream):
        return [torch.full((s,), 77, dtype=torch.uint8, device="cuda") for s in sizes for _ in range(4)]


def test_replay_after_larger_calls_on_the_stream():
    """A captured graph keeps the workspace and the staging buffers that it names, whatever larger calls come after
    it: its results stay right and other tensors stay untouched."""
    k, n = 2048, 8192
    layer = _layer(n, k)
    host_in, host_out = _rows(2, k, 1).pin_memory(), torch.zeros(2, n, dtype=torch.float16).pin_memory()
    mid_in, mid_out = _rows(40, k, 2).pin_memory(), torch.zeros(40, n, dtype=torch.float16)
    dev_in = _rows(100, k, 3).cuda()
    want = [layer(host_in.cuda()).cpu(), layer(mid_in.cuda()).cpu(), layer(dev_in).cpu()]
    mid_pinned = mid_out.pin_memory()
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):

        def calls():
            layer.forward_host(host_in, host_out)
            layer.forward_host(mid_in, mid_pinned)
            return layer(dev_in)

        calls()  # warm-up on the capture stream
        stream.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            dev_out = calls()
        # larger calls of every kind, then tensors in whatever became free
        wide = _layer(4 * n, k, seed=9)
        for m in (16, 128, 1000):
            wide.forward_host(_rows(m, k, m).pin_memory(), torch.zeros(m, 4 * n, dtype=torch.float16).pin_memory())
            wide(_rows(m, k, m).cuda())
        stream.synchronize()
        others = _fill_free_memory(stream, [1 << e for e in range(12, 24)] + [2 * k * 2, 40 * k * 2, 2 * n * 2, 40 * n * 2])
        for _ in range(2):
            host_out.zero_()
            mid_pinned.zero_()
            graph.replay()
            stream.synchronize()
            for got, ref in zip((host_out, mid_pinned, dev_out), want):
                assert _close(got, ref)
        assert all(bool((t == 77).all()) for t in others)


def test_alternating_shapes_settle_on_one_pair_of_staging_buffers():
    """Layers with long rows in and short rows out, and the other way round, in turn: after the first round the
    calls allocate nothing."""
    a, b = _layer(4096, 1024), _layer(1024, 4096)
    cases = [(lay, _rows(m, lay.in_features, 1).pin_memory(), torch.zeros(m, lay.out_features, dtype=torch.float16).pin_memory())
             for m in (4, 64) for lay in (a, b)]
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        for _ in range(2):
            for lay, x, out in cases:
                lay.forward_host(x, out)
        before = torch.cuda.memory_stats()["allocation.all.allocated"]
        for _ in range(5):
            for lay, x, out in cases:
                lay.forward_host(x, out)
        assert torch.cuda.memory_stats()["allocation.all.allocated"] == before
        stream.synchronize()
        for lay, x, out in cases:
            assert _close(out, lay(x.cuda()))


@pytest.mark.parametrize("call", ["forward", "forward_host"])
def test_first_call_of_a_stream_inside_a_capture(call):
    """No call has been made on the stream before it is captured, twice: each graph finds a cleared workspace whichever
    is replayed first, and so does an eager call before any replay.  100 rows share column tiles between CTAs, 2 rows
    with 272 columns do so in the stream kernel."""
    k = 2048
    shapes = [(100, 4112), (2, 272)]
    layers = [_layer(n, k, seed=n) for _, n in shapes]
    xs = [_rows(m, k, m) for m, _ in shapes]
    want = [lay(x.cuda()).cpu() for lay, x in zip(layers, xs)]  # (also loads the kernels)
    if call == "forward_host":
        for lay, x in zip(layers, xs):
            lay.forward_host(x.pin_memory())
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()
    dirty = _fill_free_memory(stream, [1 << 20, 1 << 21, 1 << 22])
    del dirty  # what the allocator hands out next for this stream is not zero
    ins = [x.pin_memory() if call == "forward_host" else x.cuda() for x in xs]
    outs = [torch.zeros(w.shape, dtype=w.dtype).pin_memory() for w in want]
    with torch.cuda.stream(stream):

        def calls():
            if call == "forward_host":
                return [lay.forward_host(x, o) for lay, x, o in zip(layers, ins, outs)]
            return [lay(x) for lay, x in zip(layers, ins)]

        graphs, results = [], []
        for _ in range(2):
            graphs.append(torch.cuda.CUDAGraph())
            with torch.cuda.graph(graphs[-1], stream=stream):
                results.append(calls())
        eager = calls()
        stream.synchronize()
        assert all(_close(g, w) for g, w in zip(eager, want))
        for i in (1, 0, 1):
            for r in results[i]:
                r.zero_()
            graphs[i].replay()
            stream.synchronize()
            assert all(_close(g, w) for g, w in zip(results[i], want)), i


def test_gate_up_inputs_of_any_shape():
    """The gate_up call takes rows however they are shaped (heads not merged, a wider matrix's first columns) and says
    no to rows that are too short."""
    k, n, m = 1024, 512, 6
    layer = _layer(n, k)
    x = _rows(m, k, 1).cuda()
    out, sf, gate_up = layer.forward_swiglu_cast(x)
    want = layer(x)
    wide = torch.cat([x, torch.ones(m, 64, dtype=torch.float16, device="cuda")], dim=1)
    for other in (x.view(m, 8, k // 8), x.view(2, m // 2, k), x.view(-1), wide):
        o, s, g = layer.forward_swiglu_cast(other)
        assert torch.equal(g, gate_up) and torch.equal(s, sf) and torch.equal(o.view(torch.uint8), out.view(torch.uint8))
    assert _close(gate_up, want)
    for bad in (x[:, : k // 2], x[:, : k // 2].contiguous(), x[0, :7]):
        with pytest.raises(ValueError):
            layer.forward_swiglu_cast(bad)


def test_first_launches_from_several_threads():
    """Threads that launch the same kernel for the first time with different amounts of shared memory (rows 17 .. 128 of
    one weight type no other test here uses)."""
    k, n = 1024, 384
    layer = _layer(n, k, dt=D.float5_e3m1)
    w = layer.dequantized_weight().float()
    xs = [_rows(m, k, m).cuda() for m in (17, 40, 64, 100, 128, 33, 80, 112)]
    torch.cuda.synchronize()
    start, outs = threading.Barrier(len(xs)), [None] * len(xs)

    def work(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            start.wait()
            outs[i] = layer(xs[i])
            torch.cuda.current_stream().synchronize()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(xs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for x, out in zip(xs, outs):
        assert out is not None and _close(out, x.float() @ w)


class _HostCalls:
    """A series of host calls through the C ABI: weights of several layers, pinned rows and results of each call."""

    def __init__(self, m, n, k, dt, layers, calls):
        gen = torch.Generator(device="cuda").manual_seed(n + m)
        self.m, self.n, self.k, self.dt, self.zp = m, n, k, dt, 1 << (dt.nbits - 1) if dt.kind == D.KIND_UINT else 0
        self.weights = [(torch.randint(0, 256, (n * k * dt.nbits // 8,), dtype=torch.uint8, device="cuda", generator=gen),
                         (torch.rand(k // 128, n, device="cuda", generator=gen) * 0.01 + 0.005).half()) for _ in range(layers)]
        self.xs = [_rows(m, k, i).pin_memory() for i in range(calls)]
        self.outs = [torch.zeros(m, n, dtype=torch.float16).pin_memory() for _ in range(calls)]
        self.staging = torch.zeros(m * (n + k), dtype=torch.float16, device="cuda")
        self.ws = torch.zeros(ops.workspace_bytes(16, n, k, dt, self.zp, 128), dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()

    def run(self):
        lib, stream = _lib.load(), torch.cuda.current_stream().cuda_stream
        for i, (x, out) in enumerate(zip(self.xs, self.outs)):
            bq, sc = self.weights[i % len(self.weights)]
            _lib.check(lib.b200q_gemm_host(x.data_ptr(), self.k, bq.data_ptr(), sc.data_ptr(), out.data_ptr(), self.n, self.m,
                                           self.n, self.k, self.dt.code, self.zp, 128, _lib.ACT_F16, self.staging.data_ptr(),
                                           self.staging.data_ptr() + 2 * self.m * self.k, self.ws.data_ptr(), self.ws.numel(),
                                           stream))

    def check(self):
        torch.cuda.synchronize()
        for i, (x, out) in enumerate(zip(self.xs, self.outs)):
            w = ops.dequantize(*self.weights[i % len(self.weights)], self.dt, 128, self.zp).float()
            assert _close(out, x.cuda().float() @ w), i
        assert int(self.ws.count_nonzero()) == 0


@pytest.mark.parametrize("m,n,k", [(1, 28672, 1024), (4, 11008, 2048), (2, 17216, 1024), (1, 5120, 5120)])
def test_chained_host_calls_whose_last_cta_owns_fewer_column_tiles(m, n, k):
    calls = _HostCalls(m, n, k, D.uint4b, 3, 18)
    for _ in range(3):
        calls.run()
    calls.check()


@pytest.mark.parametrize("m,n,other", [(1, 28672, 28704), (9, 32768, 28672)])
def test_host_calls_are_as_fast_as_those_of_a_similar_width(m, n, other):
    """One row: 28672 columns leave the last CTA fewer column tiles than 28704 do; nothing is left over in either, so both fetch
    their rows under the call before (13 us a call; 18 without).  Nine rows: 32768 columns on 128 CTAs (27 us, 28672 columns
    25; 36 on 147 CTAs, whose warps end inside column tiles)."""
    chains = [_HostCalls(m, width, 4096, D.uint4b, 4, 40) for width in (n, other)]
    best = [1e9, 1e9]
    for _ in range(6):
        for i, chain in enumerate(chains):
            chain.run()
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            chain.run()
            e1.record()
            torch.cuda.synchronize()
            best[i] = min(best[i], e0.elapsed_time(e1))
    assert best[0] <= 1.25 * best[1], best


@pytest.mark.parametrize("m,n,k,dt", [(4, 48, 14336, D.uint4b), (6, 32, 8192, D.uint4b), (5, 64, 13312, D.int3b), (1, 16, 20480, D.uint2b),
                                      (2, 16, 6144, D.uint2b), (8, 16, 512, D.int8), (16, 16, 7680, D.int8)], ids=str)
def test_narrow_layers_with_more_activations_than_their_ctas_fetch(m, n, k, dt):
    """Calls whose launch has too few CTAs to fetch the rows, and calls that have enough in between: a kernel of its own brings
    them."""
    calls = [_HostCalls(m, n, k, dt, 2, 6), _HostCalls(1, 256, 1024, D.uint4b, 2, 6)]
    for _ in range(2):
        for c in calls:
            c.run()
    for c in calls:
        c.check()


@pytest.mark.parametrize("m,n,k,dt", [(1, 16, 20480, D.uint2b), (4, 48, 14336, D.uint4b), (6, 64, 12288, D.int8), (2, 16, 6144, D.uint2b)], ids=str)
def test_rows_that_replace_others_at_the_same_address(m, n, k, dt):
    """Long chains of short calls, each on rows that a small kernel has just written over those of the call before: many launches are
    on the SMs by then, and none may see a line of the rows that were there."""
    calls = _HostCalls(m, n, k, dt, 2, 24)
    want = [x.cuda().float() @ ops.dequantize(*calls.weights[i % 2], dt, 128, calls.zp).float() for i, x in enumerate(calls.xs)]
    for _ in range(12):
        for _ in range(4):
            calls.run()
        torch.cuda.synchronize()
        assert [i for i, out in enumerate(calls.outs) if not _close(out, want[i])] == []
