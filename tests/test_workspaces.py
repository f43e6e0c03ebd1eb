"""Workspaces of GEMMs that split K between CTAs: who shares one, first launches on new streams, captures, graphs."""
import ctypes
import gc
import threading

import numpy as np
import pytest

import awesome_fusion_b200 as pkg

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

STREAMING = (40, 8192, 8192)      # 64 tiles on all the SMs: every tile is shared
SLICED = (16, 1024, 8192)         # decode kernel, K-slices


class Gemm:
    """One GEMM on torch buffers, with its result when launched alone."""

    def __init__(self, lib, m, n, k, seed):
        gen = torch.Generator(device="cuda")
        gen.manual_seed(seed)
        self.lib = lib
        self.a = torch.randn((m, k), device="cuda", generator=gen).bfloat16()
        self.b = torch.randint(-127, 128, (n, k), device="cuda", generator=gen, dtype=torch.int8)
        self.s = torch.rand((n,), device="cuda", generator=gen) * 0.01
        self.c = torch.empty((m, n), device="cuda", dtype=torch.bfloat16)
        self.args = lib.make_args(self.c, self.a, self.b, self.s, m, n, k)
        self.launch()
        torch.cuda.synchronize()
        self.want = self.c.clone()
        exact = (self.a.double() @ self.b.double().T) * self.s.double()
        assert ((self.want.double() - exact).norm() / exact.norm()).item() < 4e-3   # one rounding to bf16 is 1.7e-3
        self.clear()

    def launch(self, stream=None):
        self.lib.gemm_launch(self.args, stream if stream is not None else torch.cuda.current_stream().cuda_stream)

    def clear(self):
        self.c.fill_(float("nan"))
        torch.cuda.synchronize()

    def check(self, what):
        torch.cuda.synchronize()
        assert torch.equal(self.c, self.want), what
        self.clear()


def _new_streams(lib, count):
    out = []
    for _ in range(count):
        p = ctypes.c_void_p()
        lib.check(lib.lib.afb_stream_create(ctypes.byref(p)), "afb_stream_create")
        out.append(p.value)
    return out


@pytest.fixture(scope="module", autouse=True)
def _leave_no_streams_behind(afb):
    """These tests use up the workspaces that afb_init allocates; what runs after them finds the library as they did."""
    yield
    gc.collect()
    torch.cuda.synchronize()
    afb.finalize()
    afb.init(0)


def test_first_launches_on_new_streams_while_the_legacy_stream_is_busy(afb):
    """A stream without a workspace gets one on its first launch.  Its arrival counters are at zero when that launch counts on them,
    whatever waits on the legacy stream (nothing orders a non-blocking stream after it)."""
    g = Gemm(afb, *SLICED, seed=1)
    busy = torch.randn((8192, 8192), device="cuda").bfloat16()
    torch.cuda.synchronize()
    for s in _new_streams(afb, 12):   # more than afb_init has workspaces for
        for _ in range(4):
            busy @ busy               # on the legacy stream
        for _ in range(3):
            g.launch(s)
        g.check("first launches on a new stream")


def test_first_launch_on_a_new_stream_leaves_a_capture_elsewhere_alone(afb):
    """While one thread captures (global mode), another one's first launch on a new stream allocates."""
    g = Gemm(afb, *SLICED, seed=2)
    streams = _new_streams(afb, 12)
    graph, done = torch.cuda.CUDAGraph(), []

    def first_launches():
        try:
            for s in streams:
                g.launch(s)
            done.append(True)
        except Exception as e:   # noqa: BLE001 (reported below, outside the capture)
            done.append(e)

    x = torch.zeros(8, device="cuda")
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        x += 1
        t = threading.Thread(target=first_launches)
        t.start()
        t.join()
        x += 1
    assert done == [True], done
    g.check("launched next to a capture")
    graph.replay()
    torch.cuda.synchronize()
    assert x.tolist() == [2.0] * 8


def _captured(g):
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        for _ in range(8):
            g.launch()
    return graph


def test_graphs_of_one_capture_stream_may_run_at_the_same_time(afb):
    """Two graphs captured one after the other (torch captures on one stream) and eager launches on that very stream, all at once: the
    streaming form's partial sums and counters are each one's own."""
    gemms = [Gemm(afb, *STREAMING, seed=3), Gemm(afb, *STREAMING, seed=4), Gemm(afb, *STREAMING, seed=5)]
    graphs = [_captured(g) for g in gemms[:2]]
    sides = [torch.cuda.Stream(), torch.cuda.Stream()]
    capture_stream = torch.cuda.graph.default_capture_stream
    before = afb.stream_launch_count()
    for turn in range(10):
        for graph, side in zip(graphs, sides):
            with torch.cuda.stream(side):
                graph.replay()
        for _ in range(8):
            gemms[2].launch(capture_stream.cuda_stream)
        for i, g in enumerate(gemms):
            g.check(f"turn {turn}, GEMM {i}")
    assert afb.stream_launch_count() - before == 80   # (a graph's launches are counted when it is captured)


def test_streams_at_the_same_time(afb):
    gemms = [Gemm(afb, *STREAMING, seed=6 + i) for i in range(4)]
    streams = _new_streams(afb, 4)
    for turn in range(5):
        for _ in range(6):
            for g, s in zip(gemms, streams):
                g.launch(s)
        for i, g in enumerate(gemms):
            g.check(f"turn {turn}, stream {i}")


def test_a_graphs_workspace_is_given_back(afb):
    """Captured, replayed and destroyed eighty times: the streaming form stays in use.  32 graphs keep their workspaces of 8 MB (and as much
    again for the allocator's pages at most); after them device memory does not grow by more than two of them."""
    g = Gemm(afb, *STREAMING, seed=10)
    start = torch.cuda.mem_get_info()[0]
    for turn in range(80):
        before = afb.stream_launch_count()
        graph = _captured(g)
        assert afb.stream_launch_count() - before == 8
        graph.replay()
        g.check(f"turn {turn}")
        del graph
        gc.collect()
        torch.cuda.synchronize()
        if turn == 40:
            free = torch.cuda.mem_get_info()[0]
    assert free - torch.cuda.mem_get_info()[0] <= 32 << 20 and start - free <= 32 * 16 << 20


def test_first_streaming_launch_next_to_a_capture_and_on_the_per_thread_stream(afb):
    """A first launch on a new stream allocates while another thread captures; the per-thread default stream, one handle for many streams,
    keeps no workspace and takes the form without."""
    g = Gemm(afb, *STREAMING, seed=11)
    streams, graph, failed = _new_streams(afb, 6), torch.cuda.CUDAGraph(), []

    def first_launches():
        try:
            for s in streams:
                g.launch(s)
        except Exception as e:   # noqa: BLE001
            failed.append(e)

    x = torch.zeros(8, device="cuda")
    torch.cuda.synchronize()
    before = afb.stream_launch_count()
    with torch.cuda.graph(graph):
        x += 1
        t = threading.Thread(target=first_launches)
        t.start()
        t.join()
        x += 1
    assert not failed and afb.stream_launch_count() - before == 6
    g.check("launched next to a capture")
    graph.replay()
    torch.cuda.synchronize()
    assert x.tolist() == [2.0] * 8
    g.launch(2)   # cudaStreamPerThread
    torch.cuda.synchronize()
    assert afb.stream_launch_count() - before == 6
    assert ((g.c.float() - g.want.float()).norm() / g.want.float().norm()).item() < 1e-3   # another order of addition: a few roundings


def test_a_stream_takes_one_workspace_for_both_forms(afb, monkeypatch):
    """The streaming form, and the pair form with tiles of 224 and of 256 rows, its highest, share tiles on one stream: its first such launch takes
    a workspace for all of them; the first stream finds the one that afb_init allocated."""
    monkeypatch.setenv("AFB_PAIR_SHARE", "1")
    monkeypatch.setenv("AFB_PAIR_ROWS", "256")
    gemms = {}

    def form_of(rows):
        monkeypatch.setenv("AFB_PAIR", "0" if rows == 40 else "1")

    for rows in (40, 224, 256):
        form_of(rows)
        gemms[rows] = Gemm(afb, rows, 8192, 8192, seed=rows)   # (loads the kernels, too)
    torch.cuda.synchronize()
    afb.finalize()
    afb.init(0)

    def taken(stream, order):
        out = []
        for rows in order:
            form_of(rows)
            streamed, paired, free = afb.stream_launch_count(), afb.pair_launch_count(), torch.cuda.mem_get_info()[0]
            gemms[rows].launch(stream)
            torch.cuda.synchronize()
            out.append(free - torch.cuda.mem_get_info()[0])
            assert (afb.stream_launch_count() - streamed, afb.pair_launch_count() - paired) == ((1, 0) if rows == 40 else (0, 1))
            gemms[rows].check(f"{rows} rows")
        return out

    assert taken(torch.cuda.current_stream().cuda_stream, (40, 224, 256)) == [0, 0, 0]
    first, *later = taken(_new_streams(afb, 1)[0], (40, 224, 256, 224, 40))
    assert 0 < first <= 40 << 20 and later == [0] * 4, (first, later)
