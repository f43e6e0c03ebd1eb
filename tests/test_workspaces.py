"""Workspaces of GEMMs that split K between CTAs: who shares one, first launches on new streams, captures, graphs."""
import ctypes
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
