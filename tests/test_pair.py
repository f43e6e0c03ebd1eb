"""The pair form of the prefill variant and of the fused launches (csrc/pair.cu), forced onto small problems, against the CPU oracle.

The sizes are those at which it can go wrong: activation rows around its tile heights (steps of 32 up to 256, halves in two CTAs), one to
four stretches of K added up at the end, K that leaves raw blocks and steps incomplete, an odd number of 128-channel halves, channels that
end inside one, tiles shared by many pairs (alone and next to whole waves) or not at all, more tiles than pairs."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import afb_testlib as T
import awesome_fusion_b200 as pkg

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _check(afb, oracle, case, what, rows=None, **kw):
    from test_gpu_parity import check_close
    before = afb.pair_launch_count()
    got, _ = T.run_case(afb, case, variant=pkg.VARIANT_PREFILL, **kw)
    again, _ = T.run_case(afb, case, variant=pkg.VARIANT_PREFILL, **kw)
    assert afb.pair_launch_count() - before == 2, f"{what}: another form took the call"
    assert np.array_equal(got, again), f"{what}: two runs differ"
    assert afb.read_status()[0] == 0
    rows = list(range(case.m)) if rows is None else rows
    check_close(oracle, oracle.gemm(case, threads=8, round_w=bool(case.group), rows=rows), np.ascontiguousarray(got[rows]), what)
    return got


@pytest.fixture
def forced(monkeypatch):
    monkeypatch.setenv("AFB_PAIR", "1")
    return monkeypatch


@pytest.mark.gpu
@pytest.mark.parametrize("share", ["0", "1"])
@pytest.mark.parametrize("m", [1, 32, 33, 65, 129, 160, 225, 256, 257, 385])
@pytest.mark.parametrize("bits,group,n,k", [(8, 0, 264, 64), (8, 0, 1000, 960), (8, 0, 128, 4096), (4, 0, 392, 320), (4, 128, 520, 1152), (4, 256, 264, 2304),
                                            (4, 64, 136, 704), (8, 128, 264, 640), (8, 64, 264, 448)])
def test_rows_and_ragged_k(afb, oracle, forced, m, bits, group, n, k, share):
    forced.setenv("AFB_PAIR_SHARE", share)
    case = T.make_case(m, n, k, bits=bits, group=group, enc=m & 1, seed=m + k, scale_range=(0.005, 0.05))
    _check(afb, oracle, case, f"int{bits} g{group} {m}x{n}x{k} share {share}")


@pytest.mark.gpu
@pytest.mark.parametrize("most", ["64", "96", "128", "192", "224", "256"])
@pytest.mark.parametrize("share", ["0", "1"])
@pytest.mark.parametrize("m,n,k,bits,group", [(300, 10120, 640, 8, 0), (700, 6152, 512, 8, 0), (500, 4104, 1280, 4, 128)])
def test_tile_heights_whole_waves_and_shared_tiles(afb, oracle, forced, m, n, k, bits, group, share, most):
    forced.setenv("AFB_PAIR_ROWS", most)
    forced.setenv("AFB_PAIR_SHARE", share)
    case = T.make_case(m, n, k, bits=bits, group=group, seed=5, scale_range=(0.005, 0.05))
    _check(afb, oracle, case, f"int{bits} g{group} {m}x{n}x{k} rows {most} share {share}", rows=list(range(0, m, 7)))


@pytest.mark.gpu
@pytest.mark.parametrize("share", ["0", "1"])
@pytest.mark.parametrize("m", [40, 200])
@pytest.mark.parametrize("bits,group", [(8, 0), (8, 128), (4, 0), (4, 128), (4, 64)])
def test_zero_points_and_packed_layout(afb, oracle, forced, m, bits, group, share):
    forced.setenv("AFB_PAIR_SHARE", share)
    case = T.make_case(m, 520, 1280, bits=bits, group=group, enc=1, seed=m + bits, zero_points=True, scale_range=(0.005, 0.05))
    got = _check(afb, oracle, case, f"zero-points int{bits} g{group} m{m}")
    assert np.array_equal(got, _check(afb, oracle, oracle.prepack(case), f"packed, zero-points int{bits} g{group} m{m}"))


@pytest.mark.gpu
@pytest.mark.parametrize("scales", [[0.0, 0.03], [2.0 ** -110, 0.02], [17.0, 0.5], [-0.04, 0.04], [2.0 ** -99, 15.9]])
def test_group_scales_at_the_edges_of_the_folding(afb, oracle, forced, scales):
    """Scales that fold into the unpack next to ones that do not, in one warp: 0, below 2^-100, from 16 on, negative."""
    case = T.make_case(70, 264, 1024, bits=4, group=128, seed=9, scale_range=(0.01, 0.02))
    s = T.np_bf16_to_f32(case.scale)
    s[:, ::3], s[:, 1::3] = scales[0], scales[1]
    case.scale = T.np_bf16_rne(s)
    _check(afb, oracle, case, f"scales {scales}")


@pytest.mark.gpu
@pytest.mark.parametrize("share", ["0", "1"])
@pytest.mark.parametrize("m,n,k,gated", [(1, 72, 512, True), (33, 136, 256, True), (257, 264, 1024, True), (300, 2056, 640, True), (70, 264, 320, False), (300, 4104, 512, False), (257, 264, 1024, False), (129, 1000, 960, False)])
def test_fused_epilogue(afb, oracle, forced, m, n, k, gated, share):
    """Bias, SiLU, gate * up and the residual, in place and with padded rows, in whole and in shared tiles."""
    from test_fused import silu
    from test_gpu_parity import check_close
    forced.setenv("AFB_PAIR_SHARE", share)
    rows = 2 * n if gated else n
    case = T.make_case(m, rows, k, seed=m + n, scale_range=(0.002, 0.01))
    rng = np.random.default_rng(11)
    bias = rng.standard_normal(rows).astype(np.float32)
    v = oracle.gemm(case, threads=8) + bias[None, :]
    ldc = n + 24
    before = T.np_bf16_rne(rng.standard_normal((m, ldc), dtype=np.float32))
    want = (silu(v[:, 0::2]) * v[:, 1::2] if gated else silu(v)) + T.np_bf16_to_f32(before[:, :n])
    held = [afb.to_device(x) for x in (case.a, case.b, case.scale, bias, before)]
    d_a, d_b, d_s, d_bias, d_c = held
    try:
        count = afb.pair_launch_count()
        args = afb.make_args(d_c, d_a, d_b, d_s, m, rows, k, ldc=ldc)
        afb.gemm_fused_launch(afb.make_fused_args(args, gated=gated, activation=pkg.ACT_SILU, bias=d_bias, residual=d_c, ld_residual=ldc))
        afb.device_sync()
        got = afb.to_host(d_c, (m, ldc), np.uint16)
        assert afb.pair_launch_count() == count + 1 and afb.read_status()[0] == 0
    finally:
        for p in held:
            afb.free(p)
    check_close(oracle, want, np.ascontiguousarray(got[:, :n]), f"fused gated={gated} {m}x{n}x{k}")
    assert np.array_equal(got[:, n:], before[:, n:])


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k,gated,share", [(33, 136, 512, True, "0"), (300, 264, 896, True, "1"), (200, 520, 640, False, "0"), (200, 520, 640, False, "1")])
@pytest.mark.parametrize("zero_points,packed", [(False, False), (True, True)])
@pytest.mark.parametrize("bits,group", [(8, 0), (4, 0), (4, 128), (4, 64), (8, 128), (8, 64)])
def test_fused_epilogue_of_the_weight_formats(afb, oracle, forced, bits, group, zero_points, packed, m, n, k, gated, share):
    """Fused launches in both steps of k (groups of 64: 64 wide), with group scales folded into the weights, zero-points and pre-packed weights."""
    from test_fused import silu
    from test_gpu_parity import check_close
    forced.setenv("AFB_PAIR_SHARE", share)
    rows = 2 * n if gated else n
    case = T.make_case(m, rows, k, bits=bits, group=group, enc=m & 1, seed=m + bits + group, zero_points=zero_points,
                       scale_range=(0.002, 0.01) if bits == 8 else (0.01, 0.05))
    rng = np.random.default_rng(7)
    bias = rng.standard_normal(rows).astype(np.float32)
    residual = T.np_bf16_rne(rng.standard_normal((m, n), dtype=np.float32))
    v = oracle.gemm(case, threads=8, round_w=bool(group)) + bias[None, :]
    want = (silu(v[:, 0::2]) * v[:, 1::2] if gated else silu(v)) + T.np_bf16_to_f32(residual)
    dc = T.DeviceCase(afb, oracle.prepack(case) if packed else case)
    held = [afb.to_device(bias), afb.to_device(residual), afb.malloc(m * n * 2)]
    try:
        count = afb.pair_launch_count()
        args = dc.args()
        args.ptr_c, args.ldc = held[2], n
        afb.gemm_fused_launch(afb.make_fused_args(args, gated=gated, activation=pkg.ACT_SILU, bias=held[0], residual=held[1], ld_residual=n))
        afb.device_sync()
        got = afb.to_host(held[2], (m, n), np.uint16)
        assert afb.pair_launch_count() == count + 1 and afb.read_status()[0] == 0
    finally:
        dc.close()
        for p in held:
            afb.free(p)
    check_close(oracle, want, got, f"fused int{bits} g{group} zero-points {zero_points} packed {packed} gated {gated} {m}x{n}x{k}")


@pytest.mark.gpu
def test_silu_over_its_range(afb, forced):
    """act(v) * 1 of values from -120 to 120, +-0, infinities and NaN against 64 bits.
    (v below -88.7, where 1 + exp(-v) overflows fp32, gives -0.)"""
    k, m = 64, 64
    v = np.concatenate([np.linspace(-120, 120, 4073), [0.0, -0.0, np.inf, -np.inf, np.nan, 1e-30, -1e-30, 88.72, -88.72, -87.0, 1e30, -1e30]])
    v = T.np_bf16_to_f32(T.np_bf16_rne(np.resize(v, 64 * 64).astype(np.float32))).reshape(64, 64)
    a = np.zeros((m, k), np.float32)
    a[:, :] = v                                   # a[i, j] = v[i, j]; channel 2j of B picks k = j, channel 2j + 1 nothing: up = bias = 1
    q = np.zeros((2 * 64, k), np.int8)
    q[2 * np.arange(64), np.arange(64)] = 1
    finite = np.isfinite(v)
    a[~finite] = 0.0
    bias = np.zeros(128, np.float32)
    bias[1::2] = 1.0
    # infinities and NaN come in through the bias, one at a time, over a row of zeros
    held = [afb.to_device(x) for x in (T.np_bf16_rne(a), q.view(np.uint8), np.ones(128, np.float32), bias)]
    d_c = afb.malloc(m * 64 * 2)
    try:
        args = afb.make_args(d_c, held[0], held[1], held[2], m, 128, k, ldc=64)
        afb.gemm_fused_launch(afb.make_fused_args(args, gated=True, activation=pkg.ACT_SILU, bias=held[3])); afb.device_sync()
        got = T.np_bf16_to_f32(afb.to_host(d_c, (m, 64), np.uint16))
        x = a.astype(np.float64)
        want = np.where(x < -88.7, 0.0, x / (1 + np.exp(-np.maximum(x, -700.0))))
        # 2^-22 from ex2.approx, 2^-23 from rcp.approx, four roundings of 2^-24: below 2^-20 of the value, next to half a unit of bf16, 2^-8
        bad = np.abs(got - want) > np.abs(want) * (2.0 ** -8 + 2.0 ** -20) + 2.0 ** -126
        assert not bad.any(), [(float(p), float(q), float(r)) for p, q, r in zip(x[bad], got[bad], want[bad])][:8]
        for special, result in ((np.inf, np.inf), (-np.inf, np.nan), (np.nan, np.nan)):
            bias[0::2] = special
            b = afb.to_device(bias)
            afb.gemm_fused_launch(afb.make_fused_args(args, gated=True, activation=pkg.ACT_SILU, bias=b)); afb.device_sync()
            out = T.np_bf16_to_f32(afb.to_host(d_c, (m, 64), np.uint16))
            afb.free(b)
            assert np.all(np.isnan(out)) if np.isnan(result) else np.all(out == result), special
    finally:
        for p in held + [d_c]:
            afb.free(p)


@pytest.mark.gpu
def test_shared_tiles_in_captured_graphs_and_on_streams(afb, oracle, forced):
    """A shared launch per stream and per captured graph: workspaces of their own, counters back at zero for the next replay."""
    import torch
    from test_gpu_parity import check_close
    forced.setenv("AFB_PAIR_SHARE", "1")
    case = T.make_case(150, 1032, 1024, bits=4, group=128, seed=3, scale_range=(0.005, 0.05))
    want = oracle.gemm(case, threads=8, round_w=True)
    dcs = [T.DeviceCase(afb, case) for _ in range(3)]
    streams = [torch.cuda.Stream() for _ in range(2)]
    try:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=streams[0]):
            afb.gemm_launch(dcs[0].args(variant=pkg.VARIANT_PREFILL), torch.cuda.current_stream().cuda_stream)
        for _ in range(3):
            graph.replay()
            for dc, s in zip(dcs[1:], streams):
                afb.gemm_launch(dc.args(variant=pkg.VARIANT_PREFILL), s.cuda_stream)
        torch.cuda.synchronize()
        for dc in dcs:
            check_close(oracle, want, dc.result()[0], "captured and on streams")
    finally:
        for dc in dcs:
            dc.close()


@pytest.mark.gpu
def test_variables_and_flags_that_ask_for_another_form(afb, monkeypatch):
    case = T.make_case(256, 8192, 1024, bits=4, group=128, seed=1)

    def paired(**kw):
        before = afb.pair_launch_count()
        T.run_case(afb, case, **kw)
        return afb.pair_launch_count() - before
    assert paired() == 1 and paired(variant=pkg.VARIANT_PREFILL) == 1
    for flags in (pkg.FLAG_PREFILL_TMEM_A, pkg.FLAG_PREFILL_SMEM_B, pkg.FLAG_GROUP_EXACT):
        assert paired(flags=flags) == 0, flags
    assert paired(c_f32=True) == 0
    for name, value in (("AFB_PAIR", "0"), ("AFB_STREAM", "0"), ("AFB_STREAM", "1"), ("AFB_PREFILL_TILE_STORE", "0"), ("AFB_PREFILL_SPLIT_TAIL", "0")):
        monkeypatch.setenv(name, value)
        assert paired() == 0, name
        monkeypatch.delenv(name)


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k,bits,group,form", [
    # up to 64 rows, all tiles shared
    (64, 28672, 8192, 8, 0, "stream"), (65, 12288, 4096, 8, 0, "pair"), (128, 8192, 8192, 8, 0, "stream"), (333, 4096, 11008, 8, 0, "other"),
    # against the streaming form: the share of this form's time that is steps; few rows of int8 in shared tiles
    (128, 22528, 8192, 8, 0, "stream"), (128, 24576, 8192, 8, 0, "pair"), (192, 19200, 8192, 8, 0, "stream"), (160, 20736, 8192, 8, 0, "pair"),
    (65, 19200, 8192, 8, 64, "stream"), (96, 28672, 8192, 8, 0, "stream"), (97, 28672, 8192, 8, 0, "pair"), (128, 14336, 3072, 4, 128, "pair"),
    # short rows
    (512, 1024, 896, 8, 0, "other"), (512, 1024, 1024, 8, 0, "pair"), (512, 4096, 512, 4, 64, "other"), (512, 4096, 768, 4, 64, "pair"),
    (2048, 28672, 512, 8, 0, "other"), (128, 19200, 512, 8, 0, "pair"), (128, 18688, 512, 8, 0, "other"),
    # steps of 64 k
    (256, 8192, 1984, 8, 0, "other"), (256, 8192, 2112, 8, 0, "pair"), (300, 28672, 4160, 8, 0, "stream"), (300, 8192, 4160, 8, 0, "pair"),
    (128, 8192, 2112, 8, 0, "other"), (128, 19200, 2112, 8, 0, "pair"), (128, 28672, 2048, 4, 64, "other"), (128, 11008, 2048, 4, 64, "pair"),
    (65, 4096, 2048, 4, 64, "other"), (300, 28672, 4096, 4, 64, "stream"), (300, 8192, 4096, 4, 64, "pair"),
    # few rows and few channels, 256 rows
    (65, 1024, 3072, 4, 0, "other"), (65, 1024, 2048, 4, 0, "pair"), (256, 11008, 1536, 8, 0, "other"), (192, 11008, 1536, 8, 0, "pair"), (256, 19200, 8192, 8, 0, "other"),
    # one or two waves of the 256-row form, nearly full or not
    (2048, 4096, 1024, 8, 0, "other"), (512, 14336, 1024, 8, 0, "other"), (1280, 5504, 1024, 8, 0, "pair"), (1024, 4096, 1024, 8, 0, "other"), (1024, 4096, 1024, 4, 128, "other"),
    (512, 4096, 1024, 8, 0, "pair"), (128, 14336, 1024, 4, 0, "other"), (128, 8192, 1024, 4, 0, "pair"), (400, 7168, 1536, 8, 0, "other"),
    (384, 7168, 1536, 8, 0, "pair"), (450, 7168, 2048, 8, 0, "other"), (777, 4096, 2048, 8, 0, "pair"), (777, 4096, 2112, 8, 0, "other"),
    (640, 4096, 2112, 8, 0, "pair"), (1024, 4096, 4096, 8, 0, "other"), (777, 4096, 4096, 8, 0, "pair"), (256, 14336, 2048, 8, 0, "other"),
    (1024, 4096, 4096, 4, 128, "pair")])
def test_choice_of_the_form(afb, m, n, k, bits, group, form):
    """On both sides of each line of the automatic choice (148 SMs)."""
    streamed, paired = afb.stream_launch_count(), afb.pair_launch_count()
    args, held = _zero_args(afb, m, n, k, bits, group)
    afb.gemm_launch(args)
    afb.device_sync()
    for p in held:
        afb.free(p)
    assert (afb.stream_launch_count() - streamed, afb.pair_launch_count() - paired) == {"stream": (1, 0), "pair": (0, 1), "other": (0, 0)}[form]


def _zero_args(afb, m, n, k, bits, group, n_out=None):
    sizes = (m * k * 2, n * k * bits // 8, n * (k // group if group else 1) * 4, m * n * 2)
    held = [afb.malloc(size) for size in sizes]
    for p, size in zip(held, sizes):
        afb.memset(p, 0, size)
    a, b, s, c = held
    return afb.make_args(c, a, b, s, m, n, k, ldc=n_out, bits=bits, group=group, scale_dtype=pkg.SCALE_BF16 if group else pkg.SCALE_F32), held


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k,bits,group,gated,paired", [
    (64, 2048, 2048, 8, 0, True, 0), (65, 2048, 2048, 8, 0, True, 1), (64, 2048, 2048, 4, 128, True, 1), (8, 2048, 2048, 8, 64, True, 1), (1, 11008, 4096, 8, 0, True, 1),
    (1, 2048, 4096, 8, 0, False, 0), (1, 4096, 4096, 8, 0, False, 1), (128, 4096, 4160, 8, 0, True, 0), (129, 4096, 4160, 8, 0, True, 1),
    (128, 5504, 2112, 8, 0, True, 1), (128, 4096, 1984, 8, 0, True, 1), (128, 4096, 4160, 8, 0, False, 1), (256, 512, 512, 8, 32, True, 0)])
def test_choice_of_the_fused_form(afb, m, n, k, bits, group, gated, paired):
    """The same for fused launches: this form or the tensor-memory form."""
    before = afb.pair_launch_count()
    args, held = _zero_args(afb, m, 2 * n if gated else n, k, bits, group, n)
    afb.gemm_fused_launch(afb.make_fused_args(args, gated=gated, activation=pkg.ACT_SILU))
    afb.device_sync()
    for p in held:
        afb.free(p)
    assert afb.pair_launch_count() - before == paired


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k", [(512, 2048, 4096), (256, 8192, 8192), (120, 11008, 4096)])
def test_stretches_of_k_do_not_drift(afb, monkeypatch, m, n, k):
    """One tile per pair: K is added up in two (up to 128 rows per tile) or four (up to 64) accumulators, where the other forms cut it, too.
    The tensor cores cut off what an addition shifts out, so sums of one sign come out low, the more the longer one accumulator adds: by
    no more than in the other forms (the rounding to bf16 has a mean of zero: 2^-9 / sqrt(12) over the root of 10^6 results, 6e-7)."""
    case = T.make_case(m, n, k, seed=m)
    a, q = np.abs(T.np_bf16_to_f32(case.a)), np.abs(case.q)
    case.a, case.b = T.np_bf16_rne(a), q.view(np.uint8)
    exact = (a @ q.T.astype(np.float32)).astype(np.float64) if n * k > 3e7 else a.astype(np.float64) @ q.T.astype(np.float64)
    exact *= case.scale.astype(np.float64)
    off = []
    for pair in ("1", "0"):
        monkeypatch.setenv("AFB_PAIR", pair)
        before = afb.pair_launch_count()
        got, _ = T.run_case(afb, case, variant=pkg.VARIANT_PREFILL)
        assert afb.pair_launch_count() - before == int(pair)
        off.append(abs(((T.np_bf16_to_f32(got) - exact) / exact).mean()))
    assert off[0] < off[1] + 6e-7, off


@pytest.fixture(scope="module")
def shim(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("deal") / "libdeal.so")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-I" + os.path.join(ROOT, "awesome_fusion_b200", "csrc"),
                           "-o", out, os.path.join(ROOT, "tests", "stream_deal_shim.cc")])
    lib = ctypes.CDLL(out)
    lib.check_pair_range.argtypes = [ctypes.c_uint32] * 3 + [ctypes.POINTER(ctypes.c_uint32)]
    return lib


@pytest.mark.parametrize("pairs,tiles,blocks", [(74, 460, 17), (66, 210, 9), (3, 40, 12)])
def test_dealing_over_pairs(shim, pairs, tiles, blocks):
    """The tiles that do not fill whole waves shared, however few, and all tiles whole with a short last wave."""
    where = (ctypes.c_uint32 * 2)()
    rc = shim.check_pair_range(tiles, blocks, pairs, where)
    assert rc == 0, f"rule {rc} broken at {where[0]} tiles of {where[1]} blocks on {pairs} pairs"
