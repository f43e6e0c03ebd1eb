"""The streaming form of the decode and prefill variants (csrc/stream.cu), forced onto small problems, against the CPU oracle.

The sizes are those at which it can go wrong: activation rows around its tile heights (16, 64, 128, 192) and modes (up to 16 rows
group scales multiply fp32 sums, above that the weights), K that leaves raw blocks and steps incomplete, channels that end inside a
tile, fewer units of work than CTAs, tiles shared by many CTAs, whole waves next to shared tiles."""
import numpy as np
import pytest

import afb_testlib as T
import awesome_fusion_b200 as pkg
from test_gpu_parity import check_close

pytestmark = pytest.mark.gpu


def _check(afb, oracle, case, what, **kw):
    before = afb.stream_launch_count()
    got, _ = T.run_case(afb, case, **kw)
    again, _ = T.run_case(afb, case, **kw)
    assert afb.stream_launch_count() - before == 2, f"{what}: another form took the call"
    assert np.array_equal(got, again), f"{what}: two runs differ"
    folded = case.group and case.m > 16   # the weights are rounded to bf16 once more, as in the other prefill forms
    check_close(oracle, oracle.gemm(case, threads=8, round_w=bool(folded)), got, what)
    return got


@pytest.fixture(autouse=True)
def _forced(monkeypatch):
    monkeypatch.setenv("AFB_STREAM", "1")


@pytest.mark.parametrize("m", [1, 16, 17, 33, 64, 65, 128, 129, 192, 193, 385])
@pytest.mark.parametrize("bits,group,n,k", [(8, 0, 264, 64), (8, 0, 1000, 960), (8, 0, 128, 4096), (4, 0, 392, 320), (4, 128, 520, 1152), (4, 256, 264, 2304),
                                            (4, 64, 136, 704), (8, 128, 264, 640), (8, 64, 264, 448)])
def test_rows_and_ragged_k(afb, oracle, m, bits, group, n, k):
    case = T.make_case(m, n, k, bits=bits, group=group, enc=m & 1, seed=m + k, scale_range=(0.005, 0.05))
    _check(afb, oracle, case, f"int{bits} g{group} {m}x{n}x{k}")


@pytest.mark.parametrize("m,n,k,bits,group", [(16, 28672, 1024, 8, 0), (40, 20008, 640, 8, 0), (3, 24000, 1280, 4, 128), (128, 19200, 768, 4, 128),
                                              (700, 6152, 512, 8, 0), (1400, 4104, 512, 4, 128)])
def test_whole_waves_and_shared_tiles(afb, oracle, m, n, k, bits, group):
    case = T.make_case(m, n, k, bits=bits, group=group, seed=5, scale_range=(0.005, 0.05))
    _check(afb, oracle, case, f"int{bits} g{group} {m}x{n}x{k}")


@pytest.mark.parametrize("m", [1, 16])
@pytest.mark.parametrize("bits,group,n,k", [(8, 0, 264, 128), (8, 0, 264, 640), (8, 0, 20008, 1152), (8, 128, 19000, 384), (8, 256, 520, 2816), (4, 0, 392, 640), (4, 0, 300, 8320),
                                            (4, 128, 19000, 640), (4, 512, 264, 2560)])
def test_two_issuing_warps(afb, oracle, m, bits, group, n, k):
    """Up to 16 rows the two parts of a step (128 k each) are issued by two warps: steps that lack the second part, in tiles and in the shares of
    tiles, sums of several parts and sets of sums that are not full."""
    case = T.make_case(m, n, k, bits=bits, group=group, enc=m & 1, seed=m + k, scale_range=(0.005, 0.05))
    _check(afb, oracle, case, f"int{bits} g{group} {m}x{n}x{k}")


@pytest.mark.parametrize("m", [7, 16, 100])
@pytest.mark.parametrize("bits,group", [(8, 0), (8, 128), (4, 0), (4, 128), (4, 64)])
def test_zero_points_and_packed_layout(afb, oracle, m, bits, group):
    case = T.make_case(m, 520, 1280, bits=bits, group=group, enc=1, seed=m + bits, zero_points=True, scale_range=(0.005, 0.05))
    got = _check(afb, oracle, case, f"zero-points int{bits} g{group} m{m}")
    assert np.array_equal(got, _check(afb, oracle, oracle.prepack(case), f"packed, zero-points int{bits} g{group} m{m}"))


@pytest.mark.parametrize("m,ldc", [(9, 269), (16, 268), (1, 265)])
@pytest.mark.parametrize("bits,group", [(8, 0), (4, 128)])
def test_result_rows_that_no_tile_store_takes(afb, oracle, m, ldc, bits, group):
    """Decode calls may have any ldc and any number of channels: register stores, and nothing written outside C."""
    case = T.make_case(m, 261, 2048, bits=bits, group=group, seed=m, scale_range=(0.005, 0.05))
    _check(afb, oracle, case, f"ldc {ldc} int{bits}", ldc=ldc)


def test_bf16_group_scales_in_fp32_and_pdl(afb, oracle):
    for group, dtype, flags in [(128, 0, 0), (0, 1, 0), (128, 1, pkg.FLAG_PDL), (0, 0, pkg.FLAG_PDL)]:
        case = T.make_case(12, 776, 3072, bits=4, group=group, scale_dtype=dtype, seed=3, scale_range=(0.005, 0.05))
        _check(afb, oracle, case, f"scale dtype {dtype} flags {flags}", flags=flags)


@pytest.mark.parametrize("m", [8, 16])
def test_sums_of_few_rows_do_not_drift(afb, m):
    """The tensor cores cut off what an addition shifts out, so a sum over all of K drifts towards zero.  Sums that cancel (the second half
    of K takes back the first, but for 64 weights) show it.  A sum over 1024 k loses at most 64 times half a unit in the last place of
    24 bits, 3.8e-6 of itself and a quarter of that of the half sum, 1e-6; what the first half loses the second gives back.  (One sum
    over all of K: 6e-6.)  The rounding to bf16 has a mean of zero: 1.4e-5 divided by the square root of 229376 results or more."""
    n, k = 28672, 8192
    half = k // 2
    case = T.make_case(m, n, k, seed=m)
    a = np.abs(T.np_bf16_to_f32(case.a))
    a[:, half:] = -a[:, :half]
    a[:, -64:] *= 0.5
    q = np.abs(case.q)
    q[:, half:] = q[:, :half]
    case.a, case.b = T.np_bf16_rne(a), q.view(np.uint8)
    scale = case.scale.astype(np.float64)
    exact = (a.astype(np.float64) @ q.T.astype(np.float64)) * scale
    half_sum = ((a[:, :half].astype(np.float64) @ q[:, :half].T.astype(np.float64)) * scale).mean()
    got, _ = T.run_case(afb, case)
    off = (T.np_bf16_to_f32(got) - exact).mean() / half_sum
    assert abs(off) < 1e-6, off


@pytest.mark.parametrize("m,n,k", [(32, 24576, 512), (24, 25600, 512), (20, 24576, 768), (2048, 19456, 768)])
def test_few_units_next_to_whole_waves(afb, oracle, monkeypatch, m, n, k):
    """Fewer units of shared tiles than CTAs, next to whole waves: every tile is finished, and the arrival counters are back at zero for
    the next launch on the stream (the same, and a decode launch with K-slices).  By the automatic choice and forced."""
    case = T.make_case(m, n, k, bits=4, group=128, seed=m, scale_range=(0.005, 0.05))
    rows = list(range(0, m, 97)) if m > 64 else list(range(m))   # one or two of every row tile
    ref = oracle.gemm(case, threads=8, round_w=True, rows=rows)
    for form in (None, "1", "1"):
        monkeypatch.setenv("AFB_STREAM", form) if form else monkeypatch.delenv("AFB_STREAM")
        got, _ = T.run_case(afb, case)
        check_close(oracle, ref, np.ascontiguousarray(got[rows]), f"{m}x{n}x{k} AFB_STREAM={form}")
    monkeypatch.delenv("AFB_STREAM")
    sliced = T.make_case(16, 1024, 8192, seed=1)
    check_close(oracle, oracle.gemm(sliced, threads=8), T.run_case(afb, sliced)[0], "decode K-slices after it")


def _streamed(afb, m, n, k, **kw):
    before = afb.stream_launch_count()
    T.run_case(afb, T.make_case(m, n, k, seed=1), **kw)
    return afb.stream_launch_count() - before


def test_switches_of_the_other_forms_still_reach_them(afb, monkeypatch):
    """Variables and flags that ask for another form get it, on sizes that the streaming form would take; AFB_STREAM outranks the variables."""
    monkeypatch.delenv("AFB_STREAM")
    few, many = (16, 28672, 8192), (40, 8192, 8192)
    assert _streamed(afb, *few) == 1 and _streamed(afb, *many) == 1
    for name, value in (("AFB_DECODE_BALANCED", "1"), ("AFB_DECODE_WR", "4"), ("AFB_DECODE_SLICES", "2")):
        monkeypatch.setenv(name, value)
        assert _streamed(afb, *few) == 0 and _streamed(afb, *many) == 1, name
        monkeypatch.delenv(name)
    monkeypatch.setenv("AFB_PREFILL_IMPL", "ts")
    assert _streamed(afb, *few) == 1 and _streamed(afb, *many) == 0
    monkeypatch.setenv("AFB_STREAM", "1")
    assert _streamed(afb, *many) == 1
    monkeypatch.setenv("AFB_STREAM", "0")
    assert _streamed(afb, *few) == 0
    monkeypatch.delenv("AFB_STREAM")
    monkeypatch.delenv("AFB_PREFILL_IMPL")
    for flag in (pkg.FLAG_PREFILL_SMEM_B, pkg.FLAG_PREFILL_TMEM_A):
        assert _streamed(afb, *many, flags=flag) == 0


def test_group_sums_are_added_in_two_levels(afb):
    """128 group sums of one sign up to half of K, taken back by the other half: what is left is the error of the fp32 additions.  An addition
    at a magnitude of at most S (the half sum) is off by 2^-24 S / sqrt(3) in the root mean square; magnitudes that rise from 0 to S and fall
    again make that 2^-24 S / 3 times the square root of their number: 1.3 for 16 sums of 8 groups (1.4 with the additions inside
    them), 3.8 for one chain of 128 (2.8 measured).  All tiles are whole ones (148 SMs)."""
    m, n, k, group = 4, 18944, 16384, 128
    half, rng = k // 2, np.random.default_rng(3)
    case = T.make_case(m, 128, k, bits=4, group=group, seed=3, scale_range=(0.005, 0.05))
    a = np.abs(T.np_bf16_to_f32(case.a))
    a[:, half:] = -a[:, :half]
    u = rng.integers(0, 8, size=(n, half), dtype=np.uint8)
    b = u[:, 0::2] | (u[:, 1::2] << np.uint8(4))
    scale = T.np_bf16_rne(rng.uniform(0.005, 0.05, size=(n, half // group)).astype(np.float32))
    case.n, case.a, case.b, case.scale = n, T.np_bf16_rne(a), np.concatenate([b, b], 1), np.concatenate([scale, scale], 1)
    sums = np.stack([a[:, :half].reshape(m, -1, group)[:, i].astype(np.float64) @ u[:, i * group:(i + 1) * group].T.astype(np.float64)
                     for i in range(half // group)])   # [group of k][m][n]
    half_sum = (sums * T.np_bf16_to_f32(scale).T[:, None, :]).sum(0)
    got, _ = T.run_case(afb, case)
    off = np.sqrt(((T.np_bf16_to_f32(got) / half_sum) ** 2).mean()) * 2 ** 24
    assert off < 2, off


@pytest.mark.parametrize("m,n,k,bits,group,form", [
    (3, 28672, 8192, 8, 0, "other"), (4, 28672, 8192, 8, 0, "stream"), (4, 28672, 8192, 4, 128, "other"), (5, 28672, 8192, 4, 128, "stream"), (16, 4096, 4096, 8, 0, "other"),
    (9, 12288, 4096, 8, 0, "stream"), (8, 8192, 8192, 4, 0, "other"), (12, 8192, 8192, 4, 0, "stream"), (8, 4096, 11008, 4, 128, "stream"), (17, 12288, 1024, 4, 128, "other"),
    (40, 16384, 2048, 4, 128, "stream"), (24, 4096, 4096, 4, 0, "stream"), (40, 4096, 4096, 4, 0, "other"), (40, 4096, 4096, 8, 0, "other"), (64, 12288, 4096, 8, 0, "stream"),
    (80, 12288, 4096, 8, 0, "pair"), (128, 8192, 8192, 8, 0, "stream"), (129, 8192, 8192, 8, 0, "stream"), (200, 8192, 8192, 8, 0, "pair"), (129, 12288, 4096, 8, 0, "pair"),
    (333, 11000, 4096, 8, 0, "pair"), (333, 8192, 8192, 8, 0, "pair"), (777, 12288, 4096, 8, 0, "pair"), (777, 12288, 4096, 4, 128, "pair"), (4096, 1024, 11008, 4, 128, "pair"), (40, 28672, 2048, 4, 64, "other"),
    (40, 28672, 2048, 4, 128, "stream"), (777, 12288, 4096, 8, 128, "pair"), (40, 28672, 1024, 4, 128, "other")])
def test_choice_of_the_form(afb, monkeypatch, m, n, k, bits, group, form):
    """On both sides of the lines of the automatic choice (148 SMs): the streaming form, the pair form, or one of the others."""
    monkeypatch.delenv("AFB_STREAM")
    before, paired = afb.stream_launch_count(), afb.pair_launch_count()
    a, b, s, c = (afb.malloc(size) for size in (m * k * 2, n * k * bits // 8, n * (k // group if group else 1) * 4, m * n * 2))
    try:
        for p, size in ((a, m * k * 2), (b, n * k * bits // 8), (s, n * (k // group if group else 1) * 4)):
            afb.memset(p, 0, size)
        afb.gemm_launch(afb.make_args(c, a, b, s, m, n, k, bits=bits, group=group, scale_dtype=pkg.SCALE_BF16 if group else pkg.SCALE_F32))
        afb.device_sync()
    finally:
        for p in (a, b, s, c):
            afb.free(p)
    assert (afb.stream_launch_count() - before, afb.pair_launch_count() - paired) == {"stream": (1, 0), "pair": (0, 1), "other": (0, 0)}[form]


def test_dependent_launches_in_a_chain(afb):
    """GEMMs of a decode loop back to back with AFB_FLAG_PDL, each reading what the one before it wrote, all in the streaming form: eagerly
    and captured, the bits of launches that wait for one another."""
    torch = pytest.importorskip("torch")
    gen = torch.Generator(device="cuda")
    gen.manual_seed(5)
    h, m, layers = 8192, 16, 4
    weights = [torch.randint(-127, 128, (h, h), device="cuda", generator=gen, dtype=torch.int8) for _ in range(layers)]
    scale = torch.full((h,), 1.0 / (73.6 * h ** 0.5), device="cuda")   # keeps the activations near N(0, 1)
    x = [torch.randn((m, h), device="cuda", generator=gen).bfloat16()] + [torch.empty((m, h), device="cuda", dtype=torch.bfloat16) for _ in range(layers)]

    def chain(flags, wait):
        for i, w in enumerate(weights):
            afb.gemm_launch(afb.make_args(x[i + 1], x[i], w, scale, m, h, h, flags=flags), torch.cuda.current_stream().cuda_stream)
            if wait:
                torch.cuda.synchronize()

    def clear():
        for t in x[1:]:
            t.fill_(float("nan"))
        torch.cuda.synchronize()

    before = afb.stream_launch_count()
    chain(0, True)
    assert afb.stream_launch_count() - before == layers
    want = [t.clone() for t in x]
    assert all(0.5 < t.float().std().item() < 2 for t in want)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        chain(pkg.FLAG_PDL, False)
    for turn in range(6):
        clear()
        if turn % 2:
            graph.replay()
        else:
            for _ in range(3):
                chain(pkg.FLAG_PDL, False)
        torch.cuda.synchronize()
        for i, (got, ref) in enumerate(zip(x, want)):
            assert torch.equal(got, ref), f"turn {turn}, layer {i}"
