"""What is measured of this framework: the mixed-precision GEMM C = A (bf16) x dequant(B)^T at the sizes, weight formats and entry points
that a program serving a language model uses it with.

listed()   the cases that are timed by name
draw(rng)  one more case of the same ranges
prepare / run / work / tolerance   of one case

A case's "kind" says how the program calls the framework:
  eager   torch.ops.afb.bf16_aintb_gemm from Python, one GEMM per pass: a model whose layers are called one by one
  block   the four projections of one transformer block (query/key/value, output, gate/up, down) through the operator, captured once in
          a CUDA graph with FLAG_PDL as a serving loop keeps it; a pass is one replay
  gemm    afb_gemm_launch on buffers that the program owns
  gated   afb_gemm_fused_launch: act(gate) * up + residual of a gated MLP, on weights that afb_prepack_gated laid out once
  pack    afb_prepack of a weight matrix in the reference's [K, N] layout: what loading a model costs, matrix by matrix
"""
import math

import torch

import awesome_fusion_b200 as afb
import awesome_fusion_b200.torch_op  # noqa: F401  (registers torch.ops.afb)

_LARGEST = 4096 * 28672 * 8192   # m * n * k of the largest listed case


def _case(kind, m, n, k, bits, group=0, zero=False, offset=False, packed=False, **more):
    return dict(kind=kind, m=m, n=n, k=k, bits=bits, group=group, zero=zero, offset=offset, packed=packed, **more)


def listed():
    cases = [
        # the smallest call: one token, one attention projection, called from Python; latency of the call and of the kernel
        ("eager-m1-int8", _case("eager", 1, 4096, 4096, 8)),
        # one token through the projections of a block of a 4096-wide model, int8 weights: the decode loop of a single user
        ("block-m1-int8", _case("block", 1, 11008, 4096, 8)),
        # sixteen users decoding together on group-scaled int4 weights
        ("block-m16-int4", _case("block", 16, 11008, 4096, 4, 128)),
        # the large MLP projection for a handful of tokens (a few users, or drafted tokens being verified), int4 with zero-points
        ("decode-m5-int4-zero", _case("gemm", 5, 28672, 8192, 4, 128, zero=True)),
        # the same projection in int8 for the largest batch of the decode range
        ("decode-m16-int8", _case("gemm", 16, 28672, 8192, 8)),
        # a batch of 40 decoding users, more than the decode range: square projection, stored with offset 128 as the reference stores it
        ("batch-m40-int8", _case("gemm", 40, 8192, 8192, 8, offset=True)),
        # a batch of 128 on the large int4 projection
        ("batch-m128-int4", _case("gemm", 128, 28672, 8192, 4, 128)),
        # a short prompt of odd length on a matrix whose edges fall inside tiles, called from Python
        ("prompt-m333-int8", _case("eager", 333, 11000, 4096, 8)),
        # a prompt of 2048 tokens, up projection, int8
        ("prompt-m2048-int8", _case("gemm", 2048, 11008, 4096, 8)),
        # the largest: 4096 tokens on the large int4 projection
        ("prompt-m4096-int4", _case("gemm", 4096, 28672, 8192, 4, 128)),
        # gate and up projection of a gated MLP with its activation and the residual, pre-packed weights
        ("mlp-m1000-int8", _case("gated", 1000, 11008, 4096, 8, packed=True)),
        # loading one matrix of the reference's layout
        ("load-kn-int8", _case("pack", 0, 11008, 4096, 8)),
    ]
    return [dict(c, name=name) for name, c in cases]


def _log_uniform(rng, lo, hi, multiple):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / multiple)) * multiple))


def draw(rng):
    kind = rng.choice(["eager", "block", "gemm", "gemm", "gemm", "gemm", "gemm", "gemm", "gated", "pack"])
    n, k = _log_uniform(rng, 1024, 28672, 8), _log_uniform(rng, 1024, 11008, 128)
    bits = rng.choice([8, 4])
    group = rng.choice([128, 128, 64, 0]) if bits == 4 else 0
    zero = bool(group) and kind in ("gemm", "gated") and rng.random() < 0.4
    offset = rng.random() < 0.3
    packed = kind == "gated" or (kind == "gemm" and rng.random() < 0.3)
    if kind == "pack":
        return _case("pack", 0, n, k, 8, offset=offset)
    if kind == "block":   # n is the width of the MLP here, k that of the model
        k = _log_uniform(rng, 1024, 8192, 128)
        n = _log_uniform(rng, 2 * k, 4 * k, 128)
        return _case("block", _log_uniform(rng, 1, 16, 1), n, k, bits, group and 128, offset=offset)
    m = _log_uniform(rng, 1, 4096, 1) if kind != "gated" else _log_uniform(rng, 64, 4096, 1)
    m = max(1, min(m, _LARGEST // (n * k * (2 if kind == "gated" else 1))))
    return _case(kind, m, n, k, bits, group, zero=zero, offset=offset, packed=packed)


class _Maker:
    """Inputs from a seed: activations ~ N(0, 1), integers uniform over their range, positive scales, zero-points near the middle."""

    def __init__(self, seed):
        self.gen = torch.Generator(device="cuda")
        self.gen.manual_seed(seed)

    def activations(self, m, k):
        return torch.randn((m, k), device="cuda", generator=self.gen, dtype=torch.float32).to(torch.bfloat16)

    def weights(self, rows, cols, bits, offset):
        if bits == 4:   # two per byte along K; every byte is a legal pair
            return torch.randint(0, 256, (rows, cols // 2), device="cuda", generator=self.gen, dtype=torch.uint8)
        q = torch.randint(-127, 128, (rows, cols), device="cuda", generator=self.gen, dtype=torch.int8)
        return q ^ -128 if offset else q

    def scales(self, n, k, group):
        if group:
            s = torch.rand((n, k // group), device="cuda", generator=self.gen) * 0.045 + 0.005
            return s.to(torch.bfloat16)
        return torch.rand((n,), device="cuda", generator=self.gen) * 0.009 + 0.001

    def zeros(self, n, k, group, offset):
        z = torch.randint(-3, 4, (n, k // group), device="cuda", generator=self.gen, dtype=torch.int16)
        return ((z + 8 if offset else z) & 15).to(torch.uint8)


def _args(lib, case, c, a, b, scale, n, zero=None, ldc=None, layout=afb.LAYOUT_COL):
    return lib.make_args(c, a, b, scale, case["m"], n, case["k"], ldc=ldc, bits=case["bits"], group=case["group"], layout=layout, zero=zero,
                         encoding=afb.ENC_OFFSET if case["offset"] else afb.ENC_TWOS,
                         scale_dtype=afb.SCALE_BF16 if scale.dtype == torch.bfloat16 else afb.SCALE_F32)


def _block_shapes(case):
    h, f = case["k"], case["n"]
    return [(3 * h, h), (h, h), (2 * f, h), (h, f)]


def prepare(case, seed):
    lib = afb.load()
    lib.init(torch.cuda.current_device())
    make = _Maker(seed)
    m, n, k, bits, group, offset = (case[key] for key in ("m", "n", "k", "bits", "group", "offset"))
    kind = case["kind"]
    stream = torch.cuda.current_stream().cuda_stream
    state = dict(case=case, lib=lib, stream=stream)
    if kind == "block":
        calls = [(make.activations(m, ck), make.weights(cn, ck, bits, offset), make.scales(cn, ck, group), bits, group, offset, afb.FLAG_PDL)
                 for cn, ck in _block_shapes(case)]
        for call in calls:   # a kernel's first call is made outside the capture
            torch.ops.afb.bf16_aintb_gemm(*call)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = [torch.ops.afb.bf16_aintb_gemm(*call) for call in calls]
        state.update(graph=graph, out=out, keep=calls)
    elif kind == "eager":
        state["call"] = (make.activations(m, k), make.weights(n, k, bits, offset), make.scales(n, k, group), bits, group, offset)
    elif kind == "pack":
        b = make.weights(k, n, bits, offset)
        out = torch.empty((n, k), device="cuda", dtype=torch.int8)
        args = lib.make_args(None, None, b, None, 1, n, k, bits=bits, layout=afb.LAYOUT_ROW)
        state.update(args=args, out=out, keep=b)
    else:
        a = make.activations(m, k)
        rows = [(make.weights(n, k, bits, offset), make.scales(n, k, group), make.zeros(n, k, group, offset) if case["zero"] else None)
                for _ in range(2 if kind == "gated" else 1)]
        c = torch.empty((m, n), device="cuda", dtype=torch.bfloat16)
        b, scale, zero = rows[0]
        if kind == "gated":
            b2 = torch.empty((2 * n, b.shape[1]), device="cuda", dtype=b.dtype)
            scale2 = torch.cat([scale, scale])
            zero2 = torch.cat([zero, zero]) if zero is not None else None
            lib.prepack_gated(_args(lib, case, c, a, b, scale, n, zero), *rows[1], b2, k, scale2, zero2, stream)
            residual = make.activations(m, n)
            args = lib.make_fused_args(_args(lib, case, c, a, b2, scale2, 2 * n, zero2, n, afb.LAYOUT_COL_PACKED), gated=True,
                                       activation=afb.ACT_SILU, residual=residual, ld_residual=n)
            keep = (a, b2, scale2, zero2, residual)
            torch.cuda.synchronize()   # the projections' own buffers go
        else:
            layout = afb.LAYOUT_COL
            if case["packed"]:
                lib.prepack(_args(lib, case, c, a, b, scale, n), b, k, stream)   # in place
                layout = afb.LAYOUT_COL_PACKED
            args = _args(lib, case, c, a, b, scale, n, zero, layout=layout)
            keep = (a, b, scale, zero)
        state.update(args=args, out=c, keep=keep)
    return state


def run(state):
    kind = state["case"]["kind"]
    if kind == "block":
        state["graph"].replay()
        return state["out"]
    if kind == "eager":
        return torch.ops.afb.bf16_aintb_gemm(*state["call"])
    if kind == "pack":
        state["lib"].prepack(state["args"], state["out"], state["case"]["k"], state["stream"])
    elif kind == "gated":
        state["lib"].gemm_fused_launch(state["args"], state["stream"])
    else:
        state["lib"].gemm_launch(state["args"], state["stream"])
    return state["out"]


def _gemm_work(m, n, k, bits, group, zero):
    scales = n * (k // group) * (2 + int(zero)) if group else n * 4
    return 2 * m * k + n * k * bits // 8 + scales + 2 * m * n, 2 * m * n * k


def work(case):
    m, n, k = case["m"], case["n"], case["k"]
    fmt = (case["bits"], case["group"], case["zero"])
    if case["kind"] == "pack":
        return {"bytes": 2 * n * k, "flops": 0}
    if case["kind"] == "block":
        parts = [_gemm_work(m, cn, ck, *fmt) for cn, ck in _block_shapes(case)]
        return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}
    if case["kind"] == "gated":   # 2n rows of B, n columns of C, the residual read
        nbytes, flops = _gemm_work(m, 2 * n, k, *fmt)
        return {"bytes": nbytes, "flops": flops}
    nbytes, flops = _gemm_work(m, n, k, *fmt)
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """Against the same path in 64 bits the results are off by 1.7e-3 (2-norm): one rounding to bf16, half a unit in the last place at most
    (2^-9 of the value).  Group scales above 16 activation rows: each weight is rounded to bf16 once more, before the sum (2.4e-3 in all).
    Each is stated four times over; the largest difference of one value as three units in the last place of a bf16, 3 * 2^-7, and for the
    gated product, where the gate's and the up projection's errors meet, twice that."""
    if case["kind"] == "pack":
        return "exact"
    finest = 128 if case["bits"] == 4 else 64   # smallest scale group of the kernels for up to 16 rows
    twice = bool(case["group"]) and (case["m"] > 16 or case["kind"] == "gated" or case["group"] < finest)
    return {"rel": 1e-2 if twice else 7e-3, "max": 0.05 if case["kind"] == "gated" or twice else 0.025}
