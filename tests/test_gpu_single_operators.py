"""Operators that are launched by themselves have kernels of their own (``csrc/solo.h``).  They are held to the stage of a program with the
same handle - bit for bit where both add up in one order - and otherwise to 64-bit arithmetic, at the edges of their tiles and of the
rules that choose them."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from native_pi0 import _native
from native_pi0.attention import ResidentAttention
from native_pi0.dense import ResidentDense
from native_pi0.linear import NativeStageProgram
from native_pi0.normalization import ResidentNorm
from native_pi0.primitives import ResidentNVFP4
from native_pi0.quantization import PackedNVFP4


def codes(rng, rows, k, scale):
    return PackedNVFP4(rng.integers(0, 256, size=(rows, k // 2), dtype=np.uint8), rng.integers(40, 61, size=(rows, k // 16), dtype=np.uint8),
                       np.float32(scale), (rows, k))


def outputs(op):
    tensors = [op.output, getattr(op, "output_scales", None), getattr(op, "residual_output", None), getattr(op, "normalized", None)]
    return [t.view(torch.uint8) for t in tensors if t is not None]


def library(op):
    return getattr(op, "library", None) or op._library


def budget(op, nanoseconds):
    _native.check(library(op).set_native_model_wait_budget(op.handle, nanoseconds), "wait budget")


def counters(op):
    total = ctypes.c_int()
    _native.check(library(op).read_native_model_counters(op.handle, None, None, 0, ctypes.byref(total)), "counters")
    counts, expected = ((ctypes.c_uint * total.value)() for _ in range(2))
    _native.check(library(op).read_native_model_counters(op.handle, counts, expected, total.value, None), "counters")
    return list(counts), list(expected)


def launch_form(op):
    """CTAs that share a tile, its columns, splits of K; None where the operator runs as a program of one stage."""
    values = (ctypes.c_int * 5)()
    _native.check(library(op).operator_launch_form(op.handle, values, 5), "launch form")
    return tuple(values[1:4]) if values[0] == 2 else None


def alone_and_as_a_stage(op):
    """Three launches of ``op`` give the bits of a program of that one stage, counters included."""
    with NativeStageProgram(None, [(op, [])]) as program:
        for t in outputs(op):
            t.zero_()
        program.forward()
        assert program.status()["code"] == 0
        want = [t.clone() for t in outputs(op)]
    for launch in range(3):
        for t in outputs(op):
            t.zero_()
        op.forward()
        status = op.status()
        assert status["code"] == 0 and status["epoch"] == launch + 1
        counts, expected = counters(op)
        assert counts == expected and max(counts) > 0
        for got, w in zip(outputs(op), want):
            assert torch.equal(got, w)


@pytest.mark.parametrize("rows,n,k,block_n,tiled,workers,ctas,width", [
    (1, 128, 64, 128, False, 148, 1, 64),            # a single K group, two tiles
    (51, 2560, 1024, 64, True, 148, 1, 64),
    (51, 640, 320, 32, False, 148, 1, 32),           # 32-wide tiles with scales of their own, half-filled last slot
    (129, 384, 1152, 128, False, 148, 1, 64),        # one row in the second band
    (640, 8192, 1088, 128, False, 148, 1, 128),      # K not in whole slots
    (256, 16384, 1024, 128, True, 148, 1, 128),      # tile-major blocks as wide as the tiles
    (256, 16384, 1024, 128, True, 2, 2, 192),        # one pair of CTAs: 192-wide tiles over blocks of 128 rows, the last of 86 cut
    (640, 8192, 1088, 128, False, 7, 2, 192),        # three pairs: odd number of row bands, K not in whole groups of scale atoms
    (300, 4096, 2048, 64, True, 2, 2, 192),          # blocks of 64 rows, a band of 44 rows
    (768, 32768, 2048, 128, True, 148, 2, 192),      # pairs on all SMs, seven tiles each
])
@pytest.mark.parametrize("out,act", [("f32", "none"), ("bf16", "none"), ("fp4", "none"), ("fp4", "gelu"), ("fp4", "geglu"), ("fp4", "relu2")])
def test_nvfp4_projection(rows, n, k, block_n, tiled, workers, ctas, width, out, act):
    if act == "geglu" and n % 256:
        pytest.skip("GeGLU takes whole pairs of 128 columns")
    rng, m = np.random.default_rng(rows + n + k), -(-rows // 128) * 128
    g = torch.Generator(device="cuda").manual_seed(rows)
    added = out != "f32" and act != "geglu"
    with ResidentNVFP4(None, codes(rng, m, k, 1.0), codes(rng, n, k, 0.01), workers=workers, rows=rows, block_n=block_n, tiled_weight=tiled,
                       output_dtype={"f32": torch.float32, "bf16": torch.bfloat16, "fp4": torch.uint8}[out], output_gelu=act == "gelu",
                       output_geglu=act == "geglu", output_relu2=act == "relu2",
                       bias=torch.randn(n, generator=g, device="cuda") if added else None,
                       residual=torch.randn(m, n, generator=g, device="cuda") if added else None) as op:
        assert launch_form(op) == (ctas, width, 1)
        alone_and_as_a_stage(op)


@pytest.mark.parametrize("rows,n,k,block_n,workers,own", [
    (64, 2048, 16384, 64, 148, False), (73, 2048, 16384, 64, 148, True), (64, 2176, 16384, 64, 148, True), (64, 2048, 16128, 64, 148, True),
    (64, 2048, 16384, 128, 148, True), (64, 2048, 16384, 64, 31, True), (1, 256, 32768, 64, 4, False),
])
def test_few_rows_over_a_long_k(rows, n, k, block_n, workers, own):
    """One tile for each of a few CTAs runs as a program of one stage; more rows, tiles, CTAs or a shorter K do not."""
    rng = np.random.default_rng(n)
    with ResidentNVFP4(None, codes(rng, 128, k, 1.0), codes(rng, n, k, 0.01), workers=workers, rows=rows, block_n=block_n, output_dtype=torch.bfloat16) as op:
        assert (launch_form(op) is not None) == own
        op.forward()
        assert op.status()["code"] == 0


@pytest.mark.parametrize("workers", [1, 3, 148])
@pytest.mark.parametrize("rows,n,k", [(1, 104, 504), (65, 1000, 1152), (333, 1000, 1152), (820, 4400, 1088), (256, 9000, 640)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float8_e4m3fn])
def test_dense_projection(rows, n, k, dtype, workers):
    g = torch.Generator(device="cuda").manual_seed(rows + n + k)
    randn = lambda *s: torch.randn(*s, generator=g, device="cuda")          # noqa: E731
    for kind in (dict(output_dtype=torch.float32), dict(output_dtype=torch.float32, bias=randn(n), residual=randn(rows, n)), dict(bias=randn(n), residual=randn(rows, n))):
        with ResidentDense(None, randn(rows, k).to(dtype), randn(n, k).to(dtype), alpha=0.05, workers=workers, **kind) as op:
            if workers == 1 or (rows, workers) == (820, 3):
                assert launch_form(op)[0] == workers // 3 + 1                                     # (one CTA; one pair with several tiles)
            alone_and_as_a_stage(op)


@pytest.mark.parametrize("rows,n,k,dtype,workers,width,splits", [
    (768, 2048, 16384, torch.float8_e4m3fn, 148, 256, 2), (513, 1930, 8192, torch.float8_e4m3fn, 148, 256, 2), (300, 1200, 8192, torch.bfloat16, 148, 192, 4),
    (512, 512, 12288, torch.float8_e4m3fn, 148, 64, 3), (256, 64, 16384, torch.float8_e4m3fn, 148, 64, 4),      # two 32-column pieces: pairs without one
    (256, 200, 24576, torch.float8_e4m3fn, 6, 256, 3), (129, 128, 16384, torch.bfloat16, 6, 128, 3),            # one cluster of six
])
def test_dense_projection_over_a_long_k(rows, n, k, dtype, workers, width, splits):
    """K split over the pairs of a cluster: sums of parts, repeated bit for bit and no further from 64 bits than one sum over all of K."""
    g = torch.Generator(device="cuda").manual_seed(k + n)
    a, b = torch.randn(rows, k, generator=g, device="cuda").to(dtype), torch.randn(n, k, generator=g, device="cuda").to(dtype)
    with ResidentDense(None, a, b, output_dtype=torch.float32, workers=workers) as op:
        assert launch_form(op) == (2, width, splits)
        exact = a.double() @ b.double().T
        bound = 2.0 ** -22 * k ** 0.5 * (a.double().abs() @ b.double().abs().T)              # (FP32 sums of K terms)
        with NativeStageProgram(None, [(op, [])]) as program:
            program.forward()
            single = float((op.logical_output.double() - exact).norm())
        want = op.forward().clone()
        assert op.status()["code"] == 0 and bool(((want.double() - exact).abs() <= bound).all())
        assert float((want.double() - exact).norm()) <= 1.02 * single
        for _ in range(3):
            op.output.fill_(float("nan"))
            assert torch.equal(op.forward(), want)
    bias, residual = torch.randn(n, generator=g, device="cuda"), torch.randn(rows, n, generator=g, device="cuda").bfloat16()
    with ResidentDense(None, a, b, bias=bias, residual=residual, workers=workers) as op:
        assert launch_form(op)[2] == splits
        assert torch.equal(op.forward(), (want + residual.float() + bias.bfloat16().float()).bfloat16())


@pytest.mark.parametrize("nq,nk,heads,prefix,splits,workers", [
    (1, 1, 1, None, 1, 148), (1, 16, 8, None, 1, 148), (16, 17, 8, 3, 1, 148),                # one row; whole and ragged pieces of 16 keys
    (17, 256, 8, None, 1, 2), (300, 256, 3, 100, 1, 148),                                     # heads that do not divide the 128 rows of a tile
    (784, 784, 8, None, 4, 148), (700, 816, 8, None, 4, 148), (769, 819, 8, 0, 4, 40),        # several tiles per CTA
    (51, 819, 8, 768, 13, 148), (51, 819, 8, 768, 13, 3), (101, 920, 8, 819, 13, 148), (2, 2000, 8, 1500, 32, 148),
    (300, 300, 8, None, 2, 16), (10, 487, 8, 477, 13, 148), (16, 17, 8, 3, 16, 148),          # few workers; many ranges of few rows; ranges without a key
])
def test_attention_of_heads_with_one_kv_head(nq, nk, heads, prefix, splits, workers):
    g = torch.Generator(device="cuda").manual_seed(nq + nk)
    make = lambda n, h: torch.randn(1, n, h, 256, generator=g, device="cuda").bfloat16()      # noqa: E731
    q, k, v = make(nq, heads), make(nk, 1), make(nk, 1)
    scores = torch.einsum("qhd,kd->hqk", q[0].double(), k[0, :, 0].double()) / 16
    if prefix is not None:
        scores[:, 0, prefix + 1:] = -torch.inf
    want = torch.einsum("hqk,kd->qhd", scores.softmax(-1), v[0, :, 0].double())
    error = lambda y: float((y.double() - want).norm() / want.norm())                         # noqa: E731
    # (rows of Q that do not lie one behind another: the stage of the persistent kernel)
    wide = torch.nn.functional.pad(q, (0, 0, 0, 1))[:, :, :heads]
    with ResidentAttention(None, wide, k, v, workers=workers, prefix=prefix, splits=splits, head_dim=256, path="tcgen05") as op:
        stage = op.forward().reshape(nq, heads, 256).clone()
        assert op.status()["code"] == 0
    with ResidentAttention(None, q, k, v, workers=workers, prefix=prefix, splits=splits, head_dim=256, path="tcgen05") as op:
        for launch in range(3):
            op.output.fill_(float("nan"))
            if splits > 1:
                op.poison_partials()
            got = op.forward().reshape(nq, heads, 256).clone()
            assert op.status()["code"] == 0
            # probabilities, partial rows and rows are rounded to BF16, each off by a part in 2^8 / sqrt(3) in the mean at most; the stage rounds
            # the same ones, and only the row sums add up in another order (FP32), which now and then moves a result to the next BF16 value
            assert error(got) <= 2 ** -8 * ((3 if splits > 1 else 2) / 3) ** 0.5 and error(got) <= 1.002 * error(stage)
            off = (got.double() - stage.double()).abs()
            assert bool((off <= 2 ** -7 * stage.double().abs() + 2 ** -16).all()) and float((off > 0).double().mean()) <= 0.01
            if launch:
                assert torch.equal(got, first)
            first = got
        if splits > 1:
            state = op.read_split_counts()
            assert state["epoch"] == 3 and all(c == 3 * splits for c in state["counts"])


def test_merge_handle_launched_by_itself():
    """The merge stage of a split attention merges the partial rows of its owner's last launch again, whenever its handle was asked for."""
    g = torch.Generator(device="cuda").manual_seed(12)
    q, k = (torch.randn(1, n, h, 256, generator=g, device="cuda").bfloat16() for n, h in ((51, 8), (819, 1)))
    with ResidentAttention(None, q, k, k, workers=148, splits=13, head_dim=256) as op:
        alone = op.forward().clone()
        merge = op.merge_handle
        for _ in range(2):
            want = op.forward().clone()
            op.output.zero_()
            _native.check(op.library.launch_op(merge, torch.cuda.current_stream().cuda_stream), "merge")
            assert torch.equal(op.output, want) and op.status()["code"] == 0
        assert float((want.double() - alone.double()).norm() / want.double().norm()) <= 1e-3
        state = op.read_split_counts()
        assert all(c == 13 * state["epoch"] for c in state["counts"])


def test_partial_rows_of_split_attention():
    """An operator holds partial rows for its configured ranges and no more, launched by itself or not: 64 of 128 rows here, 4 MiB."""
    g = torch.Generator(device="cuda").manual_seed(11)
    q, k = (torch.randn(1, n, h, 256, generator=g, device="cuda").bfloat16() for n, h in ((51, 8), (819, 1)))
    ops, output = [], torch.empty(1, 51, 8, 256, dtype=torch.bfloat16, device="cuda")
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    try:
        for _ in range(32):
            ops.append(ResidentAttention(None, q, k, k, workers=148, splits=8, head_dim=256, output=output))
            ops[-1].forward()
        torch.cuda.synchronize()
        assert before - torch.cuda.mem_get_info()[0] <= 32 * (4 << 20) * 1.25                 # (statistics, programs, whole pages)
    finally:
        for op in ops:
            op.close()


@pytest.mark.parametrize("batches,nq,nk,heads,kv_heads,head_dim,prefix,workers", [
    (1, 1, 1, 1, 1, 72, None, 148), (1, 16, 17, 2, 2, 72, 3, 148),                            # one row; ragged pieces of 16 keys
    (3, 256, 256, 16, 16, 72, None, 148), (2, 129, 240, 16, 16, 72, None, 148),               # one row in an image's second tile
    (3, 200, 196, 4, 2, 72, None, 5), (1, 130, 256, 3, 1, 72, 0, 148),                        # several tiles per CTA; query heads that share KV heads
])
def test_attention_of_heads_stored_128_apart(batches, nq, nk, heads, kv_heads, head_dim, prefix, workers):
    g = torch.Generator(device="cuda").manual_seed(nq + nk)
    make = lambda n, h: torch.nn.functional.pad(torch.randn(batches, n, h, head_dim, generator=g, device="cuda"), (0, 128 - head_dim)).bfloat16()      # noqa: E731
    q, k, v = make(nq, heads), make(nk, kv_heads), make(nk, kv_heads)
    kd, vd = (t[..., :head_dim].double().repeat_interleave(heads // kv_heads, 2) for t in (k, v))
    scores = torch.einsum("bqhd,bkhd->bhqk", q[..., :head_dim].double(), kd) * head_dim ** -0.5
    if prefix is not None:
        scores[:, :, 0, prefix + 1:] = -torch.inf
    want = torch.einsum("bhqk,bkhd->bqhd", scores.softmax(-1), vd)
    error = lambda y: float((y - want).norm() / want.norm())                                  # noqa: E731
    with ResidentAttention(None, q, k, v, workers=workers, prefix=prefix, head_dim=head_dim, path="tcgen05") as op:
        with NativeStageProgram(None, [(op, [])]) as program:
            stage = program.forward().reshape(want.shape).double()
            assert program.status()["code"] == 0
        for _ in range(3):
            op.output.fill_(float("nan"))
            got = op.forward().reshape(want.shape).double()
            assert op.status()["code"] == 0
            assert error(got) <= 2 ** -8 * (2 / 3) ** 0.5 and error(got) <= 1.002 * error(stage)      # (as above)
            assert bool(((got - stage).abs() <= 2 ** -7 * stage.abs() + 2 ** -16).all())


@pytest.mark.parametrize("rows,width", [(1, 16), (51, 1024), (592, 2048), (593, 1168), (2000, 64)])
def test_norm(rows, width):
    g = torch.Generator(device="cuda").manual_seed(rows + width)
    x, r = (torch.randn(rows, width, generator=g, device="cuda").bfloat16() for _ in range(2))
    gamma, beta = torch.randn(width, generator=g, device="cuda"), torch.randn(width, generator=g, device="cuda")
    for kw in (dict(precision="fp4", gamma=gamma, keep_bf16=True), dict(kind="layer", precision="fp4", gamma=gamma, beta=beta), dict(precision="fp8", gamma=gamma),
               dict(kind="layer", precision="bf16", gamma=gamma, beta=beta, residual=r), dict(precision="bf16", gamma=gamma, inverse_scale=beta, residual=r),
               dict(precision="factor"), dict(precision="fp4", quantize_only=True)):
        with ResidentNorm(None, x, workers=148, row_alignment=128, **kw) as op:
            alone_and_as_a_stage(op)


def test_wait_budget_of_an_operator():
    """The budget given to an operator handle bounds the waits of its launches, whether it is given before the first or later.  A tile of K =
    131072 on one SM keeps the draining warps waiting for more than 100 us."""
    g = torch.Generator(device="cuda").manual_seed(3)
    a, b = (torch.randn(64, 131072, generator=g, device="cuda").bfloat16() for _ in range(2))
    with ResidentDense(None, a, b, workers=1) as op:
        for _ in range(2):
            budget(op, 20_000)
            op.forward()
            status = op.status()
            assert status["code"] == 2 and status["aborted"] == 1 and status["stage"] == 0
            budget(op, 2_000_000_000)
            good = op.forward().clone()
            assert op.status()["code"] == 0
            assert float((good.double() - a.double() @ b.double().T).norm() / good.double().norm()) < 3e-3


def test_wait_budget_begins_behind_the_kernel_in_front():
    """CTAs that are let in early do not count their predecessor's time as their own: about a millisecond on one SM, in front of operators that may
    wait for 100 us."""
    g = torch.Generator(device="cuda").manual_seed(4)
    randn = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()                 # noqa: E731
    with ResidentDense(None, randn(64, 131072), randn(512, 131072), workers=1) as long, \
            ResidentDense(None, randn(64, 1024), randn(128, 1024), workers=148) as gemm, \
            ResidentAttention(None, randn(1, 51, 8, 256), randn(1, 819, 1, 256), randn(1, 819, 1, 256), workers=148, splits=13) as attention:
        for op in (gemm, attention):
            want = op.forward().clone()
            budget(op, 100_000)
            for _ in range(2):
                start, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
                start.record()
                long.forward()
                end.record()
                torch.cuda.synchronize()
                assert start.elapsed_time(end) > 0.3                                          # (three times the budget)
                long.forward()
                got = op.forward()
                assert op.status()["code"] == 0 and torch.equal(got, want)
        assert long.status()["code"] == 0


@pytest.mark.parametrize("rows,n,k,workers", [(64, 64, 524288, 1), (256, 256, 1048576, 8)])      # one CTA; K split over the pairs of a cluster
def test_a_tile_that_gave_up_is_not_finished(rows, n, k, workers):
    """A draining warp whose wait for some 450 us of MMAs runs out leaves its tile unwritten and uncounted, in every pair that shares it."""
    g = torch.Generator(device="cuda").manual_seed(k)
    a, b = (torch.randn(r, 4096, generator=g, device="cuda").to(torch.float8_e4m3fn).repeat(1, k // 4096) for r in (rows, n))
    with ResidentDense(None, a, b, workers=workers) as op:
        good = op.forward().clone()
        counts, expected = counters(op)
        assert op.status()["code"] == 0 and counts == expected and max(counts) > 0
        for _ in range(2):
            op.output.fill_(float("nan"))
            budget(op, 5_000)
            op.forward()
            counts, expected = counters(op)
            assert sum(counts) < sum(expected)
            assert op.status()["code"] == 2 and bool(torch.isnan(op.output[:rows, :n]).any())
            budget(op, 2_000_000_000)
            assert torch.equal(op.forward(), good) and op.status()["code"] == 0


def test_attention_whose_partners_do_not_arrive_is_not_finished():
    """Another stream keeps all but one or two SMs for some 600 us: the first tiles wait for the partial rows of others that have no place to run,
    give up after 50 us and are not counted; those that come later see it and end."""
    g = torch.Generator(device="cuda").manual_seed(4)
    randn = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()                 # noqa: E731
    other = torch.cuda.Stream()
    with ResidentDense(None, randn(768, 16384), randn(32768, 16384), workers=147) as long, \
            ResidentAttention(None, randn(1, 51, 8, 256), randn(1, 819, 1, 256), randn(1, 819, 1, 256), workers=148, splits=13) as op:
        want = op.forward().clone()
        counts, expected = counters(op)
        assert op.status()["code"] == 0 and counts == expected
        long.forward()
        torch.cuda.synchronize()
        budget(op, 50_000)
        with torch.cuda.stream(other):
            long.forward()
        op.forward()
        counts, expected = counters(op)
        assert op.status()["code"] == 2 and sum(counts) < sum(expected)
        budget(op, 2_000_000_000)
        for _ in range(3):
            assert torch.equal(op.forward(), want)
        assert op.status()["code"] == 0 and counters(op)[0] == counters(op)[1]
