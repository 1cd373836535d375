"""Operators that are launched by themselves have kernels of their own (``csrc/solo.h``).  They are held to the stage of a program with the
same handle - bit for bit where both add up in one order - and otherwise to 64-bit arithmetic, at the edges of their tiles and of the
rules that choose them."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from native_pi0.linear import NativeStageProgram
from native_pi0.normalization import ResidentNorm


def outputs(op):
    tensors = [op.output, getattr(op, "output_scales", None), getattr(op, "residual_output", None), getattr(op, "normalized", None)]
    return [t.view(torch.uint8) for t in tensors if t is not None]


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
        for got, w in zip(outputs(op), want):
            assert torch.equal(got, w)


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
