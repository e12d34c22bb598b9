"""Edges of the kernels that serve ragged sizes, static activations and few rows of grouped weights: outputs on any
byte boundary, rows read in place or through the padded layout, tiles with one live row or column.  Everything that
is bytes or int32 is compared exactly, with the CPU oracle or with the one-thread-per-output kernel (itself held
to the oracle elsewhere); so is fp32, whose every rounding is part of the contract."""
import numpy as np
import pytest

from tests import workloads as wl
from tests.test_gpu_parity import ctx, dev, torch  # noqa: F401  (fixtures)

pytestmark = pytest.mark.gpu


def bits(a):
    return a.view(np.uint32)


@pytest.mark.parametrize("n", [1, 3, 31, 33, 62, 64, 66, 97, 129, 250, 257, 514])
@pytest.mark.parametrize("rows,lead,extra", [(129, 0, 0), (161, 1, 2), (300, 2, 5), (140, 16, 32), (131, 4, 8)])
def test_byte_outputs_on_any_boundary(torch, ctx, n, rows, lead, extra):
    """int8 tiles whose rows start `lead` bytes into a row pitch of n + lead + extra: both tile kernels (and the
    narrow tiles of the second), with bias and zero point, nothing written beside the window."""
    from volvoxai_b200 import w8a8
    c = wl.single_linear(rows=rows, k=100, n=n, seed=n + rows)
    bias = np.arange(n, dtype=np.int32) * 37 - 900
    weight = w8a8.Weight.from_i8(ctx, c["w"], c["ws"], bias_i32=bias)
    x = dev(torch, c["x"])
    want = ctx.linear_i8(weight, x, 0.05, 3, route=w8a8.ROUTE_SIMT)
    for route in (w8a8.ROUTE_TCGEN05, w8a8.ROUTE_TCGEN05_PAIR):
        wide = torch.full((rows, lead + n + extra), 99, dtype=torch.int8, device="cuda")
        ctx.linear_i8(weight, x, 0.05, 3, out=wide[:, lead:lead + n], route=route)
        assert torch.equal(wide[:, lead:lead + n], want)
        assert (wide[:, :lead] == 99).all() and (wide[:, lead + n:] == 99).all()
    weight.close()


@pytest.mark.parametrize("n", [2, 30, 34, 64, 130, 258])
@pytest.mark.parametrize("lead", [0, 1, 4])
def test_word_outputs_on_any_boundary(torch, ctx, n, lead):
    """fp32 tiles and their SiLU * Mul form, rows `lead` words into the row pitch."""
    from volvoxai_b200 import w8a8
    rows = 150
    c = wl.single_linear(rows=rows, k=100, n=n, seed=n + lead)
    weight = w8a8.Weight.from_i8(ctx, c["w"], c["ws"], bias_f32=c["bias"])
    x = dev(torch, c["x"])
    want = ctx.linear_f32(weight, x, route=w8a8.ROUTE_SIMT)
    for route in (w8a8.ROUTE_TCGEN05, w8a8.ROUTE_TCGEN05_PAIR):
        wide = torch.full((rows, lead + n + 3), 99.0, device="cuda")
        ctx.linear_f32(weight, x, out=wide[:, lead:lead + n], route=route)
        assert torch.equal(wide[:, lead:lead + n], want)
        assert (wide[:, :lead] == 99).all() and (wide[:, lead + n:] == 99).all()
    wide = torch.full((rows, lead + n // 2 + 3), 99.0, device="cuda")
    ctx.linear_f32_fused(weight, x, silu_mul=True, out=wide[:, lead:lead + n // 2])
    g, u = want[:, 0::2].double(), want[:, 1::2].double()
    y = g / (1.0 + torch.exp(-g)) * u
    # four roundings and an expf of at most 2 ulp: 1e-6 of the value covers eight
    assert (wide[:, lead:lead + n // 2].double() - y).abs().le(1e-6 * y.abs() + 1e-30).all()
    assert (wide[:, :lead] == 99).all() and (wide[:, lead + n // 2:] == 99).all()
    weight.close()
