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


@pytest.mark.parametrize("k", [1, 31, 33, 257, 1023, 1025, 2047, 4097, 8190, 8195])
@pytest.mark.parametrize("rows", [1, 3, 700])
def test_quantizer_any_width_and_alignment(torch, ctx, oracle, k, rows):
    """Widths around the threads-per-row steps of the any-alignment quantizer, on a base 4 bytes off; an invalid, a
    zero, a very small and a very large row."""
    rng = np.random.default_rng(k * 3 + rows)
    x = rng.standard_normal((rows, k)).astype(np.float32)
    if rows > 4:
        x[1] = 0
        x[2, k // 2] = np.inf
        x[3] *= np.float32(1e-35)
        x[4] *= np.float32(1e30)
    qo, so, vo = oracle.quantize_rows(x)
    flat = torch.empty(rows * k + 1, device="cuda")
    flat[1:] = dev(torch, x).flatten()
    kpad = (k + 127) // 128 * 128
    q, s, v = ctx.quantize_rows(flat[1:].view(rows, k), ldq=kpad)
    q, s, v = q.cpu().numpy(), s.cpu().numpy(), v.cpu().numpy()
    assert np.array_equal(v != 0, vo != 0)
    assert np.array_equal(q[:, :k], qo) and (q[:, k:] == 0).all()
    assert np.array_equal(bits(s[vo != 0]), bits(so[vo != 0])) and np.isnan(s[vo == 0]).all()


@pytest.mark.parametrize("rows,k", [(r, k + d) for r, ks in ((5000, (128, 256, 512, 1024)), (3, (256, 512, 1024, 2048, 4096, 8192))) for k in ks for d in (0, 1)])
def test_quantizer_elements_per_thread(torch, ctx, oracle, rows, k):
    """Widths on both sides of each step in the any-alignment quantizer's elements per thread, with 32 threads per row and
    with up to 256."""
    x = np.random.default_rng(k + rows).standard_normal((rows, k)).astype(np.float32)
    x[1, k - 1] = -np.inf
    x[2] *= np.float32(1e-36)
    qo, so, vo = oracle.quantize_rows(x)
    flat = torch.empty(rows * k + 1, device="cuda")
    flat[1:] = dev(torch, x).flatten()
    kpad = (k + 127) // 128 * 128
    q, s, v = (t.cpu().numpy() for t in ctx.quantize_rows(flat[1:].view(rows, k), ldq=kpad))
    assert np.array_equal(v != 0, vo != 0)
    assert np.array_equal(q[:, :k], qo) and (q[:, k:] == 0).all()
    assert np.array_equal(bits(s[vo != 0]), bits(so[vo != 0])) and np.isnan(s[vo == 0]).all()


@pytest.mark.parametrize("n", [1, 3, 31, 33, 62, 64, 66, 97, 129, 250, 257, 514])
@pytest.mark.parametrize("rows,lead,extra", [(129, 0, 0), (161, 1, 2), (300, 2, 5), (140, 16, 32), (131, 4, 8)])
def test_byte_outputs_on_any_boundary(torch, ctx, n, rows, lead, extra):
    """int8 tiles whose rows start `lead` bytes into a row pitch of n + lead + extra: both tile kernels, with bias and zero
    point, nothing written beside the window."""
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


@pytest.mark.parametrize("n", [4, 28, 36, 64, 132, 260, 2052])
@pytest.mark.parametrize("rows", [129, 150, 289])
def test_word_outputs_on_eight_byte_boundaries(torch, ctx, rows, n):
    """fp32 tiles and their SiLU * Mul form in a window whose rows start on 8 bytes and not on 16 (stored in pairs of
    words), and on 4 (in words): equal to the 16-byte aligned form, nothing written beside the window."""
    from volvoxai_b200 import w8a8
    c = wl.single_linear(rows=rows, k=100, n=n, seed=n + rows)
    weight = w8a8.Weight.from_i8(ctx, c["w"], c["ws"], bias_f32=c["bias"])
    x = dev(torch, c["x"])

    def window(width, lead, pitch, call):
        wide = torch.full((rows, pitch), 99.0, device="cuda")
        call(wide[:, lead:lead + width])
        assert (wide[:, :lead] == 99).all() and (wide[:, lead + width:] == 99).all()
        return wide[:, lead:lead + width].clone()

    calls = [(n, lambda out, r=r: ctx.linear_f32(weight, x, out=out, route=r)) for r in (w8a8.ROUTE_TCGEN05, w8a8.ROUTE_TCGEN05_PAIR)]
    calls.append((n // 2, lambda out: ctx.linear_f32_fused(weight, x, silu_mul=True, out=out)))
    for width, call in calls:
        want = window(width, 0, (width + 7) // 4 * 4, call)
        for lead, pitch in ((2, width + 2 + width % 2), (2, width + 4 + width % 2), (1, width + 1), (2, width + 3 - width % 2)):
            assert torch.equal(window(width, lead, pitch, call), want)
    weight.close()


@pytest.mark.parametrize("rows,k,n", [(129, 1600, 128), (257, 2048, 100), (512, 2000, 4096), (600, 4096, 1000), (300, 1537, 386)])
def test_narrow_pair_tiles(torch, ctx, rows, k, n):
    """Long K and few tiles: 256 x 128 tiles by pairs of CTAs, every kind of output, equal to the single-CTA kernel."""
    from volvoxai_b200 import w8a8
    c = wl.single_linear(rows=rows, k=k, n=n, seed=rows + k + n)
    weight = w8a8.Weight.from_i8(ctx, c["w"], c["ws"], bias_f32=c["bias"], bias_i32=np.arange(n, dtype=np.int32) * 11 - 300)
    x = dev(torch, c["x"])
    for call in (lambda r: ctx.linear_acc_i32(weight, x, route=r), lambda r: ctx.linear_f32(weight, x, route=r),
                 lambda r: ctx.linear_i8(weight, x, 0.1, -5, route=r)):
        y = call(w8a8.ROUTE_AUTO)
        assert "pair-narrow" in w8a8.last_route()
        assert torch.equal(y, call(w8a8.ROUTE_TCGEN05))
    weight.close()


@pytest.mark.parametrize("n", [1, 33, 64, 66, 129, 250])
@pytest.mark.parametrize("rows,lead,extra", [(129, 0, 0), (161, 1, 2), (300, 2, 5), (140, 16, 32), (131, 4, 8)])
def test_byte_outputs_of_the_narrow_tiles(torch, ctx, n, rows, lead, extra):
    """The same windows from the 256 x 128 tiles, which the automatic route takes from padded K 1664 on."""
    from volvoxai_b200 import w8a8
    c = wl.single_linear(rows=rows, k=1600, n=n, seed=n + rows)
    weight = w8a8.Weight.from_i8(ctx, c["w"], c["ws"], bias_i32=np.arange(n, dtype=np.int32) * 37 - 900)
    x = dev(torch, c["x"])
    wide = torch.full((rows, lead + n + extra), 99, dtype=torch.int8, device="cuda")
    ctx.linear_i8(weight, x, 0.05, 3, out=wide[:, lead:lead + n])
    assert "pair-narrow" in w8a8.last_route()
    assert torch.equal(wide[:, lead:lead + n], ctx.linear_i8(weight, x, 0.05, 3, route=w8a8.ROUTE_SIMT))
    assert (wide[:, :lead] == 99).all() and (wide[:, lead + n:] == 99).all()
    weight.close()


@pytest.mark.parametrize("rows,k,n,lead,want", [(512, 1664, 2050, 0, "pair-narrow"), (300, 2048, 388, 0, "pair-narrow"), (300, 2048, 386, 1, "pair-narrow"),
                                                (512, 1700, 2048, 2, "pair-narrow"), (2048, 2048, 8192, 0, "tcgen05-pair-i8"),
                                                (2048, 2048, 8192, 3, "tcgen05-pair-i8"), (4096, 256, 2560, 1, "tcgen05-pair-i8"),
                                                (4090, 256, 2564, 2, "tcgen05-pair-i8")])
def test_silu_tail_of_the_paired_tiles(torch, ctx, rows, k, n, lead, want):
    """The SiLU * Mul tail of both paired tile widths, rows on 16 bytes, on 8 and on 4: bit-equal to the decode kernel's tail
    (rows are independent of each other, 64 at a time take that kernel), nothing written beside the window."""
    from volvoxai_b200 import w8a8
    c = wl.single_linear(rows=rows, k=k, n=n, seed=rows + n)
    weight = w8a8.Weight.from_i8(ctx, c["w"], c["ws"], bias_f32=c["bias"])
    x = dev(torch, c["x"])
    half = n // 2
    wide = torch.full((rows, lead + half + (lead and 5)), 99.0, device="cuda")
    ctx.linear_f32_fused(weight, x, silu_mul=True, out=wide[:, lead:lead + half])
    assert want in w8a8.last_route(), w8a8.last_route()
    assert (wide[:, :lead] == 99).all() and (wide[:, lead + half:] == 99).all()
    for r in (0, 64, 128, 224, rows // 128 * 64, rows - 64):
        part = ctx.linear_f32_fused(weight, x[r:r + 64], silu_mul=True)
        assert "decode-rows" in w8a8.last_route()
        assert torch.equal(wide[r:r + 64, lead:lead + half], part)
    weight.close()


@pytest.mark.parametrize("in_u8", [False, True])
@pytest.mark.parametrize("rows,k,n", [(1, 128, 40), (40, 48, 33), (128, 256, 130), (130, 16, 65), (200, 1283, 50), (300, 576, 1536),
                                      (700, 2064, 300)])
def test_static_rows_in_place_and_padded(torch, ctx, oracle, in_u8, rows, k, n):
    """Codes read where they are (whole 16-byte pieces) or through the padded layout, with and without a zero point,
    from an unaligned base, and with the output lying over the input."""
    from volvoxai_b200 import w8a8
    rng = np.random.default_rng(rows + k + n + in_u8)
    x = rng.integers(0, 256, size=(rows, k)).astype(np.uint8) if in_u8 else rng.integers(-128, 128, size=(rows, k)).astype(np.int8)
    w = rng.integers(-127, 128, size=(n, k), dtype=np.int8)
    ws = rng.uniform(0.001, 0.02, size=n).astype(np.float32)
    b = rng.integers(-500, 500, size=n).astype(np.int32)
    weight = w8a8.Weight.from_i8(ctx, w, ws, bias_i32=b)
    for zero in ((128, 7) if in_u8 else (0, -9)):
        want = oracle.qlinear_i8u8(x, w, b, ws, np.zeros(n, np.int32), 0.05, zero, 0.6, 4)
        xd = dev(torch, x)
        assert np.array_equal(ctx.qlinear_device(weight, xd, 0.05, zero, 0.6, 4).cpu().numpy(), want)
        off = torch.empty(rows * k + 1, dtype=xd.dtype, device="cuda")
        off[1:] = xd.flatten()
        assert np.array_equal(ctx.qlinear_device(weight, off[1:].view(rows, k), 0.05, zero, 0.6, 4).cpu().numpy(), want)
        if not in_u8:
            # one buffer: the output's rows start where the input does
            both = torch.zeros(max(rows * k, rows * n), dtype=torch.int8, device="cuda")
            both[:rows * k] = xd.flatten()
            xin = both[:rows * k].view(rows, k)
            out = both[:rows * n].view(rows, n)
            w8a8._check(ctx._L.vxb_qlinear_device(ctx.handle, weight.handle, w8a8._ptr(xin), rows, 0.05, zero, 0.6, 4,
                                                  w8a8.DT_I8, w8a8.DT_I8, w8a8._ptr(out), n, 0))
            assert np.array_equal(out.cpu().numpy(), want)
    weight.close()


@pytest.mark.parametrize("scale", [1e-12, 3e-9, 0.0371, 1.9999999, 5e8, 3e9])
@pytest.mark.parametrize("unsigned,zero", [(False, 0), (False, -128), (True, 255), (True, 3)])
def test_quantize_linear_scales_and_extremes(torch, ctx, oracle, scale, unsigned, zero):
    """Scales on both sides of the fast division's range (and the all-ones significand just below 2), ties, the
    largest and smallest magnitudes, infinities and NaN."""
    s = np.float32(scale)
    ties = (np.arange(-600, 600, dtype=np.float32) * np.float32(0.5) * s).astype(np.float32)
    near = np.concatenate([np.nextafter(ties, np.float32(np.inf)), np.nextafter(ties, np.float32(-np.inf))])
    ext = np.array([0.0, -0.0, 1e-45, -1e-45, 1e-38, 3.4e38, -3.4e38, np.inf, -np.inf, np.nan, 4096, -4097, 1e20], np.float32)
    x = np.tile(np.concatenate([ties, near, ext, ext * s]), 4)
    got = ctx.quantize_linear(dev(torch, x), float(s), zero, unsigned).cpu().numpy()
    assert np.array_equal(got, oracle.quantize_linear(x, float(s), zero, unsigned))


@pytest.mark.parametrize("count", [1, 15, 16, 17, 255, 257, 4095, 4096, 4097, 8191, 12289])
@pytest.mark.parametrize("lead", [0, 1, 3])
def test_boundary_ops_last_blocks_and_unaligned_inputs(torch, ctx, oracle, count, lead):
    """Counts around a thread's 16 elements and a block's 4096, inputs `lead` elements off."""
    rng = np.random.default_rng(count + lead)
    x = (rng.standard_normal(count + lead) * 3).astype(np.float32)
    xd, x = dev(torch, x)[lead:], x[lead:]
    for scale, zero, unsigned in ((0.05, -3, False), (1e-12, 3, True)):
        assert np.array_equal(ctx.quantize_linear(xd, scale, zero, unsigned).cpu().numpy(), oracle.quantize_linear(x, scale, zero, unsigned))
    for dtype, lo, hi, zero in ((np.int8, -128, 128, -7), (np.uint8, 0, 256, 130)):
        c = rng.integers(lo, hi, size=count + lead).astype(dtype)
        cd, c = dev(torch, c)[lead:], c[lead:]
        assert np.array_equal(bits(ctx.dequantize_linear(cd, 0.031, zero).cpu().numpy()), bits(oracle.dequantize_linear(c, 0.031, zero)))
        for unsigned in (False, True):
            assert np.array_equal(ctx.requantize_linear(cd, 0.031, zero, 0.05, 4, unsigned).cpu().numpy(),
                                  oracle.requantize_linear(c, 0.031, zero, 0.05, 4, unsigned))


@pytest.mark.parametrize("group", [32, 64, 128, 256])
@pytest.mark.parametrize("rows,k,n", [(5, 300, 1), (8, 640, 129), (9, 4096, 100), (17, 1283, 300), (33, 896, 64), (64, 2176, 257),
                                      (7, 272, 10000), (40, 384, 19200), (12, 4224, 70), (5, 2048, 4200), (3, 8200, 1540)])
def test_grouped_few_rows(torch, ctx, oracle, group, rows, k, n):
    """Every token-slot count and both tile heights of the few-row kernel: ragged channels, a last stage half empty, a
    last group cut short, more tiles than SMs; rows one past a slot count take the next one."""
    from volvoxai_b200 import _lib, w8a8
    rng = np.random.default_rng(group + rows * 7 + k + n)
    w = rng.integers(-127, 128, size=(n, k), dtype=np.int8)
    words = wl.pack_w8_words(w)
    gs = rng.uniform(0.001, 0.05, size=(n, (k + group - 1) // group)).astype(np.float32)
    bias = rng.standard_normal(n).astype(np.float32)
    x = (rng.standard_normal((rows, k)) * 2).astype(np.float32)
    x[1] = 0
    x[2, k // 3] = np.nan
    wg = w8a8.Weight.from_w8_words(ctx, words, gs, k, group, bias_f32=bias)
    wide = torch.full((rows, n + 5), 99.0, device="cuda")
    ctx.linear_f32(wg, dev(torch, x), out=wide[:, 2:2 + n])
    assert "tcgen05-grouped-i8" in _lib.last_route()
    got = wide.cpu().numpy()
    assert (got[:, :2] == 99).all() and (got[:, 2 + n:] == 99).all()
    y, want = got[:, 2:2 + n], oracle.packed_linear_w8_grouped(x, words, gs, group, bias)
    assert np.array_equal(np.isnan(y), np.isnan(want))
    ok = ~np.isnan(want)
    assert np.array_equal(bits(y[ok]), bits(want[ok]))
    wg.close()


@pytest.mark.parametrize("rows,k,n", [(1200, 100, 4096), (2500, 576, 2064), (4097, 65, 1304)])
def test_wide_silu_tiles(torch, ctx, rows, k, n):
    """A full wave of tiles: the SiLU * Mul tail through TMA tile stores, ragged rows, a last tile half empty, a row pitch
    wider than the output; bit-equal to the general kernel's tail (the same operations), which an unaligned output takes."""
    from volvoxai_b200 import w8a8
    c = wl.single_linear(rows=rows, k=k, n=n, seed=rows + n)
    weight = w8a8.Weight.from_i8(ctx, c["w"], c["ws"], bias_f32=c["bias"])
    x = dev(torch, c["x"])
    wide = torch.full((rows, n // 2 + 8), 99.0, device="cuda")
    ctx.linear_f32_fused(weight, x, silu_mul=True, out=wide[:, 4:4 + n // 2])
    assert "wide-silu" in w8a8.last_route()
    odd = torch.full((rows, n // 2 + 1), 99.0, device="cuda")
    ctx.linear_f32_fused(weight, x, silu_mul=True, out=odd[:, 1:])
    assert "wide" not in w8a8.last_route()
    assert torch.equal(wide[:, 4:4 + n // 2], odd[:, 1:])
    assert (wide[:, :4] == 99).all() and (wide[:, 4 + n // 2:] == 99).all()
    weight.close()


@pytest.mark.parametrize("rows,k", [(1, 64), (5, 1000), (64, 1024), (700, 576), (40, 9000)])
def test_rmsnorm_products_near_and_far_from_one(torch, ctx, rows, k):
    """The normalized rows against the same arithmetic in 64 bits: ordinary rows, rows scaled to 1e-25 and 1e25, gammas
    of 0, 1e-33 and 1e30."""
    rng = np.random.default_rng(rows + k)
    x = rng.standard_normal((rows, k)).astype(np.float32)
    x[rows // 2] *= np.float32(1e-25)
    x[rows // 3] *= np.float32(1e25 if rows > 3 else 1)
    g = (1 + 0.1 * rng.standard_normal(k)).astype(np.float32)
    g[:4] = 0, 1e-33, 1e30, -1
    y, q, s, v = ctx.rmsnorm_quantize_rows(dev(torch, x), dev(torch, g), 1e-30, ldq=(k + 127) // 128 * 128)
    x64 = x.astype(np.float64)
    want = (x64 / np.sqrt((x64 ** 2).mean(axis=1, keepdims=True) + float(np.float32(1e-30))) * g.astype(np.float64)).astype(np.float32)
    y = y.cpu().numpy()
    # one rounding to fp32 each; a 64-bit rounding can tip it in a handful of elements, by one place
    assert (np.abs(y.view(np.int32).astype(np.int64) - want.view(np.int32)) <= 1).all() and (y != want).mean() <= 1e-4


@pytest.mark.parametrize("tiny,gain", [(1e-33, 1e15), (3e-36, 1e16), (1.35 * 2.0 ** -100, 1.77 * 2.0 ** 60), (1e-38, 1e18)])
@pytest.mark.parametrize("form", ["aligned", "unaligned", "single launch"])
def test_rmsnorm_tiny_elements_under_large_gammas(torch, ctx, form, tiny, gain):
    """Elements whose normalized value x * inv lies near or below the smallest fp32 and comes back into range by a large
    gamma, in rows with an rms of about 1e9: every form of the operator within one place of 64 bits."""
    from volvoxai_b200 import w8a8
    rows, k = 2, 640
    rng = np.random.default_rng(5)
    x = (rng.standard_normal((rows, k)) * 1e9).astype(np.float32)
    g = (1 + 0.1 * rng.standard_normal(k)).astype(np.float32)
    x[:, 7::64] = tiny * rng.uniform(0.5, 2, size=(rows, 10))
    g[7::64] = gain * rng.uniform(0.5, 2, size=10)
    x64 = x.astype(np.float64)
    want = (x64 / np.sqrt((x64 ** 2).mean(axis=1, keepdims=True) + float(np.float32(1e-6))) * g.astype(np.float64)).astype(np.float32)
    if form == "single launch":
        c = wl.single_linear(rows=rows, k=k, n=64, seed=3)
        weight = w8a8.Weight.from_i8(ctx, c["w"], c["ws"])
        y = torch.empty((rows, k), device="cuda")
        ctx.rmsnorm_linear_f32_fused(weight, dev(torch, x), dev(torch, g), 1e-6, norm_out=y)
        assert "decode-fused" in w8a8.last_route()
        weight.close()
    else:
        flat = torch.empty(rows * k + 1, device="cuda")
        at = 1 if form == "unaligned" else 0
        flat[at:at + rows * k] = dev(torch, x).flatten()
        y = ctx.rmsnorm_quantize_rows(flat[at:at + rows * k].view(rows, k), dev(torch, g), 1e-6, ldq=k)[0]
    y = y.cpu().numpy()
    assert (np.abs(bits(y).astype(np.int64) - bits(want).astype(np.int64)) <= 1).all()


@pytest.mark.parametrize("rows,k,n", [(65, 1024, 3080), (100, 1152, 200), (128, 4096, 1000), (66, 64, 4000)])
def test_rows_past_64_in_tiles(torch, ctx, rows, k, n):
    """65 to 128 rows outside the small weights take the tile kernels: every output equal to the decode kernel's."""
    from volvoxai_b200 import w8a8
    c = wl.single_linear(rows=rows, k=k, n=n, seed=rows + k + n)
    weight = w8a8.Weight.from_i8(ctx, c["w"], c["ws"], bias_f32=c["bias"], bias_i32=np.arange(n, dtype=np.int32) * 5 - 300)
    x = dev(torch, c["x"])
    res = torch.randn((rows, n), device="cuda")
    for call in (lambda r: ctx.linear_acc_i32(weight, x, route=r), lambda r: ctx.linear_f32(weight, x, route=r),
                 lambda r: ctx.linear_i8(weight, x, 0.1, -5, route=r)):
        y = call(w8a8.ROUTE_AUTO)
        assert "tcgen05" in w8a8.last_route() and "decode" not in w8a8.last_route()
        assert torch.equal(y, call(w8a8.ROUTE_DECODE))
    assert torch.equal(ctx.linear_f32_fused(weight, x, residual=res), ctx.linear_f32(weight, x, route=w8a8.ROUTE_DECODE) + res)
    weight.close()


@pytest.mark.parametrize("rows,k,n", [(65, 1536, 2050), (97, 1100, 1022), (128, 100, 3090), (80, 1100, 66)])
def test_rows_past_64_in_the_decode_kernel(torch, ctx, rows, k, n):
    """65 to 128 rows where unaligned outputs and the SiLU * Mul tail keep the decode kernel: equal to the tile kernels'."""
    from volvoxai_b200 import w8a8
    c = wl.single_linear(rows=rows, k=k, n=n, seed=rows + k + n)
    weight = w8a8.Weight.from_i8(ctx, c["w"], c["ws"], bias_f32=c["bias"], bias_i32=np.arange(n, dtype=np.int32) * 5 - 300)
    x = dev(torch, c["x"])
    res = torch.randn((rows, n), device="cuda")
    tiles = ctx.linear_f32(weight, x, route=w8a8.ROUTE_TCGEN05)

    def decoded(y):
        assert "decode-rows" in w8a8.last_route()
        return y

    assert torch.equal(decoded(ctx.linear_f32(weight, x)), tiles)
    assert torch.equal(decoded(ctx.linear_acc_i32(weight, x)), ctx.linear_acc_i32(weight, x, route=w8a8.ROUTE_TCGEN05))
    assert torch.equal(decoded(ctx.linear_f32_fused(weight, x, residual=res)), tiles + res)
    s = decoded(ctx.linear_f32_fused(weight, x, silu_mul=True)).double()
    g, u = tiles[:, 0::2].double(), tiles[:, 1::2].double()
    y = g / (1.0 + torch.exp(-g)) * u
    assert (s - y).abs().le(1e-6 * y.abs() + 1e-30).all()      # four roundings and an expf of at most 2 ulp
    y8 = ctx.linear_i8(weight, x, 0.1, -5)
    assert torch.equal(y8, ctx.linear_i8(weight, x, 0.1, -5, route=w8a8.ROUTE_TCGEN05))
    weight.close()


def test_native_and_ctypes_calls_agree(torch, ctx, monkeypatch):
    """The eight device calls in both forms, and with outputs, residuals and norm weights that are not torch's."""
    from tests.test_torch_calls import Memory
    from volvoxai_b200 import w8a8
    rows, k, n = 9, 300, 66
    c = wl.single_linear(rows=rows, k=k, n=n, seed=1)
    weight = w8a8.Weight.from_i8(ctx, c["w"], c["ws"], bias_f32=c["bias"], bias_i32=np.arange(n, dtype=np.int32))
    x, res = dev(torch, c["x"]), torch.randn((rows, n), device="cuda")
    gamma = torch.rand(k, device="cuda") + 0.5
    q = torch.randint(-128, 128, (rows, k), dtype=torch.int8, device="cuda")
    outs = {"y": torch.empty((rows, n), device="cuda"), "norm": torch.empty((rows, k), device="cuda")}

    def memory(t):
        return Memory(t.data_ptr(), t.stride(0))

    def into(call):
        for t in outs.values():
            t.zero_()
        call()
        return torch.cat([t.flatten() for t in outs.values()])

    calls = [lambda: ctx.linear_f32(weight, x), lambda: ctx.linear_f32_fused(weight, x, residual=res), lambda: ctx.linear_f32_fused(weight, x, silu_mul=True),
             lambda: ctx.rmsnorm_linear_f32_fused(weight, x, gamma, 1e-6), lambda: ctx.linear_i8(weight, x, 0.1, 3),
             lambda: ctx.qlinear_device(weight, q, 0.05, -3, 0.5, 4, out_unsigned=True), lambda: ctx.quantize_linear(x, 0.1, 5),
             lambda: ctx.dequantize_linear(q, 0.1, 5), lambda: ctx.requantize_linear(q, 0.1, 5, 0.2, 7, unsigned=True)]
    native = [call() for call in calls]
    native.append(into(lambda: ctx.rmsnorm_linear_f32_fused(weight, x, gamma, 1e-6, norm_out=outs["norm"], out=outs["y"])))
    assert torch.equal(native[-1], into(lambda: ctx.rmsnorm_linear_f32_fused(weight, x, memory(gamma), 1e-6, norm_out=memory(outs["norm"]), out=memory(outs["y"]))))
    assert torch.equal(into(lambda: ctx.linear_f32_fused(weight, x, residual=memory(res), out=outs["y"]))[:rows * n], native[1].flatten())
    assert torch.equal(into(lambda: ctx.linear_f32(weight, x, out=memory(outs["y"])))[:rows * n], native[0].flatten())
    monkeypatch.setattr(w8a8, "_torch_calls", None)
    for call, want in zip(calls, native):
        got = call()
        assert got.dtype == want.dtype and torch.equal(got, want)
    weight.close()


@pytest.mark.parametrize("captured", [False, True])
def test_small_calls_back_to_back(torch, ctx, captured):
    """Calls on both sides of the line up to which the quantizer lets its GEMM in before its own wait, and single-launch
    calls on both sides of theirs, one after the other through one context's scratch without a pause, in a stream and
    replayed from a graph: each output as when it is computed alone."""
    from volvoxai_b200 import w8a8
    shapes = [(6, 640, 1472), (8, 128, 300), (64, 1024, 1000), (16, 1024, 1000), (1, 576, 128), (3, 257, 64), (1, 576, 300), (33, 576, 200),
              (128, 128, 600), (2, 1024, 64), (7, 2048, 500)]
    weights, xs, want, outs = [], [], [], []
    for i, (rows, k, n) in enumerate(shapes):
        c = wl.single_linear(rows=rows, k=k, n=n, seed=i)
        weights.append(w8a8.Weight.from_i8(ctx, c["w"], c["ws"], bias_f32=c["bias"]))
        xs.append(dev(torch, c["x"]))
        want.append(ctx.linear_f32(weights[i], xs[i], route=w8a8.ROUTE_SIMT))
        outs.append(torch.empty_like(want[i]))
        torch.cuda.synchronize()

    def all_calls():
        for w, x, y in zip(weights, xs, outs):
            ctx.linear_f32(w, x, out=y)

    stream = torch.cuda.Stream()
    ctx.set_stream(stream.cuda_stream)
    try:
        with torch.cuda.stream(stream):
            all_calls()
            stream.synchronize()
            graph = torch.cuda.CUDAGraph()
            if captured:
                with torch.cuda.graph(graph, stream=stream):
                    all_calls()
            for _ in range(20):
                for y in outs:
                    y.zero_()
                graph.replay() if captured else all_calls()
                stream.synchronize()
                for y, ref in zip(outs, want):
                    assert torch.equal(y, ref)
    finally:
        ctx.set_stream(None)
    for w in weights:
        w.close()
