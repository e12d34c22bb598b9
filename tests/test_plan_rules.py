"""Where the automatic routes change over (no GPU): each rule at its line and on both sides of it."""
import pytest

from volvoxai_b200 import _lib, w8a8


def pick(rows, k, n, **kw):
    plan, why = w8a8.plan(rows, k, n, sm_count=148, **kw)
    assert plan is not None, why
    return plan


@pytest.mark.parametrize("rows,k,n,decode", [(64, 4096, 14336, True), (65, 1024, 3072, True), (128, 1024, 3073, False), (65, 1025, 64, False),
                                             (128, 576, 64, True)])
def test_rows_past_64_keep_the_decode_kernel_for_small_weights_only(rows, k, n, decode):
    for epilogue in (_lib.EPI_ACC, _lib.EPI_F32, _lib.EPI_I8):
        assert (pick(rows, k, n, epilogue=epilogue)["id"] == "DECODE_ROWS") == decode


@pytest.mark.parametrize("kw,inside,outside", [
    ({"out_store_aligned": False}, [(128, 1536, 4736), (80, 1536, 9472), (65, 100, 5000)], [(65, 1537, 1024), (81, 64, 4737), (80, 64, 9473)]),
    ({"out_store_aligned": False, "epilogue": _lib.EPI_ACC}, [(124, 1152, 3224)], [(66, 1537, 64)]),
    ({"out_store_aligned": False, "epilogue": _lib.EPI_I8}, [(80, 768, 4736), (128, 512, 4736)], [(128, 512, 4737), (65, 512, 4737), (80, 896, 3073), (65, 1025, 64)]),
    ({"out_store_aligned": True, "epilogue": _lib.EPI_I8}, [(128, 1024, 3072)], [(65, 128, 3073)]),
    ({"fused_tail": 2}, [(128, 1536, 4736), (96, 576, 9472)], [(97, 1536, 4738), (65, 1664, 1024), (65, 64, 9474)]),
    ({"fused_tail": 2, "out_store_aligned": False}, [(96, 1024, 6000)], [(97, 1024, 6000)]),
])
def test_rows_past_64_by_what_the_output_costs_in_tiles(kw, inside, outside):
    """Unaligned outputs and the SiLU * Mul tail keep the decode kernel further than the small weights above."""
    for shape in inside:
        assert pick(*shape, **kw)["id"] == "DECODE_ROWS", shape
    for shape in outside:
        assert pick(*shape, **kw)["id"] != "DECODE_ROWS", shape
    for rows, k, n in inside + outside:
        assert pick(64, k, n, **kw)["id"] == "DECODE_ROWS" and pick(129, k, n, **kw)["id"] != "DECODE_ROWS"


@pytest.mark.parametrize("rows,k,n,want", [(512, 4096, 4096, "TCGEN05_PAIR_NARROW"), (1024, 4096, 4096, "TCGEN05"), (2048, 4096, 4096, "TCGEN05_PAIR"),
                                           (512, 1536, 4096, "TCGEN05"), (512, 1537, 4096, "TCGEN05_PAIR_NARROW")])
def test_long_k_takes_the_cheapest_waves(rows, k, n, want):
    assert pick(rows, k, n, epilogue=_lib.EPI_I8)["id"] == want
    plan = pick(rows, k, n, epilogue=_lib.EPI_I8, pair_clusters=0)
    assert plan["id"] == "TCGEN05"


def test_silu_tail_from_a_full_wave_of_tiles():
    assert pick(4096, 576, 3072, fused_tail=2)["id"] == "TCGEN05_WIDE_SILU"
    assert pick(1280, 576, 3584, fused_tail=2)["id"] == "TCGEN05"                  # 140 tiles
    assert pick(1408, 576, 3584, fused_tail=2)["id"] == "TCGEN05_WIDE_SILU"        # 154
    assert pick(4096, 576, 3072, fused_tail=2, out_store_aligned=False)["id"] == "TCGEN05_PAIR"
    assert pick(4096, 1537, 3072, fused_tail=2)["id"] == "TCGEN05_PAIR"


@pytest.mark.parametrize("rows,n,tile", [(64, 14336, (64, 128)), (8, 14336, (16, 128)), (8, 9472, (16, 64)), (17, 9473, (32, 128)), (65, 4096, (128, 128))])
def test_grouped_rows_up_to_64_have_the_weights_as_m(rows, n, tile):
    plan = pick(rows, 4096, n, weight_kind=_lib.WEIGHT_GROUPED, group_size=128)
    assert plan["id"] == "GROUPED_TCGEN05" and (plan["tile_rows"], plan["tile_columns"]) == tile


@pytest.mark.parametrize("rows,k,per_row", [(64, 1024, 256), (148, 1024, 256), (149, 1024, 128), (296, 1024, 128), (297, 1024, 64), (2368, 1024, 64),
                                            (2369, 1024, 32), (777, 576, 32), (300, 576, 64), (592, 576, 64), (593, 576, 32), (4736, 256, 32), (4737, 256, 8),
                                            (64, 124, 8), (64, 128, 32), (1184, 128, 32), (1185, 128, 8), (592, 4096, 256), (593, 4096, 128),
                                            (40, 8192, 256)])
def test_quantizer_threads_per_row(rows, k, per_row):
    """Doubled while the launch stays within 256 threads per SM and a thread keeps a float4, or within 1024 and it keeps four
    (two at K up to 256)."""
    plan = pick(rows, k, 4096, fp32_input=True)
    assert plan["quantizer"] == 2 and plan["quantizer_grid"] == -(-rows // (256 // per_row))


@pytest.mark.parametrize("rows,k,n,want", [(4, 8192, 1536, "GEMV_GROUPED"), (3, 8192, 1537, "GROUPED_TCGEN05"), (4, 8191, 4000, "GEMV_GROUPED"), (4, 14336, 2048, "GROUPED_TCGEN05"),
                                           (2, 14336, 4096, "GEMV_GROUPED"), (4, 8191, 4097, "GROUPED_TCGEN05")])
def test_three_and_four_grouped_rows(rows, k, n, want):
    assert pick(rows, k, n, weight_kind=_lib.WEIGHT_GROUPED, group_size=128)["id"] == want
