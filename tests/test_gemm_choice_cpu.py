"""Which kernel and tile the expert GEMMs take: the rules, which need no GPU."""
import pytest

from deepep_efa_b200 import _ext

C = _ext.load()


@pytest.mark.parametrize("rows,groups,n,k,swiglu,how,columns", [
    # few K blocks: a wide tile costs twice a narrow one (us, 128 / 256 columns: 9.4 / 12.2, 37.5 / 43.7, 26.1 / 32.0)
    (16 * 256, 16, 1280, 128, False, {}, 128),
    (16 * 512, 16, 1280, 1024, True, {}, 128),
    (8 * 512, 8, 4096, 512, False, {}, 128),
    # the same layers with more of them (108 / 97, 187 / 154)
    (16 * 512, 16, 2560, 4096, True, {}, 256),
    (8 * 512, 8, 4096, 7168, False, {}, 256),
    # tiles that are dealt out at once either way
    (8 * 128, 8, 1024, 7168, True, {}, 128),
    # room for 128 rows in every group, nothing said about how many come: two groups in use 32.2 / 39.9, so narrow as without a choice
    (32 * 128, 32, 2560, 7168, True, dict(ends=True), 128),
    (32 * 128, 32, 2560, 7168, True, dict(ends=True, rows_hint=4), 128),
    (32 * 128, 32, 2560, 7168, True, dict(ends=True, rows_hint=1000), 256),
    # 16 groups of 111 rows each fill 48 tiles, not the 87 of a tile too many per group (11.6 / 16.6)
    (16 * 512, 16, 768, 1280, True, dict(ends=True, rows_hint=1776), 128),
    # a plan whose tiles are all in use says so
    (64 * 128, 64, 2816, 4096, True, dict(ends=True, rows_hint=64 * 128), 256),
    (64 * 128, 64, 4096, 1408, False, dict(ends=True, rows_hint=64 * 128), 256),
    # tiles with few rows in them (118 / 116 for the layer of 300 tokens), and with many
    (60 * 512, 60, 2048, 512, False, dict(ends=True, rows_hint=600), 256),
    (60 * 512, 60, 2048, 384, False, dict(ends=True, rows_hint=60 * 120), 128),
    # groups of 100 rows fill 32 tiles, though there are rows for 25 (38.9 / 46.5)
    (32 * 100, 32, 2560, 1024, True, {}, 128),
    # an odd number of 128 columns
    (64 * 512, 64, 4096 + 128, 4096, False, {}, 128),
])
def test_promotion_tile_width(rows, groups, n, k, swiglu, how, columns):
    assert C.promotion_columns(rows, groups, n, k, swiglu, **how) == columns


@pytest.mark.parametrize("rows,groups,n,k,how,form", [
    # few K blocks stay rows, as pairs where two tiles of rows are full (us, rows / columns: 11.6 / 15.9, 7.4 / 11.6, 124 / 132)
    (64 * 256, 64, 512, 256, {}, "row pairs"),
    (64 * 300, 64, 512, 256, {}, "rows"),
    (64 * 128, 64, 512, 128, dict(ends=True, zero_tail=True), "rows"),
    (64 * 800, 64, 1408, 512, dict(mn_major=True), "row pairs"),
    # two rounds of small tiles against one of large ones (16.3 / 19.2; 18.2 / 20.2), and a single one of either (13.9 / 12.0)
    (64 * 100, 64, 512, 1024, dict(mn_major=True), "rows"),
    (64 * 128, 64, 512, 1024, dict(ends=True, zero_tail=True), "rows"),
    (8 * 128, 8, 2048, 1024, dict(ends=True, zero_tail=True), "columns 128"),
    # half of an odd last tile of 256 features is empty (41 / 47; 29.4 / 42.7)
    (64 * 210, 64, 128, 5056, dict(ends=True, zero_tail=True), "rows"),
    # the layers of the training step
    (64 * 128, 64, 2816, 4096, dict(ends=True, zero_tail=True), "columns 128"),
    (64 * 128, 64, 4096, 1408, dict(ends=True, zero_tail=True), "columns 128"),
    (64 * 832, 64, 4096, 1408, dict(ends=True, zero_tail=True), "columns 256"),
    (64 * 832, 64, 1408, 4096, dict(mn_major=True, ends=True, zero_tail=True), "columns 256"),
    # a layout with room for more rows than come
    (64 * 256, 64, 1408, 512, dict(ends=True), "rows"),
    (64 * 256, 64, 1408, 2048, dict(ends=True), "columns 256"),
    (64 * 128, 64, 512, 1024, dict(ends=True), "rows"),
    (160 * 128, 160, 128, 2240, dict(ends=True), "rows"),
    # what the columns' kernel does not take, and one SM
    (8 * 512, 8, 192, 4096, {}, "row pairs"),
    (8 * 512, 8, 256, 4096, dict(num_sms=1), "rows"),
])
def test_form_of_bf16_products(rows, groups, n, k, how, form):
    assert C.bf16_form(rows, groups, n, k, **how) == form


@pytest.mark.parametrize("swiglu,how", [(True, {}), (False, {}), (True, dict(ends=True, rows_hint=64 * 512))])
def test_promotion_without_registers_for_wide_tiles(swiglu, how):
    """A build whose 256-column kernel did not get the registers that its warps move between them takes 128 columns, which compute the same."""
    size = (64 * 512, 64, 4096, 4096, swiglu)
    assert C.promotion_columns(*size, **how) == 256
    assert C.promotion_columns(*size, fits=False, **how) == 128
