"""The rule for the tiles of plain products (the products themselves are tested on the GPU)."""
import pytest

from fbamtrain_b200.ops import native as nv


@pytest.fixture
def columns():
    if not nv.available():
        pytest.skip("kernel library not built")
    lib = nv.lib()
    yield lambda m, n, max_ctas, a_mn=0: lib.fbam_gemm_tile_columns(m, n, max_ctas, a_mn)
    lib.fbam_set_reserved_sms(0)


def test_narrow_tiles_fit_the_ctas_of_the_launch(columns):
    """9 x 16 tiles of 64 columns: one wave of the whole machine, two of what a pipeline rank or a limited launch may use."""
    assert columns(9 * 128, 16 * 64, 0) == 64
    assert columns(9 * 128, 16 * 64, 144) == 64
    assert columns(9 * 128, 16 * 64, 143) == 128
    assert columns(9 * 128, 16 * 64, 71) == 256
    assert columns(9 * 128, 16 * 64, 500) == 64
    assert columns(9 * 128, 32 * 64, 0) == 128 and columns(9 * 128, 64 * 64, 0) == 256
    assert nv.lib().fbam_set_reserved_sms(16) == 0
    assert columns(9 * 128, 16 * 64, 0) == 128
    assert columns(9 * 128, 32 * 64, 0) == 256
    assert columns(9 * 128, 14 * 64, 0) == 64


@pytest.mark.parametrize("n,wide", [(8, 64), (64, 64), (72, 128), (128, 128), (136, 256), (4096, 256)])
def test_many_rows_take_the_tile_that_the_columns_fill(columns, n, wide):
    """More tiles than CTAs: 64 columns and fewer used to be padded to 128 there."""
    assert columns(200 * 128, n, 0) == wide


@pytest.mark.parametrize("m,a_mn,few", [(1, 0, True), (8, 0, True), (9, 0, False), (32, 1, True), (33, 1, False)])
def test_very_few_rows_take_some_forty_tiles(columns, m, a_mn, few):
    """148, 64 and 32 tiles of 64 columns."""
    assert [columns(m, n, 0, a_mn) for n in (9472, 4096, 2048)] == ([256, 128, 64] if few else [64, 64, 64])
    assert columns(m, 9472, 36, a_mn) == 256
