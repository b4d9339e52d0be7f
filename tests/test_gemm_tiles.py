"""How wide the grouped GEMMs make their tiles: a rule on the sizes and on how many CTAs run, not on one chip's SM count."""
import pytest


def _ops():
    from memfabric_hybrid_b200._loader import _pymf

    return _pymf.ops


@pytest.mark.parametrize("ctas", [1, 20, 74, 132, 148])
def test_wide_tiles_when_every_cta_gets_two(mf, ctas):
    ops = _ops()
    G, N = 4, 2048
    first = -(-2 * ctas // (N // 256))  # m-tiles from which there are two wide tiles per CTA
    for m in (first - 1, first, first + 1):
        if m < 2 * G:
            continue
        want = 256 if m >= first else 128
        assert ops.gemm_tile(G, m * 128, N, ctas) == want
        assert ops.gemm_tile(G, m * 128 - 127, N, ctas) == want
        assert ops.gemm_mx_tile(G, m * 128, N, ops.GEMM_EPI_BF16, ctas) == want
        assert ops.gemm_mx_tile(G, m * 128, N, ops.GEMM_EPI_SWIGLU_FP8 | ops.GEMM_B_PACKED, ctas) == want


def test_other_conditions(mf):
    ops = _ops()
    assert ops.gemm_tile(4, 1 << 20, 2048 + 128, 148) == 128  # no whole wide tiles
    assert ops.gemm_tile(64, 127 * 128, 1 << 14, 148) == 128  # fewer than two m-tiles per group
    assert ops.gemm_mx_tile(64, 64 * 128, 7168, ops.GEMM_EPI_BF16, 148) == 224  # one m-tile per group
    assert ops.gemm_mx_tile(64, 65 * 128, 7168, ops.GEMM_EPI_BF16, 148) == 256
    assert ops.gemm_mx_tile(64, 64 * 128, 7168, ops.GEMM_EPI_SWIGLU, 148) == 256
    assert ops.gemm_mx_tile(8, 8 * 128, 7168, ops.GEMM_EPI_BF16, 148) == 128  # 8 x 32 tiles of 224 columns are fewer than 2 x 148
    assert ops.gemm_mx_tile(8, 8 * 128, 7168, ops.GEMM_EPI_BF16, 128) == 224  # but not fewer than 2 x 128
