"""Which kernel and which pipeline shape a single copy takes: by size and alignment, and by whether it stays in one GPU's memory."""
import pytest

KiB, MiB = 1 << 10, 1 << 20
LOCAL = (32 * KiB, 4, 2, 0)
LINK, LINK_LARGE = (16 * KiB, 4, 1, 0), (32 * KiB, 4, 2, 1)


@pytest.mark.parametrize("n,local,link", [(1, None, None), (4 * MiB - 1, None, None), (4 * MiB, None, LINK), (24 * MiB - 1, None, LINK), (24 * MiB, LOCAL, LINK),
                                          (256 * MiB - 1, LOCAL, LINK), (256 * MiB, LOCAL, LINK_LARGE), (3 << 30, LOCAL, LINK_LARGE)])
@pytest.mark.parametrize("rel", [0, 1, 8])
def test_route(mf, n, local, link, rel):
    base = 1 << 40
    for off in (0, 5):
        assert mf.native.xcopy_shape(base + off + rel, 2 * base + off, n, True) == (local if rel == 0 else None)
        assert mf.native.xcopy_shape(base + off + rel, 2 * base + off, n, False) == (link if rel == 0 else None)
