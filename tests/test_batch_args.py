"""Batch copies on a CPU-only pool: how the address lists may be handed over, and placement of elements that follow one another
in the same backed range, leave it, or leave the pool."""
import numpy as np
import pytest

from conftest import free_port

MiB = 1 << 20


@pytest.fixture(scope="module")
def pool():
    from memfabric_hybrid_b200.parallel.pool import open_pool

    p = open_pool(0, 1, -1, 0, dram_bytes=8 * MiB, store_url=f"tcp://127.0.0.1:{free_port()}")
    yield p
    p.close()


def _fill(addr, n, seed):
    from memfabric_hybrid_b200.utils.tensors import host_array_from_gva

    view = host_array_from_gva(addr, n)
    view[:] = np.random.default_rng(seed).integers(0, 256, n, dtype=np.uint8)
    return view


@pytest.mark.parametrize("make", [list, tuple, lambda v: np.array(v, dtype=np.uint64), lambda v: [np.uint64(x) for x in v]])
@pytest.mark.parametrize("count", [1, 2, 400])
def test_sequences(mf, pool, make, count):
    base = pool.dram()
    src = _fill(base, 64 * count, count)
    dst = _fill(base + 4 * MiB, 64 * count, count + 1)
    order = np.random.default_rng(3).permutation(count)
    srcs = make([base + 64 * i for i in range(count)])
    dsts = make([base + 4 * MiB + 64 * int(i) for i in order])
    assert pool.handle.copy_data_batch(srcs, dsts, make([64] * count), count, mf.bm.BmCopyType.G2G, 0) == 0, mf.get_last_err_msg()
    assert (dst.reshape(count, 64)[order] == src.reshape(count, 64)).all()


@pytest.mark.parametrize("bad", [[-1], ["a"], [1 << 64], [1.5], 7, None])
def test_what_is_no_sequence_of_addresses_raises(mf, pool, bad):
    with pytest.raises(TypeError):
        pool.handle.copy_data_batch(bad, [pool.dram()], [64], 1, mf.bm.BmCopyType.G2G, 0)


@pytest.mark.parametrize("at", [0, 1, 5])
@pytest.mark.parametrize("side", ["src", "dst"])
def test_one_element_outside_refuses_the_batch(mf, pool, at, side):
    """The element that leaves the pool by its last byte is found behind elements that stay inside; nothing is copied."""
    base = pool.dram()
    src, dst = _fill(base, 6 * 64, 1), _fill(base + 4 * MiB, 6 * 64, 2)
    before = dst.copy()
    srcs, dsts = [base + 64 * i for i in range(6)], [base + 4 * MiB + 64 * i for i in range(6)]
    (srcs if side == "src" else dsts)[at] = base + 8 * MiB - 63
    assert pool.handle.copy_data_batch(srcs, dsts, [64] * 6, 6, mf.bm.BmCopyType.G2G, 0) != 0
    assert (dst == before).all()
    assert src.size == 6 * 64


@pytest.mark.parametrize("pattern", ["llgg", "glgl", "gggl", "lggg"])
def test_elements_of_several_groups_keep_their_data(mf, pool, pattern):
    """Pool and ordinary host memory alternate on the source side: runs of one group, switches back and forth."""
    base = pool.dram()
    local = np.random.default_rng(8).integers(0, 256, 64 * 12, dtype=np.uint8)
    pooled = _fill(base, 64 * 12, 9)
    dst = _fill(base + 4 * MiB, 64 * 12, 10)
    kinds = (pattern * 3)[:12]
    srcs = [local.ctypes.data + 64 * i if k == "l" else base + 64 * i for i, k in enumerate(kinds)]
    assert pool.handle.copy_data_batch(srcs, [base + 4 * MiB + 64 * i for i in range(12)], [64] * 12, 12, mf.bm.BmCopyType.AUTO, 0) == 0
    for i, k in enumerate(kinds):
        want = local if k == "l" else pooled
        assert (dst[64 * i:64 * i + 64] == want[64 * i:64 * i + 64]).all(), i


@pytest.mark.parametrize("kind,per_element", [("local", 3), ("registered", 4), ("pool_then_registered", 3)])
def test_placing_elements_that_share_no_range_costs_their_own_look_ups(mf, pool, kind, per_element):
    """Elements with a side outside the pool's windows are placed one by one. Per element: two look-ups for the class of a side
    outside the windows and its owner, and one per side that has to lie in the pool; none for remembering ranges that are of no use."""
    n = 200
    base = pool.dram()
    outside = np.random.default_rng(11).integers(0, 256, 64 * n, dtype=np.uint8)
    inside = _fill(base, 64 * n, 12)
    dst = _fill(base + 4 * MiB, 64 * n, 13)
    if kind != "local":
        assert pool.handle.register(outside.ctypes.data, outside.size) == 0, mf.get_last_err_msg()
    try:
        from_pool = [kind == "pool_then_registered" and i % 2 == 0 for i in range(n)]
        srcs = [base + 64 * i if p else outside.ctypes.data + 64 * i for i, p in enumerate(from_pool)]
        before = mf.native.va_lookups()
        assert pool.handle.copy_data_batch(srcs, [base + 4 * MiB + 64 * i for i in range(n)], [64] * n, n, mf.bm.BmCopyType.AUTO, 0) == 0
        assert mf.native.va_lookups() - before <= per_element * n + 8
        for i, p in enumerate(from_pool):
            assert (dst[64 * i:64 * i + 64] == (inside if p else outside)[64 * i:64 * i + 64]).all(), i
    finally:
        if kind != "local":
            assert pool.handle.unregister(outside.ctypes.data) == 0
