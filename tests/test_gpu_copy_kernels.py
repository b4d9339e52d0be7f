"""Edges of the copy kernels on one GPU, bytes against bytes: vectors put together from two neighbours at every relative alignment,
tiles and their remainders, batches around the list lengths at which a launch takes a larger parameter block or a further piece,
chunk remainders, batches that are not aligned, and an enqueued copy that follows the copy which writes its source."""
import numpy as np
import pytest

from conftest import free_port

pytestmark = pytest.mark.gpu

KiB, MiB = 1 << 10, 1 << 20


@pytest.fixture(scope="module")
def pool():
    import torch

    from memfabric_hybrid_b200.parallel.pool import open_pool

    torch.cuda.set_device(0)
    p = open_pool(0, 1, 0, 192 * MiB, store_url=f"tcp://127.0.0.1:{free_port()}")
    yield p
    p.close()


def _regions(pool, n):
    import torch

    from memfabric_hybrid_b200.utils.tensors import device_tensor_from_gva

    src, dst = device_tensor_from_gva(pool.hbm(), n), device_tensor_from_gva(pool.hbm() + 96 * MiB, n)
    src.random_(0, 256, generator=torch.Generator(device="cuda").manual_seed(n & 0xFFFF))
    dst.fill_(0xA5)
    torch.cuda.synchronize()
    return src, dst


@pytest.mark.parametrize("rel", range(16))
@pytest.mark.parametrize("n", [31, 8 * KiB + 1, 148 * 2 * 8 * KiB + 17, 20 * MiB + 5])
def test_every_relative_alignment(mf, pool, rel, n):
    import torch

    src, dst = _regions(pool, n + 64)
    for doff in (0, 5):
        dst.fill_(0xA5)
        torch.cuda.synchronize()
        soff = (rel + doff) % 16
        assert pool.handle.copy_data(pool.hbm() + soff, pool.hbm() + 96 * MiB + 16 + doff, n, mf.bm.BmCopyType.G2G, 0) == 0, mf.get_last_err_msg()
        lo = 16 + doff
        assert torch.equal(dst[lo:lo + n], src[soff:soff + n])
        assert bool((dst[:lo] == 0xA5).all()) and bool((dst[lo + n:] == 0xA5).all())


@pytest.mark.parametrize("n", [24 * MiB - 16, 24 * MiB, 24 * MiB + 16, 32 * KiB * 148 * 5 + 48])
def test_both_sides_of_the_bulk_copy_threshold(mf, pool, n):
    import torch

    src, dst = _regions(pool, n + 64)
    assert pool.handle.copy_data(pool.hbm() + 7, pool.hbm() + 96 * MiB + 23, n, mf.bm.BmCopyType.G2G, 0) == 0, mf.get_last_err_msg()
    assert torch.equal(dst[23:23 + n], src[7:7 + n])
    assert bool((dst[:23] == 0xA5).all()) and bool((dst[23 + n:] == 0xA5).all())


def _batch(rng, count, unit, top, aligned=16):
    """Blocks of 1..top units in a shuffled order with gaps between them: offsets and sizes in bytes."""
    sizes = (rng.integers(1, top + 1, count) * unit).astype(np.int64)
    slot = top * unit + 32
    offs = rng.permutation(count).astype(np.int64) * slot + rng.integers(0, 2, count) * aligned
    return offs, sizes, slot * count


@pytest.mark.parametrize("stream", [False, True])
@pytest.mark.parametrize("unit,top", [(16, 3), (16, 600), (8 * KiB, 1), (4112, 7)])
@pytest.mark.parametrize("count", [1, 2, 32, 33, 168, 169, 504, 505, 504 + 1344, 504 + 1344 + 1, 3000])
def test_bulk_batches(mf, pool, count, unit, top, stream):
    import torch

    if count * (top * unit + 32) > 90 * MiB:
        pytest.skip("larger than the region")
    rng = np.random.default_rng(count * 7 + unit)
    so, sizes, span = _batch(rng, count, unit, top)
    do = rng.permutation(count).astype(np.int64) * (top * unit + 32)
    src, dst = _regions(pool, span + 64)
    srcs, dsts = [int(pool.hbm() + o) for o in so], [int(pool.hbm() + 96 * MiB + o) for o in do]
    szs = [int(z) for z in sizes]
    if stream:
        assert pool.handle.copy_data_batch_on_stream(srcs, dsts, szs, mf.bm.BmCopyType.G2G, torch.cuda.current_stream().cuda_stream, 0) == 0
        torch.cuda.synchronize()
    else:
        assert pool.handle.copy_data_batch(srcs, dsts, szs, count, mf.bm.BmCopyType.G2G, 0) == 0, mf.get_last_err_msg()
    s, d = src.cpu().numpy(), dst.cpu().numpy()
    want = np.full_like(d, 0xA5)
    for a, b, z in zip(so, do, sizes):
        want[b:b + z] = s[a:a + z]
    assert (d == want).all()


@pytest.mark.parametrize("count", [3, 168, 169, 1000])
@pytest.mark.parametrize("shift", [1, 2, 8])
def test_batches_off_the_16_byte_grid(mf, pool, count, shift):
    rng = np.random.default_rng(count + shift)
    so, sizes, span = _batch(rng, count, 100, 50, aligned=shift)
    do = rng.permutation(count).astype(np.int64) * (50 * 100 + 32)
    src, dst = _regions(pool, span + 64)
    assert pool.handle.copy_data_batch([int(pool.hbm() + o) for o in so], [int(pool.hbm() + 96 * MiB + o) for o in do], [int(z) for z in sizes], count,
                                       mf.bm.BmCopyType.G2G, 0) == 0, mf.get_last_err_msg()
    s, d = src.cpu().numpy(), dst.cpu().numpy()
    want = np.full_like(d, 0xA5)
    for a, b, z in zip(so, do, sizes):
        want[b:b + z] = s[a:a + z]
    assert (d == want).all()


@pytest.mark.parametrize("kind", ["small", "shifted", "bulk", "batch"])
def test_enqueued_copies_keep_stream_order(mf, pool, kind):
    """Forty hops, each reading what the one before wrote: a copy that overlaps its predecessor's end must not read too early."""
    import torch

    from memfabric_hybrid_b200.utils.tensors import device_tensor_from_gva

    n = {"small": 3000, "shifted": 3 * MiB + 1, "bulk": 25 * MiB, "batch": 8 * MiB}[kind]
    step = 2 if kind == "shifted" else 0
    base, hop, G2G = pool.hbm(), 40 * MiB, mf.bm.BmCopyType.G2G
    first = device_tensor_from_gva(base, n)
    first.random_(0, 256, generator=torch.Generator(device="cuda").manual_seed(4))
    want = first.clone()
    st = torch.cuda.current_stream().cuda_stream
    at = base
    for i in range(40):
        to = base + (hop if i % 2 == 0 else 0) + step * (i + 1)
        if kind == "batch":
            blk = n // 2048
            order = np.random.default_rng(i).permutation(2048)
            rc = pool.handle.copy_data_batch_on_stream([int(at + o * blk) for o in order], [int(to + o * blk) for o in order], [blk] * 2048, G2G, st, 0)
        else:
            rc = pool.handle.copy_data_on_stream(at, to, n, G2G, st, 0)
        assert rc == 0, mf.get_last_err_msg()
        at = to
    torch.cuda.synchronize()
    assert torch.equal(device_tensor_from_gva(at, n), want)


@pytest.mark.parametrize("form", ["single", "batch", "engine"])
def test_a_copy_without_a_stream_does_not_wait_for_the_default_stream(mf, pool, form):
    """Buffers of the caller's own device memory are copied while the default stream is busy with something else."""
    import torch

    n = {"single": 512 * KiB, "batch": 512 * KiB, "engine": 8 * MiB}[form]
    mine = torch.randint(0, 256, (n,), dtype=torch.uint8, device="cuda")
    host = torch.empty(n, dtype=torch.uint8).pin_memory()
    to, T = pool.hbm() + 4 * MiB, mf.bm.BmCopyType
    busy = torch.cuda.Event()
    for turn in range(2):  # the first round loads the kernels
        torch.cuda.synchronize()
        torch.cuda._sleep(2000 if turn == 0 else 600_000_000)  # at least 0.3 s
        busy.record()
        if form == "batch":
            rc = pool.handle.copy_data_batch([mine.data_ptr() + i * 4096 for i in range(n // 4096)], [to + i * 4096 for i in range(n // 4096)][::-1],
                                             [4096] * (n // 4096), n // 4096, T.L2G, 0)
        else:
            rc = pool.handle.copy_data(mine.data_ptr(), to, n, T.L2G, 0)
            if form == "engine":
                rc |= pool.handle.copy_data(to, host.data_ptr(), n, T.G2H, 0)
        still = not busy.query()
        assert rc == 0, mf.get_last_err_msg()
    assert still, "the copy waited for the default stream"
    torch.cuda.synchronize()


@pytest.mark.parametrize("polls", [-1, 0])
@pytest.mark.parametrize("kernel", ["single", "batch"])
def test_a_bulk_copy_that_gives_up_waiting_says_so(mf, pool, kernel, polls):
    """With a limit of no polls at all the first wait for a load runs out; the loads that are on their way are waited for, the word is
    set and the kernel ends. With the ordinary limit everything arrives and the word stays as it was."""
    import torch

    n = 26 * MiB
    src, dst = _regions(pool, n)
    fault = torch.zeros(1, dtype=torch.int32).pin_memory()
    st = torch.cuda.current_stream().cuda_stream
    if kernel == "single":
        rc = mf.native.xcopy_shaped(dst.data_ptr(), src.data_ptr(), n, 32 * KiB, 4, 2, 0, 0, st, polls, fault.data_ptr())
    else:
        blk = n // 416
        rc = mf.native.batch_bulk([src.data_ptr() + i * blk for i in range(416)], [dst.data_ptr() + i * blk for i in range(416)], [blk] * 416, st, polls,
                                  fault.data_ptr())
    assert rc == 0
    torch.cuda.synchronize()
    assert int(fault[0]) == (1 if polls == 0 else 0)
    assert torch.equal(dst, src) == (polls != 0)
    # the context is as usable as before
    assert pool.handle.copy_data(pool.hbm(), pool.hbm() + 96 * MiB, n, mf.bm.BmCopyType.G2G, 0) == 0 and torch.equal(dst, src)


@pytest.mark.parametrize("n", [8 * KiB + 5, 24 * KiB + 1, 64 * KiB + 3, 256 * KiB + 1])
@pytest.mark.parametrize("step", [1, 2, 7])
def test_short_shifted_copies_keep_stream_order(mf, pool, n, step):
    """Grids of a few CTAs, of which several copies are resident at once, read through the L1 what the copies just before them wrote
    over the data that still older ones had read: other data every round."""
    import torch

    from memfabric_hybrid_b200.utils.tensors import device_tensor_from_gva

    base, hop, G2G = pool.hbm(), MiB, mf.bm.BmCopyType.G2G
    st = torch.cuda.current_stream().cuda_stream
    g = torch.Generator(device="cuda").manual_seed(n + step)
    first, ends, wants = device_tensor_from_gva(base, n), [], []
    for _ in range(12):
        data = torch.randint(0, 256, (n,), dtype=torch.uint8, device="cuda", generator=g)
        first.copy_(data)
        at = base
        for i in range(31):
            to = base + (hop if i % 2 == 0 else 0) + step * (i // 2 + 1)
            assert pool.handle.copy_data_on_stream(at, to, n, G2G, st, 1) == 0, mf.get_last_err_msg()
            at = to
        ends.append(device_tensor_from_gva(at, n).clone())
        wants.append(data)
    for turn, (end, want) in enumerate(zip(ends, wants)):
        assert torch.equal(end, want), turn


@pytest.mark.parametrize("count", [505, 504 + 1344 + 1, 3000])
def test_batches_in_several_pieces_replay_from_a_graph(mf, pool, count):
    """A captured batch of several chained launches between two others: the second reads what the batch writes, the batch what the
    first wrote; new data before every replay."""
    import torch

    blk = 4 * KiB
    n = count * blk
    order = np.random.default_rng(count).permutation(count)
    src, dst = _regions(pool, n)
    fresh, out = torch.empty_like(src), torch.empty_like(src)
    perm = torch.from_numpy(order).cuda()
    a, b = pool.hbm(), pool.hbm() + 96 * MiB
    srcs, dsts = [a + i * blk for i in range(count)], [b + int(o) * blk for o in order]
    stream = torch.cuda.Stream()
    T = mf.bm.BmCopyType

    def work():
        h = stream.cuda_stream
        assert pool.handle.copy_data_on_stream(fresh.data_ptr(), a, n, T.L2G, h, 1) == 0, mf.get_last_err_msg()
        assert pool.handle.copy_data_batch_on_stream(srcs, dsts, [blk] * count, T.G2G, h, 1) == 0, mf.get_last_err_msg()
        assert pool.handle.copy_data_on_stream(b, out.data_ptr(), n, T.G2L, h, 1) == 0, mf.get_last_err_msg()

    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        work()  # loads the kernels
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            work()
        g = torch.Generator(device="cuda").manual_seed(count)
        for turn in range(6):
            fresh.copy_(torch.randint(0, 256, (n,), dtype=torch.uint8, device="cuda", generator=g))
            out.zero_()
            for _ in range(2):
                graph.replay()
            assert torch.equal(out.view(count, blk)[perm], fresh.view(count, blk)), turn
    torch.cuda.synchronize()
    del graph


def test_batches_of_two_threads_on_one_stream(mf, pool):
    """Pieces of two batches are enqueued in any interleaving; each arrives whole, and what follows on the stream sees both."""
    import threading

    import torch

    from memfabric_hybrid_b200.utils.tensors import device_tensor_from_gva

    count, blk, rounds = 2500, 4 * KiB, 8
    n = count * blk
    st = torch.cuda.current_stream().cuda_stream
    bases = [(pool.hbm() + k * 24 * MiB, pool.hbm() + 96 * MiB + k * 24 * MiB) for k in range(2)]
    srcs = [device_tensor_from_gva(a, n) for a, _ in bases]
    for k, s in enumerate(srcs):
        s.random_(0, 256, generator=torch.Generator(device="cuda").manual_seed(k))
    torch.cuda.synchronize()
    orders = [[np.random.default_rng(10 * k + r).permutation(count) for r in range(rounds)] for k in range(2)]
    rcs = []

    def issue(k):
        torch.cuda.set_device(0)
        for r in range(rounds):
            a, b = bases[k]
            rcs.append(pool.handle.copy_data_batch_on_stream([a + i * blk for i in range(count)], [b + int(o) * blk for o in orders[k][r]], [blk] * count,
                                                             mf.bm.BmCopyType.G2G, st, 1))

    threads = [threading.Thread(target=issue, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    seen = [device_tensor_from_gva(b, n).clone() for _, b in bases]
    assert rcs == [0] * (2 * rounds)
    for k in range(2):
        assert torch.equal(seen[k].view(count, blk)[torch.from_numpy(orders[k][-1]).cuda()], srcs[k].view(count, blk)), k
