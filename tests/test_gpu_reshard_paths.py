"""The two ways a tile of the reshard kernel moves (rows and columns, or runs in destination order), on parameters whose sizes sit at
the edges: one row, fewer rows than a tile, widths just below and at the narrowest run, shards that end inside a row and inside a
tile, tables much longer than the grid is wide. Against the gather + slice + cast oracle."""
import pytest

pytestmark = pytest.mark.gpu


def _specs():
    from memfabric_hybrid_b200.models.llama import ParamSpec

    return [
        ParamSpec("norm", (8,), "rep", False),
        ParamSpec("one_row", (4, 4096), "col", False),          # at TP 4: one row
        ParamSpec("narrow", (130, 4 * 1016), "row", False),     # 1016 columns at TP 4, 2032 at TP 2
        ParamSpec("wide", (131, 4 * 1024), "row", False),       # 1024 columns at TP 4: the narrowest run
        ParamSpec("tall", (1028, 24), "col", False),            # narrow, but contiguous
        ParamSpec("block", (512, 512), "col", True),
        ParamSpec("ragged_rows", (516, 264), "col", True),      # no whole blocks: stays bf16
        ParamSpec("split", (256, 2048), "row", True),
        ParamSpec("odd_blocks", (1536, 384), "col", True),      # three blocks wide: the last tile is half empty
        ParamSpec("many", (2048, 4096), "col", True),
        ParamSpec("many_bf16", (2052, 4096), "vocab", False),
        ParamSpec("last", (16,), "rep", False),
    ]


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("world,tp", [(1, 1), (1, 4), (2, 2), (3, 4), (8, 4)])
def test_paths(world, tp, fp8):
    import torch

    from memfabric_hybrid_b200.ops.reshard import ReshardPlan, emulated_reshard, reference_reshard
    from memfabric_hybrid_b200.parallel.heap import EmulatedHeap

    plans = [ReshardPlan(_specs(), world, (r + tp - 1) % tp, tp, fp8=fp8) for r in range(world)]
    p0 = plans[0]
    flat = torch.zeros(p0.shard_elems * world, dtype=torch.bfloat16, device="cuda")
    flat[:p0.total_elems] = torch.randn(p0.total_elems, generator=torch.Generator(device="cuda").manual_seed(5), device="cuda").to(torch.bfloat16)
    heap = EmulatedHeap(world, p0.shard_elems * 2 + 4096)
    off = heap.alloc(p0.shard_elems * 2)
    for r in range(world):
        heap.tensor(r, off, (p0.shard_elems,), torch.bfloat16).copy_(flat[r * p0.shard_elems:(r + 1) * p0.shard_elems])
    for r, (dst, scales, status) in enumerate(emulated_reshard(heap, plans, off)):
        assert status == 0
        ref = reference_reshard(flat, plans[r])
        for e in plans[r].entries:
            n = e.nrows * e.ncols
            if not e.quant:
                assert torch.equal(dst[e.dst_off:e.dst_off + 2 * n].view(torch.bfloat16), ref[e.spec.name].reshape(-1)), (r, e.spec.name)
                continue
            q, s = ref[e.spec.name]
            got_s = scales[e.scale_off:e.scale_off + s.numel()].view_as(s)
            # The oracle divides by 448, the kernel multiplies by its reciprocal: one unit in the last place of the scale, and a
            # value that lies within that of a rounding boundary may fall on the neighbouring e4m3 value.
            torch.testing.assert_close(got_s, s, rtol=2.5e-7, atol=0)
            got = dst[e.dst_off:e.dst_off + n].view(torch.float8_e4m3fn).view(e.nrows, e.ncols)
            assert float((got.float() != q.float()).float().mean()) < 2e-3, (r, e.spec.name)
