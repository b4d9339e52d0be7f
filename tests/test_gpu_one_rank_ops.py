"""The operators on a heap of one rank, where they take their own ways: the MoE layer writes and gathers its rows directly, the layer
epilogue runs without barriers. Sizes at the edges of the work split; against the PyTorch oracles."""
import pytest

from conftest import free_port

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def heap():
    import torch

    from memfabric_hybrid_b200.parallel.heap import SymmetricHeap

    torch.cuda.set_device(0)
    h = SymmetricHeap(0, 1, 0, 1 << 30, store_url=f"tcp://127.0.0.1:{free_port()}")
    yield h
    h.close()


def _weights(E, H, I, seed):
    import torch

    from memfabric_hybrid_b200.ops import fp8_gemm as F

    g = torch.Generator(device="cuda").manual_seed(seed)
    wg, wu = (torch.randn(E, I, H, generator=g, device="cuda") * H ** -0.5 for _ in range(2))
    w2 = torch.randn(E, H, I, generator=g, device="cuda") * I ** -0.5
    return F.quant_weight_mx_torch(F.interleave_gate_up(wg, wu)) + F.quant_weight_mx_torch(w2)


def _check(out, ref):
    scale = float(ref.abs().max()) + 1e-6
    err = (out.float() - ref).abs()
    # the bounds of the emulated-rank tests: a flipped e4m3 rounding of the intermediate moves single elements by a step
    assert float(err.max()) <= 1e-1 * scale and float(err.mean()) <= 4e-3 * scale
    assert float((err > 4e-2 * scale).float().mean()) < 1e-3


# tokens: one, fewer and more than there are CTAs; hidden 128 (one block), 384 (three), 4096 (exactly one trip of a CTA), 4224 and 8320
# (a second and a third trip); topk 1, 8 (one group) and 10 (a second group of pairs per token)
@pytest.mark.parametrize("T,H,E,K,I", [(1, 128, 4, 2, 128), (3, 384, 8, 8, 128), (130, 512, 8, 1, 256), (700, 1024, 16, 8, 256), (40, 4096, 4, 4, 128),
                                       (33, 4224, 4, 2, 128), (9, 8320, 4, 3, 128), (65, 512, 16, 10, 128), (64, 512, 16, 8, 384)])
def test_moe_layer(heap, T, H, E, K, I):
    import torch

    from memfabric_hybrid_b200.ops.moe import FusedMoE, moe_reference, route

    w = _weights(E, H, I, 3)
    layer = FusedMoE(heap, T + 5, H, E, K, I, *w, capacity_factor=2.0)
    g = torch.Generator(device="cuda").manual_seed(T)
    for turn in range(3):  # the scratch counters have to be clean for the next call, whatever its size
        n = T if turn != 1 else max(1, T // 2)
        x = torch.randn(n, H, generator=g, device="cuda").to(torch.bfloat16)
        idx, tw = route(torch.randn(n, E, generator=g, device="cuda"), K)
        out = layer(x, idx, tw)
        assert layer.check_status() == 0
        _check(out, moe_reference([x], [idx], [tw], [w], E, I)[0])
        ref_call = out.clone()
        layer.dispatch(x, idx, tw)  # the phases one by one give the same
        layer.experts()
        assert torch.equal(layer.combine(n), ref_call)
    assert layer.launches == 3 * 8


def test_moe_layer_skips_masked_pairs(heap):
    """Pairs with expert -1 are not routed: their weight does not enter the sum, and tokens without any pair come out zero."""
    import torch

    from memfabric_hybrid_b200.ops.moe import FusedMoE, moe_reference, route

    T, H, E, K, I = 50, 512, 8, 4, 128
    w = _weights(E, H, I, 4)
    layer = FusedMoE(heap, T, H, E, K, I, *w)
    g = torch.Generator(device="cuda").manual_seed(1)
    x = torch.randn(T, H, generator=g, device="cuda").to(torch.bfloat16)
    idx, tw = route(torch.randn(T, E, generator=g, device="cuda"), K)
    drop = torch.rand(T, K, generator=g, device="cuda") < 0.4
    drop[7] = True
    masked = torch.where(drop, torch.full_like(idx, -1), idx)
    out = layer(x, masked, tw)
    assert layer.check_status() == 0
    _check(out, moe_reference([x], [idx], [torch.where(drop, torch.zeros_like(tw), tw)], [w], E, I)[0])
    assert float(out[7].float().abs().max()) == 0.0


def _routed_layer(heap, T, H, E, K, I, seed, **kw):
    import torch

    from memfabric_hybrid_b200.ops.moe import FusedMoE, route

    layer = FusedMoE(heap, T, H, E, K, I, *_weights(E, H, I, seed), **kw)
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(T, H, generator=g, device="cuda").to(torch.bfloat16)
    return (layer, x) + route(torch.randn(T, E, generator=g, device="cuda"), K)


@pytest.mark.parametrize("change", ["gone", "in_place"])
def test_combine_needs_nothing_of_what_dispatch_was_given(heap, change):
    """Routing that was a temporary of the dispatch call, its memory handed out again; and routing changed before combine."""
    import torch

    T, K = 60, 4
    layer, x, idx, tw = _routed_layer(heap, T, 512, 8, K, 128, 21)
    want = layer(x, idx, tw * 2.5).clone()
    torch.cuda.synchronize()
    if change == "gone":
        layer.dispatch(x, idx.clone(), tw * 2.5)
        torch.cuda.synchronize()
        reused = [torch.full((T, K), v, device="cuda", dtype=d) for d, v in ((torch.int32, 0), (torch.float32, 100.0)) for _ in range(4)]
    else:
        idx, tw = idx.clone(), tw * 2.5
        layer.dispatch(x, idx, tw)
        idx.zero_()
        tw.fill_(100.0)
    layer.experts()
    assert torch.equal(layer.combine(T), want) and layer.check_status() == 0
    if change == "gone":
        del reused


@pytest.mark.parametrize("asked", [1, 30, 64])
def test_combine_sums_the_tokens_that_were_dispatched(heap, asked):
    """Another count given to combine() selects rows of the result, it does not reach past the routing of this call."""
    import torch

    T, most = 40, 64
    layer, x, idx, tw = _routed_layer(heap, most, 512, 8, 4, 128, 22)
    x, idx, tw = x[:T].clone(), idx[:T].clone(), tw[:T].clone()
    want = layer(x, idx, tw).clone()
    layer.st.out.fill_(7.0)
    layer.dispatch(x, idx, tw)
    layer.experts()
    assert layer.combine(asked).shape == (asked, 512)
    assert torch.equal(layer.st.out[:T], want) and bool((layer.st.out[T:] == 7.0).all())


@pytest.mark.parametrize("K", [1, 2, 3, 6])
def test_combine_keeps_an_infinite_weight_infinite(heap, K):
    """The rows of a token are read four at a time; the slots that hold no row add nothing, whatever the first weight is."""
    import torch

    T = 5
    layer, x, idx, tw = _routed_layer(heap, T, 512, 8, K, 128, 23)
    tw = tw.clone()
    plain = layer(x, idx, tw).float()
    tw[2, 0] = float("inf")
    out = layer(x, idx, tw).float()
    assert bool(out[2].isinf().all())
    keep = [0, 1, 3, 4]
    assert torch.equal(out[keep], plain[keep]) and layer.check_status() == 0


def test_moe_layer_looks_at_its_weights_on_every_call(heap):
    import torch

    from memfabric_hybrid_b200.ops.moe import FusedMoE, route

    T, H, E, K, I = 4, 256, 4, 2, 128
    layer = FusedMoE(heap, T, H, E, K, I, *_weights(E, H, I, 6))
    x = torch.ones(T, H, dtype=torch.bfloat16, device="cuda")
    idx, tw = route(torch.randn(T, E, device="cuda"), K)
    want = layer(x, idx, tw).clone()
    layer.w2_s.unsqueeze_(0)  # the same scales in another shape are as good
    layer.w13_s = layer.w13_s.flatten()
    assert torch.equal(layer(x, idx, tw), want)
    layer.w2_q.transpose_(1, 2)  # the same tensor, but its rows no longer follow one another
    with pytest.raises(AssertionError):
        layer(x, idx, tw)
    layer.w2_q.transpose_(1, 2)
    layer.w2_s.squeeze_(0)
    layer.w2_s = layer.w2_s[1:]  # too few scales
    with pytest.raises(AssertionError):
        layer(x, idx, tw)


def test_moe_layer_replays_and_follows_itself(heap):
    """The launches of a layer overlap the end of the one before: captured three in a row, and eagerly with new inputs every time."""
    import torch

    from memfabric_hybrid_b200.ops.moe import FusedMoE, route

    T, H, E, K, I = 64, 512, 8, 4, 256
    layer = FusedMoE(heap, T, H, E, K, I, *_weights(E, H, I, 8), device_epochs=True)
    g = torch.Generator(device="cuda").manual_seed(2)

    def batch():
        x = torch.randn(T, H, generator=g, device="cuda").to(torch.bfloat16)
        return (x,) + route(torch.randn(T, E, generator=g, device="cuda"), K)

    inputs = batch()
    ref = layer(*inputs).clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        for _ in range(3):
            out = layer(*inputs)
    for _ in range(5):
        layer.st.out.zero_()
        graph.replay()
        assert torch.equal(out, ref)
    for _ in range(30):
        inputs = batch()
        a = layer(*inputs).clone()
        torch.cuda.synchronize()
        layer(*batch())  # what follows must not reach into the call before it, nor be reached by it
        assert torch.equal(layer(*inputs), a)
    assert layer.check_status() == 0
    del graph


def test_moe_overflow_is_reported_and_the_kernel_ends(heap):
    """Everything goes to one expert of a layer whose receive buffer holds a fraction of it."""
    import torch

    from memfabric_hybrid_b200.ops.moe import FusedMoE

    T, H, E, K, I = 1500, 256, 4, 2, 128
    layer = FusedMoE(heap, T, H, E, K, I, *_weights(E, H, I, 5), capacity_factor=0.25)
    x = torch.zeros(T, H, dtype=torch.bfloat16, device="cuda")
    idx = torch.tensor([[0, 1]], dtype=torch.int32, device="cuda").repeat(T, 1)
    layer(x, idx, torch.full((T, K), 0.5, device="cuda"))
    assert layer.check_status() == 2  # MF_DEV_ERR_BOUNDS


@pytest.mark.parametrize("T", [1, 7, 300, 4099])
@pytest.mark.parametrize("H", [8, 2048, 4096, 4104, 8192, 16384])
def test_epilogue(heap, T, H):
    import torch

    from memfabric_hybrid_b200.ops.allreduce import AllReduceRMSNorm, reference

    if T * H > 300 * 16384 and H > 4104:
        pytest.skip("heap space")
    mark = heap._bump.used
    ar = AllReduceRMSNorm(heap, T, H)
    g = torch.Generator(device="cuda").manual_seed(T + H)
    w = (1.0 + 0.1 * torch.randn(H, generator=g, device="cuda")).to(torch.bfloat16)
    for n, with_res in ((T, True), (max(1, T // 2), False), (T, True)):
        x = torch.randn(n, H, generator=g, device="cuda").to(torch.bfloat16)
        res = torch.randn(n, H, generator=g, device="cuda").to(torch.bfloat16) if with_res else None
        ar.x[:n].copy_(x)
        out, h = ar(n, res, w)
        ref_out, ref_h = reference([x], res, w, 1e-6)
        assert out.shape == (n, H) and ar.check_status() == 0
        assert torch.equal(h.float(), ref_h)  # one rounding of an exact sum of two bf16 numbers
        torch.testing.assert_close(out.float(), ref_out, rtol=2 ** -7, atol=1e-6)  # bf16 rounding (2^-8) and 32-bit sums
    heap._bump.used = mark


def _launched(call):
    """Names of the kernels that `call` launches."""
    import torch
    from torch.profiler import ProfilerActivity, profile

    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        call()
        torch.cuda.synchronize()
    return " ".join(e.key for e in prof.key_averages())


@pytest.mark.parametrize("algo,ctas,kernel", [("auto", 0, "residual_rmsnorm"), ("oneshot", 0, "oneshot"), ("twoshot", 0, "twoshot"), ("auto", 4, "oneshot"),
                                              ("twoshot", 8, "twoshot")])
def test_epilogue_of_one_rank_runs_the_algorithm_that_was_named(heap, algo, ctas, kernel):
    import torch

    from memfabric_hybrid_b200.ops.allreduce import AllReduceRMSNorm, reference

    T, H = 24, 2048
    mark = heap._bump.used
    ar = AllReduceRMSNorm(heap, T, H)
    g = torch.Generator(device="cuda").manual_seed(9)
    x, res = (torch.randn(T, H, generator=g, device="cuda").to(torch.bfloat16) for _ in range(2))
    w = torch.ones(H, dtype=torch.bfloat16, device="cuda")
    ref_out, ref_h = reference([x], res, w, 1e-6)

    def call():
        ar.x[:T].copy_(x)
        call.got = ar(T, res, w, algo=algo, ctas=ctas)

    call()
    assert kernel in _launched(call)
    out, h = call.got
    assert torch.equal(h.float(), ref_h) and ar.check_status() == 0
    torch.testing.assert_close(out.float(), ref_out, rtol=2 ** -7, atol=1e-6)
    heap._bump.used = mark


def test_epilogue_reads_its_settings_on_every_call(heap):
    import torch

    from memfabric_hybrid_b200.ops.allreduce import AllReduceRMSNorm, reference

    T, H = 6, 1024
    mark = heap._bump.used
    ar = AllReduceRMSNorm(heap, T, H)
    x = torch.randn(T, H, device="cuda").to(torch.bfloat16)
    w = torch.ones(H, dtype=torch.bfloat16, device="cuda")
    for eps in (1e-6, 0.5, 1e-6):
        ar.eps = eps
        ar.x[:T].copy_(x)
        torch.testing.assert_close(ar(T, None, w)[0].float(), reference([x], None, w, eps)[0], rtol=2 ** -7, atol=1e-6)
    heap._bump.used = mark


@pytest.mark.parametrize("whole", [True, False])
def test_moe_layer_reads_its_limits_on_every_call(heap, whole):
    """A dispatch in arrival mode whose tiles never fill up: the first GEMM gives up after the layer's present `wait_ns`."""
    import time

    import torch

    layer, x, idx, tw = _routed_layer(heap, 16, 256, 4, 2, 128, 31, overlap=True)
    layer(x, idx, tw)
    assert layer.check_status() == 0
    took = {}
    for wait_ns in (1_000_000, 700_000_000):
        layer.wait_ns = wait_ns
        if whole:
            layer(x, idx, tw)
            assert layer.check_status() == 0
        layer.dispatch(x, idx, tw)
        layer.st.arrive.zero_()  # as if the senders' counts had been lost
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        layer.experts()
        torch.cuda.synchronize()
        took[wait_ns] = time.perf_counter() - t0
        assert layer.check_status() == 4  # the arrival wait ran out
        layer.st.status.zero_()
    assert took[1_000_000] < 0.3 < took[700_000_000], took


@pytest.mark.parametrize("H", [512, 8192, 16384])
def test_epilogue_of_one_rank_checks_its_input_first(heap, H):
    """With the bounds check on, an input outside the heap (valid memory here) is refused before anything is read or written."""
    import torch

    from memfabric_hybrid_b200.ops.allreduce import AllReduceRMSNorm

    T = 7
    mark = heap._bump.used
    ar = AllReduceRMSNorm(heap, T, H)
    outside = torch.ones(T, H, dtype=torch.bfloat16, device="cuda")
    w = torch.ones(H, dtype=torch.bfloat16, device="cuda")
    ar.out.fill_(3.0)
    ar.residual_out.fill_(3.0)
    heap.set_check_bounds(True)
    try:
        inside = list(ar._x_ptrs)
        ar._x_ptrs = [outside.data_ptr()] * 2
        ar(T, outside, w)
        assert ar.check_status() == 2  # MF_DEV_ERR_BOUNDS
        assert bool((ar.out == 3.0).all()) and bool((ar.residual_out == 3.0).all())
        ar.status.zero_()
        ar._x_ptrs = inside
        ar.x.zero_()
        ar(T, outside, w)
        assert ar.check_status() == 0 and bool((ar.residual_out == 1.0).all())
    finally:
        heap.set_check_bounds(False)
    heap._bump.used = mark


@pytest.mark.parametrize("n", [12, 5])
def test_results_are_tensors_of_their_own(heap, n):
    """What a caller does to the shape of a result stays with that tensor: the next call returns the ordinary one."""
    import torch

    from memfabric_hybrid_b200.models.llama import ParamSpec
    from memfabric_hybrid_b200.ops.allreduce import AllReduceRMSNorm
    from memfabric_hybrid_b200.ops.reshard import Resharder, ReshardPlan

    T, H = 12, 512
    mark = heap._bump.used
    ar = AllReduceRMSNorm(heap, T, H)
    w = torch.ones(H, dtype=torch.bfloat16, device="cuda")
    layer, x, idx, tw = _routed_layer(heap, T, H, 4, 2, 128, 41)
    rs = Resharder(heap, ReshardPlan([ParamSpec("a", (256, 128), "col", True), ParamSpec("b", (64,), "rep", False)], 1, 0, 1, fp8=True))
    calls = [lambda: ar(n, None, w), lambda: (layer(x[:n], idx[:n], tw[:n]),), lambda: (*rs()["a"], rs()["b"])]
    for call in calls:
        shapes = [t.shape for t in call()]
        first = call()
        for t in first:
            t.unsqueeze_(0)
            t.transpose_(0, 1)
        again = call()
        assert [t.shape for t in again] == shapes
        assert all(t is not f for t, f in zip(again, first))
        assert all(t.data_ptr() == f.data_ptr() for t, f in zip(again, first))
    assert ar.out.shape == (T, H) and layer.st.out.shape == (T, H)
    heap._bump.used = mark
