"""Performance cases of the library on one GPU: what a serving or training process asks of it, through its public Python API.

    copy       one contiguous copy inside the pooled HBM (Big Memory, G2G), blocking or on the caller's stream
    kv         one batch call that moves the KV blocks of some requests: pool to pool, offload to pooled DRAM, reload
    allreduce  sum + residual + RMSNorm of a tensor-parallel layer (here with one rank: the fused epilogue)
    moe        a mixture-of-experts layer: dispatch with fp8 quantisation, two block-scaled grouped GEMMs, weighted combine
    reshard    a flat bf16 training shard turned into inference weights, as bf16 or as block-scaled e4m3
    expert_ffn the expert FFN on operands with free-form fp32 scales: row quantiser + grouped GEMM, twice

`listed()` are fixed cases, `draw(rng)` gives others of the same ranges. The pool, the symmetric heap and the operators that own
heap memory are opened once per process and configuration, as a program that uses the library does.
"""
from __future__ import annotations

import socket
import weakref

import numpy as np
import torch

import memfabric_hybrid_b200 as mf
from memfabric_hybrid_b200.models import LlamaConfig, param_specs
from memfabric_hybrid_b200.ops import fp8_gemm as F
from memfabric_hybrid_b200.ops.allreduce import AllReduceRMSNorm
from memfabric_hybrid_b200.ops.moe import FusedMoE, route
from memfabric_hybrid_b200.ops.reshard import Resharder, ReshardPlan
from memfabric_hybrid_b200.parallel.heap import SymmetricHeap
from memfabric_hybrid_b200.parallel.pool import open_pool
from memfabric_hybrid_b200.utils.tensors import device_tensor_from_gva

KiB, MiB, GiB = 1 << 10, 1 << 20, 1 << 30
PAGE = 4 * KiB


def listed():
    return [
        # One cache page between two slots of the pool, waited for: what a block manager's copy-on-write does; latency only.
        {"name": "copy_page", "kind": "copy", "bytes": 16 * KiB, "src_off": 0, "dst_off": 0, "stream": False},
        # A slice of a bf16 tensor that starts at an odd element, into an aligned buffer, with an odd count of elements.
        {"name": "copy_slice", "kind": "copy", "bytes": 5_242_882, "src_off": 34, "dst_off": 0, "stream": True},
        # The bandwidth figure that the reference publishes: 1 GiB per transfer.
        {"name": "copy_1gib", "kind": "copy", "bytes": GiB, "src_off": 0, "dst_off": 0, "stream": True},
        # One request's KV cache (61 layers, a 128 KiB and a 16 KiB block each) between slots of the HBM pool.
        {"name": "kv_move_1", "kind": "kv", "way": "move", "requests": 1, "layers": 61, "large": 128 * KiB, "small": 16 * KiB, "stream": False},
        # The same for a batch of 32 requests: a long descriptor list.
        {"name": "kv_move_32", "kind": "kv", "way": "move", "requests": 32, "layers": 61, "large": 128 * KiB, "small": 16 * KiB, "stream": False},
        # Preempted requests leave for pooled host DRAM, and come back.
        {"name": "kv_offload_8", "kind": "kv", "way": "offload", "requests": 8, "layers": 61, "large": 128 * KiB, "small": 16 * KiB, "stream": False},
        {"name": "kv_reload_8", "kind": "kv", "way": "reload", "requests": 8, "layers": 61, "large": 128 * KiB, "small": 16 * KiB, "stream": False},
        # The epilogue of a tensor-parallel layer in a decode step of 32 sequences.
        {"name": "allreduce_decode", "kind": "allreduce", "tokens": 32, "hidden": 8192},
        # An MoE layer in a decode step (bound by the weight stream) and in prefill (bound by the tensor cores).
        {"name": "moe_decode", "kind": "moe", "tokens": 128, "hidden": 7168, "experts": 32, "topk": 8, "inter": 2048},
        {"name": "moe_prefill", "kind": "moe", "tokens": 4096, "hidden": 7168, "experts": 32, "topk": 8, "inter": 2048},
        # Weight update of an RL step: a quarter of a Llama-3-8B's layers with embedding and head, cast to e4m3.
        {"name": "reshard_fp8", "kind": "reshard", "layers": 8, "hidden": 4096, "heads": 32, "kv_heads": 8, "ffn": 14336, "vocab": 128256, "tp": 1,
         "fp8": True},
        # Experts whose weights were quantised elsewhere with free-form scales, about 256 rows each, ragged.
        {"name": "expert_ffn_fp32_scales", "kind": "expert_ffn", "rows": 8191, "hidden": 7168, "experts": 32, "inter": 2048},
    ]


def _log(rng, lo, hi):
    """A whole number of [lo, hi], spread over its logarithm."""
    return min(hi, max(lo, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choice(["copy", "copy", "kv", "kv", "allreduce", "moe", "moe", "reshard", "expert_ffn"])
    if kind == "copy":
        n = _log(rng, 4 * KiB, GiB)
        # Page moves are whole and aligned; tensor slices start and end at any element of two bytes.
        if rng.random() < 0.5:
            n, so, do = max(1, n // PAGE) * PAGE, rng.randrange(16) * 256, rng.randrange(16) * 256
        else:
            n, so, do = n // 2 * 2, rng.randrange(64) * 2, rng.randrange(64) * 2
        return {"kind": "copy", "bytes": n, "src_off": so, "dst_off": do, "stream": rng.random() < 0.5}
    if kind == "kv":
        way = rng.choice(["move", "move", "offload", "reload"])
        return {"kind": "kv", "way": way, "requests": _log(rng, 1, 32 if way == "move" else 8), "layers": rng.randrange(24, 62),
                "large": rng.choice([32, 64, 96, 128]) * KiB, "small": rng.choice([4, 8, 12, 16]) * KiB, "stream": rng.random() < 0.3}
    if kind == "allreduce":
        return {"kind": "allreduce", "tokens": _log(rng, 1, 4096), "hidden": rng.choice([2048, 4096, 5120, 7168, 8192])}
    if kind == "moe":
        return {"kind": "moe", "tokens": _log(rng, 1, 4096), "hidden": rng.choice([2048, 4096, 7168]), "experts": rng.choice([8, 16, 32]),
                "topk": rng.choice([2, 4, 6, 8]), "inter": rng.choice([768, 1024, 1536, 2048])}
    if kind == "reshard":
        return {"kind": "reshard", "layers": rng.randrange(1, 9), "hidden": rng.choice([2048, 4096]), "heads": 32, "kv_heads": 8,
                "ffn": rng.choice([5632, 8192, 14336]), "vocab": rng.choice([32000, 128256]), "tp": rng.choice([1, 2, 4]), "fp8": rng.random() < 0.6}
    return {"kind": "expert_ffn", "rows": _log(rng, 16, 16384), "hidden": rng.choice([2048, 4096, 7168]), "experts": rng.choice([8, 16, 32]),
            "inter": rng.choice([768, 1024, 1536, 2048])}


# ---------------------------------------------------------------------------------------------- what a process keeps open


class _Lease:
    """Gives `item` back to `idle` when the state that holds the lease is gone."""

    def __init__(self, idle: list, item):
        self.item = item
        weakref.finalize(self, idle.append, item)


def _store_url():
    with socket.socket() as s:
        s.bind(("127.0.0.1", 0))
        return "tcp://127.0.0.1:%d" % s.getsockname()[1]


HBM_SLOT, DRAM_SLOT, SLOTS = 2 * (GiB + MiB), 320 * MiB, 4
_pool = None
_pool_idle = []


def _pool_slot():
    """(lease, HBM address, DRAM address) of an unused part of the pool: 1 GiB + 1 MiB for sources and as much for destinations."""
    global _pool
    if _pool is None:
        _pool = open_pool(0, 1, torch.cuda.current_device(), SLOTS * HBM_SLOT, dram_bytes=SLOTS * DRAM_SLOT, store_url=_store_url())
        _pool_idle.extend(range(SLOTS))
    if not _pool_idle:
        raise MemoryError("every slot of the pool is in use")
    lease = _Lease(_pool_idle, _pool_idle.pop())
    return lease, _pool.hbm() + lease.item * HBM_SLOT, _pool.dram() + lease.item * DRAM_SLOT


_heap = None
_heap_key = None
_heap_idle = []


def _heap_operator(key, nbytes, copies, make):
    """Lease of an operator made by `make(heap)`; the heap holds `copies` of `nbytes` each and serves one configuration at a time."""
    global _heap, _heap_key, _heap_idle
    if key != _heap_key:
        _heap_idle.clear()
        _heap_idle = []
        _heap_key = None
        if _heap is not None:
            _heap.close()
            _heap = None
        torch.cuda.empty_cache()
        _heap = SymmetricHeap(0, 1, torch.cuda.current_device(), copies * nbytes, store_url=_store_url())
        _heap_key = key
    op = _heap_idle.pop() if _heap_idle else make(_heap)
    return _Lease(_heap_idle, op)


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


# ---------------------------------------------------------------------------------------------- copies in the pool


def _prepare_copy(c, seed):
    lease, base, _ = _pool_slot()
    src, dst, n = base + c["src_off"], base + HBM_SLOT // 2 + c["dst_off"], c["bytes"]
    device_tensor_from_gva(src, n).random_(0, 256, generator=_generator(seed))
    out = device_tensor_from_gva(dst, n)
    out.zero_()
    stream = torch.cuda.current_stream().cuda_stream
    return {"lease": lease, "handle": _pool.handle, "src": src, "dst": dst, "bytes": n, "stream": stream if c["stream"] else None, "out": out}


def _run_copy(s):
    h, t = s["handle"], mf.bm.BmCopyType.G2G
    if s["stream"] is None:
        rc = h.copy_data(s["src"], s["dst"], s["bytes"], t, 0)
    else:
        rc = h.copy_data_on_stream(s["src"], s["dst"], s["bytes"], t, s["stream"], 0)
    if rc != 0:
        raise RuntimeError(f"copy failed ({rc}): {mf.get_last_err_msg()}")
    return s["out"]


def _kv_sizes(c):
    return [c["large"], c["small"]] * (c["layers"] * c["requests"])


def _kv_blocks(c, rng, base):
    """Addresses of a request batch's blocks: shuffled slots of one large block each, twice as many as are used, every block at a
    random 4 KiB step of its slot."""
    sizes = np.array(_kv_sizes(c), dtype=np.int64)
    pick = rng.permutation(2 * len(sizes))[: len(sizes)].astype(np.int64)
    steps = (rng.random(len(sizes)) * ((c["large"] - sizes) // PAGE + 1)).astype(np.int64)
    return [int(base + a) for a in pick * c["large"] + steps * PAGE]


def _prepare_kv(c, seed):
    lease, hbm, dram = _pool_slot()
    rng = np.random.default_rng(seed)
    sizes = _kv_sizes(c)
    span = 2 * len(sizes) * c["large"]
    src = dram if c["way"] == "reload" else hbm
    dst = dram if c["way"] == "offload" else hbm + HBM_SLOT // 2
    srcs, dsts = _kv_blocks(c, rng, src), _kv_blocks(c, rng, dst)
    device_tensor_from_gva(src, span).random_(0, 256, generator=_generator(seed))
    out = device_tensor_from_gva(dst, span)
    out.zero_()
    stream = torch.cuda.current_stream().cuda_stream
    return {"lease": lease, "handle": _pool.handle, "srcs": srcs, "dsts": dsts, "sizes": sizes, "stream": stream if c["stream"] else None, "out": out}


def _run_kv(s):
    h, t = s["handle"], mf.bm.BmCopyType.G2G
    if s["stream"] is None:
        rc = h.copy_data_batch(s["srcs"], s["dsts"], s["sizes"], len(s["sizes"]), t, 0)
    else:
        rc = h.copy_data_batch_on_stream(s["srcs"], s["dsts"], s["sizes"], t, s["stream"], 0)
    if rc != 0:
        raise RuntimeError(f"batch copy failed ({rc}): {mf.get_last_err_msg()}")
    return s["out"]


# ---------------------------------------------------------------------------------------------- layer epilogue


def _prepare_allreduce(c, seed):
    T, H = c["tokens"], c["hidden"]
    lease = _heap_operator(("allreduce", T, H), 3 * (T * H * 2 + MiB), 6, lambda heap: AllReduceRMSNorm(heap, T, H, eps=1e-6))
    ar, g = lease.item, _generator(seed)
    weight = (1.0 + 0.1 * torch.randn(H, generator=g, device="cuda")).to(torch.bfloat16)
    residual = torch.randn(T, H, generator=g, device="cuda").to(torch.bfloat16)
    x = torch.randn(T, H, generator=g, device="cuda").to(torch.bfloat16)
    for _ in range(2):  # calls alternate between two input buffers: the producing GEMM's result stands in both
        ar.x[:T].copy_(x)
        ar(T, residual, weight)
    return {"lease": lease, "ar": ar, "tokens": T, "residual": residual, "weight": weight}


def _run_allreduce(s):
    return s["ar"](s["tokens"], s["residual"], s["weight"])


# ---------------------------------------------------------------------------------------------- mixture of experts


def _expert_weights(experts, hidden, inter, seed, quantise):
    g = _generator(seed)
    w13_q = torch.empty(experts, 2 * inter, hidden, dtype=torch.float8_e4m3fn, device="cuda")
    w13_s = torch.empty(experts, 2 * inter // 128, hidden // 128, dtype=torch.float32, device="cuda")
    w2_q = torch.empty(experts, hidden, inter, dtype=torch.float8_e4m3fn, device="cuda")
    w2_s = torch.empty(experts, hidden // 128, inter // 128, dtype=torch.float32, device="cuda")
    for e in range(experts):
        gate, up = (torch.randn(inter, hidden, generator=g, device="cuda") * hidden ** -0.5 for _ in range(2))
        w13_q[e], w13_s[e] = quantise(F.interleave_gate_up(gate, up))
        w2_q[e], w2_s[e] = quantise(torch.randn(hidden, inter, generator=g, device="cuda") * inter ** -0.5)
    return w13_q, w13_s, w2_q, w2_s


def _prepare_moe(c, seed):
    T, H, E, K, I = c["tokens"], c["hidden"], c["experts"], c["topk"], c["inter"]

    def make(heap):
        return FusedMoE(heap, T, H, E, K, I, *_expert_weights(E, H, I, 7, F.quant_weight_mx_torch), capacity_factor=2.0)

    nbytes = (T * K + 128 * (E + 1)) * (3 * H + H // 32 + 256) + 16 * MiB
    lease = _heap_operator(("moe", T, H, E, K, I), nbytes, 1, make)
    # One layer serves every batch: it goes back at once, a batch is the state.
    layer, g = lease.item, _generator(seed)
    x = torch.randn(T, H, generator=g, device="cuda").to(torch.bfloat16)
    idx, w = route(torch.randn(T, E, generator=g, device="cuda"), K)
    return {"layer": layer, "x": x, "idx": idx, "w": w}


def _run_moe(s):
    return s["layer"](s["x"], s["idx"], s["w"])


# ---------------------------------------------------------------------------------------------- weight update


def _plan(c):
    cfg = LlamaConfig(layers=c["layers"], hidden=c["hidden"], heads=c["heads"], kv_heads=c["kv_heads"], ffn=c["ffn"], vocab=c["vocab"])
    return ReshardPlan(param_specs(cfg), 1, c["tp"] - 1, c["tp"], fp8=c["fp8"])


def _prepare_reshard(c, seed):
    plan = _plan(c)
    key = ("reshard",) + tuple(c[k] for k in ("layers", "hidden", "heads", "kv_heads", "ffn", "vocab", "tp", "fp8"))
    lease = _heap_operator(key, plan.shard_elems * 2 + 2 * MiB, 4, lambda heap: Resharder(heap, plan))
    rs, g = lease.item, _generator(seed)
    step = 1 << 26
    for lo in range(0, plan.shard_elems, step):
        n = min(step, plan.shard_elems - lo)
        rs.shard[lo:lo + n] = torch.randn(n, generator=g, device="cuda", dtype=torch.float32).mul_(0.02).to(torch.bfloat16)
    rs.dst.zero_()
    return {"lease": lease, "rs": rs}


def _run_reshard(s):
    rs = s["rs"]
    rs()  # the weights by name are views of the two buffers below
    return [rs.dst, rs.scales] if rs.plan.scale_floats else [rs.dst]


# ---------------------------------------------------------------------------------------------- expert FFN with free-form scales


def _prepare_expert_ffn(c, seed):
    M, H, E, I = c["rows"], c["hidden"], c["experts"], c["inter"]
    g = _generator(seed)
    weights = _expert_weights(E, H, I, seed, F.quant_weight_torch)
    # Routed rows fall on the experts as softmax-routed tokens do; every expert's rows start at a multiple of 128.
    counts = torch.bincount(torch.randint(0, E, (M,), generator=g, device="cuda"), minlength=E).to(torch.int32)
    ends = torch.cumsum((counts + 127) // 128 * 128, 0, dtype=torch.int32)
    offsets = torch.cat([torch.zeros(1, dtype=torch.int32, device="cuda"), ends])
    R = (M + 127) // 128 * 128 + E * 128
    x = torch.randn(R, H, generator=g, device="cuda").to(torch.bfloat16)
    h = torch.zeros(R, I, dtype=torch.bfloat16, device="cuda")
    y = torch.zeros(R, H, dtype=torch.bfloat16, device="cuda")
    return {"weights": weights, "counts": counts, "offsets": offsets, "x": x, "h": h, "y": y}


def _run_expert_ffn(s):
    w13_q, w13_s, w2_q, w2_s = s["weights"]
    q, scale = F.quant_rows_fp8(s["x"])
    h = F.grouped_gemm(q, scale, w13_q, w13_s, s["offsets"], s["counts"], mode="swiglu", out=s["h"])
    q, scale = F.quant_rows_fp8(h)
    return F.grouped_gemm(q, scale, w2_q, w2_s, s["offsets"], s["counts"], out=s["y"])


# ---------------------------------------------------------------------------------------------- the interface


_KINDS = {
    "copy": (_prepare_copy, _run_copy),
    "kv": (_prepare_kv, _run_kv),
    "allreduce": (_prepare_allreduce, _run_allreduce),
    "moe": (_prepare_moe, _run_moe),
    "reshard": (_prepare_reshard, _run_reshard),
    "expert_ffn": (_prepare_expert_ffn, _run_expert_ffn),
}


def prepare(case, seed):
    state = _KINDS[case["kind"]][0](case, seed)
    state["run"] = _KINDS[case["kind"]][1]
    return state


def run(state):
    return state["run"](state)


def work(case):
    """Bytes that have to be read or written once, and multiply-add operations (two each) of the contractions."""
    c = case
    if c["kind"] == "copy":
        return {"bytes": 2 * c["bytes"], "flops": 0}
    if c["kind"] == "kv":
        return {"bytes": 2 * sum(_kv_sizes(c)), "flops": 0}
    if c["kind"] == "allreduce":
        return {"bytes": 4 * c["tokens"] * c["hidden"] * 2 + 2 * c["hidden"], "flops": 0}
    if c["kind"] == "reshard":
        plan = _plan(c)
        return {"bytes": plan.bytes_pulled() + plan.dst_bytes + 4 * plan.scale_floats, "flops": 0}
    rows = c["tokens"] * c["topk"] if c["kind"] == "moe" else c["rows"]
    touched = c["experts"] * (1 - (1 - 1 / c["experts"]) ** rows)  # experts that get a row at all
    weights = touched * 3 * c["hidden"] * c["inter"] * (1 + 4 / 16384)
    acts = 4 * c["hidden"] * (c["tokens"] if c["kind"] == "moe" else rows)
    return {"bytes": weights + acts, "flops": 2 * rows * 3 * c["hidden"] * c["inter"]}


def tolerance(case):
    if case["kind"] == "allreduce":
        return {"rel": 5e-3}  # bf16 results of 32-bit sums
    if case["kind"] in ("moe", "expert_ffn"):
        return {"rel": 1e-2}  # bf16 results; a sum in another order moves some intermediate values to the next e4m3 value
    return "exact"  # copies; block casts, whose maxima and roundings do not depend on an order
