// `ops` submodule: raw launchers of the fused compute+collective kernels. Arguments are device addresses (ints) and a
// CUDA stream handle; the torch-facing wrappers live in memfabric_hybrid_b200/ops.
#include <pybind11/stl.h>

#include <cuda_runtime.h>

#include "../kernels/mf_kernels.h"
#include "pymf_parts.h"

namespace py = pybind11;

namespace {

// What one AllReduceRMSNorm object keeps between calls.
struct AllReducePlan {
    mf_allreduce_args_t a{};
    int world{1}, hidden{0};
};

// What one MoE layer of a rank keeps between calls, and the launches of a call: in Python the four of them took about 60 us,
// more than a small layer runs on the GPU.
struct MoePlan {
    mf_moe_dispatch_args_t d{};
    mf_moe_combine_args_t c{};
    void *h1Q{nullptr}, *h1Sf{nullptr};
    int world{1}, hidden{0}, topk{0}, experts{0}, inter{0};
    uint32_t dispatchChannel{0}, combineChannel{0};
    uint64_t timeoutNs{0}, waitNs{0};  // limits of the layer, set anew by every call
    int *arrive{nullptr};

    int Dispatch(uint64_t x, uint64_t idx, uint64_t w, int T, uint64_t epoch, bool overlap, int dedupMinPairs, uint64_t stream)
    {
        d.x = (const void *)x;
        d.topkIdx = (const int *)idx;
        d.topkW = (const float *)w;
        d.T = c.T = T;
        d.arrive = overlap ? arrive : nullptr;
        d.dedupMinPairs = dedupMinPairs;
        // One CTA per token: small batches get a small grid (its grid-wide barriers are cheaper), large ones every SM.
        return mf_k_moe_dispatch_rank(&d, world, hidden, topk, experts, dispatchChannel, epoch, timeoutNs, T > 1 ? T : 1, (mf_stream_t)stream);
    }
    int Experts(uint64_t w13Q, uint64_t w13S, int w13Packed, uint64_t w2Q, uint64_t w2S, int w2Packed, bool overlap, uint64_t stream)
    {
        const int el = experts / world, rows = c.cap;
        const int mode1 = MF_GEMM_EPI_SWIGLU_FP8 | (w13Packed ? (int)MF_GEMM_B_PACKED : 0), mode2 = MF_GEMM_EPI_BF16 | (w2Packed ? (int)MF_GEMM_B_PACKED : 0);
        const int rc = overlap ? mf_k_moe_grouped_gemm_mx_gated(d.recvX, d.recvSf, (const void *)w13Q, (const float *)w13S, h1Q, h1Sf, d.expertOffset,
                                                                d.expertCount, el, rows, 2 * inter, hidden, mode1, 0, arrive, waitNs, d.status, 0,
                                                                (mf_stream_t)stream)
                               : mf_k_moe_grouped_gemm_mx(d.recvX, d.recvSf, (const void *)w13Q, (const float *)w13S, h1Q, h1Sf, d.expertOffset,
                                                          d.expertCount, el, rows, 2 * inter, hidden, mode1, 0, d.status, 0, (mf_stream_t)stream);
        if (rc != MF_K_OK) {
            return rc;
        }
        return mf_k_moe_grouped_gemm_mx(h1Q, (const uint32_t *)h1Sf, (const void *)w2Q, (const float *)w2S, const_cast<void *>(c.y), nullptr, d.expertOffset,
                                        d.expertCount, el, rows, hidden, inter, mode2, 0, d.status, 0, (mf_stream_t)stream);
    }
    // Of the tokens that were dispatched, whatever count the caller asks to see.
    int Combine(uint64_t epoch, uint64_t stream)
    {
        // One warp per 2 KiB piece of a returned row; alone, a rank has no rows to return and one warp sums each 1 KiB of a token.
        const long long pieces = world == 1 ? (long long)c.T * ((hidden / 8 + 63) / 64) : (long long)c.T * topk * ((hidden / 8 + 127) / 128);
        const int ctas = (int)((pieces + 7) / 8 < 65536 ? (pieces + 7) / 8 : 65536);
        return mf_k_moe_combine_rank(&c, world, hidden, topk, experts / world, combineChannel, epoch, timeoutNs, ctas > 1 ? ctas : 1, (mf_stream_t)stream);
    }
};

}  // namespace

void BindOps(py::module_ &m)
{
    py::module_ ops = m.def_submodule("ops", "raw launchers of the fused kernels");

    ops.attr("AR_AUTO") = (int)MF_AR_AUTO;
    ops.attr("AR_ONESHOT") = (int)MF_AR_ONESHOT;
    ops.attr("AR_TWOSHOT") = (int)MF_AR_TWOSHOT;
    ops.attr("AR_NVLS") = (int)MF_AR_NVLS;
    ops.attr("AR_ONESHOT_NOTAIL") = (int)MF_AR_ONESHOT_NOTAIL;
    ops.attr("ALLREDUCE_ARGS_BYTES") = (int)sizeof(mf_allreduce_args_t);

    // Packs one argument block (to be copied to device memory by the caller).
    ops.def("pack_allreduce_args", [](uint64_t meta, uint64_t x, uint64_t residual, uint64_t weight, uint64_t residualOut, uint64_t out, uint64_t status,
                                       uint64_t epochState) {
        mf_allreduce_args_t a{};
        a.meta = (const void *)meta;
        a.x = (const void *)x;
        a.residual = (const void *)residual;
        a.weight = (const void *)weight;
        a.residualOut = (void *)residualOut;
        a.out = (void *)out;
        a.status = (int *)status;
        a.epochState = (unsigned long long *)epochState;
        return py::bytes((const char *)&a, sizeof(a));
    }, py::arg("meta"), py::arg("x"), py::arg("residual"), py::arg("weight"), py::arg("residual_out"), py::arg("out"), py::arg("status"),
       py::arg("epoch_state") = 0);
    ops.attr("GEMM_EPI_BF16") = (int)MF_GEMM_EPI_BF16;
    ops.attr("GEMM_EPI_SWIGLU") = (int)MF_GEMM_EPI_SWIGLU;
    ops.attr("GEMM_EPI_SWIGLU_FP8") = (int)MF_GEMM_EPI_SWIGLU_FP8;
    ops.attr("MOE_MAX_SIBLINGS") = (int)MF_MOE_MAX_SIBLINGS;
    ops.def("moe_grouped_gemm_mx", [](uint64_t a, uint64_t aSf, uint64_t b, uint64_t bScale, uint64_t out, uint64_t outSf, uint64_t groupOffset,
                                      uint64_t groupCount, int G, int rowsTotal, int N, int K, int mode, int tileN, uint64_t status, int ctas,
                                      uint64_t stream, uint64_t arrive, uint64_t waitNs) {
        if (arrive != 0) {
            return mf_k_moe_grouped_gemm_mx_gated((const void *)a, (const uint32_t *)aSf, (const void *)b, (const float *)bScale, (void *)out,
                                                  (void *)outSf, (const int *)groupOffset, (const int *)groupCount, G, rowsTotal, N, K, mode, tileN,
                                                  (const int *)arrive, waitNs, (int *)status, ctas, (mf_stream_t)stream);
        }
        return mf_k_moe_grouped_gemm_mx((const void *)a, (const uint32_t *)aSf, (const void *)b, (const float *)bScale, (void *)out, (void *)outSf,
                                        (const int *)groupOffset, (const int *)groupCount, G, rowsTotal, N, K, mode, tileN, (int *)status, ctas,
                                        (mf_stream_t)stream);
    }, py::arg("a"), py::arg("a_sf"), py::arg("b"), py::arg("b_scale"), py::arg("out"), py::arg("out_sf"), py::arg("group_offset"),
            py::arg("group_count"), py::arg("G"), py::arg("rows_total"), py::arg("N"), py::arg("K"), py::arg("mode"), py::arg("tile_n") = 0,
            py::arg("status") = 0, py::arg("ctas") = 0, py::arg("stream") = 0, py::arg("arrive") = 0, py::arg("wait_ns") = 0);
    ops.def("gemm_tile", &mf_k_gemm_tile, py::arg("G"), py::arg("rows_total"), py::arg("N"), py::arg("ctas"));
    ops.def("gemm_mx_tile", &mf_k_gemm_mx_tile, py::arg("G"), py::arg("rows_total"), py::arg("N"), py::arg("mode"), py::arg("ctas"));
    ops.attr("GEMM_B_PACKED") = (int)MF_GEMM_B_PACKED;
    ops.attr("GEMM_ARRIVAL_EXPIRED") = (int)MF_K_GEMM_ARRIVAL_EXPIRED;
    ops.attr("GEMM_PIPELINE_EXPIRED") = (int)MF_K_GEMM_PIPELINE_EXPIRED;
    ops.def("moe_grouped_gemm", [](uint64_t a, uint64_t aScale, uint64_t b, uint64_t bScale, uint64_t out, uint64_t groupOffset, uint64_t groupCount,
                                   int G, int rowsTotal, int N, int K, int mode, uint64_t status, int ctas, uint64_t stream) {
        return mf_k_moe_grouped_gemm((const void *)a, (const float *)aScale, (const void *)b, (const float *)bScale, (void *)out,
                                     (const int *)groupOffset, (const int *)groupCount, G, rowsTotal, N, K, mode, (int *)status, ctas, (mf_stream_t)stream);
    }, py::arg("a"), py::arg("a_scale"), py::arg("b"), py::arg("b_scale"), py::arg("out"), py::arg("group_offset"), py::arg("group_count"), py::arg("G"),
            py::arg("rows_total"), py::arg("N"), py::arg("K"), py::arg("mode"), py::arg("status") = 0, py::arg("ctas") = 0, py::arg("stream") = 0);
    ops.def("quant_rows_fp8", [](uint64_t x, uint64_t q, uint64_t scale, int rows, int K, uint64_t rowLimit, uint64_t stream) {
        return mf_k_quant_rows_fp8((const void *)x, (void *)q, (float *)scale, rows, K, (const int *)rowLimit, (mf_stream_t)stream);
    }, py::arg("x"), py::arg("q"), py::arg("scale"), py::arg("rows"), py::arg("K"), py::arg("row_limit") = 0, py::arg("stream") = 0);
    ops.attr("MOE_DISPATCH_ARGS_BYTES") = (int)sizeof(mf_moe_dispatch_args_t);
    ops.attr("MOE_COMBINE_ARGS_BYTES") = (int)sizeof(mf_moe_combine_args_t);
    ops.def("pack_moe_dispatch_args", [](uint64_t meta, uint64_t x, uint64_t topkIdx, uint64_t topkW, uint64_t cnt, uint64_t recvX, uint64_t recvSf,
                                         uint64_t recvMeta, uint64_t recvSib, uint64_t localCnt, uint64_t cursor, uint64_t expertOffset, uint64_t expertCount,
                                         uint64_t routed, uint64_t status, int T, int cap, uint64_t arrive, int dedupMinPairs, uint64_t epochState) {
        mf_moe_dispatch_args_t a{};
        a.arrive = (int *)arrive;
        a.dedupMinPairs = dedupMinPairs;
        a.epochState = (unsigned long long *)epochState;
        a.meta = (const void *)meta;
        a.x = (const void *)x;
        a.topkIdx = (const int *)topkIdx;
        a.topkW = (const float *)topkW;
        a.cnt = (int *)cnt;
        a.recvX = (void *)recvX;
        a.recvSf = (uint32_t *)recvSf;
        a.recvMeta = (int4 *)recvMeta;
        a.recvSib = (int2 *)recvSib;
        a.localCnt = (int *)localCnt;
        a.cursor = (int *)cursor;
        a.expertOffset = (int *)expertOffset;
        a.expertCount = (int *)expertCount;
        a.routed = (int4 *)routed;
        a.status = (int *)status;
        a.T = T;
        a.cap = cap;
        return py::bytes((const char *)&a, sizeof(a));
    }, py::arg("meta"), py::arg("x"), py::arg("topk_idx"), py::arg("topk_w"), py::arg("cnt"), py::arg("recv_x"), py::arg("recv_sf"), py::arg("recv_meta"),
            py::arg("recv_sib"), py::arg("local_cnt"), py::arg("cursor"), py::arg("expert_offset"), py::arg("expert_count"), py::arg("routed"),
            py::arg("status"), py::arg("T"), py::arg("cap"), py::arg("arrive") = 0, py::arg("dedup_min_pairs") = 0, py::arg("epoch_state") = 0);
    ops.def("pack_moe_combine_args", [](uint64_t meta, uint64_t y, uint64_t recvMeta, uint64_t recvSib, uint64_t expertOffset, uint64_t expertCount,
                                        uint64_t retY, uint64_t routed, uint64_t out, uint64_t status, int T, int cap, int retRows, uint64_t epochState) {
        mf_moe_combine_args_t a{};
        a.epochState = (unsigned long long *)epochState;
        a.meta = (const void *)meta;
        a.y = (const void *)y;
        a.recvMeta = (const int4 *)recvMeta;
        a.recvSib = (const int2 *)recvSib;
        a.expertOffset = (const int *)expertOffset;
        a.expertCount = (const int *)expertCount;
        a.retY = (void *)retY;
        a.routed = (const int4 *)routed;
        a.out = (void *)out;
        a.status = (int *)status;
        a.T = T;
        a.cap = cap;
        a.retRows = retRows;
        return py::bytes((const char *)&a, sizeof(a));
    }, py::arg("meta"), py::arg("y"), py::arg("recv_meta"), py::arg("recv_sib"), py::arg("expert_offset"), py::arg("expert_count"), py::arg("ret_y"),
            py::arg("routed"), py::arg("out"), py::arg("status"), py::arg("T"), py::arg("cap"), py::arg("ret_rows"), py::arg("epoch_state") = 0);
    ops.def("moe_dispatch", [](uint64_t argsDev, int nEmulated, int rankCount, int H, int K, int E, uint32_t channel, uint64_t epoch, uint64_t timeoutNs,
                               int ctas, uint64_t stream) {
        return mf_k_moe_dispatch((const mf_moe_dispatch_args_t *)argsDev, nEmulated, rankCount, H, K, E, channel, epoch, timeoutNs, ctas,
                                 (mf_stream_t)stream);
    }, py::arg("args_dev"), py::arg("n_emulated"), py::arg("rank_count"), py::arg("H"), py::arg("K"), py::arg("E"), py::arg("channel"), py::arg("epoch"),
            py::arg("timeout_ns") = 0, py::arg("ctas") = 0, py::arg("stream") = 0);
    ops.def("moe_combine", [](uint64_t argsDev, int nEmulated, int rankCount, int H, int K, int EL, uint32_t channel, uint64_t epoch, uint64_t timeoutNs,
                              int ctas, uint64_t stream) {
        return mf_k_moe_combine((const mf_moe_combine_args_t *)argsDev, nEmulated, rankCount, H, K, EL, channel, epoch, timeoutNs, ctas,
                                (mf_stream_t)stream);
    }, py::arg("args_dev"), py::arg("n_emulated"), py::arg("rank_count"), py::arg("H"), py::arg("K"), py::arg("EL"), py::arg("channel"), py::arg("epoch"),
            py::arg("timeout_ns") = 0, py::arg("ctas") = 0, py::arg("stream") = 0);
    ops.attr("RESHARD_DESC_BYTES") = (int)sizeof(mf_reshard_desc_t);
    ops.attr("RESHARD_ARGS_BYTES") = (int)sizeof(mf_reshard_args_t);
    ops.def("pack_reshard_desc", [](uint64_t srcFlatOff, uint64_t dstOff, uint64_t scaleOff, uint32_t colsFull, uint32_t r0, uint32_t c0, uint32_t nrows,
                                    uint32_t ncols, uint32_t tileStart, uint32_t quant) {
        mf_reshard_desc_t d{srcFlatOff, dstOff, scaleOff, colsFull, r0, c0, nrows, ncols, tileStart, quant, 0};
        return py::bytes((const char *)&d, sizeof(d));
    });
    ops.def("pack_reshard_args", [](uint64_t meta, uint64_t srcShard, uint64_t dst, uint64_t dstScale, uint64_t descs, uint64_t status, uint64_t shardElems,
                                    uint32_t ndesc, uint32_t totalTiles) {
        mf_reshard_args_t a{};
        a.meta = (const void *)meta;
        a.srcShard = (const void *)srcShard;
        a.dst = (void *)dst;
        a.dstScale = (float *)dstScale;
        a.descs = (const mf_reshard_desc_t *)descs;
        a.status = (int *)status;
        a.shardElems = shardElems;
        a.ndesc = ndesc;
        a.totalTiles = totalTiles;
        return py::bytes((const char *)&a, sizeof(a));
    });
    ops.def("reshard", [](uint64_t argsDev, int nEmulated, int rankCount, uint32_t channel, uint64_t epoch, uint64_t timeoutNs, int ctas, uint64_t stream) {
        return mf_k_reshard((const mf_reshard_args_t *)argsDev, nEmulated, rankCount, channel, epoch, timeoutNs, ctas, (mf_stream_t)stream);
    }, py::arg("args_dev"), py::arg("n_emulated"), py::arg("rank_count"), py::arg("channel"), py::arg("epoch"), py::arg("timeout_ns") = 0,
            py::arg("ctas") = 0, py::arg("stream") = 0);
    py::class_<AllReducePlan>(ops, "AllReducePlan")
        .def(py::init([](uint64_t meta, uint64_t residualOut, uint64_t out, uint64_t status, uint64_t epochState, int world, int hidden) {
            AllReducePlan p;
            p.a.meta = (const void *)meta;
            p.a.residualOut = (void *)residualOut;
            p.a.out = (void *)out;
            p.a.status = (int *)status;
            p.a.epochState = (unsigned long long *)epochState;
            p.world = world;
            p.hidden = hidden;
            return p;
        }))
        .def("run", [](const AllReducePlan &p, uint64_t x, uint64_t residual, uint64_t weight, int T, float eps, int algo, uint32_t channel, uint64_t epoch,
                       uint64_t timeoutNs, int ctas, uint64_t stream) {
            mf_allreduce_args_t a = p.a;
            a.x = (const void *)x;
            a.residual = (const void *)residual;
            a.weight = (const void *)weight;
            return mf_k_allreduce_rmsnorm_rank(&a, p.world, T, p.hidden, eps, algo, channel, epoch, timeoutNs, ctas, (mf_stream_t)stream);
        });
    py::class_<MoePlan>(ops, "MoePlan")
        .def(py::init([](uint64_t meta, uint64_t cnt, uint64_t recvX, uint64_t recvSf, uint64_t recvMeta, uint64_t recvSib, uint64_t localCnt,
                         uint64_t cursor, uint64_t expertOffset, uint64_t expertCount, uint64_t routed, uint64_t arrive, uint64_t status, uint64_t h1Q,
                         uint64_t h1Sf, uint64_t y, uint64_t retY, uint64_t out, int cap, int retRows, int world, int hidden, int topk, int experts,
                         int inter, uint32_t dispatchChannel, uint32_t combineChannel, uint64_t epochD, uint64_t epochC) {
            MoePlan p;
            p.d.meta = p.c.meta = (const void *)meta;
            p.d.cnt = (int *)cnt;
            p.d.recvX = (void *)recvX;
            p.d.recvSf = (uint32_t *)recvSf;
            p.d.recvMeta = (int4 *)recvMeta;
            p.c.recvMeta = (const int4 *)recvMeta;
            p.d.recvSib = (int2 *)recvSib;
            p.c.recvSib = (const int2 *)recvSib;
            p.d.localCnt = (int *)localCnt;
            p.d.cursor = (int *)cursor;
            p.d.expertOffset = (int *)expertOffset;
            p.c.expertOffset = (const int *)expertOffset;
            p.d.expertCount = (int *)expertCount;
            p.c.expertCount = (const int *)expertCount;
            p.d.routed = (int4 *)routed;
            p.c.routed = (const int4 *)routed;
            p.d.status = p.c.status = (int *)status;
            p.d.epochState = (unsigned long long *)epochD;
            p.c.epochState = (unsigned long long *)epochC;
            p.d.cap = p.c.cap = cap;
            p.c.y = (const void *)y;
            p.c.retY = (void *)retY;
            p.c.out = (void *)out;
            p.c.retRows = retRows;
            p.h1Q = (void *)h1Q;
            p.h1Sf = (void *)h1Sf;
            p.arrive = (int *)arrive;
            p.world = world;
            p.hidden = hidden;
            p.topk = topk;
            p.experts = experts;
            p.inter = inter;
            p.dispatchChannel = dispatchChannel;
            p.combineChannel = combineChannel;
            return p;
        }))
        .def("limits", [](MoePlan &p, uint64_t timeoutNs, uint64_t waitNs) {
            p.timeoutNs = timeoutNs;
            p.waitNs = waitNs;
        })
        .def("dispatch", &MoePlan::Dispatch)
        .def("experts", &MoePlan::Experts)
        .def("combine", &MoePlan::Combine)
        .def("run", [](MoePlan &p, uint64_t x, uint64_t idx, uint64_t w, int T, uint64_t w13Q, uint64_t w13S, int w13Packed, uint64_t w2Q, uint64_t w2S,
                       int w2Packed, uint64_t epochD, uint64_t epochC, bool overlap, int dedupMinPairs, uint64_t timeoutNs, uint64_t waitNs,
                       uint64_t stream) {
            p.timeoutNs = timeoutNs;
            p.waitNs = waitNs;
            int rc = p.Dispatch(x, idx, w, T, epochD, overlap, dedupMinPairs, stream);
            if (rc == MF_K_OK) {
                rc = p.Experts(w13Q, w13S, w13Packed, w2Q, w2S, w2Packed, overlap, stream);
            }
            return rc == MF_K_OK ? p.Combine(epochC, stream) : rc;
        });
    ops.def("allreduce_rmsnorm", [](uint64_t argsDev, int nEmulated, int rankCount, int T, int H, float eps, int algo, uint32_t channel, uint64_t epoch,
                                    uint64_t timeoutNs, int ctas, uint64_t stream) {
        return mf_k_allreduce_rmsnorm((const mf_allreduce_args_t *)argsDev, nEmulated, rankCount, T, H, eps, algo, channel, epoch, timeoutNs, ctas,
                                      (mf_stream_t)stream);
    }, py::arg("args_dev"), py::arg("n_emulated"), py::arg("rank_count"), py::arg("T"), py::arg("H"), py::arg("eps"), py::arg("algo"),
            py::arg("channel"), py::arg("epoch"), py::arg("timeout_ns") = 0, py::arg("ctas") = 0, py::arg("stream") = 0);
}
