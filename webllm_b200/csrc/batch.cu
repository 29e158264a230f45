// Command batches: record many linear / dequant calls once, submit them together, replay at will.
// Replaces CommandBatch (src/gpu/pipeline.ts:55-117), which packs every dispatch of a forward pass into
// one command encoder and one submit to avoid ~110 us of CPU cost per dispatch. Here a batch is a CUDA
// graph captured from the context's stream. A recorded linear call waits for the calls before it whose tensors it
// reads or overwrites, and for no others: a decode-size call is a few microseconds of latency on a part of the chip, and in
// stream order a layer of them was a chain of those: the seven projections of a 0.5B layer at M = 4 11.9 -> 8.4 us a submit.
// Whatever else is recorded keeps stream order with everything before and after it (the reference's endPass).
#include "common.cuh"

namespace wb {

namespace {

bool overlap(const char *a0, const char *a1, const char *b0, const char *b1) { return a0 < b1 && b0 < a1; }

// The nodes that whatever the stream captures next would wait for.
int capture_state(wb_context *ctx, cudaGraph_t *graph, std::vector<cudaGraphNode_t> *nodes)
{
    cudaStreamCaptureStatus st;
    unsigned long long id;
    const cudaGraphNode_t *deps = nullptr;
    const cudaGraphEdgeData *edges = nullptr;
    size_t n = 0;
    WB_CUDA(cudaStreamGetCaptureInfo_v3(ctx->stream, &st, &id, graph, &deps, &edges, &n));
    if (st != cudaStreamCaptureStatusActive) return fail(WB_ERR_BAD_ARG, "the stream of this context is not being captured");
    nodes->assign(deps, deps + n);
    return WB_OK;
}

int set_capture_state(wb_context *ctx, std::vector<cudaGraphNode_t> &nodes)
{
    WB_CUDA(cudaStreamUpdateCaptureDependencies_v2(ctx->stream, nodes.data(), nullptr, nodes.size(), cudaStreamSetCaptureDependencies));
    return WB_OK;
}

}  // namespace

// Before and after the launch of a recorded call that is one kernel, reads [r0, r1) and constants, and writes [w0, w1).
int record_before(wb_context *ctx, const void *r0, uint64_t r_bytes, const void *w0, uint64_t w_bytes)
{
    BatchOrder &o = ctx->order;
    std::vector<cudaGraphNode_t> now, deps;
    cudaGraph_t graph;
    WB_CHECK(capture_state(ctx, &graph, &now));
    if (now != o.left) o.ops.clear(), o.base = now;  // something else was captured: it, and all before it, comes first
    BatchOrder::Op op;
    op.r0 = (const char *)r0, op.r1 = op.r0 + r_bytes, op.w0 = (const char *)w0, op.w1 = op.w0 + w_bytes;
    // from the last one back, without those that an earlier find already waits for (a plain chain stays one: each call waits for the
    // call before it and may start its prologue under it)
    op.before.assign(o.ops.size(), false);
    for (size_t i = o.ops.size(); i-- > 0;) {
        BatchOrder::Op &b = o.ops[i];
        if (op.before[i] || !(overlap(op.r0, op.r1, b.w0, b.w1) || overlap(op.w0, op.w1, b.r0, b.r1) || overlap(op.w0, op.w1, b.w0, b.w1))) continue;
        deps.push_back(b.node);
        b.leaf = false, op.before[i] = true;
        for (size_t k = 0; k < b.before.size(); k++)
            if (b.before[k]) op.before[k] = true;
    }
    // At most so many abreast: the graph's branches are streams that the driver sets up at wb_batch_end (a layer 0.6 ms, in sequence
    // 0.2), and a chip full of decode-size calls gains nothing from more. (Layer at M = 4, abreast 1 / 2 / 4 / all 7, us a submit at
    // the clocks of an idle chip: 28.7, 20.5, 17.1, 15.7.)
    constexpr size_t kWidth = 8;
    if (deps.empty() && o.ops.size() >= kWidth) {
        const size_t i = o.ops.size() - kWidth;
        deps.push_back(o.ops[i].node);
        o.ops[i].leaf = false, op.before[i] = true;
        for (size_t k = 0; k < o.ops[i].before.size(); k++)
            if (o.ops[i].before[k]) op.before[k] = true;
    }
    if (deps.empty()) deps = o.base;
    if (deps.size() > 1) {  // one node to wait for
        cudaGraphNode_t join;
        WB_CUDA(cudaGraphAddEmptyNode(&join, graph, deps.data(), deps.size()));
        deps.assign(1, join);
    }
    o.ops.push_back(op);
    return set_capture_state(ctx, deps);
}

int record_after(wb_context *ctx)
{
    BatchOrder &o = ctx->order;
    std::vector<cudaGraphNode_t> now;
    cudaGraph_t graph;
    WB_CHECK(capture_state(ctx, &graph, &now));
    if (now.size() != 1) return fail(WB_ERR_CUDA, "a recorded call left %d graph nodes", (int)now.size());
    o.ops.back().node = now[0];
    // whatever is captured by other means waits for all of them (by way of those that no other call waits for)
    now.clear();
    for (const BatchOrder::Op &b : o.ops)
        if (b.leaf) now.push_back(b.node);
    WB_CHECK(set_capture_state(ctx, now));
    return capture_state(ctx, &graph, &o.left);
}

}  // namespace wb

struct wb_batch {
    wb_context *ctx = nullptr;
    cudaGraphExec_t exec = nullptr;
    uint64_t launches = 0;  // kernels per replay
};

using namespace wb;

extern "C" {

int wb_batch_begin(wb_context *ctx)
{
    if (!ctx) return fail(WB_ERR_BAD_ARG, "context is NULL");
    WB_CUDA(cudaSetDevice(ctx->device));
    if (ctx->capturing) return fail(WB_ERR_BAD_ARG, "a batch is already being recorded on this context");
    WB_CUDA(cudaStreamSynchronize(ctx->stream));
    WB_CUDA(cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal));
    ctx->capturing = true;
    ctx->order = BatchOrder();
    ctx->launches_at_capture = ctx->launches;
    return WB_OK;
}

int wb_batch_end(wb_context *ctx, wb_batch **out)
{
    if (!ctx || !out) return fail(WB_ERR_BAD_ARG, "wb_batch_end: NULL argument");
    WB_CUDA(cudaSetDevice(ctx->device));
    if (!ctx->capturing) return fail(WB_ERR_BAD_ARG, "wb_batch_end without wb_batch_begin");
    cudaGraph_t g = nullptr;
    cudaError_t e = cudaStreamEndCapture(ctx->stream, &g);
    ctx->capturing = false;
    ctx->order = BatchOrder();
    const uint64_t recorded = ctx->launches - ctx->launches_at_capture;
    ctx->launches = ctx->launches_at_capture;  // recording launches nothing
    WB_CUDA(e);
    wb_batch *b = new wb_batch();
    b->ctx = ctx;
    b->launches = recorded;
    e = cudaGraphInstantiate(&b->exec, g, 0);
    cudaGraphDestroy(g);
    if (e != cudaSuccess) {
        delete b;
        WB_CUDA(e);
    }
    *out = b;
    return WB_OK;
}

int wb_batch_submit(wb_batch *b)
{
    if (!b) return fail(WB_ERR_BAD_ARG, "batch is NULL");
    WB_CUDA(cudaSetDevice(b->ctx->device));
    WB_CUDA(cudaGraphLaunch(b->exec, b->ctx->stream));
    b->ctx->launches += b->launches;
    return WB_OK;
}

int wb_batch_destroy(wb_batch *b)
{
    if (!b) return WB_OK;
    cudaSetDevice(b->ctx->device);
    cudaStreamSynchronize(b->ctx->stream);
    if (b->exec) cudaGraphExecDestroy(b->exec);
    delete b;
    return WB_OK;
}

}  // extern "C"
