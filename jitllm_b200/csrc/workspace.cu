// Places for a call's converted activations where no call of another stream or graph can reach them while it runs.
//
// The kernels that took these calls before read the activations themselves, so calls of one context on several streams, graphs
// replayed side by side, and a graph beside plain calls were all independent, and stay so:
//   the context's own stream (host-pointer calls, trials)   the scratch, which only that stream's call uses at the time
//   a stream that is being captured                         memory of the graph's own, kept until the graph is gone
//   any other stream                                        a slot of its own, for the first eight streams of a context
// Streams are told apart by cudaStreamGetId, which unlike a handle never comes back for another stream; inside a capture, where
// it may not be asked, by the handle.
#include "jl_internal.cuh"

#define JL_MAX_PLACES 64      // graphs' places in use at once; a call that finds none runs on a kernel that needs none

static void CUDART_CB place_gone(void *flag) {
    auto *f = static_cast<std::shared_ptr<std::atomic<bool>> *>(flag);
    (*f)->store(true);
    delete f;
}

bool jl_stream_query(cudaStream_t s, jl_stream_state *q) {
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    q->graph = nullptr;
    q->stream = (unsigned long long)(uintptr_t)s;
    if (cudaStreamGetCaptureInfo(s, &st, &q->capture, &q->graph) != cudaSuccess) { cudaGetLastError(); return false; }
    if (st == cudaStreamCaptureStatusActive) return true;
    q->graph = nullptr;
    if (st != cudaStreamCaptureStatusNone || cudaStreamGetId(s, &q->stream) != cudaSuccess) { cudaGetLastError(); return false; }
    return true;
}

// `bytes` for the calls that a capture takes on one stream (one after the other there): allocated at the first of them, under
// the thread's relaxed capture mode, and given back once the graph, what was instantiated from it and its launches are
// gone -- the runtime then drops the user object that the graph holds.
void *jl_capture_place(jl_ctx *ctx, const jl_stream_state &st, size_t bytes) {
    jl_place *free_place = nullptr;
    for (jl_place &p : ctx->places) {
        if (p.gone->load()) {
            if (p.cap >= bytes && (!free_place || p.cap < free_place->cap)) free_place = &p;
        } else if (p.capture == st.capture && p.stream == st.stream && p.cap >= bytes) {
            return p.mem;
        }
    }
    jl_place q = {};
    if (free_place) {
        q.mem = free_place->mem; q.cap = free_place->cap;
    } else {
        if (ctx->places.size() >= JL_MAX_PLACES) return nullptr;
        q.cap = (bytes + 0xFFFF) & ~(size_t)0xFFFF;
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
        if (cudaThreadExchangeStreamCaptureMode(&mode) != cudaSuccess) { cudaGetLastError(); return nullptr; }
        const cudaError_t e = cudaMalloc(&q.mem, q.cap);
        cudaThreadExchangeStreamCaptureMode(&mode);
        if (e != cudaSuccess) { cudaGetLastError(); return nullptr; }
        ctx->places.push_back(jl_place{q.mem, q.cap, 0, 0, std::make_shared<std::atomic<bool>>(true)});
        free_place = &ctx->places.back();
    }
    auto flag = std::make_shared<std::atomic<bool>>(false);
    auto *held = new std::shared_ptr<std::atomic<bool>>(flag);
    cudaUserObject_t obj = nullptr;
    if (cudaUserObjectCreate(&obj, held, place_gone, 1, cudaUserObjectNoDestructorSync) != cudaSuccess) {
        cudaGetLastError();
        delete held;
        return nullptr;
    }
    if (cudaGraphRetainUserObject(st.graph, obj, 1, cudaGraphUserObjectMove) != cudaSuccess) {
        cudaGetLastError();
        cudaUserObjectRelease(obj, 1);
        return nullptr;
    }
    free_place->capture = st.capture; free_place->stream = st.stream; free_place->gone = flag;
    return q.mem;
}

// Frees the places whose graphs are gone (jl_reserve, uploads), or all (jl_close).
void jl_places_free(jl_ctx *ctx, bool all) {
    for (size_t i = 0; i < ctx->places.size();) {
        if (all || ctx->places[i].gone->load()) {
            cudaFree(ctx->places[i].mem);
            ctx->places[i] = ctx->places.back();
            ctx->places.pop_back();
        } else {
            i++;
        }
    }
}

// Slots of at least `bytes` (jl_reserve, uploads). Without memory for them the calls run on the kernels that need none.
int jl_xop_reserve(jl_ctx *ctx, size_t bytes) {
    bytes = (bytes + 255) & ~(size_t)255;
    if (ctx->xop_slot >= bytes) return JL_OK;
    JL_CUDA(ctx, cudaDeviceSynchronize());       // an earlier launch may still read the old slots
    if (ctx->xop) cudaFree(ctx->xop);
    ctx->xop = nullptr; ctx->xop_slot = 0; ctx->xop_streams = 0;
    if (cudaMalloc(&ctx->xop, bytes * JL_XOP_SLOTS) != cudaSuccess) { cudaGetLastError(); ctx->xop = nullptr; return JL_OK; }
    ctx->xop_slot = bytes;
    return JL_OK;
}

void *jl_operand_place(jl_ctx *ctx, cudaStream_t s, size_t bytes) {
    if (s == ctx->stream) return ctx->scratch_cap >= bytes ? ctx->scratch : nullptr;
    jl_stream_state st;
    if (!jl_stream_query(s, &st)) return nullptr;
    if (st.graph) return jl_capture_place(ctx, st, bytes);
    if (ctx->xop_slot < bytes) return nullptr;
    int i = 0;
    while (i < ctx->xop_streams && ctx->xop_stream[i] != st.stream) i++;
    if (i == JL_XOP_SLOTS) return nullptr;
    if (i == ctx->xop_streams) ctx->xop_stream[ctx->xop_streams++] = st.stream;
    return (uint8_t *)ctx->xop + (size_t)i * ctx->xop_slot;
}
