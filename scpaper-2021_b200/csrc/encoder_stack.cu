// A stack of encoder layers as one host call.  Issuing a layer's four to six kernels costs the host
// 2.7 us each, more than they take on the GPU for short batches (72 launches, 230 us, for twelve layers
// of one 128-token sequence that run in 280 us), so a plan remembers the launches of a call as a CUDA
// graph - programmatic dependencies included - and replays them with one launch when a call comes
// with the same arguments again.  The layers' numbers are read at every replay like at every launch:
// nothing but the list of launches is kept.
//
// A call is captured when its arguments (input, mask, lengths: addresses and kind) are seen for the
// second time; up to PLAN_GRAPHS argument sets are kept, calls with others issue the kernels one by
// one.  So do calls on a stream that is being captured, where the launches join the caller's graph.
#include <mutex>
#include <new>
#include <vector>

#include <string.h>

#include "common.cuh"
#include "kernels.h"

namespace et {
namespace {

constexpr int PLAN_GRAPHS = 8;
constexpr int PLAN_SEEN = 16;

struct StackKey {
    const et_half* x;
    const et_half* mask;
    const int32_t* valid_len;
    int mask_kind;
    bool operator==(const StackKey& o) const {
        return x == o.x && mask == o.mask && valid_len == o.valid_len && mask_kind == o.mask_kind;
    }
};

struct StackGraph {
    StackKey key;
    cudaGraphExec_t exec;
    long long launches;
};

}  // namespace
}  // namespace et

struct et_encoder_stack {
    std::mutex mutex;
    std::vector<et_encoder_layer_t> layers;
    int batch, seq;
    et_half* buf[2];
    void* workspace;
    size_t workspace_bytes;
    int device;
    cudaStream_t capture_stream = nullptr;
    bool graphs_off = false;
    std::vector<et::StackGraph> graphs;
    et::StackKey seen[et::PLAN_SEEN];
    int n_seen = 0, next_seen = 0;
};

namespace et {
namespace {

int run_layers(et_encoder_stack* p, const StackKey& k, cudaStream_t stream) {
    const et_half* cur = k.x;
    for (size_t i = 0; i < p->layers.size(); ++i) {
        et_half* out = p->buf[i & 1];
        const int st = et_encoder_layer_fwd(&p->layers[i], cur, out, p->batch, p->seq, k.mask_kind, k.mask,
                                            k.valid_len, p->workspace, p->workspace_bytes, stream);
        if (st != ET_OK) return st;
        cur = out;
    }
    return ET_OK;
}

void drop_graphs(et_encoder_stack* p) {
    for (StackGraph& g : p->graphs) cudaGraphExecDestroy(g.exec);
    p->graphs.clear();
    p->n_seen = p->next_seen = 0;
}

bool seen_before(et_encoder_stack* p, const StackKey& k) {
    for (int i = 0; i < p->n_seen; ++i)
        if (p->seen[i] == k) return true;
    p->seen[p->next_seen] = k;
    p->next_seen = (p->next_seen + 1) % PLAN_SEEN;
    if (p->n_seen < PLAN_SEEN) ++p->n_seen;
    return false;
}

// Captures the call's launches; on any failure graphs are switched off and the caller issues them.
StackGraph* capture(et_encoder_stack* p, const StackKey& k) {
    if (!p->capture_stream &&
        cudaStreamCreateWithFlags(&p->capture_stream, cudaStreamNonBlocking) != cudaSuccess)
        p->capture_stream = nullptr;
    StackGraph g = {k, nullptr, 0};
    if (p->capture_stream &&
        cudaStreamBeginCapture(p->capture_stream, cudaStreamCaptureModeThreadLocal) == cudaSuccess) {
        const long long before = et_launch_count();
        const int st = run_layers(p, k, p->capture_stream);
        g.launches = et_launch_count() - before;
        count_launches(-g.launches);  // (captured, not launched)
        cudaGraph_t graph = nullptr;
        if (cudaStreamEndCapture(p->capture_stream, &graph) == cudaSuccess && st == ET_OK && graph)
            if (cudaGraphInstantiate(&g.exec, graph, 0) != cudaSuccess) g.exec = nullptr;
        if (graph) cudaGraphDestroy(graph);
    }
    if (!g.exec) {
        cudaGetLastError();
        p->graphs_off = true;
        return nullptr;
    }
    p->graphs.push_back(g);
    return &p->graphs.back();
}

}  // namespace
}  // namespace et

extern "C" {

int et_encoder_stack_create(const et_encoder_layer_t* const* layers, int n_layers, int batch, int seq,
                            et_half* buf0, et_half* buf1, void* workspace, size_t workspace_bytes,
                            et_encoder_stack_t** stack) {
    if (!layers || n_layers <= 0 || batch <= 0 || seq <= 0 || !buf0 || !buf1 || !workspace || !stack)
        return ET_ERR_INVALID_ARG;
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess) return ET_ERR_NO_DEVICE;
    et_encoder_stack* p = new (std::nothrow) et_encoder_stack;
    if (!p) return ET_ERR_WORKSPACE;
    p->layers.resize(static_cast<size_t>(n_layers));
    for (int i = 0; i < n_layers; ++i) {
        if (!layers[i]) {
            delete p;
            return ET_ERR_INVALID_ARG;
        }
        p->layers[i] = *layers[i];
        const size_t need = et_encoder_layer_workspace_bytes(layers[i], batch, seq);
        if (need == 0 || need > workspace_bytes) {
            delete p;
            return need == 0 ? ET_ERR_SHAPE : ET_ERR_WORKSPACE;
        }
    }
    p->batch = batch;
    p->seq = seq;
    p->buf[0] = buf0;
    p->buf[1] = buf1;
    p->workspace = workspace;
    p->workspace_bytes = workspace_bytes;
    p->device = dev;
    *stack = p;
    return ET_OK;
}

int et_encoder_stack_fwd(et_encoder_stack_t* stack, const et_encoder_layer_t* const* layers, const et_half* x,
                         int mask_kind, const et_half* mask, const int32_t* valid_len, et_stream stream) {
    if (!stack || !x) return ET_ERR_INVALID_ARG;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    std::lock_guard<std::mutex> lock(stack->mutex);
    if (layers)  // descriptions changed since: the recorded launches are not these layers' any more
        for (size_t i = 0; i < stack->layers.size(); ++i)
            if (memcmp(&stack->layers[i], layers[i], sizeof(et_encoder_layer_t)) != 0) {
                et::drop_graphs(stack);
                for (size_t j = 0; j < stack->layers.size(); ++j) stack->layers[j] = *layers[j];
                break;
            }
    const et::StackKey key = {x, mask, valid_len, mask_kind};
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    int dev = -1;
    const bool replayable = !stack->graphs_off && cudaGetDevice(&dev) == cudaSuccess && dev == stack->device &&
                            cudaStreamIsCapturing(s, &cs) == cudaSuccess &&
                            cs == cudaStreamCaptureStatusNone;
    if (replayable) {
        et::StackGraph* g = nullptr;
        for (et::StackGraph& c : stack->graphs)
            if (c.key == key) g = &c;
        if (!g && stack->graphs.size() < et::PLAN_GRAPHS && et::seen_before(stack, key))
            g = et::capture(stack, key);
        if (g) {
            et::count_launches(g->launches);
            return cudaGraphLaunch(g->exec, s) == cudaSuccess ? ET_OK : ET_ERR_CUDA;
        }
    }
    return et::run_layers(stack, key, s);
}

int et_encoder_stack_destroy(et_encoder_stack_t* stack) {
    if (!stack) return ET_ERR_INVALID_ARG;
    et::drop_graphs(stack);
    if (stack->capture_stream) cudaStreamDestroy(stack->capture_stream);
    delete stack;
    return ET_OK;
}

}  // extern "C"
