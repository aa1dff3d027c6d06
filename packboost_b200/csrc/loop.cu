// The host side of a round, one call each way: the feature lists go up, the phases of the round are
// enqueued (or replayed as one CUDA graph), the decision log comes down; a log is replayed into node
// arrays.  Through the interpreter these steps cost 0.3 to 0.4 ms a round, more than a small table's
// round takes on the device.

#include <new>

#include "common.cuh"

namespace pb {

namespace {

constexpr int kLoopSlots = 8;

struct RoundLoop {
    cudaEvent_t logged[kLoopSlots] = {};
    cudaGraphExec_t exec = nullptr;
    bool no_graph = false;  // a capture failed: rounds are launched one kernel at a time
    int64_t graph_k = 0, graph_launches = 0, replays = 0;
    ~RoundLoop() {
        if (exec) cudaGraphExecDestroy(exec);
        for (auto e : logged)
            if (e) cudaEventDestroy(e);
    }
};

// lists: device [max_depth][3][k]: global ids, local rows, positions of the sampled features
int enqueue_round(const pb_train_state* st, const int32_t* lists, int64_t k, int64_t apply_previous, void* stream) {
    int rc = pb_round_begin(st, apply_previous, stream);
    for (int64_t d = 0; d < st->max_depth && rc == PB_OK; ++d) {
        const int32_t* l = lists + d * 3 * k;
        rc = pb_depth_hist_score(st, d, l + k, l + 2 * k, k, k, stream);
        if (rc == PB_OK) rc = pb_depth_select(st, d, l, k, stream);
        if (rc == PB_OK) rc = pb_depth_partition(st, d, stream);
    }
    return rc == PB_OK ? pb_round_end(st, stream) : rc;
}

int capture_round(RoundLoop* loop, const pb_train_state* st, const int32_t* lists, int64_t k) {
    cudaStream_t side = nullptr;
    PB_CUDA_TRY(cudaStreamCreateWithFlags(&side, cudaStreamNonBlocking));
    const int64_t before = pb_launch_count();
    cudaGraph_t graph = nullptr;
    cudaError_t e = cudaStreamBeginCapture(side, cudaStreamCaptureModeThreadLocal);
    int rc = PB_OK;
    if (e == cudaSuccess) {
        rc = enqueue_round(st, lists, k, 1, side);
        const cudaError_t end = cudaStreamEndCapture(side, &graph);
        e = rc ? cudaSuccess : end;
    }
    if (rc == PB_OK && e == cudaSuccess) e = cudaGraphInstantiate(&loop->exec, graph, 0);
    if (graph) cudaGraphDestroy(graph);
    cudaStreamDestroy(side);
    if (rc) return rc;
    if (e != cudaSuccess) return fail_cuda(e, "round graph");
    loop->graph_k = k;
    loop->graph_launches = pb_launch_count() - before;
    return PB_OK;
}

}  // namespace

}  // namespace pb

using namespace pb;

extern "C" void* pb_loop_create(void) {
    RoundLoop* l = new (std::nothrow) RoundLoop();
    if (!l) return nullptr;
    for (auto& e : l->logged)
        if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) {
            delete l;
            return nullptr;
        }
    return l;
}

extern "C" void pb_loop_destroy(void* loop) { delete static_cast<RoundLoop*>(loop); }

extern "C" int pb_loop_submit(void* loop_, const pb_train_state* st, int64_t slot, const int32_t* lists_host, int32_t* lists_dev,
                              int64_t k, void* log_host, int64_t apply_previous, int64_t use_graph, void* stream_) {
    RoundLoop* loop = static_cast<RoundLoop*>(loop_);
    PB_REQUIRE(loop && st && lists_host && lists_dev && log_host, "null argument");
    PB_REQUIRE(slot >= 0 && slot < kLoopSlots, "slot out of range");
    PB_REQUIRE(k >= 1 && k <= st->n_features_total, "feature count out of range");
    cudaStream_t stream = (cudaStream_t)stream_;
    void* log_dev = nullptr;
    int64_t log_bytes = 0;
    int rc = pb_round_log_buffer(st, &log_dev, &log_bytes);
    if (rc) return rc;
    PB_CUDA_TRY(cudaMemcpyAsync(lists_dev, lists_host, (size_t)(st->max_depth * 3 * k) * 4, cudaMemcpyHostToDevice, stream));
    // the launches of a round are the same every time: from the second round on they are replayed
    const bool graph = use_graph && apply_previous;
    if (graph && !loop->no_graph && (!loop->exec || loop->graph_k != k)) {
        if (loop->exec) cudaGraphExecDestroy(loop->exec);
        loop->exec = nullptr;
        if (capture_round(loop, st, lists_dev, k) != PB_OK) {
            loop->no_graph = true;
            cudaGetLastError();  // (an argument error shows again in the launches below)
        }
    }
    if (graph && loop->exec) {
        PB_CUDA_TRY(cudaGraphLaunch(loop->exec, stream));
        ++loop->replays;
    } else {
        rc = enqueue_round(st, lists_dev, k, apply_previous, stream_);
        if (rc) return rc;
    }
    PB_CUDA_TRY(cudaMemcpyAsync(log_host, log_dev, (size_t)log_bytes, cudaMemcpyDeviceToHost, stream));
    PB_CUDA_TRY(cudaEventRecord(loop->logged[slot], stream));
    return PB_OK;
}

extern "C" int pb_loop_wait(void* loop, int64_t slot) {
    PB_REQUIRE(loop && slot >= 0 && slot < kLoopSlots, "slot out of range");
    PB_CUDA_TRY(cudaEventSynchronize(static_cast<RoundLoop*>(loop)->logged[slot]));
    return PB_OK;
}

extern "C" int pb_loop_release_graph(void* loop_) {
    RoundLoop* loop = static_cast<RoundLoop*>(loop_);
    PB_REQUIRE(loop, "null argument");
    if (loop->exec) {
        const cudaGraphExec_t exec = loop->exec;
        loop->exec = nullptr;
        PB_CUDA_TRY(cudaGraphExecDestroy(exec));
    }
    return PB_OK;
}

extern "C" int pb_loop_counts(void* loop, int64_t* graph_launches, int64_t* replays) {
    PB_REQUIRE(loop && graph_launches && replays, "null argument");
    *graph_launches = static_cast<RoundLoop*>(loop)->graph_launches;
    *replays = static_cast<RoundLoop*>(loop)->replays;
    return PB_OK;
}

// Node arrays of a round's tree from its decision log, children numbered as they are appended
// (packboost/booster.py:172-190, 527-563).  Arrays hold 2^(max_depth + 1) - 1 nodes.
extern "C" int pb_tree_from_log(const void* log_head, const void* log_winners, int64_t max_depth, int32_t* feature,
                                int32_t* threshold, int32_t* left, int32_t* right, double* value, uint8_t* is_leaf,
                                int64_t* n_nodes) {
    PB_REQUIRE(log_head && log_winners && feature && threshold && left && right && value && is_leaf && n_nodes, "null argument");
    PB_REQUIRE(max_depth >= 1 && max_depth <= PB_MAX_DEPTH, "max_depth out of range");
    const pb_round_log_header* h = static_cast<const pb_round_log_header*>(log_head);
    const pb_winner* winners = static_cast<const pb_winner*>(log_winners);
    if (h->faults != 0) return fail_arg("a wait inside a histogram kernel ran into its limit: the round's sums are not complete");
    const int64_t cap = (2ll << max_depth) - 1;
    auto leaf = [&](int64_t n, double v) {
        feature[n] = -1;
        threshold[n] = 0;
        left[n] = right[n] = -1;
        value[n] = v;
        is_leaf[n] = 1;
    };
    int64_t n = 1;
    leaf(0, h->root_value);
    for (int64_t d = 0; d < max_depth && h->n_ctx[d] > 0; ++d) {
        PB_REQUIRE(h->n_ctx[d] <= (1 << d), "log is damaged: %d nodes at depth %d", h->n_ctx[d], (int)d);
        for (int i = 0; i < h->n_ctx[d]; ++i) {
            const pb_winner& w = winners[(1 << d) - 1 + i];
            if (w.tree_node < 0 || w.tree_node >= n) return fail_arg("device and host child numbering disagree");
            if (w.feature < 0) {
                leaf(w.tree_node, w.left_value);
                continue;
            }
            if (w.left_id != n || w.right_id != n + 1 || n + 2 > cap) return fail_arg("device and host child numbering disagree");
            feature[w.tree_node] = w.feature;
            threshold[w.tree_node] = w.threshold;
            left[w.tree_node] = (int32_t)n;
            right[w.tree_node] = (int32_t)n + 1;
            is_leaf[w.tree_node] = 0;
            leaf(n, w.left_value);
            leaf(n + 1, w.right_value);
            n += 2;
        }
    }
    if (n != h->n_tree_nodes) return fail_arg("device and host tree sizes disagree");
    *n_nodes = n;
    return PB_OK;
}
