// Batch of many resident lattices advanced together (C ABI wake_batch_* in
// include/wake_gpu.h). No reference counterpart: the reference steps one
// LatticeGrid per object and call (src/grid/lattice_grid_2d.cpp:195-265); a
// parameter sweep or a serving loop runs one such object per job. Here every
// member keeps its own state, geometry, parameters and force history (it is an
// ordinary wake_grid), and one step of the whole batch is one launch of k_step_cells_batch: the listed cells of
// every member, then the pure cells of every member.
//
// Each launch reads the member's step arguments from a device table, so members
// of any size share a launch and the per-node arithmetic is the single-lattice
// arithmetic: a member's results do not depend on what else is in the batch.
#include <chrono>
#include <cstring>
#include <string>
#include <vector>

#include "engine.cuh"

using namespace wk;

struct wake_batch {
    struct Member {
        wake_grid* g;
        cudaStream_t saved_stream;  // the member's stream before it joined
    };
    int Q = 0, storage = 0;
    std::vector<Member> members;
    cudaStream_t stream = nullptr;
    bool own_stream = false;

    DevMem d_dom, d_pure, d_listed;
    std::vector<BatchDom> up_dom;  // table as last uploaded
    int n_pure = 0, n_listed = 0;
    bool thermal = false;  // some member has a coupled temperature
    long long state_bytes = 0;  // one state buffer of every member
    int coll = 0, les = 0;
    int parity = 0;  // batch steps taken, mod 2

    // cell lists are rebuilt when the members or any member's geometry change
    std::vector<std::pair<const wake_grid*, unsigned long long>> layout;
    unsigned shape = 0;  // bumped when launch shapes or table addresses change
    // host seconds spent in wake_batch_step: preparing members and tables, capturing and
    // instantiating graphs, issuing launches (a launch that waits for queue space counts here)
    double host_s[3] = {0.0, 0.0, 0.0};

    int tpb = 64;

    cudaGraphExec_t graph = nullptr;
    int graph_steps = 0, graph_parity = -1;
    unsigned graph_shape = ~0u;

    ~wake_batch() {
        if (stream && cudaStreamSynchronize(stream) == cudaSuccess) {
            d_dom.release();
            d_pure.release();
            d_listed.release();
        }
        if (graph) cudaGraphExecDestroy(graph);
        if (own_stream && stream) cudaStreamDestroy(stream);
    }
    void drop_graph() {
        if (graph) cudaGraphExecDestroy(graph);
        graph = nullptr;
        graph_shape = ~0u;
    }
};

namespace {

bool valid_batch(wake_batch* b) {
    if (!b) {
        set_error(WAKE_ERR_INVALID, "null wake_batch handle");
        return false;
    }
    return true;
}

// Rebuild the concatenated cell lists when the membership or a member's geometry changed.
int build_cells(wake_batch* b) {
    std::vector<std::pair<const wake_grid*, unsigned long long>> layout;
    layout.reserve(b->members.size());
    for (const auto& m : b->members) layout.emplace_back(m.g, m.g->units_version);
    if (layout == b->layout) return WAKE_OK;
    // queued steps may still read the old lists: let them finish, then lists can move freely
    WK_CUDA(cudaStreamSynchronize(b->stream));
    std::vector<uint2> pure, listed;
    for (std::size_t i = 0; i < b->members.size(); ++i) {
        const wake_grid* g = b->members[i].g;
        const unsigned m = static_cast<unsigned>(i);
        if (!g->narrow()) continue;  // stepped by its own launches
        if (g->mem_on) listed.push_back(make_uint2(m, LISTED_SUM));
        for (unsigned w : g->cells.units)
            if (!(w & UNIT_PURE)) listed.push_back(make_uint2(m, w));
        // its pure cells, linear and listed, in node order
        const auto cell = [&](unsigned i, unsigned nodes, bool zh) {
            pure.push_back(make_uint2(m | (nodes - 1u) << 24 | (zh ? 1u << 30 : 0u), i));
        };
        unsigned e = g->cells.general;
        const std::vector<uint4>& list = g->cells.cells;
        const auto listed_before = [&](unsigned i) {
            for (; e < list.size() && list[e].x < i; ++e) cell(list[e].x, list[e].y & 0xffu, list[e].y & LIST_ZH);
        };
        for (std::size_t c = 0; c < g->h_kind.size(); ++c) {
            if (!(g->h_kind[c] & CELL_PURE)) continue;
            const unsigned i = static_cast<unsigned>(c) * CELL;
            listed_before(i);
            cell(i, std::min<unsigned>(CELL, static_cast<unsigned>(g->N) - i), g->h_kind[c] & CELL_ZH);
        }
        listed_before(0xffffffffu);
    }
    WK_CUDA(b->d_pure.grow(sizeof(uint2) * std::max<std::size_t>(1, pure.size())));
    WK_CUDA(b->d_listed.grow(sizeof(uint2) * std::max<std::size_t>(1, listed.size())));
    if (!pure.empty())
        WK_CUDA(cudaMemcpyAsync(b->d_pure.p, pure.data(), sizeof(uint2) * pure.size(), cudaMemcpyHostToDevice, b->stream));
    if (!listed.empty())
        WK_CUDA(cudaMemcpyAsync(b->d_listed.p, listed.data(), sizeof(uint2) * listed.size(), cudaMemcpyHostToDevice,
                                b->stream));
    WK_CUDA(cudaStreamSynchronize(b->stream));  // the host vectors go out of scope
    b->n_pure = static_cast<int>(pure.size());
    b->n_listed = static_cast<int>(listed.size());
    b->layout = std::move(layout);
    b->up_dom.clear();  // force a table upload
    ++b->shape;
    return WAKE_OK;
}

// Step-argument table of the current members; uploaded when changed.
int build_tables(wake_batch* b) {
    const std::size_t n = b->members.size();
    std::vector<BatchDom> dom(n);
    bool thermal = false;
    b->state_bytes = 0;
    for (std::size_t i = 0; i < n; ++i) {
        wake_grid* g = b->members[i].g;
        BatchDom d;
        std::memset(&d, 0, sizeof d);
        d.a = grid_step_args(g);
        d.buf[0] = g->A.p;
        d.buf[1] = g->B.p;
        d.tbuf[0] = g->tbuf(0);
        d.tbuf[1] = g->tbuf(1);
        d.cur0 = g->cur ^ b->parity;
        d.alone = g->narrow() ? 0 : 1;
        dom[i] = d;
        thermal = thermal || g->th.on;
        b->state_bytes += static_cast<long long>(g->elem) * g->Q * g->pitch;
    }
    if (thermal != b->thermal) {
        b->thermal = thermal;
        ++b->shape;  // a captured graph holds the other kernel
    }
    if (dom.size() == b->up_dom.size() &&
        (dom.empty() || std::memcmp(dom.data(), b->up_dom.data(), sizeof(BatchDom) * n) == 0))
        return WAKE_OK;
    // a captured graph keeps launch shapes and table addresses, not the table contents; only the launches of a member
    // that is stepped by itself hold its arguments by value
    for (std::size_t i = 0; i < n; ++i)
        if (dom[i].alone && i < b->up_dom.size() && std::memcmp(&dom[i], &b->up_dom[i], sizeof(BatchDom)) != 0) {
            ++b->shape;
            break;
        }
    WK_CUDA(cudaStreamSynchronize(b->stream));  // queued steps may still read the old table
    const void* old_dom = b->d_dom.p;
    WK_CUDA(b->d_dom.grow(sizeof(BatchDom) * std::max<std::size_t>(1, n)));
    if (n) WK_CUDA(cudaMemcpyAsync(b->d_dom.p, dom.data(), sizeof(BatchDom) * n, cudaMemcpyHostToDevice, b->stream));
    WK_CUDA(cudaStreamSynchronize(b->stream));
    b->up_dom = std::move(dom);
    if (old_dom != b->d_dom.p) ++b->shape;
    return WAKE_OK;
}

int batch_steps(wake_batch* b, int n) {
    for (int s = 0; s < n; ++s) {
        BatchArgs a{};
        a.dom = b->d_dom.as<BatchDom>();
        a.listed = b->d_listed.as<uint2>();
        a.nlisted = static_cast<unsigned>(b->n_listed);
        a.pure = b->d_pure.as<uint2>();
        a.npure = static_cast<unsigned>(b->n_pure);
        a.parity = b->parity;
        a.evict_first = fits_l2(b->members[0].g, b->state_bytes);
        WK_CUDA(launch_batch_any(b->Q, b->coll, b->storage, b->les != 0, a, b->thermal, b->tpb, b->stream));
        for (std::size_t i = 0; i < b->up_dom.size(); ++i) {
            if (!b->up_dom[i].alone) continue;
            wake_grid* g = b->members[i].g;
            StepArgs one = b->up_dom[i].a;
            grid_step_buffers(g, b->up_dom[i].cur0 ^ b->parity, one);
            WK_CUDA(launch_cells_any(b->Q, b->coll, b->storage, b->les != 0, one, b->tpb, b->stream));
        }
        b->parity ^= 1;
    }
    return WAKE_OK;
}

// Prepare every member and the tables for the next steps.
int batch_prepare(wake_batch* b) {
    if (b->members.empty()) return WAKE_OK;
    const wake_grid* g0 = b->members[0].g;
    for (const auto& m : b->members) {
        if (m.g->collision != g0->collision || m.g->les != g0->les)
            return set_error(WAKE_ERR_INVALID, "wake_batch: members differ in collision model or LES switch");
    }
    if (b->coll != g0->collision || b->les != g0->les) {
        b->coll = g0->collision;
        b->les = g0->les;
        ++b->shape;  // a captured graph holds the other model's kernel
    }
    for (const auto& m : b->members) {
        const int r = grid_prepare(m.g);
        if (r) return r;
    }
    int r = build_cells(b);
    if (r) return r;
    return build_tables(b);
}

}  // namespace

extern "C" {

wake_batch* wake_batch_create(int q, int storage) {
    if (!(q == 9 || q == 19 || q == 27) || storage < 0 || storage > 3) {
        set_error(WAKE_ERR_INVALID, "wake_batch_create: invalid lattice or storage");
        return nullptr;
    }
    auto* b = new wake_batch();
    b->Q = q;
    b->storage = storage;
    cudaError_t e = cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking);
    if (e == cudaSuccess) b->own_stream = true;
    if (e != cudaSuccess) {
        set_error(WAKE_ERR_CUDA, std::string("wake_batch_create: ") + cudaGetErrorString(e));
        delete b;
        return nullptr;
    }
    return b;
}

void wake_batch_destroy(wake_batch* b) {
    if (!b) return;
    if (b->stream) cudaStreamSynchronize(b->stream);
    for (auto& m : b->members) wake_grid_set_stream(m.g, m.saved_stream);
    delete b;
}

int wake_batch_add(wake_batch* b, wake_grid* g) {
    if (!valid_batch(b) || !grid_valid(g)) return WAKE_ERR_INVALID;
    if (g->Q != b->Q || g->storage != b->storage)
        return set_error(WAKE_ERR_INVALID, "wake_batch_add: lattice or storage differs from the batch");
    for (const auto& m : b->members)
        if (m.g == g) return set_error(WAKE_ERR_INVALID, "wake_batch_add: grid is already a member");
    // the member's work (preparation, reads) is ordered on the batch stream from now on
    WK_CUDA(cudaStreamSynchronize(g->stream));
    const cudaStream_t saved = g->own_stream ? nullptr : g->stream;
    int r = wake_grid_set_stream(g, b->stream);
    if (r) return r;
    b->members.push_back({g, saved});
    return static_cast<int>(b->members.size()) - 1;
}

int wake_batch_remove(wake_batch* b, wake_grid* g) {
    if (!valid_batch(b) || !grid_valid(g)) return WAKE_ERR_INVALID;
    for (std::size_t i = 0; i < b->members.size(); ++i) {
        if (b->members[i].g != g) continue;
        WK_CUDA(cudaStreamSynchronize(b->stream));
        const cudaStream_t saved = b->members[i].saved_stream;
        b->members.erase(b->members.begin() + static_cast<long>(i));
        return wake_grid_set_stream(g, saved);
    }
    return set_error(WAKE_ERR_INVALID, "wake_batch_remove: grid is not a member");
}

int wake_batch_size(wake_batch* b) { return valid_batch(b) ? static_cast<int>(b->members.size()) : WAKE_ERR_INVALID; }

int wake_batch_set_stream(wake_batch* b, void* stream) {
    if (!valid_batch(b)) return WAKE_ERR_INVALID;
    WK_CUDA(cudaStreamSynchronize(b->stream));
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (!s) {
        if (!b->own_stream) {
            WK_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
            b->own_stream = true;
        } else {
            s = b->stream;
        }
    } else if (b->own_stream) {
        cudaStreamDestroy(b->stream);
        b->own_stream = false;
    }
    b->stream = s;
    for (auto& m : b->members) {
        const int r = wake_grid_set_stream(m.g, s);
        if (r) return r;
    }
    b->drop_graph();
    return WAKE_OK;
}

int wake_batch_use_graph(wake_batch* b, int steps_per_graph) {
    if (!valid_batch(b)) return WAKE_ERR_INVALID;
    if (steps_per_graph < 0) return set_error(WAKE_ERR_INVALID, "negative graph size");
    b->graph_steps = steps_per_graph > 0 && steps_per_graph % 2 ? steps_per_graph + 1 : steps_per_graph;
    b->drop_graph();
    return WAKE_OK;
}

int wake_batch_set_block(wake_batch* b, int threads_bulk, int threads_general) {
    if (!valid_batch(b)) return WAKE_ERR_INVALID;
    if (threads_bulk < 32 || threads_bulk > WK_FAST_MAX_THREADS || threads_bulk % 32 || threads_general < 32 ||
        threads_general > 512 || threads_general % 32)
        return set_error(WAKE_ERR_INVALID, "wake_batch_set_block: bulk 32 or 64 (the step kernel's bound), "
                                           "general 32..512, multiples of 32");
    b->tpb = threads_bulk;  // one launch steps the general rows too
    b->drop_graph();
    return WAKE_OK;
}

int wake_batch_get_block(wake_batch* b) { return valid_batch(b) ? b->tpb : WAKE_ERR_INVALID; }

int wake_batch_set_kernel(wake_batch* b, int variant) {
    if (!valid_batch(b)) return WAKE_ERR_INVALID;
    if (variant < 0 || variant > 2) return set_error(WAKE_ERR_INVALID, "wake_batch_set_kernel: variant 0, 1 or 2");
    return WAKE_OK;  // every variant gives the same results; a batch has the direct kernel only
}

int wake_batch_step(wake_batch* b, int n) {
    if (!valid_batch(b)) return WAKE_ERR_INVALID;
    if (n < 0) return set_error(WAKE_ERR_INVALID, "negative step count");
    if (n == 0 || b->members.empty()) return WAKE_OK;
    using clock = std::chrono::steady_clock;
    auto t0 = clock::now();
    auto lap = [&](int phase) {
        const auto t = clock::now();
        b->host_s[phase] += std::chrono::duration<double>(t - t0).count();
        t0 = t;
    };
    int r = batch_prepare(b);
    lap(0);
    if (r) return r;
    int done = 0;
    const int gs = b->graph_steps;
    if (gs > 0 && n >= gs) {
        if (!b->graph || b->graph_shape != b->shape || b->graph_parity != b->parity) {
            b->drop_graph();
            const int p0 = b->parity;
            cudaGraph_t graph = nullptr;
            WK_CUDA(cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal));
            r = batch_steps(b, gs);
            const cudaError_t e = cudaStreamEndCapture(b->stream, &graph);
            b->parity = p0;
            if (r) {
                if (graph) cudaGraphDestroy(graph);
                return r;
            }
            if (e != cudaSuccess) return set_error(WAKE_ERR_CUDA, std::string("batch graph capture: ") + cudaGetErrorString(e));
            const cudaError_t e2 = cudaGraphInstantiate(&b->graph, graph, 0);
            cudaGraphDestroy(graph);
            if (e2 != cudaSuccess) {
                b->graph = nullptr;
                return set_error(WAKE_ERR_CUDA, std::string("batch graph instantiate: ") + cudaGetErrorString(e2));
            }
            const cudaError_t e3 = cudaGraphUpload(b->graph, b->stream);
            if (e3 != cudaSuccess) return set_error(WAKE_ERR_CUDA, std::string("batch graph upload: ") + cudaGetErrorString(e3));
            b->graph_shape = b->shape;
            b->graph_parity = p0;
        }
        lap(1);
        while (n - done >= gs) {  // gs is even: the parity returns to graph_parity
            WK_CUDA(cudaGraphLaunch(b->graph, b->stream));
            done += gs;
        }
    }
    r = batch_steps(b, n - done);
    for (auto& m : b->members) grid_advanced(m.g, n);
    lap(2);
    return r;
}

int wake_batch_host_seconds(wake_batch* b, double* prepare_s, double* capture_s, double* launch_s) {
    if (!valid_batch(b)) return WAKE_ERR_INVALID;
    if (prepare_s) *prepare_s = b->host_s[0];
    if (capture_s) *capture_s = b->host_s[1];
    if (launch_s) *launch_s = b->host_s[2];
    return WAKE_OK;
}

int wake_batch_synchronize(wake_batch* b) {
    if (!valid_batch(b)) return WAKE_ERR_INVALID;
    WK_CUDA(cudaStreamSynchronize(b->stream));
    for (std::size_t i = 0; i < b->members.size(); ++i) {
        const int r = grid_check_status(b->members[i].g);
        if (r) return set_error(r, "wake_batch member " + std::to_string(i) + ": " + wake_gpu_last_error());
    }
    return WAKE_OK;
}

int wake_batch_info(wake_batch* b, long long* nodes, int* bulk_rows, int* general_rows, int* launches_per_step) {
    if (!valid_batch(b)) return WAKE_ERR_INVALID;
    const int r = batch_prepare(b);
    if (r) return r;
    long long nn = 0;
    for (const auto& m : b->members) nn += m.g->N;
    if (nodes) *nodes = nn;
    if (bulk_rows) *bulk_rows = b->n_pure;
    if (general_rows) *general_rows = b->n_listed;
    if (launches_per_step) {
        *launches_per_step = b->n_pure + b->n_listed > 0 ? 1 : 0;
        for (const BatchDom& d : b->up_dom) *launches_per_step += d.alone;
    }
    return WAKE_OK;
}

// Time `steps` real steps for each block size of {32, 64, 128, 256} within the
// kernel's launch bound (plain launches, CUDA events on the batch stream) and keep
// the fastest. The members advance `steps` per size tried; results do not depend on
// the block size.
int wake_batch_autotune(wake_batch* b, int steps, int* best_threads) {
    if (!valid_batch(b)) return WAKE_ERR_INVALID;
    if (steps < 1) return set_error(WAKE_ERR_INVALID, "wake_batch_autotune: steps must be positive");
    if (b->members.empty()) return WAKE_OK;
    int r = batch_prepare(b);
    if (r) return r;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    WK_CUDA(cudaEventCreate(&e0));
    if (cudaEventCreate(&e1) != cudaSuccess) {
        cudaEventDestroy(e0);
        return set_error(WAKE_ERR_CUDA, "wake_batch_autotune: event creation failed");
    }
    const int keep = b->tpb;
    int best = keep;
    float best_ms = -1.f;
    for (int t : {32, 64, 128, 256}) {
        if (t > WK_FAST_MAX_THREADS) break;
        b->tpb = t;
        cudaEventRecord(e0, b->stream);
        r = batch_steps(b, steps);
        cudaEventRecord(e1, b->stream);
        if (r) break;
        for (auto& m : b->members) grid_advanced(m.g, steps);
        float ms = 0.f;
        if (cudaEventSynchronize(e1) != cudaSuccess || cudaEventElapsedTime(&ms, e0, e1) != cudaSuccess) {
            r = set_error(WAKE_ERR_CUDA, "wake_batch_autotune: timing failed");
            break;
        }
        if (best_ms < 0.f || ms < best_ms) {
            best_ms = ms;
            best = t;
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    b->tpb = r ? keep : best;
    b->drop_graph();
    if (best_threads) *best_threads = b->tpb;
    return r;
}

}  // extern "C"
