// Host state of one resident lattice (wake_grid) shared by the single-lattice
// engine (engine.cu) and the batch of many lattices (batch.cu).
#pragma once

#include <algorithm>
#include <string>
#include <vector>

#include "common.cuh"
#include "kernels.cuh"
#include "wake_gpu.h"

namespace wk {

// ---------------------------------------------------------------- host lattice tables
struct HostLat {
    int Q = 0, D = 0;
    int cx[27], cy[27], cz[27], opp[27];
    float w[27];
    explicit HostLat(int q) : Q(q) {
        auto fill = [&](auto lat) {
            using L = decltype(lat);
            D = L::D;
            for (int k = 0; k < Q; ++k) {
                cx[k] = L::cx(k);
                cy[k] = L::cy(k);
                cz[k] = L::cz(k);
                opp[k] = L::opp(k);
                w[k] = L::w(k);
            }
        };
        if (q == 9) fill(Lat<9>{});
        else if (q == 19) fill(Lat<19>{});
        else fill(Lat<27>{});
    }
};

// Bounding box (inclusive) and shape of a device rasteriser call (k_rasterise in engine.cu).
struct RasterBox {
    int x0, x1, y0, y1, z0, z1;
};
struct RasterShape {
    int kind;     // 0 circle, 1 sphere, 2 rotated ellipse
    float c[3];   // centre
    float p[4];   // circle / sphere: r^2; ellipse: cos, sin, 1/a^2, 1/b^2
};

cudaError_t launch_cells_any(int Q, int coll, int store, bool les, const StepArgs& a, int tpb, cudaStream_t stream);
cudaError_t launch_batch_any(int Q, int coll, int store, bool les, const BatchArgs& b, bool thermal, int tpb,
                             cudaStream_t stream);
cudaError_t launch_tiles_any(int Q, int coll, int store, bool les, const StepArgs& a, const TileArgs& t,
                             cudaStream_t stream);
cudaError_t launch_rows_any(int Q, int store, bool les, const StepArgs& a, int rows, int tpb, cudaStream_t stream);
cudaError_t launch_rows_pipe_any(int Q, int store, bool les, int cap, const StepArgs& a, const PipeArgs& p,
                                 cudaStream_t stream);

// Listed cells of k_step_cells on the device (cells.cuh), for one set of flags.
struct CellList {
    DevMem list, records, d_units, slot, contrib;
    unsigned general = 0;               // the first cells of `list`, with records; the others are pure
    std::vector<uint4> cells;           // the list with its LIST_* bits
    std::vector<unsigned> units;        // for `mode` (0: not made yet)
    int mode = 0, slots = 0;
    long long stride = 3;               // doubles of one half of contrib
    unsigned long long version = 0;     // geom_version it was built for (0: never)
    void release() {
        for (DevMem* m : {&list, &records, &d_units, &slot, &contrib}) m->release();
    }
    std::size_t bytes() const { return list.bytes + records.bytes + d_units.bytes + slot.bytes + contrib.bytes; }
};

}  // namespace wk

using wk::DevMem;
using wk::HostLat;
using wk::Physics;
using wk::Geo;
using wk::Links;
using wk::Launch;
using wk::StepArgs;

struct wake_grid {
    int Q = 0, D = 0, nx = 0, ny = 0, nz = 0, storage = 0;
    long long N = 0, pitch = 0;
    std::size_t elem = 4;
    HostLat lat{9};

    DevMem A, B;       // state buffers
    int cur = 0;       // 0: A holds the current state, 1: B
    // State machine. m_f (FP32) holds the reference-visible f^k whenever mf_valid.
    // `pending`: A/B do not hold Collide(f^k) for the current collision parameters
    // (fresh initial state, or tau / model / body force changed since the last
    // collide); the next step re-collides f^k from m_f first, exactly like the
    // reference, whose step k+1 starts by colliding f^k with that step's parameters.
    bool pending = true;
    bool mf_valid = false;
    float collided_g[3] = {0.f, 0.f, 0.f};  // body force the state buffers were collided with
    float last_step_g[3] = {0.f, 0.f, 0.f};  // body force of the last executed step
    DevMem d_types, d_flags, d_status, d_nodestart;
    // Cell types live in two copies: `types` on the host (single-cell edits, face setters,
    // reads) and d_types on the device (flag builds, link candidates, the shape rasterisers).
    // The flags say which copy holds edits the other lacks; copies move only when needed.
    std::vector<uint8_t> types;
    bool types_host_newer = true;
    bool types_dev_newer = false;
    bool geom_dirty = true;

    int collision = WAKE_MRT, les = 0;
    Physics phys{};
    int inflow = 0, outflow = 0, lid = 0, periodic_y = 0, periodic_z = 0;
    float uin[3] = {0.f, 0.f, 0.f}, rho_out = 1.0f, uw[3] = {0.f, 0.f, 0.f};

    std::vector<int> link_node, link_q;
    std::vector<float> link_delta, link_uw;  // uw: 3 per link
    DevMem d_link_node, d_link_rec, d_link_mom;
    std::vector<int> dev_link_node;  // node of each uploaded link
    int dev_links = 0;         // links currently on the device (the flags refer to these)
    bool links_dirty = false;  // host links differ from the device copy

    int mem_on = 0, hist_cap = 0;
    float center[3] = {0.f, 0.f, 0.f}, rmax = 0.f;
    DevMem d_left, d_hist;  // MemLeft, history
    // the history's length as read last, the value of mem_issued then (~0: never); calls that issued steps with forces on
    long long hist_seen = 0;
    unsigned long long seen_at = ~0ull, mem_issued = 0;
    // whether the last step's force may still be outstanding, and whether steps were captured into a caller's graph, whose
    // replays leave forces unseen by the host
    bool mem_left = false, mem_captured = false;

    // k_step_cells: what the linear cells and the segments are, and the cells that are listed
    DevMem d_kind, d_seg;
    unsigned long long seg_version = 0;  // geom_version of d_seg
    std::vector<uint8_t> h_kind, h_seg;
    wk::CellList cells;
    unsigned long long units_version = 0;  // a fresh number whenever units are made (next_geom_version)
    long long cell_nodes = 0;  // nodes of the segments that are not all solid
    // Identity of the current flags / cell lists: a fresh process-wide number at every
    // rebuild (next_geom_version), so a batch never takes a new grid that happens to
    // reuse a destroyed grid's address for the old one.
    unsigned long long geom_version = 0;

    int l2_bytes = 0;  // L2 cache of the lattice's device
    int tpb = 0, xchunks = 1, rows = 1, tpb_cells = 64;
    // step kernels: 0 automatic, 1 direct (k_step_cells over the whole lattice), 2 to 4 a bulk kernel for the
    // rows whose every node is a pure gather (ROW_FAST) beside k_step_cells for the other rows (`rest`):
    // 2 persistent tiles (k_step_tiles), 3 one block per row (k_step_rows, TRT), 4 rows moved through shared
    // memory by bulk copies (k_step_rows_pipe, TRT; the automatic choice for 16-bit storage).
    int kernel_variant = 0;
    DevMem d_row_kind, d_row_list, d_tiles;  // ROW_* byte per row; ROW_FAST rows (row | bits << 28); tiles of them
    int n_row_fast = 0, n_tiles = 0;
    wk::CellList rest;
    bool narrow() const { return static_cast<long long>(Q) * pitch < (1ll << 32); }
    bool tiles_fit() const { return kernel_variant == 2 && wk::tile_row_ok(nx, static_cast<int>(elem)) && !th.on; }
    bool rows_fit() const { return kernel_variant == 3 && collision == WAKE_TRT && nx % 2 == 0 && narrow() && !th.on; }
    int pipe_cap() const { return nx <= 256 ? 256 : 512; }
    bool pipe_fits() const {
        const bool chosen = kernel_variant == 4 || (kernel_variant == 0 && storage != 0);
        return chosen && collision == WAKE_TRT && nx % 2 == 0 && nx <= 512 &&
               (static_cast<long long>(nx) * static_cast<long long>(elem)) % 16 == 0 && narrow() && !th.on &&
               rows < (1 << 28);
    }
    // (the row tables of the current flags exist once prepared)
    bool use_tiles() const { return tiles_fit(); }
    bool use_rows() const { return rows_fit() && n_row_fast > 0; }
    bool use_pipe() const { return pipe_fits() && n_row_fast > 0; }
    bool by_rows() const { return use_tiles() || use_rows() || use_pipe(); }
    int tpb_rows() const { return nx <= 64 ? 32 : 64; }
    cudaStream_t stream = nullptr;
    bool own_stream = false;
    cudaStream_t side = nullptr;  // forked stream of the rows beside a bulk kernel
    cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
    long long k = 0;

    DevMem m_f, m_rho, m_ux, m_uy, m_uz, m_speed, m_diag;
    DevMem m_an;  // field analytics: vorticity (2D) or omega x/y/z + Q (3D), and the |max| word

    // coupled D2Q5 temperature (D2Q9 lattices): post-collision populations in TA / TB
    // (same parity as A / B), FP32 start-up populations in m_t
    wk::Thermal th{};
    DevMem TA, TB, m_t;
    bool mt_valid = false;
    float* tbuf(int which) const { return static_cast<float*>(which == 0 ? TA.p : TB.p); }

    // CUDA graph of `graph_steps` fused steps starting from buffer parity graph_cur
    cudaGraphExec_t graph = nullptr;
    int graph_steps = 0, graph_cur = -1;
    float graph_g[3] = {0.f, 0.f, 0.f};
    bool graph_ok = false;

    // Optional CUDA-event timing of every pure-gather (bulk) launch; plain launches only.
    bool time_bulk = false;
    std::vector<cudaEvent_t> t_ev;  // pairs (start, end), reused
    std::size_t t_used = 0;         // events recorded since the last read

    explicit wake_grid(int q) : lat(q) {}
    ~wake_grid() {
        // every queued use of the blocks ends here, so they go back to the cache
        // (no device-wide cudaFree while other lattices run)
        bool idle = true;
        if (stream) idle = cudaStreamSynchronize(stream) == cudaSuccess;
        if (side) idle = idle && cudaStreamSynchronize(side) == cudaSuccess;
        if (idle) {
            DevMem* all[] = {&A, &B, &d_types, &d_flags, &d_status, &d_nodestart, &d_link_node, &d_link_rec,
                             &d_link_mom, &d_left, &d_hist, &d_kind, &d_seg, &d_row_kind, &d_row_list, &d_tiles, &m_f,
                             &m_rho, &m_ux, &m_uy, &m_uz, &m_speed, &m_diag, &TA, &TB, &m_t, &m_an};
            cells.release();
            rest.release();
            for (DevMem* m : all) m->release();
        }
        for (cudaEvent_t e : t_ev) cudaEventDestroy(e);
        if (graph) cudaGraphExecDestroy(graph);
        if (own_stream && stream) cudaStreamDestroy(stream);
        if (side) cudaStreamDestroy(side);
        if (ev_fork) cudaEventDestroy(ev_fork);
        if (ev_join) cudaEventDestroy(ev_join);
    }

    void* buf(int which) { return which == 0 ? A.p : B.p; }

    Geo geo() const {
        Geo g{};
        g.nx = nx;
        g.ny = ny;
        g.nz = nz;
        g.by_nx = wk::FastDiv::of(static_cast<unsigned>(nx));
        g.by_ny = wk::FastDiv::of(static_cast<unsigned>(ny));
        g.periodic_y = (D == 3) ? periodic_y : 0;
        g.periodic_z = (D == 3) ? periodic_z : 0;
        g.pitch = pitch;
        for (int a = 0; a < 3; ++a) g.uin[a] = uin[a];
        g.rho_out = rho_out;
        for (int q = 0; q < Q; ++q) {
            // 2 w_q rho_0 / cs^2 (c_q . u_w) in the reference's float order (d2q9_streaming.ispc:49-53)
            const float ci_uw = float(lat.cx[q]) * uw[0] + float(lat.cy[q]) * uw[1] + float(lat.cz[q]) * uw[2];
            g.mom[q] = lid ? 2.0f * lat.w[q] * 1.0f * 3.0f * ci_uw : 0.0f;
        }
        return g;
    }
    Links links() const {
        Links l{};
        l.node_start = d_nodestart.as<int>();
        l.rec = d_link_rec.as<uint4>();
        l.mom = d_link_mom.as<float>();
        l.count = dev_links;
        return l;
    }
    Launch launch() const { return Launch{tpb, xchunks, rows, stream, ny, nz}; }
    int blocks() const { return rows * xchunks; }

    void invalidate_graph() { graph_ok = false; }

    void choose_block(int want) {
        const int full = ((nx + 31) / 32) * 32;
        if (want > 0) tpb = want;
        else if (full <= 512) tpb = full;
        else {
            int best = 256;
            long long best_waste = -1;
            for (int t : {256, 384, 512}) {
                const long long chunks = (nx + t - 1) / t;
                const long long waste = chunks * t - nx;
                if (best_waste < 0 || waste < best_waste) {
                    best = t;
                    best_waste = waste;
                }
            }
            tpb = best;
        }
        xchunks = (nx + tpb - 1) / tpb;
        rows = ny * nz;
        tpb_cells = want > 0 ? std::max(32, std::min(want, WK_FAST_MAX_THREADS)) : WK_FAST_MAX_THREADS;
    }
};

namespace wk {

// Validity check that records the error (WAKE_ERR_INVALID) for a null handle.
bool grid_valid(wake_grid* g);
// Bring a lattice to the point where its state buffers hold Collide(f^k) for the
// current geometry and parameters (rebuilds flags, re-collides when pending) and
// its cell list is built.
int grid_prepare(wake_grid* g);
unsigned long long next_geom_version();
// Step arguments of one lattice: the direct range and its listed cells, or the rows beside a bulk kernel
// (buffers left for the caller).
StepArgs grid_step_args(const wake_grid* g, bool rest = false);
bool fits_l2(const wake_grid* g, long long bytes);
// Its buffers: the state in buf(cur), the step's output in the other one.
void grid_step_buffers(wake_grid* g, int cur, StepArgs& a);
// The last step left its force outstanding.
void grid_force_left(wake_grid* g);
// Bookkeeping after n steps run outside wake_grid_step (by a batch).
void grid_advanced(wake_grid* g, int n);
// Error status word of the lattice: WAKE_OK or WAKE_ERR_NUMERIC (synchronizes its stream).
int grid_check_status(wake_grid* g);

}  // namespace wk
