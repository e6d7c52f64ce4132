// Step kernel over cells: up to CELL consecutive nodes of the linear node order (z * ny + y) * nx + x, stepped by one
// warp (two nodes per thread in packed FP32, pairs2.cuh) or two (one node per thread). One launch steps the lattice.
//
// Cells ignore the row ends, so nearly every warp is full whatever nx is. Rows cut into 64-node pieces leave lanes
// idle wherever nx is no multiple of 64 (81-node rows: 64 + 17; 81^3 sphere channel, D3Q19 FP32: 26.2 -> 14.4 us a
// step, 97^3 38.9 -> 26.1, 160^3 152 -> 112). A node's pull sources are its own index plus one of three x, y
// and z offsets (the periodic wraps included), so a load costs one or two integer adds.
//
// Two kinds of cells. A pure one, all in segments of pure gathers (FL_FAST), reads nothing but its class and the
// populations: the linear cells (node number / CELL) by their index, the others from a list. The general ones are
// listed, each node with a 16-byte record built when the geometry changes: which pulls bounce back, which
// of those are momentum-exchange or moving-wall links, where its curved links start. The
// general path is a latency chain (record -> populations -> curved links); the record
// replaces one flag read per direction in it, the packed links a serial walk per link.
// The blocks of the listed cells are spread over the first part of the launch (which_block), so the chain runs
// under the linear cells. Each general cell leaves the sum of its momentum exchange in a slot; the next step's
// launch adds the slots up (a host read of the history does it after the last step), where nothing waits for it.
//
// How a node is computed goes by its segment, never by its cell: a node's result does not depend on the launch
// shape or on what else shares the launch.
#pragma once

#include "stream_collide.cuh"

namespace wk {

// A segment is CELL nodes of a row, from its start (the last one of a row may be shorter). PURE: its every node is a
// pure gather. A model's arithmetic goes by a node's segment, so the result does not depend on the cells either.
enum SegKind : uint8_t { SEG_GENERAL = 0, SEG_PURE = 1, SEG_SOLID = 2 };
// Linear cells: PURE, all in SEG_PURE segments and stepped as a cell; ZH, holds Zou-He nodes.
enum : uint8_t { CELL_PURE = 1u, CELL_ZH = 2u };
// What a listed cell holds, in bits 8 .. of its node count (k_records): of each half, nodes to step,
// momentum-exchange links; Zou-He nodes of a pure one. The host makes the units of the cells from them.
constexpr unsigned LIST_LIVE = 1u << 8, LIST_MEM = 1u << 10, LIST_ZH = 1u << 12;  // LIVE, MEM << half
// How the general cells of a model are split into units (warps): whole cells in pairs, or halves, one node per thread.
enum ListMode { LIST_WHOLE = 1, LIST_HALVES = 2 };
constexpr unsigned UNIT_PURE = 2u;

// Word 0 of a node record: bits 0..26 the pulls that bounce back, and these.
constexpr unsigned CN_LIVE = 1u << 31, CN_ZH_IN = 1u << 30, CN_ZH_OUT = 1u << 29;
// Word 1: the momentum-exchange links (mem_links). Word 2: the pulls that bounce off a moving wall, and from bit
// CN_WALL_SHIFT (D2Q9) those that bounce at the lattice's y faces. Word 3: bits 1..18 the populations that curved
// links replace, from bit CN_LINK_SHIFT the position of the first of these links among the cell's.
constexpr int CN_WALL_SHIFT = 16;
constexpr int CN_LINK_SHIFT = 19;
constexpr unsigned CN_LINKS = (1u << CN_LINK_SHIFT) - 2u;

// Offsets from a node to its pull sources: m for c = +1 (the source at -1), p for c = -1.
// A pure or in-range pull never crosses a non-periodic face, so the wraps apply unconditionally.
struct PullOffsets {
    int xm, xp, ym, yp, zm, zp;
};
template <int Q>
__device__ __forceinline__ PullOffsets pull_offsets(const Geo& g, unsigned i) {
    const int nx = g.nx, ny = g.ny;
    const unsigned row = g.by_nx.quot(i);
    const int x = static_cast<int>(i - row * static_cast<unsigned>(nx));
    PullOffsets o;
    o.xm = x == 0 ? nx - 1 : -1;
    o.xp = x == nx - 1 ? 1 - nx : 1;
    int y = static_cast<int>(row);
    if constexpr (Lat<Q>::D == 3) {
        const unsigned z = g.by_ny.quot(row);
        y = static_cast<int>(row - z * static_cast<unsigned>(ny));
        const int plane = nx * ny;
        o.zm = z == 0 ? (g.nz - 1) * plane : -plane;
        o.zp = z == static_cast<unsigned>(g.nz - 1) ? (1 - g.nz) * plane : plane;
    } else {
        o.zm = o.zp = 0;
    }
    o.ym = y == 0 ? (ny - 1) * nx : -nx;
    o.yp = y == ny - 1 ? (1 - ny) * nx : nx;
    return o;
}
// How a pure cell gathers. INSIDE: a whole cell of which no node pulls across a face, so direction q's source is the
// node's index minus one constant and its address one addition to a per-launch base, which cell_pairs takes for a lane's
// second node too without asking whether it exists (a shorter cell near the lattice's end would read past the
// plane). ROW_ENDS: as INSIDE in y and z, but a row ends in the cell, whose end nodes wrap in x, or the cell is
// shorter. FACES: a y or z face is in reach.
enum CellGather { INSIDE, ROW_ENDS, FACES };
template <int Q>
__host__ __device__ __forceinline__ CellGather cell_gather(const Geo& g, unsigned i0, int count) {
    const unsigned nx = g.nx, last = i0 + count - 1, r0 = g.by_nx.quot(i0), r1 = g.by_nx.quot(last);
    const unsigned z = Lat<Q>::D == 3 ? g.by_ny.quot(r0) : 0u, y0 = r0 - z * g.ny, y1 = y0 + (r1 - r0);
    const bool in_y = y0 > 0u && y1 < static_cast<unsigned>(g.ny) - 1u;
    const bool in_z = Lat<Q>::D == 2 || (z > 0u && z < static_cast<unsigned>(g.nz) - 1u);
    if (!in_y || !in_z) return FACES;
    return count == CELL && r0 == r1 && i0 != r0 * nx && last != r0 * nx + nx - 1u ? INSIDE : ROW_ENDS;
}
template <int Q>
__device__ __forceinline__ int pull_offset(const PullOffsets& o, int q) {
    using L = Lat<Q>;
    int d = 0;
    if (L::cz(q)) d += L::cz(q) > 0 ? o.zm : o.zp;
    if (L::cy(q)) d += L::cy(q) > 0 ? o.ym : o.yp;
    if (L::cx(q)) d += L::cx(q) > 0 ? o.xm : o.xp;
    return d;
}

// The temperature populations pulled by node i (D2Q5 directions 1..4 are D2Q9's): anti-bounce-back at the
// isothermal y walls, bounce-back at solid nodes; r = 0 for a pure node.
__device__ __forceinline__ void cell_t5(const Thermal& th, const float* tin, long long P, unsigned i, const PullOffsets& d, const uint4& r,
                                        float t[5]) {
    t[0] = tin[i];
#pragma unroll
    for (int q = 1; q < 5; ++q) {
        const bool bounce = ((r.x & ~r.z) >> q) & 1u;  // a moving wall passes the temperature on
        const float v = tin[bounce ? D2Q5::opp(q) * P + i : q * P + (i + pull_offset<9>(d, q))];
        const bool wall = (r.z >> (CN_WALL_SHIFT + q)) & 1u;
        const float tw = D2Q5::cy(q) > 0 ? th.t_south : th.t_north;
        t[q] = wall ? __fadd_rn(-v, __fmul_rn(2.0f * D2Q5::w(q), tw)) : v;
    }
}

// Where the populations are. One lattice: base pointers of every plane from the kernel's parameters
// (constant memory, so an address is one multiply-add on the node index), for any lattice size.
template <int Q, class T>
struct OneLattice {
    static constexpr bool UNIFORM = Q != 9;  // one node per thread: addresses from the warp's first node (cell_one)
    const StepArgs& a;
    L2Policy ld;
    __device__ __forceinline__ const T* in(int q, unsigned e) const { return static_cast<const T*>(a.in[q]) + e; }
    __device__ __forceinline__ const T* pull(int q, unsigned e) const { return static_cast<const T*>(a.pull[q]) + e; }
    __device__ __forceinline__ T* out(int q, unsigned e) const { return static_cast<T*>(a.out[q]) + e; }
    __device__ __forceinline__ const float* tin() const { return a.th.tin; }
    __device__ __forceinline__ float* tout() const { return a.th.tout; }
    __device__ __forceinline__ int cur() const { return a.cur; }
};
// A member of a batch, whose arguments are in device memory: 32-bit element offsets from its
// two buffers (the host steps members with Q * pitch >= 2^32 by themselves).
template <int Q, class T>
struct OneMember {
    static constexpr bool UNIFORM = false;
    const T* f;
    T* g;
    const float* t_in;
    float* t_out;
    unsigned P;
    int nx, plane, c;
    L2Policy ld;
    __device__ __forceinline__ const T* in(int q, unsigned e) const { return f + (q * P + e); }
    __device__ __forceinline__ const T* pull(int q, unsigned e) const {
        using L = Lat<Q>;
        return f + (q * P - (L::cx(q) + L::cy(q) * nx + L::cz(q) * plane) + e);
    }
    __device__ __forceinline__ T* out(int q, unsigned e) const { return g + (q * P + e); }
    __device__ __forceinline__ const float* tin() const { return t_in; }
    __device__ __forceinline__ float* tout() const { return t_out; }
    __device__ __forceinline__ int cur() const { return c; }
};

// The curved links of a cell (Bouzidi linear interpolation from post-collision values,
// d3q19_curved.ispc:36-68). They are consecutive in the link array, so the warp evaluates them one per lane,
// 128 with their loads in flight together, and each node picks its values up from shared memory (`sm`, 128 values
// per warp); a node that walked its own links would wait for them one after the other.
// put(node 0 / 1 of this lane, q, value); wa, wb: the records' words 3.
template <int S, class Put>
__device__ __forceinline__ void curved_links(const typename Codec<S>::T* fin, long long P, const Links& B, unsigned first,
                                             unsigned count, unsigned wa, unsigned wb, float* sm, L2Policy ld, Put put) {
    constexpr int R = 4;
    const unsigned lane = threadIdx.x & 31;
    const unsigned pa = wa >> CN_LINK_SHIFT, pb = wb >> CN_LINK_SHIFT;
    for (unsigned k0 = 0; k0 < count; k0 += 32 * R) {  // uniform
        uint4 r[R];
        float x[R], y[R];
#pragma unroll
        for (int j = 0; j < R; ++j)
            if (k0 + 32 * j < count) r[j] = __ldg(B.rec + first + min(k0 + 32 * j + lane, count - 1));
#pragma unroll
        for (int j = 0; j < R; ++j)
            if (k0 + 32 * j < count) {
                const float w = S == STORE_F32 ? 0.0f : rt_w19(static_cast<int>(r[j].z & 0xffu));  // of both planes
                x[j] = load_f<S>(fin + (static_cast<long long>(r[j].z & 0xffu) * P + r[j].x), w, ld);
                y[j] = load_f<S>(fin + (static_cast<long long>((r[j].z >> 8) & 0xffu) * P + r[j].y), w, ld);
            }
#pragma unroll
        for (int j = 0; j < R; ++j)
            if (k0 + 32 * j < count) {
                const float c = __uint_as_float(r[j].w);
                float m = 0.0f;
                if (r[j].z & LINK_MOVES) m = __ldg(B.mom + first + min(k0 + 32 * j + lane, count - 1));
                sm[32 * j + lane] = c * x[j] + (1.0f - c) * y[j] - m;
            }
        __syncwarp();
#pragma unroll
        for (int q = 1; q < 19; ++q) {
            const unsigned below = ((1u << q) - 1u) & CN_LINKS;
            const unsigned ka = pa + __popc(wa & below) - k0, kb = pb + __popc(wb & below) - k0;
            if (((wa >> q) & 1u) && ka < 32u * R) put(0, q, sm[ka]);
            if (((wb >> q) & 1u) && kb < 32u * R) put(1, q, sm[kb]);
        }
        __syncwarp();
    }
}

// One warp: append the force of the last step from its partial sums, if one is outstanding: 256 strided sums
// of the slots and a fixed tree, whatever the launch, so the force is reproducible bit for bit.
__device__ __forceinline__ void mem_sum(const MemCfg& M) {
    const int lane = threadIdx.x & 31;
    const double* part = M.left->part;
    if (!part) return;
    const int slots = M.left->slots;
    const unsigned step = M.left->steps;
#pragma unroll 1
    for (int c = 0; c < 3; ++c) {  // one component at a time: this rare path must not set the kernel's registers
        double s[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) s[k] = 0.0;
        for (int j = lane; j < slots; j += 256) {
#pragma unroll
            for (int k = 0; k < 8; ++k)
                if (j + 32 * k < slots) s[k] += part[3 * static_cast<long long>(j + 32 * k) + c];
        }
#pragma unroll
        for (int o = 4; o > 0; o >>= 1)
#pragma unroll
            for (int k = 0; k < o; ++k) s[k] += s[k + o];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s[0] += __shfl_down_sync(0xffffffffu, s[0], o);
        if (lane == 0) M.hist[3 * static_cast<long long>(step % static_cast<unsigned>(M.hist_cap)) + c] = s[0];
    }
    __syncwarp();
    if (lane == 0) M.left->steps = step + 1u;
}

// The same at the start of a step that reads buffer `cur`, which leaves its own partial sums outstanding.
__device__ __forceinline__ void mem_sum_step(const MemCfg& M, int cur) {
    mem_sum(M);
    __syncwarp();
    if ((threadIdx.x & 31) == 0) {
        M.left->part = M.contrib + cur * M.stride;
        M.left->slots = M.slots;
    }
}

// The momentum exchange of a cell's (half cell's) nodes, in all lanes, to its slot.
__device__ __forceinline__ void mem_leave(const MemCfg& M, double acc[3], int slot, int cur) {
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc[c] += __shfl_down_sync(0xffffffffu, acc[c], o);
    if ((threadIdx.x & 31) == 0) {
        double* p = M.contrib + (cur * M.stride + 3 * static_cast<long long>(slot));
        for (int c = 0; c < 3; ++c) p[c] = acc[c];
    }
}

// Tell the host of a non-finite node. A lattice that has diverged has them everywhere: only the first of an SM go to the
// one word in L2 (a batch of sixteen 48^3 FP16 MRT lattices, all diverged: 82 us a step, 469 with an atomic each).
__device__ __forceinline__ void flag_nonfinite(unsigned* status) {
    if (!(*status & ERR_NONFINITE)) atomicOr(status, ERR_NONFINITE);
}

// This warp's values of curved links (D3Q19).
__device__ __forceinline__ float* link_values() {
    __shared__ float v[WK_FAST_MAX_THREADS / 32][128];
    return v[threadIdx.x >> 5];
}

// One cell, two nodes per thread. FP32: lane and lane + 32; 16-bit storage: the adjacent pair 2 lane, 2 lane + 1,
// which leaves with one 32-bit store per plane where the cell starts on an even node. PURE: a pure cell, zh telling
// whether it holds Zou-He nodes; otherwise the general cell `entry`. The two are compiled apart: the general
// path's live values would cost the pure one registers, hence loads in flight.
// Bound by memory: 152 B a node, of which D3Q19 FP32 256x128x128 moves 5.8 TB/s (110.0 us a step;
// 118.2 with one warp per row segment).
template <int Q, int COLL, int S, bool LES, bool PURE, class At>
__device__ __forceinline__ void cell_pairs(const StepArgs& a, const At& at, uint4 cell, int entry, bool zh) {
    using L = Lat<Q>;
    using T = typename Codec<S>::T;
    constexpr bool HS = S != STORE_F32;
    const unsigned i0 = cell.x;
    const int count = static_cast<int>(cell.y & 0xffu);
    const int lane = threadIdx.x & 31;
    const int oa = HS ? 2 * lane : lane, ob = HS ? 2 * lane + 1 : lane + 32;
    bool va = oa < count, vb = ob < count;
    unsigned ia = i0 + oa, ib = i0 + ob;
    uint4 ra = make_uint4(0u, 0u, 0u, 0u), rb = ra;
    bool mem = false;  // uniform: the cell holds momentum-exchange nodes
    if constexpr (!PURE) {
        ra = __ldg(a.records + (static_cast<long long>(entry) * CELL + oa));
        rb = __ldg(a.records + (static_cast<long long>(entry) * CELL + ob));
        va = (ra.x & CN_LIVE) != 0u;
        vb = (rb.x & CN_LIVE) != 0u;
        if (a.mem.enabled) mem = __any_sync(0xffffffffu, (ra.y | rb.y) != 0u);
    }
    if (PURE && !va && !vb) return;  // the lanes of a general cell stay together for its links and its sum
    const unsigned mem_a = ra.y, mem_b = rb.y;  // 0 for a node that is not stepped
    // a node that is not stepped (solid, past the end) is computed as a copy of its partner
    // (a lane without any reads the cell's first node)
    if (!va && !vb) ia = ib = i0, ra = rb = make_uint4(0u, 0u, 0u, 0u);
    else if (!va) ia = ib, ra = rb;
    else if (!vb) ib = ia, rb = ra;
    const long long P = a.geo.pitch;
    const CellGather way = PURE ? cell_gather<Q>(a.geo, i0, count) : FACES;  // uniform
    const bool words = HS && (a.geo.nx & 1) == 0;  // 16-bit pairs lie in one row, every source row on a word boundary
    float2 f[Q];
    PullOffsets da, db;
    if (PURE && way == INSIDE) {
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            const T* p = at.pull(q, ia);
            if (HS && L::cx(q) == 0 && words) {
                const unsigned w = ld_pop(reinterpret_cast<const unsigned*>(p), at.ld);
                f[q] = make_float2(raw_lo<S>(w), raw_hi<S>(w));
            } else {
                f[q] = make_float2(load_raw<S>(p, at.ld), load_raw<S>(p + (HS ? 1 : 32), at.ld));
            }
        }
    } else if (PURE && way == ROW_ENDS) {
        const unsigned nx = a.geo.nx;
        const unsigned xa = ia - a.geo.by_nx.quot(ia) * nx, xb = ib - a.geo.by_nx.quot(ib) * nx;
        const unsigned am = xa == 0u ? ia + nx : ia, ap = xa == nx - 1u ? ia - nx : ia;  // c_x = +1 / -1
        const unsigned bm = xb == 0u ? ib + nx : ib, bp = xb == nx - 1u ? ib - nx : ib;
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            if (HS && L::cx(q) == 0 && words) {
                const unsigned w = ld_pop(reinterpret_cast<const unsigned*>(at.pull(q, ia)), at.ld);
                f[q] = make_float2(raw_lo<S>(w), raw_hi<S>(w));
            } else {
                f[q] = make_float2(load_raw<S>(at.pull(q, L::cx(q) > 0 ? am : (L::cx(q) < 0 ? ap : ia)), at.ld),
                                   load_raw<S>(at.pull(q, L::cx(q) > 0 ? bm : (L::cx(q) < 0 ? bp : ib)), at.ld));
            }
        }
    } else if (PURE) {
        da = pull_offsets<Q>(a.geo, ia);
        db = pull_offsets<Q>(a.geo, ib);
#pragma unroll
        for (int q = 0; q < Q; ++q)
            f[q] = make_float2(load_raw<S>(at.in(q, ia + pull_offset<Q>(da, q)), at.ld),
                               load_raw<S>(at.in(q, ib + pull_offset<Q>(db, q)), at.ld));
    } else {
        da = pull_offsets<Q>(a.geo, ia);
        db = pull_offsets<Q>(a.geo, ib);
        f[0] = make_float2(load_raw<S>(at.in(0, ia), at.ld), load_raw<S>(at.in(0, ib), at.ld));
#pragma unroll
        for (int q = 1; q < Q; ++q) {
            const T* pa = at.in(q, ia + pull_offset<Q>(da, q));
            const T* pb = at.in(q, ib + pull_offset<Q>(db, q));
            if ((ra.x >> q) & 1u) pa = at.in(L::opp(q), ia);
            if ((rb.x >> q) & 1u) pb = at.in(L::opp(q), ib);
            f[q] = make_float2(load_raw<S>(pa, at.ld), load_raw<S>(pb, at.ld));
        }
        if (ra.z | rb.z) {  // pulls that bounced off a moving wall
#pragma unroll
            for (int q = 1; q < Q; ++q) {
                if ((ra.z >> q) & 1u) f[q].x += a.geo.mom[q];
                if ((rb.z >> q) & 1u) f[q].y += a.geo.mom[q];
            }
        }
        if constexpr (Q == 19) {
            if (cell.w)
                curved_links<S>(at.in(0, 0u), P, a.links, cell.z, cell.w, ra.w, rb.w, link_values(), at.ld,
                                [&](int h, int q, float v) {
                                    if (h == 0) f[q].x = v;
                                    else f[q].y = v;
                                });
        }
    }
    if (zh || !PURE) {
        unsigned za, zb;  // FL_ZH_IN / FL_ZH_OUT of the two nodes
        if (!PURE) {
            za = (ra.x & CN_ZH_IN ? FL_ZH_IN : 0u) | (ra.x & CN_ZH_OUT ? FL_ZH_OUT : 0u);
            zb = (rb.x & CN_ZH_IN ? FL_ZH_IN : 0u) | (rb.x & CN_ZH_OUT ? FL_ZH_OUT : 0u);
        } else {
            za = a.flags[ia] & (FL_ZH_IN | FL_ZH_OUT);
            zb = a.flags[ib] & (FL_ZH_IN | FL_ZH_OUT);
        }
        if (za) zou_he_half<Q, HS>(f, 0, static_cast<uint8_t>(za), a.geo);
        if (zb) zou_he_half<Q, HS>(f, 1, static_cast<uint8_t>(zb), a.geo);
    }
    if (mem) {
        double acc[3] = {0.0, 0.0, 0.0};
        if (mem_a | mem_b) {
#pragma unroll
            for (int q = 1; q < Q; ++q) {
                if ((mem_a >> q) & 1u) mem_add<Q>(q, f[q].x, 0, 0, a.mem, acc);
                if ((mem_b >> q) & 1u) mem_add<Q>(q, f[q].y, 0, 0, a.mem, acc);
            }
        }
        mem_leave(a.mem, acc, __ldg(a.mem.slot + 2 * entry), at.cur());
    }
    float2 rho, u[3];
    collide_pairs2<Q, COLL, S, LES>(f, a.phys, bc2(a.phys.g[1]),
                                    a.phys.g[0] != 0.0f || a.phys.g[1] != 0.0f || a.phys.g[2] != 0.0f, rho, u);
    if ((va && (!(rho.x > 0.0f) || !(fabsf(u[0].x) < 1e30f))) || (vb && (!(rho.y > 0.0f) || !(fabsf(u[0].y) < 1e30f))))
        flag_nonfinite(a.status);
    if (va && vb) {
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            T* p = at.out(q, ia);
            if (HS && (i0 & 1u) == 0u) {  // (uniform)
                store_pair<S>(p, f[q]);
            } else {
                store_raw<S>(p, f[q].x);
                store_raw<S>(p + (HS ? 1 : 32), f[q].y);
            }
        }
    } else if (va || vb) {
#pragma unroll
        for (int q = 0; q < Q; ++q) store_raw<S>(at.out(q, ia), va ? f[q].x : f[q].y);  // ia = ib where one is not stepped
    }
}

// Half a cell (32 nodes), one node per thread; known: how a pure one gathers (cell_gather), below 0 if to be found.
template <int Q, int COLL, int S, bool LES, bool TH, bool PURE, class At>
__device__ __forceinline__ void cell_one(const StepArgs& a, const At& at, uint4 cell, int entry, bool zh, int half,
                                         int known = -1) {
    using L = Lat<Q>;
    using C = Codec<S>;
    using T = typename C::T;
    const unsigned i0 = cell.x;
    const int count = static_cast<int>(cell.y & 0xffu);
    const int lane = threadIdx.x & 31, o = 32 * half + lane;
    unsigned i = i0 + o;
    // UNIFORM: a plane's address is a uniform one, of the half cell's first node, and the lane's 32-bit offset, which
    // takes no instruction per plane (D3Q27 F16 MRT 256^3 box: 621 -> 595 us a step). Elsewhere it was up to 5 % slower
    // (D2Q9) or 12 % (a batch of two 160^3 F16 boxes, whose bases are not parameters: 216 -> 241).
    const unsigned at0 = At::UNIFORM ? i0 + 32 * half : i, off = At::UNIFORM ? lane : 0;
    bool v = o < count;
    uint4 r = make_uint4(0u, 0u, 0u, 0u);
    bool mem = false;  // uniform: the half cell holds momentum-exchange nodes
    if constexpr (!PURE) {
        r = __ldg(a.records + (static_cast<long long>(entry) * CELL + o));
        v = (r.x & CN_LIVE) != 0u;
        if (a.mem.enabled) mem = __any_sync(0xffffffffu, r.y != 0u);
    }
    if (!v) {
        if (PURE) return;
        i = i0;  // stays for the links and the sum; reads the cell's first node and stores nothing
        r = make_uint4(0u, 0u, 0u, 0u);
    }
    const long long P = a.geo.pitch;
    PullOffsets d;
    float f[Q];
    const int way = !PURE ? FACES : (known >= 0 ? known : cell_gather<Q>(a.geo, i0, count));  // uniform
    if (PURE && way == INSIDE) {
#pragma unroll
        for (int q = 0; q < Q; ++q) f[q] = load_f<S>(at.pull(q, at0) + off, L::w(q), at.ld);
    } else if (PURE && way == ROW_ENDS) {
        const unsigned nx = a.geo.nx, x = i - a.geo.by_nx.quot(i) * nx;
        if constexpr (At::UNIFORM) {
            const unsigned om = x == 0u ? off + nx : off, op = x == nx - 1u ? off : off + nx;  // c_x = +1, and -1 from at0 - nx
#pragma unroll
            for (int q = 0; q < Q; ++q)
                f[q] = load_f<S>(at.pull(q, L::cx(q) < 0 ? at0 - nx : at0) + (L::cx(q) > 0 ? om : (L::cx(q) < 0 ? op : off)),
                                 L::w(q), at.ld);
        } else {
            const unsigned im = x == 0u ? i + nx : i, ip = x == nx - 1u ? i - nx : i;  // c_x = +1 / -1
#pragma unroll
            for (int q = 0; q < Q; ++q)
                f[q] = load_f<S>(at.pull(q, L::cx(q) > 0 ? im : (L::cx(q) < 0 ? ip : i)), L::w(q), at.ld);
        }
    } else if (PURE) {
        d = pull_offsets<Q>(a.geo, i);
#pragma unroll
        for (int q = 0; q < Q; ++q) f[q] = load_f<S>(at.in(q, i + pull_offset<Q>(d, q)), L::w(q), at.ld);
    } else {
        d = pull_offsets<Q>(a.geo, i);
        f[0] = load_f<S>(at.in(0, i), L::w(0), at.ld);
#pragma unroll
        for (int q = 1; q < Q; ++q) {
            const T* p = at.in(q, i + pull_offset<Q>(d, q));
            if ((r.x >> q) & 1u) p = at.in(L::opp(q), i);
            f[q] = load_f<S>(p, L::w(q), at.ld);
        }
        if (Q == 9 ? r.z & 0xffffu : r.z) {
#pragma unroll
            for (int q = 1; q < Q; ++q)
                if ((r.z >> q) & 1u) f[q] += a.geo.mom[q];
        }
        if constexpr (Q == 19) {
            if (cell.w)
                curved_links<S>(at.in(0, 0u), P, a.links, cell.z, cell.w, r.w, 0u, link_values(), at.ld,
                                [&](int, int q, float x) { f[q] = x; });
        }
    }
    if (zh || !PURE) {
        const unsigned z = !PURE ? (r.x & CN_ZH_IN ? FL_ZH_IN : 0u) | (r.x & CN_ZH_OUT ? FL_ZH_OUT : 0u) : a.flags[i];
        if (z & FL_ZH_IN) zou_he_inlet<Q>(f, a.geo.uin);
        if (z & FL_ZH_OUT) zou_he_outlet<Q>(f, a.geo.rho_out);
    }
    Physics ph = a.phys;  // a coupled temperature adds the node's buoyancy to the body force
    float t5[5], Tn = 0.f;
    if constexpr (TH) {
        if (a.th.on) {
            if (PURE && way != FACES) d = pull_offsets<Q>(a.geo, i);
            cell_t5(a.th, at.tin(), P, i, d, r, t5);
            Tn = sum_t5(t5);
            ph.g[1] = buoyant_gy(a.th, a.phys.g[1], Tn);
        }
    }
    float rho, u[3];
    node_moments<Q>(f, ph.g, rho, u);
    if (mem) {
        double acc[3] = {0.0, 0.0, 0.0};
        if (r.y) {
            const unsigned y = a.geo.by_nx.quot(i);  // (2D: the torque's arm)
#pragma unroll
            for (int q = 1; q < Q; ++q)
                if ((r.y >> q) & 1u)
                    mem_add<Q>(q, f[q], static_cast<int>(i - y * a.geo.nx), static_cast<int>(y), a.mem, acc);
        }
        mem_leave(a.mem, acc, __ldg(a.mem.slot + 2 * entry + half), at.cur());
    }
    if (!v) return;
    if (!(rho > 0.0f) || !(fabsf(u[0]) < 1e30f)) flag_nonfinite(a.status);
    collide<Q, COLL, LES>(f, rho, u, ph);
#pragma unroll
    for (int q = 0; q < Q; ++q) store_f<S>(at.out(q, at0) + off, f[q], L::w(q));
    if constexpr (TH) {
        if (a.th.on) {
            collide_t5(t5, Tn, u, a.th.omega_t);
#pragma unroll
            for (int q = 0; q < 5; ++q) __stcs(at.tout() + q * P + i, t5[q]);
        }
    }
}

// Units (warps) of a pure cell, and the mode of the listed ones.
template <int Q, int COLL, int S, bool TH>
__host__ __device__ constexpr unsigned pure_units() {
    return pure_pairs<Q, COLL, S>() && !TH ? 1u : CELL / 32u;
}
template <int Q, int COLL, int S, bool TH>
__host__ __device__ constexpr ListMode list_mode() {
    return all_pairs<Q, COLL, S>() && !TH ? LIST_WHOLE : LIST_HALVES;
}

// Unit `word` = entry * 4 + (UNIT_PURE for a pure cell) + (half) of a listed cell.
template <int Q, int COLL, int S, bool LES, bool TH, class At>
__device__ __forceinline__ void listed_unit(const StepArgs& a, const At& at, unsigned word) {
    const int entry = static_cast<int>(word >> 2), half = static_cast<int>(word & 1u);
    const uint4 cell = __ldg(a.list + entry);
    if (word & UNIT_PURE) {
        const bool zh = (cell.y & LIST_ZH) != 0u;
        if constexpr (pure_units<Q, COLL, S, TH>() == 1u) cell_pairs<Q, COLL, S, LES, true>(a, at, cell, -1, zh);
        else cell_one<Q, COLL, S, LES, TH, true>(a, at, cell, -1, zh, half);
    } else if constexpr (list_mode<Q, COLL, S, TH>() == LIST_WHOLE) {
        cell_pairs<Q, COLL, S, LES, false>(a, at, cell, entry, false);
    } else {
        cell_one<Q, COLL, S, LES, TH, false>(a, at, cell, entry, false, half);
    }
}

// Register budgets (blocks of up to 64 threads): common.cuh.
template <int Q, int COLL, int S, bool LES, bool TH, bool BATCH>
constexpr int cell_min_blocks() {
    if (Q == 27 && COLL == COLL_MRT && S == STORE_F32 && (LES || BATCH)) return WK_PAIRS27_MIN_BLOCKS;
    if (!pure_pairs<Q, COLL, S>() || (TH && !BATCH)) return Q == 9 ? (TH ? 16 : 18) : (Q == 19 ? 12 : 8);
    if (Q != 9) return WK_PAIRS_MIN_BLOCKS;
    return BATCH ? WK_PAIRS9_BATCH_MIN_BLOCKS : WK_PAIRS9_MIN_BLOCKS;
}

// The work units of warp `warp` of the pure blocks (block index b of them): `run` units (cells, or half cells), those
// of a block's warps adjacent. load(u), the unit's class or entry, goes out while the unit before it is stepped.
template <class Load, class Step>
__device__ __forceinline__ void walk(unsigned b, unsigned warp, unsigned units, unsigned run, Load load, Step step) {
    const unsigned wpb = blockDim.x >> 5;
    unsigned u = b * (wpb * run) + warp;
    if (u >= units) return;
    auto d = load(u);
#pragma unroll 1
    for (unsigned k = 0; k < run && u < units; ++k) {
        const unsigned next = u + wpb;
        const auto dn = load(min(next, units - 1u));
        step(u, d);
        u = next;
        d = dn;
    }
}

// Block index among the listed (first = true) or the pure blocks of a launch. Every 2^spread-th block is a listed
// one until all are placed (list_blocks << spread is about 60 % of the blocks): the listed cells' latency chain
// then never holds more than a few of the device's block slots at once, and none of it is left at the end.
// All of them at the front held half the slots for 20 us on a 160^3 sphere channel. Every other step takes the
// pure cells from the end (`reverse`): what the last step wrote last is still in L2 (256x128x128: 112.1 -> 110.0 us, 160^3
// 113.5 -> 111.8; lattices that are read evict-first are within 2 % either way).
__device__ __forceinline__ unsigned which_block(unsigned list_blocks, unsigned spread, bool reverse, bool& first) {
    const unsigned b = blockIdx.x, k = b >> spread;
    first = k < list_blocks && (b & ((1u << spread) - 1u)) == 0u;
    const unsigned pb = b - min(list_blocks, k + 1u);
    return first ? k : (reverse ? gridDim.x - list_blocks - 1u - pb : pb);
}

// A step's launch may start before the step before it has ended (launch_step), as that one's blocks end: wait for its
// results. The blocks come up and take over where they had the latency of a launch between steps: D2Q9
// 400x160 in a graph 3.5 -> 3.2 us a step, as plain launches 6.1 -> 3.4 (the host's rate of launches), 1024x512 MRT 7.9 -> 7.6
// and 10.2 -> 7.8; D3Q19 48^3 sphere 5.95 -> 5.6, 256x128x128 110.4 -> 110.0. Letting the next launch start as
// soon as every block of this one runs was slower (1024x512 BGK 9.4, 8.6 without, in graphs).
__device__ __forceinline__ void after_last_step() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// One step of one lattice: the listed cells and the pure cells of cells 0 .. cells - 1.
template <int Q, int COLL, int S, bool LES, bool TH>
__global__ void __launch_bounds__(WK_FAST_MAX_THREADS, (cell_min_blocks<Q, COLL, S, LES, TH, false>())) k_step_cells(const StepArgs a) {
    after_last_step();
    const OneLattice<Q, typename Codec<S>::T> at{a, read_policy(a.evict_first)};
    constexpr unsigned W = pure_units<Q, COLL, S, TH>();
    bool listed;
    const unsigned block = which_block(a.list_blocks, a.spread, a.reverse, listed);
    if (listed) {
        unsigned k = block * (blockDim.x >> 5) + (threadIdx.x >> 5);
        if (a.mem.enabled && k-- == 0)  // the first warp
            mem_sum_step(a.mem, a.cur);
        else if (k < a.nunits)
            listed_unit<Q, COLL, S, LES, TH>(a, at, __ldg(a.units + k));
        return;
    }
    // 3D, one node per thread: a warp with several half cells takes both halves of a cell in turn and classifies it once
    // (256^3 boxes, F16 MRT: D3Q19 454 -> 420 us a step, D3Q27 667 -> 621; D2Q9 2048x1024 MRT 26.9 -> 27.9, so not there)
    constexpr bool TURN = W == 2u && Q != 9;
    const unsigned per = TURN ? min(a.run, W) : 1u;
    unsigned warp = threadIdx.x >> 5;
    if constexpr (TURN) warp = __shfl_sync(0xffffffffu, warp, 0);  // known to the compiler as the warp's
    walk(
        block, warp, a.cells * W / per, a.run / per, [&](unsigned u) { return static_cast<unsigned>(__ldg(a.cell_kind + u * per / W)); },
        [&](unsigned u, unsigned kind) {
            if (!(kind & CELL_PURE)) return;
            const unsigned i0 = u * per / W * CELL;
            const uint4 cell = make_uint4(i0, min(CELL + 0u, a.nodes - i0), 0u, 0u);
            if constexpr (W == 1u) {
                cell_pairs<Q, COLL, S, LES, true>(a, at, cell, -1, (kind & CELL_ZH) != 0);
            } else if constexpr (!TURN) {
                cell_one<Q, COLL, S, LES, TH, true>(a, at, cell, -1, (kind & CELL_ZH) != 0, u % W);
            } else {
                const int way = cell_gather<Q>(a.geo, i0, cell.y);
                const unsigned h0 = u * per % W;
#pragma unroll 1
                for (unsigned h = h0; h < h0 + per; ++h)
                    cell_one<Q, COLL, S, LES, TH, true>(a, at, cell, -1, (kind & CELL_ZH) != 0, static_cast<int>(h), way);
            }
        });
}

// ------------------------------------------------------------------ many lattices
// A batch advances many independent lattices (same Q, collision model and storage; any sizes,
// parameters and geometry) with one launch. Each member's step arguments live in device memory; its
// buffers swap with the batch's step parity, so the table stays valid while the members step together.
struct BatchDom {
    StepArgs a;        // fin / fout (th.tin / th.tout) unused: taken from buf[] (tbuf[]) by parity
    void* buf[2];      // the member's two state buffers
    float* tbuf[2];    // its two temperature buffers (thermal members)
    int cur0;          // index of the buffer holding the state at batch parity 0
    int alone;         // 1: stepped by its own launches (Q * pitch >= 2^32)
};

constexpr unsigned LISTED_SUM = 0xffffffffu;

struct BatchArgs {
    const BatchDom* dom;
    const uint2* listed;  // (member, unit of its list, or LISTED_SUM)
    const uint2* pure;    // (member | (nodes - 1) << 24 | zh << 30, first node) of every pure cell
    unsigned nlisted, npure, list_blocks, spread, run;
    int parity;           // batch step parity of this launch
    int evict_first;      // policy of the population loads
};

template <int Q, int S>
__device__ __forceinline__ OneMember<Q, typename Codec<S>::T> batch_at(const BatchDom& d, int parity, L2Policy ld) {
    using T = typename Codec<S>::T;
    const int c = d.cur0 ^ parity;
    return {static_cast<const T*>(d.buf[c]), static_cast<T*>(d.buf[c ^ 1]), d.tbuf[c], d.tbuf[c ^ 1],
            static_cast<unsigned>(d.a.geo.pitch), d.a.geo.nx, d.a.geo.nx * d.a.geo.ny, c, ld};
}

template <int Q, int COLL, int S, bool LES, bool TH>
__global__ void __launch_bounds__(WK_FAST_MAX_THREADS, (cell_min_blocks<Q, COLL, S, LES, TH, true>()))
    k_step_cells_batch(const BatchArgs b) {
    after_last_step();
    constexpr unsigned W = pure_units<Q, COLL, S, false>();
    const L2Policy ld = read_policy(b.evict_first);
    bool listed;
    const unsigned block = which_block(b.list_blocks, b.spread, b.parity, listed);
    if (listed) {
        const unsigned k = block * (blockDim.x >> 5) + (threadIdx.x >> 5);
        if (k >= b.nlisted) return;
        const uint2 r = __ldg(b.listed + k);
        const BatchDom& d = b.dom[r.x];
        const StepArgs& a = d.a;
        if (r.y == LISTED_SUM) {  // the member's force of the last step
            mem_sum_step(a.mem, d.cur0 ^ b.parity);
        } else {
            const auto at = batch_at<Q, S>(d, b.parity, ld);
            if (TH && a.th.on) listed_unit<Q, COLL, S, LES, TH>(a, at, r.y);
            else listed_unit<Q, COLL, S, LES, false>(a, at, r.y);
        }
        return;
    }
    unsigned warp = threadIdx.x >> 5;
    // known to the compiler as the warp's: its table entry is then addressed once for the warp (512 channels FP16 388 -> 375 us)
    if constexpr (W == 1u) warp = __shfl_sync(0xffffffffu, warp, 0);
    walk(
        block, warp, b.npure * W, b.run, [&](unsigned u) { return __ldg(b.pure + u / W); },
        [&](unsigned u, uint2 r) {
            const BatchDom& d = b.dom[r.x & 0xffffffu];
            const StepArgs& a = d.a;
            const auto at = batch_at<Q, S>(d, b.parity, ld);
            const uint4 cell = make_uint4(r.y, ((r.x >> 24) & 63u) + 1u, 0u, 0u);
            const bool zh = ((r.x >> 30) & 1u) != 0u;
            if constexpr (TH) {
                if (a.th.on) {
#pragma unroll 1
                    for (int h = u % W; h < 2; h += W) cell_one<Q, COLL, S, LES, true, true>(a, at, cell, -1, zh, h);
                    return;
                }
            }
            if constexpr (W == 1u) cell_pairs<Q, COLL, S, LES, true>(a, at, cell, -1, zh);
            else cell_one<Q, COLL, S, LES, false, true>(a, at, cell, -1, zh, u % W);
        });
}

}  // namespace wk
