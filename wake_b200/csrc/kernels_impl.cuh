// Kernel instantiations and launch tables for one lattice. Included by
// kernels_q{9,19,27}.cu with WK_Q defined, so the three lattices compile in
// parallel translation units.
#pragma once

#include "kernels.cuh"

#ifndef WK_Q
#error "define WK_Q before including kernels_impl.cuh"
#endif

#define WK_CAT2(a, b) a##b
#define WK_CAT(a, b) WK_CAT2(a, b)

namespace wk {

// Per-node flag byte from the cell types (see FL_* in lattice.cuh).
template <int Q>
__global__ void k_flags(const uint8_t* __restrict__ types, uint8_t* __restrict__ flags, const Geo geo,
                        const FlagCfg cfg, int xchunks) {
    using L = Lat<Q>;
    const int row = blockIdx.x / xchunks;
    const int x = (blockIdx.x - row * xchunks) * blockDim.x + threadIdx.x;
    if (x >= geo.nx) return;
    const int nx = geo.nx, ny = geo.ny, nz = geo.nz;
    const int y = row % ny, z = row / ny;
    const long long i = static_cast<long long>(row) * nx + x;
    const uint8_t t = types[i] & FL_TYPE;
    uint8_t fl = t;
    if (t != CT_SOLID) {
        bool zh = false;
        if (cfg.zh_rule == 1) {
            const bool interior_row = (y >= 1) && (y <= ny - 2);
            if (cfg.inflow && x == 0 && interior_row) { fl |= FL_ZH_IN; zh = true; }
            if (cfg.outflow && x == nx - 1 && interior_row) { fl |= FL_ZH_OUT; zh = true; }
        } else if (cfg.zh_rule == 2) {
            if (cfg.inflow && x == 0 && t == CT_INFLOW) { fl |= FL_ZH_IN; zh = true; }
            if (cfg.outflow && x == nx - 1 && t == CT_OUTFLOW) { fl |= FL_ZH_OUT; zh = true; }
        }
        bool fast = true;  // Zou-He nodes gather purely too; the formula is applied after the gather
        (void)zh;
        bool mem = false;
#pragma unroll
        for (int q = 1; q < Q; ++q) {
            // pull source x - c_q
            const int sx = L::cx(q) ? wrap<Q>(x - L::cx(q), nx) : x;
            int sy = y - L::cy(q), sz = z - L::cz(q);
            if (L::cy(q) && geo.periodic_y) sy = wrap<Q>(sy, ny);
            if (L::cz(q) && geo.periodic_z) sz = wrap<Q>(sz, nz);
            if (sy < 0 || sy >= ny || sz < 0 || sz >= nz) {
                fast = false;
            } else {
                const uint8_t ts = types[(static_cast<long long>(sz) * ny + sy) * nx + sx] & FL_TYPE;
                if (ts == CT_SOLID || ts == CT_MOVING_WALL) fast = false;
            }
            // momentum-exchange link to x + c_q (forces_momentum_exchange.ispc:38-52)
            if (cfg.mem_enabled && t == CT_FLUID) {
                const int xn = L::cx(q) ? wrap<Q>(x + L::cx(q), nx) : x;
                const int yn = y + L::cy(q), zn = z + L::cz(q);
                if (yn >= 0 && yn < ny && zn >= 0 && zn < nz) {
                    const uint8_t tn = types[(static_cast<long long>(zn) * ny + yn) * nx + xn] & FL_TYPE;
                    if (tn == CT_SOLID || tn == CT_MOVING_WALL) {
                        const float rx = __fsub_rn(__fadd_rn(float(x), 0.5f * float(L::cx(q))), cfg.center[0]);
                        const float ry = __fsub_rn(__fadd_rn(float(y), 0.5f * float(L::cy(q))), cfg.center[1]);
                        const float rz = __fsub_rn(__fadd_rn(float(z), 0.5f * float(L::cz(q))), cfg.center[2]);
                        float r2 = __fadd_rn(__fmul_rn(rx, rx), __fmul_rn(ry, ry));
                        if (L::D == 3) r2 = __fadd_rn(r2, __fmul_rn(rz, rz));
                        if (cfg.r_max <= 0.0f || r2 <= cfg.r_max_sq) mem = true;
                    }
                }
            }
        }
        if (fast) fl |= FL_FAST;
        if (mem) fl |= FL_MEM;
    }
    flags[i] = fl;
}

// Node records of the listed general cells (cells.cuh), one block of CELL threads per cell, and every listed cell's
// LIST_* bits: the first `general` are general, the others pure.
template <int Q>
__global__ void __launch_bounds__(CELL)
    k_records(const uint8_t* __restrict__ flags, uint4* __restrict__ list, unsigned general,
              uint4* __restrict__ records, const Links links, const Geo geo, const FlagCfg cfg) {
    using L = Lat<Q>;
    const uint4 c = list[blockIdx.x];
    if (blockIdx.x >= general) {
        const bool zh = threadIdx.x < c.y && (flags[c.x + threadIdx.x] & (FL_ZH_IN | FL_ZH_OUT));
        if (__syncthreads_or(zh) && threadIdx.x == 0) list[blockIdx.x].y = c.y | LIST_ZH;
        return;
    }
    uint4 r = make_uint4(0u, 0u, 0u, 0u);
    if (threadIdx.x < c.y) {
        const unsigned i = c.x + threadIdx.x;
        const uint8_t fl = flags[i];
        if ((fl & FL_TYPE) != CT_SOLID) {
            r.x = CN_LIVE | (fl & FL_ZH_IN ? CN_ZH_IN : 0u) | (fl & FL_ZH_OUT ? CN_ZH_OUT : 0u);
            unsigned hit = 0;
            if (fl & FL_BFL) {
                const int first = links.node_start[i];
                r.w = (static_cast<unsigned>(first) - c.z) << CN_LINK_SHIFT;
                for (int k = first; k < links.count && links.rec[k].x == i; ++k) r.w |= 1u << ((links.rec[k].z >> 16) & 0xffu);
            }
            const int row = static_cast<int>(i / geo.nx), x = static_cast<int>(i % geo.nx);
            const int y = row % geo.ny, z = row / geo.ny;
#pragma unroll
            for (int q = 1; q < Q; ++q) {
                const int sx = L::cx(q) ? wrap<Q>(x - L::cx(q), geo.nx) : x;
                int sy = y - L::cy(q), sz = z - L::cz(q);
                if (L::cy(q) && geo.periodic_y) sy = wrap<Q>(sy, geo.ny);
                if (L::cz(q) && geo.periodic_z) sz = wrap<Q>(sz, geo.nz);
                if (sy < 0 || sy >= geo.ny || sz < 0 || sz >= geo.nz) {
                    r.x |= 1u << q;  // half-way wall at the lattice's face
                    if (Q == 9) r.z |= 1u << (CN_WALL_SHIFT + q);
                    continue;
                }
                const uint8_t t = flags[(static_cast<long long>(sz) * geo.ny + sy) * geo.nx + sx] & FL_TYPE;
                if (t == CT_SOLID || t == CT_MOVING_WALL) {
                    r.x |= 1u << q;
                    hit |= 1u << q;
                    if (t == CT_MOVING_WALL) r.z |= 1u << q;
                }
            }
            if (fl & FL_MEM) r.y = mem_links<Q>(hit, x, y, z, geo, cfg.center, cfg.r_max, cfg.r_max_sq);
        }
    }
    records[static_cast<long long>(blockIdx.x) * CELL + threadIdx.x] = r;
    const bool live = (r.x & CN_LIVE) != 0u;
    const unsigned half = threadIdx.x >> 5;
    unsigned bits = 0;
    for (unsigned h = 0; h < 2; ++h) {
        if (__syncthreads_or(half == h && live)) bits |= LIST_LIVE << h;
        if (__syncthreads_or(half == h && r.y != 0u)) bits |= LIST_MEM << h;
    }
    if (threadIdx.x == 0) list[blockIdx.x].y = c.y | bits;
}

// Pull-free read of f^0 (state buffer holding pre-collision populations).
template <int Q, int S>
__global__ void __launch_bounds__(512) k_direct(const void* fin_v, const uint8_t* flags, Geo geo, Physics phys,
                                                Out out, int xchunks, Thermal th) {
    using L = Lat<Q>;
    using C = Codec<S>;
    const typename C::T* fin = static_cast<const typename C::T*>(fin_v);
    const int row = blockIdx.x / xchunks;
    const int x = (blockIdx.x - row * xchunks) * blockDim.x + threadIdx.x;
    if (x >= geo.nx) return;
    const long long i = static_cast<long long>(row) * geo.nx + x;
    float f[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) f[q] = C::load_plain(fin + q * geo.pitch + i, L::w(q));
    if (out.f) {
#pragma unroll
        for (int q = 0; q < Q; ++q) out.f[q * geo.pitch + i] = f[q];
    }
    if (out.macro) {
        float g[3] = {phys.g[0], phys.g[1], phys.g[2]};
        if (th.on) {  // local buoyancy of the state's temperature (sum of the current temperature buffer)
            float t5[5];
#pragma unroll
            for (int q = 0; q < 5; ++q) t5[q] = th.tin[q * geo.pitch + i];
            g[1] = buoyant_gy(th, phys.g[1], sum_t5(t5));
        }
        float rho, u[3];
        node_moments<Q>(f, g, rho, u);
        store_macro(out, i, rho, u);
    }
    (void)flags;
}

namespace {
constexpr int kQ = WK_Q;

unsigned blocks_of(unsigned units, int tpb) {
    const unsigned wpb = static_cast<unsigned>(tpb) / 32u;
    return (units + wpb - 1u) / wpb;
}

// Blocks of a launch over `units` pure units, and how they are laid out. Two units per warp where the blocks
// still fill the device (148 SMs, 10 or more blocks each) several times over: a block's start costs about a tenth
// of a one-unit block's life (D3Q19 FP32 160^3: 119 us with one, 112 with two, 115 with eight; D2Q9 1024x512 MRT,
// 8192 blocks of one unit: 8.2 / 7.8 / 9.3); smaller lattices need the blocks to even out the end (97^3: 25.9 / 26.1 /
// 31.0; 48^3: 5.6 / 7.2 / 16). `four`: four units from 59,200 blocks, on D3Q19 and FP16C lattices (256^3 box, two / four:
// D3Q19 FP32 TRT 414 / 399, F16 MRT 417 / 412, D3Q27 FP16C MRT 733 / 721; D3Q27 F16 BGK 588 / 599 and FP32 BGK
// 568 / 570, so not there), and in batches but D3Q27 ones (512 channels FP32 / FP16 431 / 375 and 404 / 348).
unsigned plan(unsigned units, int tpb, unsigned list_blocks, bool four, unsigned& run, unsigned& spread) {
    unsigned blocks = blocks_of(units, tpb);
    run = blocks >= 148u * 400u && four ? 4u : (blocks >= 148u * 40u ? 2u : 1u);
    blocks = list_blocks + (blocks + run - 1u) / run;
    spread = 0;
    while (list_blocks && (static_cast<unsigned long long>(list_blocks) << (spread + 1)) <= blocks / 5ull * 3ull) ++spread;
    return blocks;
}

// Launch a step kernel; early: it may start before the kernel before it on the stream has ended (after_last_step).
template <class A>
void launch_step(void (*kernel)(A), unsigned blocks, int tpb, cudaStream_t st, const A& a, bool early) {
    cudaLaunchConfig_t c{};
    c.gridDim = dim3(blocks);
    c.blockDim = dim3(static_cast<unsigned>(tpb));
    c.stream = st;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    c.attrs = &at;
    c.numAttrs = early ? 1 : 0;
    (void)cudaLaunchKernelEx(&c, kernel, a);  // the caller reads the error
}

template <int C, int S, bool LES, bool TH>
void cells_one(StepArgs& a, int tpb, cudaStream_t st) {
    a.list_blocks = blocks_of(a.nunits + (a.mem.enabled ? 1u : 0u), tpb);
    const unsigned blocks = plan(a.cells * pure_units<kQ, C, S, TH>(), tpb, a.list_blocks, kQ == 19 || S == STORE_F16C, a.run, a.spread);
    if (blocks) launch_step(k_step_cells<kQ, C, S, LES, TH>, blocks, tpb, st, a, a.early != 0);
}
template <int C, int S, bool LES, bool TH>
void batch_one(BatchArgs& b, int tpb, cudaStream_t st) {
    b.list_blocks = blocks_of(b.nlisted, tpb);
    const unsigned blocks = plan(b.npure * pure_units<kQ, C, S, false>(), tpb, b.list_blocks, kQ != 27, b.run, b.spread);
    if (blocks) launch_step(k_step_cells_batch<kQ, C, S, LES, TH>, blocks, tpb, st, b, true);
}
template <int C, int S, bool LES>
void initial_one(const float* f0, void* A, void* B, const uint8_t* flags, const Geo& g, const Physics& p,
                 const Launch& L) {
    k_initial<kQ, C, S, LES><<<L.rows * L.xchunks, L.tpb, 0, L.stream>>>(f0, A, B, flags, g, p, L.xchunks);
}
// Persistent tile kernel: TILE_CTAS_PER_SM CTAs per SM (capped by the work), dynamic shared
// memory opted in once per kernel instantiation.
template <auto Kernel>
cudaError_t tiles_launch(unsigned smem, int work, cudaStream_t st, const StepArgs& a, const TileArgs& t) {
    static bool ready = false;
    if (!ready) {
        const cudaError_t e =
            cudaFuncSetAttribute(Kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
        if (e != cudaSuccess) return e;
        ready = true;
    }
    int sms = 148;
    int dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int blocks = std::max(1, std::min(work, TILE_CTAS_PER_SM * sms));
    Kernel<<<blocks, TILE_THREADS, smem, st>>>(a, t);
    return cudaGetLastError();
}

template <int C, int S, bool LES>
cudaError_t tiles_one(const StepArgs& a, const TileArgs& t, cudaStream_t st) {
    constexpr unsigned smem = tile_smem_bytes<kQ, S>();
    if (t.ntiles <= 0) return cudaSuccess;
    return tiles_launch<k_step_tiles<kQ, C, S, LES>>(smem, t.ntiles, st, a, t);
}
using TilesFn = cudaError_t (*)(const StepArgs&, const TileArgs&, cudaStream_t);
using CellsFn = void (*)(StepArgs&, int, cudaStream_t);
using BatchFn = void (*)(BatchArgs&, int, cudaStream_t);
using InitFn = void (*)(const float*, void*, void*, const uint8_t*, const Geo&, const Physics&, const Launch&);

#if WK_Q == 9  // [LES][coupled temperature]
#define WK_4(F, C, S) {{F<C, S, false, false>, F<C, S, false, true>}, {F<C, S, true, false>, F<C, S, true, true>}}
#else
#define WK_4(F, C, S) {{F<C, S, false, false>, nullptr}, {F<C, S, true, false>, nullptr}}
#endif
#define WK_TABLE(F)                                                                    \
    {{WK_4(F, 0, 0), WK_4(F, 0, 1), WK_4(F, 0, 2), WK_4(F, 0, 3)},                     \
     {WK_4(F, 1, 0), WK_4(F, 1, 1), WK_4(F, 1, 2), WK_4(F, 1, 3)},                     \
     {WK_4(F, 2, 0), WK_4(F, 2, 1), WK_4(F, 2, 2), WK_4(F, 2, 3)}}
const CellsFn kCells[3][4][2][2] = WK_TABLE(cells_one);
const BatchFn kBatch[3][4][2][2] = WK_TABLE(batch_one);
#undef WK_4
#undef WK_TABLE
#define WK_IROW(C, S) {initial_one<C, S, false>, initial_one<C, S, true>}
const InitFn kInit[3][4][2] = {{WK_IROW(0, 0), WK_IROW(0, 1), WK_IROW(0, 2), WK_IROW(0, 3)},
                               {WK_IROW(1, 0), WK_IROW(1, 1), WK_IROW(1, 2), WK_IROW(1, 3)},
                               {WK_IROW(2, 0), WK_IROW(2, 1), WK_IROW(2, 2), WK_IROW(2, 3)}};
#define WK_SROW(C, S) {tiles_one<C, S, false>, tiles_one<C, S, true>}
const TilesFn kTiles[3][4][2] = {{WK_SROW(0, 0), WK_SROW(0, 1), WK_SROW(0, 2), WK_SROW(0, 3)},
                                 {WK_SROW(1, 0), WK_SROW(1, 1), WK_SROW(1, 2), WK_SROW(1, 3)},
                                 {WK_SROW(2, 0), WK_SROW(2, 1), WK_SROW(2, 2), WK_SROW(2, 3)}};
#undef WK_IROW
#undef WK_SROW

bool valid(int coll, int store) { return coll >= 0 && coll < 3 && store >= 0 && store < 4; }
}  // namespace

cudaError_t WK_CAT(launch_cells_q, WK_Q)(int coll, int store, bool les, StepArgs a, int tpb, cudaStream_t stream) {
    if (!valid(coll, store)) return cudaErrorInvalidValue;
    const CellsFn f = kCells[coll][store][les ? 1 : 0][a.th.on ? 1 : 0];
    if (!f) return cudaErrorInvalidValue;
    f(a, tpb, stream);
    return cudaGetLastError();
}

cudaError_t WK_CAT(launch_batch_q, WK_Q)(int coll, int store, bool les, BatchArgs b, bool thermal, int tpb,
                                        cudaStream_t stream) {
    if (!valid(coll, store)) return cudaErrorInvalidValue;
    const BatchFn f = kBatch[coll][store][les ? 1 : 0][thermal ? 1 : 0];
    if (!f) return cudaErrorInvalidValue;
    f(b, tpb, stream);
    return cudaGetLastError();
}

cudaError_t WK_CAT(launch_tiles_q, WK_Q)(int coll, int store, bool les, const StepArgs& a, const TileArgs& t,
                                        cudaStream_t stream) {
    if (!valid(coll, store)) return cudaErrorInvalidValue;
    return kTiles[coll][store][les ? 1 : 0](a, t, stream);
}

cudaError_t WK_CAT(launch_initial_q, WK_Q)(int coll, int store, bool les, const float* f0, void* a, void* b,
                                          const uint8_t* flags, const Geo& geo, const Physics& phys,
                                          const Launch& L) {
    if (!valid(coll, store)) return cudaErrorInvalidValue;
    kInit[coll][store][les ? 1 : 0](f0, a, b, flags, geo, phys, L);
    return cudaGetLastError();
}

cudaError_t WK_CAT(launch_materialise_q, WK_Q)(int store, const void* fin, const uint8_t* flags, const Geo& geo,
                                              const Links& links, const Physics& phys, const Out& out,
                                              const Launch& L, int direct, const Thermal& th) {
    const int blocks = L.rows * L.xchunks;
#define WK_MAT(S)                                                                               \
    if (direct) k_direct<kQ, S><<<blocks, L.tpb, 0, L.stream>>>(fin, flags, geo, phys, out, L.xchunks, th); \
    else k_materialise<kQ, S><<<blocks, L.tpb, 0, L.stream>>>(fin, flags, geo, links, phys, out, L.xchunks, th)
    switch (store) {
        case 0: WK_MAT(0); break;
        case 1: WK_MAT(1); break;
        case 2: WK_MAT(2); break;
        case 3: WK_MAT(3); break;
        default: return cudaErrorInvalidValue;
    }
#undef WK_MAT
    return cudaGetLastError();
}

#if WK_Q == 9
cudaError_t launch_initial_thermal_q9(int coll, int store, bool les, const float* f0, const float* t0, void* a, void* b,
                                      float* ta, float* tb, const uint8_t* flags, const Geo& geo, const Physics& phys,
                                      const Thermal& th, const Launch& L) {
    if (!valid(coll, store)) return cudaErrorInvalidValue;
    const int blocks = L.rows * L.xchunks;
#define WK_TI(C, S, LES) \
    k_initial_thermal<C, S, LES><<<blocks, L.tpb, 0, L.stream>>>(f0, t0, a, b, ta, tb, flags, geo, phys, th, L.xchunks)
    switch (coll * 8 + store * 2 + (les ? 1 : 0)) {
        case 0: WK_TI(0, 0, false); break;
        case 1: WK_TI(0, 0, true); break;
        case 2: WK_TI(0, 1, false); break;
        case 3: WK_TI(0, 1, true); break;
        case 4: WK_TI(0, 2, false); break;
        case 5: WK_TI(0, 2, true); break;
        case 6: WK_TI(0, 3, false); break;
        case 7: WK_TI(0, 3, true); break;
        case 8: WK_TI(1, 0, false); break;
        case 9: WK_TI(1, 0, true); break;
        case 10: WK_TI(1, 1, false); break;
        case 11: WK_TI(1, 1, true); break;
        case 12: WK_TI(1, 2, false); break;
        case 13: WK_TI(1, 2, true); break;
        case 14: WK_TI(1, 3, false); break;
        case 15: WK_TI(1, 3, true); break;
        case 16: WK_TI(2, 0, false); break;
        case 17: WK_TI(2, 0, true); break;
        case 18: WK_TI(2, 1, false); break;
        case 19: WK_TI(2, 1, true); break;
        case 20: WK_TI(2, 2, false); break;
        case 21: WK_TI(2, 2, true); break;
        case 22: WK_TI(2, 3, false); break;
        case 23: WK_TI(2, 3, true); break;
        default: return cudaErrorInvalidValue;
    }
#undef WK_TI
    return cudaGetLastError();
}
#endif

cudaError_t WK_CAT(launch_flags_q, WK_Q)(const uint8_t* types, uint8_t* flags, const Geo& geo, const FlagCfg& cfg,
                                        const Launch& L) {
    k_flags<kQ><<<L.rows * L.xchunks, L.tpb, 0, L.stream>>>(types, flags, geo, cfg, L.xchunks);
    return cudaGetLastError();
}

// Whole-row TRT kernel (rows.cuh): one block per row of the lattice.
cudaError_t WK_CAT(launch_rows_q, WK_Q)(int store, bool les, const StepArgs& a, int rows, int tpb,
                                       cudaStream_t stream) {
    if (rows <= 0) return cudaSuccess;
    switch (store * 2 + (les ? 1 : 0)) {
        case 0: k_step_rows<kQ, 0, false><<<rows, tpb, 0, stream>>>(a); break;
        case 1: k_step_rows<kQ, 0, true><<<rows, tpb, 0, stream>>>(a); break;
        case 2: k_step_rows<kQ, 1, false><<<rows, tpb, 0, stream>>>(a); break;
        case 3: k_step_rows<kQ, 1, true><<<rows, tpb, 0, stream>>>(a); break;
        case 4: k_step_rows<kQ, 2, false><<<rows, tpb, 0, stream>>>(a); break;
        case 5: k_step_rows<kQ, 2, true><<<rows, tpb, 0, stream>>>(a); break;
        case 6: k_step_rows<kQ, 3, false><<<rows, tpb, 0, stream>>>(a); break;
        case 7: k_step_rows<kQ, 3, true><<<rows, tpb, 0, stream>>>(a); break;
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

namespace {  // internal linkage: every lattice's translation unit has its own pipe_one (kQ differs)
// Pipelined whole-row TRT kernel (rowpipe.cuh): as many CTAs as fit on the device (capped by
// the rows), dynamic shared memory opted in once per instantiation.
template <int S, bool LES, int CAP>
cudaError_t pipe_one(const StepArgs& a, const PipeArgs& p, cudaStream_t stream) {
    constexpr unsigned smem = pipe_smem_bytes<kQ, S, CAP>();
    static int slots = 0;  // resident CTAs on the device
    if (slots == 0) {
        cudaError_t e = cudaFuncSetAttribute(k_step_rows_pipe<kQ, S, LES, CAP>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
        if (e != cudaSuccess) return e;
        // the stages are the kernel's working set: all of the SM's unified memory as shared memory
        e = cudaFuncSetAttribute(k_step_rows_pipe<kQ, S, LES, CAP>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                 cudaSharedmemCarveoutMaxShared);
        if (e != cudaSuccess) return e;
        int per_sm = 0, sms = 0, dev = 0;
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_step_rows_pipe<kQ, S, LES, CAP>,
                                                          pipe_threads<CAP>(), smem);
        if (e != cudaSuccess) return e;
        if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
        if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
        slots = std::max(1, per_sm * sms);
    }
    const int blocks = std::min(p.nrows, slots);
    if (blocks <= 0) return cudaSuccess;
    k_step_rows_pipe<kQ, S, LES, CAP><<<blocks, pipe_threads<CAP>(), smem, stream>>>(a, p);
    return cudaGetLastError();
}
}  // namespace

cudaError_t WK_CAT(launch_rows_pipe_q, WK_Q)(int store, bool les, int cap, const StepArgs& a, const PipeArgs& p,
                                            cudaStream_t stream) {
    const int sel = (cap > 256 ? 8 : 0) + store * 2 + (les ? 1 : 0);
    switch (sel) {
        case 0: return pipe_one<0, false, 256>(a, p, stream);
        case 1: return pipe_one<0, true, 256>(a, p, stream);
        case 2: return pipe_one<1, false, 256>(a, p, stream);
        case 3: return pipe_one<1, true, 256>(a, p, stream);
        case 4: return pipe_one<2, false, 256>(a, p, stream);
        case 5: return pipe_one<2, true, 256>(a, p, stream);
        case 6: return pipe_one<3, false, 256>(a, p, stream);
        case 7: return pipe_one<3, true, 256>(a, p, stream);
        case 8: return pipe_one<0, false, 512>(a, p, stream);
        case 9: return pipe_one<0, true, 512>(a, p, stream);
        case 10: return pipe_one<1, false, 512>(a, p, stream);
        case 11: return pipe_one<1, true, 512>(a, p, stream);
        case 12: return pipe_one<2, false, 512>(a, p, stream);
        case 13: return pipe_one<2, true, 512>(a, p, stream);
        case 14: return pipe_one<3, false, 512>(a, p, stream);
        case 15: return pipe_one<3, true, 512>(a, p, stream);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t WK_CAT(launch_records_q, WK_Q)(const uint8_t* flags, uint4* list, unsigned n, unsigned general,
                                          uint4* records, const Links& links, const Geo& geo, const FlagCfg& cfg,
                                          cudaStream_t stream) {
    if (n == 0) return cudaSuccess;
    k_records<kQ><<<n, CELL, 0, stream>>>(flags, list, general, records, links, geo, cfg);
    return cudaGetLastError();
}

}  // namespace wk
