// Fused pull-stream + boundary + moments + momentum-exchange + collide kernels.
//
// State between steps is the POST-collision population buffer g^k (A/B
// ping-pong, SoA planes [q][node], plane pitch a multiple of 64 elements).
// The reference keeps the post-stream, pre-collision f^k instead
// (src/grid/lattice_grid_2d.cpp:195-265): f^{k+1} = ZouHe(BFL(Stream(Collide(f^k)))).
// With g^k = Collide(f^k), one fused launch computes, per node,
//
//   f^{k+1}(x) = ZouHe(BFL(Pull(g^k)))(x)      -- reference steps 3-5
//   rho, u, momentum exchange from f^{k+1}(x)   -- reference step 6 + scenario MEM
//   g^{k+1}(x) = Collide(f^{k+1}(x))            -- next step's collide
//
// so every quantity the reference exposes after k steps is available from
// g^{k-1} (re-gathered by the materialise kernel), and one step moves
// 2*Q*sizeof(pop) + 1 flag byte per node through HBM.
#pragma once

#include "common.cuh"
#include "lattice.cuh"
#include "pairs2.cuh"

namespace wk {

// Device-side error word bits (read by the host after a launch sequence).
enum : unsigned { ERR_NONFINITE = 1u, ERR_BAD_CONFIG = 2u };

// Division of a 31-bit unsigned value by a run-time constant d: n / d = (n * m) >> (31 + l) with
// l = ceil(log2 d), m = ceil(2^(31 + l) / d) < 2^32 (exact for n < 2^31: n (m d - 2^(31+l)) < 2^(31+l)).
struct FastDiv {
    unsigned m, s;  // s = l - 1; m = 0 for d = 1
    static FastDiv of(unsigned d) {
        if (d <= 1u) return {0u, 0u};
        unsigned l = 0;
        while ((1ull << l) < d) ++l;
        return {static_cast<unsigned>(((1ull << (31 + l)) + d - 1) / d), l - 1u};
    }
    __host__ __device__ __forceinline__ unsigned quot(unsigned n) const {
        return m ? static_cast<unsigned>((static_cast<unsigned long long>(n) * m) >> 32) >> s : n;
    }
};

struct Geo {
    int nx, ny, nz;
    FastDiv by_nx, by_ny;
    int periodic_y, periodic_z;   // 3D: wrap y / z instead of half-way bounce-back walls
    long long pitch;              // elements per population plane
    float uin[3];                 // Zou-He inlet velocity
    float rho_out;                // Zou-He outlet density
    float mom[27];                // moving-wall term 2 w_q 3 (c_q . u_w) (d2q9_streaming.ispc:49-53)
};

// Curved-boundary (BFL) links sorted by fluid node. rec: x = fluid node, y = node of the second
// population, z = plane of the first population | plane of the second << 8 | direction replaced << 16 |
// LINK_MOVES, w = bits of the first population's coefficient c: the replaced value is
// c f_first(node) + (1 - c) f_second - mom, with (first, second) of the branch delta takes
// (d3q19_curved.ispc:36-68).
constexpr unsigned LINK_MOVES = 1u << 24;
struct Links {
    const int* node_start;        // [N] first link of the node, read only where FL_BFL is set
    const uint4* rec;             // [n]
    const float* mom;             // [n] moving-wall term, read only where LINK_MOVES is set
    int count;
};

struct MemLeft {                  // in device memory: what the steps so far left of the forces
    const double* part;           // the last step's force, `slots` partial sums, while it is not in the history yet
    int slots;
    unsigned steps;               // number of entries written to the history
};

struct MemCfg {                   // momentum-exchange monitor
    int enabled;
    float center[3];
    // Every unit of the listed cells with momentum-exchange links owns one slot of `contrib` (slot[2 * entry + half];
    // a whole cell's is slot[2 * entry]), numbered in node order, in the half of `contrib` of the buffer the step
    // reads (stride doubles apart). The next launch sums them in slot order: the force is reproducible bit for bit.
    // Any list of cells that holds these nodes gives the same sums, and `left` says where they are: a graph that a
    // caller captured may follow steps over another list.
    const int* slot;
    int slots;
    double* contrib;              // [2][slots][3]
    long long stride;
    MemLeft* left;
    double* hist;                 // [hist_cap][3]: (Fx, Fy, Tz) in 2D, (Fx, Fy, Fz) in 3D
    int hist_cap;
};

struct Out {                      // optional outputs of the materialise kernel, null for those not wanted
    float* f;                     // FP32 f^k planes (pitch as the state buffers)
    int macro;                    // some moment is wanted
    float* rho;
    float* ux;
    float* uy;
    float* uz;
    float* speed;
};
__device__ __forceinline__ void store_macro(const Out& out, long long i, float rho, const float u[3]) {
    if (out.rho) out.rho[i] = rho;
    if (out.ux) out.ux[i] = u[0];
    if (out.uy) out.uy[i] = u[1];
    if (out.uz) out.uz[i] = u[2];
    if (out.speed) out.speed[i] = sqrtf(u[0] * u[0] + u[1] * u[1] + u[2] * u[2]);
}

template <int Q>
__device__ __forceinline__ int wrap(int v, int n) {
    v += (v < 0) ? n : 0;
    v -= (v >= n) ? n : 0;
    return v;
}

// Pure gather of a node whose pull sources are all in range (after the periodic
// wraps) and plain fluid: the three x positions and the row bases of the
// (dy, dz) shifts are built once, then each load is a warp-uniform plane
// pointer plus a 32-bit in-plane offset.
template <int Q, int S>
__device__ __forceinline__ void gather_pure(const typename Codec<S>::T* __restrict__ fin, const Geo& G, int x, int y,
                                            int z, float f[Q]) {
    using L = Lat<Q>;
    using C = Codec<S>;
    const long long P = G.pitch;
    const int nx = G.nx, ny = G.ny, nz = G.nz;
    const int xs[3] = {x == nx - 1 ? 0 : x + 1, x, x == 0 ? nx - 1 : x - 1};  // source x for cx = -1, 0, +1
    int ys[3] = {y + 1, y, y - 1}, zs[3] = {z + 1, z, z - 1};                // source rows for c = -1, 0, +1
    if (G.periodic_y) {
        ys[0] = ys[0] == ny ? 0 : ys[0];
        ys[2] = ys[2] < 0 ? ny - 1 : ys[2];
    }
    if (G.periodic_z) {
        zs[0] = zs[0] == nz ? 0 : zs[0];
        zs[2] = zs[2] < 0 ? nz - 1 : zs[2];
    }
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        const unsigned off =
            static_cast<unsigned>((zs[L::cz(q) + 1] * ny + ys[L::cy(q) + 1]) * nx + xs[L::cx(q) + 1]);
        f[q] = C::load(fin + q * P + off, L::w(q));
    }
}

// Pull f^{k+1}(x) out of g^k.
template <int Q, int S>
__device__ __forceinline__ void gather(const typename Codec<S>::T* __restrict__ fin, const Geo& G,
                                       const uint8_t* __restrict__ flags, const Links& B, int x, int y, int z,
                                       long long i, uint8_t fl, float f[Q]) {
    using L = Lat<Q>;
    using C = Codec<S>;
    const long long P = G.pitch;
    const int nx = G.nx, ny = G.ny, nz = G.nz;
    if (fl & FL_FAST) {
        gather_pure<Q, S>(fin, G, x, y, z, f);
        if (fl & FL_ZH_IN) zou_he_inlet<Q>(f, G.uin);
        if (fl & FL_ZH_OUT) zou_he_outlet<Q>(f, G.rho_out);
        return;
    }
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        const int o = L::opp(q);
        const int sx = L::cx(q) ? wrap<Q>(x - L::cx(q), nx) : x;
        int sy = y - L::cy(q), sz = z - L::cz(q);
        if (L::cy(q) && G.periodic_y) sy = wrap<Q>(sy, ny);
        if (L::cz(q) && G.periodic_z) sz = wrap<Q>(sz, nz);
        const bool inr = (sy >= 0) && (sy < ny) && (sz >= 0) && (sz < nz);
        if (!inr) {
            f[q] = C::load(fin + o * P + i, L::w(o));  // domain wall: half-way bounce-back
            continue;
        }
        const long long s = (static_cast<long long>(sz) * ny + sy) * nx + sx;
        const uint8_t t = flags[s] & FL_TYPE;
        if (t == CT_SOLID) {
            f[q] = C::load(fin + o * P + i, L::w(o));
        } else if (t == CT_MOVING_WALL) {
            f[q] = C::load(fin + o * P + i, L::w(o)) + G.mom[q];
        } else {
            f[q] = C::load(fin + q * P + s, L::w(q));
        }
    }
    if constexpr (Q == 19) {
        if (fl & FL_BFL) {
            // Bouzidi linear interpolation from post-collision values (d3q19_curved.ispc:36-68).
            for (int k = B.node_start[i]; k < B.count; ++k) {
                const uint4 r = B.rec[k];
                if (r.x != i) break;
                const int o = static_cast<int>((r.z >> 16) & 0xffu);
                const float w = rt_w19(o), c = __uint_as_float(r.w);
                const float fi = C::load(fin + static_cast<long long>(r.z & 0xffu) * P + i, w);
                const float f2 = C::load(fin + static_cast<long long>((r.z >> 8) & 0xffu) * P + r.y, w);
                const float val = c * fi + (1.0f - c) * f2 - ((r.z & LINK_MOVES) ? B.mom[k] : 0.0f);
#pragma unroll
                for (int qq = 0; qq < Q; ++qq)
                    if (qq == o) f[qq] = val;
            }
        }
    }
    if (fl & FL_ZH_IN) zou_he_inlet<Q>(f, G.uin);
    if (fl & FL_ZH_OUT) zou_he_outlet<Q>(f, G.rho_out);
}

// Momentum-exchange links of a fluid node (forces_momentum_exchange.ispc:33-63): bit q where a Solid / MovingWall
// node at x + c_q (x periodic, y / z in range) lies within r_max of the centre. `hit` has bit q where the
// pull of direction q bounced off such a node. The filter's float roundings are the reference's: no contraction.
template <int Q>
__device__ __forceinline__ unsigned mem_links(unsigned hit, int x, int y, int z, const Geo& G, const float center[3],
                                              float r_max, float r_max_sq) {
    using L = Lat<Q>;
    unsigned links = 0;
#pragma unroll
    for (int q = 1; q < Q; ++q) {
        if (!(hit & (1u << L::opp(q)))) continue;
        const int yn = y + L::cy(q), zn = z + L::cz(q);
        if (yn < 0 || yn >= G.ny || zn < 0 || zn >= G.nz) continue;
        const float rx = __fsub_rn(__fadd_rn(float(x), 0.5f * float(L::cx(q))), center[0]);
        const float ry = __fsub_rn(__fadd_rn(float(y), 0.5f * float(L::cy(q))), center[1]);
        const float rz = __fsub_rn(__fadd_rn(float(z), 0.5f * float(L::cz(q))), center[2]);
        float r2 = __fadd_rn(__fmul_rn(rx, rx), __fmul_rn(ry, ry));
        if (L::D == 3) r2 = __fadd_rn(r2, __fmul_rn(rz, rz));
        if (r_max <= 0.0f || r2 <= r_max_sq) links |= 1u << q;
    }
    return links;
}

// Their contributions F += 2 f_q c_q for one direction, and in 2D the torque r x F about the centre (x, y the node's).
template <int Q>
__device__ __forceinline__ void mem_add(int q, float f, int x, int y, const MemCfg& M, double acc[3]) {
    using L = Lat<Q>;
    const double f2 = 2.0 * static_cast<double>(f);
    if (L::cx(q)) acc[0] += L::cx(q) > 0 ? f2 : -f2;
    if (L::cy(q)) acc[1] += L::cy(q) > 0 ? f2 : -f2;
    if constexpr (L::D == 2) {
        const float rx = __fsub_rn(__fadd_rn(float(x), 0.5f * float(L::cx(q))), M.center[0]);
        const float ry = __fsub_rn(__fadd_rn(float(y), 0.5f * float(L::cy(q))), M.center[1]);
        acc[2] += double(rx) * (f2 * L::cy(q)) - double(ry) * (f2 * L::cx(q));
    } else if (L::cz(q)) {
        acc[2] += L::cz(q) > 0 ? f2 : -f2;
    }
}

// D2Q5 temperature coupled to a D2Q9 flow (no reference counterpart; the
// reference's thermal solver uses a D2Q9 temperature and one domain-averaged
// force, src/thermal/thermal_solver.cpp:83-123, src/scenarios/thermal_convection.cpp:70).
// Per node: T = sum g, the flow collides with the body force g + (0, beta_g (T - T_ref)),
// the temperature relaxes to w_q T (1 + 3 c_q.u) with omega_t (first-order equilibrium
// as thermal_kernels.ispc:32). Streaming: anti-bounce-back g_q = -g*_opp + 2 w_q T_wall
// through the y walls (Dirichlet), bounce-back at solid nodes (adiabatic).
struct Thermal {
    int on;
    float omega_t, t_ref, beta_g, t_south, t_north;
    const float* tin;  // post-collision temperature populations of the last step [5][pitch]
    float* tout;
};

struct D2Q5 {  // rest, +x, +y, -x, -y; c_s^2 = 1/3
    __host__ __device__ static constexpr int cx(int q) { return q == 1 ? 1 : (q == 3 ? -1 : 0); }
    __host__ __device__ static constexpr int cy(int q) { return q == 2 ? 1 : (q == 4 ? -1 : 0); }
    __host__ __device__ static constexpr int opp(int q) { return q == 0 ? 0 : (q + 1) % 4 + 1; }
    __host__ __device__ static constexpr float w(int q) { return q == 0 ? 1.0f / 3.0f : 1.0f / 6.0f; }
};

__device__ __forceinline__ float sum_t5(const float t[5]) {
    float T = t[0];
#pragma unroll
    for (int q = 1; q < 5; ++q) T = __fadd_rn(T, t[q]);
    return T;
}

// Body force of a node with temperature T: g + (0, beta_g (T - T_ref), 0), explicit roundings.
__device__ __forceinline__ float buoyant_gy(const Thermal& th, float gy, float T) {
    return __fadd_rn(gy, __fmul_rn(th.beta_g, __fsub_rn(T, th.t_ref)));
}

// BGK relaxation of the temperature populations toward w_q T (1 + 3 c_q.u).
__device__ __forceinline__ void collide_t5(float t[5], float T, const float u[3], float om) {
#pragma unroll
    for (int q = 0; q < 5; ++q) {
        const float cu = __fadd_rn(__fmul_rn(float(D2Q5::cx(q)), u[0]), __fmul_rn(float(D2Q5::cy(q)), u[1]));
        const float geq = __fmul_rn(__fmul_rn(D2Q5::w(q), T), __fadd_rn(1.0f, __fmul_rn(3.0f, cu)));
        t[q] = __fsub_rn(t[q], __fmul_rn(om, __fsub_rn(t[q], geq)));
    }
}

struct StepArgs {
    const void* fin;
    void* fout;
    int cur;                  // index of the buffer fin is
    // plane q of fin, of fin moved by minus direction q's pull offset c_x + c_y nx + c_z nx ny, and of fout
    const void *in[27], *pull[27];
    void* out[27];
    const uint8_t* flags;
    unsigned* status;
    Geo geo;
    Links links;
    MemCfg mem;
    Physics phys;
    unsigned nodes;           // nx ny nz
    unsigned cells;           // cells of the direct range of k_step_cells (0: the listed cells only)
    const uint8_t* cell_kind;  // CELL_* of every cell
    unsigned run;             // units per warp of the direct range
    int reverse;              // the sweep runs from the lattice's end (every other step)
    int evict_first;          // policy of the population loads (read_policy)
    int early;                // host: the launch may start before the stream's last kernel has ended (launch_step)
    unsigned nunits, list_blocks, spread;
    const unsigned* units;    // units of the listed cells (cells.cuh)
    const uint4* list;        // listed cells: first node, node count | LIST_* bits, first curved link, links
    const uint4* records;     // [nlist][CELL] node records (cells.cuh)
    Thermal th;            // D2Q9 lattices only; th.on = 0 otherwise
    const uint8_t* row_kind;  // per-row descriptor bytes of k_step_rows (rows.cuh); one block per row
};

constexpr int CELL = 64;  // nodes per cell (cells.cuh)

// Value stored for population q: FP32 holds f, FP16 / BF16 / FP16C hold h = f / w - 1.
// load_h / store_h move the stored value itself (no decode) for the h-space math.
template <int S>
__device__ __forceinline__ float load_raw(const typename Codec<S>::T* p, L2Policy pol) {
    if constexpr (S == STORE_F32) {
        return ld_pop(p, pol);
    } else {
        const unsigned short v = ld_pop(reinterpret_cast<const unsigned short*>(p), pol);
        if constexpr (S == STORE_F16) return __half2float(__ushort_as_half(v));
        else if constexpr (S == STORE_F16C) return f16c_decode(v);
        else return __bfloat162float(__ushort_as_bfloat16(v));
    }
}
template <int S>
__device__ __forceinline__ void store_raw(typename Codec<S>::T* p, float v) {
    if constexpr (S == STORE_F32) {
        *p = v;
    } else {
        unsigned short h;
        if constexpr (S == STORE_F16) h = __half_as_ushort(__float2half_rn(v));
        else if constexpr (S == STORE_F16C) h = static_cast<unsigned short>(f16c_encode(v));
        else h = __bfloat16_as_ushort(__float2bfloat16_rn(v));
        *reinterpret_cast<unsigned short*>(p) = h;
    }
}
// The same for the decoded population (w its weight).
template <int S>
__device__ __forceinline__ float load_f(const typename Codec<S>::T* p, float w, L2Policy pol) {
    const float v = load_raw<S>(p, pol);
    return S == STORE_F32 ? v : fmaf(w, v, w);
}
template <int S>
__device__ __forceinline__ void store_f(typename Codec<S>::T* p, float f, float w) {
    store_raw<S>(p, S == STORE_F32 ? f : fmaf(f, 1.0f / w, -1.0f));
}

// The two 16-bit values of a 32-bit word (little endian: node x in the low half) as floats,
// and two floats stored as one rounded 16-bit pair.
template <int S>
__device__ __forceinline__ float raw_lo(unsigned w) {
    if constexpr (S == STORE_F16) return __half2float(__ushort_as_half(static_cast<unsigned short>(w & 0xffffu)));
    else if constexpr (S == STORE_F16C) return f16c_decode(w & 0xffffu);
    else return __bfloat162float(__ushort_as_bfloat16(static_cast<unsigned short>(w & 0xffffu)));
}
template <int S>
__device__ __forceinline__ float raw_hi(unsigned w) {
    if constexpr (S == STORE_F16) return __half2float(__ushort_as_half(static_cast<unsigned short>(w >> 16)));
    else if constexpr (S == STORE_F16C) return f16c_decode(w >> 16);
    else return __bfloat162float(__ushort_as_bfloat16(static_cast<unsigned short>(w >> 16)));
}
template <int S>
__device__ __forceinline__ void store_pair(typename Codec<S>::T* p, float2 v) {
    unsigned w;
    if constexpr (S == STORE_F16) {
        const __half2 h = __floats2half2_rn(v.x, v.y);  // .x in the low half
        w = *reinterpret_cast<const unsigned*>(&h);
    } else if constexpr (S == STORE_F16C) {
        w = f16c_encode2(v);
    } else {
        const __nv_bfloat162 h = __floats2bfloat162_rn(v.x, v.y);
        w = *reinterpret_cast<const unsigned*>(&h);
    }
    *reinterpret_cast<unsigned*>(p) = w;
}

// Zou-He on one of the two nodes of a packed pair (lane 0 = .x, 1 = .y); the
// formulas work on f, so shifted values are decoded and encoded around them.
template <int Q, bool HS>
__device__ __forceinline__ void zou_he_half(float2* f, int lane, uint8_t fl, const Geo& G) {
    using L = Lat<Q>;
    float t[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        const float v = lane ? f[q].y : f[q].x;
        t[q] = HS ? fmaf(L::w(q), v, L::w(q)) : v;
    }
    if (fl & FL_ZH_IN) zou_he_inlet<Q>(t, G.uin);
    if (fl & FL_ZH_OUT) zou_he_outlet<Q>(t, G.rho_out);
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        const float v = HS ? fmaf(t[q], 1.0f / L::w(q), -1.0f) : t[q];
        if (lane) f[q].y = v;
        else f[q].x = v;
    }
}

// Re-gather f^k from g^{k-1} and write FP32 populations and/or macroscopic fields
// (the reference's f_src and its rho/u/speed arrays after step k,
// lattice_grid_2d.cpp:257-262). Solid nodes report their frozen populations.
template <int Q, int S>
__global__ void __launch_bounds__(512) k_materialise(const void* fin_v, const uint8_t* flags, Geo geo, Links links,
                                                     Physics phys, Out out, int xchunks, Thermal th) {
    using L = Lat<Q>;
    using C = Codec<S>;
    using T = typename C::T;
    const T* fin = static_cast<const T*>(fin_v);
    const int row = blockIdx.x / xchunks;
    const int x = (blockIdx.x - row * xchunks) * blockDim.x + threadIdx.x;
    if (x >= geo.nx) return;
    const int y = row % geo.ny, z = row / geo.ny;
    const long long i = static_cast<long long>(row) * geo.nx + x;
    const uint8_t fl = flags[i];
    float f[Q];
    if ((fl & FL_TYPE) == CT_SOLID) {
#pragma unroll
        for (int q = 0; q < Q; ++q) f[q] = C::load(fin + q * geo.pitch + i, L::w(q));
    } else {
        gather<Q, S>(fin, geo, flags, links, x, y, z, i, fl, f);
    }
    if (out.f) {
#pragma unroll
        for (int q = 0; q < Q; ++q) out.f[q * geo.pitch + i] = f[q];
    }
    if (out.macro) {
        float g[3] = {phys.g[0], phys.g[1], phys.g[2]};
        if (th.on) {  // the step's local buoyancy: T^k is the sum of the current post-collision temperature
            float t5[5];
#pragma unroll
            for (int q = 0; q < 5; ++q) t5[q] = th.tin[q * geo.pitch + i];
            g[1] = buoyant_gy(th, phys.g[1], sum_t5(t5));
        }
        float rho, u[3];
        node_moments<Q>(f, g, rho, u);
        store_macro(out, i, rho, u);
    }
}

// Initial collide of a coupled flow + temperature state (f^0 and T populations
// g^0 in FP32 scratch): A <- Collide(f^0) with the local buoyancy, TA <- Collide_T(g^0);
// B <- f^0, TB <- g^0. Solid nodes copy through.
template <int COLL, int S, bool LES>
__global__ void __launch_bounds__(512) k_initial_thermal(const float* f0, const float* t0, void* a_v, void* b_v,
                                                         float* ta, float* tb, const uint8_t* flags, Geo geo,
                                                         Physics phys, Thermal th, int xchunks) {
    using L = Lat<9>;
    using C = Codec<S>;
    using T = typename C::T;
    const int row = blockIdx.x / xchunks;
    const int x = (blockIdx.x - row * xchunks) * blockDim.x + threadIdx.x;
    if (x >= geo.nx) return;
    const long long i = static_cast<long long>(row) * geo.nx + x;
    const long long P = geo.pitch;
    float f[9], t5[5];
#pragma unroll
    for (int q = 0; q < 9; ++q) f[q] = f0[q * P + i];
#pragma unroll
    for (int q = 0; q < 5; ++q) t5[q] = t0[q * P + i];
    T* A = static_cast<T*>(a_v);
    T* Bf = static_cast<T*>(b_v);
#pragma unroll
    for (int q = 0; q < 9; ++q) C::store(Bf + q * P + i, f[q], L::w(q));
#pragma unroll
    for (int q = 0; q < 5; ++q) tb[q * P + i] = t5[q];
    if ((flags[i] & FL_TYPE) != CT_SOLID) {
        const float Tn = sum_t5(t5);
        Physics ph = phys;
        ph.g[1] = buoyant_gy(th, phys.g[1], Tn);
        float rho, u[3];
        node_moments<9>(f, ph.g, rho, u);
        collide<9, COLL, LES>(f, rho, u, ph);
        collide_t5(t5, Tn, u, th.omega_t);
    }
#pragma unroll
    for (int q = 0; q < 9; ++q) C::store(A + q * P + i, f[q], L::w(q));
#pragma unroll
    for (int q = 0; q < 5; ++q) ta[q * P + i] = t5[q];
}

// Initial collide from FP32 populations f^0: buffer A <- g^0 = Collide(f^0)
// (solid nodes copy through, d2q9_collision_bgk.ispc:22-28), buffer B <- f^0.
// B's fluid entries are overwritten by the first step; until then B is the
// reference's f_src, and its solid entries stay the frozen populations.
template <int Q, int COLL, int S, bool LES>
__global__ void __launch_bounds__(512) k_initial(const float* f0, void* a_v, void* b_v, const uint8_t* flags,
                                                 Geo geo, Physics phys, int xchunks) {
    using L = Lat<Q>;
    using C = Codec<S>;
    using T = typename C::T;
    const int row = blockIdx.x / xchunks;
    const int x = (blockIdx.x - row * xchunks) * blockDim.x + threadIdx.x;
    if (x >= geo.nx) return;
    const long long i = static_cast<long long>(row) * geo.nx + x;
    float f[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) f[q] = f0[q * geo.pitch + i];
    T* A = static_cast<T*>(a_v);
    T* Bf = static_cast<T*>(b_v);
#pragma unroll
    for (int q = 0; q < Q; ++q) C::store(Bf + q * geo.pitch + i, f[q], L::w(q));
    if ((flags[i] & FL_TYPE) != CT_SOLID) {
        float rho, u[3];
        node_moments<Q>(f, phys.g, rho, u);
        collide<Q, COLL, LES>(f, rho, u, phys);
    }
#pragma unroll
    for (int q = 0; q < Q; ++q) C::store(A + q * geo.pitch + i, f[q], L::w(q));
}

}  // namespace wk
