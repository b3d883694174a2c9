// Fused stage kernel of the second-order Euler step: Green-Gauss gradients,
// smooth-switch limiter, MUSCL + Roe flux, per-cell sums, RK update, ghost
// fill and residual partials of one tile of T cells in one CTA, one launch
// per RK stage (calc_gradients + calc_limiters + calc_time_derivatives +
// update_cells + update_bounds of explicit.cpp:112-417 for one stage).
//
// A tile stages the states of its cells, of their face neighbours (ring 1)
// and of the ring-1 cells' other neighbours (ring 2).  The gradient phase
// gives one thread (or 2 or 4 lanes, each with its share of the variables,
// which do not mix there) a cell of the tile or of ring 1: it computes the
// limited gradients in registers and leaves, for every flux edge of the cell,
// the cell's face state in shared memory.  The flux phase then reads the two
// face states of an edge from consecutive addresses, and nothing else of the
// cells.  The limited gradients never leave the registers: per stage the
// kernel reads the stage state, the base state and the constant geometry once
// and writes the new state.  Ring-1 gradients are computed by every tile that
// borders the cell (the same arithmetic in each, so the results are identical
// and, in the exact policy, bit-identical to the reference's).
//
// The geometry of the gradient phase is stored per (gradient cell, face), in
// the order the threads read it: FP64 holds the cell's Green-Gauss
// coefficient (the gradient is the sum of a_f (q_nb - q), since a closed cell's
// face normals sum to zero) and the vector to the face centre; FP32 and the exact
// policy hold what the face value needs.  FP32 takes the face values
// q_i + (q_j - q_i) g, the limiter per face and the Roe flux on the unit normal
// with the roundings that its one-ring kernels have: its results are pinned bit
// for bit, since flows amplify another order of operations to 1e-4 and more of
// the residual norms.  (The FP64 forms in FP32 take 301 us per step of a 20-step
// call at 998k cells, these 352; they are nearer to 64 bits, but other results.)
// It goes from global memory straight into registers, with coalesced 16- or
// 32-byte loads issued before the dependency wait.
//
// What bounds it and why this form: the former kernel kept gradients,
// centroids and edge arrays in shared memory and gathered them again per edge.
// Its shared-memory wavefronts (about 345 per 32 cells) and its instructions
// (46 warp instructions per cell in FP32) each took 37-40 us of a 998k-cell
// stage by themselves.  The flux edges' geometry and the cells' 1 / area come
// through shared memory too, copied before the dependency wait: loaded where
// they are used, each of the two flux passes and the update waited an L2
// latency for them (998k cells FP64: 723 us per RK5 step, 676 with the copies).
// Now, of a 998k-cell stage: FP32 45 warp instructions per cell at 66 % of the
// issue rate, 63 us; FP64 58, latency-bound at 16 warps per SM, 125 us.
#pragma once
#include "fv_tile.cuh"

namespace fvgpu {

// Shared-memory layout of one fused tile, in bytes from the start.
//  - state planes [max_slots] of the staged states;
//  - face-state planes of the flux edges' first and second cells
//    [2 * max_flux]; the flux leaving the first cell and entering the second
//    replaces them, and after the per-cell sums the store holds the residual
//    warp sums;
//  - the base state of the owned cells (FP64, [T][4]);
//  - the flux edges' geometry [max_flux][4] and 1 / area of the owned cells;
//  - the limited gradients (and, exact, the limiters) of owned cells with a
//    boundary ghost, for the ghost fill; viscous: the unlimited gradients of
//    every slot, the limiters, and the tile's e2 and ar.
struct FusedSmem {
    int q, fs, qb, gx, gy, lm, eg, ria, gl, gd, e2, ar, total, total_grad, total_run;
    int ls, lf, lt;  // plane strides (units)
};
template <class M>
inline FusedSmem fused_smem(int max_slots, int max_grad, int max_flux, int max_ghost, int T, bool viscous) {
    constexpr int NU = (int)(4 * sizeof(typename M::S) / 16);
    FusedSmem L{};
    L.ls = max_slots;
    L.lf = 2 * max_flux;
    L.lt = viscous ? max_grad : T;
    int o = 0;
    L.q = o; o += 16 * NU * max_slots;
    // the face states, the time step's {u, v, c} or the residual warp sums
    L.fs = o; o += std::max({32 * NU * max_flux, 16 * NU * max_grad, (kFusedThreads / 32) * 4 * (int)sizeof(double)});
    L.qb = o; o += 32 * T;
    L.gx = o; o += 16 * NU * L.lt;
    L.gy = o; o += 16 * NU * L.lt;
    L.lm = o; if (M::exact || viscous) o += 16 * NU * L.lt;
    L.eg = o; o += 16 * NU * max_flux;
    L.ria = o; o += 8 * T;
    L.total = o;
    // the run kernel keeps the tile's ghosts behind that
    L.gd = o; o += 16 * NU * max_ghost;
    L.gl = o; o += (8 * max_ghost + 15) / 16 * 16;
    L.e2 = o; if (viscous) o += 16 * NU * max_flux;
    L.ar = o; if (viscous) o += (4 * NU * max_grad + 15) / 16 * 16;
    L.total_run = o;
    // the gradient kernel of the split layout and the dt kernel: the states
    // and {u, v, c} of the gradient slots
    L.total_grad = L.fs + 16 * NU * max_grad;
    return L;
}

// Dynamic shared memory of a CTA at most: 227 KB with the kernels' static
// variables (under 1 KB).
constexpr size_t kSmemMost = 226 * 1024;

struct FusedParams {
    Params P;
    int T;
    int threads;               // threads per CTA: T, 2T (FV_SCHED_TILE2) or lanes * T
    int lanes;                 // lanes per cell of the gradient and update phases: 1 or 4 (exact only)
    int nf;                    // faces per gradient slot: 3 (triangles only) or 4
    int max_slots, max_grad, max_flux;
    // [n_tiles][2]: {slot_off, halo_off, flux_off, n_flux},
    // {n1, n2, owned cells | ghosts << 16, ghost_off}
    const int4* info;
    const int32_t* halo;       // device cell of each ring-1, then ring-2 slot
    // per gradient slot (T owned, then n1 ring-1 slots of every tile) four
    // face words: neighbour slot (0xFFFF = no face) | face-state unit << 16
    // (flux edge + max_flux on the edge's second side) | kWordGhost (the
    // neighbour is a boundary ghost) | kWordNoFlux (not a flux edge).  FP32
    // with nf = 3: the fourth word holds `sl`.
    const uint4* hd;
    // per gradient slot and face, at nf * slot_off + f * (T + n1) + slot:
    // FP64 S[4] {a_x, a_y, d_x, d_y}; exact S[4] {n_x, n_y, length (negative
    // on the edge's second side), weight} and S[2] {d_x, d_y} in rec2 (d: face
    // centre - centroid); FP32 as exact, the weight negative with the length
    const void* rec;
    const void* rec2;
    const void* sl;            // per gradient slot: FP64 1 / (K sqrt(A))^3; FP32 A; exact double2 {1 / A, (K sqrt(A))^3}
    // S[4] per flux edge: n_x, n_y, length and, exact, the signed zero that a
    // boundary ghost's zero gradient adds; first order: its two slots in the
    // bits of the fourth (edge_slots)
    const void* eg;
    const double* ria;         // [n_own] 1 / area
    const void* area;          // S [n_total]
    FusedSmem L;               // shared-memory layout (fused_smem)
    // boundary ghosts of the tiles' owned cells, one thread each: {interior
    // slot | group << 16, device cell}, and S[4] {n_x, n_y, d_x, d_y}
    const int2* gl;
    const void* gd;
    int max_ghost;             // ghosts of a tile at most
    const void* e2;            // viscous: S[4] per flux edge {t_x, t_y, 1 / distance, 0} (t: unit vector of c_i - c_j)
    const void* ar;            // viscous: S per gradient slot: the area
};

constexpr uint32_t kWordGhost = 0x40000000u, kWordNoFlux = 0x80000000u;
constexpr int kMaxFluxUnits = 0x3FFF;  // 2 * max_flux at most
__device__ __forceinline__ int word_nbr(uint32_t w) { return (int)(w & 0xFFFFu); }
__device__ __forceinline__ int word_unit(uint32_t w) { return (int)((w >> 16) & 0x3FFFu); }

__device__ __forceinline__ uint32_t edge_slots(float e3) { return __float_as_uint(e3); }
__device__ __forceinline__ uint32_t edge_slots(double e3) { return (uint32_t)__double_as_longlong(e3); }

// One 4-vector of S at a 16- or 32-byte aligned global address.
__device__ __forceinline__ void ldg4(const float* p, float* v) {
    const float4 x = __ldg(reinterpret_cast<const float4*>(p));
    v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
}
__device__ __forceinline__ void ldg4(const double* p, double* v) {  // one 256-bit load
    asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]), "=d"(v[3]) : "l"(p));
}

// NV consecutive variables (from v0) of 4-vectors kept in shared-memory
// planes of 16-byte units (FP32 one float4 plane, FP64 two double2 planes
// `stride` units apart), so that reads of random slots are free of bank
// conflicts.
template <class S, int NV>
struct Planes;
template <int NV>
struct Planes<float, NV> {
    __device__ static __forceinline__ void get(const uint4* p, int, int r, int v0, float* v) {
        const float* a = reinterpret_cast<const float*>(p + r) + v0;
        if (NV == 4) {
            const float4 x = *reinterpret_cast<const float4*>(a);
            v[0] = x.x; v[1 % NV] = x.y; v[2 % NV] = x.z; v[3 % NV] = x.w;
        } else if (NV == 2) {
            const float2 x = *reinterpret_cast<const float2*>(a);
            v[0] = x.x; v[1 % NV] = x.y;
        } else {
            v[0] = a[0];
        }
    }
    __device__ static __forceinline__ void put(uint4* p, int, int r, int v0, const float* v) {
        float* a = reinterpret_cast<float*>(p + r) + v0;
        if (NV == 4) *reinterpret_cast<float4*>(a) = make_float4(v[0], v[1 % NV], v[2 % NV], v[3 % NV]);
        else if (NV == 2) *reinterpret_cast<float2*>(a) = make_float2(v[0], v[1 % NV]);
        else a[0] = v[0];
    }
    // asynchronous copy of the whole 4-vector at global g into slot r
    __device__ static __forceinline__ void stage(uint4* p, int, int r, const float* g) { cpa16(p + r, g); }
};
template <int NV>
struct Planes<double, NV> {
    __device__ static __forceinline__ void get(const uint4* p, int stride, int r, int v0, double* v) {
        if (NV == 4) {
            const double2 x = reinterpret_cast<const double2*>(p)[r];
            const double2 y = reinterpret_cast<const double2*>(p + stride)[r];
            v[0] = x.x; v[1 % NV] = x.y; v[2 % NV] = y.x; v[3 % NV] = y.y;
        } else if (NV == 2) {
            const double2 x = reinterpret_cast<const double2*>(p + (v0 >> 1) * stride)[r];
            v[0] = x.x; v[1 % NV] = x.y;
        } else {
            v[0] = reinterpret_cast<const double*>(p + (v0 >> 1) * stride + r)[v0 & 1];
        }
    }
    __device__ static __forceinline__ void put(uint4* p, int stride, int r, int v0, const double* v) {
        if (NV == 4) {
            reinterpret_cast<double2*>(p)[r] = make_double2(v[0], v[1 % NV]);
            reinterpret_cast<double2*>(p + stride)[r] = make_double2(v[2 % NV], v[3 % NV]);
        } else if (NV == 2) {
            reinterpret_cast<double2*>(p + (v0 >> 1) * stride)[r] = make_double2(v[0], v[1 % NV]);
        } else {
            reinterpret_cast<double*>(p + (v0 >> 1) * stride + r)[v0 & 1] = v[0];
        }
    }
    __device__ static __forceinline__ void stage(uint4* p, int stride, int r, const double* g) {
        cpa16(p + r, g);
        cpa16(p + stride + r, g + 2);
    }
};

// NV consecutive values of a 4-vector in global memory
template <class S, int NV>
__device__ __forceinline__ void ldv(const S* a, S* v) {
    if (NV == 4 && sizeof(S) == 4) {
        const float4 x = *reinterpret_cast<const float4*>(a);
        v[0] = (S)x.x; v[1 % NV] = (S)x.y; v[2 % NV] = (S)x.z; v[3 % NV] = (S)x.w;
    } else if (NV >= 2 && sizeof(S) == 8) {
#pragma unroll
        for (int i = 0; i < NV / 2; ++i) {
            const double2 x = reinterpret_cast<const double2*>(a)[i];
            v[2 * i] = (S)x.x; v[(2 * i + 1) % NV] = (S)x.y;
        }
    } else {
#pragma unroll
        for (int i = 0; i < NV; ++i) v[i] = a[i];
    }
}
template <class S, int NV>
__device__ __forceinline__ void stv(S* a, const S* v) {
    if (NV == 4 && sizeof(S) == 4) {
        *reinterpret_cast<float4*>(a) = make_float4((float)v[0], (float)v[1 % NV], (float)v[2 % NV], (float)v[3 % NV]);
    } else if (NV >= 2 && sizeof(S) == 8) {
#pragma unroll
        for (int i = 0; i < NV / 2; ++i)
            reinterpret_cast<double2*>(a)[i] = make_double2((double)v[2 * i], (double)v[(2 * i + 1) % NV]);
    } else {
#pragma unroll
        for (int i = 0; i < NV; ++i) a[i] = v[i];
    }
}

// The NV-variable shares of the 4 / NV lanes of one cell (consecutive lanes
// of a warp, all in the same branch), as one 4-vector in every lane.
template <class S, int NV>
__device__ __forceinline__ void share(const S* v, S* all) {
    if (NV == 4) {
#pragma unroll
        for (int k = 0; k < 4; ++k) all[k] = v[k % NV];
    } else {
        constexpr int LP = 4 / NV;
        const int lane = threadIdx.x & 31, first = lane & ~(LP - 1);
        const unsigned m = ((1u << LP) - 1u) << first;
#pragma unroll
        for (int k = 0; k < 4; ++k) all[k] = __shfl_sync(m, v[k % NV], first + k / NV);
    }
}
// this lane's share of a 4-vector
template <class S, int NV>
__device__ __forceinline__ void own_share(const S* all, int v0, S* v) {
    if (NV == 4) {
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k % NV] = all[k];
    } else if (NV == 2) {
        v[0] = v0 ? all[2] : all[0];
        v[1 % NV] = v0 ? all[3] : all[1];
    } else {
        v[0] = v0 == 0 ? all[0] : v0 == 1 ? all[1] : v0 == 2 ? all[2] : all[3];
    }
}

// guard_face (fv_tile.cuh) of a face state held in shares
template <class S, int NV, bool EXACT>
__device__ __forceinline__ void guard_share(const Params& P, S* qf, const S* qc) {
    if (!P.positivity_guard) return;
    S a[4];
    share<S, NV>(qf, a);
    if (face_state_bad<S, EXACT>(P, a)) {
#pragma unroll
        for (int i = 0; i < NV; ++i) qf[i] = qc[i];
    }
}

// One gradient slot's geometry: face words and records.
template <class M, int NF>
struct SlotGeo {
    using S = typename M::S;
    static constexpr bool faces = M::exact || sizeof(S) == 4;  // face values (rec2), or differences
    uint32_t w[NF];
    S sl[M::exact ? 2 : 1];
    S a[NF][4];
    S d[faces ? NF : 1][2];
    __device__ __forceinline__ bool face(int f) const { return f < 3 || word_nbr(w[f]) != 0xFFFF; }
    __device__ __forceinline__ S dx(int f) const { if constexpr (faces) return d[f][0]; else return a[f][2]; }
    __device__ __forceinline__ S dy(int f) const { if constexpr (faces) return d[f][1]; else return a[f][3]; }
    __device__ __forceinline__ static void prefetch(const FusedParams& FP, uint32_t slot_off, uint32_t G, uint32_t r) {
        auto pf = [](const void* p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p)); };
        pf(FP.hd + (slot_off + r));
#pragma unroll
        for (int f = 0; f < NF; ++f) pf((const S*)FP.rec + 4 * (size_t)(NF * slot_off + r + f * G));
    }
    __device__ __forceinline__ void load(const FusedParams& FP, uint32_t slot_off, uint32_t G, uint32_t r) {
        const uint4 h = __ldg(FP.hd + (slot_off + r));
        w[0] = h.x; w[1] = h.y; w[2] = h.z;
        if constexpr (NF == 4) w[NF - 1] = h.w;
        if constexpr (M::exact) {
            const double2 x = __ldg(reinterpret_cast<const double2*>(FP.sl) + (slot_off + r));
            sl[0] = x.x; sl[1] = x.y;
        } else if constexpr (NF == 3 && sizeof(S) == 4) {
            sl[0] = __uint_as_float(h.w);
        } else {
            sl[0] = __ldg((const S*)FP.sl + (slot_off + r));
        }
        const uint32_t b = NF * slot_off + r;
#pragma unroll
        for (int f = 0; f < NF; ++f) {
            ldg4((const S*)FP.rec + 4 * (size_t)(b + f * G), a[f]);
            if constexpr (M::exact) {
                const double2 x = __ldg(reinterpret_cast<const double2*>(FP.rec2) + (b + f * G));
                d[f][0] = x.x; d[f][1] = x.y;
            } else if constexpr (faces) {
                const float2 x = __ldg(reinterpret_cast<const float2*>(FP.rec2) + (b + f * G));
                d[f][0] = x.x; d[f][1] = x.y;
            }
        }
    }
};

// CFL or constant time step of owned cell c (slot l) and of its boundary
// ghosts from {u, v, c, rho} of the tile's slots (calc_dt of
// examples/forwardStep/main.cpp:140-185 and examples/naca/main.cpp:142-183;
// VISC, fast policies: and the viscous kinds, AR the slots' areas).
// edge(el, e): normal and length of flux edge el; A: the cell's area, which is
// its ghosts' too.  Returns the ordered-key minimum of the values written.
template <class M, int NF, bool VISC, class Edge>
__device__ __forceinline__ unsigned long long fused_cell_dt(const FusedParams& FP, const TileIO& io, const uint32_t* fw,
                                                            const uint4* W, int l, int c, int halo_off,
                                                            typename M::S A, Edge edge, double& di,
                                                            const typename M::S* AR = nullptr) {
    using S = typename M::S;
    const Params& P = FP.P;
    const S cfl = (S)P.cfl;
    const bool sum = P.dt_kind == 1 || (VISC && P.dt_kind == 4), constant = P.dt_kind == 0;
    const bool visc = VISC && P.dt_kind >= 3;
    unsigned long long kmin = ~0ull;
    S ws[4];
    Planes<S, 4>::get(W, FP.max_grad, l, 0, ws);
    S acc = sum ? S(0) : S(1);
    // viscous kinds (see tile_cell_dt_visc): C mu / pr max(4 / 3, gamma) / rho le^2 / A
    const S vc = VISC ? S(2) * (S)(P.mu / P.pr) * fast::tmax(S(4.0 / 3.0), (S)P.gamma) : S(0);
    const S vs = VISC ? vc * fast::rcp(ws[3]) * fast::rcp(A) : S(0);
#pragma unroll
    for (int f = 0; f < NF; ++f) {
        const uint32_t w = fw[f];
        const int o = word_nbr(w);
        if (f == 3 && o == 0xFFFF) continue;
        const bool ghost = (w & kWordGhost) != 0;
        S e[4], wn[4];
        const int u = word_unit(w);
        const bool side = u >= FP.max_flux;
        edge(side ? u - FP.max_flux : u, e);
        Planes<S, 4>::get(W, FP.max_grad, o, 0, wn);
        double dg = P.dt_const;
        if constexpr (M::exact) {
            if (sum) {
                const double es = ws[2] + fabs(ws[0] * e[0] + ws[1] * e[1]);
                const double en = wn[2] + fabs(wn[0] * e[0] + wn[1] * e[1]);
                const double center = side ? exact::dmax(en, es) : exact::dmax(es, en);
                acc += center * e[2];
                if (ghost) {
                    double d = 0.;
                    d += center * e[2];
                    dg = cfl * A / d;
                }
            } else if (!constant) {
                const double es = (ws[2] + fabs(ws[0])) * e[0] + (ws[2] + fabs(ws[1])) * e[1];
                acc = exact::dmin(acc, cfl * (A / e[2]) / fabs(es));
                if (ghost) {
                    const double en = (wn[2] + fabs(wn[0])) * e[0] + (wn[2] + fabs(wn[1])) * e[1];
                    dg = exact::dmin(1.0, cfl * (A / e[2]) / fabs(en));
                }
            }
        } else if (visc) {
            const S le2 = e[2] * e[2], vn = vc * fast::rcp(wn[3]) * le2 * fast::rcp(AR[o]);
            if (sum) {
                const S center = fast::tmax(ws[2] + fabs(ws[0] * e[0] + ws[1] * e[1]) + vs * le2,
                                            wn[2] + fabs(wn[0] * e[0] + wn[1] * e[1]) + vn);
                acc += center * e[2];
                if (ghost) dg = (double)(cfl * A * fast::rcp(center * e[2]));
            } else {
                const S es = (ws[2] + fabs(e[0] * ws[0]) + fabs(e[1] * ws[1])) * e[2] + vs * le2;
                acc = fast::tmin(acc, cfl * A * fast::rcp(es));
                if (ghost) {
                    const S en = (wn[2] + fabs(e[0] * wn[0]) + fabs(e[1] * wn[1])) * e[2] + vn;
                    dg = (double)fast::tmin(S(1), cfl * A * fast::rcp(en));
                }
            }
        } else if (sum) {
            const S center = fast::tmax(ws[2] + fabs(fast::dot2(ws[0], e[0], ws[1], e[1])),
                                        wn[2] + fabs(fast::dot2(wn[0], e[0], wn[1], e[1])));
            acc = fast::madd(center, e[2], acc);
            if (ghost) dg = (double)(cfl * A * fast::rcp(center * e[2]));
        } else if (!constant) {
            const S es = fast::dot2(ws[2] + fabs(ws[0]), e[0], ws[2] + fabs(ws[1]), e[1]);
            acc = fast::tmin(acc, cfl * A * fast::rcp(e[2] * fabs(es)));
            if (ghost) {
                const S en = fast::dot2(wn[2] + fabs(wn[0]), e[0], wn[2] + fabs(wn[1]), e[1]);
                dg = (double)fast::tmin(S(1), cfl * A * fast::rcp(e[2] * fabs(en)));
            }
        }
        if (ghost) {
            io.dt[FP.halo[halo_off + o - FP.T]] = dg;
            kmin = kmin_(kmin, tkey(dg));
        }
    }
    if constexpr (M::exact) di = constant ? P.dt_const : (sum ? cfl * A / acc : acc);
    else di = constant ? P.dt_const : (double)(sum ? cfl * A * fast::rcp(acc) : acc);
    io.dt[c] = di;
    return kmin_(kmin, tkey(di));
}
// {u, v, c, rho} of a state, in the reference's arithmetic (exact) or the fast one
template <class M>
__device__ __forceinline__ void fused_speeds(double gamma, const typename M::S* q, typename M::S* w) {
    if constexpr (M::exact) {
        const double gm1 = gamma - 1;
        bool ok = true;
        const exact::Recip r = exact::recip(q[0], ok);
        w[0] = exact::quot(q[1], r, ok);
        w[1] = exact::quot(q[2], r, ok);
        double c2 = exact::quot((gm1 * (q[3] - exact::quot(0.5, r, ok) * (q[1] * q[1] + q[2] * q[2]))) * gamma, r, ok);
        if (!ok) {
            w[0] = q[1] / q[0];
            w[1] = q[2] / q[0];
            c2 = (gm1 * (q[3] - 0.5 / q[0] * (q[1] * q[1] + q[2] * q[2]))) * gamma / q[0];
        }
        w[2] = sqrt(c2);
    } else {
        fast::speeds((typename M::S)gamma, q, w);
    }
    w[3] = q[0];
}

// Gradients and limiters of gradient slot r (this lane's variables), and the
// face states of its flux edges into shared memory.  PH: see fused_tile.
template <class M, int NV, int NF, int PH, bool VISC = false>
__device__ __forceinline__ void fused_slot(const FusedParams& FP, const TileIO& io, unsigned char* smem_raw,
                                           const SlotGeo<M, NF>& geo, int r, int v0, int c0, int halo_off, int flux_off) {
    using S = typename M::S;
    using PL = Planes<S, NV>;
    const Params& P = FP.P;
    const FusedSmem& L = FP.L;
    const int T = FP.T;
    uint4* Q = reinterpret_cast<uint4*>(smem_raw + L.q);
    uint4* FS = reinterpret_cast<uint4*>(smem_raw + L.fs);
    uint4* GX = reinterpret_cast<uint4*>(smem_raw + L.gx);
    uint4* GY = reinterpret_cast<uint4*>(smem_raw + L.gy);
    uint4* LM = reinterpret_cast<uint4*>(smem_raw + L.lm);
    S qs[NV], gx[NV], gy[NV], lim[NV];
    PL::get(Q, L.ls, r, v0, qs);
    if constexpr (PH == 2) {
        const size_t g = r < T ? (size_t)(c0 + r) : (size_t)__ldg(FP.halo + halo_off + r - T);
        ldv<S, NV>((const S*)io.gx + 4 * g + v0, gx);
        ldv<S, NV>((const S*)io.gy + 4 * g + v0, gy);
    } else if constexpr (M::exact) {
        double qmn[NV], qmx[NV];
#pragma unroll
        for (int k = 0; k < NV; ++k) { gx[k] = 0; gy[k] = 0; qmn[k] = qs[k]; qmx[k] = qs[k]; lim[k] = 1; }
#pragma unroll
        for (int f = 0; f < NF; ++f) {
            if (!geo.face(f)) continue;
            const double nx = geo.a[f][0], ny = geo.a[f][1], le = geo.a[f][2], g = geo.a[f][3];
            const bool side = (geo.a[f][2] < 0.);  // a negative length marks the edge's second cell
            const double len = fabs(le);
            double qn[NV];
            PL::get(Q, L.ls, word_nbr(geo.w[f]), v0, qn);
#pragma unroll
            for (int k = 0; k < NV; ++k) {
                if (!side) {
                    const double fl = (qs[k] * (1.0 - g) + qn[k] * g) * len;
                    gx[k] += fl * nx; gy[k] += fl * ny;
                } else {
                    const double fl = (qn[k] * (1.0 - g) + qs[k] * g) * len;
                    gx[k] -= fl * nx; gy[k] -= fl * ny;
                }
                qmn[k] = exact::dmin(qmn[k], qn[k]); qmx[k] = exact::dmax(qmx[k], qn[k]);
            }
        }
        const double invA = geo.sl[0], K3a = geo.sl[1];
        const double tol = 1e-15;
        // the divisions of a group of variables together (exact::quot)
        constexpr int GK = NV == 4 ? 1 : NV;
#pragma unroll
        for (int k0 = 0; k0 < NV; k0 += GK) {
            double sig[GK], y[GK][NF];
            bool on[GK][NF], ok = true, limited = false;
#pragma unroll
            for (int i = 0; i < GK; ++i) {
                const int k = k0 + i;
                gx[k] *= invA; gy[k] *= invA;
                const double delta_max = qmx[k] - qs[k];
                const double delta_min = qmn[k] - qs[k];
                const double d2 = (delta_max - delta_min) * (delta_max - delta_min);
                if (d2 <= K3a) sig[i] = 1.;
                else if (d2 <= 2 * K3a) {
                    const double z = (d2 / K3a - 1.0);
                    sig[i] = 2.0 * z * z * z - 3.0 * z * z + 1.0;
                } else sig[i] = 0.;
                limited |= sig[i] < 1.0;
            }
            if (!limited) continue;  // sig = 1: lim = 1
#pragma unroll
            for (int i = 0; i < GK; ++i) {
                const int k = k0 + i;
#pragma unroll
                for (int f = 0; f < NF; ++f) {
                    on[i][f] = false;
                    y[i][f] = 0.;
                    if (!geo.face(f)) continue;
                    const double dqg = gx[k] * geo.dx(f) + gy[k] * geo.dy(f);
                    on[i][f] = sig[i] < 1.0 && (dqg > tol || dqg < -tol);
                    const double num = on[i][f] ? (dqg > tol ? qmx[k] - qs[k] : qmn[k] - qs[k]) : 0.;
                    const double den = on[i][f] ? dqg : 1.;
                    y[i][f] = exact::quot(num, exact::recip(den, ok), ok);
                }
            }
            if (P.limiter == 2) {
#pragma unroll
                for (int i = 0; i < GK; ++i)
#pragma unroll
                    for (int f = 0; f < NF; ++f) {
                        const double z = y[i][f];
                        y[i][f] = exact::quot(z * z + 2.0 * z, exact::recip(z * z + z + 2.0, ok), ok);
                    }
            } else {
#pragma unroll
                for (int i = 0; i < GK; ++i)
#pragma unroll
                    for (int f = 0; f < NF; ++f) y[i][f] = exact::limiter_func(P.limiter, y[i][f]);
            }
            if (!ok) {  // an operand out of exact::quot's range
#pragma unroll
                for (int i = 0; i < GK; ++i)
#pragma unroll
                    for (int f = 0; f < NF; ++f) {
                        if (!on[i][f]) continue;
                        const int k = k0 + i;
                        const double dqg = gx[k] * geo.dx(f) + gy[k] * geo.dy(f);
                        y[i][f] = exact::limiter_func(P.limiter, (dqg > tol ? qmx[k] - qs[k] : qmn[k] - qs[k]) / dqg);
                    }
            }
#pragma unroll
            for (int i = 0; i < GK; ++i)
#pragma unroll
                for (int f = 0; f < NF; ++f) {
                    if (!geo.face(f)) continue;
                    double lv = on[i][f] ? y[i][f] : 1.0;
                    lv = sig[i] + (1.0 - sig[i]) * lv;
                    lim[k0 + i] = exact::dmin(lim[k0 + i], lv);
                }
        }
    } else if constexpr (sizeof(S) == 4) {
        float qmn[NV], qmx[NV], sig[NV];
#pragma unroll
        for (int k = 0; k < NV; ++k) { gx[k] = 0; gy[k] = 0; qmn[k] = qs[k]; qmx[k] = qs[k]; lim[k] = 1; }
#pragma unroll
        for (int f = 0; f < NF; ++f) {
            if (!geo.face(f)) continue;
            const float nx = geo.a[f][0], ny = geo.a[f][1], le = geo.a[f][2], g = geo.a[f][3];
            float qn[NV];
            PL::get(Q, L.ls, word_nbr(geo.w[f]), v0, qn);
#pragma unroll
            for (int k = 0; k < NV; ++k) {
                // q_i + (q_j - q_i) g of the edge's first and second cells i and
                // j; on the second side le and g are negative
                const float fl = fast::fma_(qn[k] - qs[k], g, le < 0.f ? qn[k] : qs[k]) * le;
                gx[k] = fast::fma_(fl, nx, gx[k]);
                gy[k] = fast::fma_(fl, ny, gy[k]);
                qmn[k] = fast::vmin(qmn[k], qn[k]);
                qmx[k] = fast::vmax(qmx[k], qn[k]);
            }
        }
        const float A = geo.sl[0], invA = fast::rcp(A), Ka = (float)P.K * fast::sqrt_(A), K3a = Ka * Ka * Ka;
        const float rK3a = fast::rcp(K3a), tol = 1e-15f;
        bool limited = false;
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            gx[k] *= invA;
            gy[k] *= invA;
            const float d = qmx[k] - qmn[k], d2 = d * d;
            if (d2 <= K3a) sig[k] = 1;
            else if (d2 <= 2 * K3a) {
                const float y = d2 * rK3a - 1.f;
                sig[k] = (2.f * y - 3.f) * y * y + 1.f;
            } else sig[k] = 0;
            limited |= sig[k] < 1.f;
        }
        if (limited) {
            auto apply = [&](auto kind) {
#pragma unroll
                for (int k = 0; k < NV; ++k) {
                    if (!(sig[k] < 1.f)) continue;
                    const float mx = qmx[k] - qs[k], mn = qmn[k] - qs[k];
                    float least = 1.f;  // of phi: the limiter grows with it, rounding included
#pragma unroll
                    for (int f = 0; f < NF; ++f) {
                        if (!geo.face(f)) continue;
                        const float dqg = gx[k] * geo.dx(f) + gy[k] * geo.dy(f);
                        const bool up = dqg > tol;
                        const float phi = fast::limiter_ratio(kind(), up ? mx : mn, dqg);
                        if (up || dqg < -tol) least = fast::vmin(least, phi);
                    }
                    lim[k] = fast::vmin(1.f, fast::fma_(1.f - sig[k], least, sig[k]));
                    gx[k] *= lim[k];
                    gy[k] *= lim[k];
                }
            };
            if (P.limiter == 2) apply([] { return 2; });
            else if (P.limiter == 1) apply([] { return 1; });
            else apply([&] { return P.limiter; });
        }
    } else {
        S mn[NV], mx[NV], sig[NV];
#pragma unroll
        for (int k = 0; k < NV; ++k) { gx[k] = 0; gy[k] = 0; mn[k] = 0; mx[k] = 0; lim[k] = 1; }
#pragma unroll
        for (int f = 0; f < NF; ++f) {
            if (!geo.face(f)) continue;
            S qn[NV];
            PL::get(Q, L.ls, word_nbr(geo.w[f]), v0, qn);
#pragma unroll
            for (int k = 0; k < NV; ++k) {
                const S d = qn[k] - qs[k];
                gx[k] = fast::fma_(geo.a[f][0], d, gx[k]);
                gy[k] = fast::fma_(geo.a[f][1], d, gy[k]);
                mn[k] = fast::vmin(mn[k], d);
                mx[k] = fast::vmax(mx[k], d);
            }
        }
        bool limited = false;
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            sig[k] = fast::smooth_switch(mx[k] - mn[k], geo.sl[0]);
            limited |= sig[k] < S(1);
        }
        if (limited && (!VISC || P.order2)) {
            auto apply = [&](auto kind) {
#pragma unroll
                for (int k = 0; k < NV; ++k) {
                    // the largest and smallest g . d over the faces
                    // give the strictest ratio of each sign
                    S up = 0, lo = 0;
#pragma unroll
                    for (int f = 0; f < NF; ++f) {
                        if (!geo.face(f)) continue;
                        const S dq = fast::fma_(gy[k], geo.dy(f), gx[k] * geo.dx(f));
                        up = fast::vmax(up, dq);
                        lo = fast::vmin(lo, dq);
                    }
                    lim[k] = fast::limiter_min(kind(), sig[k], mx[k], mn[k], up, lo);
                    if constexpr (!VISC) {  // the face gradient takes the unlimited ones
                        gx[k] *= lim[k];
                        gy[k] *= lim[k];
                    }
                }
            };
            if (P.limiter == 2) apply([] { return 2; });
            else if (P.limiter == 1) apply([] { return 1; });
            else apply([&] { return P.limiter; });
        }
    }
    if constexpr (M::exact && PH == 0) {
        // the adjoint keeps a stage's gradients and limiters
        if (io.gx != nullptr && r < T) {
            stv<S, NV>((S*)io.gx + 4 * (size_t)(c0 + r) + v0, gx);
            stv<S, NV>((S*)io.gy + 4 * (size_t)(c0 + r) + v0, gy);
            stv<S, NV>((S*)io.lim + 4 * (size_t)(c0 + r) + v0, lim);
        }
    }
    if constexpr (PH == 1) {
        stv<S, NV>((S*)io.gx + 4 * (size_t)(c0 + r) + v0, gx);
        stv<S, NV>((S*)io.gy + 4 * (size_t)(c0 + r) + v0, gy);
    } else {
        if constexpr (VISC) {
            PL::put(GX, L.lt, r, v0, gx);
            PL::put(GY, L.lt, r, v0, gy);
        }
        uint32_t any = 0;
#pragma unroll
        for (int f = 0; f < NF; ++f) {
            if (!geo.face(f)) continue;
            S qf[NV];
#pragma unroll
            for (int k = 0; k < NV; ++k) {
                if constexpr (M::exact) qf[k] = qs[k] + (gx[k] * geo.dx(f) + gy[k] * geo.dy(f)) * lim[k];
                else if constexpr (VISC)
                    qf[k] = P.order2 ? fast::fma_(fast::fma_(gy[k], geo.dy(f), fast::mul_(gx[k], geo.dx(f))), lim[k], qs[k]) : qs[k];
                else qf[k] = fast::fma_(gy[k], geo.dy(f), fast::fma_(gx[k], geo.dx(f), qs[k]));
            }
            guard_share<S, NV, M::exact>(P, qf, qs);
            if (!(geo.w[f] & kWordNoFlux)) PL::put(FS, L.lf, word_unit(geo.w[f]), v0, qf);
            any |= geo.w[f];
        }
        if (any & kWordGhost) {
            // a ghost's face state is its cell value (gradient 0); the
            // cell's own gradients are kept for the ghost fill
#pragma unroll
            for (int f = 0; f < NF; ++f) {
                if (!geo.face(f) || !(geo.w[f] & kWordGhost)) continue;
                const int u = word_unit(geo.w[f]), el = u < FP.max_flux ? u : u - FP.max_flux;
                S qn[NV];
                PL::get(Q, L.ls, word_nbr(geo.w[f]), v0, qn);
                if constexpr (M::exact) {
                    // the signed zero that the ghost's zero gradient adds
                    const double z = reinterpret_cast<const double*>(smem_raw + L.eg)[4 * el + 3];
#pragma unroll
                    for (int k = 0; k < NV; ++k) qn[k] += z;
                }
                PL::put(FS, L.lf, u < FP.max_flux ? u + FP.max_flux : el, v0, qn);
            }
            if constexpr (!VISC) {
                PL::put(GX, L.lt, r, v0, gx);
                PL::put(GY, L.lt, r, v0, gy);
            }
            if constexpr (M::exact || VISC) PL::put(LM, L.lt, r, v0, lim);
        }
    }
}

// Sum of the fluxes of owned cell uc (this lane's variables) in reference edge
// order and RK update (update_cells, explicit.cpp:368-378); res: its residual
// terms when partial sums are due.  ghosts: the tile fills boundary ghosts.
template <class M, int NV, int NF, bool REMOTE>
__device__ __forceinline__ void fused_update(const FusedParams& FP, const TileIO& io, unsigned char* smem_raw,
                                             const uint32_t* own, int uc, int v0, int c0, int tc, double dtc,
                                             const double& s_dt, bool ghosts, const PartIO& pio, double* res) {
    using S = typename M::S;
    using PL = Planes<S, NV>;
    const Params& P = FP.P;
    const FusedSmem& L = FP.L;
    uint4* FS = reinterpret_cast<uint4*>(smem_raw + L.fs);
    const double* QB = reinterpret_cast<const double*>(smem_raw + L.qb);
    const double* RA = reinterpret_cast<const double*>(smem_raw + L.ria);
    const int c = c0 + uc;
    double qt[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) qt[k] = 0.;
    const double ra = RA[uc];  // 1 / area
    double A = 1.;
    if (M::exact || io.partials != nullptr) A = (double)__ldg((const S*)FP.area + c);
    bool ok = M::exact ? exact::quot_range(A) && exact::quot_range(ra) : true;
#pragma unroll
    for (int f = 0; f < NF; ++f) {
        if (f == 3 && word_nbr(own[f]) == 0xFFFF) continue;
        S fe[NV];
        PL::get(FS, L.lf, word_unit(own[f]), v0, fe);
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            if constexpr (M::exact) qt[k] += exact::quot(fe[k], exact::recip_of(A, ra), ok);
            else qt[k] += (double)fe[k];
        }
    }
    if (M::exact && !ok) {
#pragma unroll
        for (int k = 0; k < NV; ++k) qt[k] = 0.;
#pragma unroll
        for (int f = 0; f < NF; ++f) {
            if (f == 3 && word_nbr(own[f]) == 0xFFFF) continue;
            S fe[NV];
            PL::get(FS, L.lf, word_unit(own[f]), v0, fe);
#pragma unroll
            for (int k = 0; k < NV; ++k) qt[k] += (double)fe[k] / A;
        }
    }
    if constexpr (!M::exact) {
#pragma unroll
        for (int k = 0; k < NV; ++k) qt[k] *= ra;
    }
    {
        if (io.ctrl != nullptr && P.global_dt) {
            dtc = s_dt;
            if (tc < 0) {  // a tile across two cases of a batch: this cell's case
                const int k = P.cell_case[c];
                unsigned long long key = ~0ull;
                for (int i = 0; i < kDtSlots; ++i) key = kmin_(key, io.dtkeys[(size_t)k * kDtSlots + i]);
                const double d0 = io.dt[P.case_cell0[k]];
                dtc = (d0 != d0) ? d0 : tkey_inv(key);
            }
        }
        double qb[NV], qnew[NV];
        ldv<double, NV>(QB + 4 * uc + v0, qb);
        if constexpr (M::exact) {
#pragma unroll
            for (int k = 0; k < NV; ++k) qnew[k] = qb[k] + qt[k] * dtc * io.alpha;
        } else {
            const double da = dtc * io.alpha;
#pragma unroll
            for (int k = 0; k < NV; ++k) qnew[k] = fma(qt[k], da, qb[k]);
        }
        S qs[NV];
#pragma unroll
        for (int k = 0; k < NV; ++k) qs[k] = (S)qnew[k];
        if (sizeof(S) == 8) {
            stv<double, NV>(io.q_out + 4 * (size_t)c + v0, qnew);
        } else {
            stv<S, NV>((S*)io.s_out + 4 * (size_t)c + v0, qs);
            if (io.write_f64) stv<double, NV>(io.q_out + 4 * (size_t)c + v0, qnew);
        }
        if constexpr (REMOTE) {
            // this cell's new state into every part that reads it
            const RemoteIO& R = *pio.remote;
            if (c < R.n_band) {
                for (int i = R.cell_off[c]; i < R.cell_off[c + 1]; ++i) {
                    const int2 d = R.cell_dst[i];
                    stv<S, NV>((S*)R.dst[d.x] + 4 * (size_t)d.y + v0, qs);
                }
            }
        }
        if (ghosts) PL::put(reinterpret_cast<uint4*>(smem_raw + L.q), L.ls, uc, v0, qs);  // for fused_ghosts
        if (io.partials != nullptr) {
#pragma unroll
            for (int k = 0; k < NV; ++k) res[k] = qt[k] * qt[k] * A;
        }
    }
}

// Ghost fill of the tile's boundary ghosts (update_bounds, explicit.cpp:380-417),
// one thread each, once every thread has stored its cell's new state.  O2: from
// the limited gradients, else from the cell value.  gl, gd: the tile's entries.
template <class M, bool REMOTE, bool O2, bool VISC = false>
__device__ __forceinline__ void fused_ghosts(const FusedParams& FP, const TileIO& io, unsigned char* smem_raw,
                                             const int2* gl, const typename M::S* gd, int n, const PartIO& pio) {
    using S = typename M::S;
    using P4 = Planes<S, 4>;
    const Params& P = FP.P;
    const FusedSmem& L = FP.L;
    const int N = P.n_real;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const int2 e = gl[i];
        const int uc = e.x & 0xFFFF, group = e.x >> 16, g = e.y;
        S qs[4], qint[4], b[4];
        const S n0 = gd[4 * i], n1 = gd[4 * i + 1];
        P4::get(reinterpret_cast<const uint4*>(smem_raw + L.q), L.ls, uc, 0, qs);
        if (O2 && (!VISC || P.order2)) {
            S gx[4], gy[4], lm[4];
            const S d0 = gd[4 * i + 2], d1 = gd[4 * i + 3];
            P4::get(reinterpret_cast<const uint4*>(smem_raw + L.gx), L.lt, uc, 0, gx);
            P4::get(reinterpret_cast<const uint4*>(smem_raw + L.gy), L.lt, uc, 0, gy);
            if constexpr (M::exact || VISC) P4::get(reinterpret_cast<const uint4*>(smem_raw + L.lm), L.lt, uc, 0, lm);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if constexpr (M::exact) qint[k] = qs[k] + (gx[k] * d0 + gy[k] * d1) * lm[k];
                else if constexpr (VISC) qint[k] = fast::fma_(fast::fma_(gy[k], d1, fast::mul_(gx[k], d0)), lm[k], qs[k]);
                else qint[k] = fast::fma_(gy[k], d1, fast::fma_(gx[k], d0, qs[k]));
            }
            guard_share<S, 4, M::exact>(P, qint, qs);
        } else {
#pragma unroll
            for (int k = 0; k < 4; ++k) qint[k] = qs[k];
        }
        if constexpr (M::exact) exact::bc<4>(P, group, g - N, b, qint, n0, n1);
        else fast::bc<4, S>(P, group, g - N, b, qint, n0, n1);
        if (sizeof(S) == 8) {
            stv<S, 4>((S*)io.q_out + 4 * (size_t)g, b);
        } else {
            stv<S, 4>((S*)io.s_out + 4 * (size_t)g, b);
            if (io.write_f64) {
                double bd[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) bd[k] = (double)b[k];
                stv<double, 4>(io.q_out + 4 * (size_t)g, bd);
            }
        }
        if constexpr (REMOTE) {
            const RemoteIO& R = *pio.remote;
            const int go = g - N;
            if (go < R.n_own_ghost)
                for (int j = R.ghost_off[go]; j < R.ghost_off[go + 1]; ++j) {
                    const int2 d = R.ghost_dst[j];
                    stv<S, 4>((S*)R.dst[d.x] + 4 * (size_t)d.y, b);
                }
        }
    }
}

// Residual partial sums of tile t: a butterfly over the cells of a warp (lanes
// of equal variables), then the warps in order.  The warp sums share the flux
// store once every thread has read its fluxes.
template <int NV>
__device__ __forceinline__ void fused_partials(const TileIO& io, unsigned char* store, int t, int v0, double* res) {
    constexpr int V = 4, LP = V / NV;
#pragma unroll
    for (int k = 0; k < NV; ++k)
#pragma unroll
        for (int o = 16; o >= LP; o >>= 1) res[k] += __shfl_xor_sync(0xffffffffu, res[k], o);
    double* red = reinterpret_cast<double*>(store);
    __syncthreads();
    if ((threadIdx.x & 31) < LP)
#pragma unroll
        for (int k = 0; k < NV; ++k) red[(threadIdx.x >> 5) * V + v0 + k] = res[k];
    __syncthreads();
    if (threadIdx.x < V) {
        const int nw = blockDim.x >> 5;
        double s = 0.;
        for (int w = 0; w < nw; ++w) s += red[w * V + threadIdx.x];
        io.partials[(size_t)t * V + threadIdx.x] = s;
    }
}

// One tile t.  Returns false when the step is inactive (nothing written).
// NV: variables per lane of the gradient and update phases (4 / NV lanes per cell).
// PH 0: the whole stage.  PH 1: the limited gradients of the owned cells only,
// written to io.gx, io.gy; PH 2: the stage with the gradients read from there
// (FP64's split layout).  PH 3: the step's time step only.
// PART: a decomposition part's tile, whose owned cells come from the tile
// info (a part owns fewer real cells than its local mesh holds).
template <class M, int FLUX, int NV, int NF, int PH, bool REMOTE, bool PART>
__device__ __forceinline__ bool fused_tile(const FusedParams& FP, const TileIO& io, const int t, const PartIO& pio) {
    using S = typename M::S;
    using PL = Planes<S, NV>;
    using P4 = Planes<S, 4>;
    constexpr int V = 4, LP = V / NV;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ double s_dt;
    const Params& P = FP.P;
    const int N = P.n_real, T = FP.T;
    const int4 ia = FP.info[2 * t], ib = FP.info[2 * t + 1];
    const int slot_off = ia.x, halo_off = ia.y, flux_off = ia.z, n_flux = ia.w;
    const int n1 = ib.x, nh = ib.x + ib.y, n_ghost = ib.z >> 16;
    const int c0 = t * T, nown = PART ? (ib.z & 0xFFFF) : min(T, N - c0);
    const int G = T + n1;
    const FusedSmem& L = FP.L;
    uint4* Q = reinterpret_cast<uint4*>(smem_raw + L.q);
    uint4* FS = reinterpret_cast<uint4*>(smem_raw + L.fs);
    double* QB = reinterpret_cast<double*>(smem_raw + L.qb);
    const S* EG = reinterpret_cast<const S*>(smem_raw + L.eg);
    double* RA = reinterpret_cast<double*>(smem_raw + L.ria);
    const bool global_dt = io.ctrl != nullptr && P.global_dt;
    const int l = threadIdx.x;
    const int r0 = l / LP, rstep = blockDim.x / LP;  // gradient slots of this lane
    const int v0 = (l % LP) * NV;                    // its first variable
    // ---- constant tile data first (may overlap the previous kernel's tail):
    // the first gradient slot's geometry and the halo indices, into registers
    SlotGeo<M, NF> geo;
    geo.load(FP, slot_off, G, min(r0, G - 1));
    const int h0 = l < nh ? __ldg(FP.halo + halo_off + l) : 0;
    // the second pass's slot: its lines into L1, so that it is not waited for
    if (r0 + rstep < G && PH != 3) geo.prefetch(FP, slot_off, G, r0 + rstep);
    if constexpr (PH == 0 || PH == 2) {
        constexpr int C = (int)sizeof(S) / 4;  // 16-byte chunks per edge
        const uint4* src = reinterpret_cast<const uint4*>((const S*)FP.eg + 4 * (size_t)flux_off);
        uint4* dst = reinterpret_cast<uint4*>(smem_raw + L.eg);
        for (int i = l; i < C * n_flux; i += blockDim.x) cpa16(dst + i, src + i);
        if (l < nown) cpa8(RA + l, FP.ria + c0 + l);
    }
    // the owned cell of the update phase (r0 < nown there) and its faces
    const int uc = r0;
    uint32_t own[NF];
#pragma unroll
    for (int f = 0; f < NF; ++f) own[f] = geo.w[f];
    // the tile's case (batches); -1: the tile spans two cases
    const int tc = (global_dt && P.n_cases > 1) ? P.tile_case[t] : 0;
    // reference cell 0 of the tile's case, whose dt carries the NaN rule of min_dt
    const int cell0 = (P.n_cases > 1 && tc >= 0) ? P.case_cell0[tc] : P.cell0;
    pdl_wait();
    // every load of data written by earlier kernels is issued here together
    const bool inactive = t_inactive(io.ctrl);
    if constexpr (REMOTE) {
        // a band tile reads halo cells: wait for the senders' epoch of this
        // stage's input (bounded; a tile that gives up is skipped)
        __shared__ int s_gave_up;
        const RemoteIO& R = *pio.remote;
        if (threadIdx.x == 0) {
            s_gave_up = 0;
            if (!inactive && t < R.n_band_tiles) {
                const unsigned long long need = io.ctrl->step * (unsigned long long)pio.stages + pio.stage;
                for (int i = 0; i < R.n_src && !s_gave_up; ++i) {
                    const unsigned long long* f = R.my_flags + R.src[i];
                    long long polls = 0;
                    while (ld_acquire_sys_u64(f) < need) {
                        if (++polls > R.limit) {
                            atomicExch(R.err, 1);
                            s_gave_up = 1;
                            break;
                        }
                        __nanosleep(256);
                    }
                }
            }
        }
        __syncthreads();
        if (s_gave_up) { cpa_wait(); return false; }
    }
    double dtc = 0.;
    if ((PH == 0 || PH == 2) && !global_dt && uc < nown) dtc = io.dt[c0 + uc];
    // the owned states and, behind them, the base states, in 16-byte chunks of
    // consecutive threads (a CTA has at least T threads)
    constexpr int NU = (int)sizeof(S) / 4;
    const uint4* gq = reinterpret_cast<const uint4*>((const S*)io.q_stage + 4 * (size_t)c0) + l;
    const uint4* gb = reinterpret_cast<const uint4*>(io.q_base + 4 * (size_t)c0) + l;
    if (l < NU * nown) cpa16(NU == 1 ? Q + l : Q + (l & 1) * L.ls + (l >> 1), gq);
    if (NU == 2 && l + T < 2 * nown) cpa16(Q + (l & 1) * L.ls + ((l + T) >> 1), gq + T);
    for (int h = l; h < nh; h += blockDim.x) {
        const int g = h == l ? h0 : __ldg(FP.halo + halo_off + h);
        P4::stage(Q, L.ls, T + h, (const S*)io.q_stage + 4 * (size_t)g);
    }
    cpa_commit();
    if (PH == 0 || PH == 2) {
        if (l < 2 * nown) cpa16(QB + 2 * l, gb);
        if (l + T < 2 * nown) cpa16(QB + 2 * (l + T), gb + T);
    }
    cpa_commit();
    if ((PH == 0 || PH == 2) && global_dt && tc >= 0 && threadIdx.x < 32) {
        // min_dt (explicit.cpp:555-564) of the tile's case; a NaN in its dt[0] wins
        const unsigned long long* keys = io.dtkeys + (size_t)tc * kDtSlots;
        const double d0 = io.dt[cell0];
        unsigned long long k = kmin_(keys[threadIdx.x], keys[threadIdx.x + 32]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) k = kmin_(k, __shfl_xor_sync(0xffffffffu, k, o));
        if (threadIdx.x == 0) s_dt = (d0 != d0) ? d0 : tkey_inv(k);
    }
    cpa_wait_prior();  // the states; the base state is awaited before the update
    if (inactive) {
        cpa_wait();
        return false;
    }
    __syncthreads();

    // ---- gradients, limiters and face states of the owned cells and ring 1
    // (calc_gradients + calc_limiters, explicit.cpp:112-258, and the MUSCL
    // states of calc_time_derivatives, 297-320)
    if constexpr (PH == 3) {
        uint4* W = FS;
        for (int r = l; r < G; r += blockDim.x) {
            if (r >= nown && r < T) continue;
            S q[V], w[V];
            P4::get(Q, L.ls, r, 0, q);
            fused_speeds<M>(P.gamma, q, w);
            P4::put(W, FP.max_grad, r, 0, w);
        }
        __syncthreads();
        unsigned long long kmin = ~0ull;
        double di;
        auto edge = [&](int el, S* e) { ldg4((const S*)FP.eg + 4 * (size_t)(flux_off + el), e); };
        if (l < nown)
            kmin = fused_cell_dt<M, NF, false>(FP, io, own, W, l, c0 + l, halo_off, __ldg((const S*)FP.area + c0 + l), edge, di);
        tile_dt_reduce(P, T, io, t, l, nown, kmin);
        return true;
    }
    const int gslots = PH == 1 ? nown : G;
    for (int r = r0; r < gslots;) {
        // unused slots of a last, partial tile and ring-1 ghosts have no faces
        if (word_nbr(geo.w[0]) != 0xFFFF) {
            fused_slot<M, NV, NF, PH>(FP, io, smem_raw, geo, r, v0, c0, halo_off, flux_off);
        }
        r += rstep;
        if (r >= gslots) break;
        geo.load(FP, slot_off, G, r);
    }
    if constexpr (PH == 1) return true;
    __syncthreads();

    // ---- one flux per flux edge (calc_time_derivatives, explicit.cpp:321-350)
    for (int el = l; el < n_flux; el += blockDim.x) {
        S e[4], qL[V], qR[V], f[V];
        e[0] = EG[4 * el]; e[1] = EG[4 * el + 1]; e[2] = EG[4 * el + 2];
        P4::get(FS, L.lf, el, 0, qL);
        P4::get(FS, L.lf, el + FP.max_flux, 0, qR);
        if constexpr (M::exact) {
            exact::flux_dev<FLUX>(P.gamma, f, qL, qR, e[0], e[1]);
#pragma unroll
            for (int k = 0; k < V; ++k) f[k] *= e[2];
        } else {
            fast::flux_le<FLUX, true>((S)P.gamma, f, qL, qR, e[0], e[1], e[2]);
        }
#pragma unroll
        for (int k = 0; k < V; ++k) qL[k] = -f[k];
        P4::put(FS, L.lf, el, 0, qL);
        P4::put(FS, L.lf, el + FP.max_flux, 0, f);
    }
    cpa_wait();  // the base state
    __syncthreads();

    // ---- per-cell sums in reference edge order, RK update, ghost fill
    // (update_cells + update_bounds, explicit.cpp:368-417)
    double res[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) res[k] = 0.;
    if (uc < nown) {
        fused_update<M, NV, NF, REMOTE>(FP, io, smem_raw, own, uc, v0, c0, tc, dtc, s_dt, n_ghost != 0, pio, res);
    }
    if (n_ghost != 0) {
        __syncthreads();
        fused_ghosts<M, REMOTE, true>(FP, io, smem_raw, FP.gl + ib.w, (const S*)FP.gd + 4 * (size_t)ib.w, n_ghost, pio);
    }
    if (io.partials != nullptr) fused_partials<NV>(io, smem_raw + L.fs, t, v0, res);
    if constexpr (REMOTE) {
        // every band tile counts itself once its stores are visible; the
        // last one releases this stage's epoch to the readers
        const RemoteIO& R = *pio.remote;
        if (t < R.n_band_tiles) {
            __syncthreads();
            if (threadIdx.x == 0) {
                __threadfence_system();
                const unsigned long long epoch = io.ctrl->step * (unsigned long long)pio.stages + pio.stage + 1;
                const unsigned long long done = atomicAdd(R.ctr, 1ull) + 1ull;
                if (done == epoch * (unsigned long long)R.n_band_tiles) {
                    __threadfence_system();
                    for (int d = 0; d < R.n_dst; ++d) st_release_sys_u64(R.flag[d], epoch);
                }
            }
        }
    }
    return true;
}

// Register budget of the one-lane kernel, as CTAs of 256 threads per SM: FP32
// 64 registers (32 warps per SM), FP64 128 (16 warps).  Measured at sizes beyond
// the run kernel, us per RK5 step: FP32 with 64 | 48 | 80 registers, forward step
// 163k cells 79 | 79 | 78, 315k 123 | 133 | 126, 998k 346 | 384 | 389, NACA 1M
// 316 | 376 | 351, strips of 422k cells 176 | 202 | 191 (48 registers spill);
// FP64 with 128 | 80 registers (which spill), 163k 133 | 128, 315k 241 | 254,
// 998k 679 | 693.
template <class M>
struct FusedBlocks { static constexpr int v = sizeof(typename M::S) == 4 ? 4 : 2; };

// One CTA per tile, tiles [0, grid).
template <class M, int FLUX, int NV, int NF>
__global__ void __launch_bounds__(NV == 4 ? kTileMax : kFusedThreads, NV == 4 ? FusedBlocks<M>::v : 1)
    k_tile_fused(FusedParams FP, TileIO io) {
    pdl_trigger();
    fused_tile<M, FLUX, NV, NF, 0, false, false>(FP, io, (int)blockIdx.x, PartIO{});
}

// FP64's split layout, over the same tiles with the same
// arithmetic: gradients, then the rest of the stage; and the time step (the
// first kernel of a step).
template <class M, int NF>
__global__ void __launch_bounds__(kTileMax) k_tile_fused_grad(FusedParams FP, TileIO io) {
    pdl_trigger();
    fused_tile<M, 1, 4, NF, 1, false, false>(FP, io, (int)blockIdx.x, PartIO{});
}
template <class M, int NF>
__global__ void __launch_bounds__(kTileMax) k_tile_fused_flux(FusedParams FP, TileIO io) {
    pdl_trigger();
    fused_tile<M, 1, 4, NF, 2, false, false>(FP, io, (int)blockIdx.x, PartIO{});
}

template <class M, int NF>
__global__ void __launch_bounds__(kTileMax) k_tile_fused_dt(FusedParams FP, TileIO io) {
    pdl_trigger();
    fused_tile<M, 1, 4, NF, 3, false, true>(FP, io, (int)blockIdx.x, PartIO{});
    // the step's first kernel: the work-list tile counters of its stage
    // kernels start at zero (every kernel that used them has completed)
    if (io.work_reset != nullptr && blockIdx.x == 0 && threadIdx.x < kWorkSlots) io.work_reset[threadIdx.x] = 0;
}

// A decomposition part's launches, one CTA per tile.  MODE 1: tiles
// [pio.t0, pio.t0 + grid) (the band and interior launches); MODE 2: the halo
// exchange inside the launch (pio.remote).
template <class M, int FLUX, int NF, int MODE>
__global__ void __launch_bounds__(kTileMax) k_tile_fused_part(FusedParams FP, TileIO io, PartIO pio) {
    pdl_trigger();
    fused_tile<M, FLUX, 4, NF, 0, MODE == 2, true>(FP, io, (MODE == 1 ? pio.t0 : 0) + (int)blockIdx.x, pio);
}

// Work-list schedule: as many CTAs as fit on the device at once, each taking
// the next tile from the launch's counter (reset by the step's dt kernel)
// until none is left, so no CTA waits at a tail of unevenly sized tiles.
// The counter is read only after the dependency wait.
template <class M, int FLUX, int NF>
__global__ void __launch_bounds__(kTileMax) k_tile_fused_work(FusedParams FP, TileIO io, int n_tiles) {
    pdl_trigger();
    pdl_wait();
    __shared__ int s_t;
    for (;;) {
        if (threadIdx.x == 0) s_t = atomicAdd(io.work, 1);
        __syncthreads();
        const int t = s_t;
        if (t >= n_tiles) return;
        if (!fused_tile<M, FLUX, 4, NF, 0, false, true>(FP, io, t, PartIO{})) return;
        __syncthreads();  // every thread is done with this tile's shared memory (and s_t)
    }
}

template <class M>
struct FusedLaunch {
    // lays out the tiles' shared memory (FP.L); the bytes of the largest launch
    // but the run kernel's
    static size_t smem(FusedParams& FP) {
        FP.L = fused_smem<M>(FP.max_slots, FP.max_grad, FP.max_flux, FP.max_ghost, FP.T, FP.P.flux == 5);
        return (size_t)std::max(FP.L.total, FP.L.total_grad);
    }
    static cudaError_t prepare(FusedParams& FP) {
        static std::mutex mu;
        std::lock_guard<std::mutex> lock(mu);
        cudaError_t e = cudaSuccess;
        const size_t bytes = smem(FP);
        auto set = [&](const void* fn) {
            // only ever raised: a solver created earlier may launch with more
            cudaFuncAttributes fa{};
            if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, fn);
            if (e == cudaSuccess && (size_t)fa.maxDynamicSharedSizeBytes < bytes)
                e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
            if (e == cudaSuccess)
                e = cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout,
                                         (int)cudaSharedmemCarveoutMaxShared);
        };
        auto all = [&](auto f, auto n) {
            constexpr int F = decltype(f)::value, NF = decltype(n)::value;
            for (const void* fn :
                 {(const void*)k_tile_fused<M, F, 4, NF>, (const void*)k_tile_fused_part<M, F, NF, 1>,
                  (const void*)k_tile_fused_part<M, F, NF, 2>, (const void*)k_tile_fused_work<M, F, NF>})
                set(fn);
            if constexpr (M::exact) set((const void*)k_tile_fused<M, F, 1, NF>);
            set((const void*)k_tile_fused_dt<M, NF>);
            if constexpr (!M::exact && sizeof(typename M::S) == 8)
                for (const void* fn : {(const void*)k_tile_fused_grad<M, NF>, (const void*)k_tile_fused_flux<M, NF>})
                    set(fn);
        };
        using One = std::integral_constant<int, 1>;
        using Three = std::integral_constant<int, 3>;
        using Four = std::integral_constant<int, 4>;
        if (FP.nf == 3) all(One{}, Three{});
        else all(One{}, Four{});
        if constexpr (M::exact) {
            using Two = std::integral_constant<int, 2>;
            if (FP.nf == 3) all(Two{}, Three{});
            else all(Two{}, Four{});
        }
        return e;
    }
    // CTAs of the work-list schedule: the device's resident capacity
    static int work_grid(FusedParams& FP, int n_tiles) {
        int dev = 0, sms = 0, nb = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(
            &nb, FP.nf == 3 ? k_tile_fused_work<M, 1, 3> : k_tile_fused_work<M, 1, 4>, FP.T, smem(FP));
        return std::max(1, std::min(n_tiles, sms * std::max(nb, 1)));
    }
    template <class... A, class... B>
    static void go(void (*k)(A...), int grid, int threads, size_t sm, cudaStream_t st, bool pdl, const B&... args) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)grid);
        cfg.blockDim = dim3((unsigned)threads);
        cfg.dynamicSmemBytes = sm;
        cfg.stream = st;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = at;
        cfg.numAttrs = pdl ? 1 : 0;
        cudaLaunchKernelEx(&cfg, k, args...);
    }
    template <int F, int NF>
    static void stage_f(const FusedParams& FP, const TileIO& io, cudaStream_t st, bool pdl, int n_tiles, int grid,
                        const PartIO* part) {
        const size_t sm = (size_t)FP.L.total;
        const int tp = FP.lanes == 1 ? FP.threads : FP.T;  // a part's launch: one lane per cell
        if (io.work) go(k_tile_fused_work<M, F, NF>, grid, FP.T, sm, st, pdl, FP, io, n_tiles);
        else if (part && part->remote) go(k_tile_fused_part<M, F, NF, 2>, n_tiles, tp, sm, st, pdl, FP, io, *part);
        else if (part) go(k_tile_fused_part<M, F, NF, 1>, n_tiles, tp, sm, st, pdl, FP, io, *part);
        else if (M::exact && FP.lanes == 4) go(k_tile_fused<M, F, M::exact ? 1 : 4, NF>, n_tiles, FP.threads, sm, st, pdl, FP, io);
        else go(k_tile_fused<M, F, 4, NF>, n_tiles, FP.threads, sm, st, pdl, FP, io);
    }
    // io.work != nullptr: the work-list schedule on `grid` CTAs
    // part: a decomposition part's launch (its tile offset, in-launch exchange)
    static void stage(const FusedParams& FP, const TileIO& io, cudaStream_t st, bool pdl, int n_tiles, int grid,
                      const PartIO* part = nullptr) {
        if constexpr (M::exact) {
            if (FP.P.flux == 2) {
                if (FP.nf == 3) stage_f<2, 3>(FP, io, st, pdl, n_tiles, grid, part);
                else stage_f<2, 4>(FP, io, st, pdl, n_tiles, grid, part);
                return;
            }
        }
        if (FP.nf == 3) stage_f<1, 3>(FP, io, st, pdl, n_tiles, grid, part);
        else stage_f<1, 4>(FP, io, st, pdl, n_tiles, grid, part);
    }
    // the time step (phase 3); FP64: the split layout's two kernels
    // (phase 1: gradients; phase 2: the rest)
    template <int NF>
    static void split_f(const FusedParams& FP, const TileIO& io, cudaStream_t st, bool pdl, int n_tiles, int phase) {
        const FusedSmem& L = FP.L;
        if (phase == 3) go(k_tile_fused_dt<M, NF>, n_tiles, FP.T, L.total_grad, st, pdl, FP, io);
        else if constexpr (M::exact || sizeof(typename M::S) == 4) return;
        else if (phase == 2) go(k_tile_fused_flux<M, NF>, n_tiles, FP.T, L.total, st, pdl, FP, io);
        else go(k_tile_fused_grad<M, NF>, n_tiles, FP.T, L.total_grad, st, pdl, FP, io);
    }
    static void split(const FusedParams& FP, const TileIO& io, cudaStream_t st, bool pdl, int n_tiles, int phase) {
        if (FP.nf == 3) split_f<3>(FP, io, st, pdl, n_tiles, phase);
        else split_f<4>(FP, io, st, pdl, n_tiles, phase);
    }
};

namespace tile {
cudaError_t prepare_fused(int precision, FusedParams& FP);
size_t smem_fused(int precision, FusedParams& FP);
int work_grid_fused(int precision, FusedParams& FP, int n_tiles);
void launch_fused(int precision, const FusedParams& FP, const TileIO& io, cudaStream_t st, bool pdl, int n_tiles,
                  int grid, const PartIO* part = nullptr);
// the time step and FP64's split kernels over the fused kernel's tiles (FusedLaunch::split)
void launch_fused_split(int precision, const FusedParams& FP, const TileIO& io, cudaStream_t st, bool pdl, int n_tiles,
                        int phase);
}  // namespace tile

}  // namespace fvgpu
