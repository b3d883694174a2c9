// Persistent run kernel of the Roe kinds and, in FP64, the Navier-Stokes kind: all the time steps of a launch in one
// cooperative kernel with one resident CTA per tile, for meshes whose tiles fit
// the device at once.
//
// On such meshes a kernel of a step takes 5 to 30 us, and most of that is not
// work: launch and drain, constant tile data fetched again, and every phase of
// a tile waiting out its own latency with a few warps.  Here a CTA keeps its
// tile's geometry in registers and shared memory for the whole run, a stage
// starts at a grid barrier, and what has no place in the chain is taken off it:
// the time step is computed from the states staged for the first stage, its
// global minimum is awaited only before that stage's update, and the residual
// norms, the time and the stop criteria of a step (explicit.cpp:717-726,
// 752-800) are evaluated beside the gradients of the next one's first stage,
// by every CTA from the same values in the same order, so that all take the
// same decision.  A first stage that turns out not to run has written nothing
// that is read later.
//
// Every wait is bounded: a CTA that gives up records the failure, the others
// see it at their next wait, and the kernel ends.
#pragma once
#include "fv_fused.cuh"
#include "fv_launch.h"

namespace fvgpu {

constexpr int kMaxStages = 16;
struct PersistIO {
    double* qbase[2];
    void* sbase[2];
    void* tmp[2];
    double* dt;
    // residual partial sums, by the step modulo 2: with one stage a CTA may
    // store its next ones while another still reads these (between the two lies
    // only the time step's barrier, which a CTA joins before it reads)
    double* partials;              // [2][n_tiles][4] (stencils: [2][CTAs])
    unsigned long long* keys;      // [3][n_cases][kDtSlots], by the step modulo 3
    Ctrl* ctrl;
    const RunLimits* limits;
    PrintRec* hist;
    int hist_cap;
    unsigned* bar;                 // arrivals at the grid barrier, zero at launch
    int n_tiles, n_cases, f32;
    int max_steps;                 // steps of this launch at most
    int polls;                     // polls of a wait at most
    int ns;
    double alpha[kMaxStages];
};

// Grid barrier: arrive() publishes the CTA's writes, wait() blocks until every
// CTA has arrived as often as this one.
struct GridSync {
    unsigned* bar;
    int* err;
    int most;  // polls of a wait
    unsigned target = 0;
    __device__ __forceinline__ void arrive() {
        __syncthreads();
        target += gridDim.x;
        if (threadIdx.x == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
    }
    __device__ __forceinline__ bool wait() {
        __shared__ int s_ok;
        if (threadIdx.x == 0) {
            int ok = 1, polls = 0;
            for (;;) {
                unsigned v;
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
                if ((int)(v - target) >= 0) break;
                if (++polls > most || ((polls & 1023) == 0 && *(volatile int*)err)) {
                    atomicExch(err, 1);
                    ok = 0;
                    break;
                }
            }
            s_ok = ok;
        }
        __syncthreads();
        return s_ok != 0;
    }
};

struct RunState {
    unsigned long long step;
    double time;
    double R[4], R0[4], Rraw[4];
    int active, need_R, n_hist;
};
__device__ __forceinline__ bool run_divides(unsigned long long step, unsigned long long every) {
    if (every == 1) return true;
    if (((step | every) >> 32) == 0) return (uint32_t)step % (uint32_t)every == 0;
    return step % every == 0;
}
// Stop criteria of the step about to start (explicit.cpp:717-726).
template <int V = 4>
__device__ __forceinline__ void run_step_start(RunState& c, const RunLimits& L) {
    double Rmax = 1.0;
    if (c.step > 0) {
        Rmax = 0.0;
#pragma unroll
        for (int k = 0; k < V; ++k) Rmax = exact::dmax(c.R[k], Rmax);
    }
    const bool stop = c.step >= L.max_step || c.time >= L.max_time || Rmax < L.tolerance;
    c.active = !stop;
    c.need_R = !stop && (c.step == 0 || L.tolerance > 1.01e-16 || run_divides(c.step, L.print_interval));
}
// The end of a step (one warp): residual norms from the tiles' partial sums
// (strided by lane, then a butterfly), time (dt: the step's), print record,
// the next step's stop criteria.  partials: [n][V], V = 4 or 1.
template <int V = 4>
__device__ __forceinline__ void run_step_end(const PersistIO& D, RunState& c, const RunLimits& lim, double dt,
                                             const double* partials, int n) {
    const int lane = threadIdx.x & 31;
    const bool need_R = c.need_R != 0;
    const unsigned long long step = c.step;
    double s[4] = {0, 0, 0, 0};
    if (need_R) {
        for (int b = lane; b < n; b += 32) {
            if constexpr (V == 1) {
                s[0] += __ldcg(partials + b);
            } else {
                const double2* p = reinterpret_cast<const double2*>(partials + (size_t)b * 4);
                const double2 x = __ldcg(p), y = __ldcg(p + 1);
                s[0] += x.x; s[1] += x.y; s[2] += y.x; s[3] += y.y;
            }
        }
#pragma unroll
        for (int k = 0; k < V; ++k)
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) s[k] += __shfl_xor_sync(0xffffffffu, s[k], o);
        if (lane < V) {
            const double v = lane == 0 ? s[0] : lane == 1 ? s[1] : lane == 2 ? s[2] : s[3];
            const double r = sqrt(v);
            c.Rraw[lane] = r;
            if (step == 0) c.R0[lane] = r;
            c.R[lane] = step == 0 ? r : r / c.R0[lane];
        }
        __syncwarp();
    }
    if (lane == 0) {
        if ((step == 0 || run_divides(step, lim.print_interval)) && c.n_hist < D.hist_cap) {
            if (blockIdx.x == 0) {
                PrintRec& r = D.hist[c.n_hist];
                r.step = step;
                r.time = c.time;
#pragma unroll
                for (int k = 0; k < V; ++k) r.R[k] = step == 0 ? 1.0 : c.R[k];
            }
            ++c.n_hist;
        }
        c.time += dt;
        c.step = step + 1;
        run_step_start<V>(c, lim);
    }
    __syncwarp();
}

// min_dt (explicit.cpp:555-564) from a case's keys, one warp: a NaN in dt[0] wins
__device__ __forceinline__ double run_min_dt(const unsigned long long* keys, const double* dt, int cell0) {
    const int lane = threadIdx.x & 31;
    const double d0 = __ldcg(dt + cell0);
    unsigned long long k = kmin_(__ldcg(keys + lane), __ldcg(keys + lane + 32));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) k = kmin_(k, __shfl_xor_sync(0xffffffffu, k, o));
    return (d0 != d0) ? d0 : tkey_inv(k);
}

// le times the Navier-Stokes flux of flux edge el (examples/flatPlate/main.cpp:
// 126-225): the Roe flux of the face states minus the viscous terms of the
// corrected face gradient (gradient_for_diffusion, explicit.cpp:70-109).
template <class S, int NF>
__device__ __forceinline__ void run_viscous_flux(const FusedParams& FP, const unsigned char* smem_raw, const S* EG,
                                                 int el, const S* qL, const S* qR, const S* e, S* f) {
    using P4 = Planes<S, 4>;
    const FusedSmem& L = FP.L;
    const uint32_t ij = edge_slots(EG[4 * el + 3]);
    const int li = (int)(ij & 0xFFFF), lj = (int)(ij >> 16);
    const S* E2 = reinterpret_cast<const S*>(smem_raw + L.e2) + 4 * el;
    const S t0 = E2[0], t1 = E2[1], rl = E2[2];
    S gxi[4], gyi[4], gxj[4], gyj[4], qi[4], qj[4], gx[4], gy[4];
    P4::get(reinterpret_cast<const uint4*>(smem_raw + L.gx), L.lt, li, 0, gxi);
    P4::get(reinterpret_cast<const uint4*>(smem_raw + L.gx), L.lt, lj, 0, gxj);
    P4::get(reinterpret_cast<const uint4*>(smem_raw + L.gy), L.lt, li, 0, gyi);
    P4::get(reinterpret_cast<const uint4*>(smem_raw + L.gy), L.lt, lj, 0, gyj);
    P4::get(reinterpret_cast<const uint4*>(smem_raw + L.q), L.ls, li, 0, qi);
    P4::get(reinterpret_cast<const uint4*>(smem_raw + L.q), L.ls, lj, 0, qj);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const S bx = S(0.5) * (gxi[k] + gxj[k]), by = S(0.5) * (gyi[k] + gyj[k]);
        const S corr = bx * t0 + by * t1 - (qi[k] - qj[k]) * rl;
        gx[k] = bx - corr * t0;
        gy[k] = by - corr * t1;
    }
    fast::roe<S>((S)FP.P.gamma, f, qL, qR, e[0], e[1]);
    fast::ns_viscous<S>(FP.P, f, qL, qR, gx, gy, e[0], e[1]);
#pragma unroll
    for (int k = 0; k < 4; ++k) f[k] *= e[2];
}

// The time loop of tile blockIdx.x.  NV, NF: as in fused_tile; O2: second order
// (two-ring tiles), else the face states are the cell values (one ring).  FLUX 5
// (Navier-Stokes, O2; fast policies): the face gradients of its viscous terms
// come from the same gradients, with or without MUSCL face states (order2).
template <class M, int FLUX, int NV, int NF, bool O2>
__device__ __forceinline__ void run_tile(const FusedParams& FP, const PersistIO& D) {
    using S = typename M::S;
    using P4 = Planes<S, 4>;
    constexpr int V = 4, LP = V / NV, NU = (int)sizeof(S) / 4;
    constexpr bool VISC = FLUX == 5;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ RunState c;
    __shared__ double s_dt, s_time;
    const Params& P = FP.P;
    const int T = FP.T, t = (int)blockIdx.x;
    const int4 ia = FP.info[2 * t], ib = FP.info[2 * t + 1];
    const int slot_off = ia.x, halo_off = ia.y, flux_off = ia.z, n_flux = ia.w, n_ghost = ib.z >> 16;
    const int n1 = ib.x, nh = O2 ? ib.x + ib.y : ib.x, nown = ib.z & 0xFFFF;
    const int c0 = t * T, G = T + n1;
    const FusedSmem& L = FP.L;
    uint4* Q = reinterpret_cast<uint4*>(smem_raw + L.q);
    uint4* FS = reinterpret_cast<uint4*>(smem_raw + L.fs);
    double* QB = reinterpret_cast<double*>(smem_raw + L.qb);
    const S* EG = reinterpret_cast<const S*>(smem_raw + L.eg);
    double* RA = reinterpret_cast<double*>(smem_raw + L.ria);
    const int l = threadIdx.x, warp = l >> 5, nw = blockDim.x >> 5;
    const int r0 = l / LP, rstep = blockDim.x / LP, v0 = (l % LP) * NV, uc = r0;
    // ---- the tile's constant data, once
    SlotGeo<M, NF> geo;
    uint32_t own[NF];
    if constexpr (O2) {
        geo.load(FP, slot_off, G, min(r0, G - 1));
#pragma unroll
        for (int f = 0; f < NF; ++f) own[f] = geo.w[f];
    } else {
        const uint4 h = __ldg(FP.hd + (slot_off + min(r0, G - 1)));
        own[0] = h.x; own[1] = h.y; own[2] = h.z;
        if constexpr (NF == 4) own[NF - 1] = h.w;
    }
    // the faces of owned cell l (the time step has one thread per cell)
    uint32_t dtw[NF];
    {
        const uint4 h = __ldg(FP.hd + (slot_off + min(l, G - 1)));
        dtw[0] = h.x; dtw[1] = h.y; dtw[2] = h.z;
        if constexpr (NF == 4) dtw[NF - 1] = h.w;
    }
    const int h0 = l < nh ? __ldg(FP.halo + halo_off + l) : 0;
    const S area = l < nown ? __ldg((const S*)FP.area + c0 + l) : S(1);
    {
        const uint4* src = reinterpret_cast<const uint4*>((const S*)FP.eg + 4 * (size_t)flux_off);
        uint4* dst = reinterpret_cast<uint4*>(smem_raw + L.eg);
        for (int i = l; i < NU * n_flux; i += blockDim.x) cpa16(dst + i, src + i);
        if (l < nown) cpa8(RA + l, FP.ria + c0 + l);
        const uint4* gsrc = reinterpret_cast<const uint4*>((const S*)FP.gd + 4 * (size_t)ib.w);
        for (int i = l; i < NU * n_ghost; i += blockDim.x) cpa16(reinterpret_cast<uint4*>(smem_raw + L.gd) + i, gsrc + i);
        for (int i = l; i < n_ghost; i += blockDim.x) cpa8(smem_raw + L.gl + 8 * i, FP.gl + ib.w + i);
        if constexpr (VISC) {
            const uint4* esrc = reinterpret_cast<const uint4*>((const S*)FP.e2 + 4 * (size_t)flux_off);
            for (int i = l; i < NU * n_flux; i += blockDim.x) cpa16(reinterpret_cast<uint4*>(smem_raw + L.e2) + i, esrc + i);
            for (int i = l; i < G; i += blockDim.x)
                cpa<(int)sizeof(S)>((S*)(smem_raw + L.ar) + i, (const S*)FP.ar + slot_off + i);
            // boundary ghosts have no gradient
            for (int i = l; i < NU * L.lt; i += blockDim.x)
                reinterpret_cast<uint4*>(smem_raw + L.gx)[i] = reinterpret_cast<uint4*>(smem_raw + L.gy)[i] = make_uint4(0, 0, 0, 0);
        }
        cpa_wait();
    }
    const int tc = (P.global_dt && P.n_cases > 1) ? P.tile_case[t] : 0;
    const int cell0 = (P.n_cases > 1 && tc >= 0) ? P.case_cell0[tc] : P.cell0;
    const int nkeys = D.n_cases * kDtSlots;
    const RunLimits lim = *D.limits;
    if (l == 0) {
        c.step = D.ctrl->step;
        c.time = D.ctrl->time;
#pragma unroll
        for (int k = 0; k < 4; ++k) { c.R[k] = D.ctrl->R[k]; c.R0[k] = D.ctrl->R0[k]; c.Rraw[k] = D.ctrl->Rraw[k]; }
        c.n_hist = 0;
        run_step_start(c, lim);
    }
    GridSync sync{D.bar, &D.ctrl->failed, D.polls};
    sync.arrive();
    TileIO io{};
    io.dt = D.dt;
    io.ctrl = D.ctrl;
    bool pending = false;  // a step has ended whose norms and time are not evaluated yet
    const double* part = nullptr;  // its partial sums
    int n = 0;
    for (bool go = c.active != 0; go && n < D.max_steps; ++n) {
        unsigned long long* keys = D.keys + (size_t)(n % 3) * nkeys;
        const int b = D.ns == 1 ? (n & 1) : 0;  // a single stage alternates the base buffers
        double* part_out = D.partials + (size_t)(n & 1) * D.n_tiles * V;
        io.dtkeys = keys;
        io.q_base = D.qbase[b];
        const void* in = D.sbase[b];
        double dtc = 0.;
        for (int k = 0; k < D.ns; ++k) {
            const bool last = k == D.ns - 1;
            void* out_s;
            if (D.ns == 1) {
                out_s = D.sbase[1 - b];
                io.q_out = D.qbase[1 - b];
            } else if (last) {
                out_s = D.sbase[b];
                io.q_out = D.qbase[b];
            } else {
                out_s = D.tmp[k & 1];
                io.q_out = D.f32 ? nullptr : (double*)out_s;
            }
            io.s_out = D.f32 ? out_s : nullptr;
            io.write_f64 = last ? 1 : 0;
            io.partials = last ? part_out : nullptr;
            io.q_stage = in;
            io.alpha = D.alpha[k];
            // ---- the stage's input is complete
            if (!sync.wait()) return;
            const uint4* gq = reinterpret_cast<const uint4*>((const S*)in + 4 * (size_t)c0);
            for (int i = l; i < NU * nown; i += blockDim.x)
                cpa16(NU == 1 ? Q + i : Q + (i & 1) * L.ls + (i >> 1), gq + i);
            for (int h = l; h < nh; h += blockDim.x) {
                const int g = h == l ? h0 : __ldg(FP.halo + halo_off + h);
                P4::stage(Q, L.ls, T + h, (const S*)in + 4 * (size_t)g);
            }
            if (k == 0) {
                const uint4* gb = reinterpret_cast<const uint4*>(io.q_base + 4 * (size_t)c0);
                for (int i = l; i < 2 * nown; i += blockDim.x) cpa16(QB + 2 * i, gb + i);
            }
            cpa_wait();
            __syncthreads();
            if (k == 0) {
                // ---- the step's time step, from the same states
                for (int r = l; r < G; r += blockDim.x) {
                    if (r >= nown && r < T) continue;
                    S q[V], w[V];
                    P4::get(Q, L.ls, r, 0, q);
                    fused_speeds<M>(P.gamma, q, w);
                    P4::put(FS, FP.max_grad, r, 0, w);
                }
                __syncthreads();
                unsigned long long kmin = ~0ull;
                double di = 0.;
                auto edge = [&](int el, S* e) { e[0] = EG[4 * el]; e[1] = EG[4 * el + 1]; e[2] = EG[4 * el + 2]; };
                if (l < nown)
                    kmin = fused_cell_dt<M, NF, VISC>(FP, io, dtw, FS, l, c0 + l, halo_off, area, edge, di,
                                                      reinterpret_cast<const S*>(smem_raw + L.ar));
                tile_dt_reduce(P, T, io, t, l, nown, kmin);
                sync.arrive();
                if (!P.global_dt && uc < nown) dtc = __ldcg(D.dt + c0 + uc);
                // the next step's keys: its set was last read two steps ago
                if (blockIdx.x == 0)
                    for (int i = l; i < nkeys; i += blockDim.x) D.keys[(size_t)((n + 1) % 3) * nkeys + i] = ~0ull;
                if (pending && warp == nw - 1) run_step_end(D, c, lim, s_time, part, D.n_tiles);
            }
            // ---- face states
            if constexpr (O2) {
                if (r0 < G && word_nbr(geo.w[0]) != 0xFFFF)
                    fused_slot<M, NV, NF, 0, VISC>(FP, io, smem_raw, geo, r0, v0, c0, halo_off, flux_off);
                for (int r = r0 + rstep; r < G; r += rstep) {
                    SlotGeo<M, NF> g2;
                    g2.load(FP, slot_off, G, r);
                    if (word_nbr(g2.w[0]) != 0xFFFF)
                        fused_slot<M, NV, NF, 0, VISC>(FP, io, smem_raw, g2, r, v0, c0, halo_off, flux_off);
                }
                __syncthreads();
            } else if (k == 0) {
                __syncthreads();
            }
            if (k == 0) {
                pending = false;
                if (!c.active) { go = false; break; }
            }
            // ---- fluxes
            for (int el = l; el < n_flux; el += blockDim.x) {
                S e[4], qL[V], qR[V], f[V];
                e[0] = EG[4 * el]; e[1] = EG[4 * el + 1]; e[2] = EG[4 * el + 2];
                if constexpr (O2) {
                    P4::get(FS, L.lf, el, 0, qL);
                    P4::get(FS, L.lf, el + FP.max_flux, 0, qR);
                } else {
                    const uint32_t ij = edge_slots(EG[4 * el + 3]);
                    P4::get(Q, L.ls, (int)(ij & 0xFFFF), 0, qL);
                    P4::get(Q, L.ls, (int)(ij >> 16), 0, qR);
                }
                if constexpr (M::exact) {
                    exact::flux_dev<FLUX>(P.gamma, f, qL, qR, e[0], e[1]);
#pragma unroll
                    for (int i = 0; i < V; ++i) f[i] *= e[2];
                } else if constexpr (VISC) {
                    run_viscous_flux<S, NF>(FP, smem_raw, EG, el, qL, qR, e, f);
                } else {
                    fast::flux_le<FLUX, O2>((S)P.gamma, f, qL, qR, e[0], e[1], e[2]);
                }
#pragma unroll
                for (int i = 0; i < V; ++i) qL[i] = -f[i];
                P4::put(FS, L.lf, el, 0, qL);
                P4::put(FS, L.lf, el + FP.max_flux, 0, f);
            }
            if (k == 0) {
                // ---- every tile's time step is known
                if (!sync.wait()) return;
                if (P.global_dt) {
                    if (warp == 0 && tc >= 0) {
                        const double d = run_min_dt(keys + (size_t)tc * kDtSlots, D.dt, cell0);
                        if (l == 0) s_dt = d;
                    }
                    if (warp == 1) {
                        const double d = run_min_dt(keys, D.dt, P.cell0);
                        if (l == 32) s_time = d;
                    }
                } else if (l == 0) {
                    s_time = __ldcg(D.dt + P.cell0);
                }
                if (P.n_cases > 1 && blockIdx.x == 0) {
                    // each case of a batch keeps its own time: time += dt[0] of that case
                    for (int i = l; i < P.n_cases; i += blockDim.x) {
                        const double e0 = __ldcg(D.dt + P.case_cell0[i]);
                        double e = e0;
                        if (P.global_dt && e0 == e0) {
                            unsigned long long key = ~0ull;
                            for (int j = 0; j < kDtSlots; ++j) key = kmin_(key, __ldcg(keys + (size_t)i * kDtSlots + j));
                            e = tkey_inv(key);
                        }
                        P.case_time[i] += e;
                    }
                }
            }
            __syncthreads();
            // ---- update
            double res[NV];
#pragma unroll
            for (int i = 0; i < NV; ++i) res[i] = 0.;
            if (uc < nown)
                fused_update<M, NV, NF, false>(FP, io, smem_raw, own, uc, v0, c0, tc, dtc, s_dt, n_ghost != 0, PartIO{}, res);
            if (n_ghost != 0) {
                __syncthreads();
                fused_ghosts<M, false, O2, VISC>(FP, io, smem_raw, reinterpret_cast<const int2*>(smem_raw + L.gl),
                                           reinterpret_cast<const S*>(smem_raw + L.gd), n_ghost, PartIO{});
            }
            if (last) fused_partials<NV>(io, smem_raw + L.fs, t, v0, res);
            sync.arrive();
            in = out_s;
        }
        if (go) { pending = true; part = part_out; }
    }
    if (pending) {  // the launch's last step
        if (!sync.wait()) return;
        if (warp == nw - 1) run_step_end(D, c, lim, s_time, part, D.n_tiles);
        __syncthreads();
    }
    if (blockIdx.x == 0 && l == 0) {
        Ctrl* o = D.ctrl;
        o->step = c.step;
        o->time = c.time;
#pragma unroll
        for (int k = 0; k < 4; ++k) { o->R[k] = c.R[k]; o->R0[k] = c.R0[k]; o->Rraw[k] = c.Rraw[k]; }
        o->active = c.active;
        o->need_R = c.need_R;
        o->n_hist = c.n_hist;
    }
}

// THREADS per CTA and CTAs per SM of the register budget
template <class M, int FLUX, int NV, int NF, bool O2, int THREADS, int BLOCKS>
__global__ void __launch_bounds__(THREADS, BLOCKS)
    k_run(const __grid_constant__ FusedParams FP, const __grid_constant__ PersistIO D) {
    run_tile<M, FLUX, NV, NF, O2>(FP, D);
}

// A candidate run kernel of a solver, in order of preference.
struct RunKernel {
    const void* fn = nullptr;
    int threads = 0;
};
constexpr int kRunKernels = 4;
template <class M>
struct RunLaunch {
    // The candidates from the most threads and registers per tile down: while
    // the device has room, more threads shorten a tile's chain (one pass over
    // the gradient slots and the flux edges instead of two).  Measured, us per
    // step (k[0] | k[1] | k[2] | k[3] | separate kernels; -: no candidate or no
    // room): forward step 10,206 cells FP64_EXACT 46.5 | 47.2 | 54.9 | 85.7 |
    // 57.9, FP64 - | 26.8 | 27.4 | 36.3 | 43.7, FP32 - | 21.5 | 26.4 | 32.9 |
    // 35.9; 98,784 cells FP32 - | - | - | 54.3 | 61.7; NACA 65,536 cells FP64
    // - | - | - | 49.7 | 57.9; Sod tube (first order) 32,000 cells FP64 - | 8.8 |
    // 8.9 | 9.1 | 16.2; flat plate (Navier-Stokes) 13,200 cells FP64 - | 40.0 |
    // 43.1 | 55.5 | 99.6 (two kernels a stage, whose limiter, Green-Gauss and
    // viscous time-step divisions the run kernel's form does not have).
    template <int F, int NF, bool O2>
    static void list(const FusedParams& FP, RunKernel* k) {
        constexpr int low = sizeof(typename M::S) == 4 ? 4 : 2, high = O2 ? low / 2 : low;
        const int two = std::min(2 * FP.T, kTileMax);
        if constexpr (M::exact && O2) k[0] = {(const void*)k_run<M, F, 2, NF, O2, kFusedThreads, 1>, std::min(4 * FP.T, kFusedThreads)};
        k[1] = {(const void*)k_run<M, F, 4, NF, O2, kTileMax, high>, two};
        k[2] = {(const void*)k_run<M, F, 4, NF, O2, kTileMax, low>, two};
        k[3] = {(const void*)k_run<M, F, 4, NF, O2, kTileMax, low>, FP.T};
    }
    static void kernels(const FusedParams& FP, RunKernel* k) {
        const bool o2 = FP.P.order2 != 0;
        auto pick = [&](auto f) {
            constexpr int F = decltype(f)::value;
            if (o2) {
                if (FP.nf == 3) list<F, 3, true>(FP, k);
                else list<F, 4, true>(FP, k);
            } else if constexpr (sizeof(typename M::S) == 8) {  // (FP32: separate kernels)
                if (FP.nf == 3) list<F, 3, false>(FP, k);
                else list<F, 4, false>(FP, k);
            }
        };
        if constexpr (M::exact) {
            if (FP.P.flux == 2) { pick(std::integral_constant<int, 2>{}); return; }
        }
        if constexpr (sizeof(typename M::S) == 8 && !M::exact) {
            if (FP.P.flux == 5) {
                if (FP.nf == 3) list<5, 3, true>(FP, k);
                else list<5, 4, true>(FP, k);
                return;
            }
        }
        pick(std::integral_constant<int, 1>{});  // the fast policies' two Roe kinds are one function
    }
};

namespace tile {
// The candidate run kernels (kRunKernels entries, fn null where there is none).
void run_kernels(int precision, const FusedParams& FP, RunKernel* k);
}  // namespace tile

}  // namespace fvgpu
