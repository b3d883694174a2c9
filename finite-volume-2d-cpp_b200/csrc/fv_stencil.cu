// Stage and run kernels of the diffusion kind over its stencils (fv_stencil.h).
//
// One pass per stage instead of a gradient kernel and a flux kernel: a tile
// stages the states of its two rings, and a thread sums its cell's at most
// NF^2 terms.  Nothing but states passes between stages, so the step's cost is
// the coefficients (in registers for a whole run, where the tiles fit the
// device at once) and the latency of a grid barrier or of a launch.  Measured,
// us per RK5 step, FP64 | FP32, two kernels a stage -> here: 512 cells 28 -> 13 |
// 26 -> 13, 24,000 cells 33 -> 14 | 30 -> 14, 125,000 cells 58 -> 19 | 54 -> 17,
// 145,800 cells 61 -> 20 | 52 -> 18; a launch per stage: 168,200 cells 74 -> 25 |
// 65 -> 23, 720,000 cells 271 -> 72 | 160 -> 64.
#include "fv_persist.cuh"
#include "fv_stencil.h"

namespace fvgpu {
namespace {

// The stencil of one cell: two slots to a word.
template <class S, int NF>
struct Stencil {
    static constexpr int K = NF * NF;
    double a[K];
    uint32_t w[(K + 1) / 2];
    __device__ __forceinline__ void load(const StencilParams& SP, int c) {
        const size_t N = (size_t)SP.P.n_real;
#pragma unroll
        for (int k = 0; k < (K + 1) / 2; ++k) w[k] = 0;
#pragma unroll
        for (int k = 0; k < K; ++k) {
            a[k] = __ldg(SP.coef + k * N + c);
            w[k / 2] |= (uint32_t)__ldg(SP.slot + k * N + c) << (16 * (k & 1));
        }
    }
    __device__ __forceinline__ int slot(int k) const { return (int)(w[k / 2] >> (16 * (k & 1)) & 0x7FFF); }
    __device__ __forceinline__ bool ghost(int f) const { return w[f / 2] >> (16 * (f & 1)) & 0x8000; }
    __device__ __forceinline__ bool any_ghost() const {
        uint32_t any = 0;
#pragma unroll
        for (int k = 0; k < (K + 1) / 2; ++k) any |= w[k];
        return any & 0x80008000u;
    }
    // the time derivative: FP64 sums of the differences from the cell's state
    __device__ __forceinline__ double qt(const S* q, int l) const {
        const double qc = q[l];
        double s[2] = {0., 0.};
#pragma unroll
        for (int k = 0; k < K; ++k) s[k & 1] = fma(a[k], (double)q[slot(k)] - qc, s[k & 1]);
        return s[0] + s[1];
    }
    // the cell's ghosts (copy boundaries) take its new state
    template <class F>
    __device__ __forceinline__ void ghosts(const StencilParams& SP, int halo_off, F write) const {
        if (!any_ghost()) return;
#pragma unroll
        for (int f = 0; f < NF; ++f)
            if (ghost(f)) write(__ldg(SP.halo + halo_off + slot(f) - SP.T));
    }
};

// sum over the block of r, valid in thread 0
__device__ __forceinline__ double block_sum(double r) {
    __shared__ double red[32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = r;
    __syncthreads();
    r = 0.;
    if (threadIdx.x == 0)
        for (int w = 0; w < (int)blockDim.x >> 5; ++w) r += red[w];
    return r;
}

// One stage of every tile.  dtkeys (a step's first stage): the step end's view of
// the constant time step, one value per case; a time-step kernel over all cells
// wrote one per cell (21 us of a step; 1,002,528 cells FP64: a step 170 us with
// it, 139 without).
template <class S, int NF>
__global__ void __launch_bounds__(kTileMax) k_stencil_stage(const __grid_constant__ StencilParams SP, TileIO io) {
    pdl_trigger();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    S* q = reinterpret_cast<S*>(smem_raw);
    const Params& P = SP.P;
    const int l = threadIdx.x, t = blockIdx.x, c = t * SP.T + l;
    const int4 inf = __ldg(SP.info + t);
    const bool on = l < inf.z;
    Stencil<S, NF> st;
    double A = 0.;
    if (on) {
        st.load(SP, c);
        A = __ldg(SP.area + c);
    }
    int h0 = l < inf.y ? __ldg(SP.halo + inf.x + l) : 0;
    pdl_wait();
    const bool inactive = t_inactive(io.ctrl);
    const S* in = (const S*)io.q_stage;
    double qb = 0.;
    if (on) {
        qb = io.q_base[c];
        q[l] = in[c];
    }
    for (int h = l; h < inf.y; h += blockDim.x) q[SP.T + h] = in[h == l ? h0 : __ldg(SP.halo + inf.x + h)];
    __syncthreads();
    if (inactive) return;
    if (io.dtkeys != nullptr && t == 0) {
        for (int i = l; i < P.n_cases; i += blockDim.x) {
            io.dtkeys[(size_t)i * kDtSlots] = tkey(P.dt_const);
            io.dt[P.n_cases > 1 ? P.case_cell0[i] : P.cell0] = P.dt_const;
        }
    }
    double res = 0.;
    if (on) {
        const double qt = st.qt(q, l), qnew = fma(qt, P.dt_const * io.alpha, qb);
        res = qt * qt * A;
        auto write = [&](int g) {
            if constexpr (sizeof(S) == 8) io.q_out[g] = qnew;
            else {
                ((S*)io.s_out)[g] = (S)qnew;
                if (io.write_f64) io.q_out[g] = g == c ? qnew : (double)(S)qnew;
            }
        };
        write(c);
        st.ghosts(SP, inf.x, write);
    }
    if (io.partials != nullptr) {
        const double s = block_sum(res);
        if (l == 0) io.partials[t] = s;
    }
}

// All the steps of a launch (see fv_persist.cuh), one resident CTA per SM with
// as many tiles as that takes: the fewer CTAs, the shorter the barrier (125,000
// cells FP64, us per RK5 step: 977 CTAs of one tile 29, 140 CTAs of seven 19).
// A cell's stencil, base and stage states stay in its thread's registers; the
// halo's states are the only loads of a stage.  With several stages the norms
// and stop criteria of a step are evaluated beside the next one's first stage,
// which writes to a stage buffer only; a single-stage step waits for them.
template <class S, int NF, int THREADS>
__global__ void __launch_bounds__(THREADS)
    k_run_stencil(const __grid_constant__ StencilParams SP, const __grid_constant__ PersistIO D) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ RunState c;
    const Params& P = SP.P;
    const int x = threadIdx.x, T = SP.T, sub = x / T, l = x - sub * T, t = blockIdx.x * (blockDim.x / T) + sub;
    S* q = reinterpret_cast<S*>(smem_raw) + (size_t)sub * SP.max_slots;
    const int cell = t * T + l, warp = x >> 5, nw = (int)blockDim.x >> 5;
    const int4 inf = t < D.n_tiles ? __ldg(SP.info + t) : make_int4(0, 0, 0, 0);
    const bool on = l < inf.z;
    Stencil<S, NF> st;
    double qb = 0.;
    S qs = S(0);
    if (on) {
        st.load(SP, cell);
        qb = D.qbase[0][cell];
        qs = ((const S*)D.sbase[0])[cell];
    }
    const int h0 = l < inf.y ? __ldg(SP.halo + inf.x + l) : 0;
    const RunLimits lim = *D.limits;
    if (x == 0) {
        c.step = D.ctrl->step;
        c.time = D.ctrl->time;
        c.R[0] = D.ctrl->R[0]; c.R0[0] = D.ctrl->R0[0]; c.Rraw[0] = D.ctrl->Rraw[0];
        c.n_hist = 0;
        run_step_start<1>(c, lim);
    }
    GridSync sync{D.bar, &D.ctrl->failed, D.polls};
    sync.arrive();
    bool pending = false;
    int n = 0;
    const double* part = nullptr;  // the pending step's partial sums
    for (bool go = c.active != 0; go && n < D.max_steps; ++n) {
        const int b = D.ns == 1 ? (n & 1) : 0;
        const S* in = (const S*)D.sbase[b];
        double* part_out = D.partials + (size_t)(n & 1) * gridDim.x;
        for (int k = 0; k < D.ns; ++k) {
            const bool last = k == D.ns - 1;
            S* out = (S*)(D.ns == 1 ? D.sbase[1 - b] : last ? D.sbase[b] : D.tmp[k & 1]);
            double* out64 = D.qbase[D.ns == 1 ? 1 - b : b];
            if (!sync.wait()) return;
            if (D.ns == 1 && pending) {
                if (warp == nw - 1) run_step_end<1>(D, c, lim, P.dt_const, part, gridDim.x);
                __syncthreads();
                pending = false;
            }
            if ((k == 1 || D.ns == 1) && !c.active) { go = false; break; }
            for (int h = l; h < inf.y; h += T) q[T + h] = __ldcg(in + (h == l ? h0 : __ldg(SP.halo + inf.x + h)));
            if (on) q[l] = qs;
            __syncthreads();
            if (k == 0 && pending && warp == nw - 1) run_step_end<1>(D, c, lim, P.dt_const, part, gridDim.x);
            if (k == (D.ns == 1 ? 0 : 1) && blockIdx.x == 0)
                for (int i = x; P.n_cases > 1 && i < P.n_cases; i += blockDim.x) P.case_time[i] += P.dt_const;
            double qt = 0.;
            if (on) {
                qt = st.qt(q, l);
                const double qnew = fma(qt, P.dt_const * D.alpha[k], qb);
                qs = (S)qnew;
                auto write = [&](int g, double v) {
                    out[g] = qs;
                    if (sizeof(S) == 4 && last) out64[g] = v;
                };
                write(cell, qnew);
                st.ghosts(SP, inf.x, [&](int g) { write(g, (double)qs); });
                if (last) qb = qnew;
            }
            if (last && c.need_R) {
                const double s = block_sum(on ? qt * qt * __ldg(SP.area + cell) : 0.);
                if (x == 0) part_out[blockIdx.x] = s;
            }
            sync.arrive();
            if (k == 0) pending = false;
            in = out;
        }
        if (go) { pending = true; part = part_out; }
    }
    if (pending) {  // the launch's last step
        if (!sync.wait()) return;
        if (warp == nw - 1) run_step_end<1>(D, c, lim, P.dt_const, part, gridDim.x);
        __syncthreads();
    }
    if (blockIdx.x == 0 && x == 0) {
        Ctrl* o = D.ctrl;
        o->step = c.step;
        o->time = c.time;
        o->R[0] = c.R[0]; o->R0[0] = c.R0[0]; o->Rraw[0] = c.Rraw[0];
        o->active = c.active;
        o->need_R = c.need_R;
        o->n_hist = c.n_hist;
    }
}

}  // namespace

const void* stencil_run_kernel(bool f32, int nf, int* threads) {
    // 64 registers; 80 for the quadrilaterals' stencils
    *threads = nf == 3 ? 1024 : 768;
    if (f32) return nf == 3 ? (const void*)k_run_stencil<float, 3, 1024> : (const void*)k_run_stencil<float, 4, 768>;
    return nf == 3 ? (const void*)k_run_stencil<double, 3, 1024> : (const void*)k_run_stencil<double, 4, 768>;
}

void launch_stencil_stage(bool f32, const StencilParams& SP, const TileIO& io, int n_tiles, cudaStream_t st, bool pdl) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)n_tiles);
    cfg.blockDim = dim3((unsigned)SP.T);
    cfg.dynamicSmemBytes = (size_t)SP.max_slots * (f32 ? 4 : 8);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = pdl ? 1 : 0;
    auto go = [&](auto k) { cudaLaunchKernelEx(&cfg, k, SP, io); };
    if (f32) { if (SP.nf == 3) go(k_stencil_stage<float, 3>); else go(k_stencil_stage<float, 4>); }
    else if (SP.nf == 3) go(k_stencil_stage<double, 3>);
    else go(k_stencil_stage<double, 4>);
}

}  // namespace fvgpu
