// Discrete adjoint kernels of the explicit step (FP64, Euler, V = 4).
//
// Each kernel owns what it writes and gathers what flows into it, so results do
// not depend on scheduling.  The flux, the gradient + limiter and the linear
// parts (MUSCL, RK update) are differentiated in reverse by hand; the boundary
// functions and the time step come from the primal functions of
// fv_physics_exact.cuh on dual numbers (fv_dual.cuh, Dual<4> seeded on one
// cell's 4 conserved variables).  Reference arithmetic followed: gradients
// explicit.cpp:112-171, limiters 174-258, MUSCL + flux 261-364, update 368-378,
// ghost fill 380-417, min_dt 555-564; Roe flux examples/forwardStep/main.cpp:
// 72-135; CFL time step forwardStep/main.cpp:140-185.
#include <algorithm>

#include "fv_adjoint.h"
#include "fv_dual.cuh"
#include "fv_physics_exact.cuh"

namespace fvgpu {
namespace {

using D4 = Dual<4>;
using D1 = Dual<1>;
constexpr int kAB = 128;  // threads per block
constexpr int kFaces = 4;
constexpr uint32_t kNone = 0xFFFFFFFFu;

__device__ __forceinline__ void ld4(const double* __restrict__ a, int c, double* v) {
    const double2* p = reinterpret_cast<const double2*>(a + 4 * (size_t)c);
    const double2 x = p[0], y = p[1];
    v[0] = x.x; v[1] = x.y; v[2] = y.x; v[3] = y.y;
}
__device__ __forceinline__ void st4(double* a, int c, const double* v) {
    double2* p = reinterpret_cast<double2*>(a + 4 * (size_t)c);
    p[0] = make_double2(v[0], v[1]);
    p[1] = make_double2(v[2], v[3]);
}
__device__ __forceinline__ void add4(double* a, int c, const double* v) {
    double w[4];
    ld4(a, c, w);
    for (int k = 0; k < 4; ++k) w[k] += v[k];
    st4(a, c, w);
}
__device__ __forceinline__ void seed(D4* x, const double* v) {
#pragma unroll
    for (int k = 0; k < 4; ++k) { x[k] = D4(v[k]); x[k].d[k] = 1.0; }
}
__device__ __forceinline__ void constant(D4* x, const double* v) {
#pragma unroll
    for (int k = 0; k < 4; ++k) x[k] = D4(v[k]);
}
// MUSCL face state q + (g . d) lim with the positivity guard (returns true
// when the guard replaced it by the cell value)
__device__ __forceinline__ bool recon(const Params& P, const double* q, const double* gx, const double* gy,
                                      const double* lim, double dx, double dy, double* out) {
#pragma unroll
    for (int k = 0; k < 4; ++k) out[k] = q[k] + (gx[k] * dx + gy[k] * dy) * lim[k];
    if (!P.positivity_guard) return false;
    const double p = (P.gamma - 1.0) * (out[3] - 0.5 / out[0] * (out[1] * out[1] + out[2] * out[2]));
    if (!(out[0] > 0.0) || !(p > 0.0)) {
#pragma unroll
        for (int k = 0; k < 4; ++k) out[k] = q[k];
        return true;
    }
    return false;
}

__device__ __forceinline__ double signum(double x) { return x < 0.0 ? -1.0 : 1.0; }  // of the duals' fabs

// Roe flux f(a, b) and its reverse: la = (df/da)^T lam, lb = (df/db)^T lam.
// Branches (minimum, maximum, absolute values) follow the primal values.  One
// reverse sweep costs about three fluxes and gives both sides; forward
// tangents cost five fluxes a side.
__device__ __forceinline__ void roe_reverse(double gamma, const double* a, const double* b, double n0, double n1,
                                            const double* lam, double* f, double* la, double* lb) {
    const double g1 = gamma - 1.0;
    const double ri = 1.0 / a[0], rj = 1.0 / b[0];
    const double uL = a[1] * ri, vL = a[2] * ri, uR = b[1] * rj, vR = b[2] * rj;
    const double kL = 0.5 * (uL * uL + vL * vL), kR = 0.5 * (uR * uR + vR * vR);
    const double pL = g1 * (a[3] - a[0] * kL), pR = g1 * (b[3] - b[0] * kR);
    const double VL = uL * n0 + vL * n1, VR = uR * n0 + vR * n1;
    const double HL = a[3] + pL, HR = b[3] + pR, hL = HL * ri, hR = HR * rj;
    const double sL = sqrt(a[0]), sR = sqrt(b[0]);
    const double w = 1.0 / (sL + sR);
    const double u = (uL * sL + uR * sR) * w, v = (vL * sL + vR * sR) * w, h = (hL * sL + hR * sR) * w;
    const double q2 = u * u + v * v;
    const double c2 = g1 * (h - 0.5 * q2), c = sqrt(c2);
    const double V = u * n0 + v * n1, rho = sL * sR;
    const double dp = pR - pL, dV = VR - VL, dr = b[0] - a[0], du = uR - uL, dv = vR - vL;
    const bool left = VL - c < V - c, right = V + c < VR + c;
    const double x1 = left ? VL - c : V - c, x5 = right ? VR + c : V + c;
    const double l1 = fabs(x1), l2 = fabs(V), l5 = fabs(x5);
    const double rc = rho * c, i2 = 0.5 / c2;
    const double A1 = dp - rc * dV, A5 = dp + rc * dV, A0 = dr - 2.0 * dp * i2;
    const double k1 = l1 * A1 * i2, k0 = l2 * A0, kr = l2 * rho, k5 = l5 * A5 * i2;
    const double d = k5 - k1, s = k1 + k0 + k5;
    f[0] = 0.5 * (a[0] * VL + b[0] * VR - s);
    f[1] = 0.5 * (a[1] * VL + b[1] * VR + (pL + pR) * n0 - (s * u + d * c * n0 + kr * (du - dV * n0)));
    f[2] = 0.5 * (a[2] * VL + b[2] * VR + (pL + pR) * n1 - (s * v + d * c * n1 + kr * (dv - dV * n1)));
    f[3] = 0.5 * (HL * VL + HR * VR - ((k1 + k5) * h + d * c * V + k0 * q2 * 0.5 + kr * (u * du + v * dv - V * dV)));
    // ---- reverse (xB: the adjoint of x)
    const double m0 = 0.5 * lam[0], m1 = 0.5 * lam[1], m2 = 0.5 * lam[2], m3 = 0.5 * lam[3];
    const double nl = m1 * n0 + m2 * n1 + m3 * V;  // -adjoint of c d
    const double t0 = m0 + m1 * u + m2 * v;
    const double k1B = -(t0 + m3 * h - c * nl), k5B = -(t0 + m3 * h + c * nl);
    const double k0B = -(t0 + 0.5 * m3 * q2);
    const double krB = -(m1 * (du - dV * n0) + m2 * (dv - dV * n1) + m3 * (u * du + v * dv - V * dV));
    double uB = -(m1 * s + m3 * kr * du), vB = -(m2 * s + m3 * kr * dv), hB = -m3 * (k1 + k5);
    double q2B = -0.5 * m3 * k0;
    double cB = -d * nl, VB = -m3 * (c * d - kr * dV);
    const double duB = -kr * (m1 + m3 * u), dvB = -kr * (m2 + m3 * v);
    double dVB = kr * nl;
    const double A1B = k1B * l1 * i2, A5B = k5B * l5 * i2, A0B = k0B * l2;
    const double i2B = k1B * l1 * A1 + k5B * l5 * A5 - 2.0 * dp * A0B;
    const double dpB = A1B + A5B - 2.0 * i2 * A0B;
    dVB += rc * (A5B - A1B);
    const double rcB = dV * (A5B - A1B);
    const double rhoB = krB * l2 + rcB * c;
    cB += rcB * rho;
    VB += signum(V) * (k0B * A0 + krB * rho);
    const double x1B = signum(x1) * k1B * A1 * i2, x5B = signum(x5) * k5B * A5 * i2;
    cB += x5B - x1B;
    double VLB = -dVB, VRB = dVB;
    if (left) VLB += x1B; else VB += x1B;
    if (right) VRB += x5B; else VB += x5B;
    const double c2B = 0.5 * cB / c - 2.0 * i2 * i2 * i2B;
    hB += g1 * c2B;
    q2B -= 0.5 * g1 * c2B;
    uB += 2.0 * u * q2B + n0 * VB;
    vB += 2.0 * v * q2B + n1 * VB;
    // one side: x = a or b with its primitives, weight sx w, and adjoints so far
    auto side = [&](const double* x, double r, double ux, double vx, double kx, double Vx, double Hx, double hx, double sx,
                    double so, double pB, double VxB, double rB, double uxB, double vxB, double* l) {
        const double ws = sx * w;
        VxB += m0 * x[0] + m1 * x[1] + m2 * x[2] + m3 * Hx;
        const double hxB = hB * ws;
        const double HB = m3 * Vx + hxB * r;
        pB += m1 * n0 + m2 * n1 + HB;
        uxB += uB * ws + n0 * VxB;
        vxB += vB * ws + n1 * VxB;
        const double sB = (uB * (ux - u) + vB * (vx - v) + hB * (hx - h)) * w + rhoB * so;
        l[0] = m0 * Vx + rB - hxB * hx * r - (uxB * ux + vxB * vx) * r + 0.5 * sB / sx + g1 * kx * pB;
        l[1] = m1 * Vx + uxB * r - g1 * ux * pB;
        l[2] = m2 * Vx + vxB * r - g1 * vx * pB;
        l[3] = HB + g1 * pB;
    };
    side(a, ri, uL, vL, kL, VL, HL, hL, sL, sR, -dpB, VLB, -A0B, -duB, -dvB, la);
    side(b, rj, uR, vR, kR, VR, HR, hR, sR, sL, dpB, VRB, A0B, duB, dvB, lb);
}

// phi(y) and phi'(y) of the limiter kinds
__device__ __forceinline__ void limiter_slope(int kind, double y, double& phi, double& slope) {
    phi = 0.0;
    slope = 0.0;
    if (kind == 1) {  // Michalak, y_t = 2
        const bool one = y >= 2.0;
        phi = one ? 1.0 : y - 0.25 * y * y;
        slope = one ? 0.0 : 1.0 - 0.5 * y;
    } else if (kind == 2) {
        const double n = y * y + 2.0 * y, r = 1.0 / (y * y + y + 2.0);
        phi = n * r;
        slope = (2.0 * y + 2.0 - phi * (2.0 * y + 1.0)) * r;
    } else if (kind == 3) {
        phi = y > 0.0 ? (y < 1.0 ? y : 1.0) : 0.0;
        slope = (y > 0.0 && y < 1.0) ? 1.0 : 0.0;
    }
}

// ---------------------------------------------------------------------------
// Ghost fill in reverse: 4 lanes per cell with boundary ghosts, lane m with
// variable m of the interior face state (and of the boundary state) seeded on a
// scalar dual, so that a lane evaluates one tangent instead of four.  The other
// cells' lam_g start at 0 in k_adj_residual.
__global__ void __launch_bounds__(64) k_adj_ghosts(Params P, AdjFaces F, AdjStage S) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int N = P.n_real, m = t & 3;
    if ((t >> 2) >= F.n_bcells) return;
    const int i = F.bcells[t >> 2];
    const bool rec = P.order2 && !S.zero_grad;
    double qi[4], gxi[4] = {0, 0, 0, 0}, gyi[4] = {0, 0, 0, 0}, limi[4] = {0, 0, 0, 0};
    ld4(S.qs1, i, qi);
    if (rec) { ld4(S.gx, i, gxi); ld4(S.gy, i, gyi); ld4(S.lim, i, limi); }
    auto own = [&](const double* v) { return m == 0 ? v[0] : m == 1 ? v[1] : m == 2 ? v[2] : v[3]; };
    double aq = 0., agx = 0., agy = 0., alim = 0.;
    for (int f = 0; f < kFaces; ++f) {
        const uint32_t w = F.nbr[(size_t)f * N + i];
        if (w == kNone) continue;
        const int j = (int)(w & 0x7FFFFFFFu);
        if (j < N) continue;
        const int gb = j - N;
        double lb[4];
        ld4(S.lam_next, j, lb);
        const double dx = P.g_dx[gb], dy = P.g_dy[gb], n0 = P.g_nx[gb], n1 = P.g_ny[gb];
        double x[4];
        bool guarded = false;
        if (rec) guarded = recon(P, qi, gxi, gyi, limi, dx, dy, x);
        else for (int k = 0; k < 4; ++k) x[k] = qi[k];
        const int group = P.ghost_group[gb];
        const int kind = P.group_bc[group];
        const double* bv = P.ghost_bv ? P.ghost_bv + 4 * (size_t)gb : P.group_bv + 4 * group;
        D1 xd[4], bvd[4], bd[4];
        auto along = [&](double sx, double sb) {  // J^T lam of the seeded variable
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                xd[k] = D1(x[k]);
                xd[k].d[0] = k == m ? sx : 0.;
                bvd[k] = D1(bv[k]);
                bvd[k].d[0] = k == m ? sb : 0.;
            }
            exact::bc_state<4>(kind, P.gamma, bvd, bd, xd, n0, n1);
            double r = 0.;
#pragma unroll
            for (int k = 0; k < 4; ++k) r += lb[k] * bd[k].d[0];
            return r;
        };
        const double lx = along(1., 0.);
        // boundary state of an inflow / far-field ghost
        if (kind == 2 || kind == 3 || kind == 5) S.lam_bv[4 * (size_t)gb + m] += along(0., 1.);
        aq += lx;
        if (rec && !guarded) {
            agx += lx * dx * own(limi);
            agy += lx * dy * own(limi);
            alim += lx * (own(gxi) * dx + own(gyi) * dy);
        }
    }
    const size_t k = 4 * (size_t)i + m;
    S.lam_next[k] += aq;
    if (S.lam_gx) { S.lam_gx[k] = agx; S.lam_gy[k] = agy; S.lam_lim[k] = alim; }
}

// sum over the 4 lanes of a cell of x[m], in lane m
__device__ __forceinline__ double transpose_sum(const double* x) {
    const int lane = threadIdx.x & 3;
    const double a0 = (lane & 2) ? x[2] : x[0], a1 = (lane & 2) ? x[3] : x[1];  // kept
    const double s0 = (lane & 2) ? x[0] : x[2], s1 = (lane & 2) ? x[1] : x[3];  // sent
    const double b0 = a0 + __shfl_xor_sync(0xffffffffu, s0, 2), b1 = a1 + __shfl_xor_sync(0xffffffffu, s1, 2);
    const double k = (lane & 1) ? b1 : b0, t = (lane & 1) ? b0 : b1;
    return k + __shfl_xor_sync(0xffffffffu, t, 1);
}

// Flux residual and RK update in reverse: 4 lanes per cell, one per face.
// Bound by the latency of one face's chain; a thread per cell with forward
// tangents (255 registers, three faces one after the other) took 50 us a
// stage at 10,206 cells, this kernel 17.
__global__ void __launch_bounds__(kAB, 3) k_adj_residual(Params P, AdjFaces F, AdjStage S) {
    const int tid = blockIdx.x * blockDim.x + threadIdx.x;
    const int N = P.n_real, i = min(tid >> 2, N - 1), f = tid & 3;
    const bool live = (tid >> 2) < N;
    const bool o2 = P.order2 != 0;
    const double ad = S.alpha * S.dt;
    const size_t s = (size_t)f * N + i;
    const uint32_t w = live ? F.nbr[s] : kNone;
    const int j = (int)(w & 0x7FFFFFFFu), side = (int)(w >> 31);
    double oq[4] = {0, 0, 0, 0}, ogx[4] = {0, 0, 0, 0}, ogy[4] = {0, 0, 0, 0}, olim[4] = {0, 0, 0, 0}, qt[4] = {0, 0, 0, 0};
    if (w != kNone) {
        double qi[4], qj[4], xi[4], xj[4], ln[4], lF[4], fl[4], lx[4], lo[4];
        double gxi[4] = {0, 0, 0, 0}, gyi[4] = {0, 0, 0, 0}, limi[4] = {0, 0, 0, 0};
        ld4(S.qs, i, qi);
        ld4(S.qs, j, qj);
        ld4(S.lam_next, i, ln);
        const double n0 = F.nx[s], n1 = F.ny[s], le = F.le[s], dx = F.dsx[s], dy = F.dsy[s];
        bool gi = false;
        if (o2) {
            ld4(S.gx, i, gxi); ld4(S.gy, i, gyi); ld4(S.lim, i, limi);
            gi = recon(P, qi, gxi, gyi, limi, dx, dy, xi);
            if (j < N) {
                double gxj[4], gyj[4], limj[4];
                ld4(S.gx, j, gxj); ld4(S.gy, j, gyj); ld4(S.lim, j, limj);
                recon(P, qj, gxj, gyj, limj, F.dnx[s], F.dny[s], xj);
            } else {
                for (int k = 0; k < 4; ++k) xj[k] = qj[k];  // ghosts: zero gradient
            }
        } else {
            for (int k = 0; k < 4; ++k) { xi[k] = qi[k]; xj[k] = qj[k]; }
        }
        // dL/dF: qt_left -= F le / A_left, qt_right += F le / A_right
        const double ci = (side ? le : -le) / F.area[i];
#pragma unroll
        for (int k = 0; k < 4; ++k) lF[k] = ci * ad * ln[k];
        if (j < N) {
            double lnj[4];
            ld4(S.lam_next, j, lnj);
            const double cj = (side ? -le : le) / F.area[j];
#pragma unroll
            for (int k = 0; k < 4; ++k) lF[k] += cj * ad * lnj[k];
        }
        double la[4], lb[4];
        if (side) roe_reverse(P.gamma, xj, xi, n0, n1, lF, fl, la, lb);
        else roe_reverse(P.gamma, xi, xj, n0, n1, lF, fl, la, lb);
#pragma unroll
        for (int k = 0; k < 4; ++k) { lx[k] = side ? lb[k] : la[k]; lo[k] = side ? la[k] : lb[k]; }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            qt[k] = ci * fl[k];
            oq[k] = lx[k];
            if (o2 && !gi) {
                ogx[k] = lx[k] * dx * limi[k];
                ogy[k] = lx[k] * dy * limi[k];
                olim[k] = lx[k] * (gxi[k] * dx + gyi[k] * dy);
            }
        }
        if (j >= N) st4(S.lam_cur, j, lo);  // the ghost's own adjoint (this cell owns it)
    }
    // lane m keeps variable m
    const unsigned ghosts = __ballot_sync(0xffffffffu, w != kNone && j >= N);
    const bool bcell = ((ghosts >> (threadIdx.x & 28)) & 15u) != 0;
    const double tq = transpose_sum(oq), tt = transpose_sum(qt);
    const size_t k = 4 * (size_t)i + f;
    const double lnk = live ? S.lam_next[k] : 0.0;
    if (live) {
        S.lam_cur[k] = tq;
        S.lam_qn[k] += lnk;
    }
    if (o2) {
        const double tx = transpose_sum(ogx), ty = transpose_sum(ogy), tl = transpose_sum(olim);
        if (live) {  // cells with ghosts hold the ghost fill's contribution
            S.lam_gx[k] = bcell ? S.lam_gx[k] + tx : tx;
            S.lam_gy[k] = bcell ? S.lam_gy[k] + ty : ty;
            S.lam_lim[k] = bcell ? S.lam_lim[k] + tl : tl;
        }
    }
    if (S.dt_partials) {
        __shared__ double red[kAB];
        red[threadIdx.x] = S.alpha * lnk * tt;
        __syncthreads();
        for (int r = kAB / 2; r > 0; r >>= 1) {
            if (threadIdx.x < r) red[threadIdx.x] += red[threadIdx.x + r];
            __syncthreads();
        }
        if (threadIdx.x == 0) S.dt_partials[blockIdx.x] = red[0];
    }
}

// Gradient and limiter of variable k of cell c in reverse, one thread per (real
// cell, variable): the operator is block-diagonal over the variables.  Leaves
// the adjoint of the cell's own value in out[0] and of its neighbours' values
// in out[1 + face] ([5][4 n_real]), which k_adj_gather collects.
__global__ void __launch_bounds__(kAB) k_adj_gradlim(Params P, AdjFaces F, AdjStage S, double* __restrict__ out) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int N = P.n_real, c = t >> 2, k = t & 3;
    if (c >= N) return;
    const double* qs = S.qs;
    const double q = qs[t], iA = 1.0 / F.area[c];
    double qn[kFaces], ax[kFaces], ay[kFaces], ox = 0., oy = 0., gx = 0., gy = 0., mx = q, mn = q;
    int imx = -1, imn = -1;
    bool has[kFaces];
#pragma unroll
    for (int f = 0; f < kFaces; ++f) {
        const size_t s = (size_t)f * N + c;
        const uint32_t w = F.nbr[s];
        has[f] = w != kNone;
        qn[f] = ax[f] = ay[f] = 0.;
        if (!has[f]) continue;
        const int side = (int)(w >> 31);
        qn[f] = qs[4 * (size_t)(w & 0x7FFFFFFFu) + k];
        // weights of the neighbour's and the own value in the face's term
        const double g = F.g[s], m = (side ? -F.le[s] : F.le[s]) * iA, wn = side ? 1.0 - g : g;
        ax[f] = m * F.nx[s];
        ay[f] = m * F.ny[s];
        gx += ax[f] * (q + (qn[f] - q) * wn);
        gy += ay[f] * (q + (qn[f] - q) * wn);
        ox += ax[f] * (1.0 - wn);
        oy += ay[f] * (1.0 - wn);
        ax[f] *= wn;
        ay[f] *= wn;
        if (qn[f] < mn) { mn = qn[f]; imn = f; }
        if (mx < qn[f]) { mx = qn[f]; imx = f; }
    }
    const double Ka = P.K * sqrt(F.area[c]), K3a = Ka * Ka * Ka, tol = 1e-15;
    const double dd = mx - mn, d2 = dd * dd;
    double sig = 0., sslope = 0.;  // sig and d sig / d d2
    if (d2 <= K3a) sig = 1.;
    else if (d2 <= 2 * K3a) {
        const double y = d2 / K3a - 1.0;
        sig = 2.0 * y * y * y - 3.0 * y * y + 1.0;
        sslope = (6.0 * y * y - 6.0 * y) / K3a;
    }
    // the face that sets the limiter (the first of equal ones)
    double lim = 1., phi_m = 1., slope_m = 0., y_m = 0., dq_m = 1., dx_m = 0., dy_m = 0.;
    bool any = false;
#pragma unroll
    for (int f = 0; f < kFaces; ++f) {
        if (!has[f]) continue;
        const double dx = F.dsx[(size_t)f * N + c], dy = F.dsy[(size_t)f * N + c];
        const double dq = gx * dx + gy * dy;
        double phi = 1., slope = 0., y = 0.;
        if (sig < 1.0 && (dq > tol || dq < -tol)) {
            y = (dq > tol ? mx - q : mn - q) / dq;
            limiter_slope(P.limiter, y, phi, slope);
        }
        const double lv = sig + (1.0 - sig) * phi;
        if (lv < lim) {
            lim = lv; phi_m = phi; slope_m = slope; y_m = y; dq_m = dq; dx_m = dx; dy_m = dy;
            any = true;
        }
    }
    double gxB = S.lam_gx[t], gyB = S.lam_gy[t], mxB = 0., mnB = 0., qB = 0.;
    if (any) {
        const double lB = S.lam_lim[t];
        const double sB = lB * (1.0 - phi_m) * sslope * 2.0 * dd;
        mxB += sB;
        mnB -= sB;
        const double yB = lB * (1.0 - sig) * slope_m;
        if (yB != 0.) {
            const double dB = yB / dq_m;  // of the delta; the slope's own part through dq
            if (dq_m > 0.) mxB += dB; else mnB += dB;
            qB -= dB;
            const double dqB = -dB * y_m;
            gxB += dqB * dx_m;
            gyB += dqB * dy_m;
        }
    }
    qB += gxB * ox + gyB * oy;
    if (imx < 0) qB += mxB;
    if (imn < 0) qB += mnB;
    const size_t n4 = 4 * (size_t)N;
    out[t] = qB;
#pragma unroll
    for (int f = 0; f < kFaces; ++f) {
        if (!has[f]) continue;
        double v = gxB * ax[f] + gyB * ay[f];
        if (imx == f) v += mxB;
        if (imn == f) v += mnB;
        out[(1 + f) * n4 + t] = v;
    }
}
// lam_cur += what k_adj_gradlim left for each cell: its own part and its slot in
// each neighbour (F.rev); a ghost's from its interior cell.
__global__ void __launch_bounds__(256) k_adj_gather(int N, AdjFaces F, const double* __restrict__ part, double* lam_cur) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int m = t >> 2, k = t & 3;
    if (m >= N) return;
    const size_t n4 = 4 * (size_t)N;
    double acc = part[t];
#pragma unroll
    for (int f = 0; f < kFaces; ++f) {
        const size_t s = (size_t)f * N + m;
        const uint32_t w = F.nbr[s];
        if (w == kNone) continue;
        const int c = (int)(w & 0x7FFFFFFFu);
        if (c < N) acc += part[(1 + F.rev[s]) * n4 + 4 * (size_t)c + k];
        else lam_cur[4 * (size_t)c + k] += part[(1 + f) * n4 + t];
    }
    lam_cur[t] += acc;
}

__global__ void k_add(double* y, const double* x, size_t n) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        y[i] += x[i];
}

// out = sum of p[0..n) in a fixed order: each of the block's threads sums a
// contiguous run, then a fixed tree over the threads.
constexpr int kSumThreads = 256;
__global__ void __launch_bounds__(kSumThreads) k_sum(const double* p, int n, double* out) {
    __shared__ double red[kSumThreads];
    const int per = (n + kSumThreads - 1) / kSumThreads;
    const int a = threadIdx.x * per, b = min(n, a + per);
    double s = 0.0;
    for (int i = a; i < b; ++i) s += p[i];
    red[threadIdx.x] = s;
    __syncthreads();
    for (int w = kSumThreads / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) *out = red[0];
}

__device__ __forceinline__ double key_inv(unsigned long long k) {
    if (k == ~0ull) return __longlong_as_double(0x7ff8000000000000ll);
    const unsigned long long b = (k & 0x8000000000000000ull) ? (k & 0x7fffffffffffffffull) : ~k;
    return __longlong_as_double((long long)b);
}

__global__ void k_dt_finalize(const unsigned long long* keys, const double* dt_cells, int cell0, double* dt_fill,
                              int n, double* dt_out) {
    unsigned long long key = ~0ull;
    for (int i = 0; i < 64; ++i) key = keys[i] < key ? keys[i] : key;
    const double d0 = dt_cells[cell0];
    const double mn = (d0 != d0) ? d0 : key_inv(key);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) dt_fill[i] = mn;
    if (blockIdx.x == 0 && threadIdx.x == 0) *dt_out = mn;
}

__global__ void k_argmin(const double* dt_cells, int n, const double* dt_n, int* argmin) {
    const double v = *dt_n;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        if (dt_cells[i] == v) atomicMin(argmin, i);
}

// CFL time step of cell a (forwardStep calc_dt kind) with one stencil cell seeded
__device__ D4 dt_cell_d(const Params& P, const AdjFaces& F, const double* q, int a, int seed_cell) {
    const int N = P.n_real;
    const double gamma = P.gamma, gm1 = gamma - 1, cfl = P.cfl;
    auto load = [&](int c, D4* x) {
        double v[4];
        ld4(q, c, v);
        if (c == seed_cell) seed(x, v); else constant(x, v);
    };
    auto sound = [&](const D4* x) {
        return sqrt((gm1 * (x[3] - 0.5 / x[0] * (x[1] * x[1] + x[2] * x[2]))) * gamma / x[0]);
    };
    if (a >= N) {  // ghost: its one face to the interior cell
        const int gb = a - N, i = P.ghost_cell[gb];
        D4 qs[4], qn[4];
        load(i, qs); load(a, qn);
        const double n0 = P.g_nx[gb], n1 = P.g_ny[gb], le = P.g_le[gb];
        const D4 es = sound(qs) + fabs(qs[1] / qs[0] * n0 + qs[2] / qs[0] * n1);
        const D4 en = sound(qn) + fabs(qn[1] / qn[0] * n0 + qn[2] / qn[0] * n1);
        const D4 center = dmax(es, en);
        return cfl * F.area[a] / (center * le);
    }
    D4 qs[4];
    load(a, qs);
    const D4 cs = sound(qs);
    D4 acc(0.0);
    for (int f = 0; f < kFaces; ++f) {
        const size_t s = (size_t)f * N + a;
        const uint32_t w = F.nbr[s];
        if (w == kNone) continue;
        const int j = (int)(w & 0x7FFFFFFFu), side = (int)(w >> 31);
        const double n0 = F.nx[s], n1 = F.ny[s], le = F.le[s];
        D4 qn[4];
        load(j, qn);
        const D4 es = cs + fabs(qs[1] / qs[0] * n0 + qs[2] / qs[0] * n1);
        const D4 en = sound(qn) + fabs(qn[1] / qn[0] * n0 + qn[2] / qn[0] * n1);
        const D4 center = side ? dmax(en, es) : dmax(es, en);
        acc += center * le;
    }
    return cfl * F.area[a] / acc;
}

__global__ void k_adj_dt(Params P, AdjFaces F, const double* q, const double* lam_dt, const int* argmin,
                         double* lam_q) {
    const int a = *argmin;
    const int N = P.n_real;
    if (a < 0 || a >= P.n_total) return;
    // one thread per stencil cell of the arg-min cell
    int c = -1;
    const int l = threadIdx.x;
    if (a >= N) {
        if (l < 2) c = l ? a : P.ghost_cell[a - N];
    } else if (l == 0) {
        c = a;
    } else if (l <= kFaces) {
        const uint32_t w = F.nbr[(size_t)(l - 1) * N + a];
        if (w != kNone) c = (int)(w & 0x7FFFFFFFu);
        // a neighbour across several faces is its first one's: its derivative holds all of them
        for (int f = 0; f < l - 1; ++f) {
            const uint32_t v = F.nbr[(size_t)f * N + a];
            if (v != kNone && (int)(v & 0x7FFFFFFFu) == c) c = -1;
        }
    }
    if (c < 0) return;
    const D4 d = dt_cell_d(P, F, q, a, c);
    double g[4];
    for (int k = 0; k < 4; ++k) g[k] = *lam_dt * d.d[k];
    add4(lam_q, c, g);
}

__device__ __forceinline__ double pres(double gamma, const double* q) {
    return (gamma - 1) * (q[3] - 0.5 / q[0] * (q[1] * q[1] + q[2] * q[2]));
}

// sum_t p(q[interior of ghost t]) le over the listed ghosts: strided by thread,
// then a fixed tree.
constexpr int kLossThreads = 128;
__device__ __forceinline__ double loss_sum(const Params& P, const double* q, const int32_t* ghosts, int n) {
    __shared__ double red[kLossThreads];
    double s = 0.0;
    for (int t = threadIdx.x; t < n; t += kLossThreads) {
        const int gb = ghosts[t];
        double v[4];
        ld4(q, P.ghost_cell[gb], v);
        s += pres(P.gamma, v) * P.g_le[gb];
    }
    red[threadIdx.x] = s;
    __syncthreads();
    for (int w = kLossThreads / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
        __syncthreads();
    }
    return red[0];
}
__global__ void __launch_bounds__(kLossThreads) k_loss(Params P, const double* q, const double* dt_n,
                                                       const int32_t* ghosts, int n, double* loss) {
    const double s = loss_sum(P, q, ghosts, n);
    if (threadIdx.x == 0) *loss += s * *dt_n;
}

__global__ void __launch_bounds__(kLossThreads) k_loss_adjoint(Params P, const double* q, const double* dt_n,
                                                               const int32_t* ghosts, int n, double w, double* lam_q,
                                                               double* lam_dt) {
    const double gm1 = P.gamma - 1.0, dt = *dt_n;
    for (int t = threadIdx.x; t < n; t += kLossThreads) {
        const int c = P.ghost_cell[ghosts[t]];
        // a cell with several listed ghosts (consecutive ones) is its first one's
        if (t > 0 && P.ghost_cell[ghosts[t - 1]] == c) continue;
        double v[4];
        ld4(q, c, v);
        const double u = v[1] / v[0], vv = v[2] / v[0];
        const double dp[4] = {gm1 * 0.5 * (u * u + vv * vv), -gm1 * u, -gm1 * vv, gm1};
        for (int r = t; r < n && P.ghost_cell[ghosts[r]] == c; ++r) {
            const double le = P.g_le[ghosts[r]];
            double g[4];
            for (int k = 0; k < 4; ++k) g[k] = w * dt * le * dp[k];
            add4(lam_q, c, g);
        }
    }
    const double s = loss_sum(P, q, ghosts, n);
    if (threadIdx.x == 0) *lam_dt += w * s;
}

int blocks_for(int n) { return (n + kAB - 1) / kAB; }

}  // namespace

int adj_residual_blocks(const Params& P) { return blocks_for(4 * P.n_real); }

void adj_launch_ghosts(const Params& P, const AdjFaces& F, const AdjStage& S, cudaStream_t st) {
    if (F.n_bcells) k_adj_ghosts<<<(4 * F.n_bcells + 63) / 64, 64, 0, st>>>(P, F, S);
}
void adj_launch_residual(const Params& P, const AdjFaces& F, const AdjStage& S, cudaStream_t st) {
    k_adj_residual<<<blocks_for(4 * P.n_real), kAB, 0, st>>>(P, F, S);
}
void adj_launch_gradlim(const Params& P, const AdjFaces& F, const AdjStage& S, double* part, cudaStream_t st) {
    k_adj_gradlim<<<blocks_for(4 * P.n_real), kAB, 0, st>>>(P, F, S, part);
    k_adj_gather<<<(4 * P.n_real + 255) / 256, 256, 0, st>>>(P.n_real, F, part, S.lam_cur);
}
void adj_launch_add(double* y, const double* x, size_t n, cudaStream_t st) {
    const int b = (int)std::min<size_t>((n + 255) / 256, 148 * 16);
    k_add<<<b > 0 ? b : 1, 256, 0, st>>>(y, x, n);
}
void adj_launch_sum(const double* partials, int n, double* out, cudaStream_t st) {
    k_sum<<<1, kSumThreads, 0, st>>>(partials, n, out);
}
void adj_launch_dt_finalize(const unsigned long long* keys, const double* dt_cells, int cell0, double* dt_fill, int n,
                            double* dt_out, cudaStream_t st) {
    const int b = std::min((n + 255) / 256, 148 * 8);
    k_dt_finalize<<<b > 0 ? b : 1, 256, 0, st>>>(keys, dt_cells, cell0, dt_fill, n, dt_out);
}
void adj_launch_dt(const Params& P, const AdjFaces& F, const double* q, const double* dt_cells, const double* dt_n,
                   const double* lam_dt, double* lam_qn, int* argmin, cudaStream_t st) {
    cudaMemsetAsync(argmin, 0x7F, sizeof(int), st);
    const int b = std::min((P.n_total + 255) / 256, 148 * 8);
    k_argmin<<<b > 0 ? b : 1, 256, 0, st>>>(dt_cells, P.n_total, dt_n, argmin);
    k_adj_dt<<<1, 32, 0, st>>>(P, F, q, lam_dt, argmin, lam_qn);
}
void adj_launch_loss(const Params& P, const double* q, const double* dt_n, const int32_t* ghosts, int n_ghosts,
                     double* loss, cudaStream_t st) {
    k_loss<<<1, kLossThreads, 0, st>>>(P, q, dt_n, ghosts, n_ghosts, loss);
}
void adj_launch_loss_adjoint(const Params& P, const double* q, const double* dt_n, const int32_t* ghosts,
                             int n_ghosts, double w, double* lam_q, double* lam_dt, cudaStream_t st) {
    k_loss_adjoint<<<1, kLossThreads, 0, st>>>(P, q, dt_n, ghosts, n_ghosts, w, lam_q, lam_dt);
}

}  // namespace fvgpu
