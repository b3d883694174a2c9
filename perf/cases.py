"""The timed cases of the explicit finite-volume step.

A case is one piece of work that a program built on this framework has it do:
it holds a mesh and a solver, hands over a state, runs some time steps and
takes the state back (or, for the adjoint, asks for a gradient).  The meshes
and physics are those of the benchmark workloads and the examples: the Sod
tube, the Mach 3 forward-facing step, the NACA 0012 O-grid, batched Riemann
strips, the Navier-Stokes flat plate and airfoil, the heat equation, and
Burgers + diffusion with residual smoothing.

``exact`` restates the time loop in 64-bit PyTorch: geometry from the element
mesh, Green-Gauss gradients, smooth-switch limiter, MUSCL, Roe / Burgers /
diffusion fluxes, the boundary states, the time steps and the RK update.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "finite-volume-2d-cpp_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import fvgpu  # noqa: E402
import meshgen  # noqa: E402
import physics as P  # noqa: E402

N_BINS = 16  # inflow density bins of the adjoint cases


# ------------------------------------------------------------------- cases --
def listed():
    return [
        # The shock-tube example at its own order of size: the drop-in program
        # in its default precision, host arrays in and out.  Steps take a few
        # microseconds of work, so launches and latency are what a user waits for.
        dict(name="sod_example", kind="sod", nx=100, ny=4, precision="fp64_exact", steps=200, host=True),
        # The Sod benchmark, 32,000 cells: first order, RK1.
        dict(name="sod_400x40", kind="sod", nx=400, ny=40, precision="fp64", steps=100, host=False),
        # The forward-step example's size (about 10,000 cells), second order,
        # drop-in precision, host arrays.
        dict(name="step_example", kind="step", nx=45, ny=0, precision="fp64_exact", steps=30, host=True),
        # An everyday production mesh, 99,000 cells, FP32-bulk.
        dict(name="step_100k_fp32", kind="step", nx=140, ny=0, precision="fp32", steps=30, host=False),
        # The headline benchmark: 998,000 cells, FP32-bulk and plain FP64.
        dict(name="step_1m_fp32", kind="step", nx=445, ny=0, precision="fp32", steps=20, host=False),
        dict(name="step_1m_fp64", kind="step", nx=445, ny=0, precision="fp64", steps=10, host=False),
        # Steady airfoil with local time steps and Michalak's limiter: an
        # engineering grid in FP64 and the benchmark's O-grid in FP32-bulk.
        dict(name="naca_65k_fp64", kind="naca", nx=256, ny=128, precision="fp64", steps=20, host=False),
        dict(name="naca_1m_fp32", kind="naca", nx=1024, ny=512, precision="fp32", steps=10, host=False),
        # Many independent cases in one solver: strips of uneven, odd sizes.
        dict(name="strips_48_fp32", kind="strips", nx=30000, ny=48, precision="fp32", steps=10, host=False),
        # The flat-plate example's quadrilateral mesh: Navier-Stokes, local steps.
        dict(name="plate_example", kind="plate", nx=120, ny=110, precision="fp64", steps=30, host=False),
        # The heat-transfer example's physics on 125,000 triangles.
        dict(name="heat_125k_fp64", kind="heat", nx=250, ny=250, precision="fp64", steps=20, host=False),
        # Backward direction: loss and gradient of the forward step.
        dict(name="adjoint_10k", kind="adjoint", nx=45, ny=0, precision="fp64_exact", steps=20, host=True),
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    kind = rng.choice(["sod", "step", "step", "step", "naca", "naca", "strips", "plate", "transient", "heat",
                       "smooth", "adjoint"])
    prec = rng.choice(["fp64_exact", "fp64", "fp32", "fp32"])
    nx = ny = 0
    if kind == "sod":
        nx, ny = _log(rng, 40, 1600), _log(rng, 2, 160)
    elif kind == "step":
        nx = 5 * _log(rng, 4, 88)
    elif kind == "naca":
        nx = _log(rng, 48, 1000)
        ny = max(8, int(nx * rng.uniform(0.25, 0.5)))
    elif kind == "strips":
        nx, ny = _log(rng, 300, 40000), rng.randint(3, 48)  # largest strip's cells, strips
    elif kind == "plate":
        nx, ny = _log(rng, 24, 700), _log(rng, 20, 700)
    elif kind == "transient":
        nx = _log(rng, 48, 500)
        ny = max(8, int(nx * rng.uniform(0.25, 0.5)))
    elif kind in ("heat", "smooth"):
        nx, ny = _log(rng, 16, 600), _log(rng, 16, 600)
    else:
        nx, prec = 5 * _log(rng, 4, 12), "fp64_exact"
    cells = _cells(dict(kind=kind, nx=nx, ny=ny))
    most = 25 if kind == "adjoint" else max(4, min(200, int(6e6 / cells)))
    return dict(kind=kind, nx=nx, ny=ny, precision=prec, steps=rng.randint(max(2, most // 2), most),
                host=kind == "adjoint" or (cells < 20000 and rng.random() < 0.5))


def _cells(case):
    nx, ny, kind = case["nx"], case["ny"], case["kind"]
    if kind in ("step", "adjoint"):
        return round(2 * nx * nx * (3 - 2.4 * 0.2))
    if kind == "strips":
        return int(ny * nx * 0.45)
    return nx * ny * (1 if kind == "plate" else 2)


def work(case):
    """Per RK stage: the stage and base states read, the new state written, and
    the mesh (indices, normal, length, face centre and weight of each edge;
    centroid and area of each cell) read once; the state in and out."""
    n, ph = _cells(case), _physics(case, None)
    sz = 4 if case["precision"] == "fp32" else 8
    epc = 2.0 if case["kind"] == "plate" else 1.5
    stages = case["steps"] * len(_alpha(case))
    grads = ph.order2 or ph.diffusive
    per = ph.V * (2 * sz + 8) + epc * (8 + sz * (6 if grads else 3)) + sz * (3 if grads else 1)
    flux = {1: 20, 2: 60, 4: 150}[ph.V] + (120 if ph.flux == "ns" else 0) + (20 * ph.V if ph.order2 else 0)
    flops = epc * flux + (2 * epc * (18 if ph.order2 else 8) * ph.V if grads else 0) + 6 * ph.V
    k = 4.0 if case["kind"] == "adjoint" else 1.0  # forward, recomputation and the reverse sweep
    return {"bytes": k * stages * n * per + 4.0 * 8 * ph.V * n, "flops": k * stages * n * flops}


# ------------------------------------------------------------------ inputs --
def _step_mesh(n, seed, jitter=0.2):
    """[0,3]x[0,1] without the step x > 0.6, y < 0.2: a lattice of spacing 1/n
    (n a multiple of 5) with jittered interior nodes, each quadrilateral split
    along its shorter diagonal.  Groups: wall, inlet, outlet, step."""
    nxl, nyl, si, sj, h = 3 * n, n, 3 * n // 5, n // 5, 1.0 / n
    J, I = np.meshgrid(np.arange(nyl + 1), np.arange(nxl + 1), indexing="ij")
    keep = ~((I > si) & (J < sj))
    lut = np.where(keep, np.cumsum(keep.ravel()).reshape(keep.shape) - 1, -1)
    bnd = (I == 0) | (I == nxl) | (J == 0) | (J == nyl) | ((I == si) & (J <= sj)) | ((J == sj) & (I >= si))
    d = np.random.default_rng(seed).uniform(-jitter * h, jitter * h, size=(2,) + I.shape)
    d[:, bnd] = 0.0
    x, y = I * h + d[0], J * h + d[1]
    quad = ~((I[:-1, :-1] >= si) & (J[:-1, :-1] < sj))
    a, b, c, e = (lut[s][quad] for s in (np.s_[:-1, :-1], np.s_[:-1, 1:], np.s_[1:, 1:], np.s_[1:, :-1]))
    x, y = x[keep], y[keep]
    ac = (x[a] - x[c]) ** 2 + (y[a] - y[c]) ** 2 <= (x[b] - x[e]) ** 2 + (y[b] - y[e]) ** 2
    t1 = np.where(ac, (a, b, c), (a, b, e)).T
    t2 = np.where(ac, (a, c, e), (b, c, e)).T
    cells = np.concatenate([np.stack([t1, t2], 1).reshape(-1, 3), np.full((2 * a.size, 1), -1)], 1)
    parts = [(0, lut[0, :si + 1]), (0, lut[sj, si:]), (0, lut[nyl, ::-1]), (1, lut[::-1, 0]),
             (2, lut[sj:, nxl]), (3, lut[:sj + 1, si])]
    seg = np.concatenate([np.stack([w[:-1], w[1:]], 1) for _, w in parts])
    grp = np.concatenate([np.full(w.size - 1, g) for g, w in parts])
    return meshgen.ElementMesh(x, y, cells.astype(np.int32), seg.astype(np.int32), grp.astype(np.int32),
                               ["wall", "inlet", "outlet", "step"])


def _meshes(case, seed):
    """The element meshes of a case (one, or one per strip)."""
    kind, nx, ny = case["kind"], case["nx"], case["ny"]
    if kind == "sod":
        return [meshgen.sod_strip(nx, ny)]
    if kind in ("step", "adjoint"):
        return [_step_mesh(nx, seed)]
    if kind in ("naca", "transient"):
        em = meshgen.naca_ogrid(nx, ny, r_far=50.0, jitter=0.05, seed=seed)
        if kind == "transient":
            em.group_names = ["wall", "farfield"]
        return [em]
    if kind == "strips":
        n = np.exp(np.random.default_rng([nx, ny]).uniform(math.log(max(64, nx // 20)), math.log(nx), ny))
        return [meshgen.riemann_strip(max(4, int(v / 16))) for v in n]
    if kind == "plate":
        n0 = max(2, nx // 4)
        # the example's gradings, eased on finer meshes so that the smallest
        # cell stays of the same relative size
        r = lambda g, n, of: g ** min(1.0, of / n)  # noqa: E731
        return [meshgen.flat_plate(n0, nx - n0, ny, r_up=r(1.2, n0, 30), r_plate=r(1.1, nx - n0, 90),
                                   r_y=r(1.1, ny, 110))]
    return [meshgen.rect_tri(nx, ny, 1.0, 1.0, side_names=("wall", "wall"))]


def _physics(case, ems):
    kind = case["kind"]
    if kind == "sod":
        return P.sod()
    if kind in ("step", "adjoint"):
        ph = P.forward_step(cfl=0.5 if kind == "adjoint" else 0.8)
        ph.positivity_guard = True
        return ph
    if kind == "naca":
        return P.naca()
    if kind == "strips":
        return P.riemann_strip()
    if kind == "plate":
        return P.flat_plate(cfl=1.0)
    if kind == "transient":
        return P.naca_transient(cfl=1.0)
    h = 1.0 / max(case["nx"], case["ny"])
    return P.heat(dt=0.05 * h * h) if kind == "heat" else P.burgers_diffusion(dt=0.05 * h * h)


def _alpha(case):
    return P.RK1_ALPHA if case["kind"] == "sod" else P.RK5_ALPHA


def _centres(em):
    """Centroids of the real cells, then the midpoints of the boundary segments."""
    tri = em.cells[:, 3] < 0
    c = np.where(tri[:, None] & (np.arange(4) == 3), em.cells[:, :1], em.cells)
    w = np.where(tri, 3.0, 4.0)
    xy = []
    for v in (em.nodes_x, em.nodes_y):
        s = v[c[:, 0]] + v[c[:, 1]] + v[c[:, 2]] + np.where(tri, 0.0, v[c[:, 3]])
        xy.append(np.concatenate([s / w, v[em.bnd_nodes].mean(1)]))
    return xy


def _waves(rng, x, y, amp, modes=4):
    """A smooth field of zero mean and about `amp` in size: long and shorter waves of random direction and phase."""
    s = np.zeros_like(x)
    for m in range(modes):
        k = 2 * math.pi * (m + 1) * rng.uniform(0.6, 1.4)
        t, ph = rng.uniform(0, 2 * math.pi, 2)
        s += amp / modes * np.sin(k * (math.cos(t) * x + math.sin(t) * y) + ph)
    return s


def _initial(case, ems, seed):
    """A state of the flow under way, [cells and ghosts of each mesh][V]: the
    case's free stream with waves of some percent and a shock, the strips' and
    the tube's two states, a warm disc, a swirl."""
    rng, kind, out = np.random.default_rng([seed, 17]), case["kind"], []
    for em in ems:
        x, y = _centres(em)
        if kind == "heat":
            x0, y0 = rng.uniform(0.4, 0.6, 2)
            out.append((np.hypot(x - x0, y - y0) < 0.16)[:, None] + _waves(rng, x, y, 0.1)[:, None])
            continue
        if kind == "smooth":
            out.append(np.stack([_waves(rng, x, y, 0.5), _waves(rng, x, y, 0.5)], 1))
            continue
        if kind in ("sod", "strips"):
            m = x < 0.5
            if kind == "sod":
                f = rng.uniform(0.9, 1.1, 4)
                st = (f[0], 0.0, f[1], 0.125 * f[2], 0.0, 0.1 * f[3])
            else:
                st = tuple(rng.uniform(lo, hi) for lo, hi in ((0.1, 1.0), (-0.5, 0.5), (0.1, 1.0)) * 2)
            rho, u, p = (np.where(m, st[i], st[i + 3]) * (1 + _waves(rng, x, y, 0.01)) for i in range(3))
            v = _waves(rng, x, y, 0.01)
        else:
            mach = {"step": 3.0, "naca": 0.8, "plate": 0.2, "transient": 0.8}[kind]
            amp = {"step": 0.06, "naca": 0.03, "plate": 0.005, "transient": 0.02}[kind]
            xs, ys = (x, y) if kind != "plate" else (x, 5 * y)
            if kind in ("naca", "transient"):  # waves in the angle and in the logarithm of the distance
                xs = np.arctan2(y, x - 0.5) / math.pi
                ys = 0.25 * np.log(np.hypot(x - 0.5, y) + 0.1)
                xs = np.abs(xs)
            rho = 1.4 * (1 + _waves(rng, xs, ys, amp))
            p = 1.0 + _waves(rng, xs, ys, amp)
            u = mach * (1 + _waves(rng, xs, ys, amp))
            v = (0.014 if kind == "naca" else 0.0) + mach * _waves(rng, xs, ys, amp)
            if kind == "step":  # a shock ahead of the step
                m = x > 0.45 + 0.3 * (y - rng.uniform(0.3, 0.5)) ** 2
                rho, p, u = np.where(m, 1.6 * rho, rho), np.where(m, 2.0 * p, p), np.where(m, 0.85 * u, u)
        out.append(np.stack([rho, rho * u, rho * v, p / 0.4 + 0.5 * rho * (u * u + v * v)], 1))
    # reference numbering of a batch: the real cells of every case, then every case's ghosts
    n = [em.cells.shape[0] for em in ems]
    return np.ascontiguousarray(np.concatenate([o[:k] for o, k in zip(out, n)] + [o[k:] for o, k in zip(out, n)]))


def _theta(seed):
    rng = np.random.default_rng([seed, 23])
    return np.concatenate([[3.0 + rng.uniform(-0.05, 0.05)], rng.normal(0.0, 0.01, N_BINS)])


# -------------------------------------------------------------- the passes --
def prepare(case, seed):
    ems = _meshes(case, seed)
    ph = _physics(case, ems)
    mesh = [fvgpu.Mesh.from_elements(em) for em in ems]
    mesh = fvgpu.Mesh.batch(mesh) if case["kind"] == "strips" else mesh[0]
    if case["kind"] == "adjoint":
        adj = fvgpu.Adjoint(mesh, ph, case["steps"], checkpoint_every=10, n_bins=N_BINS)
        return {"case": case, "adjoint": adj, "theta": _theta(seed)}
    solver = fvgpu.Solver(mesh, ph, case["precision"])
    q = _initial(case, ems, seed)
    st = {"case": case, "solver": solver, "alpha": _alpha(case)}
    if case["host"]:
        st["q"] = q.ravel()
        return st
    # device arrays and one stream for the solver and the program's own work
    st["stream"] = torch.cuda.Stream()
    solver.set_stream(st["stream"].cuda_stream)
    st["q"] = torch.from_numpy(q).cuda()
    st["out"] = torch.empty_like(st["q"])
    # FP32-bulk results carry single precision: the program keeps them so
    st["out32"] = torch.empty_like(st["q"], dtype=torch.float32) if case["precision"] == "fp32" else None
    return st


def run(state):
    case = state["case"]
    if "adjoint" in state:
        loss, grad = state["adjoint"].gradient(state["theta"])
        return {"loss": np.array([loss]), "grad": grad}
    s, single = state["solver"], case["precision"] == "fp32"
    kept = np.float32 if single else np.float64
    if case["host"]:
        s.set_state(state["q"])
        info = s.run(case["steps"], alpha=state["alpha"])
        q = s.get_state().astype(kept, copy=False)
    else:
        s.set_state_ptr(state["q"].data_ptr(), device=True)
        info = s.run(case["steps"], alpha=state["alpha"])
        s.get_state_ptr(state["out"].data_ptr(), device=True)
        q = state["out"]
        if single:
            with torch.cuda.stream(state["stream"]):
                q = state["out32"].copy_(q)
    times = s.case_times() if case["kind"] == "strips" else np.array([info["time"]])
    return {"q": q, "R": info["R"].astype(kept), "times": times.astype(kept)}


# ------------------------------------------------------- the 64-bit answer --
class _Geometry:
    """Edges, normals, areas, centroids and Green-Gauss weights of an element
    mesh: the first cell of an edge is the lower-numbered one, boundary
    segment b's ghost is cell n + b, mirrored across the edge."""

    def __init__(self, ems, dev):
        offs, c0, b0 = [], 0, 0
        nodes, cells, seg, grp, case = [], [], [], [], []
        for k, em in enumerate(ems):
            base = sum(v.shape[1] for v in nodes)
            nodes.append(np.stack([em.nodes_x, em.nodes_y]))
            cells.append(np.where(em.cells < 0, -1, em.cells.astype(np.int64) + base))
            seg.append(em.bnd_nodes.astype(np.int64) + base)
            grp.append(em.bnd_group)
        self.names = ems[0].group_names
        X = torch.from_numpy(np.concatenate(nodes, 1)).to(dev)
        C = torch.from_numpy(np.concatenate(cells)).to(dev)
        S = torch.from_numpy(np.concatenate(seg)).to(dev)
        self.group = torch.from_numpy(np.concatenate(grp).astype(np.int64)).to(dev)
        per = [(em.cells.shape[0], em.bnd_nodes.shape[0]) for em in ems]
        ids = torch.arange(len(ems), device=dev)
        self.case = torch.cat([torch.repeat_interleave(ids, torch.tensor([p[i] for p in per], device=dev))
                               for i in (0, 1)])
        n, nb = C.shape[0], S.shape[0]
        tri = C[:, 3] < 0
        self.n, self.nb, self.nf = n, nb, torch.where(tri, 3.0, 4.0).to(X.dtype)
        side = [torch.stack([C[:, 0], C[:, 1]]), torch.stack([C[:, 1], C[:, 2]]),
                torch.stack([C[:, 2], torch.where(tri, C[:, 0], C[:, 3])]), torch.stack([C[~tri, 3], C[~tri, 0]])]
        owner = torch.cat([torch.arange(n, device=dev).repeat(3), torch.arange(n, device=dev)[~tri]])
        ab = torch.cat(side, 1)
        big = X.shape[1] + 1
        key = ab.min(0).values * big + ab.max(0).values
        uniq, inv = torch.unique(key, return_inverse=True)
        E = uniq.numel()
        i = torch.full((E,), n, device=dev).scatter_reduce(0, inv, owner, "amin")
        j = torch.full((E,), -1, device=dev).scatter_reduce(0, inv, owner, "amax")
        be = torch.searchsorted(uniq, S.min(1).values * big + S.max(1).values)
        j[be] = n + torch.arange(nb, device=dev)
        a, b = uniq // big, uniq % big
        mid, d = 0.5 * (X[:, a] + X[:, b]), X[:, b] - X[:, a]
        self.le = torch.sqrt((d * d).sum(0))
        nrm = torch.stack([-d[1], d[0]]) / self.le
        c4 = torch.where(C < 0, C[:, :1], C)
        cc = (X[:, c4[:, 0]] + X[:, c4[:, 1]] + X[:, c4[:, 2]] + torch.where(tri, 0.0, X[:, c4[:, 3]])) / self.nf
        nrm = torch.where(((mid - cc[:, i]) * nrm).sum(0) < 0, -nrm, nrm)
        p = [X[:, c4[:, k]] for k in range(4)]
        tri_area = lambda u, v, w: 0.5 * torch.abs((v - u)[0] * (w - u)[1] - (w - u)[0] * (v - u)[1])  # noqa: E731
        area = tri_area(p[0], p[1], p[2]) + torch.where(tri, 0.0, tri_area(p[0], p[2], p[3]))
        gi = i[be]
        dist = torch.sqrt(((mid[:, be] - cc[:, gi]) ** 2).sum(0))
        self.cc = torch.cat([cc, mid[:, be] + dist * nrm[:, be]], 1)
        self.area = torch.cat([area, area[gi]])
        self.i, self.j, self.nrm, self.mid, self.be, self.gi = i, j, nrm, mid, be, gi
        self.g = torch.sqrt(((mid - self.cc[:, i]) ** 2).sum(0)) / torch.sqrt(((self.cc[:, i] - self.cc[:, j]) ** 2).sum(0))
        self.di, self.dj = mid - self.cc[:, i], mid - self.cc[:, j]


def _pressure(q, gm1=0.4):
    return gm1 * (q[3] - 0.5 / q[0] * (q[1] * q[1] + q[2] * q[2]))


def _roe(ph, a, b, n):
    gm1 = ph.gamma - 1
    pL, pR = _pressure(a, gm1), _pressure(b, gm1)
    uL, vL, uR, vR = a[1] / a[0], a[2] / a[0], b[1] / b[0], b[2] / b[0]
    VL, VR = uL * n[0] + vL * n[1], uR * n[0] + vR * n[1]
    sL, sR = torch.sqrt(a[0]), torch.sqrt(b[0])
    rho, w = sL * sR, sL + sR
    u, v = (uL * sL + uR * sR) / w, (vL * sL + vR * sR) / w
    h = ((a[3] + pL) / a[0] * sL + (b[3] + pR) / b[0] * sR) / w
    q2 = u * u + v * v
    c = torch.sqrt(gm1 * (h - 0.5 * q2))
    V = u * n[0] + v * n[1]
    l1, l2, l5 = torch.abs(torch.minimum(V - c, VL - c)), torch.abs(V), torch.abs(torch.maximum(V + c, VR + c))
    dp, dV = pR - pL, VR - VL
    k1, k0 = l1 * (dp - rho * c * dV) / (2 * c * c), l2 * ((b[0] - a[0]) - dp / (c * c))
    kr, k5 = l2 * rho, l5 * (dp + rho * c * dV) / (2 * c * c)
    return torch.stack([
        0.5 * (a[0] * VL + b[0] * VR) - 0.5 * (k1 + k0 + k5),
        0.5 * (a[1] * VL + b[1] * VR + (pL + pR) * n[0])
        - 0.5 * (k1 * (u - c * n[0]) + k0 * u + kr * (uR - uL - dV * n[0]) + k5 * (u + c * n[0])),
        0.5 * (a[2] * VL + b[2] * VR + (pL + pR) * n[1])
        - 0.5 * (k1 * (v - c * n[1]) + k0 * v + kr * (vR - vL - dV * n[1]) + k5 * (v + c * n[1])),
        0.5 * ((a[3] + pL) * VL + (b[3] + pR) * VR)
        - 0.5 * (k1 * (h - c * V) + k0 * q2 * 0.5 + kr * (u * (uR - uL) + v * (vR - vL) - V * dV) + k5 * (h + c * V))])


def _phi(ph, y):
    if ph.limiter == "venkat":
        return (y * y + 2 * y) / (y * y + y + 2)
    if ph.limiter == "michalak":
        return torch.where(y >= 2, 1.0, y - 0.25 * y * y)
    return torch.clamp(y, 0.0, 1.0)


def _boundary(ph, G, bv, q):
    """Ghost states from the interior face states q [V][ghosts]."""
    n, out = G.nrm[:, G.be], torch.zeros_like(q)
    for k, name in enumerate(G.names):
        kind = ph.bcs[name][0]
        m = G.group == k
        if not bool(m.any()):
            continue
        x, nn = q[:, m], n[:, m]
        if kind == "copy":
            b = x
        elif kind == "tangent":
            b = torch.stack([-nn[1], nn[0]])
        elif kind == "wall":
            d = 2 * (nn[0] * x[1] + nn[1] * x[2])
            b = torch.stack([x[0], x[1] - nn[0] * d, x[2] - nn[1] * d, x[3]])
        elif kind == "noslip":
            b = torch.stack([x[0], -x[1], -x[2], x[3]])
        else:
            f, gm1 = bv[:, m], ph.gamma - 1
            u, v = x[1] / x[0], x[2] / x[0]
            un, p = u * nn[0] + v * nn[1], _pressure(x, gm1)
            c = torch.sqrt(ph.gamma * p / x[0])
            pa, ua, va = _pressure(f, gm1), f[1] / f[0], f[2] / f[0]
            energy = lambda pb, r, m1, m2: pb / gm1 + 0.5 / r * (m1 * m1 + m2 * m2)  # noqa: E731
            rc = x[0] * c
            if kind == "inlet_outlet":
                sub_in = torch.stack([f[0], f[1], f[2], energy(p, f[0], f[1], f[2])])
            else:
                pb = 0.5 * (pa + p - rc * (nn[0] * (ua - u) + nn[1] * (va - v)))
                r = f[0] + (pb - pa) / (c * c)
                m1 = r * (ua - nn[0] * (pa - pb) / rc)
                m2 = (r if kind == "farfield_b0" else m1) * (va - nn[1] * (pa - pb) / rc)
                sub_in = torch.stack([r, m1, m2, energy(pb, r, m1, m2)])
            r = x[0] + (pa - p) / (c * c)
            m1 = r * (u + nn[0] * (p - pa) / rc)
            m2 = (r if kind == "farfield_b0" else m1) * (va + nn[1] * (p - pa) / rc)
            sub_out = torch.stack([r, m1, m2, energy(pa, r, m1, m2)])
            sup = u * u + v * v > c * c
            b = torch.where(un < 0, torch.where(sup, f, sub_in), torch.where(sup, x, sub_out))
        out = out.index_copy(1, torch.nonzero(m)[:, 0], b)
    return out


def _guarded(ph, face, cell):
    if not ph.positivity_guard:
        return face
    bad = ~(face[0] > 0) | ~(_pressure(face, ph.gamma - 1) > 0)
    return torch.where(bad, cell, face)


def _time_steps(ph, G, q):
    """dt of every cell and ghost."""
    if ph.dt_kind == "const":
        return torch.full_like(G.area, ph.dt_const)
    u, v = q[1] / q[0], q[2] / q[0]
    c = torch.sqrt(ph.gamma * _pressure(q, ph.gamma - 1) / q[0])
    i, j, n, le, A = G.i, G.j, G.nrm, G.le, G.area
    if ph.dt_kind in ("cfl_sum", "visc_sum"):
        s = [c[k] + torch.abs(u[k] * n[0] + v[k] * n[1]) for k in (i, j)]
        if ph.dt_kind == "visc_sum":
            s = [e + 2 * torch.clamp(torch.tensor(ph.gamma), min=4 / 3).item() / q[0][k] * (ph.mu / ph.pr) * le * le / A[k]
                 for e, k in zip(s, (i, j))]
        w = torch.maximum(s[0], s[1]) * le
        return ph.cfl * A / torch.zeros_like(A).index_add(0, i, w).index_add(0, j, w)
    dt = torch.ones_like(A)
    for k in (i, j):
        if ph.dt_kind == "cfl_min_signed":
            e = (c[k] + torch.abs(u[k])) * n[0] + (c[k] + torch.abs(v[k])) * n[1]
            d = ph.cfl * (A[k] / le) / torch.abs(e)
        else:
            e = (c[k] + torch.abs(n[0] * u[k]) + torch.abs(n[1] * v[k])) * le
            d = ph.cfl * A[k] / (e + 2 * max(4 / 3, ph.gamma) / q[0][k] * (ph.mu / ph.pr) * le * le / A[k])
        dt = dt.scatter_reduce(0, k, d, "amin")
    return dt


def _gradients(ph, G, q):
    """Green-Gauss gradients and limiters of the real cells (ghosts: 0 and 1)."""
    n, i, j = G.n, G.i, G.j
    qi, qj = q[:, i], q[:, j]
    f = (qi * (1 - G.g) + qj * G.g) * G.le
    add = lambda w: (torch.zeros_like(q).index_add(1, i, w).index_add(1, j, -w) / G.area)[:, :n]  # noqa: E731
    gx, gy = add(f * G.nrm[0]), add(f * G.nrm[1])
    lim = torch.ones_like(gx)
    if ph.order2:
        ext = lambda how: q.scatter_reduce(1, i.expand_as(qj), qj, how).scatter_reduce(  # noqa: E731
            1, j.expand_as(qi), qi, how)[:, :n]
        mx, mn, qc = ext("amax"), ext("amin"), q[:, :n]
        K3 = (ph.K * torch.sqrt(G.area[:n])) ** 3
        d2 = (mx - mn) ** 2
        y = d2 / K3 - 1
        sig = torch.where(d2 <= K3, 1.0, torch.where(d2 <= 2 * K3, 2 * y ** 3 - 3 * y ** 2 + 1, 0.0))
        for k, d in ((i, G.di), (j, G.dj)):
            m = k < n
            k, d = k[m], d[:, m]
            dq = gx[:, k] * d[0] + gy[:, k] * d[1]
            num = torch.where(dq > 0, mx[:, k] - qc[:, k], mn[:, k] - qc[:, k])
            tiny = torch.abs(dq) <= 1e-15
            y = num / torch.where(tiny, 1.0, dq)
            lv = torch.where(tiny | (sig[:, k] >= 1), 1.0, _phi(ph, y))
            lv = sig[:, k] + (1 - sig[:, k]) * lv
            lim = lim.scatter_reduce(1, k.expand_as(lv), lv, "amin")
    pad = lambda t, v: torch.cat([t, torch.full_like(q[:, n:], v)], 1)  # noqa: E731
    return pad(gx, 0.0), pad(gy, 0.0), pad(lim, 1.0)


def _face_gradient(G, q, gx, gy):
    i, j = G.i, G.j
    t = G.cc[:, i] - G.cc[:, j]
    length = torch.sqrt((t * t).sum(0))
    t = t / length
    bx, by = 0.5 * (gx[:, i] + gx[:, j]), 0.5 * (gy[:, i] + gy[:, j])
    corr = bx * t[0] + by * t[1] - (q[:, i] - q[:, j]) / length
    return bx - corr * t[0], by - corr * t[1]


def _viscous(ph, a, b, gx, gy, n):
    q = 0.5 * (a + b)
    u, v, E, r = q[1] / q[0], q[2] / q[0], q[3] / q[0], q[0]
    ux, uy = (gx[1] - u * gx[0]) / r, (gy[1] - u * gy[0]) / r
    vx, vy = (gx[2] - v * gx[0]) / r, (gy[2] - v * gy[0]) / r
    cT = (ph.gamma - 1) / ph.r
    tx = cT * ((gx[3] - E * gx[0]) / r - (u * ux + v * vx))
    ty = cT * ((gy[3] - E * gy[0]) / r - (u * uy + v * vy))
    div = ux + vy
    txx, tyy, txy = 2 * ph.mu * (ux - div / 3), 2 * ph.mu * (vy - div / 3), ph.mu * (uy + vx)
    k = ph.cp * ph.mu / ph.pr
    f1, f2 = u * txx + v * txy + k * tx, u * txy + v * tyy + k * ty
    z = torch.zeros_like(f1)
    return torch.stack([z, n[0] * txx + n[1] * txy, n[0] * txy + n[1] * tyy, n[0] * f1 + n[1] * f2])


def _stage(ph, G, q):
    """Time derivatives of the real cells, with the gradients and limiters."""
    i, j, n = G.i, G.j, G.n
    gx = gy = lim = None
    if ph.order2 or ph.diffusive:
        gx, gy, lim = _gradients(ph, G, q)
    a, b = q[:, i], q[:, j]
    if ph.order2:
        a = _guarded(ph, a + (gx[:, i] * G.di[0] + gy[:, i] * G.di[1]) * lim[:, i], a)
        b = _guarded(ph, b + (gx[:, j] * G.dj[0] + gy[:, j] * G.dj[1]) * lim[:, j], b)
    if ph.diffusive:
        fx, fy = _face_gradient(G, q, gx, gy)
    if ph.flux == "diffusion":
        F = -(fx * G.nrm[0] + fy * G.nrm[1])
    elif ph.flux == "burgers_diffusion":
        Va, Vb = (w[0] * G.nrm[0] + w[1] * G.nrm[1] for w in (a, b))
        F = 0.5 * (Va * a + Vb * b) - 0.5 * torch.maximum(torch.abs(Va), torch.abs(Vb)) * (b - a)
        F = F - (fx * G.nrm[0] + fy * G.nrm[1])
    else:
        F = _roe(ph, a, b, G.nrm)
        if ph.flux == "ns":
            F = F - _viscous(ph, a, b, fx, fy, G.nrm)
    F = F * G.le
    qt = (torch.zeros_like(q).index_add(1, i, -F).index_add(1, j, F) / G.area)[:, :n]
    if ph.smooth:
        q0, inner = qt, j < n
        for _ in range(2):
            s = torch.zeros_like(qt).index_add(1, i[inner], qt[:, j[inner]]).index_add(1, j[inner], qt[:, i[inner]])
            qt = (q0 + 0.6 * s) / (1 + 0.6 * G.nf)
    return qt, gx, gy, lim


def _filled(ph, G, bv, real, gx=None, gy=None, lim=None):
    """The state with its ghosts filled from the interior face states."""
    c = real[:, G.gi]
    face = c
    if ph.order2 and gx is not None:
        d = G.mid[:, G.be] - G.cc[:, G.gi]
        face = _guarded(ph, c + (gx[:, G.gi] * d[0] + gy[:, G.gi] * d[1]) * lim[:, G.gi], c)
    return torch.cat([real, _boundary(ph, G, bv, face)], 1)


def _loop(ph, G, bv, q, alpha, steps, at_start=None):
    """The time loop; returns the state, the residual norms and the times of the cases."""
    cases = int(G.case.max()) + 1
    times = torch.zeros(cases, dtype=q.dtype, device=q.device)
    first = [int(torch.nonzero(G.case[:G.n] == k)[0, 0]) for k in range(cases)]
    q, R, R0 = _filled(ph, G, bv, q[:, :G.n]), None, None
    for step in range(steps):
        dt = _time_steps(ph, G, q)
        if ph.global_dt:
            least = torch.stack([dt[G.case == k].min() for k in range(cases)])
            times = times + least
            dt = least[G.case]
        else:
            times = times + dt[first]
        if at_start is not None:
            at_start(q, times, dt)
        base, x = q[:, :G.n], q
        for a in alpha:
            qt, gx, gy, lim = _stage(ph, G, x)
            x = _filled(ph, G, bv, base + qt * dt[:G.n] * a, gx, gy, lim)
        R = torch.sqrt((qt * qt * G.area[:G.n]).sum(1))
        R0 = R if step == 0 else R0
        R = R if step == 0 else R / R0
        q = x
    return q, R, times


def _far_field(ph, G, like):
    bv = torch.zeros(4, G.nb, dtype=like.dtype, device=like.device)
    for k, name in enumerate(G.names):
        if ph.bcs[name][1] is not None:
            bv[:, G.group == k] = torch.tensor(ph.bcs[name][1], dtype=like.dtype, device=like.device)[:, None]
    return bv


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    ems = _meshes(case, seed)
    ph, G = _physics(case, ems), _Geometry(ems, dev)
    if case["kind"] == "adjoint":
        return _exact_adjoint(case, seed, ph, G, dev)
    with torch.no_grad():
        q = torch.from_numpy(_initial(case, ems, seed)).to(dev).T.contiguous()
        q, R, times = _loop(ph, G, _far_field(ph, G, q) if ph.V == 4 else None, q, _alpha(case), case["steps"])
    q = q.T.contiguous()
    return {"q": q.cpu().numpy().ravel() if case["host"] else q, "R": R.cpu().numpy(), "times": times.cpu().numpy()}


def _exact_adjoint(case, seed, ph, G, dev):
    """Loss and gradient by reverse-mode differentiation of the loop above."""
    theta = torch.tensor(_theta(seed), dtype=torch.float64, device=dev, requires_grad=True)
    far, gm1 = ph.bcs["inlet"][1], ph.gamma - 1
    rho0 = far[0]
    p0 = gm1 * (far[3] - 0.5 * (far[1] ** 2 + far[2] ** 2) / far[0])
    mach, flow = theta[0], [k for k, s in enumerate(G.names) if ph.bcs[s][0] == "inlet_outlet"]
    y = G.mid[1, G.be]
    bins = torch.clamp(torch.floor(y * N_BINS), 0, N_BINS - 1).long()
    rho = torch.full_like(y, rho0)
    rho = torch.where(G.group == G.names.index("inlet"), rho0 * (1 + theta[1 + bins]), rho)
    bv = torch.stack([rho, rho * mach, torch.zeros_like(rho), p0 / gm1 + 0.5 * rho * mach * mach])
    bv = torch.where(functools.reduce(torch.logical_or, [G.group == k for k in flow]), bv, 0.0)
    one = torch.ones(G.n + G.nb, dtype=torch.float64, device=dev)
    q = torch.stack([rho0 * one, rho0 * mach * one, 0 * one, (p0 / gm1 + 0.5 * rho0 * mach * mach) * one])
    face = G.group == G.names.index("step")
    cell, le, loss = G.gi[face], G.le[G.be[face]], []

    def at_start(state, times, dt):
        loss.append(dt[0] * (_pressure(state[:, cell], gm1) * le).sum())

    _loop(ph, G, bv, q, _alpha(case), case["steps"], at_start)
    total = sum(loss)
    grad, = torch.autograd.grad(total, theta)
    return {"loss": total.detach().reshape(1).cpu().numpy(), "grad": grad.cpu().numpy()}
