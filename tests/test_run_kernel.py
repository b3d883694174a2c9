"""The persistent run kernel (all steps of a run in one cooperative launch, for
meshes whose tiles fit the device at once) against the separate kernels of the
split layout, which take the same faces and cells through the same arithmetic:
the states have the same bits.  Residual norms are reduced in another order
over the tiles, so within 1e-12 relative, as against the oracle.  The
Navier-Stokes kind computes its gradients by other (equivalent) formulas: a few
ulps per stage, 1e-12 over the steps taken here."""
import numpy as np
import pytest

import fvgpu
import meshgen
import physics as P
from cases import CASES, random_euler_state
from test_mixed_elements import mixed_strip

pytestmark = pytest.mark.gpu

R_RTOL = 1e-12
PRECISIONS = ("fp64_exact", "fp64", "fp32")
ROE = [n for n in sorted(CASES) if CASES[n]["phys"]().V == 4 and CASES[n]["phys"]().flux in ("roe_fs", "roe_st")
       and CASES[n]["phys"]().dt_kind in ("const", "cfl_sum", "cfl_min_signed")]


def bits_equal(a, b):
    a = np.ascontiguousarray(a); b = np.ascontiguousarray(b)
    return a.shape == b.shape and a.tobytes() == b.tobytes()


def euler(order2, global_dt=True):
    return P.Physics(V=4, flux="roe_fs", order2=order2, limiter="venkat" if order2 else "zero",
                     K=5.0 if order2 else 7.5, dt_kind="cfl_sum", cfl=0.5, global_dt=global_dt,
                     bcs={"wall": ("wall", None), "ends": ("copy", None)})


def smooth_state(g):
    """A smooth field with gradients everywhere, ghosts included."""
    x, y = np.asarray(g["ccx"]), np.asarray(g["ccy"])
    rho = 1.0 + 0.3 * np.sin(9 * x + 1) * np.cos(7 * y)
    u, v, p = 0.4 * np.cos(5 * x), 0.3 * np.sin(6 * y + x), 1.0 + 0.2 * np.cos(8 * x * y + 1)
    return np.stack([rho, rho * u, rho * v, p / 0.4 + 0.5 * rho * (u * u + v * v)], 1).ravel()


def pair(mesh, ph, precision, tile_cells=0):
    """(solver on the run kernel, solver on separate kernels)"""
    return (fvgpu.Solver(mesh, ph, precision, tile_cells=tile_cells),
            fvgpu.Solver(mesh, ph, precision, tile_cells=tile_cells, stage_kernels="split"))


def compare(a, b, q0, steps, alpha, same=bits_equal, separate=False, **kw):
    """separate: both run separate kernels (FP32 in first order)"""
    out = []
    for s in (a, b):
        s.set_state(q0)
        r = s.run(steps, alpha=alpha, **kw)
        out.append((s.get_state(), r, s.last_run_stats()[1]))
    (qa, ra, la), (qb, rb, lb) = out
    if separate:
        assert la == lb
    else:
        assert la <= 2 * (1 + steps // 2048) and (la < lb or ra["step"] == 0)      # one cooperative launch against kernels per stage
    assert ra["step"] == rb["step"]
    assert same(qa, qb)
    np.testing.assert_allclose(ra["time"], rb["time"], rtol=0 if same is bits_equal else 1e-12, atol=0)
    np.testing.assert_allclose(ra["R"], rb["R"], rtol=R_RTOL if same is bits_equal else 1e-9, atol=0)
    return ra


@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("name", ROE)
def test_same_bits_as_separate_kernels(name, precision, oracle):
    case = CASES[name]
    em = case["mesh"]()
    mesh = fvgpu.Mesh.from_elements(em)
    q0 = case["ic"](oracle.build_mesh(em))
    for tile_cells in (0, 64):
        ph = case["phys"]()
        compare(*pair(mesh, ph, precision, tile_cells), q0, case["steps"], case["alpha"],
                separate=precision == "fp32" and not ph.order2)


# cells: fewer than one tile, exactly one, one and two cells, a partial last
# tile, more than one tile per SM and (FP64, FP32) more than two, where
# the kernel with fewer threads or registers takes over
@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("order2", (False, True))
@pytest.mark.parametrize("nx, ny", [(1, 1), (8, 8), (13, 5), (31, 23), (130, 130), (180, 180)])
def test_sizes(nx, ny, order2, precision):
    mesh = fvgpu.Mesh.from_elements(meshgen.rect_tri(nx, ny, 1.0, 0.8))
    q0 = smooth_state(mesh.geometry())
    for alpha in (P.RK1_ALPHA, P.RK5_ALPHA):
        compare(*pair(mesh, euler(order2, global_dt=nx != 31), precision), q0, 5, alpha,
                separate=precision == "fp32" and not order2)


@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("order2", (False, True))
def test_quadrilaterals(order2, precision):
    mesh = fvgpu.Mesh.from_elements(mixed_strip())
    compare(*pair(mesh, euler(order2), precision), smooth_state(mesh.geometry()), 12, P.RK5_ALPHA,
            separate=precision == "fp32" and not order2)


@pytest.mark.parametrize("order2", (False, True))
@pytest.mark.parametrize("nx, ny", [(3, 2), (24, 16), (130, 130)])
def test_navier_stokes(nx, ny, order2):
    mesh = fvgpu.Mesh.from_elements(meshgen.rect_tri(nx, ny, 1.0, 0.8))
    for dt_kind in ("cfl_sum", "cfl_min_signed", "visc_min", "visc_sum"):
        ph = euler(order2, global_dt=dt_kind != "visc_min")
        ph.flux, ph.diffusive = "ns", True
        ph.dt_kind, ph.mu, ph.pr, ph.cp, ph.r = dt_kind, 2e-3, 0.72, 3.5, 1.0

        def same(a, b):
            a, b = a.reshape(-1, 4), b.reshape(-1, 4)
            return np.all(np.abs(a - b).max(0) <= 1e-12 * np.abs(b).max(0))
        compare(*pair(mesh, ph, "fp64"), smooth_state(mesh.geometry()), 6, P.RK5_ALPHA, same=same)


@pytest.mark.parametrize("precision", PRECISIONS)
def test_navier_stokes_plate(precision, oracle):
    """Graded cells, inflow, outflow and no-slip ghosts; FP64 alone has a run
    kernel for it, the others keep the separate kernels."""
    case = CASES["flat_plate"]
    em = case["mesh"]()
    mesh = fvgpu.Mesh.from_elements(em)
    s = fvgpu.Solver(mesh, case["phys"](), precision)
    s.set_state(case["ic"](oracle.build_mesh(em)))
    s.run(8, alpha=case["alpha"])
    assert (s.last_run_stats()[1] <= 2) == (precision == "fp64")


@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("name", ("sod", "step_o2_venk5"))
def test_stops_records_and_continuation(name, precision, oracle):
    case = CASES[name]
    em = case["mesh"]()
    mesh = fvgpu.Mesh.from_elements(em)
    q0 = case["ic"](oracle.build_mesh(em))
    a, b = pair(mesh, case["phys"](), precision)
    b.set_state(q0)
    full = b.run(11, alpha=case["alpha"])
    t5 = []
    b.set_state(q0)
    b.run(11, alpha=case["alpha"], on_print=lambda step, t, R: t5.append((step, t, R)))
    # by time: the first step whose start is not before max_time ends the run
    sep = precision == "fp32" and name == "sod"
    r = compare(a, b, q0, 100, case["alpha"], max_time=t5[6][1], separate=sep)
    assert r["step"] == 6
    # by residual, midway between two records (a falling norm that starts at 1; else at once)
    compare(a, b, q0, 30, case["alpha"], tolerance=np.sqrt(max(t5[7][2]) * max(t5[8][2])), separate=sep)
    # records at an interval, and a run cut in three
    got, want = [], []
    a.set_state(q0)
    a.run(11, alpha=case["alpha"], print_interval=3, on_print=lambda step, t, R: got.append((step, t, R)))
    b.set_state(q0)
    b.run(11, alpha=case["alpha"], print_interval=3, on_print=lambda step, t, R: want.append((step, t, R)))
    assert [(x[0], x[1]) for x in got] == [(x[0], x[1]) for x in want]
    np.testing.assert_allclose([x[2] for x in got], [x[2] for x in want], rtol=R_RTOL, atol=0)
    whole = a.get_state()
    a.set_state(q0)
    for stop in (4, 5, 11):
        r = a.run(stop, alpha=case["alpha"], restart=stop == 4)
    assert r["step"] == 11 and r["time"] == full["time"] and bits_equal(a.get_state(), whole)
    # no step at all
    a.set_state(q0)
    assert a.run(0, alpha=case["alpha"])["step"] == 0


def test_more_steps_than_one_launch():
    mesh = fvgpu.Mesh.from_elements(meshgen.rect_tri(6, 4, 1.0, 0.8))
    r = compare(*pair(mesh, euler(False), "fp64"), smooth_state(mesh.geometry()), 2051, P.RK1_ALPHA, print_interval=100)
    assert r["step"] == 2051


@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("tile_cells", (0, 64))
def test_batch(tile_cells, precision):
    meshes = [fvgpu.Mesh.from_elements(meshgen.riemann_strip(nx, 2)) for nx in (40, 7, 64, 33, 1)]
    mesh = fvgpu.Mesh.batch(meshes)
    q0 = smooth_state(mesh.geometry())
    a, b = pair(mesh, euler(False), precision, tile_cells)
    compare(a, b, q0, 9, P.RK1_ALPHA, separate=precision == "fp32")
    assert bits_equal(a.case_times(), b.case_times())


@pytest.mark.parametrize("order2", (False, True))
@pytest.mark.parametrize("scale", (1e-300, 1e-160, 1e-40, 1e40, 1e150, 1e300))
def test_exact_quotients_out_of_range(scale, order2, oracle):
    """FP64_EXACT's quotients are corrected estimates where the operands allow
    them and plain divisions elsewhere: the oracle's bits at any magnitude.
    (NaNs are compared as such: their payloads are the machine's.)"""
    em = mixed_strip()
    ph = euler(order2)
    g = oracle.build_mesh(em)
    q0 = random_euler_state(g.n_total, 7).reshape(-1, 4) * np.where(np.arange(g.n_total) % 3 == 0, scale, 1.0)[:, None]
    with np.errstate(all="ignore"):
        want = oracle.run_loop(g, oracle.physics(ph, em.group_names), q0.ravel(), P.RK1_ALPHA, 2)["q"]
    s = fvgpu.Solver(fvgpu.Mesh.from_elements(em), ph, "fp64_exact")
    s.set_state(q0.ravel())
    s.run(2, alpha=P.RK1_ALPHA, tolerance=-1.0)
    got = s.get_state()
    nan = np.isnan(want)
    assert np.array_equal(nan, np.isnan(got)) and bits_equal(got[~nan], want[~nan])


@pytest.mark.parametrize("precision", ("fp64", "fp32"))
@pytest.mark.parametrize("nx, ny, quads", [(1, 1, 0), (8, 8, 0), (13, 5, 0), (24, 6, 1), (130, 90, 0), (420, 260, 0)])
def test_diffusion_stencil(nx, ny, quads, precision):
    """One stencil per cell against gradients and fluxes: sums of at most a few
    dozen products of the differences between neighbouring states, so 64 ulps
    of the state's range per stage; sizes as in test_sizes, the largest beyond
    the run kernel (its stages are separate launches)."""
    em = mixed_strip(nx, ny) if quads else meshgen.rect_tri(nx, ny, 1.0, 0.8, side_names=("wall", "ends"))
    mesh = fvgpu.Mesh.from_elements(em)
    g = mesh.geometry()
    ph = P.heat(dt=0.05 * (0.2 / max(nx, ny)) ** 2)
    ph.bcs = {"wall": ("copy", None), "ends": ("copy", None)}
    x, y = np.asarray(g["ccx"]), np.asarray(g["ccy"])
    q0 = 1.0 + np.sin(9 * x + 1) * np.cos(7 * y) + (np.hypot(x - 0.5, y - 0.4) < 0.2)
    eps = 1.2e-7 if precision == "fp32" else 2.3e-16
    for alpha, steps in ((P.RK1_ALPHA, 7), (P.RK5_ALPHA, 4)):
        a, b = pair(mesh, ph, precision)
        out = []
        for s in (a, b):
            s.set_state(q0)
            r = s.run(steps, alpha=alpha)
            recs = []
            half = s.get_state()
            s.run(steps + 3, alpha=alpha, restart=False, print_interval=2, on_print=lambda n, t, R: recs.append((n, t)))
            out.append((half, s.get_state(), r, recs))
        tol = 64 * eps * (steps + 3) * len(alpha) * np.ptp(q0)
        for u, v in zip(out[0][:2], out[1][:2]):
            assert np.abs(u - v).max() <= tol
        assert out[0][2]["step"] == out[1][2]["step"] == steps and out[0][2]["time"] == out[1][2]["time"]
        assert out[0][3] == out[1][3]
        np.testing.assert_allclose(out[0][2]["R"], out[1][2]["R"], rtol=1e4 * eps)
        if mesh.n_real < 100000:
            assert a.last_run_stats()[1] <= 4


@pytest.mark.parametrize("precision", ("fp64", "fp32"))
@pytest.mark.parametrize("large", (False, True))  # True: beyond the run kernel
def test_diffusion_stops_and_batch(large, precision):
    ph = P.heat(dt=1e-7 if large else 5e-6)
    ph.bcs = {"wall": ("copy", None), "ends": ("copy", None)}
    strips = [meshgen.riemann_strip(n, 2) for n in (40, 7, 64, 1)]
    if large:
        strips += [meshgen.rect_tri(300, 280, 1.0, 0.8), meshgen.rect_tri(3, 2, 1.0, 0.8)]
    mesh = fvgpu.Mesh.batch([fvgpu.Mesh.from_elements(em) for em in strips])
    q0 = np.sin(7 * np.asarray(mesh.geometry()["ccx"]))
    eps = 1.2e-7 if precision == "fp32" else 2.3e-16
    for alpha in (P.RK1_ALPHA, P.RK5_ALPHA):
        a, b = pair(mesh, ph, precision)
        recs = []
        b.set_state(q0)
        b.run(12, alpha=alpha, on_print=lambda n, t, R: recs.append((t, R[0])))
        tol = np.sqrt(recs[8][1] * recs[9][1])
        for kw in (dict(max_time=recs[6][0]), dict(tolerance=tol), dict(max_time=0.0)):
            got = []
            for s in (a, b):
                s.set_state(q0)
                got.append((s.run(12, alpha=alpha, **kw), s.get_state(), s.case_times()))
            assert got[0][0]["step"] == got[1][0]["step"] < 12 and got[0][0]["time"] == got[1][0]["time"]
            assert np.abs(got[0][1] - got[1][1]).max() <= 64 * eps * 12 * len(alpha) * np.ptp(q0)
            assert bits_equal(got[0][2], got[1][2])
