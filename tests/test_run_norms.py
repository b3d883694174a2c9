"""Residual norms of every step of the run kernel (fv_persist.cuh) on meshes of
hundreds of tiles, one CTA each.

A step's norms are summed by every CTA from all tiles' partial sums after the CTA
has joined the next step's time-step barrier.  With a single stage the CTAs that
are ahead then store their next partial sums: `run_model` walks that order under
random interleavings, with the two sets of partial sums that the kernel keeps and,
as a control, with one."""
import random

import numpy as np
import pytest

import fvgpu
import meshgen
import physics as P
from test_run_kernel import R_RTOL, bits_equal, euler, pair, smooth_state


def run_model(n_cta, steps, sets, seed):
    """Number of reads that saw another step's partial sum."""
    rng = random.Random(seed)
    part = [[None] * n_cta for _ in range(sets)]
    arrived = [0]
    bad = [0]

    def cta(t):
        target = 0

        def arrive():
            nonlocal target
            target += n_cta
            arrived[0] += 1

        arrive()
        for n in range(steps):
            while arrived[0] < target:        # the stage's input is complete
                yield
            arrive()                          # this tile's time step is known
            if n > 0:
                for i in range(n_cta):
                    bad[0] += part[(n - 1) % sets][i] != n - 1
                    yield
            while arrived[0] < target:        # every tile's time step is known
                yield
            part[n % sets][t] = n             # update, partial sums
            yield
            arrive()

    live = [cta(t) for t in range(n_cta)]
    while live:
        # one process runs on for a while: the others lag
        g = rng.choice(live)
        for _ in range(rng.randint(1, 12)):
            if next(g, "end") == "end":
                live.remove(g)
                break
    return bad[0]


def test_partial_sums_of_a_step_stand_until_all_have_read_them():
    assert all(run_model(5, 6, 2, seed) == 0 for seed in range(100))
    assert any(run_model(5, 6, 1, seed) > 0 for seed in range(100))


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ("fp64_exact", "fp64"))
def test_every_record_of_a_single_stage_run(precision):
    mesh = fvgpu.Mesh.from_elements(meshgen.rect_tri(180, 180, 1.0, 0.8))
    assert mesh.n_real > 500 * 128
    q0 = smooth_state(mesh.geometry())
    ph = euler(False)

    def run(s, steps=150, **kw):
        recs = []
        s.set_state(q0)
        r = s.run(steps, alpha=P.RK1_ALPHA, on_print=lambda n, t, R: recs.append((n, t, tuple(R))), **kw)
        return r, recs, s.get_state()

    a, b = pair(mesh, ph, precision)
    (ra, ga, qa), (rb, gb, qb) = run(a), run(b)
    assert a.last_run_stats()[1] < b.last_run_stats()[1]
    assert [x[:2] for x in ga] == [x[:2] for x in gb] and len(ga) == 150
    np.testing.assert_allclose([x[2] for x in ga], [x[2] for x in gb], rtol=R_RTOL, atol=0)
    np.testing.assert_allclose(ra["R0"], rb["R0"], rtol=R_RTOL, atol=0)
    assert bits_equal(qa, qb)
    # twice the same, and without records (one launch)
    rc, gc, qc = run(a)
    assert ga == gc and bits_equal(ra["R"], rc["R"]) and bits_equal(qa, qc)
    a.set_state(q0)
    rd = a.run(150, alpha=P.RK1_ALPHA, tolerance=1e-300)
    assert bits_equal(ra["R"], rd["R"]) and bits_equal(ra["R0"], rd["R0"])
    # a stop by tolerance in the middle: at the first record below it
    worst = [max(x[2]) for x in ga]
    k = next(i for i in range(60, 150) if worst[i] < min(worst[1:i]))
    tol = 0.5 * (worst[k] + min(worst[1:k]))
    stops = [run(s, tolerance=tol)[0]["step"] for s in (a, b)]
    assert stops == [k + 1, k + 1]


@pytest.mark.gpu
def test_several_launches_of_many_tiles():
    """More steps than one launch takes, on some hundred CTAs."""
    mesh = fvgpu.Mesh.from_elements(meshgen.rect_tri(90, 80, 1.0, 0.8))
    q0 = smooth_state(mesh.geometry())
    out = []
    for s in pair(mesh, euler(False), "fp64"):
        s.set_state(q0)
        out.append((s.run(2100, alpha=P.RK1_ALPHA, tolerance=1e-300), s.get_state()))
    assert out[0][0]["step"] == out[1][0]["step"] == 2100 and out[0][0]["time"] == out[1][0]["time"]
    assert bits_equal(out[0][1], out[1][1])
    np.testing.assert_allclose(out[0][0]["R"], out[1][0]["R"], rtol=R_RTOL, atol=0)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ("roe", "stencil"))
def test_a_barrier_that_gives_up_is_an_error(kind):
    """No poll allowed beyond the first: the earliest CTA gives up, the others
    follow at their waits, the kernel ends and the solver serves the next run."""
    mesh = fvgpu.Mesh.from_elements(meshgen.rect_tri(130, 130, 1.0, 0.8))
    if kind == "roe":
        ph, q0 = euler(True), smooth_state(mesh.geometry())
    else:
        ph = P.heat(dt=1e-6)
        ph.bcs = {"wall": ("copy", None), "ends": ("copy", None)}
        q0 = 1 + np.sin(9 * np.asarray(mesh.geometry()["ccx"]))
    a, b = (fvgpu.Solver(mesh, ph, "fp64") for _ in range(2))
    for s in (a, b):
        s.set_state(q0)
    a.set_run_polls(0)
    with pytest.raises(fvgpu.FvError, match="gave up") as e:
        a.run(200, alpha=P.RK5_ALPHA)
    assert e.value.code == -2
    a.set_run_polls(1 << 23)
    a.set_state(q0)
    ra, rb = (s.run(20, alpha=P.RK5_ALPHA) for s in (a, b))
    assert ra["step"] == rb["step"] == 20 and ra["time"] == rb["time"]
    assert bits_equal(a.get_state(), b.get_state()) and bits_equal(ra["R"], rb["R"])
    with pytest.raises(fvgpu.FvError):
        a.set_run_polls(-1)


@pytest.mark.gpu
def test_runs_of_several_solvers_at_once():
    """Run kernels of several solvers, each on its own stream and host thread:
    a launch starts where its CTAs have room, so the runs take turns or share the
    device, with the results that each has alone."""
    import threading

    heat = P.heat(dt=1e-6)
    heat.bcs = {"wall": ("copy", None), "ends": ("copy", None)}
    jobs = []
    for nx, ny, ph, precision, alpha in ((130, 130, euler(True), "fp64", P.RK5_ALPHA), (180, 180, euler(False), "fp64", P.RK1_ALPHA),
                                         (31, 23, euler(True, global_dt=False), "fp64_exact", P.RK5_ALPHA),
                                         (130, 90, heat, "fp64", P.RK5_ALPHA)):
        mesh = fvgpu.Mesh.from_elements(meshgen.rect_tri(nx, ny, 1.0, 0.8))
        g = mesh.geometry()
        q0 = smooth_state(g) if ph is not heat else 1 + np.sin(9 * np.asarray(g["ccx"]))
        jobs.append((fvgpu.Solver(mesh, ph, precision), q0, alpha))

    def once(job):
        s, q0, alpha = job
        s.set_state(q0)
        r = s.run(40, alpha=alpha)
        return s.get_state().tobytes(), r["time"], r["R"].tobytes()

    alone = [once(j) for j in jobs]
    for s, _, _ in jobs:
        assert s.last_run_stats()[1] <= 2
    got = [[] for _ in jobs]

    def repeat(k):
        for _ in range(8):
            got[k].append(once(jobs[k]))

    threads = [threading.Thread(target=repeat, args=(k,)) for k in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k, want in enumerate(alone):
        assert len(got[k]) == 8 and all(x == want for x in got[k])
