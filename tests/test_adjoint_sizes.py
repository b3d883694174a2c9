"""The adjoint's kernels where their grids and lanes have edges: a mesh of less
than one tile, partial last blocks, several blocks; single and several stages;
first order (no gradient kernels) and both limiters.  The gradient against
central differences of the loss (h = 1e-6: truncation and rounding below 1e-8
of it; a difference interval that holds a kink of a limiter or of the arg-min
of dt departs by up to 1e-5, so 2e-5 of the norm)."""
import numpy as np
import pytest

import meshgen
import physics as P
from test_adjoint import theta0

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, alpha, order2, limiter", [(5, P.RK5_ALPHA, True, "venkat"), (5, P.RK1_ALPHA, False, "zero"),
                                                       (10, P.RK1_ALPHA, True, "michalak"), (10, P.RK5_ALPHA, False, "zero"),
                                                       (15, P.RK5_ALPHA, True, "michalak"), (25, P.RK5_ALPHA, True, "venkat")])
def test_gradient_matches_finite_differences(n, alpha, order2, limiter):
    import fvgpu

    ph = P.forward_step(order2=order2, limiter=limiter, K=5.0, cfl=0.5)
    ph.positivity_guard = True
    mesh = fvgpu.Mesh.from_elements(meshgen.forward_step(n=n))
    nb = 3
    adj = fvgpu.Adjoint(mesh, ph, n_steps=25, checkpoint_every=10, n_bins=nb, alpha=alpha)
    th = theta0(nb)
    L, g = adj.gradient(th)
    assert L == adj.loss(th)
    fd = np.zeros_like(g)
    for i in range(g.size):
        tp, tm = th.copy(), th.copy()
        tp[i] += 1e-6; tm[i] -= 1e-6
        fd[i] = (adj.loss(tp) - adj.loss(tm)) / 2e-6
    assert np.linalg.norm(g - fd) <= 2e-5 * np.linalg.norm(fd)
    adj.close()


def test_cells_with_two_common_faces():
    """Two quadrilaterals (b, a, d, c) and (b, c, e, a) with the faces a-b and b-c
    in common, in place of two triangles ahead of the step.  One of them has the
    smallest time step, whose derivative has one entry per neighbouring cell, not
    per face."""
    import fvgpu

    em = meshgen.forward_step(n=5)
    x, y = em.nodes_x, em.nodes_y
    # an inner edge of two triangles near (0.7, 0.6)
    best = None
    for i in range(em.n_cells):
        for j in range(i):
            common = np.intersect1d(em.cells[i, :3], em.cells[j, :3])
            if common.size == 2:
                d = np.hypot(x[common].mean() - 0.7, y[common].mean() - 0.6)
                if best is None or d < best[0]:
                    best = (d, i, j, common)
    _, i, j, (a, c) = best
    d, e = (np.setdiff1d(em.cells[k, :3], (a, c))[0] for k in (i, j))
    b = x.size
    em.nodes_x = np.append(x, 0.5 * (x[a] + x[c]) + 0.1 * (x[d] - x[e]))
    em.nodes_y = np.append(y, 0.5 * (y[a] + y[c]) + 0.1 * (y[d] - y[e]))
    em.cells = em.cells.copy()
    em.cells[i], em.cells[j] = (b, a, d, c), (b, c, e, a)
    mesh = fvgpu.Mesh.from_elements(em)
    ph = P.forward_step(order2=True, limiter="venkat", K=5.0, cfl=0.5)
    ph.positivity_guard = True
    s = fvgpu.Solver(mesh, ph, "fp64_exact")
    dt = s.stage_dt(P.ic_forward_step(mesh.n_total).ravel())
    assert np.argmin(dt) in (i, j)
    nb = 3
    adj = fvgpu.Adjoint(mesh, ph, n_steps=12, checkpoint_every=5, n_bins=nb, alpha=P.RK5_ALPHA)
    th = theta0(nb)
    g = adj.gradient(th)[1]
    fd = np.zeros_like(g)
    for k in range(g.size):
        tp, tm = th.copy(), th.copy()
        tp[k] += 1e-6; tm[k] -= 1e-6
        fd[k] = (adj.loss(tp) - adj.loss(tm)) / 2e-6
    assert np.linalg.norm(g - fd) <= 2e-5 * np.linalg.norm(fd)
    adj.close()
