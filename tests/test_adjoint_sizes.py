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
