"""Tiles whose shared memory lies at the limit of the run kernel: loose patches
of a few cells, whose boundary ghosts, slots and flux edges fill it."""
import numpy as np
import pytest

import fvgpu
import meshgen
import physics as P
from test_run_kernel import bits_equal, euler, smooth_state

pytestmark = pytest.mark.gpu


def patches(shapes):
    """Separate grids of m x n quadrilaterals, in rows of eight."""
    xs, ys, cells, seg, base = [], [], [], [], 0
    for d, (m, n) in enumerate(shapes):
        I, J = np.meshgrid(np.arange(m + 1), np.arange(n + 1))
        xs.append(0.125 * (d % 8) + 0.03 * I.ravel())
        ys.append(0.125 * (d // 8) + 0.03 * J.ravel())
        w = m + 1
        a = base + (np.arange(n)[:, None] * w + np.arange(m)[None]).ravel()
        cells.append(np.stack([a, a + 1, a + w + 1, a + w], 1))
        e, f = base + np.arange(m), base + np.arange(n) * w
        seg += [np.stack(s, 1) for s in ((e, e + 1), (e + n * w, e + n * w + 1), (f, f + w), (f + m, f + m + w))]
        base += w * (n + 1)
    seg = np.concatenate(seg).astype(np.int32)
    return meshgen.ElementMesh(np.concatenate(xs), np.concatenate(ys), np.concatenate(cells).astype(np.int32), seg,
                               np.zeros(len(seg), np.int32), ["wall"])


# one tile of Navier-Stokes in FP64: 240 bytes per boundary face, 256 per cell
# and 45,056 more.  The first has 232,256 bytes, which only the kernel's static
# variables push over 227 KB (232,448); the others lie well below and above
@pytest.mark.parametrize("shapes, run_kernel", [([(2, 2)] * 57 + [(3, 2)] * 4 + [(1, 1)] * 3, False),
                                                ([(2, 2)] * 50 + [(3, 2)] * 4 + [(1, 1)] * 3, True),
                                                ([(2, 2)] * 59 + [(1, 1)] * 19, False)])
def test_run_kernel_or_separate_kernels(shapes, run_kernel):
    mesh = fvgpu.Mesh.from_elements(patches(shapes))
    assert mesh.n_real <= 256
    ph = euler(True)
    ph.flux, ph.diffusive = "ns", True
    ph.dt_kind, ph.mu, ph.pr, ph.cp, ph.r = "visc_sum", 2e-3, 0.72, 3.5, 1.0
    q0 = smooth_state(mesh.geometry())
    out = []
    for sk in ("auto", "split"):
        s = fvgpu.Solver(mesh, ph, "fp64", tile_cells=256, stage_kernels=sk)
        s.set_state(q0)
        s.run(4, alpha=P.RK5_ALPHA)
        out.append((s.get_state(), s.last_run_stats()[1] <= 2))
    assert [x[1] for x in out] == [run_kernel, False]
    if run_kernel:  # other formulas: a few ulps per stage
        a, b = (x[0].reshape(-1, 4) for x in out)
        assert np.all(np.abs(a - b).max(0) <= 1e-12 * np.abs(b).max(0))
    else:
        assert bits_equal(out[0][0], out[1][0])


def test_no_arrays_for_a_run_kernel_that_has_no_room():
    """120,000 Navier-Stokes cells in FP64, beyond the run kernel: the default
    layout holds what the split layout holds (the run kernel's records would be
    some 60 MB)."""
    import torch

    n, m = 400, 300
    J, I = np.meshgrid(np.arange(m + 1), np.arange(n + 1), indexing="ij")
    a = (np.arange(m)[:, None] * (n + 1) + np.arange(n)[None]).ravel()
    e, f = np.arange(n), np.arange(m) * (n + 1)
    seg = np.concatenate([np.stack(s, 1) for s in ((e, e + 1), (e + m * (n + 1), e + m * (n + 1) + 1), (f, f + n + 1),
                                                  (f + n, f + 2 * n + 1))]).astype(np.int32)
    em = meshgen.ElementMesh(I.ravel() / n, J.ravel() / m, np.stack([a, a + 1, a + n + 2, a + n + 1], 1).astype(np.int32),
                             seg, np.zeros(len(seg), np.int32), ["wall"])
    mesh = fvgpu.Mesh.from_elements(em)
    ph = euler(True)
    ph.flux, ph.diffusive = "ns", True
    ph.dt_kind, ph.mu, ph.pr, ph.cp, ph.r = "visc_sum", 2e-3, 0.72, 3.5, 1.0

    def held(layout):
        before = torch.cuda.mem_get_info()[0]
        s = fvgpu.Solver(mesh, ph, "fp64", stage_kernels=layout)
        used = before - torch.cuda.mem_get_info()[0]
        s.close()
        return used

    held("split")  # (kernels loaded)
    held("auto")
    assert abs(held("auto") - held("split")) <= 4 << 20
