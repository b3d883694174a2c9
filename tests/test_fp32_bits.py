"""FP32 results of the second-order Roe kinds, bit for bit.  Flows amplify
rounding: under another order of operations the state of "step" moves by 7e-5 and
its residual norms by 6e-4, so no tolerance would tell a wrong kernel from
another rounding.  fp32_bits.npz
holds the states that the split and fused kernels both gave when each formed its
faces' values q_i + (q_j - q_i) g and its Roe flux on the unit normal; recorded
on a B200 by

    PYTHONPATH=finite-volume-2d-cpp_b200:oracle python tests/test_fp32_bits.py

Residual norms are sums over the cells in an order of each layout's own: 1e-12."""
import os

import numpy as np
import pytest

import fvgpu
import meshgen
import physics as P
from test_mixed_elements import mixed_strip

GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "fp32_bits.npz")


def conservative(rho, u, v, p):
    return np.stack([rho, rho * u, rho * v, p / 0.4 + 0.5 * rho * (u * u + v * v)], 1).ravel()


def strip_state(x, y):
    left = x < 0.5
    return conservative(np.where(left, 0.9, 0.3) * (1 + 0.01 * np.sin(9 * x + 1)), np.where(left, -0.3, 0.4),
                        0.01 * np.sin(7 * x + 2), np.where(left, 0.2, 0.8) * (1 + 0.01 * np.cos(8 * x + 3)))


def wave_state(mach, amp, phase=(1.0, 2.0, 0.0, 1.0)):
    a, b, c, d = phase
    return lambda x, y: conservative(1.4 * (1 + amp * np.sin(9 * x + a) * np.cos(5 * y)), mach * (1 + amp * np.cos(6 * x + b)),
                                     3 * amp * np.sin(6 * y + x + c), 1 + amp * np.cos(8 * x * y + d))


PHASES = (2.1229302854698933, 4.714243431787986, 0.8803156075416094, 3.2503713420930724)


def guarded_step():
    ph = P.forward_step(cfl=0.8)
    ph.positivity_guard = True
    return ph


def quads(dt_kind, limiter):
    return P.Physics(V=4, flux="roe_fs", order2=True, limiter=limiter, K=1.0, dt_kind=dt_kind, cfl=0.5, global_dt=True,
                     bcs={"wall": ("wall", None), "ends": ("copy", None)})


# mesh, physics, state of (x, y), steps
CASES = {
    "strip": (lambda: meshgen.riemann_strip(12), P.riemann_strip, strip_state, 120),
    "step": (lambda: meshgen.forward_step(n=10), guarded_step, wave_state(3.0, 0.06, PHASES), 200),
    "step_short": (lambda: meshgen.forward_step(n=10), guarded_step, wave_state(3.0, 0.06), 120),
    "naca": (lambda: meshgen.naca_ogrid(ni=32, nj=8, r_far=10.0), P.naca, wave_state(0.8, 0.02), 40),
    "quads": (mixed_strip, lambda: quads("cfl_sum", "venkat"), wave_state(0.4, 0.1), 40),
    "quads_minmod": (mixed_strip, lambda: quads("cfl_min_signed", "minmod"), wave_state(0.4, 0.1), 40),
}


def run(name, layout):
    make, physics, state, steps = CASES[name]
    mesh = fvgpu.Mesh.from_elements(make())
    g = mesh.geometry()
    s = fvgpu.Solver(mesh, physics(), "fp32", stage_kernels=layout)
    s.set_state(state(np.asarray(g["ccx"]), np.asarray(g["ccy"])))
    r = s.run(steps, alpha=P.RK5_ALPHA)
    return s.get_state(), np.asarray(r["R"]), r["time"]


@pytest.mark.gpu
@pytest.mark.parametrize("layout", ("auto", "split", "fused", "hybrid"))
@pytest.mark.parametrize("name", sorted(CASES))
def test_same_bits(name, layout):
    want = np.load(GOLDEN)
    q, R, t = run(name, layout)
    assert q.tobytes() == want[name + "_q"].tobytes()
    assert t == want[name + "_t"]
    np.testing.assert_allclose(R, want[name + "_R"], rtol=1e-12, atol=0)


if __name__ == "__main__":
    out = {}
    for n in sorted(CASES):
        for k, v in zip("qRt", run(n, "auto")):
            out[n + "_" + k] = v
    np.savez_compressed(GOLDEN, **out)
