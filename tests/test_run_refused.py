"""fv_run where the cooperative launch of the run kernel is refused: the captured
steps of the separate kernels take over.  The refusal is made on the host: a
preloaded function in the launch's place returns cudaErrorCooperativeLaunchTooLarge."""
import os
import shutil
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))

FAKE = """
static int calls;
int fake_calls(void) { return calls; }
int cudaLaunchCooperativeKernel(void) { ++calls; return 720; }
"""

RUN = """
import ctypes, sys
sys.path[:0] = [p for p in sys.argv[2].split(":")]
import numpy as np
import fvgpu, meshgen
import physics as P
from test_run_kernel import bits_equal, euler, smooth_state
fake = ctypes.CDLL(sys.argv[1])
heat = P.heat(dt=1e-5)
heat.bcs = {"wall": ("copy", None), "ends": ("copy", None)}
mesh = fvgpu.Mesh.from_elements(meshgen.rect_tri(31, 23, 1.0, 0.8))
q4 = smooth_state(mesh.geometry())
q1 = 1 + np.sin(9 * np.asarray(mesh.geometry()["ccx"]))
for ph, q0, alphas in ((euler(False), q4, (P.RK1_ALPHA, P.RK5_ALPHA)), (euler(True), q4, (P.RK5_ALPHA,)),
                       (heat, q1, (P.RK1_ALPHA, P.RK5_ALPHA))):
    for alpha in alphas:
        out = []
        for layout in ("auto", "split"):
            s = fvgpu.Solver(mesh, ph, "fp64", stage_kernels=layout)
            recs, before = [], fake.fake_calls()
            s.set_state(q0)
            s.run(5, alpha=alpha)
            r = s.run(30, alpha=alpha, restart=False, on_print=lambda n, t, R: recs.append((n, t)))
            assert (fake.fake_calls() - before == 2) == (layout == "auto"), (layout, fake.fake_calls() - before)
            out.append((s.get_state(), r["step"], r["time"], recs))
        assert out[0][1:] == out[1][1:] and out[0][1] == 30 and len(out[0][3]) == 25
        # (the stencils' sums have an order of their own)
        assert bits_equal(out[0][0], out[1][0]) or (ph is heat and np.abs(out[0][0] - out[1][0]).max() < 1e-12)
print("served")
"""


@pytest.mark.skipif(shutil.which("gcc") is None, reason="needs gcc")
def test_refused_launch_is_served_by_captured_steps(tmp_path):
    src, so = tmp_path / "fake.c", tmp_path / "fake.so"
    src.write_text(FAKE)
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(so), str(src)], check=True)
    root = os.path.dirname(HERE)
    paths = ":".join([HERE, os.path.join(root, "finite-volume-2d-cpp_b200"), os.path.join(root, "oracle"), root])
    r = subprocess.run([sys.executable, "-c", RUN, str(so), paths], env=dict(os.environ, LD_PRELOAD=str(so)),
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("served"), r.stdout + r.stderr
