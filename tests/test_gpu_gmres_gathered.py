"""Left-preconditioned GMRES steps whose product is written straight into the
ILU(0) sweeps' input (CSR, ILU(0)): systems of a few rows and of a ragged last
slice, the sweeps' dataflow, barrier and ELL forms (whose inputs are padded
differently), against the oracle's GMRES (pgmres.c:41-196): the solution to the
bar of the parity tests (1e-8), the iteration count give or take one."""
import os

import numpy as np
import pytest

from oracle import pyoracle
from fem_codes_gb300.mesh import skew_problem, structured_mesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,env", [
    (1, 2, {}), (3, 3, {}), (33, 31, {}), (33, 31, {"FEMGPU_SWEEP_SYNC": "barrier"}),
    (33, 31, {"FEMGPU_SWEEP_LAYOUT": "ell"}), (7, 90, {})])
def test_gmres_vs_oracle(gpu_lib, monkeypatch, nx, ny, env):
    import fem_codes_gb300 as fg
    for k in ("FEMGPU_SWEEP_SYNC", "FEMGPU_SWEEP_LAYOUT"):
        monkeypatch.delenv(k, raising=False)
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    m = structured_mesh(nx, ny, perturb=0.2, seed=17)
    p = skew_problem(m)
    ref = pyoracle.run_transport(m.x, m.y, p.node_type, m.vert, p.k, p.gamma, p.beta, p.fsrc, p.upresc, npicard=2)
    with fg.SSTransport.from_problem(m, p, scheme="CSR", reorder="NOT", precond="ILU0", solver="GMRES", kmax=30,
                                     lmax=1000, tol=1e-8) as T:
        uh, its = T.Process(2)
    for i in range(2):
        r = ref["uhist"][i, :-1]
        assert np.linalg.norm(uh[i, :-1] - r) <= 1e-8 * np.linalg.norm(r)
    assert np.all(np.abs(its - ref["iters"][:2]) <= 1)
