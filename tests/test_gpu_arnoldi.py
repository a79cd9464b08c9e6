"""The one-launch Arnoldi steps at the edges of their sizes: one unknown, fewer
than and just over half a reduction block, one reduction block to a thread block
and two (38,912 unknowns), one entry of w a thread and two (77,824), and beyond
what fits (155,648: the separate kernels).  The reference's GMRES (modified
Gram-Schmidt) takes the oracle's iteration count, plus or minus one, and its
solution to 1e-8 relative; FGMRES (classical Gram-Schmidt, its second pass from
the second restart cycle on) reaches the tolerance on the true residual."""
import numpy as np
import pytest

from oracle import pyoracle
from fem_codes_gb300.mesh import skew_problem, structured_mesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(1, 1), (127, 1), (43, 3), (304, 128), (277, 141), (512, 152), (500, 156), (432, 361)])
def test_gmres_and_fgmres_at_block_edges(gpu_lib, nx, ny):
    import fem_codes_gb300 as fg
    m = structured_mesh(nx, ny, perturb=0.2, seed=8)
    p = skew_problem(m, 1e-3)
    kw = dict(scheme="CSR", reorder="NOT", precond="ILU0", lmax=60, tol=1e-10)
    with fg.SSTransport.from_problem(m, p, solver="GMRES", kmax=7, **kw) as T:
        F, AA = T.Build(want_matrix=True)
        T.precond_setup(1)
        pat = T.pattern()
        x, it = T.solver()
        n = T.neq
    assert n == nx * ny
    xo, ito, _ = pyoracle.csr_gmres(pat["IA"], pat["JA"], AA, F, kmax=7, lmax=60, tol=1e-10)
    assert abs(it - ito) <= 1
    assert np.linalg.norm(x[:n] - xo[:n]) <= 1e-8 * np.linalg.norm(xo[:n])
    # FP32 sweeps: the plain FGMRES cycle (no look-ahead step), restarted
    with fg.SSTransport.from_problem(m, p, solver="FGMRES", precision="MIXED", kmax=9, **dict(kw, tol=1e-9)) as T:
        T.build_dev()
        T.precond_setup_dev(1)
        T.solve_dev()
        assert T.true_residual() <= 1.0001e-9
