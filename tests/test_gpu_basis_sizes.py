"""Krylov cycles around the basis size where a step's form changes: 256 basis
vectors are the last that take the one-launch steps and the columns' shared
memory, beyond it the Givens update and the back substitution work in global
scratch.

The reference's GMRES without a preconditioner fills whole cycles on a 200 x 12
mesh (484, 486 and 399 iterations by the oracle at 256, 257 and 300 vectors); a
basis of 256 is also filled with two entries of w a thread block (39,000
unknowns).  Bars: the oracle's iteration count plus or minus two (a step takes
five per cent off the residual, rounding moves it by far less), the true
residual at the tolerance, and the oracle's solution to 1e-8 relative: the
smallest singular value puts two solutions at this residual within 8.8e-9 of
each other.  FGMRES (plain, look-ahead and FP32 sweeps) reaches the tolerance
on the true residual."""
import numpy as np
import pytest

from oracle import pyoracle
from fem_codes_gb300.mesh import skew_problem, structured_mesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kmax", [256, 257, 300])
def test_gmres_fills_its_basis(gpu_lib, kmax):
    import fem_codes_gb300 as fg
    m = structured_mesh(200, 12, perturb=0.2, seed=8)
    p = skew_problem(m, 1e-3)
    with fg.SSTransport.from_problem(m, p, scheme="CSR", reorder="NOT", precond="NOT", solver="GMRES", kmax=kmax,
                                     lmax=6, tol=1e-10) as T:
        F, AA = T.Build(want_matrix=True)
        T.precond_setup(1)
        pat = T.pattern()
        x, it = T.solver()
        n, rel = T.neq, T.true_residual()
    xo, ito, _ = pyoracle.csr_gmres(pat["IA"], pat["JA"], AA, F, use_ilu0=False, kmax=kmax, lmax=6, tol=1e-10)
    assert ito > kmax and abs(it - ito) <= 2
    assert rel <= 1.01e-10
    assert np.linalg.norm(x[:n] - xo[:n]) <= 1e-8 * np.linalg.norm(xo[:n])


@pytest.mark.parametrize("kmax", [256, 257, 300])
@pytest.mark.parametrize("precision,lookahead", [("FP64", "0"), ("FP64", "1"), ("MIXED", "0")])
def test_fgmres_at_basis_sizes(gpu_lib, monkeypatch, kmax, precision, lookahead):
    import fem_codes_gb300 as fg
    monkeypatch.setenv("FEMGPU_LOOKAHEAD", lookahead)
    m = structured_mesh(160, 96, perturb=0.2, seed=1234)
    p = skew_problem(m)
    with fg.SSTransport.from_problem(m, p, scheme="CSR", reorder="SYMRCM", precond="ILU0", solver="FGMRES", kmax=kmax,
                                     lmax=20, tol=1e-8, precision=precision, ilu_blocks=8) as T:
        T.build_dev()
        T.precond_setup_dev(1)
        T.solve_dev()
        assert T.true_residual() <= 1.01e-8


def test_fgmres_fills_the_largest_one_launch_basis(gpu_lib):
    import fem_codes_gb300 as fg
    m = structured_mesh(300, 130, perturb=0.2, seed=8)
    p = skew_problem(m, 1e-3)
    with fg.SSTransport.from_problem(m, p, scheme="CSR", reorder="NOT", precond="NOT", solver="FGMRES", kmax=256,
                                     lmax=20, tol=1e-4) as T:
        T.Build()
        T.precond_setup(1)
        _, it = T.solver()
        assert it > 256 and T.true_residual() <= 1.01e-4
