"""A device-side error is reported once: the call that finds it returns it, and
the next call on the context reports only what happened since."""
import numpy as np
import pytest

from fem_codes_gb300.mesh import skew_problem, structured_mesh

pytestmark = pytest.mark.gpu

E_ZERO_PIVOT, E_BREAKDOWN = -4, -6


def test_zero_pivot_reported_once(gpu_lib):
    import fem_codes_gb300 as fg
    m = structured_mesh(24, 16, perturb=0.2, seed=2)
    p = skew_problem(m)
    with fg.SSTransport(m.x, m.y, p.node_type, m.vert, 0.0, 0.0, np.zeros(m.nnodes), const_beta=(0.0, 0.0),
                        scheme="CSR", precond="ILU0") as T:
        T.Build()
        for _ in range(2):                          # the operator is zero: reported by each set-up, not by Build
            with pytest.raises(fg.FemGpuError) as e:
                T.precond_setup()
            assert e.value.code == E_ZERO_PIVOT
            T.Build()


@pytest.mark.parametrize("solver", ["GMRES", "FGMRES"])
def test_breakdown_reported_once(gpu_lib, solver):
    import fem_codes_gb300 as fg
    m = structured_mesh(24, 16, perturb=0.2, seed=2)
    p = skew_problem(m)
    with fg.SSTransport(m.x, m.y, p.node_type, m.vert, 0.0, 0.0, np.zeros(m.nnodes), const_beta=(0.0, 0.0),
                        scheme="CSR", precond="NOT", solver=solver, kmax=20) as T:
        T.Build()
        T.precond_setup()
        for _ in range(2):                          # the first column of a zero operator has no norm
            with pytest.raises(fg.FemGpuError) as e:
                T.solver_bx(np.ones(T.neq + 1))
            assert e.value.code == E_BREAKDOWN
            T.Build()
