"""Waits of the dataflow kernels that run out, without a GPU fault: with the
context's bound at zero polls the ILU(0) factorisation, the one-launch Arnoldi
steps (GMRES and FGMRES) and the AMG's SOR sweeps give up at the first value
that is not there yet, record FEMGPU_E_TIMEOUT and return; the call reports it,
and with the default bound back the same context gives the same bits as
before."""
import numpy as np
import pytest

from fem_codes_gb300.mesh import cavity_problem, skew_problem, structured_mesh

pytestmark = pytest.mark.gpu

E_TIMEOUT = -7


def gives_up(fg, call):
    with pytest.raises(fg.FemGpuError) as e:
        call()
    assert e.value.code == E_TIMEOUT


def transport(fg, **kw):
    m = structured_mesh(96, 64, perturb=0.2, seed=5)
    return fg.SSTransport.from_problem(m, skew_problem(m), **dict(dict(scheme="CSR", lmax=40, tol=1e-8), **kw))


@pytest.mark.parametrize("blocks,precond", [(0, "ILU0"), (4, "ILU0"), (0, "ILU2")])
def test_factor_wait_runs_out_then_recovers(gpu_lib, blocks, precond):
    import fem_codes_gb300 as fg
    with transport(fg, precond=precond, solver="FGMRES", ilu_blocks=blocks) as T:
        T.Build()
        T.precond_setup()
        X0, it0 = T.solver()
        T.set_sweep_wait(0)
        gives_up(fg, T.precond_setup)
        T.set_sweep_wait(-1)
        T.precond_setup()
        X1, it1 = T.solver()
        assert it1 == it0 and np.array_equal(X0[:T.neq], X1[:T.neq])


@pytest.mark.parametrize("solver", ["GMRES", "FGMRES"])
def test_arnoldi_wait_runs_out_then_recovers(gpu_lib, solver):
    import fem_codes_gb300 as fg
    with transport(fg, precond="NOT", solver=solver, kmax=40) as T:   # no sweeps: the steps' waits alone
        T.Build()
        T.precond_setup()
        X0, it0 = T.solver(raise_on_nonconvergence=False)
        T.set_sweep_wait(0)
        gives_up(fg, T.solver)
        T.set_sweep_wait(-1)
        X1, it1 = T.solver(raise_on_nonconvergence=False)
        assert it1 == it0 and np.array_equal(X0[:T.neq], X1[:T.neq])


@pytest.mark.parametrize("nr", [1, 2, 3])
def test_sor_wait_runs_out_then_recovers(gpu_lib, nr):
    import fem_codes_gb300 as fg
    with transport(fg, precond="ILU0", solver="GMRES") as T:
        _, A = T.Build(want_matrix=True)
        pat = T.pattern()
    q = np.random.default_rng(0).standard_normal(pat["IA"].size - 1)

    def context():
        amg = fg.AMG(ncl=2, beta=0.25, nr=nr)
        amg.setup(pat["IA"], pat["JA"], A[:pat["IA"][-1]])
        return amg
    amg = context()
    z0 = amg.apply(q)
    amg.set_wait(0)
    gives_up(fg, lambda: amg.apply(q))
    amg.setup(pat["IA"], pat["JA"], A[:pat["IA"][-1]])
    amg.set_wait(-1)
    assert np.array_equal(amg.apply(q), z0)
    amg.close()


def test_navier_stokes_wait_runs_out_then_recovers(gpu_lib):
    import fem_codes_gb300 as fg
    m = structured_mesh(24, 24)
    pb = cavity_problem(m, 100.0)
    with fg.NavierStokes.from_problem(m, pb, scheme="CSR", precond="ILU0", solver="FGMRES", kmax=30, lmax=100) as ns:
        ns.Build(np.zeros(pb.neq + 1))
        F = ns.precond_setup()
        X0, it0 = ns.solver(F)
        ns.set_wait(0)
        gives_up(fg, ns.precond_setup)
        ns.set_wait(-1)
        ns.precond_setup()
        ns.set_wait(0)
        gives_up(fg, lambda: ns.solver(F))
        ns.set_wait(-1)
        X1, it1 = ns.solver(F)
        assert it1 == it0 and np.array_equal(X0, X1)
