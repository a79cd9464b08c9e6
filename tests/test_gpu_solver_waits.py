"""A preconditioner's wait that runs out inside a solve or a set-up is the
solve's error (FEMGPU_E_TIMEOUT), not a breakdown and not silence, whichever
context runs it; the AMG context reports its device calls' errors through its
status, its host calls' with the call, each once."""
import numpy as np
import pytest

from fem_codes_gb300.mesh import cavity_problem, euler_cfl_dt, refletido_problem, skew_problem, structured_mesh

pytestmark = pytest.mark.gpu

E_TIMEOUT = -7


def gives_up(fg, call):
    with pytest.raises(fg.FemGpuError) as e:
        call()
    assert e.value.code == E_TIMEOUT


@pytest.mark.parametrize("solver", ["GMRES", "FGMRES"])
def test_transport_amg(gpu_lib, solver):
    import fem_codes_gb300 as fg
    m = structured_mesh(48, 32, perturb=0.2, seed=5)
    amg = fg.AMG(ncl=2, beta=0.25)
    with fg.SSTransport.from_problem(m, skew_problem(m), scheme="CSR", precond="AMG", solver=solver, kmax=30,
                                     lmax=40, tol=1e-8) as T:
        T.set_amg(amg)
        T.Build()
        T.precond_setup()
        X0, it0 = T.solver()
        amg.set_wait(0)
        gives_up(fg, T.solver)
        if solver == "GMRES":                       # the set-up applies the cycle to F
            gives_up(fg, T.precond_setup)
        amg.set_wait(-1)
        T.Build(u=np.zeros(T.neq + 1))
        T.precond_setup()
        X1, it1 = T.solver()
        assert it1 == it0 and np.array_equal(X0[:T.neq], X1[:T.neq])
    amg.close()


@pytest.mark.parametrize("precond", ["AMG", "ILU0"])
def test_navier_stokes(gpu_lib, precond):
    """257 basis vectors: no one-launch Arnoldi step, so the preconditioner's
    waits are the only ones."""
    import fem_codes_gb300 as fg
    m = structured_mesh(24, 24)
    pb = cavity_problem(m, 100.0)
    amg = fg.AMG(ncl=1, beta=0.25)
    with fg.NavierStokes.from_problem(m, pb, scheme="CSR", precond=precond, solver="FGMRES", kmax=257, lmax=2) as ns:
        if precond == "AMG":
            ns.set_amg(amg)
        wait = amg.set_wait if precond == "AMG" else ns.set_wait
        F, _ = ns.Build(np.zeros(pb.neq + 1))
        ns.precond_setup()
        X0, it0 = ns.solver(F)
        wait(0)
        gives_up(fg, lambda: ns.solver(F))
        wait(-1)
        X1, it1 = ns.solver(F)
        assert it1 == it0 and np.array_equal(X0, X1)
    amg.close()


def test_euler_amg_setup(gpu_lib):
    import fem_codes_gb300 as fg
    m = structured_mesh(24, 16)
    pb = refletido_problem(m)
    du = np.zeros(pb.neq + 1)
    amg = fg.AMG(ncl=1, beta=0.25)
    with fg.Euler.from_problem(m, pb, scheme="CSR", precond="AMG", solver="GMRES", dt=euler_cfl_dt(m, 5.0)) as eu:
        eu.set_amg(amg)
        eu.Build(pb.u0, du)
        R0 = eu.precond_setup()                     # R := M^-1 R
        eu.Build(pb.u0, du)
        amg.set_wait(0)
        gives_up(fg, eu.precond_setup)
        amg.set_wait(-1)
        eu.Build(pb.u0, du)
        assert np.array_equal(eu.precond_setup(), R0)
    amg.close()


def test_amg_calls_report_their_own_error_once(gpu_lib):
    import torch
    import fem_codes_gb300 as fg
    m = structured_mesh(48, 32, perturb=0.2, seed=5)
    with fg.SSTransport.from_problem(m, skew_problem(m), scheme="CSR", precond="NOT") as T:
        _, A = T.Build(want_matrix=True)
        pat = T.pattern()
    amg = fg.AMG(ncl=2, beta=0.25)
    amg.setup(pat["IA"], pat["JA"], A[:pat["IA"][-1]])
    n = pat["IA"].size - 1
    q = np.random.default_rng(0).standard_normal(n)
    qd = torch.from_numpy(q).cuda()
    zd = torch.zeros_like(qd)
    torch.cuda.synchronize()
    z0 = amg.apply(q)
    assert amg.status() == 0
    amg.set_wait(0)
    amg.apply_dev(qd.data_ptr(), zd.data_ptr())
    gives_up(fg, lambda: amg.apply(q))
    amg.set_wait(-1)
    assert np.array_equal(amg.apply(q), z0)
    assert amg.status() == E_TIMEOUT and amg.status() == 0
    amg.apply_dev(qd.data_ptr(), zd.data_ptr())
    assert amg.status() == 0 and np.array_equal(zd.cpu().numpy(), z0)
    amg.close()
