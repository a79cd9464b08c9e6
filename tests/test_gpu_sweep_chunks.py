"""The dataflow sweeps' chunks at their edges: matrix blocks with fewer chunks
than a thread block has warps, chunks of fewer than 32 rows, every record width
(rows of ILU(0) to ILU(6); wide ones leave room for fewer warps and the small
ring), the ring's reach lowered, the lookahead at its least and most, and the
two sweeps in one launch or two.  The separately rounded sweeps are the
oracle's bit for bit (ILUp_precond.c:26-46); the chain-scan sweeps of the same
factor agree to the tolerances of their arithmetic (test_gpu_ilu_sweeps)."""
import os

import numpy as np
import pytest

from oracle import pyoracle
from fem_codes_gb300.mesh import skew_problem, structured_mesh
from test_gpu_ilu_sweeps import CHAIN_TOL, DS_TOL

pytestmark = pytest.mark.gpu


def apply_with(env, m, level, solver, blocks=0):
    import fem_codes_gb300 as fg
    saved = {k: os.environ.get(k) for k in env}
    try:
        for k, v in env.items():
            os.environ.pop(k, None)
            if v is not None:
                os.environ[k] = str(v)
        with fg.SSTransport.from_problem(m, skew_problem(m), scheme="CSR", reorder="NOT", precond=f"ILU{level}",
                                         solver=solver, ilu_blocks=blocks) as T:
            _, A = T.Build(want_matrix=True)
            T.precond_setup(1)
            pat = T.pattern()
            r = np.zeros(T.neq + 1)
            r[:-1] = np.random.default_rng(5).standard_normal(T.neq)
            return T.precond(r)[:-1], r, pat, A[: T.nnzero], T.ilu_chain()
    finally:
        for k, v in saved.items():
            os.environ.pop(k, None)
            if v is not None:
                os.environ[k] = v


@pytest.mark.parametrize("nx,ny,level,near,skew", [
    (1, 1, 0, None, None), (2, 3, 0, None, None), (33, 31, 0, None, 1), (20, 300, 0, 8, 64), (90, 80, 0, 8, 1),
    (33, 31, 1, None, None), (24, 40, 2, 8, None), (24, 40, 3, None, 1), (24, 40, 4, None, None), (9, 70, 5, 8, None),
    (30, 30, 6, None, None)])
def test_chunks_bitexact(gpu_lib, nx, ny, level, near, skew):
    m = structured_mesh(nx, ny, perturb=0.2, seed=17)
    env = {"FEMGPU_SWEEP_NEAR": near, "FEMGPU_SWEEP_SKEW": skew, "FEMGPU_SWEEP_FB": None, "FEMGPU_SWEEP_DS": None}
    z, r, pat, A, _ = apply_with(env, m, level, "GMRES")
    z2, _, _, _, _ = apply_with(dict(env, FEMGPU_SWEEP_FB="0"), m, level, "GMRES")
    IA, JA = np.asarray(pat["IA"]), np.asarray(pat["JA"])
    if level:
        IA, JA, LU, Dinv = pyoracle.iluk(IA, JA, A, level)
    else:
        LU, Dinv = pyoracle.ilu0(IA, JA, A)
    zo = pyoracle.ilu0_apply(IA, JA, LU, Dinv, r)[: z.size]
    assert np.array_equal(z, zo)
    assert np.array_equal(z2, zo)
    for ds, tol in ((None, DS_TOL), ("0", CHAIN_TOL)):
        zc, _, _, _, chain = apply_with(dict(env, FEMGPU_SWEEP_DS=ds), m, level, "FGMRES")
        z2, _, _, _, _ = apply_with(dict(env, FEMGPU_SWEEP_DS=ds, FEMGPU_SWEEP_FB="0"), m, level, "FGMRES")
        assert np.max(np.abs(zc - zo)) <= tol * np.max(np.abs(zo))
        assert np.array_equal(zc, z2)


@pytest.mark.parametrize("blocks", [2, 13, 64])
def test_blocks_of_few_chunks(gpu_lib, blocks):
    """Block factors against the barrier sweeps of the same factor."""
    m = structured_mesh(40, 40, perturb=0.2, seed=17)
    env = {"FEMGPU_SWEEP_SYNC": None}
    z = apply_with(env, m, 0, "GMRES", blocks)[0]
    zb = apply_with({"FEMGPU_SWEEP_SYNC": "barrier"}, m, 0, "GMRES", blocks)[0]
    assert np.array_equal(z, zb)
