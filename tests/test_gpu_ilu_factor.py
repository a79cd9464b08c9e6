"""The dataflow ILU(p) factorisation at the edges of its row slots: systems of
one row and of less than a warp's rows, rows that just fit 8 and 16 lanes and
ones that need 32, levels that do not fill a warp, and blocks of a few rows.
The factor is seen through the preconditioner application of the reference's
GMRES, whose sweeps round as the reference's: bit-identical to the oracle's
ILU(p) (ILUp_precond_setup.c:66-167, ILUp_precond.c:26-46)."""
import numpy as np
import pytest

from blockcut_ref import block_ids
from oracle import pyoracle
from fem_codes_gb300.mesh import skew_problem, structured_mesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,level,lanes,blocks", [
    (1, 1, 0, 8, 0), (2, 1, 0, 8, 0), (5, 3, 0, 8, 0), (33, 31, 0, 8, 0), (70, 9, 0, 8, 0), (40, 40, 0, 8, 13),
    (33, 31, 1, 16, 0), (24, 40, 2, 16, 0), (33, 31, 4, 32, 0), (9, 70, 5, 32, 0)])
def test_factor_bitexact(gpu_lib, nx, ny, level, lanes, blocks):
    import fem_codes_gb300 as fg
    m = structured_mesh(nx, ny, perturb=0.2, seed=17)
    with fg.SSTransport.from_problem(m, skew_problem(m), scheme="CSR", reorder="NOT", precond=f"ILU{level}",
                                     solver="GMRES", ilu_blocks=blocks) as T:
        _, AA = T.Build(want_matrix=True)
        T.precond_setup(1)
        pat = T.pattern()
        IA, JA, AA = np.asarray(pat["IA"]), np.asarray(pat["JA"]), AA[: T.nnzero]
        if blocks:
            blk = block_ids(T.ilu_blocks())
            row = np.repeat(np.arange(T.neq), np.diff(IA))
            keep = blk[row] == blk[JA]
            IA = np.concatenate([[0], np.cumsum(np.bincount(row[keep], minlength=T.neq))]).astype(np.int32)
            JA, AA = JA[keep].astype(np.int32), AA[keep]
        if level:
            IA, JA, LU, Dinv = pyoracle.iluk(IA, JA, AA, level)
        else:
            LU, Dinv = pyoracle.ilu0(IA, JA, AA)
        longest = int(np.diff(IA).max())
        assert lanes == 8 and longest <= 8 or lanes // 2 < longest <= lanes
        r = np.zeros(T.neq + 1)
        r[:-1] = np.random.default_rng(5).standard_normal(T.neq)
        z = T.precond(r)
    zo = pyoracle.ilu0_apply(IA, JA, LU, Dinv, r)
    assert np.array_equal(z[: T.neq], zo[: T.neq])
