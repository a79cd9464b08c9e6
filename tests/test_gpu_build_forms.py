"""The steady element kernel's forms (with and without a source, a reaction,
a constant velocity, either shock parameter and length) and the assembly's row
gather, on ragged sizes around the kernel's 128-element and 32-row tiles.  A
third of the vertices are prescribed, so most elements carry a gradient and a
lift term.  Storage and right-hand side are bit-identical to the oracle's
(Build_K_F_SUPG.c:30-190, csr_assembly.c:9-22); the fused product reads the
slice copy that the assembly writes, whose at most 9 terms a row (an FMA each)
stay within 9 roundings of the exact sum, the rounded terms' within 2."""
import math

import numpy as np
import pytest

from oracle import pyoracle
from fem_codes_gb300.mesh import structured_mesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,scheme,gamma,src,const,shock,hshock", [
    (1, 2, "CSR", 0.0, False, True, "CAU", "2sqrtArea"),
    (8, 8, "CSR", 0.0, False, True, "CAU", "2sqrtArea"),
    (13, 5, "CSR", 0.0, True, False, "CAU", "2sqrtArea"),
    (31, 33, "CSR", 1.5, False, True, "YZBeta", "2sqrtArea"),
    (31, 33, "CSR", 1.5, True, False, "CAU", "Option1"),
    (40, 27, "CSR", 0.0, False, False, "YZBeta", "Option2"),
    (40, 27, "EDE", 1.5, True, True, "YZBeta", "2sqrtArea"),
    (17, 19, "EDE", 0.0, False, True, "CAU", "2sqrtArea"),
    (17, 19, "EBE", 0.0, True, True, "CAU", "2sqrtArea"),
    (64, 65, "EBE", 1.5, False, False, "CAU", "2sqrtArea")])
def test_build_forms(gpu_lib, nx, ny, scheme, gamma, src, const, shock, hshock):
    import fem_codes_gb300 as fg
    m = structured_mesh(nx, ny, perturb=0.2, seed=3)
    rng = np.random.default_rng(nx * 100 + ny)
    node_type = (rng.random(m.nnodes) > 0.35).astype(np.int32)
    node_type[:2] = [0, 1]
    upresc = np.where(node_type == 0, rng.uniform(-1.0, 1.0, m.nnodes), 0.0)
    ne = len(m.vert)
    beta = np.tile([0.6, -0.8], (ne, 1)) if const else rng.uniform(-1.0, 1.0, (ne, 2))
    if not const:
        beta[::7] = 0.0
    fsrc = rng.uniform(-1.0, 1.0, (ne, 3)) if src else np.zeros((ne, 3))
    precond = "ILU0" if scheme == "CSR" else "DIAG"
    ref = pyoracle.run_transport(m.x, m.y, node_type, m.vert, 1e-3, gamma, beta, fsrc, upresc, scheme=scheme,
                                 precond="Diag" if precond == "DIAG" else precond, shock=shock, hshock=hshock,
                                 npicard=1, tol=0.5)
    vel = dict(const_beta=[0.6, -0.8]) if const else dict(beta=beta)
    opts = dict(**vel, fsrc=fsrc, scheme=scheme, reorder="NOT", shock=shock, hshock=hshock)
    with fg.SSTransport(m.x, m.y, node_type, m.vert, 1e-3, gamma, upresc, precond=precond, **opts) as T:
        F, A = T.Build(u=np.zeros(T.neq + 1), want_matrix=True)
    assert np.array_equal(A, np.asarray(ref["Afirst"]).reshape(-1))
    assert np.array_equal(F[:-1], ref["Ffirst"][: ref["neq"]])
    if scheme != "CSR":
        return
    n, IA, JA = ref["neq"], ref["IA"], ref["JA"]
    with fg.SSTransport(m.x, m.y, node_type, m.vert, 1e-3, gamma, upresc, precond="ILU0", solver="FGMRES",
                        **opts) as T:
        T.Build(u=np.zeros(T.neq + 1))
        P = np.zeros(n + 1)
        P[:-1] = rng.standard_normal(n)
        Q = T.ProductMatrixVector(P)
    for i in range(n):
        terms = A[IA[i]:IA[i + 1]] * P[JA[IA[i]:IA[i + 1]]]
        assert abs(Q[i] - math.fsum(terms)) <= 11 * 2.0**-53 * np.abs(terms).sum()
