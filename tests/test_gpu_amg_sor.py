"""The dataflow SOR sweeps of the AMG V-cycle where their schedules differ from
a mesh matrix's: one to four sweeps a side (one launch, two sweeps together,
several launches), systems of less than a warp, rows longer than the 8 and 16
entries the kernel keeps in registers, patterns that are not symmetric (a row
read by one that it does not read), a diagonal that takes the general division,
a zero right-hand side.  Bar: bit-identical to the oracle's sequential V-cycle
over the same hierarchy (amg_dpa.c:485-506, amg_solvers.c:3-33)."""
import numpy as np
import pytest

from oracle import pyoracle

pytestmark = pytest.mark.gpu


def matrix(n, per_row, seed, symmetric=True, scale=1.0):
    """A diagonally dominant CSR matrix of n rows with about per_row couplings
    a row to near and far columns, ascending."""
    rng = np.random.default_rng(seed)
    pairs = {}
    for i in range(n):
        for j in set(rng.integers(0, n, per_row // 2).tolist() + [i - 1, i + 1][: per_row]):
            if 0 <= j < n and j != i:
                pairs[i, j] = -rng.uniform(0.1, 1.0)
                if symmetric:
                    pairs.setdefault((j, i), -rng.uniform(0.1, 1.0))
    rows = [[] for _ in range(n)]
    for (i, j), v in pairs.items():
        rows[i].append((j, scale * v))
    IA, JA, AA = [0], [], []
    for i, r in enumerate(rows):
        r.append((i, scale * (1.0 + rng.uniform() + sum(abs(v) for _, v in r) / scale)))
        r.sort()
        JA += [c for c, _ in r]
        AA += [v for _, v in r]
        IA.append(len(JA))
    return np.array(IA, np.int32), np.array(JA, np.int32), np.array(AA)


@pytest.mark.parametrize("n,per_row,nr,omega,symmetric,scale", [
    (5, 2, 2, 1.0, True, 1.0), (33, 4, 1, 1.0, True, 1.0), (700, 6, 2, 0.8, True, 1.0), (700, 6, 3, 1.0, False, 1.0),
    (900, 14, 2, 1.0, False, 1.0), (400, 40, 4, 1.3, True, 1.0), (300, 4, 2, 1.0, True, 1e-180)])
def test_sweeps_bitexact(gpu_lib, n, per_row, nr, omega, symmetric, scale):
    import fem_codes_gb300 as fg
    IA, JA, AA = matrix(n, per_row, 100 + n + nr, symmetric, scale)
    amg = fg.AMG(ncl=1, beta=0.25, omega=omega, nr=nr)
    amg.setup(IA, JA, AA)
    lv = [amg.level(l) for l in range(amg.levels())]
    rng = np.random.default_rng(n)
    q = rng.standard_normal(n)
    for v in (q, np.where(rng.random(n) < 0.7, 0.0, q), np.zeros(n)):
        assert np.array_equal(amg.apply(v), pyoracle.amg_vcycle(lv, omega, nr, v))
    amg.close()
