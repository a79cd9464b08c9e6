"""The fused network layers at the edges of their tiles and of the edges they
take at a time: graphs of one node, of less than a tile and just over one, nodes
without neighbours, with up to eight and with more.  Forward pass, loss and
gradient against the oracle's network (gnn_oracle.py), bars as in
test_gpu_gnn.py: FP32 activations 1e-4 / 1e-3, bf16 activations 2e-2 / 5e-2
(relative 2-norm of z / of the gradient)."""
import numpy as np
import pytest

from oracle import gnn_oracle as go

pytestmark = pytest.mark.gpu


def graph(n, degree, seed):
    """A matrix with a symmetric pattern: each node coupled to up to `degree'
    others (node 0, when there are others, to none)."""
    rng = np.random.default_rng(seed)
    pairs = set()
    for i in range(1, n):
        for j in rng.integers(1, n, degree // 2):
            if i != j:
                pairs |= {(i, int(j)), (int(j), i)}
    rows = [[(i, 4.0 + rng.random())] for i in range(n)]
    for i, j in sorted(pairs):
        rows[i].append((j, float(rng.uniform(-1.0, 0.3))))
    IA, JA, AA = [0], [], []
    for r in rows:
        r.sort()
        JA += [c for c, _ in r]
        AA += [v for _, v in r]
        IA.append(len(JA))
    return np.array(IA, np.int32), np.array(JA, np.int32), np.array(AA)


@pytest.mark.parametrize("bf16,ztol,gtol", [(False, 1e-4, 1e-3), (True, 2e-2, 5e-2)])
@pytest.mark.parametrize("n,degree", [(1, 0), (37, 4), (64, 6), (257, 6), (300, 14), (1025, 22)])
def test_tiles_vs_oracle(gpu_lib, n, degree, bf16, ztol, gtol):
    from fem_codes_gb300.learned import MeshGNN, init_params
    IA, JA, AA = graph(n, degree, n + degree)
    theta = init_params(3)
    rng = np.random.default_rng(9)
    theta = (theta + 0.05 * rng.standard_normal(theta.size)).astype(np.float32)
    r, t = rng.standard_normal(n), rng.standard_normal(n)
    net = MeshGNN(theta, bf16=bf16)
    net.attach_csr(IA, JA, AA)
    net.set_loss("both")
    z = net.apply(r)
    loss, grad, zt = net.loss_grad(r, t)
    net.close()
    lo, g, zo = go.loss_and_grad(theta, go.graph(IA, JA, AA), r, t, act_bf16=bf16, kind=2)
    assert np.array_equal(z, zt)
    assert np.linalg.norm(z - zo) <= ztol * np.linalg.norm(zo)
    assert abs(loss - lo) <= ztol * lo
    assert np.linalg.norm(grad - g) <= gtol * np.linalg.norm(g)
