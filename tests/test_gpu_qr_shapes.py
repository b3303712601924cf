"""Small QRs on both sides of the line between the cluster and the one-CTA kernel: more than 256 rows
with at least 40 rows per column go to one CTA, as do matrices that do not fit the shared memory of
a cluster (4096 x 4).  The leaf's matrix is d^2 x n.

Tolerance: orthogonal factorisations of at most 4096 rows, some hundred roundings of 1.1e-16
relative to the norm: 1e-12 for Q^T Q and 1e-11 for the state, as in the other tests of isometry moves."""
import numpy as np
import pytest

from tests.test_gpu_ttn import _isometric

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,n", [(16, 1), (16, 6), (16, 7), (17, 1), (17, 7), (17, 8), (20, 10),
                                 (20, 11), (32, 16), (45, 2), (50, 6), (64, 1), (64, 4)])
def test_leaf_moves(tn, ctx, d, n):
    a, b, c = (1, 1), (1, 2), (2, 1)
    graph, sites = {a: [c], b: [c], c: [a, b]}, [a, a, b, b]
    rng = np.random.default_rng(d + n)
    t = {a: rng.standard_normal((d, d, n)), b: rng.standard_normal((d, d, n)),
         c: rng.standard_normal((n, n))}

    def dense(x):
        s = (x[a].reshape(d * d, n) @ x[c]) @ x[b].reshape(d * d, n).T
        return s / np.linalg.norm(s)

    for center in (c, b):
        pg = tn.ttn.TTN(graph, sites, d, t, None, ctx).isometrize_(center)
        assert _isometric(pg, center)
        assert np.linalg.norm(dense({v: pg[v] for v in graph}) - dense(t)) <= 1e-11
