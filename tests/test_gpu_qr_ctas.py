"""Householder panels of one matrix on both sides of the lines of its CTA count: 64 rows a CTA up to
one CTA per SM (152 x 64 = 9728 rows: 98^2 below, 99^2 above), one per SM up to 512 rows each
(152 x 512 = 77824: 278^2 below, 279^2 above), two per SM beyond.  The matrix is the middle
node's, D^2 x 33 (one panel of 32 columns and one of one).

Tolerance: an orthogonal factorisation of a matrix with 8e4 rows, sums of 1e3 terms in sequence at
most: 1e-12 for Q^T Q, 1e-11 for the direction of the state, as in the other tests of isometry moves."""
import numpy as np
import pytest

from tests.test_gpu_ttn import _isometric

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [98, 99, 130, 278, 279])
def test_panel_cta_counts(tn, ctx, D):
    d, n = 17, 33
    a, b, c, e = (1, 1), (1, 2), (2, 1), (3, 1)
    graph = {a: [c], b: [c], c: [a, b, e], e: [c]}
    sites = [a, a, b, b, e, e]
    rng = np.random.default_rng(D)
    tensors = {a: rng.standard_normal((d, d, D)) / d, b: rng.standard_normal((d, d, D)) / d,
               c: rng.standard_normal((D, D, n)) / D, e: rng.standard_normal((d, d, n))}
    x, y = rng.standard_normal((d, d)), rng.standard_normal((d, d))

    def direction(t):  # the state with the sites of a and b projected on x and y
        va, vb = np.einsum("ij,ijk->k", x, t[a]), np.einsum("ij,ijk->k", y, t[b])
        u = t[e] @ np.einsum("i,ijk,j->k", va, t[c], vb)
        return u / np.linalg.norm(u)

    pg = tn.ttn.TTN(graph, sites, d, tensors, None, ctx).isometrize_(e)
    assert _isometric(pg, e)
    assert np.linalg.norm(direction({v: pg[v] for v in graph}) - direction(tensors)) <= 1e-11
