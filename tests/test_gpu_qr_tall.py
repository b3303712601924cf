"""Householder panels whose CTAs have more than 1024 rows each (one row of the panel per thread): the
isometry move of a node of 560 x 560 x 33, a 313600 x 33 matrix (one panel of 32 columns and one of
one) on at most two CTAs per SM.

Tolerance: an orthogonal factorisation of a matrix with 3e5 rows, sums of 1e3 terms in sequence at
most: 1e-12 for Q^T Q, 1e-11 for the direction of the state, as in the other tests of isometry moves."""
import numpy as np
import pytest

from tests.test_gpu_ttn import _isometric

pytestmark = pytest.mark.gpu


def test_panel_of_many_rows_per_cta(tn, ctx):
    d, D, n = 32, 560, 33
    a, b, c, e = (1, 1), (1, 2), (2, 1), (3, 1)
    graph = {a: [c], b: [c], c: [a, b, e], e: [c]}
    sites = [a, a, b, b, e, e]
    rng = np.random.default_rng(5)
    tensors = {a: rng.standard_normal((d, d, D)) / 32, b: rng.standard_normal((d, d, D)) / 32,
               c: rng.standard_normal((D, D, n)) / D, e: rng.standard_normal((d, d, n))}
    x, y = rng.standard_normal((d, d)), rng.standard_normal((d, d))

    def direction(t):  # the state with the sites of a and b projected on x and y
        va, vb = np.einsum("ij,ijk->k", x, t[a]), np.einsum("ij,ijk->k", y, t[b])
        u = t[e] @ np.einsum("i,ijk,j->k", va, t[c], vb)
        return u / np.linalg.norm(u)

    pg = tn.ttn.TTN(graph, sites, d, tensors, None, ctx).isometrize_(e)
    assert _isometric(pg, e)
    assert np.linalg.norm(direction({v: pg[v] for v in graph}) - direction(tensors)) <= 1e-11
