"""Small Householder QR by a cluster of CTAs per matrix: isometry moves of trees whose link
dimensions lie on and next to the 8 columns of a CTA and the 32 rows of a warp pass, tall, square
and wide matrices (leaves of 4 rows with up to 25 columns), and more than 8 rows per lane.

Tolerance: the moves are orthogonal factorisations of matrices of at most 625 rows, whose error is
some hundred roundings of 1.1e-16 relative to the norm: 1e-12 for Q^T Q and 1e-11 for the state,
as in the other tests of isometry moves."""
import numpy as np
import pytest

from oracle import ttn_oracle as T
from tests.test_gpu_ttn import _isometric, upload

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chi", [1, 2, 3, 7, 8, 9, 16, 17, 24, 25])
def test_isometry_moves_at_column_and_row_edges(tn, ctx, chi):
    N = 16
    adj, sites = T.default_graph_sitenodes(N)
    psi = T.TTN(adj, sites, 2)
    rng = np.random.default_rng(chi)
    for v in psi.nodes:
        shape = [2 if leg[0] == "s" else chi for leg in psi.legs(v)]
        psi.tensors[v] = rng.standard_normal(shape) / np.sqrt(np.prod(shape[:-1]))
    ref = T.ttn_to_dense(psi)
    ref /= np.linalg.norm(ref)
    centers = [T.eccentric_center(adj, set(sites)), psi.nodes[0], psi.nodes[-1]]
    for center in centers:
        pg = upload(tn, ctx, psi).isometrize_(center)
        assert pg.orthocenter == center
        assert _isometric(pg, center)
        got = T.TTN(adj, sites, 2, {v: pg[v] for v in pg.labels}, center)
        assert np.linalg.norm(T.ttn_to_dense(got) - ref) <= 1e-11
