"""Long products of the tree code split into pieces of 256: on both sides of 512 rows of a QR panel
(one piece, two), of the 8192 rows where the number of pieces ends, and of the 1024 terms from
which a link contraction is split.

Tolerances as in the other tests of this code: 1e-12 for Q^T Q, 1e-11 for the direction of the state,
1e-12 relative for a product at the initial centre."""
import numpy as np
import pytest

from oracle import ttn_oracle as T
from tests.test_gpu_ttn import _isometric, upload

pytestmark = pytest.mark.gpu

A, B, C, E = (1, 1), (1, 2), (2, 1), (3, 1)
GRAPH = {A: [C], B: [C], C: [A, B, E], E: [C]}
SITES = [A, A, B, B, E, E]


def _tensors(rng, d, Da, Db, n):
    return {A: rng.standard_normal((d, d, Da)) / d, B: rng.standard_normal((d, d, Db)) / d,
            C: rng.standard_normal((Da, Db, n)) / np.sqrt(Da * Db),
            E: rng.standard_normal((d, d, n)) / d}


@pytest.mark.parametrize("Da,Db,n", [(17, 15, 65), (16, 16, 65), (73, 7, 33), (32, 16, 33),
                                     (27, 19, 33), (64, 128, 33), (91, 91, 34)])
def test_panel_products(tn, ctx, Da, Db, n):
    d = 12
    rng = np.random.default_rng(Da)
    t = _tensors(rng, d, Da, Db, n)
    x, y = rng.standard_normal((d, d)), rng.standard_normal((d, d))

    def direction(s):  # the state with the sites of a and b projected on x and y
        va, vb = np.einsum("ij,ijk->k", x, s[A]), np.einsum("ij,ijk->k", y, s[B])
        u = s[E] @ np.einsum("i,ijk,j->k", va, s[C], vb)
        return u / np.linalg.norm(u)

    pg = tn.ttn.TTN(GRAPH, SITES, d, t, None, ctx).isometrize_(E)
    assert _isometric(pg, E)
    assert np.linalg.norm(direction({v: pg[v] for v in GRAPH}) - direction(t)) <= 1e-11


@pytest.mark.parametrize("Da,Db", [(31, 33), (32, 32), (25, 41), (48, 47)])
@pytest.mark.parametrize("n", [15, 16, 40])
def test_link_contractions(tn, ctx, Da, Db, n):
    d = 7
    rng = np.random.default_rng(Da * n)
    pg = tn.ttn.TTN(GRAPH, SITES, d, _tensors(rng, d, Da, Db, n), None, ctx).isometrize_(E)
    psi = T.TTN(GRAPH, SITES, d, {v: pg[v] for v in GRAPH}, E)
    terms = []
    for i in range(5):
        o = [rng.standard_normal((d, d)) for _ in range(2)]
        terms.append((0.7, [(i, o[0] + o[0].T), (i + 1, o[1] + o[1].T)]))
    want = T.StateEnvsTTN(psi, terms).product(psi.tensors[E])
    env = tn.ttn.StateEnvsTTN(upload(tn, ctx, psi), tn.ttn.CouplingModel(terms, 6, d))
    got = env.product(psi.tensors[E])
    assert np.linalg.norm(got - want) <= 1e-12 * np.linalg.norm(want)
