"""Lanczos steps at the edges of the fused Gram-Schmidt kernel: vector lengths on and around
one part (256 elements), its clusters of 1, 2, 4 and 8 CTAs and the longest vectors it takes
(32 parts), and Krylov spaces that grow from it into the separate passes.

One two-site update of a random dense MPS (bond dimensions D1 and D3, so n = 4 D1 D3) against
the oracle's.  Tolerance: Ritz values of a few Lanczos steps with full re-orthogonalisation are
backward stable, error of order K n^(1/2) 2^-53 |H| < 1e-11 |H|; the kept spectrum as in the
other parity tests."""
import numpy as np
import pytest

from oracle import tn_oracle as O
from tests.helpers import upload_mpo, upload_mps

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d1,d3,krylovdim", [(1, 1, 3), (7, 9, 5), (8, 8, 5), (5, 13, 5),
                                             (8, 16, 4), (12, 16, 16), (16, 33, 6), (32, 64, 2),
                                             (32, 64, 5), (31, 67, 12), (40, 64, 31)])
def test_update_at_vector_length_edges(tn, ctx, d1, d3, krylovdim):
    rng = np.random.default_rng(d1 * 100 + d3)
    D = [1, d1, 6, d3, 1]
    links = [np.zeros(n, dtype=np.int64) for n in D]
    pq = np.zeros(2, dtype=np.int64)
    A = []
    for i in range(4):  # centre at site 1: left isometry before it, right isometries after it
        t = rng.standard_normal((D[i], 2, D[i + 1]))
        if i != 1:  # the wide side may exceed its rank: only scale then
            t /= np.linalg.norm(t)
        A.append(t)
    mps = O.MPS(A, links, pq, center=1)
    H = O.heisenberg_mpo(4, qn=False)
    env = tn.StateEnvs(upload_mps(tn, ctx, mps, center=1), upload_mpo(tn, ctx, H))
    e, err, eigs = tn.update_position_(env, tn.eig_solver, 1, 2, "left", maxdim=200, cutoff=1e-13,
                                       solver_krylovdim=krylovdim, solver_maxiter=2)
    eo = O.StateEnvs(mps, H)
    e_ref, spec, _ = O.update_two_site(eo, 1, "left", 200, 1, 1e-13, krylovdim, 2, 1e-14)
    assert abs(e - e_ref) <= 1e-11 * max(1.0, abs(e_ref))
    assert len(eigs) == len(spec.eigs)
    assert np.linalg.norm(eigs - spec.eigs) <= 1e-9
