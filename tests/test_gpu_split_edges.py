"""Split-precision GEMM where only part of a tile is copied, multiplied and drained: bond
dimensions on and next to the 8-row atoms, the 16-deep MMA steps, the 16-column groups and the
128 x 64 tile, and more k tiles than the step mask holds (H_eff of an MPO with many states).

Tolerance: 5 slices keep 41 bits of each operand row and drop slice products below 2^-40, so
a product of three stages is within about 3 * 2^-38 = 1e-11 of FP64 in the norm; 5e-11 is the
bound of the other split-precision tests."""
import numpy as np
import pytest

from oracle import tn_oracle as O
from tests.helpers import oracle_envs, upload_mpo, upload_mps

pytestmark = pytest.mark.gpu


def _check(tn, H, dims, p):
    rng = np.random.default_rng(sum(dims))
    N = len(dims) + 1
    D = [1, *dims, 1]
    links = [np.zeros(n, dtype=np.int64) for n in D]
    pq = np.zeros(2, dtype=np.int64)
    mps = O.MPS([rng.standard_normal((D[i], 2, D[i + 1])) / np.sqrt(D[i]) for i in range(N)],
                links, pq, center=p)
    ctx = tn.Context(0, precision="split", slices=5)
    env = tn.StateEnvs(upload_mps(tn, ctx, mps, center=p), upload_mpo(tn, ctx, H))
    env.position_(p, 2)
    Lp, Rp = oracle_envs(mps, H, p)
    v = rng.standard_normal((D[p], 2, 2, D[p + 2]))
    ref = O.heff2_apply(Lp, H.W[p], H.W[p + 1], Rp, v)
    assert np.linalg.norm(env.product(v) - ref) <= 5e-11 * np.linalg.norm(ref)


@pytest.mark.parametrize("dims", [(1, 1, 1), (7, 3, 9), (8, 8, 8), (15, 4, 17), (16, 5, 33),
                                  (33, 8, 16), (63, 8, 65), (64, 9, 31), (129, 16, 130)])
def test_split_product_at_tile_edges(tn, dims):
    _check(tn, O.heisenberg_mpo(4, qn=False), dims, 1)


def test_split_product_with_many_k_tiles(tn):
    # 5 x 4 cylinder, about 20 MPO states: the second stage runs over more than 32 k tiles
    N = 20
    H = O.mpo_from_terms(N, O.j1j2_cylinder_terms(5, 4, 1.0, 0.5), qn=False)
    _check(tn, H, [2, 4, 7, 9, 9, 9, 8, 9, 17, 5, 20, 9, 7, 9, 9, 9, 7, 4, 2], 9)
