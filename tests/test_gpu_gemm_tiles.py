"""FP64 grouped GEMM at the edges of its tiles (8 x 4 patches, 16 x 8, 16 x 16 and 32 x 32
tiles, 16-deep k chunks that run across segments): the two-site H_eff product of an MPS whose
bond dimensions sit on and next to those edges, against the oracle.

Tolerance: every output is one chain of at most w (D1 + D2) fused multiply-adds per stage, so
the relative error is below about 2 * 5 * 300 * 2^-53 = 3e-13 in the norm."""
import numpy as np
import pytest

from oracle import tn_oracle as O
from tests.helpers import oracle_envs, upload_mpo, upload_mps

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(1, 1, 1), (3, 2, 5), (4, 4, 8), (7, 9, 8), (15, 4, 17),
                                  (16, 16, 16), (31, 8, 33), (65, 20, 33), (300, 24, 280)])
def test_product_at_tile_edges(tn, ctx, dims):
    rng = np.random.default_rng(sum(dims))
    D = [1, *dims, 1]
    links = [np.zeros(n, dtype=np.int64) for n in D]
    pq = np.zeros(2, dtype=np.int64)
    mps = O.MPS([rng.standard_normal((D[i], 2, D[i + 1])) for i in range(4)], links, pq, center=1)
    H = O.heisenberg_mpo(4, qn=False)
    env = tn.StateEnvs(upload_mps(tn, ctx, mps, center=1), upload_mpo(tn, ctx, H))
    env.position_(1, 2)
    Lp, Rp = oracle_envs(mps, H, 1)
    v = rng.standard_normal((D[1], 2, 2, D[3]))
    ref = O.heff2_apply(Lp, H.W[1], H.W[2], Rp, v)
    assert np.linalg.norm(env.product(v) - ref) <= 3e-13 * np.linalg.norm(ref)
