"""FP32 presolve on column pairs whose norms differ by more than 2^64 and are not orthogonal: the
squares in the rotation angle then leave FP32's range.

The block has one row of 0.9 and, below it, a diagonal of order delta: every column is that row's
direction plus its own 1e-18 .. 1e-12, all of it exact through the QR (the first reflector is the
identity), so R^T has one column of norm 31 and 1199 of norm delta at angles of order one to each
other's sum.  The largest value is the Frobenius norm to rounding, the others lie between the
smallest and the largest delta (interlacing of a rank-one change).

Tolerance: 1e-13 of the largest value, as in the other tests of this path; LAPACK of the same
matrix is the reference."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 1200


@pytest.mark.parametrize("delta", [1.05e-18, 1.2e-18, 3e-18, 1e-17, 1e-16, 1e-12])
@pytest.mark.parametrize("sign", [1, -1])
def test_norm_ratios_beyond_the_square_range(tn, delta, sign):
    rng = np.random.default_rng(2)
    a = np.zeros((N, N))
    a[0, :] = 0.9
    a[0, 1::2] *= sign  # both signs of the inner products
    a[np.arange(1, N), np.arange(1, N)] = delta * rng.uniform(1, 1.3, N - 1)
    ctx = tn.Context(0, svd_split=0)  # every block on the multi-SM path
    _, sv, _ = tn.svd_truncate([a], cutoff=1e-30, ctx=ctx)
    s = sv[0]
    ref = np.linalg.svd(a, compute_uv=False)
    assert np.isfinite(s).all()
    assert np.abs(s - ref).max() <= 1e-13 * ref[0]
