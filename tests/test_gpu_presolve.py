"""FP32 presolve by block pairs (bj32_kernel) at the edges of its blocks: one block of columns,
one pair, an odd number of blocks, ragged last blocks, rows that are no multiple of four, more
than one row group, and the width where the older kernel takes over (1280 columns), on the
multi-SM path for every block.

Tolerance: 1e-13 of the largest value, as in the other tests of this path (the double-float
polish that follows sets the accuracy, not the presolve)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _graded(rng, r, c, decades=9.0):
    k = min(r, c)
    U, _ = np.linalg.qr(rng.standard_normal((r, k)))
    V, _ = np.linalg.qr(rng.standard_normal((c, k)))
    return (U * 10.0 ** (-decades * np.arange(k) / k)) @ V.T


def _check(tn, blocks):
    ctx = tn.Context(0, svd_split=0)  # every block on the multi-SM path
    _, sv, _ = tn.svd_truncate(blocks, cutoff=1e-20, ctx=ctx)
    for b, s in zip(blocks, sv):
        ref = np.linalg.svd(b, compute_uv=False)
        assert np.abs(s - ref).max() <= 1e-13 * ref[0], b.shape


@pytest.mark.parametrize("sizes", [[(1, 1), (2, 2), (3, 5)], [(16, 16), (17, 15), (18, 17)],
                                   [(33, 32), (40, 33), (48, 47)], [(65, 49), (64, 64), (90, 81)],
                                   [(200, 129), (129, 200), (257, 255)], [(300, 270), (20, 7)]])
def test_block_edges(tn, sizes):
    rng = np.random.default_rng(6)
    _check(tn, [_graded(rng, r, c) for r, c in sizes])


@pytest.mark.parametrize("n", [1100, 1290])
def test_longest_columns(tn, n):
    rng = np.random.default_rng(7)
    _check(tn, [_graded(rng, n + 3, n), _graded(rng, 70, 66)])


def test_flat_and_deficient_spectra(tn):
    rng = np.random.default_rng(8)
    flat, _ = np.linalg.qr(rng.standard_normal((150, 130)))
    low = rng.standard_normal((140, 9)) @ rng.standard_normal((9, 100))
    _check(tn, [flat, low, np.diag(np.r_[np.ones(60), np.full(40, 0.5)])])
