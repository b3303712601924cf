"""One-CTA block SVD at the edges of its size classes (32, 64, 96 and 112 columns, 32 to 128
rows, and just beyond, where the general path takes over): values against LAPACK for graded,
wide, tall, rank-deficient and zero blocks, all of one launch.

Tolerance 1e-13 of the largest value (the double-float factorisation carries 48 bits and at
most a few hundred operations per value: 100 * 2^-48 = 4e-13 in the worst case, 1e-13 is what
the other SVD tests hold)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EDGES = [(1, 1), (2, 1), (32, 32), (33, 32), (33, 33), (64, 20), (64, 64), (65, 64), (65, 33),
         (96, 96), (97, 96), (97, 65), (97, 97), (112, 112), (113, 112), (113, 113), (128, 112),
         (128, 97), (128, 30), (129, 40), (129, 112), (140, 130)]


def _graded(rng, r, c):
    k = min(r, c)
    U, _ = np.linalg.qr(rng.standard_normal((r, k)))
    V, _ = np.linalg.qr(rng.standard_normal((c, k)))
    return (U * 10.0 ** (-9.0 * np.arange(k) / k)) @ V.T


def _check(tn, blocks):
    ctx = tn.Context(0, svd_split=4096)  # every block on one CTA
    kept, sv, _ = tn.svd_truncate(blocks, cutoff=1e-20, ctx=ctx)
    for b, s in zip(blocks, sv):
        ref = np.linalg.svd(b, compute_uv=False)
        assert np.all(np.diff(s) <= 0)
        assert np.abs(s - ref).max() <= 1e-13 * max(ref[0], 1e-300), b.shape


@pytest.mark.parametrize("transpose", [False, True])
def test_values_at_class_edges(tn, transpose):
    rng = np.random.default_rng(3)
    blocks = [_graded(rng, r, c) for r, c in EDGES]
    _check(tn, [np.asfortranarray(b.T) for b in blocks] if transpose else blocks)


def test_each_class_alone(tn):
    # one launch each: shared memory sized by that block only
    rng = np.random.default_rng(4)
    for r, c in EDGES:
        _check(tn, [_graded(rng, r, c)])


def test_rank_deficient_and_zero_blocks(tn):
    rng = np.random.default_rng(5)
    blocks = []
    for r, c, k in [(20, 16, 3), (60, 50, 7), (90, 88, 40), (128, 100, 1)]:
        blocks.append(rng.standard_normal((r, k)) @ rng.standard_normal((k, c)))
    blocks += [np.zeros((17, 9)), np.zeros((70, 70))]
    blocks.append(np.eye(48)[:, ::-1].copy())  # equal values
    _check(tn, blocks)
