"""The block-SVD path of a bond whose blocks all lie in the one-CTA kernel's size classes (up to
128 x 112) depends on the blocks alone: one CTA each.  A fresh context, one whose tuner has settled
the same buckets on other bonds, and one with that schedule fixed give the same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ONE_CTA = 4096


def _graded(rng, r, c):
    k = min(r, c)
    U, _ = np.linalg.qr(rng.standard_normal((r, k)))
    V, _ = np.linalg.qr(rng.standard_normal((c, k)))
    return (U * 10.0 ** (-9.0 * np.arange(k) / k)) @ V.T


def _values(tn, ctx, blocks):
    return np.concatenate(tn.svd_truncate(blocks, cutoff=1e-20, ctx=ctx)[1])


@pytest.mark.parametrize("shapes", [
    [(100, 96), (80, 70), (30, 20)], [(96, 100), (60, 64)], [(112, 97), (90, 80), (66, 65), (50, 40)],
    [(128, 112)], [(100, 100)] * 33, [(100, 97)] * 32 + [(64, 64)] * 8])
def test_path_depends_on_the_blocks_alone(tn, shapes):
    rng = np.random.default_rng(11)
    made = {s: _graded(rng, *s) for s in set(shapes)}
    blocks = [made[s] for s in shapes]
    settled = tn.Context(0)
    others = [[_graded(rng, 150, 90), _graded(rng, 150, 70)],  # buckets 3 and 4, outside the classes
              [_graded(rng, 150, 120), _graded(rng, 100, 90)]]
    for bond in others:
        for _ in range(4):
            tn.svd_truncate(bond, cutoff=1e-12, ctx=settled)
    want = _values(tn, tn.Context(0, svd_split=ONE_CTA), blocks)
    assert np.array_equal(_values(tn, tn.Context(0), blocks), want)
    assert np.array_equal(_values(tn, settled, blocks), want)
    for b, s in zip(blocks, tn.svd_truncate(blocks, cutoff=1e-20, ctx=settled)[1]):
        ref = np.linalg.svd(b, compute_uv=False)
        assert np.abs(s - ref).max() <= 1e-13 * ref[0]
