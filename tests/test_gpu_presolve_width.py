"""FP32 presolve at the edges of its width: 1152 columns (a round number of block pairs) and the next,
1279 and 1280, the most that the block-pair kernel takes (its largest shared memory, two passes of
its 1024 rows), and 1281, the first that the older kernel takes, beside a small block.

Tolerance: 1e-13 of the largest value, as in the other tests of this path."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1152, 1153, 1279, 1280, 1281])
def test_values_at_the_widest(tn, n):
    rng = np.random.default_rng(n)
    ctx = tn.Context(0, svd_split=0)  # every block on the multi-SM path
    blocks = []
    for r, c in ((n + 5, n), (50, 40)):
        scale = lambda k: 10.0 ** (-4.5 * np.arange(k) / k)  # noqa: E731 - graded on both sides
        blocks.append(scale(r)[:, None] * rng.standard_normal((r, c)) * scale(c))
    _, sv, _ = tn.svd_truncate(blocks, cutoff=1e-20, ctx=ctx)
    for b, s in zip(blocks, sv):
        ref = np.linalg.svd(b, compute_uv=False)
        assert np.abs(s - ref).max() <= 1e-13 * ref[0], b.shape
