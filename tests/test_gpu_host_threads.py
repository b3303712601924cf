"""Contexts driven from several host threads on one GPU, with kernels that ask for different
amounts of dynamic shared memory: the limit that a launch needs must not be lowered by another
thread between its setting and the launch (which is then refused).

Each thread repeats one call on a context of its own and compares every result with its first one
(the same kernels on the same data: the same bits) and, for the block SVD, with LAPACK (1e-13 of the
largest value, as in the other SVD tests)."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run_threads(jobs):
    errors = []
    start = threading.Barrier(len(jobs))

    def body(job):
        try:
            start.wait(timeout=60)
            job()
        except Exception as e:  # noqa: BLE001 - handed to the test's thread
            errors.append(repr(e))

    threads = [threading.Thread(target=body, args=(j,)) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join(timeout=300)
    assert not any(t.is_alive() for t in threads)
    assert not errors, errors


def test_small_qr_of_different_sizes(tn):
    # the leaves' matrices are D^2 x 2: 4 rows (144 bytes a CTA) to 2500 (180 KB)
    def job(D, seed):
        rng = np.random.default_rng(seed)
        a, b, c = (1, 1), (1, 2), (2, 1)
        tensors = {a: rng.standard_normal((D, D, 2)), b: rng.standard_normal((D, D, 2)),
                   c: rng.standard_normal((2, 2))}
        graph, sites = {a: [c], b: [c], c: [a, b]}, [a, a, b, b]
        ctx = tn.Context(0)

        def run():
            first = None
            for _ in range(60):
                psi = tn.ttn.TTN(graph, sites, D, tensors, None, ctx).isometrize_(a)
                psi.isometrize_(b)
                got = [psi[v] for v in (a, b, c)]
                first = first or got
                assert all(np.array_equal(x, y) for x, y in zip(got, first))
        return run

    _run_threads([job(D, i) for i, D in enumerate((2, 45, 3, 50))])


def test_one_cta_svds_of_different_sizes(tn):
    def job(n, seed):
        block = np.random.default_rng(seed).standard_normal((n + 3, n))
        ref = np.linalg.svd(block, compute_uv=False)
        ctx = tn.Context(0, svd_split=4096)  # every block on one CTA

        def run():
            for _ in range(60):
                _, sv, _ = tn.svd_truncate([block], cutoff=1e-20, ctx=ctx)
                assert np.abs(sv[0] - ref).max() <= 1e-13 * ref[0]
        return run

    _run_threads([job(n, i) for i, n in enumerate((8, 100, 20, 117))])
