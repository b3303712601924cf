"""Small QRs of a lockstep group whose matrices go to different kernels: a 4096 x 4 matrix (its
columns do not fit the shared memory of a cluster: one CTA) beside a 64 x 16 one (a cluster).  Each
instance has to come out of the batch as it does alone, to the bit: which kernel takes a matrix
depends on that matrix, not on its neighbours.

The tree is a star with two sites of dimension 8 on each leaf; the sweep moves the centre through
its nodes and back to the first, and the middle node's matrix toward e is D^2 x n."""
import numpy as np
import pytest

from tests.test_gpu_ttn import _isometric

pytestmark = pytest.mark.gpu

A, B, C, E = (1, 1), (1, 2), (2, 1), (3, 1)
GRAPH = {A: [C], B: [C], C: [A, B, E], E: [C]}
SITES = [A, A, B, B, E, E]


def _state(tn, ctx, D, n, seed):
    rng = np.random.default_rng(seed)
    t = {A: rng.standard_normal((8, 8, D)), B: rng.standard_normal((8, 8, D)),
         C: rng.standard_normal((D, D, n)), E: rng.standard_normal((8, 8, n))}
    return tn.ttn.TTN(GRAPH, SITES, 8, t, None, ctx).isometrize_(E)


def _model(tn):
    rng = np.random.default_rng(9)
    op = rng.standard_normal((8, 8))
    op = 0.5 * (op + op.T)
    terms = [(1.0, [(i, op), (i + 1, op)]) for i in range(5)]
    return tn.ttn.CouplingModel(terms, 6, 8)


def test_each_matrix_by_its_own_shape(tn, ctx):
    shapes = [(64, 4), (8, 16)]
    alone = []
    for i, (D, n) in enumerate(shapes):
        env = tn.ttn.StateEnvsTTN(_state(tn, ctx, D, n, i), _model(tn))
        sw = tn.ttn.SweepDataTTN()
        tn.ttn.fullsweep_(env, [A, C, B, E], tn.eig_solver, sw, outputlevel=0)
        alone.append((env.getpsi(), sw.energy[-1]))
    batch = tn.ttn.StateEnvsTTN.batch([_state(tn, ctx, D, n, i) for i, (D, n) in enumerate(shapes)],
                                      [_model(tn), _model(tn)])
    sws = [tn.ttn.SweepDataTTN() for _ in batch]
    tn.ttn.fullsweep_batch_(batch, [A, C, B, E], tn.eig_solver, sws, outputlevel=0)
    for env, sw, (psi, energy) in zip(batch, sws, alone):
        got = env.getpsi()
        assert env.orthocenter == A and _isometric(got, A) and _isometric(psi, A)
        assert sw.energy[-1] == energy
        for v in GRAPH:
            assert np.array_equal(got[v], psi[v]), v
