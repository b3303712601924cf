"""A zero start vector is refused by the eigensolver whichever Gram-Schmidt path its length takes, in
both precisions, and leaves the context usable: the next update gives what a fresh context gives."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 8


@pytest.mark.parametrize("precision", ["fp64", "split"])
@pytest.mark.parametrize("links", ["charges", "dense"])  # n = a few; n = 2 * 2 * 64 * 64 = 16384
def test_refused_and_the_context_goes_on(tn, precision, links):
    def setup():
        ctx = tn.Context(0, precision=precision)
        W, delta, pq = tn.models.mpo_from_terms(N, tn.models.heisenberg_chain_terms(N))
        if links == "charges":
            psi = tn.MPS.product(tn.models.neel_states(N), pq, ctx)
            q = [np.asarray(psi.link_charges(i)) for i in range(N + 1)]
            t = [np.asarray(psi.site(i)) for i in range(N)]
            pos = 3
        else:  # one charge sector, links of 64
            pq = np.zeros(2, dtype=np.int32)
            delta = [np.zeros_like(d) for d in delta]
            dims = [1, 2, 4, 64, 64, 64, 4, 2, 1]
            q = [np.zeros(d, dtype=np.int32) for d in dims]
            rng = np.random.default_rng(0)
            t = [rng.standard_normal((dims[i], 2, dims[i + 1])) for i in range(N)]
            pos = 3
        return ctx, tn.MPO(W, delta, pq, ctx), pq, q, t, pos

    def update(ctx, H, pq, q, t, pos):
        env = tn.StateEnvs(tn.MPS(t, q, pq, pos, ctx), H)
        return tn.update_position_(env, tn.eig_solver, pos, 2, "left", maxdim=64, cutoff=1e-12)

    ctx, H, pq, q, t, pos = setup()
    with pytest.raises(tn.TenNetError, match="start vector is zero"):
        update(ctx, H, pq, q, [x * 0 for x in t], pos)
    after = update(ctx, H, pq, q, t, pos)
    fresh = update(*setup())
    assert after[0] == fresh[0] and np.array_equal(after[2], fresh[2])
