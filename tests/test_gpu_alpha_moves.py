"""The alpha test's parallel tail at the ends of its ranges: one to 32 populations,
one CTA to more CTAs than a warp has lanes, one alpha or one per population, flat
and gamma priors.  The sums, the log ratio of the last test and the moves equal the
oracle's from the same state (tolerances as in the parity tests of UpdateAlpha)."""
import numpy as np
import pytest

from structure_b200 import api, synth

pytestmark = pytest.mark.gpu

SEED = 0xA1FA5


@pytest.mark.parametrize("unif", [0, 1])
@pytest.mark.parametrize("popalphas", [0, 1])
@pytest.mark.parametrize("N,K", [(1, 1), (7, 2), (300, 5), (1500, 32), (4000, 17)])
def test_alpha_moves(ctx, orc, N, K, popalphas, unif):
    d = synth.snp_fmodel(N, 4, 2, [0.1, 0.2], 0.5, 0.0, N + K)
    data = api.Data(ctx, d["numalleles"], geno=d["geno"], layout=api.LAYOUT_B2G)
    c = api.Chain(ctx, data, api.model_defaults(maxpops=K, burnin=0, numreps=20, popalphas=popalphas,
                                                unifprioralpha=unif, alpha=0.8, alphapropsd=0.2), SEED)
    rng = np.random.default_rng(N + K)
    c.set(api.F_Q, rng.dirichlet(np.full(K, 0.8), N).astype(np.float32))
    for rep in range(4):
        c.set(api.F_REP, np.array([rep], np.int32))
        before = c.get(api.F_ALPHA)
        c.UpdateAlpha()
        assert c.sync() == 0
        st = c.get(api.F_STATS)
        S_o, T_o = orc.alpha_sums(c.get(api.F_LOGQ))
        np.testing.assert_allclose(st[api.ST_ALPHA_S:api.ST_ALPHA_S + K], S_o, rtol=1e-11, atol=1e-12)
        np.testing.assert_allclose(st[api.ST_ALPHA_T], T_o, rtol=1e-11, atol=1e-12)
        a_o, _ = orc.update_alpha(N, st[api.ST_ALPHA_S:api.ST_ALPHA_S + K], st[api.ST_ALPHA_T],
                                  before, SEED, rep, popalphas, unif, 10.0, 0.2, 1.0, 2.0)
        np.testing.assert_allclose(c.get(api.F_ALPHA), a_o, rtol=1e-14)
    c.close()
    data.close()
