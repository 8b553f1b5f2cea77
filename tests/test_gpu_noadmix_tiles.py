"""The no-admixture log likelihoods on 2-bit data at the edges of their tables:
every width of the population loop, odd numbers of loci (a pair's second half
empty), stages and chunks cut short, individuals beyond a word or a CTA, missing
genotypes and one-allele data.  The picked populations equal the oracle's."""
import numpy as np
import pytest

from structure_b200 import api, synth

pytestmark = pytest.mark.gpu

SEED = 0x7AB1E


def _check(ctx, orc, geno, na, K):
    L = geno.shape[2]
    data = api.Data(ctx, na, geno=geno, layout=api.LAYOUT_B2G)
    c = api.Chain(ctx, data, api.model_defaults(maxpops=K, burnin=10, numreps=10, noadmix=1,
                                                admburnin=2), SEED)
    rng = np.random.default_rng(K * 1000 + L)
    P = np.zeros((L, K, c.A), np.float32)
    for l in range(L):
        if na[l] > 0:
            P[l, :, :na[l]] = rng.dirichlet(np.full(na[l], 0.7), K)
    c.set(api.F_P, P)
    c.set(api.F_REP, np.array([5], np.int32))
    c.UpdateQ()
    assert c.sync() == 0
    Qo, lQo, _ = orc.update_q_noadmix(geno, c.get(api.F_LOGP), SEED, 5)
    np.testing.assert_array_equal(c.get(api.F_Q), Qo)
    np.testing.assert_array_equal(c.get(api.F_LOGQ), lQo)
    c.close()
    data.close()


@pytest.mark.parametrize("K", [1, 2, 3, 4, 5, 8, 9, 16, 17, 32])
@pytest.mark.parametrize("N,L", [(1, 1), (17, 65), (300, 131)])
def test_picks_match_the_oracle(ctx, orc, N, L, K):
    d = synth.snp_fmodel(N, L, 3, [0.05, 0.1, 0.2], 0.3, 0.1, N + L + K)
    _check(ctx, orc, d["geno"], d["numalleles"], K)


def test_one_allele_data(ctx, orc):
    rng = np.random.default_rng(2)
    geno = np.zeros((40, 2, 33), np.int32)
    geno[rng.random((40, 33))[:, None, :].repeat(2, 1) < 0.2] = -9
    _check(ctx, orc, geno, np.ones(33, np.int32), 4)
