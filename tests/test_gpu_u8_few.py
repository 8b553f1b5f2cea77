"""One-byte chains of few individuals take the per-genotype kernel, by a rule on
individuals, populations and alleles; around it both kernels give the oracle's draws,
counts and ratios (the bounds of test_gpu_u8.py), and a batch that mixes them the bits
of its chains alone."""
import numpy as np
import pytest

from structure_b200 import api
from test_gpu_u8 import SEED, _check, _geno

pytestmark = pytest.mark.gpu


# 4 (N - 18) against K A, more than 148 loci (one locus per CTA up to there)
@pytest.mark.parametrize("N,L,K,amax", [(19, 300, 3, 2), (20, 300, 3, 2), (32, 149, 10, 6), (33, 149, 10, 6),
                                        (33, 148, 10, 6), (1, 260, 2, 3), (67, 151, 9, 22)])
def test_around_the_rule(ctx, orc, N, L, K, amax):
    _check(ctx, orc, N, L, K, amax)


def test_batch_of_both_kernels_equals_chains_alone(ctx):
    rng = np.random.default_rng(6)
    data = []
    for N, L in ((20, 300), (150, 200)):
        geno, na = _geno(rng, N, L, 8)
        data.append(api.Data(ctx, na, geno=geno, layout=api.LAYOUT_U8))
    specs = [(d, K) for d in data for K in (1, 4, 2, 10, 4)]
    mk = lambda: [api.Chain(ctx, d, api.model_defaults(maxpops=K, burnin=1, numreps=9, freqscorr=1,
                                                       metrofreq=3, fpriormean=0.05, fpriorsd=0.05),
                            SEED + j) for j, (d, K) in enumerate(specs)]
    batched, alone = mk(), mk()
    b = api.Batch(ctx, batched)
    b.sweep(5)
    for c in alone:
        c.sweep(5)
    for x, y in zip(batched, alone):
        assert x.sync() == 0 and y.sync() == 0
        for f in (api.F_Q, api.F_P, api.F_N, api.F_M, api.F_QSUM, api.F_PSUM):
            np.testing.assert_array_equal(x.get(f), y.get(f))
        np.testing.assert_array_equal(x.get(api.F_STATS)[:4], y.get(api.F_STATS)[:4])
    b.close()
    for c in batched + alone:
        c.close()
    for d in data:
        d.close()
