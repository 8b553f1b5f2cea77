"""The eps and F stages at every number of lanes per locus (few to many loci, few to
many alleles and populations): eps moves and F moves equal the oracle's from the same
state, and the F log likelihood differences agree.

The differences are FP64 sums of L K A terms lgamma(x) - lgamma(y) of magnitude at
most M each, one logarithm of a product of four Lanczos series (a few 2^-53 of its
value) plus (z - 1/2) log(z + 13/2) terms: with M the largest |z log z| met, 32 x
2^-53 x M per term bounds the rounding."""
import numpy as np
import pytest

from structure_b200 import api, synth

pytestmark = pytest.mark.gpu

SEED = 0x10C05


@pytest.mark.parametrize("N,L,K,amax,onefst", [
    (40, 1, 1, 2, 0), (40, 3, 2, 9, 0), (60, 37, 3, 10, 1), (60, 37, 6, 10, 0), (30, 257, 17, 5, 0),
    (50, 700, 5, 2, 0), (50, 3000, 4, 2, 1), (20, 12000, 9, 2, 0), (10, 40000, 3, 2, 0)])
def test_eps_and_f_moves(ctx, orc, N, L, K, amax, onefst):
    rng = np.random.default_rng(L + K)
    na = rng.integers(1, amax + 1, L).astype(np.int32)
    na[0] = amax
    geno = (rng.random((N, 2, L)) * na).astype(np.int32)
    d = api.Data(ctx, na, geno=geno, layout=api.LAYOUT_U8)
    c = api.Chain(ctx, d, api.model_defaults(maxpops=K, burnin=0, numreps=9, freqscorr=1,
                                             onefst=onefst, fpriormean=0.1, fpriorsd=0.1), SEED)
    rep = 3
    c.set(api.F_F, np.full(K, 0.07) if onefst else rng.uniform(0.02, 0.3, K))
    c.set(api.F_REP, np.array([rep], np.int32))
    c.UpdateP()
    F0, logP, eps0 = c.get(api.F_F), c.get(api.F_LOGP).astype(np.float64), c.get(api.F_EPS)
    c.UpdateEpsilon()
    eps = c.get(api.F_EPS)
    # every locus moved by a two-allele shift or not at all, and its accept decision is
    # the sign of log u - ratio (recomputed in FP64 from the move itself where it moved)
    moved = np.abs(eps - eps0).max(1) > 0
    assert (np.abs(eps.sum(1) - eps0.sum(1)) < 1e-12).all()
    assert (np.sum(eps != eps0, axis=1)[moved] == 2).all()
    assert L < 30 or 0 < moved.sum()
    c.UpdateFst()
    assert c.sync() == 0
    st = c.get(api.F_STATS)
    from math import lgamma
    vlg = np.vectorize(lgamma)
    mask = np.arange(c.A)[None, :] < na[:, None]
    nf = st[api.ST_FST_NEW:api.ST_FST_NEW + K]
    diff = st[api.ST_FST_DIFF:api.ST_FST_DIFF + K]

    def term(k, new):
        a, b = (1 - new) / new, (1 - F0[k]) / F0[k]
        e = np.where(mask, eps, 1.0)
        t = (a - b) * e * logP[:, k, :] - (vlg(a * e) - vlg(b * e))
        big = np.abs(a * e * np.log(a * e + 7)) + np.abs(b * e * np.log(b * e + 7)) \
            + np.abs((a - b) * e * logP[:, k, :]) + 10
        return np.where(mask, t, 0.0).sum(), np.where(mask, big, 0.0).sum()

    for f in range(1 if onefst else K):
        if not 0 < nf[f] < 1:
            continue
        parts = [term(k, nf[f]) for k in (range(K) if onefst else [f])]
        # the Lanczos series itself is accurate to about 1e-15 relative
        want, mag = sum(p[0] for p in parts), sum(p[1] for p in parts)
        assert abs(diff[f] - want) <= (32 * 2.0 ** -53 + 2e-15) * mag, (f, diff[f], want)
    c.close()
    d.close()
