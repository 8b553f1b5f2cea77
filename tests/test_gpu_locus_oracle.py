"""The eps and F moves against the oracle's at 1 to 32 lanes per locus, with one and
several alleles per lane, populations beyond a locus' slots, and one F for all: every
locus' accept decision and values, the F differences, and F after its tests.

Bounds.  A log ratio of a locus is a sum of K log-gamma differences; as either side
forms them (one logarithm of a product of Lanczos series or four series by themselves,
each accurate to about 1e-15, and products z log z of magnitude at most M), its error is
at most (32 x 2^-53 + 2e-15) M a side with M the sum of the magnitudes: a decision may
differ only where log u is that close to the ratio, and the F differences agree to it.
A shift is one product and one sum, contracted or not: 4 x 2^-53 of values at most 1."""
from math import fsum, lgamma

import numpy as np
import pytest

from structure_b200 import api

pytestmark = pytest.mark.gpu

SEED = 0x10CB
S_EPS = 8
REL = 2 * (32 * 2.0 ** -53 + 2e-15)   # both sides
VLG = np.vectorize(lgamma)


def _mag(z):
    return np.abs(z * np.log(z + 7)) + 10


def _eps_ratio(orc, l, na, logP, eps, F, lam, inv, rep):
    """(ratio, magnitude, log u) of one locus' move, formed here from the draws."""
    w = orc.stream(l, 0, rep, S_EPS, SEED)
    a1 = int((int(w[0]) >> 1) / 2147483648.0 * na)
    a2 = int((int(w[1]) >> 1) / 2147483648.0 * (na - 1))
    a2 += a2 >= a1
    d = (int(w[2]) >> 1) / 2147483648.0 * inv
    fr = (1 - F) / F
    z = [fr * eps[l, a1], fr * eps[l, a2], fr * (eps[l, a1] + d), fr * (eps[l, a2] - d)]
    lp = fr * d * (logP[l, :, a1].astype(np.float64) - logP[l, :, a2])
    s = (VLG(z[0]) + VLG(z[1]) - VLG(z[2]) - VLG(z[3]) + lp).sum()
    u = (int(orc.stream(l, 1, rep, S_EPS, SEED)[0]) >> 1) / 2147483648.0
    return s, sum(_mag(x).sum() for x in z) + np.abs(fr * d * logP[l, :, a1]).sum() * 2, np.log(max(u, 1e-300))


# (lanes: 32 up to 2368 loci, 16 to 4736, 8 to 9472, 4 to 18,944, 2 to 37,888)
@pytest.mark.parametrize("L,K,amax,onefst", [
    (1, 3, 9, 0), (60, 1, 10, 0), (60, 3, 10, 1), (61, 6, 10, 0), (300, 5, 2, 0), (130, 20, 7, 1),
    (3000, 3, 5, 0), (4700, 6, 9, 1), (7000, 2, 6, 0), (15000, 5, 4, 0), (15000, 3, 2, 1),
    (30000, 7, 3, 0), (40000, 3, 4, 0), (40000, 2, 2, 1)])
def test_moves_equal_the_oracles(ctx, orc, L, K, amax, onefst):
    N, rep = 12, 5
    rng = np.random.default_rng(L * 31 + K)
    na = rng.integers(1, amax + 1, L).astype(np.int32)
    na[0] = amax
    geno = (rng.random((N, 2, L)) * na).astype(np.int32)
    d = api.Data(ctx, na, geno=geno, layout=api.LAYOUT_U8)
    m, sd = 0.1, 0.1
    c = api.Chain(ctx, d, api.model_defaults(maxpops=K, burnin=0, numreps=9, freqscorr=1, onefst=onefst,
                                             fpriormean=m, fpriorsd=sd), SEED)
    F0 = np.full(K, 0.07) if onefst else rng.uniform(0.02, 0.3, K)
    c.set(api.F_F, F0)
    c.set(api.F_REP, np.array([rep], np.int32))
    c.UpdateP()
    logP, eps0 = c.get(api.F_LOGP), c.get(api.F_EPS)
    inv = float(N) ** -0.5
    c.UpdateEpsilon()
    eps = c.get(api.F_EPS)
    want, acc = orc.update_eps(na, logP, eps0, F0, 1.0, inv, SEED, rep)
    off = np.abs(eps - want).max(1) > 4 * 2.0 ** -53
    for l in np.flatnonzero(off):
        s, mag, lu = _eps_ratio(orc, l, int(na[l]), logP, eps0, F0, 1.0, inv, rep)
        assert abs(lu - s) <= REL * mag, (l, lu, s)
    assert off.sum() <= 2 and (L < 30 or acc.sum() > 0)
    c.UpdateFst()
    assert c.sync() == 0
    st = c.get(api.F_STATS)
    nf, _ = orc.fst_diffs(na, logP, eps, F0, onefst, sd, SEED, rep)
    n = 1 if onefst else K
    new, got = st[api.ST_FST_NEW:api.ST_FST_NEW + n], st[api.ST_FST_DIFF:api.ST_FST_DIFF + n]
    np.testing.assert_allclose(new, nf[:n], rtol=1e-13)
    mask = np.arange(c.A)[None, :] < na[:, None]
    e = np.where(mask, eps, 1.0)
    for f in range(n):
        if not 0 < nf[f] < 1:
            continue
        mag, terms = 0.0, []
        for k in (range(K) if onefst else [f]):
            a, b = (1 - nf[f]) / nf[f], (1 - F0[k]) / F0[k]
            lp = (a - b) * e * logP[:, k, :]
            mag += np.where(mask, _mag(a * e) + _mag(b * e) + np.abs(lp), 0).sum()
            terms.append((lp - (VLG(a * e) - VLG(b * e)))[mask])
        # (the oracle adds the terms one after another, with an error of its own)
        diff = fsum(np.concatenate(terms))
        assert abs(got[f] - diff) <= REL * mag, (f, got[f], diff, REL * mag)
    full = np.zeros(K)
    full[:n] = got
    Fo, _ = orc.update_fst(F0, onefst, m, sd, int((na > 0).sum()), full, nf, SEED, rep)
    np.testing.assert_allclose(c.get(api.F_F), Fo, rtol=1e-13)
    c.close()
    d.close()
