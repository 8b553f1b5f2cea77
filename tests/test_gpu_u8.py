"""The data pass on one-byte genotypes: every K class and the edges of its tiles (a
pair of individuals, a CTA's pairs, a chunk of loci), up to 64 alleles and
half-missing genotypes.  Z and counts equal the oracle's FP32 draws exactly;
counts of flagged individuals only equal the oracle's counts of the same Z.

ln P(D) is the oracle's FP64 value of the same FP32 Q and P up to the FP32
rounding of the K-term mixture sums: at most K 2^-24 relative per copy, so
K 2^-24 absolute per copy's logarithm.  The Metropolis log ratios are FP64 sums
and products of the same terms as the oracle's: K 2^-52 per copy and logarithm
of a running product 2^-53 per factor, in all at most (K + 4) 2^-51 per copy."""
import numpy as np
import pytest

from structure_b200 import api

pytestmark = pytest.mark.gpu

SEED = 0x18181


def _geno(rng, N, L, amax, missing=0.08):
    na = rng.integers(1, amax + 1, L).astype(np.int32)
    na[L // 2] = amax
    geno = (rng.random((N, 2, L)) * na).astype(np.int32)
    geno[rng.random((N, 2, L)) < missing] = -9
    return geno, na


def _state(rng, N, L, K, na):
    Q = rng.dirichlet(np.full(K, 0.5), N).astype(np.float32)
    P = np.zeros((L, K, int(na.max())), np.float32)
    for l in range(L):
        P[l, :, :na[l]] = rng.dirichlet(np.ones(na[l]), K)
    return Q, P


def _check(ctx, orc, N, L, K, amax, flagged=False):
    rng = np.random.default_rng(N * 7 + L * 3 + K)
    geno, na = _geno(rng, N, L, amax)
    flags = (rng.random(N) < 0.5).astype(np.int32)
    d = api.Data(ctx, na, geno=geno, layout=api.LAYOUT_U8, popflags=flags)
    Q, P = _state(rng, N, L, K, na)
    want_z = orc.zupdate_f32(geno, Q, P, SEED, 7)
    ncnt = np.where((flags == 1)[:, None, None], want_z, -9) if flagged else want_z
    n_o = orc.counts(np.where(ncnt < 0, -9, geno), ncnt, K, int(na.max()))[0]
    m_o = orc.counts(geno, want_z, K, int(na.max()))[1]
    for store in (0, 1):
        c = api.Chain(ctx, d, api.model_defaults(maxpops=K, burnin=0, numreps=9, freqscorr=0,
                                                 metrofreq=4, store_z=store,
                                                 pfrompopflagonly=int(flagged)), SEED)
        c.set(api.F_Q, Q)
        c.set(api.F_P, P)
        c.set(api.F_REP, np.array([7], np.int32))
        c.UpdateZ()
        assert c.sync() == 0
        np.testing.assert_array_equal(c.get(api.F_N), n_o)
        np.testing.assert_array_equal(c.get(api.F_M), m_o)
        if store:
            z = c.get(api.F_Z).astype(np.int32)
            z[z == 255] = -9
            np.testing.assert_array_equal(z, want_z)
        copies = int((geno >= 0).sum())
        assert abs(c.CalcLike() - orc.calc_like(geno, Q, P)) <= max(1, copies) * (K + 1) * 2.0 ** -24
        # the Metropolis move at the next multiple of METROFREQ
        c.set(api.F_REP, np.array([8], np.int32))
        c.UpdateQ()
        assert c.sync() == 0
        T = c.get(api.F_TESTQ).astype(np.float64)
        ld = np.zeros(N)
        for line in range(2):
            g = geno[:, line, :]
            ok = g >= 0
            Pa = P.astype(np.float64)[np.arange(L)[None, :], :, np.where(ok, g, 0)]   # [N][L][K]
            t = np.einsum("ik,ilk->il", T, Pa)
            q = np.einsum("ik,ilk->il", Q.astype(np.float64), Pa)
            ld += np.where(ok, np.log(np.where(ok, t, 1.0)) - np.log(np.where(ok, q, 1.0)), 0.0).sum(1)
        got = c.get(api.F_LOGDIFF)
        # each logarithm's magnitude is at most 104 (the smallest FP32 number)
        bound = 2 * L * ((K + 4) * 2.0 ** -51 + 104 * 2.0 ** -52) + 1e-300
        assert (np.abs(got - ld) <= bound).all(), np.abs(got - ld).max()
        c.close()
    d.close()


@pytest.mark.parametrize("K", [1, 2, 3, 4, 5, 8, 9, 13, 17, 25, 32])
def test_every_k_class(ctx, orc, K):
    _check(ctx, orc, 70, 41, K, 7)


@pytest.mark.parametrize("N,L,amax", [(1, 1, 2), (2, 5, 3), (255, 3, 9), (256, 17, 4), (257, 33, 5),
                                      (600, 600, 3), (40, 12, 64)])
def test_edges_of_tiles(ctx, orc, N, L, amax):
    _check(ctx, orc, N, L, 3, amax)


def test_counts_of_flagged_individuals(ctx, orc):
    _check(ctx, orc, 131, 57, 5, 6, flagged=True)


def test_batch_equals_chains_alone(ctx):
    rng = np.random.default_rng(5)
    geno, na = _geno(rng, 150, 60, 8)
    d = api.Data(ctx, na, geno=geno, layout=api.LAYOUT_U8)
    mk = lambda: [api.Chain(ctx, d, api.model_defaults(maxpops=K, burnin=1, numreps=9, freqscorr=1,
                                                       metrofreq=3, fpriormean=0.05, fpriorsd=0.05),
                            SEED + j) for j, K in enumerate([1, 4, 2, 10, 4])]
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
    d.close()
