"""One-byte genotypes are turned to [L][N][2] on upload through tiles of 64 copies x 64
loci, and the per-genotype kernel (initial Z, counts of a given Z, FP64 draws) walks
them individuals side by side: around the tiles' edges every genotype is where the
oracle has it."""
import numpy as np
import pytest

from structure_b200 import api

pytestmark = pytest.mark.gpu

SEED = 77


@pytest.mark.parametrize("N,L", [(1, 1), (31, 65), (32, 64), (33, 63), (64, 1), (65, 129), (300, 3)])
def test_genotypes_after_upload(ctx, orc, N, L):
    K, A = 3, 6
    rng = np.random.default_rng(N + L)
    geno = rng.integers(0, A, (N, 2, L)).astype(np.int32)
    geno[rng.random((N, 2, L)) < 0.1] = -9
    d = api.Data(ctx, np.full(L, A, np.int32), geno=geno, layout=api.LAYOUT_U8)
    m = dict(maxpops=K, freqscorr=0, store_z=1)
    c = api.Chain(ctx, d, api.model_defaults(**m), SEED)

    def same(z):
        got = c.get(api.F_Z).astype(np.int32)
        got[got == 255] = -9
        np.testing.assert_array_equal(got, z)
        n, ma = orc.counts(geno, z, K, A)
        np.testing.assert_array_equal(c.get(api.F_N), n)
        np.testing.assert_array_equal(c.get(api.F_M), ma)

    same(orc.init_z(geno, K, SEED))
    Q = rng.dirichlet(np.ones(K), N).astype(np.float32)
    P = rng.dirichlet(np.ones(A), (L, K)).astype(np.float32)
    c.set(api.F_Q, Q)
    c.set(api.F_P, P)
    z = rng.integers(0, K, geno.shape).astype(np.int32)
    z[geno < 0] = -9
    c.set(api.F_Z, np.where(z < 0, 255, z).astype(np.uint8))
    same(z)
    c.UpdateZ()
    same(orc.zupdate_f32(geno, Q, P, SEED, 0))
    # FP64: ln P(D) of the state; each copy's sum of K products is K 2^-52 relative off at
    # most on either side, its logarithm (at most 115) and the running sum 2^-52 each
    c64 = api.Chain(ctx, d, api.model_defaults(precision=1, **m), SEED)
    c64.set(api.F_Q, Q)
    c64.set(api.F_P, P)
    copies = int((geno >= 0).sum())
    bound = max(1, copies) * (2 * K + 2 * 115) * 2.0 ** -52 + copies ** 2 * 115 * 2.0 ** -52
    assert abs(c64.CalcLike() - orc.calc_like(geno, Q, P)) <= bound
    c64.UpdateZ()
    m64 = c64.get(api.F_M)
    np.testing.assert_array_equal(m64.sum(1), (geno >= 0).sum((1, 2)))
    assert c.sync() == 0 and c64.sync() == 0
    c.close()
    c64.close()
    d.close()
