"""A caller may set any Q and P (st_set_state refuses none).  With negative weights the
thresholds do not increase and their sum may be negative, where the draw's rule
z = #{k < K - 1 : C_k < r} still gives 0..K-1, also in a K class wider than K.  Passes
that store Z equal the oracle's rule and the counts of its Z."""
import numpy as np
import pytest

from structure_b200 import api

pytestmark = pytest.mark.gpu

SEED = 0x2A


@pytest.mark.parametrize("layout,A,K", [(api.LAYOUT_U8, 5, K) for K in (1, 5, 7, 9, 13, 17, 25, 32)]
                         + [(api.LAYOUT_B2G, 2, K) for K in (5, 13, 17, 21, 25, 31, 32)])
def test_negative_weights_draw_within_the_populations(ctx, orc, layout, A, K):
    N, L = 37, 70
    rng = np.random.default_rng(K)
    geno = np.sort(rng.integers(0, A, (N, 2, L)), axis=1).astype(np.int32)
    geno[np.broadcast_to(rng.random((N, 1, L)) < 0.1, geno.shape)] = -9
    Q = rng.normal(0, 1, (N, K)).astype(np.float32)
    Q[0] = -1.0 / K
    Q[1] = 0.0
    P = rng.dirichlet(np.ones(A), (L, K)).astype(np.float32)
    d = api.Data(ctx, np.full(L, A, np.int32), geno=geno, layout=layout)
    c = api.Chain(ctx, d, api.model_defaults(maxpops=K, freqscorr=0, store_z=1), SEED)
    c.set(api.F_Q, Q)
    c.set(api.F_P, P)
    c.set(api.F_REP, np.array([4], np.int32))
    c.UpdateZ()
    assert c.sync() == 0
    want = orc.zupdate_f32(geno, Q, P, SEED, 4)
    z = c.get(api.F_Z).astype(np.int32)
    z[z == 255] = -9
    np.testing.assert_array_equal(z, want)
    n, m = orc.counts(geno, want, K, A)
    np.testing.assert_array_equal(c.get(api.F_N), n)
    np.testing.assert_array_equal(c.get(api.F_M), m)
    c.close()
    d.close()
