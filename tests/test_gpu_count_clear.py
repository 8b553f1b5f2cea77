"""Every sweep starts its counts at zero, also for alleles that a locus' own number leaves
out: packed genotypes are not compared with num_alleles (a monomorphic locus may be
coded by its other allele), and a caller may set any counts.  The counts after a sweep
are those of one sweep's draws: alone as in a batch, and every copy present counts
once."""
import numpy as np
import pytest

from structure_b200 import api

pytestmark = pytest.mark.gpu


def _packed(rng, N, L):
    g = rng.integers(0, 4, (L, N)).astype(np.uint32)
    w = np.full((L, (N + 15) // 16 * 16), 3, np.uint32)
    w[:, :N] = g
    packed = (w.reshape(L, -1, 16) << (2 * np.arange(16, dtype=np.uint32))).sum(2, dtype=np.uint32)
    return packed, 2 * (g != 3).sum(1)


def _model(K, **kw):
    return api.model_defaults(maxpops=K, burnin=0, numreps=9, metrofreq=2, **kw)


# few loci (several lanes each) and many (one lane each); general pass with PFROMPOPFLAGONLY
@pytest.mark.parametrize("L,K,freqscorr", [(70, 3, 1), (70, 17, 0), (1200, 5, 1), (40000, 2, 1)])
def test_understated_alleles_of_packed_loci(ctx, L, K, freqscorr):
    N = 37
    rng = np.random.default_rng(L + K)
    packed, copies = _packed(rng, N, L)
    na = rng.integers(0, 3, L).astype(np.int32)
    na[0] = 2
    d = api.Data(ctx, na, packed=packed, layout=api.LAYOUT_B2G, num_inds=N, num_loci=L)
    alone, inb = (api.Chain(ctx, d, _model(K, freqscorr=freqscorr), 99) for _ in range(2))
    b = api.Batch(ctx, [inb])
    for _ in range(3):
        alone.sweep(1)
        b.sweep(1)
        n = alone.get(api.F_N)
        np.testing.assert_array_equal(n.sum((1, 2)), copies)
        np.testing.assert_array_equal(n, inb.get(api.F_N))
        assert alone.get(api.F_M).sum() == copies.sum()
    assert alone.sync() == 0 and inb.sync() == 0
    b.close()
    alone.close()
    inb.close()
    d.close()


@pytest.mark.parametrize("L", [50, 40000])
def test_counts_set_beyond_a_locus_alleles(ctx, L):
    N, K = 6, 2
    rng = np.random.default_rng(L)
    na = rng.integers(1, 6, L).astype(np.int32)
    na[0] = 5
    geno = (rng.random((N, 2, L)) * na).astype(np.int32)
    d = api.Data(ctx, na, geno=geno, layout=api.LAYOUT_U8)
    c = api.Chain(ctx, d, _model(K, freqscorr=1), 7)
    c.set(api.F_N, np.ones((L, K, 5), np.int32))
    c.sweep(1)
    assert c.sync() == 0
    n = c.get(api.F_N)
    want = np.zeros((L, 5), np.int64)
    for a in range(5):
        want[:, a] = (geno == a).sum((0, 1))
    np.testing.assert_array_equal(n.sum(1), want)
    c.close()
    d.close()
