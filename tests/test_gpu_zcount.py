"""The counting Z pass (biallelic data, no stored Z) against the general pass,
which a chain that stores Z takes: the same Q, P and sweep give the same allele
and ancestry counts (whole numbers, exact, and equal to the oracle's counts) and
the same ln P(D).  Every K class, shapes at the edges of a word, a warp's loci, a
CTA's loci and a chunk, given tiles, and a batch that mixes both passes.

ln P(D): both passes add the same FP32 value per genotype word (at most 2e5 words
here) in FP64, in different orders: 2e5 x 2^-53 = 2.2e-11 relative.  The counting
pass first rounds each word to a quantum 2^-(47 - ceil(log2 words)), so that its
sums are exact at any tile: at most half a quantum a word more."""
import numpy as np
import pytest

from structure_b200 import api, synth

pytestmark = pytest.mark.gpu

SEED = 0x2C0DE
LIKE_RTOL = 2.2e-11


def _like_atol(N, L):
    words = L * ((N + 15) // 16)
    return words * 2.0 ** -(48 - int(np.ceil(np.log2(words))))


def _data(N, L, seed, missing=0.05):
    d = synth.snp_fmodel(N, L, 4, np.linspace(0.05, 0.25, 4), 0.4, missing, seed)
    return d["geno"], d["numalleles"]


def _state(rng, N, L, K, A):
    Q = rng.dirichlet(np.full(K, 0.3), N).astype(np.float32)
    P = rng.dirichlet(np.full(A, 0.4), (L, K)).astype(np.float32)
    return Q, P


def _chain(ctx, d, K, **kw):
    return api.Chain(ctx, d, api.model_defaults(maxpops=K, burnin=0, numreps=9, freqscorr=0,
                                                metrofreq=3, **kw), SEED)


def _compare(ctx, orc, geno, na, K, rep=4, **kw):
    N, _, L = geno.shape
    d = api.Data(ctx, na, geno=geno, layout=api.LAYOUT_B2G)
    cc, cg = _chain(ctx, d, K, **kw), _chain(ctx, d, K, store_z=1, **kw)
    Q, P = _state(np.random.default_rng(N + L + K), N, L, K, cc.A)
    for c in (cc, cg):
        c.set(api.F_Q, Q)
        c.set(api.F_P, P)
        c.set(api.F_REP, np.array([rep], np.int32))
        c.UpdateZ()
        assert c.sync() == 0
    zo = orc.zupdate_f32(geno, Q, P, SEED, rep)
    n_o, m_o = orc.counts(geno, zo, K, cc.A)
    for f, want in ((api.F_N, n_o), (api.F_M, m_o)):
        np.testing.assert_array_equal(cg.get(f), want)
        np.testing.assert_array_equal(cc.get(f), want)
    # collecting sweeps (Gibbs, Gibbs, Metropolis) from there
    for c in (cc, cg):
        c.sweep(3)
        assert c.sync() == 0
    for f in (api.F_N, api.F_M, api.F_Q, api.F_P):
        np.testing.assert_array_equal(cc.get(f), cg.get(f), err_msg=str(f))
    sc, sg, at = cc.get(api.F_STATS), cg.get(api.F_STATS), _like_atol(N, L)
    np.testing.assert_allclose(sc[:2], sg[:2], rtol=LIKE_RTOL, atol=3 * at)
    np.testing.assert_allclose(sc[2], sg[2], rtol=LIKE_RTOL, atol=6 * at * abs(sg[1]))
    assert sc[3] == sg[3] == 3
    for c in (cc, cg):
        c.close()
    d.close()


@pytest.mark.parametrize("K", [1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 16, 19, 20, 23, 32])
def test_every_k_class(ctx, orc, K):
    _compare(ctx, orc, *_data(150, 530, K), K)


@pytest.mark.parametrize("N,L", [(1, 1), (15, 31), (16, 32), (17, 33), (32, 256), (33, 257),
                                 (113, 255), (600, 40), (1037, 300)])
def test_edges_of_words_warps_and_tiles(ctx, orc, N, L):
    _compare(ctx, orc, *_data(N, L, N * L), 5)
    _compare(ctx, orc, *_data(N, L, N * L + 1), 9)


@pytest.mark.parametrize("tile", [dict(tile_t=16), dict(tile_t=112, tile_r=3), dict(tile_t=128),
                                  dict(tile_t=4096, tile_r=64)])
def test_given_tiles(ctx, orc, tile):
    _compare(ctx, orc, *_data(700, 900, 5), 6, **tile)


def test_missing_rows_loci_and_monomorphic_data(ctx, orc):
    geno, na = _data(90, 300, 77, missing=0.5)
    geno[7] = -9
    geno[:, :, 33] = -9
    _compare(ctx, orc, geno, na, 4)
    _compare(ctx, orc, geno, na, 10)
    mono = np.where(geno < 0, -9, 0).astype(np.int32)      # one allele everywhere: A = 1
    _compare(ctx, orc, mono, np.ones(300, np.int32), 3)


def test_tiny_terms_take_the_exact_logarithm(ctx):
    """Words whose products of terms leave FP32's range are logged in FP64: the
    pass on caller buffers against CalcLike (general pass) on the same Q and P."""
    import ctypes as C

    import torch
    N, L, K = 64, 256, 7
    geno, na = _data(N, L, 8)
    d = api.Data(ctx, na, geno=geno, layout=api.LAYOUT_B2G)
    c = _chain(ctx, d, K)
    Q, P = _state(np.random.default_rng(1), N, L, K, 2)
    P[::3, :, 0] = 1e-30
    P[::3, :, 1] = 1.0
    c.set(api.F_Q, Q)
    c.set(api.F_P, P)
    g2 = torch.from_numpy(synth.repack_from_int32(geno).view(np.int32)).cuda()
    q, p = torch.from_numpy(Q).cuda(), torch.from_numpy(P).cuda()
    n = torch.empty(L, K, 2, dtype=torch.int32, device="cuda")
    m = torch.empty(N, K, dtype=torch.int32, device="cuda")
    like = torch.empty(1, dtype=torch.float64, device="cuda")
    ptr = lambda t: C.c_void_p(t.data_ptr())
    assert api.lib().st_update_z_noalloc(0, ptr(g2), g2.shape[1], N, L, K, ptr(q), ptr(p), SEED, 0,
                                         ptr(n), ptr(m), ptr(like), None,
                                         C.c_void_p(torch.cuda.current_stream().cuda_stream),
                                         None) == api.ST_OK
    want = c.CalcLike()
    assert np.isfinite(want) and abs(like.item() - want) <= LIKE_RTOL * abs(want) + _like_atol(N, L)
    c.UpdateZ()
    np.testing.assert_array_equal(n.cpu().numpy(), c.get(api.F_N))
    np.testing.assert_array_equal(m.cpu().numpy(), c.get(api.F_M))
    c.close()
    d.close()


def test_batch_of_both_passes(ctx):
    """Chains that count flagged individuals only (general pass) next to chains of
    the same K class that count all: each as it is alone."""
    geno, na = _data(130, 400, 21)
    flags = (np.arange(130) % 3 > 0).astype(np.int32)
    d = api.Data(ctx, na, geno=geno, layout=api.LAYOUT_B2G, popflags=flags)
    spec = [(5, 0), (5, 1), (10, 1), (10, 0), (5, 0)]
    mk = lambda: [_chain(ctx, d, K, pfrompopflagonly=pf) for K, pf in spec]
    batched, alone = mk(), mk()
    b = api.Batch(ctx, batched)
    b.sweep(4)
    for c in alone:
        c.sweep(4)
    for cb, ca in zip(batched, alone):
        assert cb.sync() == 0 and ca.sync() == 0
        for f in (api.F_N, api.F_M, api.F_Q, api.F_P):
            np.testing.assert_array_equal(cb.get(f), ca.get(f))
    b.close()
    for c in batched + alone:
        c.close()
    d.close()
