"""The Metropolis pass and CalcLike on 2-bit data: every K class, the edges of a word, a
warp's loci, a CTA's loci and a chunk, given tiles, one-allele data and products near
FP32's lower end.  Log ratios against FP64 within the derived bound of the FP32 terms
(conftest.metro_terms_and_bound); ln P(D) of a chain without stored Z (pass without
draws) against one with (general pass): the same words' FP32 values, which the first
rounds to half a quantum each (test_gpu_zcount), summed in FP64."""
import numpy as np
import pytest

from conftest import metro_terms_and_bound
from structure_b200 import api, synth
from test_gpu_zcount import LIKE_RTOL, _chain, _data, _like_atol, _state

pytestmark = pytest.mark.gpu


def _check(ctx, geno, na, K, tiny=False, **kw):
    N, _, L = geno.shape
    d = api.Data(ctx, na, geno=geno, layout=api.LAYOUT_B2G)
    cc, cg = _chain(ctx, d, K, **kw), _chain(ctx, d, K, store_z=1, **kw)
    Q, P = _state(np.random.default_rng(N + 5 * L + K), N, L, K, cc.A)
    if tiny:
        P[::4, :, 0] = 1e-30
        P[::4, :, 1] = 1.0
    for c in (cc, cg):
        c.set(api.F_Q, Q)
        c.set(api.F_P, P)
    a, b = cc.CalcLike(), cg.CalcLike()
    assert np.isfinite(a) and abs(a - b) <= LIKE_RTOL * abs(b) + _like_atol(N, L)
    cc.set(api.F_REP, np.array([3], np.int32))       # a multiple of METROFREQ = 3
    cc.UpdateQ()
    assert cc.sync() == 0
    ld, _, bnd = metro_terms_and_bound(geno, Q, cc.get(api.F_TESTQ), P)
    assert (np.abs(cc.get(api.F_LOGDIFF) - ld) <= bnd + 1e-12).all()
    for c in (cc, cg):
        c.close()
    d.close()


@pytest.mark.parametrize("K", [1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 16, 20, 24, 32])
def test_every_k_class(ctx, K):
    _check(ctx, *_data(90, 300, K + 1), K)


@pytest.mark.parametrize("N,L", [(1, 1), (15, 31), (17, 33), (33, 257), (113, 64), (600, 40),
                                 (300, 900)])
def test_edges(ctx, N, L):
    for K in (5, 9, 17):
        _check(ctx, *_data(N, L, N * L + 2), K)


def test_tiles_alleles_and_small_terms(ctx):
    geno, na = _data(260, 700, 12)
    _check(ctx, geno, na, 6, tile_t=32, tile_r=2)
    _check(ctx, geno, na, 3, tile_t=512)
    _check(ctx, geno, na, 7, tiny=True)
    _check(ctx, geno, na, 17, tiny=True)
    _check(ctx, np.where(geno < 0, -9, 0).astype(np.int32), np.ones(700, np.int32), 4)
