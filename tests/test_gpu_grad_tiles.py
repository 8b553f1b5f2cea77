"""The FP32 gradient passes at the edges of their tiles: every class of K, single
individuals and loci, a pair cut in two, stages, chunks and CTAs cut short, missing
genotypes, and logits so large that products of terms leave FP32's safe range (the
factor-by-factor branch).  FP64 takes the same classes.

Bounds as in the gradient tests, with unit roundoff u = 2^-24 (FP32): an entry is
p (g - <p, g>), g a sum of n positive terms, so its error is at most (n + K + 16 +
2 X) u times p (g + <p, g>); X, the largest |logit - row maximum|, is the relative
error that rounding the exponent's argument adds to a softmax value.  ln P(D) sums
n_copies logarithms of relative error (K + 8 + 2 X) u each, in FP32 partial sums of 32
loci."""
import numpy as np
import pytest

from structure_b200 import api, synth
from structure_b200.grad import LogLikGrad
from test_gpu_grad import _grad_scales

pytestmark = pytest.mark.gpu


def _check(ctx, orc, N, L, K, scale, bits=32, missing=0.1):
    import torch
    d = synth.snp_fmodel(N, L, 3, [0.05, 0.1, 0.2], 0.4, missing, N + 3 * L + K)
    geno = d["geno"]
    na = np.full(L, 2, np.int32)
    data = api.Data(ctx, na, packed=d["packed"], layout=api.LAYOUT_B2G, num_inds=N, num_loci=L)
    rng = np.random.default_rng(N + L + K)
    dt = np.float32 if bits == 32 else np.float64
    ql, pl = rng.normal(0, scale, (N, K)).astype(dt), rng.normal(0, scale, (L, K, 2)).astype(dt)
    ev = LogLikGrad(ctx, data, K, precision=bits)
    ll, dq, dp, lli = ev(torch.tensor(ql, device="cuda"), torch.tensor(pl, device="cuda"),
                         per_individual=True)
    torch.cuda.synchronize()
    q64, p64 = ql.astype(np.float64), pl.astype(np.float64)
    llo, dqo, dpo, llio = orc.loglik_grad(geno, q64, p64)
    u = 2.0 ** -24 if bits == 32 else 2.0 ** -53
    X = max(np.abs(q64 - q64.max(1, keepdims=True)).max(), np.abs(p64 - p64.max(2, keepdims=True)).max())
    sq, sp = _grad_scales(geno, q64, p64)
    tiny = 1e-30 if bits == 32 else 1e-290       # below it the values themselves lose digits
    for dev, ref, s, n in ((dq, dqo, sq, 2 * L), (dp, dpo, sp, 2 * N)):
        err = np.abs(dev.cpu().numpy().astype(np.float64) - ref)
        bound = (n + K + 16 + 2 * X) * u * s + tiny
        assert (err <= bound).all(), (err / bound).max()
    copies = (geno >= 0).sum((1, 2))
    eb = copies * (K + 8 + 2 * X) * u + 40 * u * np.abs(llio)
    assert (np.abs(lli.cpu().numpy() - llio) <= eb + 1e-12).all()
    assert abs(ll.item() - llo) <= eb.sum() + 1e-12
    ev.close()
    data.close()


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("K", [1, 2, 3, 4, 5, 6, 7, 9, 11, 12, 16])
def test_every_k_class(ctx, orc, K, bits):
    _check(ctx, orc, 45, 70, K, 1.5, bits)


@pytest.mark.parametrize("N,L", [(1, 1), (2, 3), (15, 31), (17, 33), (255, 64), (257, 65), (65, 257),
                                 (700, 130)])
def test_edges_of_tiles(ctx, orc, N, L):
    _check(ctx, orc, N, L, 8, 1.5)
    _check(ctx, orc, N, L, 5, 1.5, missing=0.0)


@pytest.mark.parametrize("K", [2, 8, 13])
def test_terms_near_the_ends_of_the_range(ctx, orc, K):
    _check(ctx, orc, 40, 96, K, 18.0)
