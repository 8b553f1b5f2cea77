"""A chain in a batch has other lanes per locus than alone, and the same bits: every
state, every sum and all statistics (the F and alpha log likelihood differences and
ratios among them), and on 2-bit data the Metropolis log ratios (on one-byte data they
are FP64 atomic sums, whose order no launch fixes).  Small chains of two alleles beside
a large one, so that their 2 to 32 lanes become 1 or a few."""
import numpy as np
import pytest

from structure_b200 import api, synth

pytestmark = pytest.mark.gpu

FIELDS = [api.F_Q, api.F_LOGQ, api.F_TESTQ, api.F_P, api.F_LOGP, api.F_EPS, api.F_F, api.F_ALPHA,
          api.F_N, api.F_M, api.F_LOGDIFF, api.F_QSUM, api.F_PSUM, api.F_SUMEPS, api.F_FSTSUM,
          api.F_SUMALPHA, api.F_STATS]


def _data(ctx, N, L, layout, seed):
    d = synth.snp_fmodel(N, L, 3, np.linspace(0.02, 0.2, 3), 0.5, 0.03, seed)
    if layout == api.LAYOUT_B2G:
        return api.Data(ctx, d["numalleles"], packed=d["packed"], layout=layout, num_inds=N, num_loci=L)
    return api.Data(ctx, d["numalleles"], geno=synth.unpack_int32(d["packed"], N, 0, L), layout=layout)


# one locus; a warp's, a CTA's and several CTAs' loci at 1 to 32 lanes; large ones
# whose CTAs are 4, 8 and 16 per lane of the last sum
@pytest.mark.parametrize("layout,onefst,sizes", [
    (api.LAYOUT_B2G, 0, [1, 33, 300, 1100, 9001, 40000]),
    (api.LAYOUT_B2G, 1, [7, 255, 2500, 40000]),
    (api.LAYOUT_U8, 0, [65, 1300, 4700, 31000]),
    (api.LAYOUT_B2G, 0, [520, 37000, 40001])])
def test_statistics_do_not_depend_on_the_batch(ctx, layout, onefst, sizes):
    data = [_data(ctx, 20 + 5 * j, L, layout, 70 + j) for j, L in enumerate(sizes)]
    specs = [(d, K) for d in data for K in (1, 2, 3, 5, 20)]

    def mk():
        return [api.Chain(ctx, d, api.model_defaults(
            maxpops=K, burnin=1, numreps=9, freqscorr=1, onefst=onefst, metrofreq=2, popalphas=K % 2,
            fpriormean=0.05, fpriorsd=0.05), 900 + j) for j, (d, K) in enumerate(specs)]
    inb, alone = mk(), mk()
    b = api.Batch(ctx, inb)
    for _ in range(3):
        b.sweep(1)
        for c in alone:
            c.sweep(1)
        for x, y, (d, K) in zip(inb, alone, specs):
            assert x.sync() == 0 and y.sync() == 0
            for f in FIELDS:
                if f == api.F_LOGDIFF and layout == api.LAYOUT_U8:
                    continue
                np.testing.assert_array_equal(x.get(f), y.get(f), err_msg=f"L={d.L} K={K} field {f}")
    b.close()
    for c in inb + alone:
        c.close()
    for d in data:
        d.close()

