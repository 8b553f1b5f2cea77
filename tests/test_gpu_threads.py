"""Two host threads, each with a context of its own, launch the same kernels with
different amounts of shared memory: the limit belongs to the function, so neither may
lower it under the other.  Chains of one K class whose tiles (or allele tables) differ,
all above the default limit of 48 KB; every call succeeds and the draws are those of
the chain alone."""
import threading

import numpy as np
import pytest

from structure_b200 import api, synth

pytestmark = pytest.mark.gpu

CALLS = 1500


def _chain(ctx, kind, which):
    if kind == "one byte":
        L, A = 2600, (64, 58)[which]
        rng = np.random.default_rng(which)
        geno = rng.integers(0, A, (20, 2, L)).astype(np.int32)
        d = api.Data(ctx, np.full(L, A, np.int32), geno=geno, layout=api.LAYOUT_U8)
        return d, api.Chain(ctx, d, api.model_defaults(maxpops=6, freqscorr=0), 5)
    N, L = 512, 256
    s = synth.snp_fmodel(N, L, 3, np.linspace(0.02, 0.2, 3), 0.5, 0.03, 8)
    d = api.Data(ctx, s["numalleles"], packed=s["packed"], layout=api.LAYOUT_B2G, num_inds=N, num_loci=L)
    return d, api.Chain(ctx, d, api.model_defaults(maxpops=8, freqscorr=0, store_z=int(kind == "general"),
                                                   tile_t=(64, 192)[which]), 5)


@pytest.mark.parametrize("kind", ["counting", "general", "one byte"])
def test_two_threads_with_different_tiles(kind):
    api.lib()
    errors, counts = [], [None, None]
    start = threading.Barrier(2, timeout=60)

    def work(which):
        try:
            ctx = api.Context(0)
            d, c = _chain(ctx, kind, which)
            c.UpdateZ()
            c.sync()
            want = c.get(api.F_N)
            start.wait()
            for _ in range(CALLS):
                c.UpdateZ()
            assert c.sync() == 0
            np.testing.assert_array_equal(c.get(api.F_N), want)
            counts[which] = want.sum()
            c.close()
            d.close()
            ctx.close()
        except BaseException as e:   # reported below: a thread's exception is lost
            errors.append(e)
            start.abort()

    threads = [threading.Thread(target=work, args=(w,)) for w in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    assert all(n > 0 for n in counts)
