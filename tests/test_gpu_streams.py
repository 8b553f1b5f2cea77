"""Sweeps on a caller's stream and reads right behind them, with no wait in between: the
results are those of a chain on its context's own stream, bit for bit.  The sweeps take
milliseconds, so a read that does not follow them sees an older state."""
import numpy as np
import pytest

from structure_b200 import api, synth

pytestmark = pytest.mark.gpu

N, L, K = 1000, 20000, 5
FIELDS = [api.F_N, api.F_P, api.F_Q, api.F_EPS, api.F_F, api.F_ALPHA, api.F_M]


@pytest.fixture(scope="module")
def words():
    return synth.snp_fmodel(N, L, 3, np.linspace(0.02, 0.2, 3), 0.5, 0.03, 4)["packed"]


class Run:
    def __init__(self, words, **kw):
        self.ctx = api.Context(0)
        self.data = api.Data(self.ctx, np.full(L, 2, np.int32), packed=words, layout=api.LAYOUT_B2G,
                             num_inds=N, num_loci=L)
        m = api.model_defaults(maxpops=K, burnin=0, numreps=1 << 30, freqscorr=1, computeprob=1,
                               fpriormean=0.05, fpriorsd=0.05, **kw)
        self.chain = api.Chain(self.ctx, self.data, m, 3)
        assert self.chain.sync() == 0

    def close(self):
        self.chain.close()
        self.data.close()
        self.ctx.close()


def _same(a, b):
    for f in FIELDS:
        np.testing.assert_array_equal(a.chain.get(f), b.chain.get(f), err_msg=str(f))


@pytest.mark.parametrize("stream", ["default", "its own"])
def test_sweeps_on_a_callers_stream(words, stream):
    import torch
    ts = torch.cuda.Stream()
    a, b = Run(words, metrofreq=3), Run(words, metrofreq=3)
    torch.cuda.synchronize()
    a.ctx.set_stream(1 if stream == "default" else ts.cuda_stream)
    a.chain.sweep(40)
    b.chain.sweep(40)
    assert b.chain.sync() == 0
    _same(a, b)
    assert a.chain.sync() == 0
    a.close()
    b.close()


def test_read_after_the_context_left_the_default_stream(words):
    a, b = Run(words, metrofreq=3), Run(words, metrofreq=3)
    b.chain.sweep(40)
    assert b.chain.sync() == 0
    want = [b.chain.get(f) for f in FIELDS]
    for f, w in zip(FIELDS, want):
        a.ctx.set_stream(1)
        a.chain.set(api.F_REP, np.array([0], np.int32))
        a.chain.sweep(40)
        a.ctx.set_stream(None)
        got = a.chain.get(f)
        if f == FIELDS[0]:   # the first 40 sweeps are b's; later rounds go on from there
            np.testing.assert_array_equal(got, w)
        else:
            np.testing.assert_array_equal(got, a.chain.get(f), err_msg=str(f))
    a.close()
    b.close()


def test_captured_sweeps_replayed_on_the_default_stream(words):
    import torch
    ts = torch.cuda.Stream()
    a, b = Run(words, metrofreq=0), Run(words, metrofreq=0)
    a.chain.sweep(2 + 3 * 20)
    assert a.chain.sync() == 0
    b.ctx.set_stream(ts.cuda_stream)
    b.chain.sweep(2)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=ts):
        b.chain.sweep(20)
    for _ in range(3):
        g.replay()
    _same(b, a)   # reads b first, right behind the replays
    torch.cuda.synchronize()
    del g
    a.close()
    b.close()


@pytest.mark.parametrize("field", [api.F_N, api.F_M])
def test_counts_set_behind_queued_sweeps(words, field):
    a = Run(words, metrofreq=0)
    want = np.ones((L, K, 2) if field == api.F_N else (N, K), np.int32)
    a.chain.sweep(40)
    a.chain.set(field, want)
    assert a.chain.sync() == 0
    np.testing.assert_array_equal(a.chain.get(field), want)
    a.close()
