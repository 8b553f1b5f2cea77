"""The work that programs give this library, as cases that can be timed.

A case is one call sequence through the public entry points on seeded synthetic
data drawn from the model STRUCTURE assumes: MCMC sweeps of chains over SNP data
(biallelic, packed 2 bits a genotype) or microsatellites (many alleles, one byte a
copy), the updates called one by one as a host run loop does, one Z update on the
caller's own device buffers, and ln P(D) with its gradient.

A pass of a sweep case is UPDATEFREQ sweeps and the reads that a program makes
after them: the state it prints and the sums it writes at the end.  Ten sweeps hold
one Metropolis sweep (METROFREQ = 10), the reference's own schedule.
"""
import ctypes as C
import math

import numpy as np
import torch

from structure_b200 import api, synth
from structure_b200.grad import LogLikGrad, loglik

METROFREQ = 10


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # one Z update of a handful of individuals on the caller's buffers: the
        # smallest call there is, where launches and host work count
        dict(name="z update, tiny", kind="zupdate", inds=50, loci=100, pops=2),
        # the classic small study, one chain by st_sweep: N=200, L=100
        # microsatellites, K=3, independent frequencies
        dict(name="microsatellites, one chain", kind="sweep", data="usat", inds=200, loci=100,
             pops=3, chains=1, sweeps=100, model="indep", batch=False),
        # replicate runs of a larger microsatellite panel, batched
        dict(name="microsatellites, replicates", kind="sweep", data="usat", inds=1000, loci=300,
             pops=6, chains=8, sweeps=20, model="fmodel", batch=True),
        # one chain of ragged shape (no multiple of a word, a warp or a block)
        dict(name="snp, one ragged chain", kind="sweep", data="snp", inds=733, loci=9973, pops=3,
             chains=1, sweeps=10, model="fmodel", batch=False),
        # the updates called one by one, as a host run loop drives them
        dict(name="snp, step by step", kind="steps", data="snp", inds=1000, loci=10001, pops=4,
             sweeps=10),
        # one population per individual
        dict(name="snp, no admixture", kind="sweep", data="snp", inds=2500, loci=20000, pops=4,
             chains=1, sweeps=10, model="noadmix", batch=False),
        # a K larger than most studies use
        dict(name="snp, wide K", kind="sweep", data="snp", inds=1200, loci=12007, pops=20,
             chains=2, sweeps=10, model="fmodel", batch=True),
        # a study over K: 40 chains, K = 1..10 on four data sets of uneven shape
        dict(name="snp, study over K", kind="study", maxpops=10, sweeps=10, scale=1.0),
        # the benchmark's workload: 20 replicate chains of N=2000, L=50,000, K=5
        dict(name="snp, replicates", kind="sweep", data="snp", inds=2000, loci=50000, pops=5,
             chains=20, sweeps=10, model="fmodel", batch=True),
        # many individuals and loci, K=10, one alpha per population
        dict(name="snp, large", kind="sweep", data="snp", inds=10000, loci=100000, pops=10,
             chains=4, sweeps=10, model="popalphas", batch=True),
        # ln P(D) and its gradient in double precision, as finite differences check it
        dict(name="gradient, float64", kind="grad", inds=1000, loci=5000, pops=5, bits=64),
        # ln P(D) and its gradient, forward and backward, N=5000, L=100,000, K=8
        dict(name="gradient, float32", kind="grad", inds=5000, loci=100000, pops=8, bits=32),
    ]


def _spread(rng, lo, hi):
    """A whole number of lo..hi, even over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _cost(c):
    """About what a pass costs, to keep a drawn case below the largest listed one."""
    if c["kind"] == "study":
        return 1e8 * c["scale"] ** 2 * c["maxpops"] * (c["maxpops"] + 8) * c["sweeps"]
    n = float(c["inds"]) * c["loci"] * (c["pops"] + 8) * c.get("chains", 1) * c.get("sweeps", 1)
    return n * (4 if c.get("data") == "usat" or c.get("bits") == 64 else 1)


def draw(rng):
    most = max(_cost(c) for c in listed())
    while True:
        kind = rng.choice(["sweep"] * 6 + ["usat"] * 3 + ["steps", "zupdate", "zupdate", "study"]
                          + ["grad"] * 3)
        if kind == "sweep":
            c = dict(kind="sweep", data="snp", inds=_spread(rng, 30, 10000),
                     loci=_spread(rng, 200, 100000), pops=_spread(rng, 1, 24),
                     chains=rng.choice([1, 1, 2, 4, 8, 20]), sweeps=10,
                     model=rng.choice(["fmodel", "fmodel", "fmodel", "indep", "popalphas",
                                       "noadmix"]), batch=rng.random() < 0.7)
        elif kind == "usat":
            c = dict(kind="sweep", data="usat", inds=_spread(rng, 30, 2000),
                     loci=_spread(rng, 8, 500), pops=_spread(rng, 1, 12),
                     chains=rng.choice([1, 1, 4, 8]), sweeps=20,
                     model=rng.choice(["indep", "fmodel", "noadmix", "locprior"]),
                     batch=rng.random() < 0.7)
        elif kind == "steps":
            c = dict(kind="steps", data=rng.choice(["snp", "snp", "usat"]),
                     inds=_spread(rng, 30, 2000), loci=_spread(rng, 100, 20000),
                     pops=_spread(rng, 1, 12), sweeps=10)
            if c["data"] == "usat":
                c["loci"] = min(500, c["loci"])
        elif kind == "zupdate":
            c = dict(kind="zupdate", inds=_spread(rng, 20, 10000), loci=_spread(rng, 50, 50000),
                     pops=_spread(rng, 1, 24))
        elif kind == "study":
            c = dict(kind="study", maxpops=rng.randint(2, 10), sweeps=10,
                     scale=round(rng.uniform(0.1, 0.9), 3))
        else:
            c = dict(kind="grad", inds=_spread(rng, 100, 5000), loci=_spread(rng, 200, 100000),
                     pops=_spread(rng, 1, 16), bits=rng.choice([32, 32, 64]))
            if c["bits"] == 64:
                c["loci"] = min(10000, c["loci"])
        if c["kind"] == "zupdate" and 8 * c["loci"] * c["pops"] + 4 * c["inds"] * c["pops"] > 24 << 20:
            continue   # that entry point's scratch is 32 MiB
        if _cost(c) <= 0.9 * most:
            return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _dirichlet(n, K, a, gen):
    g = torch.distributions.Gamma(torch.full((n, K), a, device="cuda"), 1.0)
    torch.manual_seed(int(torch.randint(1 << 30, (1,), generator=gen, device="cuda")))
    x = g.sample().clamp_min(1e-12)
    return x / x.sum(1, keepdim=True)


def _snp(N, L, K, seed, missing=0.03):
    """SNP genotypes under the F model (Fst 0.05..0.25, Q ~ Dirichlet(0.3)), packed 16
    individuals a word and locus-major as int32 on the GPU, with the alleles per locus.
    The first copy seen at a locus is allele 0, as the reference's recoding leaves it."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    Kt = max(2, min(K, 10))
    Q = _dirichlet(N, Kt, 0.3, gen)
    fst = torch.linspace(0.05, 0.25, Kt, device="cuda")
    wpr = (N + 15) // 16
    packed = torch.empty(L, wpr, dtype=torch.int32, device="cuda")
    na = torch.empty(L, dtype=torch.int32, device="cuda")
    shift = (2 * torch.arange(16, device="cuda", dtype=torch.int32)).view(1, 1, 16)
    step = max(1, min(L, int(6e7) // max(1, N)))
    for l0 in range(0, L, step):
        n = min(step, L - l0)
        p = torch.rand(n, generator=gen, device="cuda").clamp(0.01, 0.99)
        sd = (p * (1 - p))[:, None].sqrt() * fst.sqrt()[None, :]
        P = (p[:, None] + sd * torch.randn(n, Kt, generator=gen, device="cuda")).clamp(1e-3, 1 - 1e-3)
        freq = P @ Q.T                                                    # [n, N]
        g = (torch.rand(n, N, generator=gen, device="cuda") < freq).to(torch.int32)
        g += torch.rand(n, N, generator=gen, device="cuda") < freq
        seen = torch.rand(n, N, generator=gen, device="cuda") >= missing
        first = seen.to(torch.uint8).argmax(1)
        flip = g[torch.arange(n, device="cuda"), first] == 2
        g = torch.where(flip[:, None], 2 - g, g)
        one = ((g > 0) & seen).any(1)
        na[l0:l0 + n] = torch.where(seen.any(1), 1 + one.to(torch.int32), 0)
        g = torch.where(seen, g, 3)
        full = torch.full((n, wpr * 16), 3, dtype=torch.int32, device="cuda")
        full[:, :N] = g
        packed[l0:l0 + n] = (full.view(n, wpr, 16) << shift).sum(2, dtype=torch.int32)
    return packed, na


def _usat(N, L, K, seed, missing=0.05):
    """Microsatellites: 2..10 alleles a locus, copies missing one by one."""
    rng = np.random.default_rng(int(seed))
    Q = rng.dirichlet(np.full(max(2, K), 0.5), N)
    cq = np.cumsum(Q, 1)
    cq[:, -1] = 1.0
    A = rng.integers(2, 11, L)
    geno = np.empty((N, 2, L), np.int32)
    for l in range(L):
        cp = np.cumsum(rng.dirichlet(np.ones(A[l]), Q.shape[1]), 1)
        cp[:, -1] = 1.0
        z = (rng.random((N, 2, 1)) > cq[:, None, :]).sum(2)
        geno[:, :, l] = (rng.random((N, 2, 1)) > cp[z]).sum(2)
    geno[rng.random((N, 2, L)) < missing] = synth.MISSING
    return synth.recode(geno)


def _model(case, K):
    kw = dict(maxpops=K, burnin=0, numreps=1 << 30, metrofreq=METROFREQ, alphapropsd=0.025,
              computeprob=1, freqscorr=1, fpriormean=0.01, fpriorsd=0.05)
    m = case.get("model", "fmodel")
    if m in ("indep", "locprior") or case.get("data") == "usat" and m == "noadmix":
        kw.update(freqscorr=0)
    if m == "popalphas":
        kw.update(popalphas=1)
    if m == "noadmix":
        kw.update(noadmix=1, admburnin=-1)
    if m == "locprior":
        kw.update(locprior=1)
    return api.model_defaults(**kw)


class _Chains:
    """Chains of a case with all that a program holds for them."""

    def __init__(self):
        self.ctx, self.datas, self.chains, self.batch, self.ev = api.Context(0), [], [], None, None

    def add_data(self, case, N, L, K, seed):
        kw = {}
        if case.get("model") == "locprior":
            kw["location"] = (np.arange(N) % 5).astype(np.int32)
        if case.get("data") == "usat":
            geno, na = _usat(N, L, K, seed)
            d = api.Data(self.ctx, na, geno=geno, **kw)
        else:
            packed, na = _snp(N, L, K, seed)
            d = api.Data(self.ctx, na.cpu().numpy(), packed=packed.cpu().numpy().view(np.uint32),
                         layout=api.LAYOUT_B2G, num_inds=N, num_loci=L, **kw)
        self.datas.append(d)
        return d

    def buffers(self, fields):
        """One page-locked array a field for all chains, and each chain's part of it."""
        self.out, self.parts = {}, [dict() for _ in self.chains]
        for name, f in fields.items():
            dt = api._DT[f]
            n = [api.lib().st_field_bytes(c.h, f) // np.dtype(dt).itemsize for c in self.chains]
            t = torch.empty(sum(n), dtype=getattr(torch, np.dtype(dt).name), pin_memory=True)
            self.out[name], at = t, 0
            for c, k in enumerate(n):
                self.parts[c][f] = t.numpy()[at:at + k]
                at += k

    def read(self):
        for c, part in zip(self.chains, self.parts):
            for f, a in part.items():
                c.get(f, out=a)
        return dict(self.out)

    def __del__(self):
        try:
            for h in ([self.batch] if self.batch else []) + ([self.ev] if self.ev else []):
                h.close()
            for h in self.chains + self.datas + [self.ctx]:
                h.close()
        except Exception:
            pass


RESULTS = dict(q=api.F_Q, qsum=api.F_QSUM, psum=api.F_PSUM, alpha=api.F_ALPHA, m=api.F_M,
               stats=api.F_STATS)
STUDY = [(300, 5000), (1000, 10000), (2500, 20000), (4000, 8000)]


def _study_shapes(case):
    return [(max(20, int(N * case["scale"])), max(50, int(L * case["scale"]))) for N, L in STUDY]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "zupdate":
        return _prepare_zupdate(case, seed)
    s = _Chains()
    s.case = case
    if kind == "grad":
        N, L, K = case["inds"], case["loci"], case["pops"]
        s.ev = LogLikGrad(s.ctx, s.add_data(case, N, L, K, seed), K, precision=case["bits"])
        s.q, s.p = (x.requires_grad_(True) for x in _logits(case, seed))
        return s
    if kind == "study":
        for j, (N, L) in enumerate(_study_shapes(case)):
            s.add_data(case, N, L, 4, seed * 4 + j)
        s.chains = [api.Chain(s.ctx, d, _model(case, K), seed * 1000 + 10 * K + j)
                    for K in range(1, case["maxpops"] + 1) for j, d in enumerate(s.datas)]
    else:
        N, L, K = case["inds"], case["loci"], case["pops"]
        d = s.add_data(case, N, L, K, seed)
        s.chains = [api.Chain(s.ctx, d, _model(case, K), seed * 1000 + j)
                    for j in range(case.get("chains", 1))]
    if kind == "steps":
        s.rep = 0
        s.buffers(dict(q=api.F_Q, p=api.F_P, eps=api.F_EPS, n=api.F_N, m=api.F_M, alpha=api.F_ALPHA,
                       f=api.F_F, stats=api.F_STATS))
        return s
    if case.get("batch", True):
        s.batch = api.Batch(s.ctx, s.chains)
    s.buffers(RESULTS)
    return s


def _logits(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed) + 7)
    dt = torch.float64 if case["bits"] == 64 else torch.float32
    N, L, K = case["inds"], case["loci"], case["pops"]
    return (torch.randn(N, K, generator=gen, device="cuda", dtype=dt),
            torch.randn(L, K, 2, generator=gen, device="cuda", dtype=dt))


def _prepare_zupdate(case, seed):
    N, L, K = case["inds"], case["loci"], case["pops"]
    gen = torch.Generator(device="cuda").manual_seed(int(seed) + 3)
    g2, _ = _snp(N, L, K, seed)
    q = _dirichlet(N, K, 0.5, gen).contiguous()
    p0 = torch.rand(L, K, generator=gen, device="cuda").clamp(1e-4, 1 - 1e-4)
    p = torch.stack([p0, 1 - p0], 2).contiguous()
    i32 = dict(dtype=torch.int32, device="cuda")
    return dict(case=case, seed=int(seed), g2=g2, q=q, p=p, n=torch.empty(L, K, 2, **i32),
                m=torch.empty(N, K, **i32), err=torch.empty(1, **i32),
                like=torch.empty(1, dtype=torch.float64, device="cuda"))


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(s):
    if isinstance(s, dict):
        return _run_zupdate(s)
    case = s.case
    if case["kind"] == "grad":
        s.q.grad = s.p.grad = None
        out = loglik(s.q, s.p, s.ev)
        out.backward()
        return dict(loglik=out.detach(), dq=s.q.grad, dp=s.p.grad)
    if case["kind"] == "steps":
        return _run_steps(s)
    if s.batch:
        s.batch.sweep(case["sweeps"])
    else:
        for c in s.chains:
            c.sweep(case["sweeps"])
    return s.read()


def _run_steps(s):
    """The loop of the reference's main program over single updates."""
    c, admix = s.chains[0], s.case.get("model", "fmodel") != "noadmix"
    for _ in range(s.case["sweeps"]):
        c.set(api.F_REP, np.array([s.rep], np.int32))
        c.UpdateP()
        c.UpdateQ()
        if admix:
            c.UpdateAlpha()
        c.UpdateEpsilon()
        c.UpdateFst()
        c.UpdateZ()
        c.DataCollection()
        s.rep += 1
    return s.read()


def _run_zupdate(s):
    c = s["case"]
    rc = api.lib().st_update_z_noalloc(
        0, C.c_void_p(s["g2"].data_ptr()), s["g2"].shape[1], c["inds"], c["loci"], c["pops"],
        C.c_void_p(s["q"].data_ptr()), C.c_void_p(s["p"].data_ptr()), s["seed"], 5,
        C.c_void_p(s["n"].data_ptr()), C.c_void_p(s["m"].data_ptr()),
        C.c_void_p(s["like"].data_ptr()), C.c_void_p(s["err"].data_ptr()),
        C.c_void_p(torch.cuda.current_stream().cuda_stream), None)
    if rc != api.ST_OK:
        raise RuntimeError("st_update_z_noalloc: %d" % rc)
    return dict(n=s["n"], m=s["m"], like=s["like"], err=s["err"])


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _sweep_work(N, L, K, A, gbits, chains):
    """Bytes and operations of one sweep of `chains` chains over one data set: the
    genotypes once, every chain's Q, P and counts once, and the K-term mixture weights
    of both copies of every genotype."""
    state = N * K * (4 + 4) + L * K * A * (4 + 4)
    return N * L * gbits / 8 + chains * state, chains * 4.0 * K * N * L


def work(case):
    kind = case["kind"]
    if kind == "grad":
        N, L, K, e = case["inds"], case["loci"], case["pops"], case["bits"] // 8
        return dict(bytes=N * L / 4 + 2 * e * (N * K + 2 * L * K), flops=16.0 * K * N * L)
    if kind == "study":
        b = f = 0.0
        for N, L in _study_shapes(case):
            for K in range(1, case["maxpops"] + 1):
                x, y = _sweep_work(N, L, K, 2, 2 if K == 1 else 0, 1)
                b, f = b + x, f + y
        return dict(bytes=b * case["sweeps"], flops=f * case["sweeps"])
    usat = case.get("data") == "usat"
    b, f = _sweep_work(case["inds"], case["loci"], case["pops"], 10 if usat else 2,
                       16 if usat else 2, case.get("chains", 1))
    return dict(bytes=b * case.get("sweeps", 1), flops=f * case.get("sweeps", 1))


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
def _unpack(packed, N, l0, l1):
    w = packed[l0:l1].to(torch.int64) & 0xFFFFFFFF
    sh = 2 * torch.arange(16, device="cuda", dtype=torch.int64)
    return ((w[:, :, None] >> sh) & 3).reshape(l1 - l0, -1)[:, :N]


def exact(case, seed):
    """ln P(D) and its gradient have a value in 64 bits; a chain's state is drawn, and has
    none apart from its generator."""
    N, L, K = (case.get(k) for k in ("inds", "loci", "pops"))
    if case["kind"] == "zupdate":
        s = _prepare_zupdate(case, seed)
        q, p = s["q"].double(), s["p"].double()
        step, like = max(1, int(4e7) // N), 0.0
        for l0 in range(0, L, step):
            l1 = min(L, l0 + step)
            g = _unpack(s["g2"], N, l0, l1)
            s0, s1 = (torch.log((p[l0:l1, :, a] @ q.T).clamp_min(1e-50)) for a in (0, 1))
            like += float(((g == 0) * 2 * s0 + (g == 1) * (s0 + s1) + (g == 2) * 2 * s1).sum())
        return dict(n=None, m=None, err=None,
                    like=torch.tensor([like], dtype=torch.float64, device="cuda"))
    if case["kind"] != "grad":
        return None
    packed, _ = _snp(N, L, K, seed)
    ql, pl = (x.double() for x in _logits(case, seed))
    Q, P = torch.softmax(ql, 1), torch.softmax(pl, 2)
    gq, gp, ll = torch.zeros_like(Q), torch.zeros_like(P), 0.0
    step = max(1, int(4e7) // N)
    for l0 in range(0, L, step):
        l1 = min(L, l0 + step)
        g = _unpack(packed, N, l0, l1)
        for a in (0, 1):
            S = P[l0:l1, :, a] @ Q.T                                      # [n, N]
            copies = (g == 2 * a) * 2.0 + (g == 1)
            ll += float((copies * torch.log(S)).sum())
            w = copies / S
            gq += w.T @ P[l0:l1, :, a]
            gp[l0:l1, :, a] += w @ Q
    return dict(loglik=torch.tensor(ll, dtype=torch.float64, device="cuda"),
                dq=Q * (gq - (Q * gq).sum(1, keepdim=True)),
                dp=P * (gp - (P * gp).sum(2, keepdim=True)))
