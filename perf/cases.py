"""Cases for timing the framework: what a user of the STRUCTURE sweep has it do.

Every case is one call sequence a program makes with its data in hand: a whole
run of one or many chains on an open context (create, sweep, read the result),
a stream of small runs through the server, or a pass over host data ahead of a
run (VCF ingest, locus filter). Sizes follow vcfpop_gb300/workloads.py (c1 to
c5) with shorter runs, since every sweep of a run does the same work.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from vcfpop_gb300 import _lib as B
from vcfpop_gb300 import structure as S


# ---------------------------------------------------------------------------
# the cases

def listed():
    return [
        # a first look at a small survey without admixture (c1): a few kernels
        # of a few microseconds a sweep, hundreds of sweeps
        dict(name="noadmix_c1", kind="run", N=200, L=2000, pops=3, K=3, nburnin=150, nreps=150),
        # the same kind of survey with admixture and alpha inferred
        dict(name="admix_small", kind="run", N=300, L=3000, pops=4, K=4, admix=1, nburnin=60, nreps=60),
        # the F model (correlated allele frequencies), which users of
        # microsatellite- and SNP-panel-sized data switch on by default
        dict(name="admix_fmodel", kind="run", N=600, L=6000, pops=4, K=4, admix=1, f=1, nburnin=6, nreps=6),
        # c2: a mid-sized SNP panel with admixture
        dict(name="admix_c2", kind="run", N=2000, L=50_000, pops=5, K=5, admix=1, nburnin=11, nreps=10),
        # a larger panel at the upper end of the K range, sizes off the tiles,
        # one alpha per cluster
        dict(name="admix_k11", kind="run", N=4999, L=40_009, pops=8, K=11, admix=1, diffalpha=1, nburnin=5, nreps=6),
        # c4 scaled down: autopolyploids of ploidy 2, 4 and 6 at 20 locations,
        # 2-8 alleles, admixture with the location prior
        dict(name="poly_locprior", kind="poly", N=1500, L=8000, pops=8, K=8, admix=1, locpriori=1, nburnin=11, nreps=10),
        # one no-admixture chain on a large panel with weak signal: sampling
        # locations as prior
        dict(name="noadmix_locprior", kind="run", N=3001, L=30_011, pops=6, K=6, locpriori=1, nburnin=11, nreps=10),
        # one no-admixture chain of c3's size class in the default (plain) form
        dict(name="noadmix_large", kind="run", N=10_000, L=60_000, pops=8, K=10, nburnin=11, nreps=10),
        # the K-sweep a study starts with (K = 1..5, some replicates) on a
        # mid-sized panel, batched on the tensor cores
        dict(name="ksweep_mid", kind="ksweep", N=2003, L=20_011, pops=5, kmax=5, reps=4, nburnin=10, nreps=1),
        # c3: K = 1..10 x 10 replicates on a biobank-sized panel (half its loci)
        dict(name="ksweep_c3", kind="ksweep", N=10_000, L=100_000, pops=8, kmax=10, reps=10, nburnin=10, nreps=1),
        # c5 scaled down: a service's stream of small independent runs
        dict(name="serve_small", kind="serve", runs=12, N=500, L=5000, nburnin=40, nreps=40),
        # the genotypes of a cohort read from VCF text
        dict(name="vcf_ingest", kind="vcf", N=2500, L=8000),
    ]


def draw(rng):
    """One more case of the same ranges."""
    def logu(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["noadmix", "admix", "admix", "fmodel", "poly", "ksweep", "ksweep", "serve", "vcf"])
    pops = rng.randint(2, 8)
    if kind == "noadmix":
        return dict(kind="run", N=logu(150, 10_000), L=logu(1500, 60_000), pops=pops, K=rng.randint(2, 10),
                    locpriori=rng.choice([0, 0, 1]), nburnin=11, nreps=10)
    if kind == "admix":
        return dict(kind="run", N=logu(200, 5000), L=logu(2000, 40_000), pops=pops, K=rng.randint(2, 11), admix=1,
                    diffalpha=rng.choice([0, 1]), nburnin=5, nreps=6)
    if kind == "fmodel":
        return dict(kind="run", N=logu(200, 1000), L=logu(1000, 6000), pops=pops, K=rng.randint(2, 6),
                    admix=rng.choice([0, 1]), f=1, singlef=rng.choice([0, 1]), nburnin=6, nreps=6)
    if kind == "poly":
        return dict(kind="poly", N=logu(200, 1500), L=logu(1000, 8000), pops=pops, K=rng.randint(2, 8),
                    admix=rng.choice([0, 1]), locpriori=rng.choice([0, 1]), nburnin=5, nreps=6)
    if kind == "ksweep":
        return dict(kind="ksweep", N=logu(1000, 8000), L=logu(15_000, 70_000), pops=pops, kmax=rng.randint(3, 10),
                    reps=rng.randint(1, 8), nburnin=10, nreps=1)
    if kind == "serve":
        return dict(kind="serve", runs=rng.randint(4, 12), N=logu(100, 500), L=logu(1000, 5000), nburnin=20,
                    nreps=rng.randint(10, 30))
    return dict(kind="vcf", N=logu(200, 2500), L=logu(1000, 8000))


# ---------------------------------------------------------------------------
# inputs: the F-model the sweep infers, drawn on the GPU from the seed

FST = 0.05
MISSING = 0.02


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 1_000_003 + 17)
    return g


def _gamma(shape, g):
    return torch._standard_gamma(shape, generator=g).clamp_min_(1e-30)


def _dirichlet(shape, g):
    x = _gamma(shape, g)
    return x / x.sum(-1, keepdim=True)


def _ancestry(N, pops, admix, g):
    """[N, pops] ancestry: Dirichlet(0.5) under admixture, else consecutive
    populations of equal size."""
    if admix:
        return _dirichlet(torch.full((N, pops), 0.5, device="cuda"), g)
    pop = torch.arange(N, device="cuda") * pops // N
    return torch.nn.functional.one_hot(pop, pops).float()


def _codes(N, L, pops, admix, seed):
    """Biallelic diploid calls in chunks of loci: copies of allele 1, 3 = missing."""
    g = _gen(seed)
    anc = _dirichlet(torch.full((L, 2), 0.5, device="cuda"), g).clamp_min_(1e-3)
    a = anc * ((1 - FST) / FST)
    f = torch.stack([_dirichlet(a, g)[:, 1] for _ in range(pops)])     # [pops, L]
    Q = _ancestry(N, pops, admix, g)
    step = max(1, (1 << 25) // N)
    for l0 in range(0, L, step):
        p = f[:, l0:l0 + step].t().contiguous() @ Q.t()                 # [chunk, N]
        u = torch.rand((3,) + p.shape, device="cuda", generator=g)
        c = (u[0] < p).to(torch.int32) + (u[1] < p).to(torch.int32)
        c = torch.where(u[2] < MISSING, 3, c)
        # every locus is polymorphic (a panel is chosen so; a monomorphic
        # locus would be dropped from the run): a heterozygote where none is
        het, alt = (c == 1).any(1), (c == 2).any(1) & (c == 0).any(1)
        c[:, 0] = torch.where(het | alt, c[:, 0], 1)
        yield c


def _packed(N, L, pops, admix, seed):
    """[L, ceil(N/16)] uint32 words on the host, as the loader hands them over."""
    Nw = (N + 15) // 16
    shift = 2 * torch.arange(16, device="cuda", dtype=torch.int64)
    out = []
    for c in _codes(N, L, pops, admix, seed):
        c = torch.nn.functional.pad(c, (0, Nw * 16 - N), value=3).view(-1, Nw, 16)
        out.append((c.to(torch.int64) << shift).sum(-1).cpu().numpy().astype(np.uint32))
    return np.concatenate(out)


def _dataset(N, L, pops, admix, seed, n_pop=1):
    popid = (np.arange(N) * n_pop // N).astype(np.int32)
    return S.Dataset(np.full(N, 2, np.int32), np.full(L, 2, np.int32), popid, n_pop,
                     packed2=_packed(N, L, pops, admix, seed))


def _poly_dataset(N, L, pops, admix, seed, n_pop):
    """Ploidy 2, 2, 4, 6 in turn, 2-8 alleles a locus, calls in ascending order."""
    g = _gen(seed)
    ploidy = torch.tensor([2, 2, 4, 6], device="cuda").repeat((N + 3) // 4)[:N]
    k = (2 + torch.arange(L, device="cuda") % 7)[torch.randperm(L, device="cuda", generator=g)]
    live = torch.arange(8, device="cuda")[None, :] < k[:, None]
    anc = _dirichlet(torch.ones((L, 8), device="cuda"), g) * live
    anc = anc / anc.sum(-1, keepdim=True)
    a = (anc * ((1 - FST) / FST)).clamp_min_(1e-3)
    f = torch.stack([_dirichlet(a, g) * live for _ in range(pops)])     # [pops, L, 8]
    Q = _ancestry(N, pops, admix, g)
    G = torch.empty((L, N, 6), dtype=torch.int8, device="cuda")
    step = max(1, (1 << 22) // N)
    slot = torch.arange(6, device="cuda")
    for l0 in range(0, L, step):
        p = torch.einsum("ip,pla->lia", Q, f[:, l0:l0 + step])          # [chunk, N, 8]
        cum = torch.cumsum(p, -1)
        u = torch.rand(cum.shape[:2] + (6,), device="cuda", generator=g) * cum[..., -1:]
        al = torch.zeros(u.shape, dtype=torch.int8, device="cuda")
        for j in range(7):
            al += u > cum[..., j:j + 1]
        al = torch.minimum(al, (k[l0:l0 + step, None, None] - 1).to(torch.int8))
        al = torch.where(slot < ploidy[None, :, None], al, 127).sort(-1).values
        miss = torch.rand(cum.shape[:2], device="cuda", generator=g) < MISSING
        al = torch.where((al == 127) | miss[..., None], -1, al)
        # the same guarantee: the first (diploid) sample is 0/1 at such a locus
        mono = torch.where(al < 0, 127, al).amin((1, 2)) == al.amax((1, 2))
        al[:, 0, 0] = torch.where(mono, 0, al[:, 0, 0])
        al[:, 0, 1] = torch.where(mono, 1, al[:, 0, 1])
        G[l0:l0 + step] = al
    popid = (np.arange(N) * n_pop // N).astype(np.int32)
    return S.Dataset(ploidy.cpu().numpy().astype(np.int32), k.cpu().numpy().astype(np.int32), popid, n_pop,
                     G=G.cpu().numpy())


def _vcf_text(N, L, seed):
    """The data lines of a VCF: nine fixed fields, then a GT call a sample."""
    call = np.array([b"0/0\t", b"0/1\t", b"1/1\t", b"./.\t"], "S4").view(np.uint8).reshape(4, 4)
    rows, l = [], 0
    for c in _codes(N, L, 4, 0, seed):
        cells = torch.from_numpy(call).cuda()[c.long()].view(c.shape[0], -1).cpu().numpy().copy()
        cells[:, -1] = ord("\n")
        head = np.array(["1\t%08d\t.\tA\tC\t.\tPASS\t.\tGT\t" % (l + j + 1) for j in range(len(cells))], "S")
        rows.append(np.concatenate([head.view(np.uint8).reshape(len(cells), -1), cells], 1).reshape(-1))
        l += len(cells)
    return np.concatenate(rows).tobytes()


# ---------------------------------------------------------------------------
# what a program has in hand, and one pass

_OPTIONS = ("admix", "locpriori", "f", "singlef", "diffalpha")


def _params(case, K, seed, **more):
    opt = {k: case[k] for k in _OPTIONS if k in case}
    return S.params(K, seed, nadmburnin=0, writelnl=1, nburnin=case["nburnin"], nreps=case["nreps"],
                    **{"admix": 0, **opt, **more})


def prepare(case, seed):
    kind = case["kind"]
    seed = int(seed)
    if kind == "vcf":
        return dict(kind=kind, text=_vcf_text(case["N"], case["L"], seed), N=case["N"])
    if kind == "serve":
        r = np.random.default_rng(seed)
        runs = []
        for j in range(case["runs"]):
            # runs of a few shapes, with and without admixture, as requests come
            N, L, K = case["N"] * (4 + j % 3) // 6, case["L"] * (3 + j % 4) // 6, 2 + j % 4
            ds = _dataset(N, L, 3, j % 2, int(r.integers(1 << 30)))
            runs.append((ds, _params(case, K, S.run_seed(seed, j + 1), admix=j % 2)))
        return dict(kind=kind, server=S.Server(), runs=runs)
    n_pop = max(2, min(20, case["N"] // 50)) if case.get("locpriori") else 1
    make = _poly_dataset if kind == "poly" else _dataset
    ds = make(case["N"], case["L"], case["pops"], case.get("admix", 0), seed, n_pop)
    ctx = S.Context(ds)
    if kind == "ksweep":
        ps = [_params(case, K, S.run_seed(seed, case["reps"] * K + j), form=B.VP_FORM_TC)
              for K in range(1, case["kmax"] + 1) for j in range(case["reps"])]
    else:
        ps = [_params(case, case["K"], S.run_seed(seed, 1))]
    ctx.sync()
    return dict(kind=kind, ds=ds, ctx=ctx, params=ps)


def run(state):
    kind = state["kind"]
    if kind == "vcf":
        packed, starts = S.vcf_pack2(state["text"], state["N"])
        return dict(packed=packed, starts=starts)
    if kind == "serve":
        sv = state["server"]
        ids = [sv.submit(ds, p) for ds, p in state["runs"]]
        out = []
        for rid in ids:
            info = sv.wait(rid)
            if info["state"] != "done":
                raise RuntimeError(info["error"])
            r = sv.result(rid)
            out.append([r["rout"], r["lnl"], r["Q"], r["ancestry"], r["freqm"]])
            sv.release(rid)
        return out
    chains = [S.Chain(state["ctx"], p) for p in state["params"]]
    S.finish(chains)
    if kind == "ksweep":
        # the labels (as one-hot Q) and lnP(D) of every chain, by which a study
        # picks K, and the state of the last chain
        out = dict(Q=np.concatenate([c.get("Q") for c in chains]), lnl=np.concatenate([c.get("LNL") for c in chains]),
                   freq=chains[-1].get("FREQ"), counts=chains[-1].get("NI"))
    else:
        c = chains[0]
        r = c.result(final=True)
        out = {k: r[k] for k in ("rout", "lnl", "Q", "ancestry", "freqm")}
        out.update(counts=c.get("NI"), copies=c.get("MI"))
    for c in chains:
        c.close()
    return out


def work(case):
    """One pass: each sweep reads the genotypes and the counts once and writes
    the frequencies and the counts once, and its arithmetic is a
    multiply-add per (copy, cluster) for the cluster weights (per call and
    cluster, two alleles, without admixture) and, for a K-sweep, the same
    again for the counts."""
    kind = case["kind"]
    if kind == "vcf":
        text = case["L"] * (4 * case["N"] + 29)
        return dict(bytes=text + case["L"] * (-(-case["N"] // 16) * 4 + 8), flops=0)
    sweeps = case["nburnin"] + case["nreps"]
    if kind == "serve":
        b = f = 0
        for j in range(case["runs"]):
            N, L, K = case["N"] * (4 + j % 3) // 6, case["L"] * (3 + j % 4) // 6, 2 + j % 4
            b += sweeps * (N * L / 4 + 3 * 4 * K * 2 * L + 8 * N * K)
            f += sweeps * 4.0 * N * L * K
        return dict(bytes=b, flops=f)
    N, L = case["N"], case["L"]
    if kind == "ksweep":
        R = case["reps"] * case["kmax"] * (case["kmax"] + 1) // 2
        return dict(bytes=sweeps * (N * L / 4 + 3 * 4 * R * 2 * L + 8 * N * R), flops=sweeps * 8.0 * N * L * R)
    K = case["K"]
    copies, KT, geno = (3.5, 5 * L, N * L * 6) if kind == "poly" else (2, 2 * L, N * L / 4)
    return dict(bytes=sweeps * (geno + 3 * 4 * K * KT + 8 * N * K), flops=sweeps * 2.0 * copies * N * L * K)


def exact(case, seed):
    """The 2-bit words and line offsets are whole numbers, and a run's outputs
    depend on its random draws: there is no value in 64 bits to give."""
    return None
