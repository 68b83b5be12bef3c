"""The work users of this framework have it do, as cases that can be timed and compared.

A case is one call of a public entry point on a seeded expression matrix of the synthetic workloads
(kinc_gb300/synthetic.py): a block of gene pairs through the worker (`call` "device": device outputs,
kinc_sim_execute_block_device; "host": Similarity.execute, one work block into host arrays), a whole
run into CCM/CMX files ("files": Similarity.run), or the eigenvalues of a pruned correlation matrix
(RMT.prune_eigenvalues).  Workers are created once per matrix, as a program that runs many blocks
does; blocks start at a work-block boundary in the middle of the pair order where there is room.
"""
import ctypes
import math
import os
import tempfile

import numpy as np
import torch

from kinc_gb300 import Similarity, _native, rmt, synthetic

WORK_BLOCK = Similarity.WORK_BLOCK_SIZE


def _case(name, call, workload, genes, samples, size, clus, corr, crit="BIC", maxclus=5, preout=False, postout=False,
          semantics="reference", precision="fp32"):
    c = dict(call=call, workload=workload, genes=genes, samples=samples, size=size, clus=clus, corr=corr, crit=crit,
             maxclus=maxclus, preout=preout, postout=postout, semantics=semantics, precision=precision)
    if name:
        c["name"] = name
    return c


def _pairs(genes):
    return genes * (genes - 1) // 2


def listed():
    return [
        # the smallest run anyone makes: a few dozen genes, to see that it works; latency is all
        _case("gmm_smallest", "host", 2, 48, 96, _pairs(48), "gmm", "spearman", "BIC", 5, True, True),
        # one 32,768-pair work block into host arrays: what the worker is asked for by KINC's block loop
        _case("gmm_work_block", "host", 2, 2500, 1000, WORK_BLOCK, "gmm", "spearman", "BIC", 5, True, True),
        # a device block of the headline workload (GMM k <= 5 + Spearman, 1,000 samples)
        _case("gmm_device_block", "device", 2, 2500, 1000, 4 * WORK_BLOCK, "gmm", "spearman", "BIC", 5, True, True),
        # a device block of the many-genes workload: 500 samples, ICL, both correlations, the default criterion
        _case("gmm_icl_both_block", "device", 5, 3500, 500, 6 * WORK_BLOCK, "gmm", "both", "ICL", 5, True, True),
        # K-means on very uneven sample counts (0-60 % missing per gene), 4,000 samples
        _case("kmeans_uneven_block", "device", 4, 800, 4000, 2 * WORK_BLOCK, "kmeans", "pearson", "BIC", 3),
        # K-means on a small odd-sized matrix, all pairs, up to five clusters
        _case("kmeans_small", "device", 4, 211, 333, _pairs(211), "kmeans", "spearman", "ICL", 5, True, False),
        # KINC's default analytic arguments on a small matrix: Pearson of all pairs, no clustering
        _case("pearson_all_pairs", "device", 1, 1000, 200, _pairs(1000), "none", "pearson"),
        # the same with every sample's own values, at odd sizes
        _case("pearson_fixed_odd", "device", 1, 1237, 611, _pairs(1237), "none", "pearson", semantics="fixed"),
        # Spearman without clustering
        _case("spearman_block", "device", 2, 2500, 1000, 8 * WORK_BLOCK, "none", "spearman"),
        # pairwise-complete Pearson of all pairs on the tensor cores
        _case("pearson_fp16_dense", "device", 3, 6000, 2000, _pairs(6000), "none", "pearson", maxclus=1,
              semantics="fixed", precision="fp16"),
        # a whole run into CCM and CMX files, read back as the next analytic does
        _case("run_to_files", "files", 2, 320, 150, _pairs(320), "gmm", "spearman", "ICL", 5, True, True),
        # RMT thresholding's step: a 1,000-row pruned matrix' eigenvalues
        dict(name="rmt_eigenvalues", call="rmt", blocks=100, block_genes=10, threshold=0.6),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(["gmm", "gmm", "gmm", "kmeans", "kmeans", "pearson", "spearman", "dense", "files", "rmt"])
    if family == "rmt":
        return dict(call="rmt", blocks=_log_int(rng, 12, 140), block_genes=rng.randint(5, 10), threshold=0.6)
    if family == "files":
        genes = _log_int(rng, 60, 380)
        return _case(None, "files", 2, genes, _log_int(rng, 60, 200), _pairs(genes), rng.choice(["gmm", "kmeans"]),
                     rng.choice(["pearson", "spearman"]), rng.choice(["BIC", "ICL"]), rng.randint(3, 5),
                     rng.random() < 0.5, rng.random() < 0.5)
    if family == "pearson":
        genes = _log_int(rng, 60, 1300)
        return _case(None, "device", 1, genes, _log_int(rng, 40, 620), _pairs(genes), "none", "pearson",
                     semantics=rng.choice(["reference", "fixed"]))
    if family == "dense":
        genes = _log_int(rng, 300, 6000)
        return _case(None, "device", 3, genes, _log_int(rng, 64, 2000), _pairs(genes), "none", "pearson", maxclus=1,
                     semantics="fixed", precision=rng.choice(["fp16", "fp16", "tf32", "3xbf16"]))
    if family == "spearman":
        genes = _log_int(rng, 60, 2500)
        return _case(None, "device", 2, genes, _log_int(rng, 40, 1200), min(_pairs(genes), 8 * WORK_BLOCK), "none",
                     "spearman")
    # clustering: any size from a few dozen genes to the device blocks above, at the same cost at most
    workload, top = (4, 4000) if family == "kmeans" else (rng.choice([2, 5]), 1000)
    genes, samples = _log_int(rng, 40, 2500), _log_int(rng, 60, top)
    most = (2 * WORK_BLOCK * 4000 if family == "kmeans" else 3 * WORK_BLOCK * 1000) // samples
    size = min(_pairs(genes), most, _log_int(rng, 700, 8 * WORK_BLOCK))
    call = "host" if size <= WORK_BLOCK and rng.random() < 0.5 else "device"
    return _case(None, call, workload, genes, samples, size, family, rng.choice(["pearson", "spearman", "both"]),
                 rng.choice(["BIC", "ICL"]), rng.randint(3, 5) if family == "gmm" else 3, rng.random() < 0.5,
                 rng.random() < 0.5)


_STREAM = None


def _stream():
    """The program's one stream (the worker reads stream 0 as its own)."""
    global _STREAM
    if _STREAM is None:
        _STREAM = torch.cuda.Stream()
    return _STREAM


def _matrix(case, seed):
    return synthetic.generate(case["workload"], genes=case["genes"], samples=case["samples"], seed=seed)


def _start(case):
    """The first pair: the middle work block if the block fits behind it."""
    total = _pairs(case["genes"])
    mid = (total // 2) // WORK_BLOCK * WORK_BLOCK
    return mid if mid + case["size"] <= total else 0


def _network(case, seed):
    return synthetic.clique_network(case["blocks"], case["block_genes"], seed=seed)


def prepare(case, seed):
    if case["call"] == "rmt":
        genes, x, y, c, r = _network(case, seed)
        return dict(call="rmt", rmt=rmt.RMT(), items=(x, y, c, r), genes=genes, threshold=case["threshold"])
    sim = Similarity(_matrix(case, seed), clusmethod=case["clus"], corrmethod=case["corr"], crit=case["crit"],
                     maxclus=case["maxclus"], preout=case["preout"], postout=case["postout"],
                     semantics=case["semantics"], precision=case["precision"])
    sim.initialize()
    state = dict(call=case["call"], sim=sim, start=_start(case), size=case["size"])
    if case["call"] == "files":
        folder = tempfile.TemporaryDirectory()
        # a reader's buffers: room for every cluster of every pair
        items = case["size"] * case["maxclus"]
        state.update(folder=folder, ccm=os.path.join(folder.name, "ccm"), cmx=os.path.join(folder.name, "cmx"),
                     ccm_bytes=np.zeros(64 + items * (16 + (case["samples"] + 1) // 2), np.uint8),
                     cmx_bytes=np.zeros(64 + items * 20, np.uint8))
    elif case["call"] == "device":
        n = case["size"]
        both = (2,) if case["corr"] == "both" else ()
        out = dict(K=torch.zeros(n, dtype=torch.int8, device="cuda"),
                   corr=torch.zeros((n, case["maxclus"]) + both, dtype=torch.float32, device="cuda"))
        if case["clus"] != "none":
            out["labels"] = torch.zeros((n, case["samples"]), dtype=torch.int8, device="cuda")
        state["out"] = out
    return state


def run(state):
    if state["call"] == "rmt":
        return {"eigenvalues": state["rmt"].prune_eigenvalues(state["items"], state["genes"], 1, state["threshold"])}
    sim = state["sim"]
    if state["call"] == "host":
        res = sim.execute(None, start=state["start"], size=state["size"])
        return {"K": res.K, "labels": res.labels, "corr": res.corr}
    if state["call"] == "files":
        sim.run(state["ccm"], state["cmx"])
        sizes = []
        for name in ("ccm", "cmx"):
            with open(state[name], "rb") as f:
                sizes.append(f.readinto(state[name + "_bytes"]))
        return {"sizes": np.array(sizes), "ccm": state["ccm_bytes"], "cmx": state["cmx_bytes"]}
    out = state["out"]
    vp = ctypes.c_void_p
    labels = vp(out["labels"].data_ptr()) if "labels" in out else None
    _native.check(_native.load().kinc_sim_execute_block_device(sim._ctx, state["start"], state["size"],
                                                               vp(out["K"].data_ptr()), labels,
                                                               vp(out["corr"].data_ptr()),
                                                               vp(_stream().cuda_stream)), sim._ctx)
    return out


#: usable share of a gene's samples, on average, in each synthetic workload
_USABLE = {1: 0.95, 2: 0.90, 3: 0.90, 4: 0.70, 5: 0.92}
#: floating-point operations per (sample, component, EM iteration) and per (sample, cluster, Lloyd iteration)
_EM_FLOPS, _LLOYD_FLOPS = 60, 9
#: EM iterations per fit and Lloyd iterations per K-means run, on average
_EM_ITERATIONS, _LLOYD_ITERATIONS = 85, 20


def work(case):
    """The matrix read once and the results written once; the operations of the method."""
    if case["call"] == "rmt":
        m = case["blocks"] * case["block_genes"]
        items = case["blocks"] * case["block_genes"] * (case["block_genes"] - 1) // 2
        return {"bytes": 13 * items + 4 * m, "flops": 4 / 3 * m ** 3}
    n, S, k = case["size"], case["samples"], case["maxclus"]
    usable = S * _USABLE[case["workload"]] ** 2
    per_pair = 1 + 4 * k * (2 if case["corr"] == "both" else 1) + (S if case["clus"] != "none" else 0)
    if case["call"] == "files":
        per_pair = S // 8
    flops = {"pearson": 8 * usable, "spearman": 6 * usable, "both": 14 * usable}[case["corr"]]
    if case["precision"] != "fp32":
        flops = 12 * S
    if case["clus"] == "gmm":
        flops += _EM_FLOPS * _EM_ITERATIONS * usable * k * (k + 1) / 2
    elif case["clus"] == "kmeans":
        # ten runs per cluster count; one cluster takes one sweep
        flops += _LLOYD_FLOPS * 10 * usable * (1 + _LLOYD_ITERATIONS * (k * (k + 1) / 2 - 1))
    return {"bytes": 4 * case["genes"] * S + n * per_pair, "flops": n * flops}


def _xy(start, size, device):
    """Linear pair index -> (x, y), x > y."""
    p = torch.arange(start, start + size, dtype=torch.int64, device=device)
    x = ((1 + torch.sqrt(1 + 8 * p.double())) / 2).long()
    x = torch.where(x * (x - 1) // 2 > p, x - 1, x)
    x = torch.where((x + 1) * x // 2 <= p, x + 1, x)
    return x, p - x * (x - 1) // 2


def _correlation(n, sx, sy, sxx, syy, sxy, minsamp=30):
    r = (n * sxy - sx * sy) / torch.sqrt((n * sxx - sx * sx) * (n * syy - sy * sy))
    return torch.where(n >= minsamp, r, torch.full_like(r, math.nan))


def _pearson_reference(gem, start, size):
    """KINC's Pearson: a pair's usable values packed to the front of an array that the pairs of a work
    block share in order, read back at the usable sample positions."""
    out = []
    S = gem.shape[1]
    pos = torch.arange(S, device=gem.device)
    end = start + size
    for b in range(start // WORK_BLOCK * WORK_BLOCK, end, WORK_BLOCK):
        count = min(WORK_BLOCK, end - b)
        x, y = _xy(b, count, gem.device)
        vx, vy = gem[x], gem[y]
        use = ~(vx.isnan() | vy.isnan())
        N = use.sum(1)
        order = torch.argsort((~use).to(torch.int8), dim=1, stable=True)
        rows = torch.arange(count, device=gem.device)
        last = torch.cummax(torch.where(pos < N[:, None], rows[:, None], -1), dim=0).values
        sums = [0.0] * 5
        for i in range(S):
            q = last[:, i].clamp(min=0)
            have = use[:, i] & (last[:, i] >= 0)
            s = order[q, i]
            a = torch.where(have, vx[q, s], 0.0)
            c = torch.where(have, vy[q, s], 0.0)
            for k, t in enumerate((a, c, a * a, c * c, a * c)):
                sums[k] = sums[k] + t
        r = _correlation(N.double(), *sums)
        out.append(r[max(0, start - b):])
    return torch.cat(out)


def _pearson_complete(gem, start, size):
    """Pearson over the samples both genes have, centred per gene first, all pairs by matrix products."""
    m = (~gem.isnan()).double()
    a = torch.nan_to_num(gem - torch.nanmean(gem, dim=1, keepdim=True))
    x, y = _xy(start, size, gem.device)
    flat = x * gem.shape[0] + y

    def pairs(u, v):
        return (u @ v.T).reshape(-1)[flat]

    return _correlation(pairs(m, m), pairs(a, m), pairs(m, a), pairs(a * a, m), pairs(m, a * a), pairs(a, a))


def _spearman(gem, start, size):
    out = []
    S = gem.shape[1]
    ranks = torch.arange(S, dtype=torch.float64, device=gem.device)
    for b in range(start, start + size, 16384):
        x, y = _xy(b, min(16384, start + size - b), gem.device)
        use = ~(gem[x].isnan() | gem[y].isnan())
        n = use.sum(1).double()
        rk = []
        for g in (x, y):
            order = torch.argsort(torch.where(use, gem[g], math.inf), dim=1, stable=True)
            rk.append(torch.empty(order.shape, dtype=torch.float64, device=gem.device).scatter_(
                1, order, ranks.expand_as(order)))
        d2 = torch.where(use, (rk[0] - rk[1]) ** 2, 0.0).sum(1)
        r = 1 - 6 * d2 / (n * (n * n - 1))
        out.append(torch.where(n >= 30, r, torch.full_like(r, math.nan)))
    return torch.cat(out)


def exact(case, seed):
    """The correlations without clustering, and the eigenvalues, in 64 bits.  Cluster labels (and what is
    correlated under them) follow single-precision trajectories from a rand() stream: no such value."""
    if case["call"] == "rmt":
        genes, x, y, _, r = _network(case, seed)
        A = np.eye(genes)
        keep = np.abs(r) >= np.float32(case["threshold"])
        A[x[keep], y[keep]] = r[keep]
        A[y[keep], x[keep]] = r[keep]
        rows = np.unique(np.concatenate([x[keep], y[keep]]))
        w = np.linalg.eigvalsh(A[np.ix_(rows, rows)])
        return {"eigenvalues": w[np.argsort(np.abs(w), kind="stable")]}
    if case["clus"] != "none" or case["corr"] == "both" or case["samples"] > 1290 and case["corr"] == "spearman":
        return None
    gem = torch.from_numpy(_matrix(case, seed)).cuda().double()
    fn = {"spearman": _spearman, "pearson": _pearson_reference if case["semantics"] == "reference"
          else _pearson_complete}[case["corr"]]
    r = fn(gem, _start(case), case["size"])
    corr = torch.full((case["size"], case["maxclus"]), math.nan, dtype=torch.float64, device=gem.device)
    corr[:, 0] = r
    return {"K": None, "corr": corr}
