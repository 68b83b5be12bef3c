"""K-means with a warp per stream of pairs: sample counts around the ring's 16-sample stages and the
4-sample steps, every cluster range it is compiled for, both rand() forms, more pairs than a warp keeps
open, very uneven usable counts, and data whose squared distances tie or nearly tie (where the rounded
square roots decide a label).  Results are the oracle's bit for bit (the tolerance of every parity test
here)."""
import numpy as np
import pytest

from kinc_gb300 import Similarity, synthetic
from oracle import pyoracle

pytestmark = pytest.mark.gpu


def _check(gem, gargs, oargs):
    sim = Similarity(gem, clusmethod="kmeans", **gargs)
    sim.initialize()
    total = sim.total_pairs()
    res = sim.execute(None, start=0, size=total)
    sim.close()
    K, labels, corr, _ = pyoracle.run_block(gem, pyoracle.params(clus_method=2, **oargs), 0, total)
    assert np.array_equal(res.K, K), f"K differs on {(res.K != K).sum()} of {total} pairs"
    multi = K > 1
    assert np.array_equal(res.labels[multi], labels[multi])
    assert np.array_equal(np.nan_to_num(res.corr, nan=9.0), np.nan_to_num(corr, nan=9.0))


@pytest.mark.parametrize("samples", [1, 2, 3, 4, 5, 15, 16, 17, 31, 32, 33, 47, 48, 49, 65, 130])
def test_sample_counts_around_stages(samples):
    rng = np.random.default_rng(samples)
    gem = rng.normal(8.0, 2.0, (12, samples)).astype(np.float32)
    _check(gem, dict(crit="BIC", corrmethod="both", preout=True, postout=True, minsamp=1, maxclus=3),
           dict(criterion=0, corr_method=2, pre_out=1, post_out=1, min_samples=1, max_clusters=3))


@pytest.mark.parametrize("minclus,maxclus", [(1, 1), (1, 2), (2, 2), (2, 5), (3, 3), (4, 5), (5, 5)])
@pytest.mark.parametrize("rand", ["glibc", "lcg"])
def test_cluster_ranges(minclus, maxclus, rand):
    gem = synthetic.generate(4, genes=16, samples=90)
    _check(gem, dict(crit="ICL", minclus=minclus, maxclus=maxclus, corrmethod="pearson", rand=rand),
           dict(criterion=1, min_clusters=minclus, max_clusters=maxclus, corr_method=0, rand_mode=int(rand == "lcg")))


def test_uneven_counts_and_many_pairs():
    rng = np.random.default_rng(3)
    gem = rng.normal(8.0, 2.0, (120, 70)).astype(np.float32)
    gem[rng.random(gem.shape) < rng.uniform(0.0, 0.9, (120, 1))] = np.nan
    _check(gem, dict(crit="BIC", corrmethod="spearman", minsamp=10, maxclus=3),
           dict(criterion=0, corr_method=1, min_samples=10, max_clusters=3))


@pytest.mark.parametrize("step,base", [(1.0, 8.0), (2.0 ** -11, 4096.0), (2.0 ** -20, 8.0), (2.0 ** -75, 0.0)])
def test_ties_and_near_ties(step, base):
    """Values on a grid of a few float spacings: many squared distances are equal or neighbours."""
    rng = np.random.default_rng(17)
    gem = (base + step * rng.integers(-12, 13, (24, 75))).astype(np.float32)
    _check(gem, dict(crit="BIC", maxclus=5), dict(criterion=0, max_clusters=5))


def test_infinite_and_constant_genes():
    gem = synthetic.generate(4, genes=14, samples=80)
    gem[1] = 3.0
    gem[2, 5] = np.inf
    gem[3, 6] = -np.inf
    gem[4] *= np.float32(1e25)
    gem[5] *= np.float32(1e-25)
    _check(gem, dict(crit="ICL", corrmethod="spearman", postout=True, maxclus=4),
           dict(criterion=1, corr_method=1, post_out=1, max_clusters=4))


def test_scratch_is_what_the_kernel_uses():
    """A warp slot holds eight open pairs (samples, labels, draws, records of the runs) and the distances and labels of
    32 runs, not 32 pairs: the worker takes that and no more (64 MB for everything else)."""
    import torch
    S, runs, draws, record = 4000, 30, 60, 4 * 3 + 1
    gem = synthetic.generate(4, genes=40, samples=S)

    def taken(matrix):
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        sim = Similarity(matrix, clusmethod="kmeans", corrmethod="pearson", maxclus=3, crit="BIC")
        sim.execute(None, start=0, size=100)
        after = torch.cuda.mem_get_info()[0]
        sim.close()
        return before - after

    taken(gem[:, :50])                                     # modules and runtime buffers
    slots = torch.cuda.get_device_properties(0).multi_processor_count * 16
    slot = 8 * (S * (8 + 1) + 4 * draws + 4 * record * runs) + 32 * S * (4 + 1)
    assert taken(gem) <= slots * (slot + 4096) + (64 << 20)
