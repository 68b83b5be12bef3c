"""GMM with one warp per pair: sample counts around the kernel's 64-sample chunks and 16-sample tails,
responsibilities in shared memory (few samples) and in global memory (many), every cluster range it is
compiled for, both criteria, correlations and packed-array semantics, the OpenCL worker's form, and
values outside its fast path (infinities, magnitudes past 1e8, constant genes).  Results are the
oracle's bit for bit (the tolerance of every parity test here)."""
import numpy as np
import pytest

from kinc_gb300 import Similarity, synthetic
from oracle import pyoracle

pytestmark = pytest.mark.gpu


def _check(gem, gargs, oargs):
    sim = Similarity(gem, clusmethod="gmm", **gargs)
    sim.initialize()
    total = sim.total_pairs()
    res = sim.execute(None, start=0, size=total)
    sim.close()
    K, labels, corr, _ = pyoracle.run_block(gem, pyoracle.params(clus_method=1, **oargs), 0, total)
    assert np.array_equal(res.K, K), f"K differs on {(res.K != K).sum()} of {total} pairs"
    multi = K > 1
    assert np.array_equal(res.labels[multi], labels[multi])
    assert np.array_equal(np.nan_to_num(res.corr, nan=9.0), np.nan_to_num(corr, nan=9.0))


def _complete(genes, samples, seed=11):
    """No missing values, so every pair has exactly `samples` usable ones; two planted clusters."""
    rng = np.random.default_rng(seed)
    side = rng.integers(0, 2, samples)
    gem = rng.normal(8.0, 1.0, (genes, samples)) + side * rng.uniform(2.0, 6.0, (genes, 1))
    return gem.astype(np.float32)


@pytest.mark.parametrize("samples", [1, 2, 15, 16, 17, 31, 33, 63, 64, 65, 80, 95, 96, 97, 127, 128, 129, 193])
def test_sample_counts_around_chunks(samples):
    _check(_complete(9, samples), dict(crit="ICL", corrmethod="both", preout=True, postout=True, minsamp=1),
           dict(criterion=1, corr_method=2, pre_out=1, post_out=1, min_samples=1))


@pytest.mark.parametrize("samples", [575, 640, 1030, 2050])
def test_responsibilities_in_global_memory(samples):
    _check(_complete(4, samples), dict(crit="BIC", corrmethod="spearman", postout=True, maxclus=4),
           dict(criterion=0, corr_method=1, post_out=1, max_clusters=4))


@pytest.mark.parametrize("minclus,maxclus", [(1, 1), (1, 2), (2, 2), (3, 5), (4, 4), (5, 5)])
@pytest.mark.parametrize("rand", ["glibc", "lcg"])
def test_cluster_ranges(minclus, maxclus, rand):
    gem = synthetic.generate(5, genes=10, samples=100)
    mode = dict(semantics="fixed", rand=rand) if rand == "lcg" else dict()
    omode = dict(semantics=1, rand_mode=1) if rand == "lcg" else dict()
    _check(gem, dict(crit="BIC", minclus=minclus, maxclus=maxclus, corrmethod="pearson", **mode),
           dict(criterion=0, min_clusters=minclus, max_clusters=maxclus, corr_method=0, **omode))


def test_values_outside_the_fast_path():
    gem = synthetic.generate(2, genes=12, samples=90)
    gem[1] *= np.float32(1e9)
    gem[2] *= np.float32(1e30)
    gem[3] *= np.float32(1e-30)
    gem[4, :7] = np.inf
    gem[5, 3] = -np.inf
    gem[6, :] = 4.0
    gem[7, ::2] = 1e8
    gem[8] = gem[9]
    _check(gem, dict(crit="ICL", corrmethod="pearson"), dict(criterion=1, corr_method=0))


def test_more_pairs_than_the_chip_holds_at_once():
    gem = synthetic.generate(2, genes=90, samples=40)
    _check(gem, dict(crit="BIC", corrmethod="spearman", preout=True, postout=True, maxclus=3),
           dict(criterion=0, corr_method=1, pre_out=1, post_out=1, max_clusters=3))


def test_block_that_fills_the_tile_kernel_s_wave():
    """Enough pairs and samples that the tile kernel is taken for the whole block and this one for a part of
    it: both give the same bits."""
    gem = synthetic.generate(2, genes=480, samples=2600)
    gem[:, 400:] = np.nan                      # few usable samples in all genes but two keep the run short
    gem[:2] = synthetic.generate(2, genes=2, samples=2600, seed=5)
    sim = Similarity(gem, clusmethod="gmm", corrmethod="spearman", crit="BIC", maxclus=2)
    sim.initialize()
    total = min(sim.total_pairs(), 97280)
    whole = sim.execute(None, start=0, size=total)
    part = sim.execute(None, start=0, size=5000)
    sim.close()
    assert np.array_equal(whole.K[:5000], part.K)
    multi = part.K > 1
    assert np.array_equal(whole.labels[:5000][multi], part.labels[multi])
    assert np.array_equal(np.nan_to_num(whole.corr[:5000], nan=9.0), np.nan_to_num(part.corr, nan=9.0))


def _slices(gem, gargs, oargs, start, size, slices):
    """The block on the GPU; the oracle on parts of it.  Returns the kernel that ran and the result."""
    sim = Similarity(gem, clusmethod="gmm", **gargs)
    res = sim.execute(None, start=start, size=size)
    kernel = sim.last_kernel()
    sim.close()
    for at, n in slices:
        K, labels, corr, _ = pyoracle.run_block(gem, pyoracle.params(clus_method=1, **oargs), start + at, n)
        got = slice(at, at + n)
        assert np.array_equal(res.K[got], K)
        assert np.array_equal(res.labels[got][K > 1], labels[K > 1])
        assert np.array_equal(res.corr[got], corr, equal_nan=True)
    return kernel, res


@pytest.mark.parametrize("samples,gargs,oargs", [
    (36, dict(maxclus=1, corrmethod="pearson", crit="BIC"), dict(max_clusters=1, corr_method=0, criterion=0)),
    (50, dict(maxclus=2, corrmethod="spearman", crit="BIC", preout=True),
     dict(max_clusters=2, corr_method=1, criterion=0, pre_out=1)),
    (64, dict(corrmethod="both", crit="ICL", preout=True, postout=True),
     dict(corr_method=2, criterion=1, pre_out=1, post_out=1)),
    (80, dict(minclus=2, maxclus=3, corrmethod="spearman", crit="ICL"),
     dict(min_clusters=2, max_clusters=3, corr_method=1, criterion=1)),
    (60, dict(maxclus=5, corrmethod="pearson", crit="BIC", semantics="fixed", rand="lcg"),
     dict(max_clusters=5, corr_method=0, criterion=0, semantics=1, rand_mode=1)),
])
def test_few_samples_run_full_waves_in_tiles(samples, gargs, oargs):
    """With few samples the tile kernel is the faster one for a full wave (20 warps of 32 pairs on every SM), this one
    for a part of it.  Both give the oracle's bits; the slices lie at a work block's start and at the wave's end."""
    import torch
    wave = torch.cuda.get_device_properties(0).multi_processor_count * 20 * 32
    genes = 600
    assert 32768 + wave <= genes * (genes - 1) // 2
    gem = synthetic.generate(2, genes=genes, samples=samples)
    kernel, whole = _slices(gem, gargs, oargs, 32768, wave, [(0, 200), (wave - 60, 60)])
    assert kernel == "tiles"
    kernel, part = _slices(gem, gargs, oargs, 32768, 3000, [])
    assert kernel == "gmm pairs"
    assert np.array_equal(whole.K[:3000], part.K)
    assert np.array_equal(whole.labels[:3000][part.K > 1], part.labels[part.K > 1])
    assert np.array_equal(whole.corr[:3000], part.corr, equal_nan=True)


@pytest.mark.parametrize("genes,samples,gargs,oargs", [
    # 16 warps a CTA, responsibilities in shared memory
    (72, 150, dict(crit="BIC", corrmethod="spearman", preout=True, postout=True), dict(criterion=0, corr_method=1, pre_out=1, post_out=1)),
    (72, 60, dict(crit="ICL", corrmethod="pearson", minclus=4, maxclus=4), dict(criterion=1, corr_method=0, min_clusters=4, max_clusters=4)),
    (64, 190, dict(crit="ICL", corrmethod="both", minclus=5, maxclus=5), dict(criterion=1, corr_method=2, min_clusters=5, max_clusters=5)),
    # 12 warps, in shared memory; 16 and 12 in global memory
    (64, 300, dict(crit="BIC", corrmethod="pearson", minclus=4, maxclus=5), dict(criterion=0, corr_method=0, min_clusters=4, max_clusters=5)),
    (64, 480, dict(crit="BIC", corrmethod="pearson", minclus=4, maxclus=5), dict(criterion=0, corr_method=0, min_clusters=4, max_clusters=5)),
    (64, 900, dict(crit="ICL", corrmethod="pearson", minclus=5, maxclus=5), dict(criterion=1, corr_method=0, min_clusters=5, max_clusters=5)),
])
def test_more_pairs_than_twelve_an_sm(genes, samples, gargs, oargs):
    """Blocks of more than 12 pairs an SM, where the number of warps is chosen by the samples; the oracle on the first
    and the last pairs."""
    gem = synthetic.generate(2, genes=genes, samples=samples)
    total = genes * (genes - 1) // 2
    import torch
    assert total > 12 * torch.cuda.get_device_properties(0).multi_processor_count
    kernel, _ = _slices(gem, gargs, oargs, 0, total, [(0, 100), (total - 30, 30)])
    assert kernel == "gmm pairs"
