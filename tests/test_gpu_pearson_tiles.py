"""Pearson without clustering on tiles of genes: sample counts around the 32-sample words, gene counts around
the tiles' edges, blocks of one, two, a few and many rows x (each takes another tile shape), blocks that begin
and end inside a row and across work blocks, sparse and complete matrices, infinities, and more samples than
the tiles take.  Correlations are the oracle's bit for bit (the tolerance of every parity test here)."""
import numpy as np
import pytest

from kinc_gb300 import Similarity
from oracle import pyoracle

pytestmark = pytest.mark.gpu


def _matrix(genes, samples, seed, missing=0.1):
    rng = np.random.default_rng(seed)
    gem = (rng.uniform(4, 12, (genes, 1)) + 2.0 * rng.standard_normal((genes, samples))).astype(np.float32)
    gem[rng.random(gem.shape) < missing * rng.uniform(0, 2, (genes, 1))] = np.nan
    return gem


def _check(gem, semantics, blocks=None, minsamp=2):
    sim = Similarity(gem, semantics=semantics, minsamp=minsamp)
    sim.initialize()
    for start, size in blocks or [(0, sim.total_pairs())]:
        res = sim.execute(None, start=start, size=size)
        K, _, corr, _ = pyoracle.run_block(gem, pyoracle.params(semantics=int(semantics == "fixed"), min_samples=minsamp),
                                           start, size)
        assert np.array_equal(res.K, K)
        assert np.array_equal(np.nan_to_num(res.corr, nan=9.0), np.nan_to_num(corr, nan=9.0))
    sim.close()


@pytest.mark.parametrize("semantics", ["reference", "fixed"])
@pytest.mark.parametrize("samples", [2, 31, 32, 33, 63, 64, 65, 100, 160, 161])
def test_sample_counts(samples, semantics):
    _check(_matrix(40, samples, samples), semantics)


@pytest.mark.parametrize("semantics", ["reference", "fixed"])
@pytest.mark.parametrize("genes", [2, 3, 15, 16, 17, 18, 33, 34, 65, 130, 300])
def test_gene_counts(genes, semantics):
    _check(_matrix(genes, 50, genes), semantics)


@pytest.mark.parametrize("semantics", ["reference", "fixed"])
@pytest.mark.parametrize("missing", [0.0, 0.03, 0.3, 0.48])
def test_missing_rates(missing, semantics):
    _check(_matrix(60, 130, 7, missing), semantics)


@pytest.mark.parametrize("semantics", ["reference", "fixed"])
def test_blocks_of_few_and_many_rows(semantics):
    gem = _matrix(600, 45, 9)
    row = lambda x: x * (x - 1) // 2  # noqa: E731
    _check(gem, semantics, [(row(500) + 17, 1), (row(500), 500), (row(500) + 100, 450), (row(400) + 399, 2),
                            (row(300) + 5, 1200), (row(590), 590 * 8), (32768, 32768), (30000, 40000)])


@pytest.mark.parametrize("semantics", ["reference", "fixed"])
def test_infinities(semantics):
    gem = _matrix(40, 70, 3)
    gem[3, 5], gem[7, 60], gem[9] = np.inf, -np.inf, gem[9] * np.float32(1e30)
    _check(gem, semantics)


@pytest.mark.parametrize("semantics", ["reference", "fixed"])
def test_more_samples_than_the_tiles_take(semantics):
    _check(_matrix(12, 4100, 2), semantics)
    _check(_matrix(12, 4096, 2), semantics)


def _sparse(genes, samples, share, seed=5):
    rng = np.random.default_rng(seed)
    gem = rng.normal(8.0, 2.0, (genes, samples)).astype(np.float32)
    gem[rng.random(gem.shape) >= share] = np.nan
    return gem


@pytest.mark.parametrize("semantics", ["reference", "fixed"])
@pytest.mark.parametrize("gem,size", [
    (_matrix(520, 40, 21), 130000),                  # many pairs: four a thread with own values, one with packed reads
    (_matrix(1360, 34, 22, 0.02), 910000),           # and four a thread with packed reads
    (_sparse(60, 90, 0.3), 1770),                    # a pair has a tenth of the samples: one thread per pair
    (_sparse(60, 90, 0.45), 1770),                   # a fifth: tiles for many pairs, one thread per pair for a few
    (_matrix(14, 6000, 23), 91),                     # more samples than fit beside 16 x 32 genes
], ids=["130k", "910k", "sparse", "half", "6000"])
def test_tile_choices(gem, size, semantics):
    """Whole work blocks from the start; few rows and few pairs; the oracle on every part (for the largest on its last
    work block, whose packed reads look back into that block only)."""
    genes = gem.shape[0]
    row = lambda x: x * (x - 1) // 2  # noqa: E731
    sim = Similarity(gem, semantics=semantics, minsamp=2)
    whole = sim.execute(None, start=0, size=size)
    last = (size - 1) // 32768 * 32768
    for start, n in [(last, size - last), (0, min(size, 500))]:
        _, _, corr, _ = pyoracle.run_block(gem, pyoracle.params(semantics=int(semantics == "fixed"), min_samples=2), start, n)
        assert np.array_equal(whole.corr[start:start + n], corr, equal_nan=True)
    for start, n in [(row(genes - 3) + 1, 1), (row(genes - 3) + 2, 7), (row(genes - 5), 2 * genes - 12), (row(genes - 7) + 2, 4 * genes)]:
        n = min(n, size - start)
        if start < 0 or n < 1:
            continue
        assert np.array_equal(sim.execute(None, start=start, size=n).corr, whole.corr[start:start + n], equal_nan=True)
    sim.close()
