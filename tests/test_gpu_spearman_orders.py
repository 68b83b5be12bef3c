"""Spearman without clustering from the genes' sample orders: sample counts around the 32-sample steps, equal
values (where the reference's sorting network decides the ranks) alone, in long runs across a step's edge and
in one gene only, signed zeros, infinities, missing and low values, too few samples, and more samples than the
orders take.  Correlations are the oracle's bit for bit (the tolerance of every parity test here); labels are
the sample states."""
import numpy as np
import pytest

from kinc_gb300 import Similarity
from oracle import pyoracle

pytestmark = pytest.mark.gpu


def _check(gem, corrmethod="spearman", **kw):
    gargs = dict(corrmethod=corrmethod, **kw)
    oargs = dict(corr_method=["pearson", "spearman", "both"].index(corrmethod))
    oargs.update({"min_samples": v if k == "minsamp" else None for k, v in kw.items() if k == "minsamp"})
    if "minexpr" in kw:
        oargs["min_expr"] = kw["minexpr"]
    sim = Similarity(gem, **gargs)
    sim.initialize()
    total = sim.total_pairs()
    res = sim.execute(None, start=0, size=total)
    sim.close()
    K, _, corr, _ = pyoracle.run_block(gem, pyoracle.params(**oargs), 0, total)
    assert np.array_equal(res.K, K)
    assert np.array_equal(np.nan_to_num(res.corr, nan=9.0), np.nan_to_num(corr, nan=9.0))
    x, y = np.tril_indices(len(gem), -1)
    low = np.float32(kw.get("minexpr", -np.inf))
    nan = np.isnan(gem[x]) | np.isnan(gem[y])
    want = np.where(nan, -9, np.where((gem[x] < low) | (gem[y] < low), -6, 0)).astype(np.int8)
    assert np.array_equal(res.labels, want)


def _normal(genes, samples, seed, missing=0.1):
    rng = np.random.default_rng(seed)
    gem = rng.normal(8.0, 2.0, (genes, samples)).astype(np.float32)
    gem[rng.random(gem.shape) < missing] = np.nan
    return gem


@pytest.mark.parametrize("samples", [1, 2, 3, 31, 32, 33, 63, 64, 65, 127, 128, 129, 160, 161, 500])
def test_sample_counts(samples):
    _check(_normal(14, samples, samples), minsamp=1)


@pytest.mark.parametrize("levels", [1, 2, 5, 40, 300])
@pytest.mark.parametrize("samples", [40, 200])
def test_equal_values(levels, samples):
    gem = _normal(16, samples, levels, missing=0.3)
    rng = np.random.default_rng(levels)
    few = rng.integers(0, levels, (10, samples)).astype(np.float32)
    gem[:10] = np.where(np.isnan(gem[:10]), np.nan, few)       # the other genes keep distinct values
    _check(gem)


def test_equal_values_in_one_sample_pair_only():
    gem = _normal(30, 150, 5, missing=0.4)
    for g in range(0, 30, 2):
        i, j = np.random.default_rng(g).choice(150, 2, replace=False)
        gem[g, j] = gem[g, i]
    _check(gem)


def test_zeros_infinities_low_values():
    gem = _normal(16, 96, 8) - np.float32(8.0)
    gem[0, :5], gem[0, 5:9] = 0.0, -0.0
    gem[1, 3], gem[2, 3], gem[2, 4] = np.inf, -np.inf, -np.inf
    gem[3, 10:12] = np.inf
    gem[4] = np.nan
    gem[5, 8:] = np.nan
    _check(gem, minexpr=-3.0)
    _check(gem, corrmethod="both", minexpr=-3.0)


def test_more_samples_than_the_orders_take():
    _check(_normal(4, 8200, 2))
    _check(_normal(4, 8192, 3))


def test_both_correlations_over_work_blocks():
    _check(_normal(270, 40, 4), corrmethod="both")
