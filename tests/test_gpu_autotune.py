"""The per-pair kernel's launch shape (kinc_sim_set_launch / kinc_sim_autotune): every shape gives
bit-identical results, the autotuner picks one of the timed candidates, and its cache answers a
second call without timing anything."""
import numpy as np
import pytest

from kinc_gb300 import Similarity, _native, synthetic

pytestmark = pytest.mark.gpu

# warps per CTA divide the kernel's warp count: 20 for GMM, 16 otherwise
SHAPES = {"gmm": [(20, 1, 8), (10, 1, 0), (4, 0, 16), (20, 0, 4)],
          "kmeans": [(16, 1, 8), (8, 1, 0), (4, 0, 16), (16, 0, 4)]}


@pytest.mark.parametrize("args", [dict(clusmethod="gmm", corrmethod="spearman", crit="BIC", preout=True,
                                       postout=True),
                                  dict(clusmethod="kmeans", corrmethod="pearson", maxclus=3, crit="BIC")],
                         ids=["gmm", "kmeans"])
def test_every_launch_shape_gives_the_same_bits(args):
    gem = synthetic.generate(2, genes=70, samples=150)
    sim = Similarity(gem, **args)
    sim.initialize()
    total = sim.total_pairs()
    want = None
    for w, r, p in SHAPES[args["clusmethod"]]:
        sim.set_launch(w, r, p)
        assert sim.launch() == {"warps_per_cta": w, "rounds": r, "prefetch": p}
        res = sim.execute(None, start=0, size=total)
        got = (res.K, res.labels[res.K > 1], np.nan_to_num(res.corr, nan=9.0).view(np.uint32))
        if want is None:
            want = got
        else:
            for a, b in zip(got, want):
                assert np.array_equal(a, b)
    sim.close()


def test_launch_shape_rejects_unsupported_values():
    gem = synthetic.generate(2, genes=20, samples=60)
    sim = Similarity(gem, clusmethod="gmm")
    sim.initialize()
    with pytest.raises(_native.SimError):
        sim.set_launch(5, 1, 8)
    with pytest.raises(_native.SimError):
        sim.set_launch(16, 1, 8)       # does not divide GMM's 20 warps
    with pytest.raises(_native.SimError):
        sim.set_launch(16, 2, 8)
    sim.close()


def test_autotune_picks_a_timed_candidate_and_caches_it(tmp_path, monkeypatch):
    monkeypatch.setenv("KINC_TUNE_CACHE", str(tmp_path / "launch.txt"))
    gem = synthetic.generate(2, genes=120, samples=200)
    sim = Similarity(gem, clusmethod="gmm", corrmethod="spearman", crit="BIC")
    sim.initialize()
    chosen, timed = sim.autotune(start=0, size=sim.total_pairs())
    assert len(timed) >= 4
    fastest = min(timed, key=lambda e: e["ms"])
    assert chosen == {k: fastest[k] for k in ("warps_per_cta", "rounds", "prefetch")}
    assert sim.launch() == chosen
    again, timed2 = sim.autotune(start=0, size=sim.total_pairs())
    assert again == chosen and timed2 == []
    assert (tmp_path / "launch.txt").read_text().count("\t") == 2
    sim.close()


def _wave():
    """Pairs the GMM tile kernel runs at once: 20 warps of 32 on every SM."""
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count * 20 * 32


def test_every_launch_shape_of_the_gmm_tile_kernel_gives_the_same_bits():
    """A block of one full wave with two genes of many samples runs in tiles, one of a part of a wave does not."""
    genes = 480
    gem = synthetic.generate(2, genes=genes, samples=2600)
    gem[:, 300:] = np.nan
    gem[:2] = synthetic.generate(2, genes=2, samples=2600, seed=5)
    sim = Similarity(gem, clusmethod="gmm", corrmethod="spearman", crit="BIC", maxclus=2, preout=True)
    sim.initialize()
    assert _wave() <= genes * (genes - 1) // 2
    want = sim.execute(None, start=0, size=3000)
    assert sim.last_kernel() == "gmm pairs"
    for shape in SHAPES["gmm"]:
        sim.set_launch(*shape)
        got = sim.execute(None, start=0, size=_wave())
        assert sim.last_kernel() == "tiles"
        assert np.array_equal(got.K[:3000], want.K)
        assert np.array_equal(got.labels[:3000][want.K > 1], want.labels[want.K > 1])
        assert np.array_equal(got.corr[:3000], want.corr, equal_nan=True)
    sim.close()


def test_autotune_times_the_kernel_that_takes_the_shape(tmp_path, monkeypatch):
    cache = tmp_path / "launch.txt"
    monkeypatch.setenv("KINC_TUNE_CACHE", str(cache))
    # GMM: the tile kernel, also where this worker's blocks run with one warp per pair
    sim = Similarity(synthetic.generate(2, genes=40, samples=600), clusmethod="gmm", corrmethod="spearman", maxclus=2)
    before = sim.execute(None, start=0, size=sim.total_pairs())
    assert sim.last_kernel() == "gmm pairs"
    _, timed = sim.autotune()
    assert sim.last_kernel() == "tiles" and len(timed) >= 4
    after = sim.execute(None, start=0, size=sim.total_pairs())
    assert sim.last_kernel() == "gmm pairs"
    assert np.array_equal(before.K, after.K) and np.array_equal(before.corr, after.corr, equal_nan=True)
    sim.close()
    assert cache.read_text().startswith("kernel=tiles ")
    # K-means with a stream of pairs: warps per CTA only
    sim = Similarity(synthetic.generate(4, genes=40, samples=80), clusmethod="kmeans", maxclus=3)
    default = sim.launch()
    _, timed = sim.autotune()
    assert sim.last_kernel() == "kmeans pairs"
    assert sorted(t["warps_per_cta"] for t in timed) == [4, 8, 16]
    assert all(t[k] == default[k] for t in timed for k in ("rounds", "prefetch"))
    sim.close()
    assert cache.read_text().count("kernel=stream ") == 1


@pytest.mark.parametrize("corr", ["pearson", "spearman", "both"])
def test_autotune_without_a_shape_to_pick(corr, tmp_path, monkeypatch):
    """Without clustering no kernel takes a shape: nothing is timed, and nothing is kept for other matrices."""
    cache = tmp_path / "launch.txt"
    monkeypatch.setenv("KINC_TUNE_CACHE", str(cache))
    sim = Similarity(synthetic.generate(1, genes=50, samples=90), corrmethod=corr)
    chosen, timed = sim.autotune()
    assert chosen == sim.launch() and timed == [] and not cache.exists()
    sim.execute(None, start=0, size=sim.total_pairs())
    assert sim.last_kernel() == "genes"
    sim.close()
