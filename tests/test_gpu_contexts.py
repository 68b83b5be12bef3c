"""Several workers of one process: what one of them sets up for its sample count and options must not take
anything from another (a kernel's shared-memory limit belongs to the kernel, not to a worker)."""
import ctypes
import threading

import numpy as np
import pytest

from kinc_gb300 import Similarity, _native, synthetic

pytestmark = pytest.mark.gpu

SORTED = dict(corrmethod="spearman", preout=True, postout=True, crit="BIC")
PLAIN = dict(corrmethod="pearson", crit="BIC")


def _same(a, b):
    assert np.array_equal(a.K, b.K)
    assert np.array_equal(a.labels[a.K > 1], b.labels[a.K > 1])
    assert np.array_equal(a.corr, b.corr, equal_nan=True)


@pytest.mark.parametrize("first,second", [
    # more shared memory in the first worker than in the second, on one kernel
    (("kmeans", 900, dict(SORTED, maxclus=3)), ("kmeans", 60, dict(PLAIN, maxclus=3))),
    (("kmeans", 300, dict(SORTED, maxclus=5)), ("kmeans", 50, dict(SORTED, maxclus=5))),
    (("gmm", 400, dict(SORTED, maxclus=6)), ("gmm", 60, dict(SORTED, maxclus=6))),
    (("none", 9000, SORTED), ("none", 8300, SORTED)),
], ids=["kmeans", "kmeans5", "gmm6", "none"])
def test_a_second_worker_with_less_shared_memory(first, second):
    def worker(clus, samples, args):
        return Similarity(synthetic.generate(4, genes=9, samples=samples), clusmethod=clus, **args)

    with_both = worker(*first)
    want = with_both.execute(None, start=0, size=with_both.total_pairs())
    other = worker(*second)
    other.execute(None, start=0, size=other.total_pairs())
    _same(with_both.execute(None, start=0, size=with_both.total_pairs()), want)
    with_both.close()
    other.close()


def test_the_allocation_free_call_between():
    import torch
    sim = Similarity(synthetic.generate(4, genes=9, samples=900), clusmethod="kmeans", maxclus=3, **SORTED)
    want = sim.execute(None, start=0, size=36)
    gem = synthetic.generate(4, genes=9, samples=60)
    params = Similarity(gem, clusmethod="kmeans", maxclus=3, **PLAIN).params
    d_gem = torch.from_numpy(gem).cuda()
    K = torch.empty(36, dtype=torch.int8, device="cuda")
    vp = ctypes.c_void_p
    _native.check(_native.load().kinc_sim_execute_block_noalloc(vp(d_gem.data_ptr()), 9, 60, ctypes.byref(params), 0, 36,
                                                                vp(K.data_ptr()), None, None, None), None)
    _same(sim.execute(None, start=0, size=36), want)
    sim.close()


@pytest.mark.parametrize("corr,size", [("pearson", 3), ("pearson", 60), ("spearman", 60)])
def test_threads_with_different_sample_counts(corr, size):
    """Four threads, a worker each, block after block: every one gets what it got alone."""
    sims = [Similarity(synthetic.generate(1, genes=60, samples=s), corrmethod=corr) for s in (70, 1900, 300, 1100)]
    want = [s.execute(None, start=1700, size=size) for s in sims]
    errors = []

    def run(sim, expected):
        try:
            for _ in range(150):
                _same(sim.execute(None, start=1700, size=size), expected)
        except Exception as e:                             # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=run, args=a) for a in zip(sims, want)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for s in sims:
        s.close()
    assert not errors, errors[0]
