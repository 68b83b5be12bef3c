"""The dense Pearson form's K = 1 and NaN columns: every pair of the range and nothing beside it, wherever the
caller's K begins and whatever is left of 16 bytes (exact)."""
import ctypes

import numpy as np
import pytest

from kinc_gb300 import Similarity, synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("max_k", [1, 2, 5])
@pytest.mark.parametrize("offset,size", [(0, 1), (1, 15), (3, 13), (5, 11), (15, 16), (8, 17), (16, 4096), (7, 7001)])
def test_k_and_empty_columns(max_k, offset, size):
    import torch

    from kinc_gb300 import _native
    gem = synthetic.generate(3, genes=150, samples=70, seed=8)
    sim = Similarity(gem, semantics="fixed", precision="fp16", maxclus=max_k)
    sim.initialize()
    L = _native.load()
    K = torch.full((offset + size + 40,), 7, dtype=torch.int8, device="cuda")
    corr = torch.full((size + 3, max_k), 2.0, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()             # the worker runs on its own stream
    vp = ctypes.c_void_p
    _native.check(L.kinc_sim_execute_block_device(sim._ctx, 321, size, vp(K.data_ptr() + offset), None,
                                                  vp(corr.data_ptr()), None), sim._ctx)
    _native.check(L.kinc_sim_synchronize(sim._ctx), sim._ctx)
    sim.close()
    K, corr = K.cpu().numpy(), corr.cpu().numpy()
    assert np.all(K[offset:offset + size] == 1)
    assert np.all(K[:offset] == 7) and np.all(K[offset + size:] == 7)
    assert np.all(np.isnan(corr[:size, 1:])) and np.all(corr[:size, 0] != 2.0)
    assert np.all(corr[size:] == 2.0)
