"""RMT's pruned matrices by connected components: component sizes around the limits of the one-warp and the
one-CTA block solver and beyond them, chains and stars (no dense blocks), scattered row numbers, several
clusters, repeated eigenvalues and negative ones.  Against numpy's eigenvalues of the whole matrix in 64 bits:
both sides are backward stable, so they differ by a few units of 2^-53 times the largest eigenvalue, far below
the rounding to 32 bits, half a unit of which is the tolerance (2^-24 relative) plus 1e-13 of the largest."""
import numpy as np
import pytest

from kinc_gb300.rmt import RMT

pytestmark = pytest.mark.gpu


def _eigenvalues(G, K, x, y, c, r, t):
    keep = np.abs(r) >= np.float32(t)
    rows = np.unique(np.concatenate([x[keep] * K + c[keep], y[keep] * K + c[keep]]))
    at = {v: i for i, v in enumerate(rows)}
    A = np.eye(len(rows))
    for i in np.flatnonzero(keep):
        a, b = at[x[i] * K + c[i]], at[y[i] * K + c[i]]
        A[a, b] = A[b, a] = r[i]
    w = np.linalg.eigvalsh(A)
    return w[np.argsort(np.abs(w), kind="stable")]


def _network(groups, kind, K=1, seed=1):
    """Components of the given sizes on a random permutation of the genes."""
    rng = np.random.default_rng(seed)
    G = sum(groups) + 7
    perm = rng.permutation(G)
    items, base = [], 0
    for n in groups:
        genes = perm[base:base + n]
        base += n
        k = int(rng.integers(0, K))
        for i in range(1, n):
            others = {"clique": range(i), "chain": [i - 1], "star": [0]}[kind]
            for j in others:
                a, b = max(genes[i], genes[j]), min(genes[i], genes[j])
                items.append((a, b, k, rng.uniform(0.7, 0.99) * (1 if kind == "clique" else rng.choice([-1, 1]))))
    for _ in range(3 * len(items) // 2):                    # items below the threshold join nothing
        a, b = rng.choice(G, 2, replace=False)
        if not any((max(a, b), min(a, b)) == (q[0], q[1]) for q in items[:50]):
            items.append((max(a, b), min(a, b), int(rng.integers(0, K)), rng.uniform(0.0, 0.5)))
    seen = {}
    for q in items:
        seen.setdefault(q[:3], q[3])
    keys = sorted(seen)
    x, y, c = (np.array(v) for v in zip(*keys))
    r = np.array([seen[k] for k in keys], np.float32)
    return G, x.astype(np.int32), y.astype(np.int32), c.astype(np.int8), r


def _check(G, K, x, y, c, r, t):
    got = RMT().prune_eigenvalues((x, y, c, r), G, K, t)
    want = _eigenvalues(G, K, x.astype(np.int64), y.astype(np.int64), c.astype(np.int64), r, t)
    assert len(got) == len(want)
    # equal magnitudes may come in either order: compare what was sorted
    got, want = np.sort(got.astype(np.float64)), np.sort(want)
    assert np.all(np.abs(got - want) <= 2.0 ** -24 * np.abs(want) + 1e-13 * np.abs(want).max())


@pytest.mark.parametrize("kind", ["clique", "chain", "star"])
@pytest.mark.parametrize("groups", [[2], [2, 3, 4, 5], [31, 32, 33, 2], [127, 128, 129], [60] * 5 + [2] * 40, [300, 5, 140, 2]])
def test_component_sizes(groups, kind):
    _check(*(lambda n: (n[0], 1) + n[1:])(_network(groups, kind)), 0.6)


def test_clusters_are_apart():
    G, x, y, c, r = _network([9, 20, 40, 3, 3, 3], "clique", K=3, seed=4)
    _check(G, 3, x, y, c, r, 0.6)


def test_repeated_eigenvalues():
    """Complete graphs with one weight: eigenvalue 1 - w repeated."""
    x, y = np.tril_indices(50, -1)
    same = (x // 10) == (y // 10)
    x, y = x[same].astype(np.int32), y[same].astype(np.int32)
    _check(50, 1, x, y, np.zeros(len(x), np.int8), np.full(len(x), 0.8, np.float32), 0.5)


@pytest.mark.parametrize("rows,a,b,value", [(6, 5, 4, np.inf), (6, 1, 0, np.inf), (40, 39, 38, -np.inf), (150, 7, 3, np.inf)])
def test_infinite_items_have_no_eigenvalues(rows, a, b, value):
    """A matrix with an infinite element has no eigenvalues: every one is NaN, whichever component it is in, and a
    search over thresholds, all of which keep such an item, finds none."""
    G, x, y, c, r = _network([rows, 4, 9], "clique")
    x, y = np.concatenate([x, [G + a]]).astype(np.int32), np.concatenate([y, [G + b]]).astype(np.int32)
    more, less = np.tril_indices(rows, -1)                 # a clique of its own behind the others, with the item in it
    other = (more != a) | (less != b)
    x, y = np.concatenate([x, G + more[other]]).astype(np.int32), np.concatenate([y, G + less[other]]).astype(np.int32)
    r = np.concatenate([r, [value], np.linspace(0.7, 0.9, other.sum())]).astype(np.float32)
    c = np.zeros(len(x), np.int8)
    keep = np.abs(r) >= np.float32(0.6)
    got = RMT().prune_eigenvalues((x, y, c, r), G + rows, 1, 0.6)
    assert len(got) == len(np.unique(np.concatenate([x[keep], y[keep]]))) and np.all(np.isnan(got))
    threshold, steps = RMT(tstart=0.7, tstep=0.05, tstop=0.5).run(items=(x, y, c, r), genes=G + rows, max_clusters=1,
                                                                  strict=False)
    assert threshold is None and len(steps) >= 4 and np.all(steps[:, 2] == -1.0)


@pytest.mark.parametrize("groups", [[90, 20], [64], [20, 3], [129] * 8, [130] * 11 + [40, 3, 2], [900, 140, 700, 129, 5]])
def test_components_that_share_a_matrix(groups):
    """One component with most of the rows, and components above the block solver's limit: solved in matrices that
    hold several of them."""
    _check(*(lambda n: (n[0], 1) + n[1:])(_network(groups, "chain", seed=8)), 0.6)
