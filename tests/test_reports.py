"""The report's order and densest prefix on the device, at sizes around a sort
tile (2048 vertices) and keys of every width, against numpy; and the sample at
out-degrees around its launch groups' bounds, against the oracle.

Whole numbers and one quotient of them, compared for equality: no tolerance."""
import numpy as np
import pytest

import kclistpp_gb300 as K
from oracle import oracle as O
from tests.test_sampling_host import bipartite_with_clique, sort_rows

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3, 33, 2047, 2048, 2049, 4097, 70001])
@pytest.mark.parametrize("keys", ["equal", "byte", "wide", "top"])
def test_order_and_prefix(ctx, n, keys):
    i = np.arange(n, dtype=np.uint32)
    pairs = np.stack([i, (i + 1) % n], axis=1)                 # a ring
    pairs = np.concatenate([pairs, np.stack([i[:-2:3], i[2::3]], axis=1)[: n // 3]]) if n > 3 else pairs
    pairs = np.unique(np.sort(pairs, axis=1), axis=0)
    g = K.build_graph(ctx, K.EdgeList.from_pairs(pairs))
    rng = np.random.default_rng(n)
    hi = {"equal": 1, "byte": 256, "wide": 1 << 40, "top": 1 << 63}[keys]
    r = rng.integers(0, hi, g.n).astype(np.uint64)
    if keys == "wide":
        r[rng.random(g.n) < 0.5] = 7                           # ties: ascending id
    info, order = K.extract_densest_seq(g, 3, 1, r)
    want = np.lexsort((np.arange(g.n), ~r))
    assert np.array_equal(order, want)
    level = np.empty(g.n, np.uint32)
    level[want] = np.arange(g.n)
    tent = K.pava(g, 3, level)
    sums = np.cumsum(tent)
    dens = sums.astype(np.float64) / np.arange(1, g.n + 1)
    at = int(np.argmax(dens))                                  # the first largest
    assert (info.n, info.cliques, info.density) == (at + 1, int(sums[at]), dens[at])
    off, cols = g.csr()
    src = np.repeat(np.arange(g.n), np.diff(off.astype(np.int64)))
    assert info.m == int(((level[src] <= at) & (level[cols] <= at)).sum())
    rho = r.astype(np.float64) * 0.75
    info2, order2 = K.extract_densest_sim(g, 3, rho)
    key = rho.astype(np.uint64)
    assert np.array_equal(order2, np.lexsort((np.arange(g.n), ~key)))
    g.close()


@pytest.mark.parametrize("a", [63, 65, 255, 258, 1023, 1026])
@pytest.mark.parametrize("k", [3, 4, 6])
def test_sample_at_group_bounds(ctx, a, k):
    pairs = bipartite_with_clique(a, a, 9)
    g = K.build_graph(ctx, K.EdgeList.from_pairs(pairs))
    og = O.Graph(pairs)
    total = og.count_cliques(k)[0]
    for target in (total + 1, max(total // 3, 1)):
        s = K.Sampling(g, k, target, 11, 8)
        all_, _, thr = O.sampling_threshold(target, total)
        want = sort_rows(*og.sampling_collect(k, 11, thr, all_, 8))
        rows, wave = s.cliques()
        assert np.array_equal(rows, want[0]) and np.array_equal(wave, want[1])
        s.passes(3)
        rho = np.zeros(og.n, np.uint32)
        for _ in range(3):
            rho = O.sampling_pass(og.n, k, want[0], want[1], 8, rho)
        assert np.array_equal(s.rho(), rho)
        s.close()
    g.close()
