"""How a root's induced rows are built (bitmap rows, walked lists looked up in
the position table), against the oracle's counts, Sim counts and Seq loads, at
out-degrees and id patterns where the routes and the table sizes change.

Whole numbers, compared for equality: no tolerance."""
import numpy as np
import pytest

import kclistpp_gb300 as K
from oracle import oracle as O

pytestmark = pytest.mark.gpu

THREADS = max(1, min(16, O.max_threads()))


def _join(*parts):
    e = np.sort(np.concatenate(parts).astype(np.int64), axis=1)
    return np.unique(e[e[:, 0] != e[:, 1]], axis=0).astype(np.uint32)


def _clique(ids):
    i, j = np.triu_indices(len(ids), 1)
    return np.stack([ids[i], ids[j]], axis=1)


def _bipartite(a, p_in, rng):
    """Degeneracy a and few cliques: out-degrees up to a without a count explosion."""
    left, right = np.arange(a), np.arange(a, 2 * a)
    parts = [np.stack(np.meshgrid(left, right, indexing="ij"), -1).reshape(-1, 2)]
    for side in (left, right):
        i, j = np.triu_indices(a, 1)
        keep = rng.random(len(i)) < p_in
        parts.append(np.stack([side[i[keep]], side[j[keep]]], axis=1))
    return _join(*parts)


def _case(name):
    rng = np.random.default_rng(3)
    if name.startswith("clique"):       # dense rows only; a word, its edge, two words
        return _clique(np.arange(int(name[6:]))), (3, 4)
    if name == "islands":               # cliques over ids far apart: walked rows
        n = 30000
        far = [rng.choice(n, 40, replace=False) for _ in range(12)]
        ring = np.stack([np.arange(n - 1), np.arange(1, n)], axis=1)
        return _join(ring, *[_clique(f) for f in far]), (3, 4, 5)
    if name == "mixed":                 # a dense core, and hubs joined to it and to far ids
        n = 20000
        core = np.arange(150)
        i, j = np.triu_indices(150, 1)
        keep = rng.random(len(i)) < 0.5
        hub = np.stack([np.repeat(rng.choice(n, 60, replace=False), 200),
                        np.where(rng.random(12000) < 0.3, rng.integers(0, 150, 12000), rng.integers(0, n, 12000))], 1)
        return _join(np.stack([core[i[keep]], core[j[keep]]], 1), hub,
                     rng.integers(0, n, (60000, 2))), (3, 4, 5)
    a = int(name[4:])                   # out-degrees around a table size and the tiers' bounds
    return _bipartite(a, 2.0 / a, rng), (3, 4)


@pytest.mark.parametrize("name", ["clique3", "clique32", "clique33", "clique64", "clique65", "clique66", "clique97",
                                  "islands", "mixed", "deep511", "deep513", "deep1026"])
def test_rows_against_oracle(ctx, name):
    pairs, ks = _case(name)
    og = O.Graph(pairs)
    g = K.build_graph(ctx, K.EdgeList.from_pairs(pairs))
    rng = np.random.default_rng(1)
    for smax in (1, 64):                # CTA per root, warp per root
        sp = K.get_schedule(g)
        sp.tier_s_max = sp.tier_s_max_seq = smax
        K.set_schedule(g, sp)
        for k in ks:
            tot, per = K.count_cliques(g, k)
            otot, oper = og.count_cliques(k)
            assert tot == otot and np.array_equal(per, oper), (smax, k)
            rho = rng.integers(0, 5, g.n).astype(np.float64)
            assert np.array_equal(K.sim_counts(g, k, rho), og.sim_counts(k, rho, THREADS)), (smax, k)
            r = rng.integers(0, 50, g.n).astype(np.uint64)
            assert np.array_equal(K.seq_passes(g, k, 1, r), og.seq_pass(k, r, O.SEQ_EDGE_STREAMS, THREADS)), (smax, k)
    g.close()
