"""The Seq kernel's last two levels over sets that a deep stream (k = 5, 6)
reaches with more than 64 candidates: every way of following the members there
(32, a slot; several slots with and without members between; more than the
scratch holds), and 32-bit values next to their cap, against the oracle.

The sets are made to order: X, a sparse graph of q vertices (and some more, so
that a stream never fits in registers), under k - 1 hubs that are joined to each
other and to X, the lowest of them to the q alone.  The DAG's order is given, so
the hubs are the roots and the last two levels run over X; `near` of the q have
loads that a prefix value can reach, the rest lie far above.

Whole numbers, compared for equality: no tolerance."""
import numpy as np
import pytest

import kclistpp_gb300 as K
from oracle import oracle as O

THREADS = max(1, min(16, O.max_threads()))
FOLLOWED = 256  # most members followed in the kernel's scratch

# (q, near): where the ways change, and beyond the word and slot edges
SETS = [(2, 1), (31, 31), (32, 9), (33, 5), (33, 33), (64, 32), (65, 33), (66, 33), (100, 40), (256, 100), (256, 200),
        (257, 128), (257, 200), (300, 33), (300, 256), (600, 256), (600, 257), (900, 32), (900, 400)]


def _graph(q, k, p, seed):
    """Pairs over the DAG's own ids: X in [0, m), hubs above."""
    rng = np.random.default_rng(seed)
    m, hubs = max(q, 70), k - 1
    i, j = np.triu_indices(m, 1)
    keep = rng.random(len(i)) < p
    pairs = [np.stack([i[keep], j[keep]], axis=1)]
    for h in range(hubs):
        x = np.arange(q if h == 0 else m)
        pairs.append(np.stack([x, np.full(len(x), m + h)], axis=1))
        pairs.append(np.stack([m + np.arange(h), np.full(h, m + h)], axis=1))
    return np.concatenate(pairs).astype(np.uint32), m, hubs


def _loads(q, near, m, hubs, seed):
    rng = np.random.default_rng(seed)
    r = np.full(m + hubs, 1 << 26, np.uint64) + rng.integers(0, 100, m + hubs).astype(np.uint64)
    r[rng.choice(q, near, replace=False)] = rng.integers(0, 64, near)
    r[m:] = rng.integers(0, 64, hubs)
    return r


def _way(np_, ni):
    """What the kernel does with a set of np_ members, ni of them in reach."""
    if np_ <= 32:
        return "slot, all"
    if ni <= 32:
        return "slot, some"
    if 2 * ni > np_ and np_ <= FOLLOWED:
        return "slots, all"
    return "slots, some" if ni <= FOLLOWED else "words"


def test_the_sets_reach_every_way():
    ways = set()
    for q, near in SETS:
        pairs, m, hubs = _graph(q, 5, 0.05, q)
        r = _loads(q, near, m, hubs, q)
        adj = np.zeros((m + hubs, m + hubs), bool)
        adj[pairs.max(1), pairs.min(1)] = True
        top, second, low = m + hubs - 1, m + 1, m
        cand = adj[top] & adj[second]            # the stream of root edge (top, second)
        assert cand.sum() > 64                   # beyond the register streams
        last = cand & adj[low]                   # the last two levels under the lowest hub
        assert last.sum() == q
        reach = int(r[m:].min()) + q * (q - 1) // 2
        ni = int((r[last] < reach).sum())
        if q > 32:
            assert ni == near
        ways.add(_way(q, ni))
    assert ways == {"slot, all", "slot, some", "slots, all", "slots, some", "words"}


@pytest.mark.gpu
@pytest.mark.parametrize("k", [5, 6])
@pytest.mark.parametrize("q,near", SETS)
def test_deep_sets(ctx, q, near, k):
    for p in (4.0 / max(q, 8), 0.15 if q <= 300 else 0.03):
        pairs, m, hubs = _graph(q, k, min(p, 1.0), 3 * q + k)
        rank = np.arange(m + hubs, dtype=np.uint32)
        og = O.Graph(pairs, rank=rank)
        g = K.build_graph(ctx, K.EdgeList.from_pairs(pairs), rank=rank)
        assert g.n == og.n == m + hubs
        r = want = _loads(q, near, m, hubs, q + k)
        for _ in range(2):
            r = K.seq_passes(g, k, 1, r)
            want = og.seq_pass(k, want.copy(), O.SEQ_EDGE_STREAMS, THREADS)
            assert np.array_equal(r, want), int((r != want).sum())
        g.close()


@pytest.mark.gpu
@pytest.mark.parametrize("k", [3, 4, 5])
@pytest.mark.parametrize("n", [5, 34, 70])
def test_loads_next_to_the_cap(ctx, n, k):
    """A 32-bit value is an offset from the root's smallest, capped at 2^31 - 16;
    a stream that could come within 64 of it takes 64-bit values."""
    i, j = np.triu_indices(n, 1)
    pairs = np.stack([i, j], axis=1).astype(np.uint32)
    og = O.Graph(pairs)
    g = K.build_graph(ctx, K.EdgeList.from_pairs(pairs))
    sp = K.get_schedule(g)
    sp.tier_s_max_seq = 1
    K.set_schedule(g, sp)
    rng = np.random.default_rng(n + k)
    cap = (1 << 31) - 16
    for below in (0, 1, 63, 64, 65, 64 + n, 64 + n * n // 2, 64 + n ** 3 // 6):
        r = (cap - below + rng.integers(-3, 4, n)).astype(np.uint64)
        r[rng.integers(0, n)] = 0                 # the smallest: the others lie next to the cap
        got = K.seq_passes(g, k, 1, r)
        want = og.seq_pass(k, r.copy(), O.SEQ_EDGE_STREAMS, THREADS)
        assert np.array_equal(got, want), (below, int((got != want).sum()))
    g.close()
