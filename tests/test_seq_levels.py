"""The Seq kernel's last two levels (whole streams in registers, members
compacted 32 to a slot, groups settled by counting or walked chain by chain)
against the oracle, at the candidate counts and loads where its routes change.

r is a vector of whole numbers and every comparison is for equality, so there
is no tolerance."""
import numpy as np
import pytest

import kclistpp_gb300 as K
from oracle import oracle as O

pytestmark = pytest.mark.gpu

THREADS = max(1, min(16, O.max_threads()))

# Out-degrees and candidate sets around one slot (32), two (64), the most
# members followed (256) and beyond; dense enough that they are reached.
SIZES = [(5, 1.0), (33, 1.0), (34, 1.0), (36, 0.95), (66, 1.0), (70, 0.9), (130, 0.7), (300, 1.0), (420, 0.8)]


def _graph(n, p, seed):
    rng = np.random.default_rng(seed)
    a = np.triu(rng.random((n, n)) < p, 1)
    return np.stack(np.nonzero(a), axis=1).astype(np.uint32)


def _loads(kind, n, rng):
    if kind == "zero":
        return np.zeros(n, np.uint64)
    if kind == "ties":      # every chain is decided by ties and single units
        return rng.integers(0, 4, n).astype(np.uint64)
    if kind == "near":      # gaps of the order of a stream's cliques
        return rng.integers(0, 20000, n).astype(np.uint64)
    if kind == "spread":    # mostly settled by counting
        return rng.integers(0, 1 << 24, n).astype(np.uint64)
    if kind == "cap":       # beyond 32 bits above the smallest value
        r = rng.integers(0, 1 << 12, n).astype(np.uint64)
        r[:: 3] += np.uint64((1 << 31) - 4000)
        r[1:: 3] += np.uint64(1 << 40)
        return r
    r = np.zeros(n, np.uint64)  # "few": a few members below, the rest far above
    r[:] = 1 << 26
    r[rng.choice(n, max(1, n // 10), replace=False)] = rng.integers(0, 64)
    return r


@pytest.mark.parametrize("loads", ["zero", "ties", "near", "spread", "cap", "few"])
@pytest.mark.parametrize("n,p", SIZES)
def test_streams_at_slot_edges(ctx, n, p, loads):
    pairs = _graph(n, p, seed=n)
    og = O.Graph(pairs)
    g = K.build_graph(ctx, K.EdgeList.from_pairs(pairs))
    sp = K.get_schedule(g)
    sp.tier_s_max_seq = 1  # every root on the CTA-per-root kernel
    K.set_schedule(g, sp)
    for k in [k for k in (4, 5, 6, 7, 8) if n ** k <= 4e11]:
        r = _loads(loads, g.n, np.random.default_rng(7 * n + k))
        got = K.seq_passes(g, k, 1, r)
        want = og.seq_pass(k, r.copy(), O.SEQ_EDGE_STREAMS, THREADS)
        assert np.array_equal(got, want), (k, int((got != want).sum()))
    g.close()
