"""Seq streams whose values differ by more than 2^31 at k >= 6, on the CTA-per-root
kernel, beside streams of the same roots whose values do not (whole numbers, the
oracle's: no tolerance)."""
import numpy as np
import pytest

import kclistpp_gb300 as K
from oracle import oracle as O

pytestmark = pytest.mark.gpu

THREADS = max(1, min(16, O.max_threads()))


@pytest.mark.parametrize("k", [6, 7, 8])
@pytest.mark.parametrize("n,p", [(18, 1.0), (34, 0.8), (70, 0.45)])
def test_wide_loads_against_oracle(ctx, n, p, k):
    rng = np.random.default_rng(n)
    i, j = np.triu_indices(n, 1)
    keep = rng.random(len(i)) < p
    pairs = np.stack([i[keep], j[keep]], axis=1).astype(np.uint32)
    og = O.Graph(pairs)
    g = K.build_graph(ctx, K.EdgeList.from_pairs(pairs))
    sp = K.get_schedule(g)
    sp.tier_s_max_seq = 1
    K.set_schedule(g, sp)
    loads = {
        "spread": rng.integers(0, 1 << 40, g.n),
        "two levels": rng.integers(0, 2, g.n) * (1 << 33) + rng.integers(0, 20, g.n),
        "one low": np.where(np.arange(g.n) == g.n // 2, 0, (1 << 35) + rng.integers(0, 20, g.n)),
        "at the bound": rng.integers(0, 2, g.n) * ((1 << 31) - 100) + rng.integers(0, 200, g.n),
    }
    for name, r in loads.items():
        r = r.astype(np.uint64)
        want = og.seq_pass(k, r, O.SEQ_EDGE_STREAMS, THREADS)
        assert np.array_equal(K.seq_passes(g, k, 1, r), want), name
    g.close()
