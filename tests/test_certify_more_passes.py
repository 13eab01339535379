"""kclpp_certify_densest on loads that rank a sparser part of the graph first:
a candidate of which a subset is denser is given up for the one that further
passes rank first, within max_passes of them.

Two cliques joined by an edge, the loads of a run that has not yet reached the
larger one: the first PAVA block is both cliques, of which K_12 alone is denser.
A pass adds 220 / 12 = 18.3 triangles (495 / 12 = 41.3 4-cliques) to a vertex of
K_12 and 84 / 9 = 9.3 (126 / 9 = 14) to one of K_9, so that a lead of 30 is gone
after a few passes and stands after one, whatever order the streams run in.
"""
import numpy as np
import pytest

import kclistpp_gb300 as K

pytestmark = pytest.mark.gpu


def _clique(lo, n):
    return [(u, v) for u in range(lo, lo + n) for v in range(u + 1, lo + n)]


@pytest.mark.parametrize("k,cliques,both", [(3, 220, 304), (4, 495, 621)])
def test_a_refuted_candidate_is_replaced(ctx, k, cliques, both):
    el = K.EdgeList.from_pairs(np.array(_clique(0, 12) + _clique(12, 9) + [(0, 12)], dtype=np.uint32))
    g = K.build_graph(ctx, el)
    rank = np.asarray(K.core_order(el))
    r = np.zeros(g.n, np.uint64)
    r[rank[12:]] = 30
    # the loads' own candidate, when there are too few passes for another
    info, mem = K.certify_densest(g, k, r, 1)
    assert (info.n, info.cliques, info.inside, info.certified) == (21, both, 0, 0), info.as_dict()
    assert len(mem) == 21
    for base in (0, 1 << 40):  # passes compare differences only
        info, mem = K.certify_densest(g, k, r + np.uint64(base), 64)
        assert info.certified and (info.n, info.cliques) == (12, cliques), info.as_dict()
        assert set(mem.tolist()) == set(rank[:12].tolist())
    # loads without room for the passes' units keep their own candidate
    r[rank[12:]] = 1 << 62
    info, _ = K.certify_densest(g, k, r, 64)
    assert (info.n, info.cliques, info.certified) == (21, both, 0), info.as_dict()
    g.close()
