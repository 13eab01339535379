"""The rows of warp-per-root roots around 32 members, where the way they are built
changes: members with a bitmap row, without one, and both in one root, with
out-neighbours among the members, below, between and beyond them.  Clique
degrees, Sim counts, prefix counts and Seq loads against the oracle (whole
numbers: no tolerance)."""
import numpy as np
import pytest

import kclistpp_gb300 as K
from oracle import oracle as O

THREADS = max(1, min(16, O.max_threads()))
SIZES = (1, 2, 3, 4, 5, 16, 31, 32, 33, 34)
STYLES = ("near", "far", "both")


def _graph(d):
    """Edges (id, lower id) with ids as the program numbers them, and the roots."""
    rng = np.random.default_rng(d)
    at, edges, roots = 8, [], []
    for style in STYLES:
        for p in (0.15, 0.6, 1.0):
            if style == "near":
                mem = at + np.arange(d)
            elif style == "far":
                mem = at + 131 * np.arange(d)
            else:
                mem = at + np.concatenate([np.arange(d // 2), 40 + 131 * np.arange(d - d // 2)])
            mem = mem.astype(np.int64)
            for i in range(d):
                edges += [(mem[i], mem[j]) for j in range(i) if rng.random() < p]
                lo = mem[i] - 1 - rng.integers(0, 60, 2)  # members or not, close below
                edges += [(mem[i], x) for x in lo if x >= at - 8]
                if rng.random() < 0.3 and i:
                    edges.append((mem[i], mem[0] - 1 - rng.integers(0, 7)))
            at = int(mem[-1]) + 2
            edges += [(at, x) for x in mem]
            roots.append(at)
            at += 10
    e = np.unique(np.array([(a, b) for a, b in edges if a != b], dtype=np.int64), axis=0)
    return e.astype(np.uint32), roots[-1] + 1, roots


def _has_row(off, cols):
    d = np.diff(off.astype(np.int64))
    row = np.zeros(len(d), bool)
    for v in np.flatnonzero(d > 1):
        c = cols[int(off[v]):int(off[v + 1])].astype(np.int64)
        row[v] = (c[-1] - c[0]) // 32 + 1 <= 2 * d[v]
    return row


@pytest.mark.parametrize("d", SIZES)
def test_the_graphs_are_what_they_are_for(d):
    edges, n, roots = _graph(d)
    og = O.Graph(edges, n, np.arange(n))
    off, cols = og.csr()
    assert [int(off[s + 1] - off[s]) for s in roots] == [d] * len(roots)
    row = _has_row(off, cols)
    kinds = {(bool(row[m].any()), bool((~row[m]).any())) for s in roots
             for m in [cols[int(off[s]):int(off[s + 1])]]}
    if d >= 16:
        assert (True, True) in kinds
    assert any(without for _, without in kinds) and (d < 3 or any(with_ for with_, _ in kinds))


@pytest.mark.gpu
@pytest.mark.parametrize("d", SIZES)
def test_small_roots_against_oracle(ctx, d):
    edges, n, _ = _graph(d)
    og = O.Graph(edges, n, np.arange(n))
    g = K.build_graph(ctx, K.EdgeList.from_pairs(edges), rank=np.arange(n))
    assert all(np.array_equal(a, b) for a, b in zip(g.csr(), og.csr()))
    sp = K.get_schedule(g)
    sp.tier_s_max = 63  # not the default: kept at every k
    sp.tier_s_max_seq = 63
    K.set_schedule(g, sp)
    rng = np.random.default_rng(d)
    for k in (3, 4, 5, 6):
        tot, per = K.count_cliques(g, k)
        otot, oper = og.count_cliques(k)
        assert tot == otot and np.array_equal(per, oper), k
        for span in (3, 1000):
            rho = rng.integers(0, span, n).astype(np.float64)
            assert np.array_equal(K.sim_counts(g, k, rho), og.sim_counts(k, rho, THREADS)), (k, span)
            r = rng.integers(0, span, n).astype(np.uint64)
            assert np.array_equal(K.seq_passes(g, k, 1, r), og.seq_pass(k, r, O.SEQ_EDGE_STREAMS, THREADS)), (k, span)
            _, level = K.sort_by_r_u64(r)
            assert np.array_equal(K.pava(g, k, level), og.pava(k, level)), (k, span)
    g.close()
