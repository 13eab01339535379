"""A tier S bound that a program sets is the one that is launched, at every k;
only a bound at its default follows k.  Counted on the host by the kernels'
names (tests/fake_cudart.c), and on the GPU the results are the oracle's
whichever kernel a root goes to (whole numbers: no tolerance)."""
import numpy as np
import pytest

import kclistpp_gb300 as K
from oracle import oracle as O
from tests import fake_cuda

THREADS = max(1, min(16, O.max_threads()))


def _clique(n):
    i, j = np.triu_indices(n, 1)
    return np.stack([i, j], axis=1).astype(np.uint32)


def test_kernels_launched(tmp_path):
    fake_cuda.run(tmp_path, """
        from tests.test_schedule_bounds import _clique
        def route(n, k, seq, smax, steal=0):
            g = K.build_graph(ctx, K.EdgeList.from_pairs(_clique(n)))
            if steal:
                sp = K.get_schedule(g)
                sp.steal_count = 1
                K.set_schedule(g, sp)
            if smax is not None:
                sp = K.get_schedule(g)
                if seq: sp.tier_s_max_seq = smax
                else: sp.tier_s_max = smax
                K.set_schedule(g, sp)
            was = [fake.fake_launches(x) for x in (b"tier_s_kernel", b"tier_m_kernel")]
            if seq: K.seq_passes(g, k, 1)
            else: K.count_cliques(g, k)
            return [fake.fake_launches(x) - y for x, y in zip((b"tier_s_kernel", b"tier_m_kernel"), was)]
        for k in (3, 4, 5, 6):
            # out-degrees 1..29
            assert route(30, k, True, None) == ([1, 0] if k <= 4 else [1, 1]), k
            for smax, want in ((1, [1, 1]), (8, [1, 1]), (15, [1, 1]), (17, [1, 1]), (29, [1, 0]), (64, [1, 0])):
                assert route(30, k, True, smax) == want, (k, smax)
            # out-degrees 1..59
            assert route(60, k, False, None) == ([1, 1] if k == 5 else [1, 0]), k
            assert route(60, k, False, None, steal=1) == ([1, 0] if k <= 4 else [1, 1]), k
            for smax, want in ((1, [1, 1]), (32, [1, 1]), (58, [1, 1]), (59, [1, 0]), (63, [1, 0])):
                assert route(60, k, False, smax) == want, (k, smax)
        """)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [3, 30, 33, 64])
@pytest.mark.parametrize("smax", [1, 31, 32, 63])
def test_results_at_set_bounds(ctx, n, smax):
    """Small roots on the CTA kernel at k <= 4, roots of 33..63 on the
    warp-per-root counting kernel at k >= 5."""
    pairs = _clique(n)
    og = O.Graph(pairs)
    g = K.build_graph(ctx, K.EdgeList.from_pairs(pairs))
    sp = K.get_schedule(g)
    sp.tier_s_max = sp.tier_s_max_seq = smax
    K.set_schedule(g, sp)
    rng = np.random.default_rng(n)
    for k in (3, 4, 5):
        tot, per = K.count_cliques(g, k)
        otot, oper = og.count_cliques(k)
        assert tot == otot and np.array_equal(per, oper), k
        rho = rng.integers(0, 5, g.n).astype(np.float64)
        assert np.array_equal(K.sim_counts(g, k, rho), og.sim_counts(k, rho, THREADS)), k
        r = rng.integers(0, 50, g.n).astype(np.uint64)
        assert np.array_equal(K.seq_passes(g, k, 1, r), og.seq_pass(k, r, O.SEQ_EDGE_STREAMS, THREADS)), k
    g.close()
