"""What a batch's concurrent branches hold of their own, and when its captured
CUDA graph may be replayed.

A batch replays the CUDA graph it captured only while the union graph's
schedule is the very one it was captured with: building a schedule again, even
an equal one, frees the root array that the captured launches read.

Every slice must equal the single-graph run bit for bit: no tolerance."""
import numpy as np
import pytest

import kclistpp_gb300 as K
from tests import fake_cuda


def _graphs():
    return [K.chung_lu(3000, 14.0, 2.4, seed=61), K.planted(3000, 6.0, 2.2, 1, 220, 220, 0.5, seed=62)]


def _check(ctx, out, els, b, ks, passes):
    for gi, el in enumerate(els):
        g = K.build_graph(ctx, el)
        for ki, k in enumerate(ks):
            assert np.array_equal(out[ki, b.slice(gi)], K.seq_passes(g, k, passes)), (gi, k)
        g.close()


def test_captures_counted_on_the_host(tmp_path):
    fake_cuda.run(tmp_path, """
        b = K.Batch(ctx, [K.chung_lu(500, 10.0, 2.4, seed=1), K.planted(500, 6.0, 2.2, 1, 90, 90, 0.5, seed=2)])
        u = b.union_graph()
        first, other = K.get_schedule(u), K.get_schedule(u)
        other.tier_s_max_seq = 8
        def captures(act=None):
            if act: act()
            n = fake.fake_instantiations()
            b.run(K.KERNEL_SEQ, [3, 5], 2)
            return fake.fake_instantiations() - n
        def twice():
            K.set_schedule(u, other)
            K.set_schedule(u, first)
        assert captures() == 1
        assert captures() == 0                              # replayed
        assert captures(lambda: K.set_schedule(u, first)) == 1
        assert captures(twice) == 1
        assert captures() == 0
        assert captures(lambda: K.autotune(u, 4)) == 1      # whichever schedule it ends at
        K.graph_shard(u, 0, 2)
        try:
            b.run(K.KERNEL_SEQ, [3, 5], 2)
            raise SystemExit("a sharded union graph ran")
        except K.KclppError as e:
            assert e.status == K.ERR_INVALID
        assert captures(lambda: K.graph_shard(u, 0, 1)) == 1
        """)


@pytest.mark.gpu
def test_equal_schedule_again_captures_again(ctx):
    els, ks = _graphs(), [3, 5]
    b = K.Batch(ctx, els)
    _check(ctx, b.run(K.KERNEL_SEQ, ks, 2), els, b, ks, 2)
    u = b.union_graph()
    first = K.get_schedule(u)
    other = K.get_schedule(u)
    other.tier_s_max_seq, other.seq_split1 = 8, 128
    launches = []
    for sp in (first, other, first):
        K.set_schedule(u, sp)
        # graphs made here may be given the memory of the schedule that was freed
        hold = [K.build_graph(ctx, el) for el in els]
        before = ctx.launches()
        out = b.run(K.KERNEL_SEQ, ks, 2)
        launches.append(ctx.launches() - before)
        _check(ctx, out, els, b, ks, 2)
        for g in hold:
            g.close()
    assert min(launches) > 1  # one launch would be a replay
    b.close()


def _deep():
    """Roots of out-degree 1100 (rows in global memory), few cliques: two halves
    joined completely, a sparse graph inside each."""
    a, rng = 1100, np.random.default_rng(4)
    parts = [np.stack(np.meshgrid(np.arange(a), np.arange(a, 2 * a), indexing="ij"), -1).reshape(-1, 2)]
    for base in (0, a):
        i, j = np.triu_indices(a, 1)
        keep = rng.random(len(i)) < 2.0 / a
        parts.append(np.stack([base + i[keep], base + j[keep]], axis=1))
    return K.EdgeList.from_pairs(np.concatenate(parts).astype(np.uint32))


def test_each_branch_has_its_rows_in_global_memory(tmp_path):
    fake_cuda.run(tmp_path, """
        from tests.test_batch_capture import _deep
        b = K.Batch(ctx, [_deep()])
        slab = 152 * 2048 * 64 * 4
        before = fake.fake_allocations(slab)
        b.run(K.KERNEL_SEQ, [3, 4, 5], 1)
        assert fake.fake_allocations(slab) - before == 3
        """)


@pytest.mark.gpu
@pytest.mark.parametrize("kernel", [K.KERNEL_SEQ, K.KERNEL_ORDER])
def test_branches_over_deep_roots_equal_single_runs(ctx, kernel):
    el, ks = _deep(), [3, 4, 5]
    b = K.Batch(ctx, [el, K.chung_lu(2000, 12.0, 2.4, seed=63)])
    g = K.build_graph(ctx, el)
    assert g.core > 1024
    for _ in range(3):
        out = b.run(kernel, ks, 2)
        for ki, k in enumerate(ks):
            want = K.seq_passes(g, k, 2) if kernel == K.KERNEL_SEQ else K.sim_passes(g, k, 2)
            assert np.array_equal(out[ki, b.slice(0)].view(np.uint64), want.view(np.uint64)), k
    b.close()


@pytest.mark.gpu
def test_replay_while_nothing_changed(ctx):
    b = K.Batch(ctx, _graphs())
    first = b.run(K.KERNEL_SEQ, [4], 2)
    before = ctx.launches()
    assert np.array_equal(b.run(K.KERNEL_SEQ, [4], 2), first)
    assert ctx.launches() - before == 1
    b.close()


@pytest.mark.gpu
def test_a_sharded_union_is_refused(ctx):
    els, ks = _graphs(), [4]
    b = K.Batch(ctx, els)
    b.run(K.KERNEL_SEQ, ks, 1)
    K.graph_shard(b.union_graph(), 0, 2)
    with pytest.raises(K.KclppError) as e:
        b.run(K.KERNEL_SEQ, ks, 1)
    assert e.value.status == K.ERR_INVALID
    K.graph_shard(b.union_graph(), 0, 1)
    _check(ctx, b.run(K.KERNEL_SEQ, ks, 1), els, b, ks, 1)
    b.close()
