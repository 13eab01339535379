"""The autotuner times the launches that a pass makes, by the root group whose
width they take.  On the host, with a clock on which a test decides what a launch
costs (tests/fake_cudart.c)."""
from tests import fake_cuda

SETUP = """
def clique(n):
    i, j = np.triu_indices(n, 1)
    return np.stack([i, j], axis=1)
def tuned(pairs, k, kernel, cost):
    g = K.build_graph(ctx, K.EdgeList.from_pairs(pairs.astype(np.uint32)))
    fn = COST(cost)
    fake.fake_cost(fn)
    best = K.autotune(g, k, kernel).best
    fake.fake_cost(COST(0))
    return best
"""


def test_a_group_without_a_launch_keeps_its_width(tmp_path):
    """Seq, k = 4, out-degrees up to 29: every root goes to the warp kernel.  The
    tier bounds all cost the same; every launch after them costs less, so that
    any width found in between is kept."""
    fake_cuda.run(tmp_path, SETUP + """
best = tuned(clique(30), 4, K.KERNEL_SEQ, lambda name, blocks, threads, n: 1.0 if n < 233 else 0.5)
assert best.tier_s_max_seq == 16 and list(best.seq_warps) == [0, 0, 0, 0], best.as_dict()
""")


def test_a_group_split_from_tier_s_is_tuned(tmp_path):
    """Counting, k = 5, out-degrees up to 59: roots above 32 are a CTA launch with
    the first group's width, quickest at 16 warps."""
    fake_cuda.run(tmp_path, SETUP + """
def cost(name, blocks, threads, n):
    return abs(threads - 512) + 1.0 if b"tier_m_kernel" in name else 1.0
best = tuned(clique(60), 5, K.KERNEL_ORDER, cost)
assert best.count_warps[0] == 16 and list(best.count_warps[1:]) == [0, 0, 0], list(best.count_warps)
""")


def test_launches_that_share_a_width_are_summed(tmp_path):
    """Counting, k = 5: 59 roots of 33..64 and 56 of 65..120 are two launches of
    one width, the first quickest at 8 warps by less than the second is at 24."""
    fake_cuda.run(tmp_path, SETUP + """
def cost(name, blocks, threads, n):
    w = threads // 32
    if b"tier_m_kernel" not in name: return 1.0
    return {59: 5.0 + 0.25 * abs(w - 8), 56: 10.0 + abs(w - 24)}.get(blocks, 100.0)
best = tuned(np.concatenate([clique(60), 60 + clique(121)]), 5, K.KERNEL_ORDER, cost)
assert best.count_warps[0] == 24, best.as_dict()
""")
