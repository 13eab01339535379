"""A sample that the device holds once but not twice: the rows are drawn again
in place, each at its wave's cursor, and the sample and its passes are those of
the oracle (whole numbers: no tolerance).  The second copy is refused by
limit_cudart.c; the device is not filled."""
import pytest

from tests import fake_cuda

SCRIPT = """
from oracle import oracle as O
from tests.test_sampling_host import bipartite_with_clique, sort_rows
for a, k, most in ((120, 4, {refused}), (1100, 3, {refused})):   # rows in shared memory; a root group in a slab too
    pairs = bipartite_with_clique(a, a, 14)
    og = O.Graph(pairs)
    total = og.count_cliques(k)[0]
    g = K.build_graph(ctx, K.EdgeList.from_pairs(pairs))
    for target in (total + 1, max(total // 3, 1)):
        all_, _, thr = O.sampling_threshold(target, total)
        want = sort_rows(*og.sampling_collect(k, 11, thr, all_, 8))
        size = len(want[0]) * (4 * k if most == "rows" else 1)
        was = limit.limit_refused()
        # the first draw's buffers are the copy's size when every clique is kept, else larger
        limit.limit_exact(size, 1 if target > total else 0)
        s = K.Sampling(g, k, target, 11, 8)
        limit.limit_off()
        assert limit.limit_refused() == was + 1
        rows, wave = s.cliques()
        assert np.array_equal(rows, want[0]) and np.array_equal(wave, want[1])
        s.passes(3)
        rho = np.zeros(og.n, np.uint32)
        for _ in range(3):
            rho = O.sampling_pass(og.n, k, want[0], want[1], 8, rho)
        assert np.array_equal(s.rho(), rho)
        s.close()
    g.close()
"""


@pytest.mark.gpu
@pytest.mark.parametrize("refused", ["rows", "waves"])
def test_sample_without_room_for_a_copy(tmp_path, refused):
    fake_cuda.run_limited(tmp_path, SCRIPT.replace("{refused}", repr(refused)))
