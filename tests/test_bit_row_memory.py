"""A graph whose bitmap rows the device has no room for: it is accepted, and
counted by walking the out-lists (whole numbers: no tolerance).  The rows'
allocations are refused by limit_cudart.c; the device is not filled."""
import pytest

from tests import fake_cuda

SCRIPT = """
from oracle import oracle as O
for el in (K.planted(3000, 6.0, 2.2, 1, 260, 260, 0.5, seed=5), K.chung_lu(3000, 16.0, 2.3, seed=3)):
    og = O.Graph(el.pairs())
    g = K.build_graph(ctx, el)
    off, cols = g.csr()
    g.close()
    d = np.diff(off.astype(np.int64))
    some = d > 1
    span = (cols[off[1:][some].astype(np.int64) - 1] - cols[off[:-1][some].astype(np.int64)]) // 32 + 1
    words = int(span[span <= 2 * d[some]].sum())
    size = 16 * (len(off) - 1) if "{refused}" == "index" else 4 * words
    assert words > 0
    was = limit.limit_refused()
    limit.limit_exact(size, 0)
    g = K.build_graph(ctx, el)
    limit.limit_off()
    assert limit.limit_refused() == was + 1
    for k in (3, 4, 5):
        assert K.count_cliques(g, k)[0] == og.count_cliques(k)[0]
        r = og.seq_pass(k, np.zeros(og.n, np.uint64))
        assert np.array_equal(K.seq_passes(g, k, 1), r)
    g.close()
"""


@pytest.mark.gpu
@pytest.mark.parametrize("refused", ["index", "rows"])
def test_graph_without_room_for_bitmap_rows(tmp_path, refused):
    fake_cuda.run_limited(tmp_path, SCRIPT.replace("{refused}", refused))
