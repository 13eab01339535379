"""A call whose device status word reports an error leaves the caller's host
vectors as they were, at sizes that go through the pinned staging (up to 24576
entries) and beyond.  On the host, with a status word that the test sets (tests/fake_cudart.c)."""
from tests import fake_cuda


def test_vectors_stay_as_they_were(tmp_path):
    fake_cuda.run(tmp_path, """
        L, u64 = K._lib, C.POINTER(C.c_uint64)
        def u(a): return a.ctypes.data_as(u64)
        def d(a): return a.ctypes.data_as(C.POINTER(C.c_double))
        for n in (10, 24575, 24576, 24577, 65000, 100000, 131070, 131071, 200000):
            off = np.concatenate([[0], np.arange(n)]).astype(np.uint64)    # a path
            g = K.graph_from_csr(ctx, off, np.arange(n - 1).astype(np.uint32))
            assert g.n == n
            calls = {
                "count": lambda v: L.kclpp_count_cliques(ctx.handle, g._h, 3, u(v), None),
                "seq": lambda v: L.kclpp_seq_passes(ctx.handle, g._h, 3, 1, K.SEQ_EDGE_STREAMS, u(v)),
                "sim_counts": lambda v: L.kclpp_sim_counts(ctx.handle, g._h, 3, d(np.zeros(n)), u(v)),
                "sim": lambda v: L.kclpp_sim_passes(ctx.handle, g._h, 3, 1, 1, d(v)),
            }
            for name, call in calls.items():
                before = np.full(n, 7.0 if name == "sim" else 7, np.float64 if name == "sim" else np.uint64)
                v = before.copy()
                fake.fake_status_word(1)
                status = call(v)
                fake.fake_status_clear()
                assert status == K.ERR_OVERFLOW, (name, n, status)
                assert np.array_equal(v, before), (name, n)
                assert call(v) == K.OK, (name, n)
            g.close()
        """)
