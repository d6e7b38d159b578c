"""Device memory accounting (cig_memory_info_get) and the position-index
budget (cig_options.index_budget_gib): the reported parts add up to the
device memory the handle actually took, the index tables stay inside the
budget, and results stay exact against the oracle when the budget leaves
most rows unindexed."""
import numpy as np
import pytest

from coincgraph_b200 import Engine
from helpers import oracle_trace, rmat_case

pytestmark = pytest.mark.gpu


def test_memory_parts_match_the_device():
    import torch

    case = rmat_case(14, 2, 500, 500, seed_offset=70)
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    with Engine("sssp", cache_gib=0.01, max_batch=500) as eng:
        eng.load_csr(case.n, case.xadj, case.adj)
        eng.init()
        for b in case.batches:
            eng.apply_batch(*b)
        m = eng.memory()
        used = free0 - torch.cuda.mem_get_info()[0]
    parts = sum(v for k, v in m.items() if k not in ("total", "pinned_host"))
    assert parts == m["total"]
    for k in ("edge_cache", "descriptors", "reverse_arena", "vertex_state", "batch_buffers"):
        assert m[k] > 0, k
    assert m["pinned_host"] > 0
    # cudaMalloc rounds every allocation up to its granule, and the CUDA
    # graphs and events hold some device memory of their own
    assert m["total"] <= used <= m["total"] + (256 << 20), (m["total"], used)


def test_index_budget_bounds_the_tables_and_keeps_results():
    case = rmat_case(13, 3, 400, 400, seed_offset=71)
    trace, _ = oracle_trace(case, "bfs")
    sizes = {}
    for budget in (0.0, 1.0 / 1024):  # default, then 1 MiB for both tables
        with Engine("bfs", cache_gib=4.0, index_budget_gib=budget) as eng:
            eng.load_csr(case.n, case.xadj, case.adj)
            eng.init()
            for i, b in enumerate(case.batches):
                eng.apply_batch(*b)
                assert np.array_equal(eng.values(), trace["batch"][i]), f"budget {budget}: batch {i}"
                xadj, adj = eng.export_csr()
                assert np.array_equal(adj, trace["rows"][i][1])
            sizes[budget] = eng.memory()["position_index"]
    assert sizes[1.0 / 1024] <= (1 << 20)
    assert sizes[0.0] > sizes[1.0 / 1024]


def test_query_buffers_follow_the_vertices_not_the_arena():
    """Query buffers of a graph whose rows take far more memory than its
    vertices: the lists of row chunks stay below 24 MiB (or 6 bytes per
    vertex), are made by the first wave that uses them, and the memory
    report follows."""
    import torch

    rng = np.random.default_rng(5)
    n = 4096
    deg = 16384  # 256 MiB of rows, over a million chunks of 64 entries, on 4,096 vertices
    xadj = np.arange(n + 1, dtype=np.uint64) * deg
    adj = rng.integers(0, n, n * deg, dtype=np.uint32)
    base = n * (64 * 4 + 3 * 8) + 2 * (n + 1) * 4 + 65536 * 24 + 8192
    with Engine("sssp", cache_gib=1.0) as eng:
        eng.load_csr(n, xadj, adj)
        eng.init()
        assert eng.memory()["query_buffers"] == 0
        eng.query_bfs([1])
        assert eng.memory()["query_buffers"] <= base
        bfs = eng.query_bfs([1, 2, 3])
        waves = eng.memory()["query_buffers"]
        slots = eng.memory()["reverse_arena"] // 4
        assert waves <= base + slots // 1024 * 36 + n // 8 + 8
        free0 = torch.cuda.mem_get_info()[0]
        sssp = eng.query_sssp([1, 2, 3])
        grown = eng.memory()["query_buffers"] - waves
        assert 0 < grown <= 24 << 20
        # the report against the device (3 n result words beside; 2 MiB granules)
        assert free0 - torch.cuda.mem_get_info()[0] <= grown + (8 << 20)
        assert (bfs != 0xFFFFFFFF).all() and (sssp <= 128 * bfs).all() and (sssp >= bfs).all()


def test_queries_answer_after_a_failed_allocation():
    """A query without device memory for its buffers (or its result) fails
    with the out-of-memory error and takes nothing; once there is memory, the
    same handle answers."""
    import torch

    import oracle
    from coincgraph_b200 import CigError, gen

    rng = np.random.default_rng(6)
    n = 1 << 20  # 256 bytes of query buffers per vertex
    g = gen.graph_from_edges(n, rng.integers(0, 2000, 200000), rng.integers(0, 2000, 200000))
    ref = oracle.Graph(g.n, g.xadj, g.adj).sssp(5, oracle.BFS)

    def fails(eng, leave):
        torch.cuda.empty_cache()
        hog = torch.empty(torch.cuda.mem_get_info()[0] - leave, dtype=torch.uint8, device="cuda")
        with pytest.raises(CigError) as err:
            eng.query_bfs(np.arange(64))
        assert err.value.code == -2, err.value  # CIG_ERR_NOMEM
        del hog
        torch.cuda.empty_cache()

    # 256 MiB for 64 results, then 300 MiB of buffers: the first, then the
    # second does not fit.
    for leave in (64 << 20, 400 << 20):
        with Engine("bfs", cache_gib=1.0) as eng:
            eng.load_csr(g.n, g.xadj, g.adj)
            eng.init()
            fails(eng, leave)
            assert eng.memory()["query_buffers"] == 0
            np.testing.assert_array_equal(eng.query_bfs([5])[0], ref)
            fails(eng, 64 << 20)  # the result buffer cannot grow
            np.testing.assert_array_equal(eng.query_bfs([5])[0], ref)
            np.testing.assert_array_equal(eng.query_bfs(np.full(64, 5))[63], ref)
