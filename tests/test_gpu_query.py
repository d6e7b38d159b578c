"""Multi-source BFS / SSSP queries (bitmask waves) against the CPU oracle.

Each row of a query result must equal the oracle's from-scratch FIFO
recompute for that source (the restated hybrid_sssp_host.cu:34-63 check with
the samples' weights), exactly, on the graph as it stands after update
batches; the batched (64-wide) and per-source (width 1) forms must agree.
"""
import numpy as np
import pytest

import oracle
from coincgraph_b200 import Engine, gen

from helpers import big_row_case, grid_case, rmat_case

pytestmark = pytest.mark.gpu

MODES = {"bfs": oracle.BFS, "sssp": oracle.SSSP}


def _sources(g, k, seed=7):
    rng = np.random.default_rng(seed)
    deg = np.diff(g.xadj.astype(np.int64))
    live = np.flatnonzero(deg > 0)
    hub = int(np.argmax(deg))
    picks = rng.choice(live, size=k - 3, replace=True)
    return np.concatenate([[0, hub, hub], picks]).astype(np.uint32)  # a repeated source too


@pytest.mark.parametrize("algo", ["bfs", "sssp"])
@pytest.mark.parametrize("k", [1, 5, 64, 70])
def test_query_matches_oracle(built, algo, k):
    g = gen.rmat(11)
    src = _sources(g, max(k, 4))[:k]
    og = oracle.Graph(g.n, g.xadj, g.adj)
    with Engine(algo, cache_gib=4.0) as eng:
        eng.load_csr(g.n, g.xadj, g.adj)
        eng.init()
        got = eng.query_bfs(src) if algo == "bfs" else eng.query_sssp(src)
    assert got.shape == (k, g.n)
    for j, s in enumerate(src):
        np.testing.assert_array_equal(got[j], og.sssp(int(s), MODES[algo]), err_msg=f"source {s}")


@pytest.mark.parametrize("cache_gib", [0.0, 0.002])
def test_query_after_updates_zero_copy_and_mixed(built, cache_gib):
    case = rmat_case(12, batches=2, dels=300, adds=300)
    og = oracle.Graph(case.n, case.xadj, case.adj)
    with Engine("sssp", cache_gib=cache_gib) as eng:
        eng.load_csr(case.n, case.xadj, case.adj)
        eng.init()
        for du, dv, au, av in case.batches:
            eng.apply_batch(du, dv, au, av)
            og.delete(du, dv)
            og.add(au, av)
        src = _sources(gen.Graph(case.n, *og.export()), 40)
        bfs = eng.query_bfs(src)
        sssp = eng.query_sssp(src)
        # Queries leave the maintained state alone.
        np.testing.assert_array_equal(eng.values(), og.sssp(0, oracle.SSSP))
    for j, s in enumerate(src):
        np.testing.assert_array_equal(bfs[j], og.sssp(int(s), oracle.BFS))
        np.testing.assert_array_equal(sssp[j], og.sssp(int(s), oracle.SSSP))


def test_query_hub_rows_and_width_forms(built):
    """Rows past the hub-split threshold (deferred grid-wide expansion) and the
    device-output form at widths 64 and 1 give the same distances."""
    import torch

    case = big_row_case()
    og = oracle.Graph(case.n, case.xadj, case.adj)
    src = np.arange(0, min(case.n, 48), dtype=np.uint32)
    with Engine("bfs", cache_gib=1.0) as eng:
        eng.load_csr(case.n, case.xadj, case.adj)
        eng.init()
        outs = {}
        for width in (64, 1):
            out = torch.empty((len(src), case.n), dtype=torch.int32, device="cuda")
            st = eng.query_device("sssp", src, out, width=width)
            assert st["waves"] == -(-len(src) // width)
            assert st["edges_scanned"] > 0 and st["source_edges"] >= st["edges_scanned"]
            outs[width] = out.cpu().numpy().view(np.uint32)
    np.testing.assert_array_equal(outs[64], outs[1])
    for j, s in enumerate(src):
        np.testing.assert_array_equal(outs[64][j], og.sssp(int(s), oracle.SSSP))


def test_query_sssp_uniform_255_weights(built):
    from coincgraph_b200.engine import FLAG_WEIGHT_U255

    g = gen.rmat(11)
    src = _sources(g, 20)
    og = oracle.Graph(g.n, g.xadj, g.adj)
    with Engine("sssp", cache_gib=1.0, flags=FLAG_WEIGHT_U255) as eng:
        eng.load_csr(g.n, g.xadj, g.adj)
        eng.init()
        got = eng.query_sssp(src)
        np.testing.assert_array_equal(eng.values(), og.sssp(0, oracle.SSSP_U255))
    for j, s in enumerate(src):
        np.testing.assert_array_equal(got[j], og.sssp(int(s), oracle.SSSP_U255))


def test_query_rejects_bad_arguments(built):
    from coincgraph_b200 import CigError

    g = gen.rmat(8)
    with Engine("bfs") as eng:
        eng.load_csr(g.n, g.xadj, g.adj)
        eng.init()
        with pytest.raises(CigError):
            eng.query_bfs(np.array([g.n], dtype=np.uint32))
        # The handle stays usable after a rejected call.
        np.testing.assert_array_equal(eng.query_bfs([0])[0], eng.values())


@pytest.mark.parametrize("pull", ["0", "32", "1000000"])  # never, default, as soon as two vertices are reached
@pytest.mark.parametrize("make", [big_row_case, lambda: grid_case(33, 1, 40), lambda: rmat_case(10, 1, 50, 50)])
def test_bfs_direction_and_depth_planes(built, make, pull, monkeypatch):
    """Bottom-up and top-down rounds in every mix, in-rows on both sides of the
    lane, warp and chunk limits, depths past the planes cleared at launch
    (grid), a tail of the last bitmap word; waves of 1, 2 and 64 sources."""
    monkeypatch.setenv("CIG_PULL_ON", pull)
    monkeypatch.setenv("CIG_PULL_OFF", "2000000" if pull == "1000000" else "64")
    case = make()
    og = oracle.Graph(case.n, case.xadj, case.adj)
    rng = np.random.default_rng(5)
    src = np.concatenate([[0, case.n - 1], rng.integers(0, case.n, 62)]).astype(np.uint32)
    ref = np.stack([og.sssp(int(s), oracle.BFS) for s in src])
    with Engine("bfs", cache_gib=1.0) as eng:
        eng.load_csr(case.n, case.xadj, case.adj)
        eng.init()
        for k in (64, 2, 1, 63):  # buffers of a wave are reused by the next
            np.testing.assert_array_equal(eng.query_bfs(src[:k]), ref[:k])


@pytest.mark.parametrize("k", [1, 2, 4, 5, 8, 9, 16, 17, 32, 33, 64])
def test_sssp_wave_widths(built, k):
    """Waves on both sides of every padded row width, rows on both sides of the
    chunk length, host-resident and cached."""
    case = big_row_case()
    og = oracle.Graph(case.n, case.xadj, case.adj)
    src = np.arange(k, dtype=np.uint32)
    with Engine("sssp", cache_gib=65536 / 2**30) as eng:
        eng.load_csr(case.n, case.xadj, case.adj)
        eng.init()
        got = eng.query_sssp(src)
    for j in range(k):
        np.testing.assert_array_equal(got[j], og.sssp(j, oracle.SSSP))


def test_bfs_wave_on_used_device_memory(built):
    """Long in-rows gathered by several warps, in buffers of a new handle that
    the memory of this process's earlier allocations serves (all bits set):
    the waves clear what they count in."""
    import torch

    case = big_row_case()  # vertex 5 has 6,000 in-edges: six chunks
    og = oracle.Graph(case.n, case.xadj, case.adj)
    src = np.concatenate([[0, 1], np.arange(7000, 7062)]).astype(np.uint32)  # 5 is two steps from 1
    ref = np.stack([og.sssp(int(s), oracle.BFS) for s in src])
    for _ in range(2):
        used = [torch.full((size // 4,), -1, dtype=torch.int32, device="cuda")
                for size in (4096, 1 << 16, 1 << 20, 1 << 24, 1 << 28) for _ in range(16)]
        torch.cuda.synchronize()
        del used
        torch.cuda.empty_cache()
        with Engine("bfs", cache_gib=1.0) as eng:
            eng.load_csr(case.n, case.xadj, case.adj)
            eng.init()
            for k in (64, 5, 64):
                np.testing.assert_array_equal(eng.query_bfs(src[:k]), ref[:k])


@pytest.mark.parametrize("k", [1, 2, 16, 17])
def test_bfs_switches_on_the_queued_rows(built, k):
    """Two steps from the sources lie 300 rows of 200 entries, a queue far
    below n / 32 vertices whose rows hold more than n entries: the round goes
    bottom-up by the lengths added up while the vertices were queued (short
    rows are not counted), on both sides of the blocks-per-SM rule.  Beside it
    a chain of 600 vertices, so that the wave ends in several hundred queue
    rounds below the limit."""
    rng = np.random.default_rng(9)
    n = 50000
    mid = np.arange(100, 400)
    chain = np.arange(1000, 1600)
    src = np.concatenate([np.repeat(np.arange(20), 300), np.repeat(mid, 200), chain[:-1], np.arange(20)])
    dst = np.concatenate([np.tile(mid, 20), rng.integers(2000, n, 300 * 200), chain[1:], np.full(20, 1000)])
    g = gen.graph_from_edges(n, src, dst)
    sources = np.arange(k, dtype=np.uint32)
    og = oracle.Graph(g.n, g.xadj, g.adj)
    import torch

    with Engine("bfs", cache_gib=1.0) as eng:
        eng.load_csr(g.n, g.xadj, g.adj)
        eng.init()
        out = torch.empty((k, n), dtype=torch.int32, device="cuda")
        st = eng.query_device("bfs", sources, out, width=64)
        got = out.cpu().numpy().view(np.uint32)
    for j, s in enumerate(sources):
        np.testing.assert_array_equal(got[j], og.sssp(int(s), oracle.BFS))
    # Top-down rounds expand the sources, the 300 rows and the chain; a
    # bottom-up round looks through the in-row of every unreached vertex.
    assert st["rows_expanded"] > 10000


@pytest.mark.parametrize("k", [4, 8, 16, 17, 32, 33, 64])
@pytest.mark.parametrize("spread", [True, False])
def test_sssp_waves_of_sparse_and_dense_masks(built, k, spread):
    """A grid, where sources far apart leave a vertex one or two bits of the
    wave (their 16-byte pieces are dealt out), and neighbouring sources leave
    it all of them; queue rounds, scan rounds and the changes between them."""
    case = grid_case(70, 1, 20)
    rng = np.random.default_rng(k)
    src = (rng.integers(0, case.n, k) if spread else 2000 + np.arange(k) // 4).astype(np.uint32)
    og = oracle.Graph(case.n, case.xadj, case.adj)
    with Engine("sssp", cache_gib=1.0) as eng:
        eng.load_csr(case.n, case.xadj, case.adj)
        eng.init()
        got = eng.query_sssp(src)
    for j, s in enumerate(src):
        np.testing.assert_array_equal(got[j], og.sssp(int(s), oracle.SSSP))


@pytest.mark.parametrize("cap", ["0", "1", "77"])
@pytest.mark.parametrize("k", [3, 13, 64])
def test_sssp_waves_with_a_full_chunk_list(built, k, cap, monkeypatch):
    """Rows of up to 20,000 entries when the list of their chunks holds none,
    one, or some of them: the rest is relaxed by the warps that met it."""
    monkeypatch.setenv("CIG_CHUNK_CAP", cap)
    case = big_row_case()
    og = oracle.Graph(case.n, case.xadj, case.adj)
    src = np.concatenate([[0, 1], np.arange(7000, 7000 + k - 2)]).astype(np.uint32)
    with Engine("sssp", cache_gib=65536 / 2**30) as eng:
        eng.load_csr(case.n, case.xadj, case.adj)
        eng.init()
        got = eng.query_sssp(src)
    for j, s in enumerate(src):
        np.testing.assert_array_equal(got[j], og.sssp(int(s), oracle.SSSP))


def test_autotune_leaves_wide_waves_alone(built):
    """The autotuner times one-source queries; a wave of 64 takes the same
    rounds in the same directions after it as before."""
    import torch

    case = grid_case(64, 1, 20)
    src = np.random.default_rng(2).integers(0, case.n, 64).astype(np.uint32)
    out = torch.empty((64, case.n), dtype=torch.int32, device="cuda")
    with Engine("bfs", cache_gib=1.0) as eng:
        eng.load_csr(case.n, case.xadj, case.adj)
        eng.init()
        before = eng.query_device("bfs", src, out, width=64)
        for _ in range(3):
            eng.autotune()
            after = eng.query_device("bfs", src, out, width=64)
            for key in ("rounds", "edges_scanned", "rows_expanded"):
                assert after[key] == before[key], key


@pytest.mark.parametrize("last", [14, 15, 16, 17, 40])
@pytest.mark.parametrize("pull", ["0", "1000000"])
def test_bfs_depths_beside_the_plane_limit(built, last, pull, monkeypatch):
    """Chains whose deepest level lies on either side of 16, where depths go
    from the planes to the result directly, top-down and bottom-up; the four
    vertices of a 16-byte store hold planes', direct and unreached entries."""
    monkeypatch.setenv("CIG_PULL_ON", pull)
    monkeypatch.setenv("CIG_PULL_OFF", "2000000")
    for n in (64, 65):
        chain = np.arange(last + 1)
        ends = np.arange(last + 1, n - 4)  # one step behind the chain's middle and end, in turn
        src = np.concatenate([chain[:-1], np.where(ends % 2, last, last // 2)])
        g = gen.graph_from_edges(n, src, np.concatenate([chain[1:], ends]))
        og = oracle.Graph(g.n, g.xadj, g.adj)
        sources = np.array([0, 3, n - 1], dtype=np.uint32)
        with Engine("bfs", cache_gib=1.0) as eng:
            eng.load_csr(g.n, g.xadj, g.adj)
            eng.init()
            got = eng.query_bfs(sources)
        for j, s in enumerate(sources):
            np.testing.assert_array_equal(got[j], og.sssp(int(s), oracle.BFS))
