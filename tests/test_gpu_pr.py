"""GPU PageRank against the FP64 oracle.

Tolerance: max relative error <= 1e-5 against the FP64 Jacobi fixed point of
the current graph (FP32 ranks with Kahan-compensated sums, epsilon 1e-9);
<= 1e-9 in FP64 mode.  With the reference's default --error=1e-6 the result
must pass the reference's own PageRankCheck bound.
"""
import numpy as np
import pytest

import oracle
from coincgraph_b200 import Engine
from coincgraph_b200.engine import FLAG_PR_FP64
from helpers import adversarial_case, big_row_case, rmat_case

pytestmark = pytest.mark.gpu


def max_rel(x, ref):
    return float(np.max(np.abs(x.astype(np.float64) - ref) / np.abs(ref)))


@pytest.mark.parametrize("fp64,eps,tol", [(False, 1e-9, 1e-5), (True, 1e-13, 1e-9)])
@pytest.mark.parametrize("make", [lambda: rmat_case(10, 4, 200, 200, seed_offset=20), adversarial_case,
                                  big_row_case])
def test_pr_stream(make, fp64, eps, tol):
    case = make()
    g = oracle.Graph(case.n, case.xadj, case.adj)
    flags = FLAG_PR_FP64 if fp64 else 0
    with Engine("pr", pr_epsilon=eps, pr_max_rounds=100000, flags=flags) as eng:
        eng.load_csr(case.n, case.xadj, case.adj)
        eng.init()
        x, ok = g.pagerank(1e-15, 100000)
        assert ok
        assert max_rel(eng.pagerank(fp64=fp64)[0], x) <= tol
        for du, dv, au, av in case.batches:
            g.delete(du, dv)
            g.add(au, av)
            s = eng.apply_batch(du, dv, au, av)
            assert s["pr_residual_l1"] <= case.n * eps * 1.01
            x, ok = g.pagerank(1e-15, 100000)
            assert ok
            assert max_rel(eng.pagerank(fp64=fp64)[0], x) <= tol
            xadj, adj = eng.export_csr()
            xo, ao = g.export()
            assert np.array_equal(xadj, xo) and np.array_equal(adj, ao)


def test_pr_reference_check_at_default_error():
    case = rmat_case(10, 3, 100, 100, seed_offset=21)
    g = oracle.Graph(case.n, case.xadj, case.adj)
    ref = oracle.RefStore(case.n, case.xadj, case.adj) if oracle.ref_available() else None
    with Engine("pr", pr_epsilon=1e-6, pr_max_rounds=100) as eng:
        eng.load_csr(case.n, case.xadj, case.adj)
        eng.init()
        for du, dv, au, av in case.batches:
            g.delete(du, dv)
            g.add(au, av)
            if ref is not None:
                ref.apply(du, dv, au, av)
            eng.apply_batch(du, dv, au, av)
            rank, res = eng.pagerank()
            assert g.pr_check(rank, res, 1e-6)["ok"] == 1.0
            if ref is not None:
                assert ref.pr_check(rank, res, 1e-6)


@pytest.mark.parametrize("fp64", [False, True])
@pytest.mark.parametrize("make", [lambda: rmat_case(9, 1, 50, 50, seed_offset=22), big_row_case])
def test_pr_round_bound_keeps_the_pending_queue(make, fp64):
    """A solve cut off by pr_max_rounds leaves every vertex above epsilon
    queued: empty batches then carry it on to the same fixed point (rows on
    both sides of the sweeps' chunk length, and rows over several segments)."""
    case = make()
    g = oracle.Graph(case.n, case.xadj, case.adj)
    du, dv, au, av = case.batches[0]
    g.delete(du, dv)
    g.add(au, av)
    x, ok = g.pagerank(1e-15, 100000)
    assert ok
    with Engine("pr", pr_epsilon=1e-9, pr_max_rounds=3, flags=FLAG_PR_FP64 if fp64 else 0) as eng:
        eng.load_csr(case.n, case.xadj, case.adj)
        eng.init()
        s = eng.apply_batch(du, dv, au, av)
        assert s["pr_rounds"] <= 3 and s["pr_residual_l1"] > case.n * 1e-9
        for _ in range(120):
            s = eng.apply_batch([], [], [], [])
        assert s["pr_residual_l1"] <= case.n * 1e-9 * 1.01
        assert max_rel(eng.pagerank(fp64=fp64)[0], x) <= 1e-6


@pytest.mark.parametrize("fp64", [False, True])
@pytest.mark.parametrize("cap", ["0", "1", "77"])
def test_pr_with_a_full_chunk_list(fp64, cap, monkeypatch):
    """Sweeps over rows of up to 20,000 entries (several segments) when the
    list of their chunks holds none, one, or some of them."""
    monkeypatch.setenv("CIG_CHUNK_CAP", cap)
    case = big_row_case()
    g = oracle.Graph(case.n, case.xadj, case.adj)
    with Engine("pr", pr_epsilon=1e-9, pr_max_rounds=100000, flags=FLAG_PR_FP64 if fp64 else 0) as eng:
        eng.load_csr(case.n, case.xadj, case.adj)
        eng.init()
        for du, dv, au, av in case.batches:
            g.delete(du, dv)
            g.add(au, av)
            s = eng.apply_batch(du, dv, au, av)
        assert s["pr_residual_l1"] <= case.n * 1e-9 * 1.01
        x, ok = g.pagerank(1e-15, 100000)
        assert ok and max_rel(eng.pagerank(fp64=fp64)[0], x) <= (1e-6 if fp64 else 1e-5)


@pytest.mark.parametrize("fp64", [False, True])
def test_pr_error_of_sweeps(fp64):
    """The ranks' error against 64 bits after a static solve by sweeps and
    after a batch.  FP64, epsilon 1e-9: what the sweeps leave, residuals of
    either sign up to 0.7 epsilon, makes 1.8e-9 (relative 2-norm; with epsilon
    itself as their threshold 2.5e-9, by queue rounds 2.2e-9 to 2.6e-9).  FP32:
    one rounding of the result, 2^-24, and that remainder, at most 0.7e-9 / 0.15
    on ranks of at least 0.15 (summed up in FP32 alone: 2e-7 to 4e-7)."""
    case = rmat_case(13, 1, 200, 200, seed_offset=23)
    g = oracle.Graph(case.n, case.xadj, case.adj)
    with Engine("pr", pr_epsilon=1e-9, pr_max_rounds=100000, flags=FLAG_PR_FP64 if fp64 else 0) as eng:
        eng.load_csr(case.n, case.xadj, case.adj)
        eng.init()
        for batch in [None, *case.batches]:
            if batch is not None:
                g.delete(*batch[:2])
                g.add(*batch[2:])
                eng.apply_batch(*batch)
            x, ok = g.pagerank(1e-15, 100000)
            assert ok
            rank = eng.pagerank(fp64=fp64)[0].astype(np.float64)
            if fp64:
                assert np.linalg.norm(rank - x) <= 2.1e-9 * np.linalg.norm(x)
            else:
                assert max_rel(rank, x) <= 2.0**-24 + 0.7e-9 / 0.15 / 0.15
