"""GPU tests of the request pool: concurrent Solve_Native calls on several
streams give exactly the results of tf_solve on the same inputs (the pool
runs the same deterministic drop-in), under a device-memory budget."""
import copy
import threading

import numpy as np
import pytest

from tflows_b200 import grids, native, pool, systems

pytestmark = pytest.mark.gpu


def _systems():
    return [systems.small_hex(12, seed=1, kind="pressure", ratio=1.02),
            systems.small_hex(24, seed=2, kind="pressure", ratio=1.02),
            systems.small_hex(10, seed=3, kind="momentum", peclet=1.0),
            systems.poly_system(2000, seed=4, kind="pressure"),
            systems.small_hex(8, seed=5, kind="pressure", tol=1e-9, miter=300, prec="icc")]


def _reference(ctx, s):
    m = native.Matrix(ctx, s.csr.row, s.csr.col, s.csr.dia)
    try:
        v, x, b = s.val.copy(), s.x0.copy(), s.b.copy()
        it, res = native.solve(ctx, m, s.solver, s.prec, v, x, b, s.miter, s.tol, s.norm)
        return x, it, res
    finally:
        m.close()


def test_pool_matches_single_solves(gpu_ctx, solve_path):
    sysl = _systems()
    ref = [_reference(gpu_ctx, s) for s in sysl]
    p = pool.Pool(workers=4, mem_budget=1 << 30)
    try:
        rids = {}

        def submitter(offset):
            for k in range(offset, 3 * len(sysl), 2):
                rids[k] = p.submit(sysl[k % len(sysl)])

        th = [threading.Thread(target=submitter, args=(o,)) for o in (0, 1)]
        for t in th:
            t.start()
        for t in th:
            t.join()
        for k in sorted(rids):
            r = p.wait(rids[k])
            x, it, res = ref[k % len(sysl)]
            assert r["niter"] == it and r["fin_res"] == res
            assert np.array_equal(r["x"], x)
            assert r["latency_ms"] >= r["queue_ms"] >= 0.0
        st = p.stats()
        assert st["completed"] == 3 * len(sysl) and st["rejected"] == 0
        assert 0 < st["peak_bytes"] <= 1 << 30
    finally:
        p.close()


def test_pool_budget(gpu_ctx):
    small = systems.small_hex(6, seed=1, kind="pressure")
    big = systems.small_hex(40, seed=1, kind="pressure")
    p = pool.Pool(workers=2, mem_budget=4 << 20)
    try:
        r_big = p.submit(big)
        r_small = p.submit(small)
        with pytest.raises(native.TFError) as e:
            p.wait(r_big)
        assert e.value.status == 2          # TF_ERR_OOM: larger than the budget
        assert p.wait(r_small)["niter"] > 0
        assert p.stats()["rejected"] == 1
    finally:
        p.close()


def test_pool_reuses_resident_structures(gpu_ctx, solve_path):
    """Requests on the same Matrix_Type arrays run on the held registration
    (no re-registration) and give the single-solve results every time, also
    with fresh right-hand sides, whichever worker's stream its kernel or its
    graph runs on."""
    s = systems.small_hex(20, seed=7, kind="pressure", ratio=1.03)
    rhs = [systems.uniform_rhs(s.n, 100 + k, zero_mean=True) for k in range(6)]
    refs = []
    for b in rhs:
        t = copy.copy(s)
        t.b = b
        refs.append(_reference(gpu_ctx, t))
    p = pool.Pool(workers=2, mem_budget=1 << 30)
    try:
        for rounds in range(2):
            rids = [p.submit(s, b=b) for b in rhs]
            for rid, (x, it, res) in zip(rids, refs):
                r = p.wait(rid)
                assert r["niter"] == it and r["fin_res"] == res
                assert np.array_equal(r["x"], x)
        res_info = p.resident()
        assert res_info["held"] >= 1 and res_info["reused"] >= 2 * len(rhs) - 2
        assert res_info["held_bytes"] <= 1 << 30
    finally:
        p.close()


def test_pool_releases_held_structures_for_new_requests(gpu_ctx):
    """Held registrations give way (least recently used first) when a new
    request needs the budget."""
    sysl = [systems.small_hex(16 + k, seed=k, kind="pressure") for k in range(4)]
    refs = [_reference(gpu_ctx, s) for s in sysl]
    # room for about two of these systems at a time
    probe = pool.Pool(workers=1, mem_budget=1 << 30)
    try:
        probe.wait(probe.submit(sysl[-1]))
        one = probe.stats()["peak_bytes"]
    finally:
        probe.close()
    budget = int(2.5 * one)
    p = pool.Pool(workers=1, mem_budget=budget)
    try:
        for rounds in range(2):
            for s, (x, it, res) in zip(sysl, refs):
                r = p.wait(p.submit(s))
                assert r["niter"] == it and np.array_equal(r["x"], x)
        info = p.resident()
        assert info["held_bytes"] <= budget and info["held"] <= 2
        assert p.stats()["peak_bytes"] <= budget
    finally:
        p.close()


def test_pool_cancel_queued_request(gpu_ctx):
    """A request still in the queue is dropped (TF_ERR_CANCELLED, x left as
    given); one that ran keeps its result; the pool keeps serving."""
    big = systems.small_hex(48, seed=6, kind="pressure", ratio=1.02)
    small = systems.small_hex(10, seed=7, kind="pressure")
    want = _reference(gpu_ctx, small)
    p = pool.Pool(workers=1, mem_budget=1 << 30)
    try:
        first = [p.submit(big) for _ in range(3)]     # one worker: these run in turn
        last = p.submit(small)
        assert p.cancel(last) == 0                     # still queued behind them
        with pytest.raises(native.TFError) as e:
            p.wait(last)
        assert e.value.status == 8                     # TF_ERR_CANCELLED
        for rid in first:
            p.wait(rid)
        assert p.cancel(first[0]) == 3                 # collected: unknown id
        again = p.submit(small)
        r = p.wait(again)
        assert p.cancel(again) == 3
        assert r["niter"] == want[1] and np.array_equal(r["x"], want[0])
    finally:
        p.close()


def test_pool_request_on_a_new_structure_is_not_passed_over_for_good(gpu_ctx):
    """300 queued requests on a held structure and one on a new structure ahead
    of them: the worker takes at most 16 of them before it."""
    known = systems.small_hex(16, seed=8, kind="pressure", ratio=1.02)
    new = systems.small_hex(11, seed=9, kind="pressure")
    want = _reference(gpu_ctx, new)
    p = pool.Pool(workers=1, mem_budget=1 << 30)
    try:
        p.wait(p.submit(known))                 # held from here on
        busy = [p.submit(known, tol=0.0, miter=20000) for _ in range(2)]
        first = p.submit(new)
        rest = [p.submit(known, tol=0.0, miter=500) for _ in range(300)]
        r = p.wait(first)
        done = p.stats()["completed"]
        assert r["niter"] == want[1] and np.array_equal(r["x"], want[0])
        # itself, the 3 before it, the 16, and what ran until wait() returned
        assert done <= 120, done
        for rid in busy + rest:
            p.wait(rid)
    finally:
        p.close()


@pytest.mark.parametrize("prec", ["jacobi", "icc"])
def test_pool_budget_counts_what_makes_solves_faster(gpu_ctx, prec, monkeypatch):
    """A budget with room for the matrix and its vectors but not for the
    one-kernel solve's layout (or the ICC records): the request is solved
    without, by the kernels a registration without them uses, and nothing
    beyond the budget is held."""
    s = systems.small_hex(24, seed=6, kind="pressure", ratio=1.02)
    s = copy.copy(s)
    s.prec = prec
    full = _reference(gpu_ctx, s)
    monkeypatch.setenv("TF_NO_RESIDENT", "1")
    monkeypatch.setenv("TF_ICC_SWEEPS", "levels")
    plain = _reference(gpu_ctx, s)
    monkeypatch.delenv("TF_NO_RESIDENT")
    monkeypatch.delenv("TF_ICC_SWEEPS")
    assert not np.array_equal(plain[0], full[0])   # sums in another order

    def served(budget):
        p = pool.Pool(workers=1, mem_budget=budget)
        try:
            for _ in range(2):
                r = p.wait(p.submit(s))
            held = p.resident()
            assert held["held"] == 1 and held["reused"] == 1
            assert p.stats()["peak_bytes"] <= budget
            return r, held["held_bytes"]
        finally:
            p.close()

    r, most = served(1 << 30)
    assert np.array_equal(r["x"], full[0])
    least, _ = 0, None
    lo, hi = 1 << 20, most
    while hi - lo > 4096:       # the smallest budget that admits the request
        mid = (lo + hi) // 2
        try:
            r, got = served(mid)
            hi, least = mid, got
            assert got <= mid
        except native.TFError as e:
            assert e.status == 2
            lo = mid
    assert least < most and np.array_equal(r["x"], plain[0])


def test_pool_icc_request_on_a_scattered_numbering(gpu_ctx):
    """The registration of an ICC request leaves out the renumbered copy, which
    ICC does not use; what it holds is what the budget counts."""
    s = copy.copy(systems.pressure_system(grids.poly_lattice_grid(12000, 4), 4, tol=1e-9,
                                          miter=300))
    s.prec = "icc"
    want = _reference(gpu_ctx, s)
    p = pool.Pool(workers=2, mem_budget=1 << 30)
    try:
        r = p.wait(p.submit(s))
        assert r["niter"] == want[1] and np.array_equal(r["x"], want[0])
        held = p.resident()
        s.prec = "jacobi"
        p.wait(p.submit(s))
        both = p.resident()
    finally:
        p.close()
    n, nnz = s.n, s.nnz
    matrix = 12 * nnz + 8 * n + 6 * 8 * n   # values, columns, rows, diagonals, vectors
    assert matrix < held["held_bytes"] < 2 * matrix + 32 * nnz + 300 * n
    assert both["held_bytes"] - held["held_bytes"] > 2 * matrix   # the copy, too
