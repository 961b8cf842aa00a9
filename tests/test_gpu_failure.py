"""Failure paths of the drop-in, made without faulting the GPU.

* The watchdog: the context's limit is set to a nanosecond, so the SpMV
  streamers' first waits for a tile's copies come after their deadline and
  give up; the solve must end with TF_ERR_TIMEOUT (the CTAs still wait for
  the copies they started, with the default limit, before exiting), and
  the same context must then solve normally again.  Run on the row-pattern
  streamer (hex) and on the CSR streamer (polyhedral), each in the graph of
  kernels, and on the exchanges of the one-kernel solve of both.
* Degenerate input the reference does not reject (Message_Mod/Error.f90 is
  never reached for it): NaN in b and a zero diagonal.  The numbers
  propagate; the drop-in must run the same iterations as the oracle (which
  is pinned to the reference's own source) and produce NaN/inf where it
  does.
"""
import numpy as np
import pytest

from oracle import oracle as O
from tflows_b200 import native, systems

pytestmark = pytest.mark.gpu


def oracle(s, val, b, miter, tol, norm, prec="jacobi"):
    v, x, bb = val.copy(), s.x0.copy(), b.copy()
    r = O.solve_native("cg", prec, s.csr.row, s.csr.col, s.csr.dia, v, x, bb, miter, tol,
                       norm=norm, threads=8)
    return x, r["niter"], r["fin_res"]


def gpu(ctx, m, s, val, b, miter, tol, norm, prec="jacobi"):
    v, x, bb = val.copy(), s.x0.copy(), b.copy()
    it, res = native.solve(ctx, m, "cg", prec, v, x, bb, miter, tol, norm)
    return x, it, res


@pytest.mark.parametrize("kind", ["hex-row-patterns", "poly-csr-tiles"])
def test_wait_limit_runs_out_then_context_recovers(kind, solve_path, monkeypatch):
    if kind == "hex-row-patterns":
        s = systems.small_hex(64, seed=4, kind="pressure", ratio=1.02)
    else:
        monkeypatch.setenv("TF_TILE_CFG", "6")   # variable CSR tiles, 4 lanes per row
        s = systems.poly_system(60000, seed=5, kind="pressure", tol=1e-10, miter=5000,
                                norm=1.0)
    ctx = native.Context(0)
    try:
        m = native.Matrix(ctx, s.csr.row, s.csr.col, s.csr.dia)
        try:
            ctx.set_wait_limit(1e-9)
            with pytest.raises(native.TFError) as e:
                gpu(ctx, m, s, s.val, s.b, 200, 1e-10, 1.0)
            assert e.value.status == 4                     # TF_ERR_TIMEOUT
            ctx.set_wait_limit(0.0)                        # back to the default
            x, it, res = gpu(ctx, m, s, s.val, s.b, 5000, 1e-10, 1.0)
            assert (m.resident_ctas > 0) == (solve_path == "one-kernel")
            ox, oit, ores = oracle(s, s.val, s.b, 5000, 1e-10, 1.0)
            assert abs(it - oit) <= max(1, 0.02 * oit) and res < 1e-10
            assert np.linalg.norm(x - ox) <= 1e-8 * np.linalg.norm(ox)
        finally:
            m.close()
    finally:
        ctx.close()


def test_icc_solve_that_times_out_leaves_the_next_solves_alone():
    """An ICC solve under a nanosecond's limit, before the matrix's first
    solve without and after it: both kinds then solve normally."""
    s = systems.small_hex(20, seed=4, kind="pressure", ratio=1.02)
    ctx = native.Context(0)
    m = native.Matrix(ctx, s.csr.row, s.csr.col, s.csr.dia)
    try:
        for _ in range(2):
            ctx.set_wait_limit(1e-9)
            with pytest.raises(native.TFError) as e:
                gpu(ctx, m, s, s.val, s.b, 200, 1e-10, 1.0, "icc")
            assert e.value.status == 4
            ctx.set_wait_limit(0.0)
            for prec in ("jacobi", "icc"):
                x, it, res = gpu(ctx, m, s, s.val, s.b, 5000, 1e-10, 1.0, prec)
                ox, oit, _ = oracle(s, s.val, s.b, 5000, 1e-10, 1.0, prec)
                assert abs(it - oit) <= max(1, 0.02 * oit) and res < 1e-10
                assert np.linalg.norm(x - ox) <= 1e-8 * np.linalg.norm(ox)
    finally:
        m.close()
        ctx.close()


def test_icc_sweep_wait_runs_out_then_context_recovers(monkeypatch):
    """One row of 5,000 lower entries is summed for some 2 ms while all other
    warps of the sweep wait for it: under a limit of 0.1 ms they give up (the
    products of such a matrix wait for nothing), under the default the solve is
    the oracle's."""
    monkeypatch.setenv("TF_ICC_SWEEPS", "one")
    n, hub = 6000, 5000
    rng = np.random.default_rng(8)
    other = np.delete(np.arange(n), hub)
    w = -rng.uniform(0.2, 1.0, n - 1)   # entries (hub, other) and (other, hub)
    i = np.arange(n)
    diag = np.full(n, 0.3)
    diag[other] -= w
    diag[hub] -= w.sum()
    r, c, v = (np.concatenate(t) for t in ((i, np.full(n - 1, hub), other),
                                           (i, other, np.full(n - 1, hub)), (diag, w, w)))
    order = np.lexsort((c, c != r, r))
    row = np.concatenate([[1], 1 + np.cumsum(np.bincount(r, minlength=n))]).astype(np.int32)
    col, dia, val = (c[order] + 1).astype(np.int32), row[:-1].copy(), v[order]
    b = rng.uniform(-1, 1, n)
    ox, ov, ob = np.zeros(n), val.copy(), b.copy()
    want = O.solve_native("cg", "icc", row, col, dia, ov, ox, ob, 20, 1e-10, norm=1.0)
    with native.Context(0) as ctx:
        m = native.Matrix(ctx, row, col, dia)
        try:
            assert m.tile_config == 3 and m.icc_kernels == 1
            for _ in range(2):
                ctx.set_wait_limit(1e-4)
                with pytest.raises(native.TFError) as e:
                    native.solve(ctx, m, "cg", "icc", val.copy(), np.zeros(n), b.copy(), 20,
                                 1e-10, 1.0)
                assert e.value.status == 4
                ctx.set_wait_limit(0.0)
                x = np.zeros(n)
                it, res = native.solve(ctx, m, "cg", "icc", val.copy(), x, b.copy(), 20, 1e-10,
                                       1.0)
                assert it == want["niter"] and res < 1e-10
                assert np.linalg.norm(x - ox) <= 1e-8 * np.linalg.norm(ox)
        finally:
            m.close()


def test_icc_sweeps_longer_than_the_limit_run_to_their_end():
    """100,000 levels of one row take some 30 ms a sweep, the products a few us:
    a limit of 5 ms is about waits that nothing moves, not about long sweeps."""
    n = 100000
    i = np.arange(n)
    lo, up = i > 0, i < n - 1
    w = -np.random.default_rng(5).uniform(0.2, 1.0, n)   # entry (i, i + 1)
    diag = 0.3 - w * up - np.roll(w, 1) * lo
    col = np.stack([i, i - 1, i + 1], 1)
    val = np.stack([diag, np.roll(w, 1), w], 1)
    keep = np.stack([i >= 0, lo, up], 1)
    row = np.concatenate([[1], 1 + np.cumsum(keep.sum(1))]).astype(np.int32)
    col, val = (col[keep] + 1).astype(np.int32), val[keep]
    b = np.random.default_rng(6).uniform(-1, 1, n)
    ox, ov, ob = np.zeros(n), val.copy(), b.copy()
    want = O.solve_native("cg", "icc", row, col, row[:-1].copy(), ov, ox, ob, 5, 1e-12, norm=1.0)
    with native.Context(0) as ctx:
        m = native.Matrix(ctx, row, col, row[:-1].copy())
        try:
            ctx.set_wait_limit(5e-3)
            x, v, bb = np.zeros(n), val.copy(), b.copy()
            it, res = native.solve(ctx, m, "cg", "icc", v, x, bb, 5, 1e-12, 1.0)
        finally:
            m.close()
    assert it == want["niter"] and np.linalg.norm(x - ox) <= 1e-8 * np.linalg.norm(ox)


def wide_halo_system(n=30000):
    """Symmetric and diagonally dominant; 256 consecutive rows refer to some 2,300
    rows outside them, more than the four a thread polls for ahead."""
    rng = np.random.default_rng(11)
    offs = [1] + list(range(3000, 18000, 3000))
    i = np.arange(n)
    w = {o: -rng.uniform(0.2, 1.0, n) for o in offs}   # entry (i, i + o)
    r = np.concatenate([np.concatenate([i[:n - o], i[o:]]) for o in offs])
    c = np.concatenate([np.concatenate([i[o:], i[:n - o]]) for o in offs])
    v = np.concatenate([np.concatenate([w[o][:n - o]] * 2) for o in offs])
    diag = 0.3 - np.bincount(r, weights=v, minlength=n)
    r, c, v = (np.concatenate([a, b]) for a, b in ((r, i), (c, i), (v, diag)))
    order = np.lexsort((c, c != r, r))   # the diagonal first
    row = np.zeros(n + 1, np.int32)
    row[1:] = np.cumsum(np.bincount(r, minlength=n))
    return row + 1, c[order].astype(np.int32) + 1, row[:-1] + 1, v[order], rng.uniform(-1, 1, n)


def test_solve_under_a_short_limit_is_right_or_times_out():
    """The one-kernel solve over wait limits around the time of its exchanges:
    a call that succeeds has the bits of an unhurried one, whatever waits were
    close to their end, and one that does not leaves the context usable."""
    row, col, dia, val, b = wide_halo_system()
    ctx = native.Context(0)
    m = native.Matrix(ctx, row, col, dia)
    try:
        def run():
            v, x, bb = val.copy(), np.zeros(len(b)), b.copy()
            return native.solve(ctx, m, "cg", "jacobi", v, x, bb, 30, 1e-300, 1.0), x

        want, x0 = run()
        assert want[0] == 30
        ended = []
        for limit in np.geomspace(1e-9, 1e-3, 60):
            ctx.set_wait_limit(limit)
            try:
                got, x = run()
                ended.append(True)
                assert got == want and np.array_equal(x, x0)
            except native.TFError as e:
                assert e.status == 4
                ended.append(False)
        assert not ended[0] and ended[-1]
        ctx.set_wait_limit(0.0)
        got, x = run()
        assert got == want and np.array_equal(x, x0)
    finally:
        m.close()
        ctx.close()


def test_right_hand_sides_after_one_that_timed_out():
    """Several right-hand sides on a matrix that fits the chip are solved one
    after another on the caller's arrays.  Over wait limits around the time of
    the first exchange (the first solve waits for its values, later ones find
    them in L2): what is written of any x has the bits of an unhurried call."""
    import torch
    row, col, dia, val, b = wide_halo_system()
    n, nrhs = len(b), 3
    B = np.stack([b, -0.5 * b[::-1], np.roll(b, 7)])
    flush = torch.zeros(1 << 25, dtype=torch.float64, device="cuda")   # larger than L2
    ctx = native.Context(0)
    m = native.Matrix(ctx, row, col, dia)
    try:
        def run():
            d = [torch.from_numpy(a).cuda() for a in (val, np.zeros((nrhs, n)), B)]
            flush.add_(1.0)
            torch.cuda.synchronize()
            try:
                r = native.solve_multi_device(ctx, m, "cg", "jacobi", nrhs,
                                              *(t.data_ptr() for t in d), 5, 1e-300, 1.0)
            except native.TFError as e:
                assert e.status == 4
                r = None
            torch.cuda.synchronize()
            return r, [t.cpu().numpy() for t in d]

        want, (v0, x0, b0) = run()
        assert want is not None
        late = 0
        for limit in np.concatenate([[1e-9], np.geomspace(2e-6, 8e-6, 300), [1e-3]]):
            ctx.set_wait_limit(limit)
            got, (v, x, bb) = run()
            if got is not None:
                assert got == want and np.array_equal(x, x0)
                continue
            late += 1
            assert ((x == x0) | (x == 0.0)).all(), limit
        assert late > 0 and got == want
        ctx.set_wait_limit(0.0)
        got, (v, x, bb) = run()
        assert got == want and all(np.array_equal(a, c) for a, c in ((v, v0), (x, x0), (bb, b0)))
    finally:
        m.close()
        ctx.close()


def test_registration_without_room():
    """Every allocation of a registration that fails ends it cleanly, but for the
    one-kernel solve's layout, an accelerator: without its memory the graph of
    kernels solves the matrix, single and several right-hand sides."""
    s = systems.small_hex(17, seed=3, kind="pressure", ratio=1.02)
    want = oracle(s, s.val, s.b, 3000, 1e-10, 1.0)
    with native.Context(0) as ctx:
        failed = 0
        while True:
            ctx.fail_allocs(failed, 1)
            try:
                m = native.Matrix(ctx, s.csr.row, s.csr.col, s.csr.dia)
                break
            except native.TFError as e:
                assert e.status == 2
                failed += 1
        try:
            assert failed > 10 and m.resident_ctas == 0
            X = np.stack([s.x0, s.x0])
            it, res = native.solve_multi(ctx, m, "cg", "jacobi", s.val.copy(), X,
                                         np.stack([s.b, s.b]), 3000, 1e-10, 1.0)
            x1, it1, res1 = gpu(ctx, m, s, s.val, s.b, 3000, 1e-10, 1.0)
            assert (it[1], res[1]) == (it1, res1) and np.array_equal(X[1], x1)
            assert abs(it1 - want[1]) <= max(1, 0.02 * want[1]) and res1 < 1e-10
            assert np.linalg.norm(x1 - want[0]) <= 1e-8 * np.linalg.norm(want[0])
        finally:
            m.close()


@pytest.mark.parametrize("skip", [0, 1, 9, 13, 16])
def test_icc_without_room_for_the_records(skip):
    """Any allocation of the one-CTA sweeps' records that fails leaves the
    kernels per level, which give every z the same bits; the sums over z are
    taken in another order."""
    s = systems.small_hex(14, seed=3, kind="pressure", ratio=1.02)
    want = oracle(s, s.val, s.b, 3000, 1e-10, 1.0, "icc")
    with native.Context(0) as ctx:
        m = native.Matrix(ctx, s.csr.row, s.csr.col, s.csr.dia)
        try:
            ctx.fail_allocs(skip, 1)   # the records are 17 allocations
            for _ in range(2):
                x, it, res = gpu(ctx, m, s, s.val, s.b, 3000, 1e-10, 1.0, "icc")
                assert it == want[1] and res < 1e-10
                assert np.linalg.norm(x - want[0]) <= 1e-8 * np.linalg.norm(want[0])
        finally:
            m.close()


def test_wait_limit_argument_checks(gpu_ctx):
    with pytest.raises(native.TFError):
        gpu_ctx.set_wait_limit(-1.0)
    gpu_ctx.set_wait_limit(0.0)


def same_propagation(g, o):
    x, it, res = g
    ox, oit, ores = o
    assert it == oit
    assert np.array_equal(np.isnan(x), np.isnan(ox))
    assert np.array_equal(np.isinf(x), np.isinf(ox))
    fin = np.isfinite(ox)
    if fin.any():
        assert np.allclose(x[fin], ox[fin], rtol=1e-8, atol=1e-12)
    assert (np.isnan(res) and np.isnan(ores)) or res == pytest.approx(ores, rel=1e-8)


@pytest.mark.parametrize("n", [6, 40])
def test_nan_in_rhs_propagates_like_the_reference(gpu_ctx, solve_path, n):
    s = systems.small_hex(n, seed=6, kind="pressure")
    b = s.b.copy()
    b[s.n // 3] = np.nan
    m = native.Matrix(gpu_ctx, s.csr.row, s.csr.col, s.csr.dia)
    try:
        g = gpu(gpu_ctx, m, s, s.val, b, 25, 1e-10, 1.0)
    finally:
        m.close()
    o = oracle(s, s.val, b, 25, 1e-10, 1.0)
    assert o[1] == 25          # NaN never compares below tol: the loop runs out
    same_propagation(g, o)


@pytest.mark.parametrize("prec", ["jacobi", "none"])
def test_zero_diagonal_propagates_like_the_reference(gpu_ctx, solve_path, prec):
    s = systems.small_hex(6, seed=7, kind="pressure")
    val = s.val.copy()
    val[s.csr.dia[11] - 1] = 0.0
    m = native.Matrix(gpu_ctx, s.csr.row, s.csr.col, s.csr.dia)
    try:
        g = gpu(gpu_ctx, m, s, val, s.b, 25, 1e-10, 1.0, prec)
    finally:
        m.close()
    same_propagation(g, oracle(s, val, s.b, 25, 1e-10, 1.0, prec))
