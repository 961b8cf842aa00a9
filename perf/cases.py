"""The work that programs have this library do, as measured cases.

Every case is one call (or one short run of calls) that a flow solver makes
in its time loop, through the library's public entry points, on matrices of
the two kinds of mesh it meets:

* ``hex``: structured blocks, cells numbered plane by plane (7 entries a
  row, repeating column offsets), optionally stretched toward the y walls;
* ``poly``: unstructured polyhedral cells (about 15 entries a row) numbered
  by sorted cell centres, as the grid generator leaves them.

Pressure matrices are symmetric Poisson operators with one pinned cell,
momentum matrices are upwind convection-diffusion operators with an inertial
diagonal.  Values, right-hand sides and fluxes come from the seed; a mesh's
topology belongs to the case.
"""
import ctypes
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "t-flows_b200"))
from tflows_b200 import batch, grids, native, pool, systems  # noqa: E402

F8 = torch.float64
DEV = "cuda"


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # The smallest solve of daily use: the pressure correction of a
        # 30^3 lid-driven cavity, run to its tolerance.  Latency decides.
        dict(name="cavity-30", path="solve", mesh="hex", nx=30, ny=30, nz=30, stretch=1.0,
             kind="pressure", solver="cg", prec="jacobi", norm=True, tol=1e-8, miter=500),
        # The largest: a pressure correction on a block of 8 M cells stretched
        # toward the walls, values already on the device.
        dict(name="channel-200", path="solve", mesh="hex", nx=200, ny=200, nz=200,
             stretch=1.02, kind="pressure", solver="cg", prec="jacobi", norm=True, tol=0.0,
             miter=50),
        # An ordinary block of odd sizes with the solver's default
        # preconditioner, incomplete Cholesky.
        dict(name="icc-hex-130k", path="solve", mesh="hex", nx=57, ny=43, nz=53, stretch=1.02,
             kind="pressure", solver="cg", prec="icc", norm=True, tol=0.0, miter=20),
        # A polyhedral mesh of a million cells: scattered numbering, long rows.
        dict(name="poly-1m", path="solve", mesh="poly", nx=100, ny=100, nz=101, stretch=1.0,
             kind="pressure", solver="cg", prec="jacobi", norm=True, tol=0.0, miter=30),
        # A small polyhedral mesh with the default preconditioner, the range
        # of x taken for the residual's norm.
        dict(name="icc-poly-21k", path="solve", mesh="poly", nx=29, ny=27, nz=27, stretch=1.0,
             kind="pressure", solver="cg", prec="icc", norm=False, tol=0.0, miter=12),
        # The drop-in call itself: host arrays in and out, one momentum
        # component, solved to its tolerance.
        dict(name="host-bicg-700k", path="host", mesh="hex", nx=101, ny=77, nz=90,
             stretch=1.02, kind="momentum", solver="bicg", prec="jacobi", norm=False,
             tol=1e-6, miter=300),
        # The three velocity components of one momentum matrix.
        dict(name="components-3", path="multi", mesh="hex", nx=71, ny=64, nz=67, stretch=1.02,
             kind="momentum", solver="bicg", prec="jacobi", norm=True, tol=0.0, miter=20,
             nrhs=3),
        # A time step's matrices built on the device from face data.
        dict(name="assemble-1m", path="assemble", nx=101, ny=103, nz=97),
        # One iteration of a caller's own Krylov loop (a sub-domain of a
        # distributed solve): residual, product, updates and sums.
        dict(name="own-loop-2m", path="loop", mesh="hex", nx=160, ny=130, nz=97, stretch=1.02),
        # Many uneven systems in one batch, uploaded, solved and fetched.
        dict(name="batch-40", path="batch", count=40, lo=1000, hi=100000, pick=4),
        # Concurrent requests for exact solves, as a server passes them on.
        dict(name="pool-24", path="pool", count=24, lo=2000, hi=200000, pick=5, workers=8),
        # The product for callers who may not allocate (a device data region).
        dict(name="noalloc-1m", path="noalloc", mesh="hex", nx=110, ny=99, nz=95, stretch=1.0),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _box(rng, lo, hi):
    """Three uneven edges whose product lies in about [lo, hi]."""
    n = _log(rng, lo, hi)
    a = n ** (1.0 / 3.0)
    nx = max(3, int(round(a * rng.uniform(0.7, 1.4))))
    ny = max(3, int(round(a * rng.uniform(0.8, 1.25))))
    nz = max(3, int(n / (nx * ny)))
    return dict(nx=nx, ny=ny, nz=nz)


def draw(rng):
    path = rng.choice(["solve"] * 6 + ["host", "multi", "assemble", "loop", "batch", "pool",
                                       "noalloc"])
    stretch = rng.choice([1.0, 1.02, 1.03])
    if path == "solve":
        mesh = rng.choice(["hex", "hex", "poly"])
        prec = rng.choice(["jacobi", "jacobi", "none", "icc"])
        kind = rng.choice(["pressure", "momentum"])
        if mesh == "hex":
            size = _box(rng, 1e3, 2.5e5 if prec == "icc" else 7e6)
        else:
            size = _box(rng, 1e3, 3e4 if prec == "icc" else 9e5)
        its = (10, 40) if kind == "pressure" else (10, 20)
        if prec == "icc":
            its = (4, 12) if kind == "pressure" else (2, 4)
        return dict(path=path, mesh=mesh, stretch=stretch if mesh == "hex" else 1.0, kind=kind,
                    solver="cg" if kind == "pressure" else "bicg", prec=prec,
                    norm=rng.random() < 0.6, tol=0.0, miter=rng.randint(*its), **size)
    if path == "host":
        return dict(path=path, mesh="hex", stretch=stretch, kind="momentum", solver="bicg",
                    prec="jacobi", norm=rng.random() < 0.5, tol=1e-6, miter=300,
                    **_box(rng, 3e3, 6e5))
    if path == "multi":
        return dict(path=path, mesh=rng.choice(["hex", "hex", "poly"]), stretch=1.0,
                    kind="momentum", solver="bicg", prec="jacobi", norm=rng.random() < 0.6,
                    tol=0.0, miter=rng.randint(10, 20), nrhs=rng.randint(2, 4),
                    **_box(rng, 3e3, 7e5))
    if path == "assemble":
        return dict(path=path, **_box(rng, 1e4, 9e5))
    if path == "loop":
        return dict(path=path, mesh=rng.choice(["hex", "hex", "poly"]), stretch=1.0,
                    **_box(rng, 1e4, 9e5))
    if path in ("batch", "pool"):
        lo = int(_log(rng, 1000, 8000))
        c = dict(path=path, count=rng.randint(6, 24), lo=lo, hi=int(lo * rng.uniform(4, 10)),
                 pick=rng.randint(0, 1 << 20))
        return dict(c, workers=rng.choice([4, 8])) if path == "pool" else c
    return dict(path=path, mesh=rng.choice(["hex", "hex", "poly"]), stretch=1.0,
                **_box(rng, 1e4, 9e5))


# ---------------------------------------------------------------------------
# Meshes and matrices (on the device, from plain torch)
# ---------------------------------------------------------------------------
class Mesh:
    """A Matrix_Type structure (diagonal first, the other columns ascending,
    1-based int32 on the host) and what values are formed from: per entry its
    column and bare face coefficient, per entry its face and the sign of the
    face's flux seen from the row, as (n, width) arrays with a mask; the
    faces' mean area and the shortest distance between cells."""

    def __init__(self, cols, mask, coef, face, sign, nfaces, vol, area, h_min):
        self.cols, self.mask, self.coef, self.face, self.sign = cols, mask, coef, face, sign
        self.nfaces, self.vol, self.area, self.h_min = nfaces, vol, area, h_min
        self.n = cols.shape[0]
        lens = mask.sum(1)
        row = torch.ones(self.n + 1, dtype=torch.int64, device=DEV)
        row[1:] += torch.cumsum(lens, 0)
        self.nnz = int(row[-1]) - 1
        self.row = row.to(torch.int32).cpu().numpy()
        self.col = (cols[mask] + 1).to(torch.int32).cpu().numpy()
        self.dia = self.row[:-1].copy()
        self.csr = systems.Csr(n=self.n, row=self.row, col=self.col, dia=self.dia, pos=None)


def _hex_mesh(nx, ny, nz, stretch):
    n = nx * ny * nz
    k = torch.arange(n, device=DEV)
    i, j, l = k // (ny * nz), (k // nz) % ny, k % nz
    half = (ny + 1) // 2
    h = torch.tensor([stretch ** min(q, ny - 1 - q) for q in range(ny)], dtype=F8, device=DEV)
    h = h / h.sum()
    hx = hz = 1.0 / max(nx, nz, half)
    cols, mask, coef, face, sign = [k], [torch.ones_like(k, dtype=torch.bool)], [], [], []
    coef.append(torch.zeros(n, dtype=F8, device=DEV))
    face.append(torch.zeros_like(k))
    sign.append(torch.zeros(n, dtype=F8, device=DEV))
    area_y = hx * hz
    dist_y = torch.zeros(ny + 1, dtype=F8, device=DEV)
    dist_y[1:ny] = 0.5 * (h[1:] + h[:-1])
    # Face f*n + c lies between cell c and its neighbour up in direction f.
    for off, ok, f, up in ((-ny * nz, i > 0, 0, 0), (-nz, j > 0, 1, 0), (-1, l > 0, 2, 0),
                           (1, l < nz - 1, 2, 1), (nz, j < ny - 1, 1, 1),
                           (ny * nz, i < nx - 1, 0, 1)):
        cols.append(k + off)
        mask.append(ok)
        face.append(f * n + (k if up else k + off).clamp_min(0))
        sign.append(torch.full((n,), 1.0 if up else -1.0, dtype=F8, device=DEV))
        if f == 1:
            c = area_y / dist_y[j + up].clamp_min(1e-30)
        else:
            c = h[j] * (hz if f == 0 else hx) / (hx if f == 0 else hz)
        coef.append(c)
    st = lambda a: torch.stack(a, 1)  # noqa: E731
    return Mesh(st(cols), st(mask), st(coef), st(face), st(sign), 3 * n, h[j] * hx * hz,
                float(h.mean() * hx), min(hx, float(h.min())))


def _poly_mesh(nx, ny, nz):
    """14 neighbours a cell (the edges of a Freudenthal tetrahedralisation
    of a jittered lattice), cells numbered by their sorted centres."""
    n = nx * ny * nz
    g = torch.Generator().manual_seed(20231 + n)
    k = torch.arange(n)
    i, j, l = k // (ny * nz), (k // nz) % ny, k % nz
    x = i + torch.rand(n, generator=g, dtype=F8) * 0.5 - 0.25
    order = torch.argsort(x)
    new = torch.empty(n, dtype=torch.int64)
    new[order] = torch.arange(n)
    wob = torch.rand(7 * n, generator=g, dtype=F8).to(DEV)
    order, new, i, j, l, k = (t.to(DEV) for t in (order, new, i, j, l, k))
    big = 1 << 60
    cols, coef, face, sign = [], [], [], []
    dirs = [(1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 1, 0), (1, 0, 1), (0, 1, 1), (1, 1, 1)]
    h = 1.0 / max(nx, ny, nz)
    for f, (a, b, c) in enumerate(dirs):
        for s in (1, -1):
            u, v, w = i + s * a, j + s * b, l + s * c
            ok = (u >= 0) & (u < nx) & (v >= 0) & (v < ny) & (w >= 0) & (w < nz)
            nb = torch.where(ok, (u * ny + v) * nz + w, torch.zeros_like(k))
            fid = f * n + (k if s > 0 else nb)
            cols.append(torch.where(ok, new[nb], torch.full_like(k, big)))
            coef.append(h * (0.4 + 0.6 * wob[fid]) / (a + b + c))
            face.append(fid)
            sign.append(torch.full((n,), float(s), dtype=F8, device=DEV))
    st = lambda a: torch.stack(a, 1)[order]  # noqa: E731
    cols, coef, face, sign = st(cols), st(coef), st(face), st(sign)
    cols, p = torch.sort(cols, 1)
    coef, face, sign = (torch.gather(t, 1, p) for t in (coef, face, sign))
    first = torch.arange(n, device=DEV)[:, None]
    mask = torch.cat([torch.ones_like(first, dtype=torch.bool), cols < big], 1)
    cols = torch.cat([first, torch.where(cols < big, cols, first)], 1)
    pad = lambda t: torch.cat([torch.zeros_like(t[:, :1]), t], 1)  # noqa: E731
    return Mesh(cols, mask, pad(coef), pad(face), pad(sign), 7 * n,
                torch.full((n,), h ** 3, dtype=F8, device=DEV), 0.4 * h * h, 0.5 * h)


@functools.lru_cache(maxsize=2)
def _large_mesh(mesh, nx, ny, nz, stretch):
    return _hex_mesh(nx, ny, nz, stretch) if mesh == "hex" else _poly_mesh(nx, ny, nz)


@functools.lru_cache(maxsize=96)
def _small_mesh(mesh, nx, ny, nz, stretch):
    return _hex_mesh(nx, ny, nz, stretch) if mesh == "hex" else _poly_mesh(nx, ny, nz)


def _mesh(c):
    small = c["nx"] * c["ny"] * c["nz"] < 300000
    return (_small_mesh if small else _large_mesh)(c["mesh"], c["nx"], c["ny"], c["nz"],
                                                   c["stretch"])


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _values(m, kind, g, cfl=0.1):
    """(n, width) values of a pressure or momentum matrix."""
    if kind == "pressure":
        v = 0.5 + torch.rand(m.n, generator=g, dtype=F8, device=DEV)
        off = m.coef * 0.5 * (v[:, None] + v[m.cols.clamp(0, m.n - 1)])
        off = torch.where(m.mask, off, torch.zeros_like(off))
        off[:, 0] = 0.0
        diag = off.sum(1)
        diag[0] += diag[0]
    else:
        flux = torch.rand(m.nfaces, generator=g, dtype=F8, device=DEV) * 2.0 - 1.0
        h = float(m.vol.mean()) ** (1.0 / 3.0)
        out = flux[m.face] * m.sign * m.area
        off = 0.1 * h * m.coef - torch.clamp(out, max=0.0)
        off = torch.where(m.mask, off, torch.zeros_like(off))
        off[:, 0] = 0.0
        diag = off.sum(1) + m.vol / (cfl * m.h_min)
    val = -off
    val[:, 0] = diag
    return val


def _rhs(m, kind, g):
    b = torch.rand(m.n, generator=g, dtype=F8, device=DEV) * 2.0 - 1.0
    return b - b.mean() if kind == "pressure" else b


def _system(c, seed, g=None):
    m = _mesh(c)
    g = _gen(seed) if g is None else g
    val = _values(m, c["kind"], g)
    return m, val, _rhs(m, c["kind"], g)


def _uneven(c, seed):
    """The systems of a batch or a pool's requests: sizes spread over the
    logarithm of [lo, hi], pressure on blocks and transport on polyhedral
    meshes in turn (topologies belong to the case, values to the seed)."""
    rng = np.random.default_rng(c["pick"])
    g = _gen(seed)
    out = []
    for k in range(c["count"]):
        a = math.exp(rng.uniform(math.log(c["lo"]), math.log(c["hi"]))) ** (1.0 / 3.0)
        nx, ny = max(3, round(a * 0.9)), max(3, round(a * 1.1))
        nz = max(3, round(a))
        d = dict(mesh="poly" if k % 2 else "hex", nx=nx, ny=ny, nz=nz, stretch=1.0,
                 kind="momentum" if k % 2 else "pressure")
        out.append((d,) + _system(d, seed, g))
    return out


# ---------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------
_ctx = None


def _context():
    global _ctx
    if _ctx is None:
        _ctx = native.Context(0)
        _ctx.torch_stream = torch.cuda.ExternalStream(_ctx.stream)
    return _ctx


class _Owned(dict):
    """A state whose handle is closed with it."""

    def __del__(self):
        h = self.pop("handle", None)
        if h is not None:
            h.close()


def _pinned(t):
    p = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    p.copy_(t)
    return p.numpy()


def prepare(case, seed):
    ctx = _context()
    path = case["path"]
    s = _Owned(case=case, ctx=ctx)
    if path in ("solve", "host", "multi"):
        m, val, b = _system(case, seed)
        s["handle"] = native.Matrix(ctx, m.row, m.col, m.dia)
        if path == "host":
            s.update(val=_pinned(val[m.mask]), b=_pinned(b), x=_pinned(torch.zeros_like(b)))
            return s
        if path == "multi":
            g = _gen(seed + 7919)
            b = torch.stack([b] + [_rhs(m, case["kind"], g) for _ in range(case["nrhs"] - 1)])
        pad = torch.zeros(m.nnz + 2, dtype=F8, device=DEV)
        pad[:m.nnz] = val[m.mask]
        s.update(val=pad[:m.nnz], b=b, x=torch.zeros_like(b))
    elif path == "assemble":
        g, csr, fc = _faces(case["nx"], case["ny"], case["nz"])
        gen = _gen(seed)
        nf = g.n_faces
        s["handle"] = native.Matrix(ctx, csr.row, csr.col, csr.dia)
        native.faces_register(ctx, s["handle"], g.faces_c, csr.pos)
        up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(DEV)  # noqa: E731
        s.update(fc=up(fc), fw=up(g.fw), vol=up(g.vol),
                 vm=0.5 + torch.rand(g.n_cells, generator=gen, dtype=F8, device=DEV),
                 flux=(2.0 * torch.rand(nf, generator=gen, dtype=F8, device=DEV) - 1.0)
                 * up(g.interior.astype(np.float64)) * g.h_mean ** 2,
                 wall=up((~g.interior).astype(np.int32)),
                 open=(torch.rand(nf, generator=gen, device=DEV) < 0.2).to(torch.int32),
                 vis=0.1 * g.h_mean, dt=0.5 * g.h_min,
                 pval=torch.empty(csr.nnz, dtype=F8, device=DEV),
                 mval=torch.empty(csr.nnz, dtype=F8, device=DEV))
    elif path == "loop":
        c = dict(case, kind="pressure")
        m, val, b = _system(c, seed)
        s["handle"] = native.Matrix(ctx, m.row, m.col, m.dia)
        z = torch.zeros_like(b)
        pad = torch.zeros(m.nnz + 2, dtype=F8, device=DEV)
        pad[:m.nnz] = val[m.mask]
        s.update(n=m.n, val=pad[:m.nnz], b=b, diag=val[:, 0].contiguous(),
                 dinv=(1.0 / val[:, 0]).contiguous(),
                 x=torch.rand(m.n, generator=_gen(seed + 3), dtype=F8, device=DEV),
                 r=z.clone(), z=z.clone(), p=b.clone(), q=z.clone(),
                 sums=torch.zeros(4, dtype=F8, device=DEV))
    elif path == "noalloc":
        m, val, b = _system(dict(case, kind="pressure"), seed)
        lib = native.load()
        vp = ctypes.c_void_p
        lib.tf_spmv_noalloc.argtypes = [ctypes.c_int, vp, vp, vp, vp, vp, vp, vp]
        s.update(lib=lib, n=m.n, row=torch.from_numpy(m.row).to(DEV),
                 col=torch.from_numpy(m.col).to(DEV), val=val[m.mask], p=b,
                 q=torch.zeros_like(b), pq=torch.zeros(1, dtype=F8, device=DEV))
    else:
        todo = []
        for d, m, val, b in _uneven(case, seed):
            pressure = d["kind"] == "pressure"
            hv, hb = val[m.mask].cpu().numpy(), b.cpu().numpy()
            nrms = float(torch.sqrt(torch.sum((b / val[:, 0]) ** 2)))
            todo.append(systems.System(
                name=d["kind"], solver="cg" if pressure else "bicg", prec="jacobi", csr=m.csr,
                val=hv, b=hb, x0=np.zeros(m.n), tol=1e-10 * nrms, miter=5000, norm=1.0))
        s["systems"] = todo
        if path == "batch":
            s["handle"] = batch.Batch(ctx, mem_budget=1 << 30, max_systems=64)
        else:
            s["handle"] = pool.Pool(workers=case["workers"], mem_budget=2 << 30)
    return s


@functools.lru_cache(maxsize=2)
def _faces(nx, ny, nz):
    g = grids.hex_grid(nx, ny, nz, stretch_y=1.02)
    csr = systems.create_matrix(g)
    return g, csr, systems.face_coef(g)


def run(s):
    c, ctx, path = s["case"], s["ctx"], s["case"]["path"]
    h = s.get("handle")
    if path in ("solve", "multi"):
        with torch.cuda.stream(ctx.torch_stream):   # a correction starts from zero
            s["x"].zero_()
        args = (s["val"].data_ptr(), s["x"].data_ptr(), s["b"].data_ptr(), c["miter"], c["tol"],
                1.0 if c["norm"] else None)
        if path == "solve":
            it, res = native.solve_device(ctx, h, c["solver"], c["prec"], *args)
        else:
            it, res = native.solve_multi_device(ctx, h, c["solver"], c["prec"], c["nrhs"], *args)
        return dict(x=s["x"], val=s["val"], b=s["b"], niter=it, res=res)
    if path == "host":
        s["x"].fill(0.0)
        it, res = native.solve_native(ctx, h, c["solver"], c["prec"], s["val"], s["x"], s["b"],
                                      c["miter"], c["tol"], 1.0 if c["norm"] else None)
        return dict(x=s["x"], val=s["val"], b=s["b"], niter=it)
    if path == "assemble":
        d = lambda k: s[k].data_ptr()  # noqa: E731
        native.assemble_pressure(ctx, h, d("fc"), d("fw"), d("vm"), d("open"), d("pval"))
        native.assemble_momentum(ctx, h, d("fc"), d("flux"), d("wall"), s["vis"], 1.0, d("vol"),
                                 s["dt"], d("mval"))
        return dict(pressure=s["pval"], momentum=s["mval"])
    if path == "loop":
        n = s["n"]
        d = {k: s[k].data_ptr() for k in ("val", "b", "diag", "dinv", "x", "r", "z", "p", "q")}
        out = s["sums"].data_ptr()
        native.residual(ctx, h, d["val"], d["b"], d["x"], d["r"])
        native.vec_nrms_sum(ctx, n, d["r"], d["diag"], out)
        native.vec_jacobi(ctx, n, d["r"], d["dinv"], d["z"], out + 8)
        native.vec_axpby(ctx, n, 1.0, d["z"], 0.5, d["p"])
        native.spmv(ctx, h, d["val"], d["p"], d["q"], out + 16)
        native.vec_axpby(ctx, n, 0.25, d["p"], 1.0, d["x"])
        native.vec_axpby(ctx, n, -0.25, d["q"], 1.0, d["r"])
        native.vec_dot(ctx, n, d["r"], d["z"], out + 24)
        return dict(x=s["x"], r=s["r"], z=s["z"], p=s["p"], q=s["q"], sums=s["sums"])
    if path == "noalloc":
        st = s["lib"].tf_spmv_noalloc(s["n"], *[s[k].data_ptr() for k in
                                                ("row", "col", "val", "p", "q", "pq")], None)
        if st:
            raise RuntimeError("tf_spmv_noalloc: status %d" % st)
        return dict(q=s["q"], pq=s["pq"])
    if path == "batch":
        ids = h.add_many(s["systems"], tol=1e-10, maxit=5000)
        h.run()
        x = [h.result(i)["x"] for i in ids]
        for i in ids:
            h.remove(i)
        return dict(x=np.concatenate(x))
    ids = [h.submit(q) for q in s["systems"]]
    return dict(x=np.concatenate([h.wait(i)["x"] for i in ids]))


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    path = case["path"]
    if path in ("batch", "pool"):
        # sizes as _uneven draws them; every system read once per iteration
        # is not a floor (small ones stay on chip): values, b and x once in,
        # x once out, and about 60 iterations' multiplications
        rng = np.random.default_rng(case["pick"])
        by = fl = 0.0
        for k in range(case["count"]):
            n = math.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"])))
            w = 15.0 if k % 2 else 7.0
            by += n * (8 * w + 32)
            fl += 60 * n * (2 * w + 12)
        return dict(bytes=by, flops=fl)
    n = float(case["nx"] * case["ny"] * case["nz"])
    if path == "assemble":
        nf = 3.0 * n
        return dict(bytes=2 * 7 * n * 8 + nf * (8 + 8 + 8 + 8 + 8) + n * 16,
                    flops=nf * 14 + n * 8)
    w = 15.0 if case["mesh"] == "poly" else 7.0
    idx = 60.0 if case["mesh"] == "poly" else 1.0   # column bytes per row
    spmv = n * (8 * w + idx + 16)
    if path == "noalloc":
        return dict(bytes=n * (12 * w + 4 + 16), flops=2 * w * n + 2 * n)
    if path == "loop":
        return dict(bytes=2 * spmv + n * (16 + 24 + 24 + 24 + 24 + 16), flops=n * (4 * w + 16))
    r = float(case.get("nrhs", 1))
    # Matrices that fit on the chip are read once per solve, others once per
    # iteration; vectors likewise (x, r, p, q and the diagonal).
    fits = n * (8 * w + 48 * r) < 1.2e8
    its = float(case["miter"])
    if case["tol"] > 0:   # to a tolerance: about three edges, or a transport's 25
        its = 3.0 * n ** (1.0 / 3.0) if case["kind"] == "pressure" else 25.0
    per = (n * (8 * w + idx) + r * n * 80) * (2.0 if case["prec"] == "icc" else 1.0)
    once = n * (16 * w + idx) + r * n * 40
    return dict(bytes=once + (0.0 if fits else its * per), flops=its * r * n * (2 * w + 12))


def tolerance(case):
    path = case["path"]
    if path in ("batch", "pool"):
        # the stopping tests leave x to about 1e-10 times the condition number
        return dict(rel=1e-6, max=1e-4)
    if path in ("assemble", "noalloc"):
        return dict(rel=1e-13, max=1e-11)
    if path == "loop":
        return dict(rel=1e-12, max=1e-10)
    # rounding of the dot products, amplified by the recurrence
    if case["tol"] > 0:
        return dict(rel=1e-6, max=1e-5)
    return dict(rel=1e-9, max=1e-7)


# ---------------------------------------------------------------------------
# The same in plain 64-bit torch
# ---------------------------------------------------------------------------
def _mul(m, val, x):
    """A x, one slot of the rows at a time."""
    acc = torch.zeros_like(x)
    for k in range(m.cols.shape[1]):
        t = val[:, k] * x[m.cols[:, k].clamp(0, m.n - 1)]
        acc += torch.where(m.mask[:, k], t, torch.zeros_like(t))
    return acc


def _icc(m, val, level):
    """Incomplete Cholesky on the matrix's own pattern as a function r -> z,
    plane after plane of cells with independent rows (level)."""
    order = torch.argsort(level, stable=True)
    cuts = torch.searchsorted(level[order], torch.arange(int(level.max()) + 2, device=DEV))
    planes = [order[a:b] for a, b in zip(cuts[:-1].tolist(), cuts[1:].tolist()) if b > a]
    n = m.n
    me = torch.arange(n, device=DEV)[:, None]
    low = m.mask & (m.cols < me)
    upp = m.mask & (m.cols > me)
    cl = m.cols.clamp(0, n - 1)
    vl, vu = torch.where(low, val, 0.0 * val), torch.where(upp, val, 0.0 * val)
    d = torch.zeros(n, dtype=F8, device=DEV)
    for r in planes:
        d[r] = 1.0 / (val[r, 0] - (d[cl[r]] * vl[r] * vl[r]).sum(1))

    def apply(res):
        y = torch.zeros_like(res)
        for r in planes:
            y[r] = (res[r] - (vl[r] * y[cl[r]]).sum(1)) * d[r]
        z = y / d
        for r in reversed(planes):
            z[r] = (z[r] - (vu[r] * z[cl[r]]).sum(1)) * d[r]
        return z
    return apply


def _cg(m, val, b, prec, norm, tol, miter, x=None, level=None):
    """Cg on the system scaled by its mean diagonal, stopped on the residual's
    root of the sum of (r / diagonal)^2 over the range of x (or norm)."""
    fn = 1.0 / float(val[:, 0].mean())
    val, b = val * fn, b * fn
    x = torch.zeros_like(b) if x is None else x.clone()
    d = val[:, 0]
    m_inv = _icc(m, val, level) if prec == "icc" else None

    def size(r):
        span = 1.0 if norm else max(1e-15, float(x.max() - x.min()))
        return float(torch.sqrt(torch.sum((r / d) ** 2))) / span

    if size(b) < tol:
        return x, 0, 0.0
    r = b - _mul(m, val, x)
    res, rho_old, p, it = size(r), 1.0, None, 0
    if res < tol or miter < 1:
        return x, 0, res
    for it in range(1, miter + 1):
        z = m_inv(r) if m_inv else (r / d if prec == "jacobi" else r)
        rho = torch.dot(z, r)
        p = z if p is None else z + (rho / rho_old) * p
        q = _mul(m, val, p)
        a = rho / torch.dot(p, q)
        x = x + a * p
        r = r - a * q
        res = size(r)
        if res < tol:
            break
        rho_old = rho
    return x, it, res


def exact(case, seed):
    path = case["path"]
    if path in ("solve", "host", "multi"):
        level = None
        if case["prec"] == "icc":
            if case["mesh"] != "hex":
                return None
            k = torch.arange(case["nx"] * case["ny"] * case["nz"], device=DEV)
            yz = case["ny"] * case["nz"]
            level = k // yz + (k // case["nz"]) % case["ny"] + k % case["nz"]
        m, val, b = _system(case, seed)
        args = (case["prec"], case["norm"], case["tol"], case["miter"])
        if path == "multi":
            g = _gen(seed + 7919)
            rhs = [b] + [_rhs(m, case["kind"], g) for _ in range(case["nrhs"] - 1)]
            got = [_cg(m, val, q, *args) for q in rhs]
            return dict(x=torch.stack([q[0] for q in got]), val=val[m.mask],
                        b=torch.stack(rhs), niter=[q[1] for q in got], res=[q[2] for q in got])
        x, it, res = _cg(m, val, b, *args, level=level)
        out = dict(x=x, val=val[m.mask], b=b, niter=it)
        if path == "solve":
            out["res"] = res
            return out
        return {k: (v.cpu().numpy() if torch.is_tensor(v) else v) for k, v in out.items()}
    if path == "assemble":
        s = prepare(case, seed)
        g, csr, _ = _faces(case["nx"], case["ny"], case["nz"])
        up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(DEV)  # noqa: E731
        inner = up(g.interior)
        c = up(g.faces_c).long() - 1
        c1, c2 = c[:, 0], torch.where(inner, c[:, 1], c[:, 0])
        pos, dia = up(csr.pos).long() - 1, up(csr.dia).long() - 1
        zero = torch.zeros(g.n_cells, dtype=F8, device=DEV)
        a = s["fc"] * (s["fw"] * s["vm"][c1] + (1.0 - s["fw"]) * s["vm"][c2])
        opened = (~inner) & (s["open"] != 0)
        d = zero.index_add(0, c1[inner], a[inner]).index_add(0, c2[inner], a[inner])
        d = d.index_add(0, c1[opened], (s["fc"] * s["vm"][c1])[opened])
        pv = torch.zeros(csr.nnz, dtype=F8, device=DEV)
        pv[pos[inner, 0]], pv[pos[inner, 1]], pv[dia] = -a[inner], -a[inner], d
        m12 = s["vis"] * s["fc"] - s["flux"].clamp(max=0.0)
        m21 = s["vis"] * s["fc"] + s["flux"].clamp(min=0.0)
        wall = inner | (s["wall"] != 0)
        d = zero.index_add(0, c1[wall], m12[wall]).index_add(0, c2[inner], m21[inner])
        mv = torch.zeros_like(pv)
        mv[pos[inner, 0]], mv[pos[inner, 1]] = -m12[inner], -m21[inner]
        mv[dia] = d + s["vol"] / s["dt"]
        return dict(pressure=pv, momentum=mv)
    if path == "loop":
        m, val, b = _system(dict(case, kind="pressure"), seed)
        x = torch.rand(m.n, generator=_gen(seed + 3), dtype=F8, device=DEV)
        r = b - _mul(m, val, x)
        z = r * (1.0 / val[:, 0])
        s0, s1 = ((r / val[:, 0]) ** 2).sum(), torch.dot(z, r)
        p = z + 0.5 * b
        q = _mul(m, val, p)
        r2 = r - 0.25 * q
        return dict(x=x + 0.25 * p, r=r2, z=z, p=p, q=q,
                    sums=torch.stack([s0, s1, torch.dot(p, q), torch.dot(r2, z)]))
    if path == "noalloc":
        m, val, b = _system(dict(case, kind="pressure"), seed)
        q = _mul(m, val, b)
        return dict(q=q, pq=torch.dot(b, q)[None])
    # batch and pool: the solutions themselves
    xs = []
    for d, m, val, b in _uneven(case, seed):
        nrms = float(torch.sqrt(torch.sum((b / val[:, 0]) ** 2)))
        xs.append(_cg(m, val, b, "jacobi", True, 1e-13 * nrms, 2000)[0].cpu().numpy())
    return dict(x=np.concatenate(xs))
