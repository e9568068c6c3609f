"""The work that programs have this library do, as measured cases.

Every case is one call (or one batch of requests) through the public entry
points, on the matrices that the library's benchmarks and tests use:
Dirichlet Laplacians of 2-D and 3-D grids and random sparse SPD matrices.  A
program registers its matrix once and then applies filters, estimates
densities of states or solves slices on it, with new vectors each time; so a
case's matrix and polynomials follow from the case alone and its vectors from
the seed, and `prepare` registers the matrix anew as a program with a new
matrix would.

Kinds of cases:

filter   ChebAv, the FP64 filter on one vector: 94-97% of a slice solve.
block    evslx_chebav_block, one FP64 filter on a block (subspace iteration).
multi    evslx_chebav_multi, FP64 or mixed precision, one polynomial per
         column (the slices that share a matrix).
kpm      evslx_kpmdos_probes, the density of states that places the slices.
nr, tr   ChebLanNr / ChebLanTr, a whole slice solve from the host's start
         vector to its eigenvalues (and vectors where asked for).
engine   the request engine serving a batch of slices of uneven matrices.
"""
import ctypes as C
import math

import numpy as np
import torch

import evsl_b200
from evsl_b200 import workloads

DEVICE = "cuda:0"
TOL = 1e-8  # residual tolerance of every solve, the benchmarks' own


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the filter of the smallest solve (100 x 100 grid, [0.6, 0.9]): latency
        dict(name="filter-2d-100", kind="filter", nx=100, ny=100, nz=1, deg=24),
        # an ordinary grid of odd sizes, cut into a few hundred slices
        dict(name="filter-3d-71", kind="filter", nx=71, ny=70, nz=69, deg=311),
        # the filter of the headline slice solve (10^6 rows, degree 1440)
        dict(name="filter-3d-100", kind="filter", nx=100, ny=100, nz=100, deg=1440),
        # no structure at all: 2 million rows of 33 entries at random columns
        dict(name="filter-random", kind="filter", random=2000000, offdiag=16, deg=40),
        # a subspace-iteration block
        dict(name="block-3d-51", kind="block", nx=51, ny=50, nz=49, deg=61, ncols=16),
        # slices of one matrix filtered together in mixed precision
        dict(name="multi-mixed-3d-100", kind="multi", nx=100, ny=100, nz=100, deg=180, spread=40, ncols=8, mixed=True),
        # the density of states of the headline matrix: 30 probes, 300 moments
        dict(name="kpm-3d-100", kind="kpm", nx=100, ny=100, nz=100, nvec=30, moments=300, damping=1),
        # a small one, as a request stream brings it
        dict(name="kpm-2d-100", kind="kpm", nx=100, ny=100, nz=1, nvec=8, moments=100, damping=1),
        # a whole solve of many pairs on the small grid: reorthogonalisation and
        # the convergence tests weigh as much as the low-degree filter
        dict(name="nr-2d-100", kind="nr", nx=101, ny=97, nz=1, lo=0.6, count=240, maxit=2000, vectors=False),
        # a mid-size solve of an interior slice, thick-restarted
        dict(name="tr-3d-30", kind="tr", nx=31, ny=30, nz=28, lo=0.9, count=40, maxit=2000, vectors=False),
        # a few pairs at the lower end of a small operator, with their vectors
        dict(name="nr-2d-47", kind="nr", nx=47, ny=34, nz=1, lo=0.05, count=20, maxit=1000, vectors=True),
        # sixteen independent operators of uneven size served together
        dict(name="engine-uneven-16", kind="engine", instances=16, nmin=1000, nmax=20000, kmin=20, kmax=50, grids=4),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid(rng, n):
    """A 2-D or 3-D grid of about n points with unequal sides."""
    if rng.random() < 0.5:
        nx = max(8, int(math.sqrt(n * rng.uniform(1.05, 1.6))))
        return nx, max(7, n // nx - (1 if n // nx == nx else 0)), 1
    nx = max(6, int((n * rng.uniform(1.1, 1.5)) ** (1 / 3)))
    ny = nx - 1 - rng.randrange(max(1, nx // 6))
    return nx, ny, max(4, min(n // (nx * ny), ny - 1 if ny > 5 else ny))


def draw(rng):
    kind = rng.choice(["filter", "filter", "filter", "block", "multi", "kpm", "kpm", "nr", "tr", "engine"])
    if kind == "filter" and rng.random() < 0.2:
        return dict(kind="filter", random=_log_int(rng, 20000, 1500000), offdiag=rng.randint(5, 16),
                    deg=_log_int(rng, 10, 40))
    if kind in ("filter", "block", "multi", "kpm"):
        n = _log_int(rng, 2000, 1000000)
        nx, ny, nz = _grid(rng, n)
        c = dict(kind=kind, nx=nx, ny=ny, nz=nz)
        if kind == "filter":
            c.update(deg=_log_int(rng, 10, 1400))
        elif kind == "block":
            c.update(deg=_log_int(rng, 10, 150), ncols=rng.randint(2, 24))
        elif kind == "multi":
            d = _log_int(rng, 20, 180)
            c.update(deg=d, spread=d // 4, ncols=rng.randint(2, 16), mixed=rng.random() < 0.6)
        else:
            c.update(nvec=rng.randint(5, 40), moments=rng.randint(60, 300), damping=rng.choice([1, 2]))
        return c
    if kind in ("nr", "tr"):
        while True:
            nx, ny, nz = _grid(rng, _log_int(rng, 2000, 25000))
            lo, count = round(rng.uniform(0.3, 1.0), 4), rng.randint(15, 80)
            # one start vector spans one copy of a repeated eigenvalue: which
            # others appear is rounding, so sides with common ratios are left out
            if np.diff(_slice(nx, ny, nz, lo, count)[1]).min() > 1e-6:
                return dict(kind=kind, nx=nx, ny=ny, nz=nz, lo=lo, count=count, maxit=2000, vectors=False)
    return dict(kind="engine", instances=rng.randint(4, 14), nmin=1000, nmax=_log_int(rng, 5000, 20000), kmin=20,
                kmax=rng.randint(30, 50), grids=rng.randrange(1 << 20))


# ---------------------------------------------------------------------------
# matrices
# ---------------------------------------------------------------------------
_LIB = None
_HOST = {}  # the last grid's host CSR: a program has its matrix in hand
_RANDOM = {}  # the last random matrix, on the device


def _library():
    global _LIB
    if _LIB is None:
        torch.zeros(1, device=DEVICE)
        _LIB = evsl_b200.Library()
    return _LIB


def _laplacian(nx, ny, nz):
    key = (nx, ny, nz)
    if key not in _HOST:
        _HOST.clear()
        _HOST[key] = workloads.laplacian_csr(nx, ny, nz)
    return _HOST[key]


def _random_csr(n, offdiag):
    """A random sparse symmetric positive definite matrix on the device, as
    workloads.random_spd_csr draws it: `offdiag` uniform columns per row,
    values in (-0.5, 0.5) after symmetrisation, each diagonal entry the row's
    absolute sum plus a number in (0, 1).  Values are multiples of 2^-40, so
    that every sum here is exact in any order.  Returns int32 row pointer and
    columns, double values and the largest absolute row sum."""
    key = (n, offdiag)
    if key in _RANDOM:
        return _RANDOM[key]
    _RANDOM.clear()
    g = torch.Generator(device=DEVICE).manual_seed(17)
    i = torch.arange(n, device=DEVICE).repeat_interleave(offdiag)
    j = torch.randint(0, n, (n * offdiag,), device=DEVICE, generator=g)
    key64 = torch.unique((torch.minimum(i, j) * n + torch.maximum(i, j))[i != j])
    del i, j
    lo, hi = key64 // n, key64 % n
    del key64
    val = torch.randint(-(1 << 39) + 1, 1 << 39, (lo.numel(),), device=DEVICE, generator=g).double() / (1 << 40)
    diag = torch.randint(1, 1 << 40, (n,), device=DEVICE, generator=g).double() / (1 << 40)
    diag.index_add_(0, lo, val.abs())
    diag.index_add_(0, hi, val.abs())
    at = torch.arange(n, device=DEVICE)
    row, col = torch.cat([lo, hi, at]), torch.cat([hi, lo, at])
    val = torch.cat([val, val, diag])
    del lo, hi
    order = torch.argsort(row * n + col)
    ia = torch.zeros(n + 1, dtype=torch.int64, device=DEVICE)
    ia[1:] = torch.cumsum(torch.bincount(row, minlength=n), 0)
    _RANDOM[key] = (ia.int(), col[order].int(), val[order], float(2 * diag.max()))
    return _RANDOM[key]


def _bounds(case):
    """[lmin, lmax] of the case's matrix."""
    if "random" in case:
        return 0.0, _random_csr(case["random"], case["offdiag"])[3]
    return 0.0, 8.0 if case["nz"] == 1 else 12.0


def _rows(case):
    return case["random"] if "random" in case else case["nx"] * case["ny"] * case["nz"]


def _register(lib, case):
    """Makes the case's matrix the library's registered one; returns what has
    to stay alive with it."""
    if "random" not in case:
        ia, ja, a = _laplacian(case["nx"], case["ny"], case["nz"])
        lib.set_csr(ia, ja, a)
        return None
    ia, ja, a, _ = _random_csr(case["random"], case["offdiag"])
    n = case["random"]
    m = evsl_b200.CsrMat(owndata=0, nrows=n, ncols=n, nnz=a.numel(),
                         ia=C.cast(ia.data_ptr(), C.POINTER(C.c_int)), ja=C.cast(ja.data_ptr(), C.POINTER(C.c_int)),
                         a=C.cast(a.data_ptr(), C.POINTER(C.c_double)))
    torch.cuda.synchronize()
    _ok(lib, lib.lib.SetAMatrix_device_csr(C.byref(m)))
    lib.n = n
    return ia, ja, a, m


def _ok(lib, rc):
    if rc != 0:
        raise RuntimeError("the library returned %d: %s" % (rc, lib.last_error()))


# ---------------------------------------------------------------------------
# polynomials
# ---------------------------------------------------------------------------
def _coefficients(deg, gamma):
    """Chebyshev coefficients of the sigma-damped delta function at `gamma` in
    (-1, 1), scaled to 1 there: what find_pol designs for that degree."""
    k = np.arange(deg + 1)
    th = math.pi / (deg + 1)
    jac = np.ones(deg + 1)
    jac[0] = 0.5
    jac[1:] = np.sin(k[1:] * th) / (k[1:] * th)
    c = np.cos(k * math.acos(gamma))
    return jac * c / np.sum(jac * c * c)


def _polynomial(case, deg, gamma):
    """(polparams, its coefficient array) for the case's spectrum."""
    lmin, lmax = _bounds(case)
    mu = _coefficients(deg, gamma)
    pol = evsl_b200.PolParams()
    _library().lib.set_pol_def(C.byref(pol))
    pol.mu = mu.ctypes.data_as(C.POINTER(C.c_double))
    pol.deg, pol.cc, pol.dd, pol.gam, pol.bar = deg, (lmax + lmin) / 2, (lmax - lmin) / 2, gamma, 0.8
    return pol, mu


def _column_filters(case):
    """(degree, gamma) of each column of a multi case: neighbouring slices."""
    m = case["ncols"]
    return [(case["deg"] + (case["spread"] * c) // max(1, m - 1), -0.9 + 0.3 * c / m) for c in range(m)]


# ---------------------------------------------------------------------------
# slices
# ---------------------------------------------------------------------------
def _spectrum(nx, ny, nz):
    """All eigenvalues of the Dirichlet Laplacian, ascending."""
    s = [4 * np.sin(np.arange(1, m + 1) * math.pi / (2 * (m + 1))) ** 2 if m > 1 else np.zeros(1) for m in (nx, ny, nz)]
    return np.sort((s[0][:, None, None] + s[1][None, :, None] + s[2][None, None, :]).ravel())


def _slice(nx, ny, nz, lo, count):
    """([a, b, lmin, lmax], eigenvalues inside) of a slice of about `count`
    eigenvalues from `lo` on, whose ends lie in gaps wide enough that no
    rounding moves an eigenvalue across them."""
    ev = _spectrum(nx, ny, nz)
    gap = np.diff(ev)
    wide = np.flatnonzero(gap > 0.3 * (ev[-1] - ev[0]) / len(ev))
    i0 = wide[min(np.searchsorted(wide, max(np.searchsorted(ev, lo) - 1, 0)), len(wide) - 2)]
    i1 = wide[min(np.searchsorted(wide, min(i0 + count, len(ev) - 2)), len(wide) - 1)]
    a, b = (float(0.5 * (ev[i] + ev[i + 1])) for i in (i0, i1))
    return [a, b, 0.0, 8.0 if nz == 1 else 12.0], ev[i0 + 1:i1 + 1]


def _instances(case):
    """The engine case's operators and slices: [((nx, ny, nz), intv, eigenvalues)]."""
    rng = np.random.default_rng(case["grids"])
    out = []
    for i in range(case["instances"]):
        n = int(np.exp(rng.uniform(np.log(case["nmin"]), np.log(case["nmax"]))))
        if i % 2 == 0:
            s = max(int(round(math.sqrt(n))), 10)
            dims = (s + 2, s - 3 - i % 3, 1)
        else:
            s = max(int(round(n ** (1 / 3))), 8)
            dims = (s + 1, s, s - 2)
        intv, ev = _slice(*dims, float(rng.uniform(0.3, 1.5)), int(rng.integers(case["kmin"], case["kmax"] + 1)))
        out.append((dims, intv, ev))
    return out


class _Served:
    """The resident matrices, requests and engine of a serving program."""

    def __init__(self, lib, case, seed):
        self.lib, self.mats, self.reqs = lib, [], []
        rng = np.random.default_rng(seed)
        for dims, intv, _ in _instances(case):
            M = lib.matrix(*workloads.laplacian_csr(*dims))
            self.mats.append(M)
            pol = lib.find_pol(intv, damping=2, thresh_int=0.8, thresh_ext=0.2, max_deg=3000)
            v = rng.standard_normal(M.n)
            self.reqs.append((M, intv, pol, v / np.linalg.norm(v)))
        self.eng = lib.engine(len(self.mats), precision=evsl_b200.PREC_FP64)

    def __del__(self):
        self.eng.free()
        for M, _, pol, _ in self.reqs:
            M.free()
            self.lib.free_pol(pol)


# ---------------------------------------------------------------------------
# prepare, run
# ---------------------------------------------------------------------------
def _vectors(case, seed, count):
    """`count` Gaussian vectors (rows), seeded, as double on the device."""
    g = torch.Generator(device=DEVICE).manual_seed(int(seed))
    return torch.randn(count, _rows(case), dtype=torch.float64, device=DEVICE, generator=g)


def prepare(case, seed):
    lib, kind = _library(), case["kind"]
    if kind == "engine":
        return dict(case=case, lib=lib, served=_Served(lib, case, seed))
    s = dict(case=case, lib=lib, keep=_register(lib, case), n=_rows(case))
    if kind in ("nr", "tr"):
        s["intv"], ev = _slice(case["nx"], case["ny"], case["nz"], case["lo"], case["count"])
        s["pol"] = lib.find_pol(s["intv"], damping=2, thresh_int=0.8, thresh_ext=0.2, max_deg=3000)
        v = np.random.default_rng(seed).standard_normal(s["n"])
        s["v"] = v / np.linalg.norm(v)
        s["nev"] = len(ev) + 4
        return s
    m = {"filter": 1, "kpm": case.get("nvec")}.get(kind, case.get("ncols"))
    s["x"] = _vectors(case, seed, m)
    if kind == "kpm":
        # the default fraction of the spectrum that is sliced in the benchmarks
        s["intv"] = (C.c_double * 4)(0.6, 1.2, *_bounds(case))
        return s
    s["y"] = torch.empty_like(s["x"])
    if kind == "multi":
        made = [_polynomial(case, d, g) for d, g in _column_filters(case)]
        s["pols"], s["mu"] = (evsl_b200.PolParams * m)(*[p for p, _ in made]), [c for _, c in made]
    else:
        s["pol"], s["mu"] = _polynomial(case, case["deg"], -0.87)
        s["work"] = torch.empty(3 if kind == "filter" else 2 * m, s["n"], dtype=torch.float64, device=DEVICE)
    return s


def run(s):
    case, lib = s["case"], s["lib"]
    kind, c = case["kind"], lib.lib
    if kind == "filter":
        _ok(lib, c.ChebAv(C.byref(s["pol"]), s["x"].data_ptr(), s["y"].data_ptr(), s["work"].data_ptr()))
        return s["y"]
    if kind == "block":
        _ok(lib, c.evslx_chebav_block(C.byref(s["pol"]), case["ncols"], s["x"].data_ptr(), s["y"].data_ptr(),
                                      s["work"].data_ptr()))
        return s["y"]
    if kind == "multi":
        prec = evsl_b200.PREC_MIXED if case["mixed"] else evsl_b200.PREC_FP64
        _ok(lib, c.evslx_chebav_multi(case["ncols"], s["pols"], s["x"].data_ptr(), s["y"].data_ptr(), prec))
        return s["y"]
    if kind == "kpm":
        mu, count = np.zeros(case["moments"] + 1), C.c_double()
        _ok(lib, c.evslx_kpmdos_probes(case["moments"], case["damping"], case["nvec"], s["intv"], s["x"].data_ptr(),
                                       mu.ctypes.data_as(C.POINTER(C.c_double)), C.byref(count)))
        return {"mu": mu, "count": count.value}
    if kind == "engine":
        sv = s["served"]
        for tag, (M, intv, pol, v) in enumerate(sv.reqs):
            sv.eng.submit_slice(M, intv, pol, 1000, TOL, v, tag)
        sv.eng.run()
        got = {}
        while (r := sv.eng.pop()) is not None:
            got[r["tag"]] = r
        # the residuals that come along are the rounding noise of converged pairs
        return {"nev": np.array([got[t]["nev"] for t in range(len(sv.reqs))]),
                "lam": np.concatenate([np.sort(got[t]["lam"]) for t in range(len(sv.reqs))])}
    if kind == "nr":
        lam, Y, _ = lib.cheblan_nr(s["intv"], case["maxit"], TOL, s["v"], s["pol"], want_vectors=case["vectors"])
    else:
        lam, Y, _ = lib.cheblan_tr(int(min(s["n"], 4 * s["nev"])), s["nev"], s["intv"], case["maxit"], TOL, s["v"],
                                   s["pol"], want_vectors=case["vectors"])
    # pairs come in the order of the filter's values; a program sorts them
    order = np.argsort(lam)
    if not case["vectors"]:
        return {"lam": lam[order]}
    Y = Y[order]
    return {"lam": lam[order], "Y": Y * np.sign(Y[:, :1])}  # a vector's sign is free: first entry positive


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _entries(case):
    """Stored entries of the case's matrix (random: expected)."""
    if "random" in case:
        return (2 * case["offdiag"] + 1) * case["random"]
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    n = nx * ny * nz
    return n + 2 * (n - n // nx) + 2 * (n - n // ny) + 2 * (n - n // nz)


def work(case):
    kind = case["kind"]
    if kind == "engine":
        # the requests' operators and start vectors in, their eigenvalues out; a
        # slice needs about 4 Lanczos steps for each of its eigenvalues
        b = f = 0.0
        for (nx, ny, nz), intv, ev in _instances(case):
            sub = dict(nx=nx, ny=ny, nz=nz)
            b += 12.0 * _entries(sub) + 4.0 * _rows(sub) + 8.0 * _rows(sub) + 8.0 * len(ev)
            f += _solve_flops(sub, intv, len(ev))
        return {"bytes": b, "flops": f}
    n, z = float(_rows(case)), float(_entries(case))
    a = 12.0 * z + 4.0 * n  # the matrix, read once
    if kind == "filter":
        return {"bytes": a + 16.0 * n, "flops": case["deg"] * (2.0 * z + 6.0 * n)}
    if kind in ("block", "multi"):
        degs = [d for d, _ in _column_filters(case)] if kind == "multi" else [case["deg"]] * case["ncols"]
        return {"bytes": a + 16.0 * n * case["ncols"], "flops": sum(degs) * (2.0 * z + 6.0 * n)}
    if kind == "kpm":
        steps = (case["moments"] + 1) // 2
        return {"bytes": a + 8.0 * n * case["nvec"] + 8.0 * case["moments"],
                "flops": steps * case["nvec"] * (2.0 * z + 8.0 * n)}
    intv, ev = _slice(case["nx"], case["ny"], case["nz"], case["lo"], case["count"])
    return {"bytes": a + 8.0 * n + 8.0 * len(ev) + (8.0 * n * len(ev) if case["vectors"] else 0.0),
            "flops": _solve_flops(case, intv, len(ev))}


def _solve_flops(case, intv, nev):
    """Filtered Lanczos to about 4 steps per eigenvalue: the filters (a slice
    of relative width w takes a degree near 5 / w), orthogonalisation against
    the growing basis and the Ritz vectors."""
    n, z, steps = float(_rows(case)), float(_entries(case)), 4.0 * nev
    deg = min(3000.0, 5.0 * (intv[3] - intv[2]) / (intv[1] - intv[0]) / 2)
    return steps * deg * (2.0 * z + 6.0 * n) + 2.0 * n * steps * steps + 2.0 * n * steps * nev


# ---------------------------------------------------------------------------
# the same in plain 64-bit arithmetic
# ---------------------------------------------------------------------------
def _plain_matrix(case):
    """The case's matrix as a torch sparse CSR tensor, built from its definition."""
    if "random" in case:
        ia, ja, a, _ = _random_csr(case["random"], case["offdiag"])
        return torch.sparse_csr_tensor(ia, ja, a, size=(case["random"],) * 2)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    n = nx * ny * nz
    at = torch.arange(n, device=DEVICE)
    x, y, z = at % nx, at // nx % ny, at // (nx * ny)
    row, col, val = [at], [at], [torch.full((n,), 6.0 if nz > 1 else 4.0, dtype=torch.float64, device=DEVICE)]
    for p, size, step in ((x, nx, 1), (y, ny, nx), (z, nz, nx * ny)):
        for inside, off in ((p > 0, -step), (p < size - 1, step)):
            row.append(at[inside])
            col.append(at[inside] + off)
            val.append(torch.full((row[-1].numel(),), -1.0, dtype=torch.float64, device=DEVICE))
    return torch.sparse_coo_tensor(torch.stack([torch.cat(row), torch.cat(col)]), torch.cat(val), (n, n)).to_sparse_csr()


def _plain_filter(A, cc, dd, mu, x):
    """sum_k mu[k, c] T_k((A - cc) / dd) x[c] for the rows x[c]; mu padded with zeros."""
    def op(v):
        return (A @ v - cc * v) / dd

    v0 = x.T.contiguous()
    v1 = op(v0)
    out = mu[0] * v0 + mu[1] * v1
    for k in range(2, mu.shape[0]):
        v0, v1 = v1, 2 * op(v1) - v0
        out += mu[k] * v1
    return out.T.contiguous()


def _plain_moments(case, A, x):
    """KPM moments and eigenvalue count of the probes x[p], one dot with the
    probe per degree."""
    M, nvec, n = case["moments"], case["nvec"], _rows(case)
    lmin, lmax = _bounds(case)
    cc, dd = (lmax + lmin) / 2, (lmax - lmin) / 2
    v = (x / x.norm(dim=1, keepdim=True)).T.contiguous()
    v0, v1, dots = v, (A @ v - cc * v) / dd, []
    for _ in range(M):
        dots.append(torch.sum(v1 * v).item())
        v0, v1 = v1, 2 * (A @ v1 - cc * v1) / dd - v0
    k = np.arange(1, M + 1)
    if case["damping"] == 1:  # Jackson
        th = math.pi / (M + 2)
        g = np.sin((k + 1) * th) / ((M + 2) * math.sin(th)) + (1 - (k + 1) / (M + 2)) * np.cos(k * th)
    else:  # Lanczos sigma
        th = math.pi / (M + 1)
        g = np.sin(k * th) / (k * th)
    t = 2 * g * np.array(dots)
    b1, b2 = (math.acos((e - cc) / dd) for e in (0.6, 1.2))
    count = -(nvec * (b2 - b1) + np.sum(t * (np.sin(k * b2) - np.sin(k * b1)) / k)) * n / (nvec * math.pi)
    return {"mu": np.concatenate([[nvec], t]) / (nvec * math.pi), "count": float(count)}


def exact(case, seed):
    kind = case["kind"]
    if kind == "engine":
        # [4 sin^2 sums of the grids]: the eigenvalues in the slices, by definition
        evs = [ev for _, _, ev in _instances(case)]
        return {"nev": None, "lam": np.concatenate(evs)}
    if kind in ("nr", "tr"):
        out = {"lam": _slice(case["nx"], case["ny"], case["nz"], case["lo"], case["count"])[1]}
        if case["vectors"]:
            out["Y"] = _plain_vectors(case["nx"], case["ny"], out["lam"])
        return out
    lmin, lmax = _bounds(case)
    x = _vectors(case, seed, {"filter": 1, "kpm": case.get("nvec")}.get(kind, case.get("ncols")))
    A = _plain_matrix(case)
    if kind == "kpm":
        return _plain_moments(case, A, x)
    cols = _column_filters(case) if kind == "multi" else [(case["deg"], -0.87)] * x.shape[0]
    mu = np.zeros((1 + max(d for d, _ in cols), len(cols)))
    for c, (d, g) in enumerate(cols):
        mu[:d + 1, c] = _coefficients(d, g)
    return _plain_filter(A, (lmax + lmin) / 2, (lmax - lmin) / 2, torch.from_numpy(mu).to(DEVICE), x)


def _plain_vectors(nx, ny, lam):
    """Unit eigenvectors of the 2-D Laplacian for its (simple) eigenvalues
    `lam`, the first entry of each positive: products of sines."""
    sx = 4 * np.sin(np.arange(1, nx + 1) * math.pi / (2 * (nx + 1))) ** 2
    sy = 4 * np.sin(np.arange(1, ny + 1) * math.pi / (2 * (ny + 1))) ** 2
    out = []
    for v in lam:
        j, i = np.unravel_index(np.argmin(np.abs(sy[:, None] + sx[None, :] - v)), (ny, nx))
        u = np.outer(np.sin((j + 1) * math.pi * np.arange(1, ny + 1) / (ny + 1)),
                     np.sin((i + 1) * math.pi * np.arange(1, nx + 1) / (nx + 1))).ravel()
        out.append(u / np.linalg.norm(u))
    return np.array(out)  # sin(i pi / (nx + 1)) > 0: first entries are positive
