"""The filter on a matrix's merged stencil (stencil.cu) gives the filtered
vector of the general kernels bit for bit."""
import ctypes as C

import numpy as np
import pytest

import evsl_b200 as E
from oracle import evsl_oracle as O

pytestmark = pytest.mark.gpu


def stencil_csr(n, entries, drop=0):
    """CSR of n rows holding `entries` (offset, value) where the column exists;
    with `drop`, row r leaves out entry (r % drop) when that is not the first."""
    r = np.arange(n, dtype=np.int64)
    rows, cols, vals = [], [], []
    for e, (off, v) in enumerate(sorted(entries)):
        keep = (r + off >= 0) & (r + off < n)
        if drop and e > 0:
            keep &= (r % drop) != e
        rows.append(r[keep])
        cols.append(r[keep] + off)
        vals.append(np.full(int(keep.sum()), v))
    rows, cols, vals = map(np.concatenate, (rows, cols, vals))
    order = np.lexsort((cols, rows))
    ia = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(rows, minlength=n), out=ia[1:])
    return ia.astype(np.int32), cols[order].astype(np.int32), vals[order]


def box9(nx):
    return [(i + nx * j, 0.1 * i + j + 3.0) for j in (-1, 0, 1) for i in (-1, 0, 1)]


def box27(nx, nxy):
    return [(i + nx * j + nxy * k, 0.01 * (i + 2 * j + 5 * k) + (7.0 if i == j == k == 0 else -0.2))
            for k in (-1, 0, 1) for j in (-1, 0, 1) for i in (-1, 0, 1)]


SHAPES = {
    # name: (rows, entries, drop); widths 5, 7, 9, 16 and 32, masks of 1, 2 and 4 bytes
    "one-row": (1, [(0, 2.5)], 0),
    "tridiagonal": (257, [(-1, -1.0), (0, 2.0), (1, -1.0)], 0),
    "line-255": (255, [(-40, -1.0), (-1, -1.0), (0, 4.0), (1, -1.0), (40, -1.0)], 0),
    "plane-7": (5003, [(-400, -1.0), (-20, -0.5), (-1, -1.0), (0, 6.1), (1, -1.0), (20, -0.5), (400, -1.0)], 0),
    "dropped-7": (4099, [(-400, -1.0), (-20, -0.5), (-1, -1.0), (0, 6.1), (1, -1.0), (20, -0.5), (400, -1.0)], 7),
    "lopsided": (3001, [(-7, 0.3), (0, 2.0), (5, 0.7), (90, -0.4)], 0),
    "no-diagonal": (1000, [(-3, 0.3), (-1, 0.6), (1, 0.6), (3, 0.3)], 0),
    "box-9": (6007, box9(60), 0),
    "eleven": (2048, [(o, 0.1 * o + 1.0) for o in range(-5, 6)], 6),
    "box-27": (9001, box27(20, 400), 0),
    "thirty-two": (3000, [(o, 1.0 / (40 + o)) for o in range(-16, 16)], 0),
    # the rows of a cluster's blocks fall on and around their edges
    "cluster-exact": (16 * 96, [(-96, -1.0), (-1, -1.0), (0, 4.0), (1, -1.0), (96, -1.0)], 0),
    "cluster-over": (16 * 96 + 1, [(-96, -1.0), (-1, -1.0), (0, 4.0), (1, -1.0), (96, -1.0)], 0),
    "cluster-halo-rows": (700, [(-200, -1.0), (-1, -1.0), (0, 4.0), (1, -1.0), (200, -1.0)], 0),
    "cluster-loop": (13000, [(-777, -1.0), (-9, -1.0), (-1, -1.0), (0, 6.0), (1, -1.0), (9, -1.0), (777, -1.0)], 0),
    "cluster-y-global": (122000, [(-3300, -1.0), (-1, -1.0), (0, 4.0), (1, -1.0), (3300, -1.0)], 0),
    # rows past the size where a thread takes two rows an offset apart
    "two-rows-5": (150001, [(-387, -1.0), (-1, -1.0), (0, 4.0), (1, -1.0), (387, -1.0)], 0),
    "two-rows-7": (160003, [(-2900, -1.0), (-53, -1.0), (-1, -1.0), (0, 6.0), (1, -1.0), (53, -1.0), (2900, -1.0)], 0),
    "two-rows-dropped": (151000, [(-900, -1.0), (-30, 0.2), (-1, -1.0), (0, 6.0), (1, -1.0), (30, 0.2), (900, -1.0)], 7),
    "two-rows-9": (155555, box9(400), 0),
    # five FP32 columns together are more than one wave of blocks
    "two-rows-fp32-9": (57601, box9(240), 0),
    "two-rows-fp32-dropped": (50001, [(-900, -1.0), (-30, 0.2), (-1, -1.0), (0, 6.0), (1, -1.0), (30, 0.2), (900, -1.0)], 7),
    # one column's threads take two rows from one wave of blocks on (227,328 rows)
    "one-wave-7": (227328, [(-2900, -1.0), (-53, -1.0), (-1, -1.0), (0, 6.0), (1, -1.0), (53, -1.0), (2900, -1.0)], 0),
    "over-one-wave-7": (227329, [(-2900, -1.0), (-53, -1.0), (-1, -1.0), (0, 6.0), (1, -1.0), (53, -1.0), (2900, -1.0)], 0),
    "over-one-wave-5-dropped": (231001, [(-487, -1.0), (-1, 0.3), (0, 4.0), (1, 0.3), (487, -1.0)], 5),
    "over-one-wave-9": (230400, box9(480), 0),
    # the march's stride is more than half the rows: one row per thread again
    "wide-offset-one-column": (230001, [(-120000, -1.0), (-1, -1.0), (0, 4.0), (1, -1.0), (120000, -1.0)], 0),
    "wide-offset": (150100, [(-80000, -1.0), (-1, -1.0), (0, 4.0), (1, -1.0), (80000, -1.0)], 0),
}


def polynomial(lib, deg, bound):
    """A polparams of exactly `deg` with seeded coefficients (and their array)."""
    pol = E.PolParams()
    lib.lib.set_pol_def(C.byref(pol))
    mu = np.random.default_rng(deg).standard_normal(deg + 1)
    pol.mu = mu.ctypes.data_as(C.POINTER(C.c_double))
    pol.deg, pol.cc, pol.dd = deg, 0.1 * bound, bound
    return pol, mu


# one launch per degree, and one cluster of the largest, a middle and the
# smallest size (stencils too wide or too long for a cluster take the former)
@pytest.mark.parametrize("blocks", [-1, 0, 4, 1])
@pytest.mark.parametrize("shape", sorted(SHAPES))
def test_stencil_filter_is_bitwise(gpu_lib, shape, blocks):
    n, entries, drop = SHAPES[shape]
    ia, ja, a = stencil_csr(n, entries, drop)
    gpu_lib.set_csr(ia, ja, a)
    assert gpu_lib.row_pattern_count() > 0
    v = O.seeded_normal(n, 3)
    bound = max(np.abs(a).max() * len(entries), 1.0)
    # degrees 1 to 8: every remainder of the three-degree update of y, at the
    # first and at a later write
    for deg in range(1, 9):
        pol, mu = polynomial(gpu_lib, deg, bound)
        try:
            gpu_lib.lib.evslcu_set_stencil_cluster(blocks)
            gpu_lib.set_filter_kernel("merged-stencil")
            y = gpu_lib.chebav(pol, v)
            gpu_lib.set_filter_kernel(0)  # SELL storage, pinned to the oracle elsewhere
            assert np.array_equal(y, gpu_lib.chebav(pol, v)), deg
        finally:
            gpu_lib.set_filter_kernel(-1)
            gpu_lib.lib.evslcu_set_stencil_cluster(0)


def test_dictionaries_that_do_not_merge_keep_the_other_kernels(gpu_lib):
    """More than 32 entries, and rows whose columns do not increase: the filter,
    the products, several columns (against the SELL kernel) and KPM (against the
    matrix without its dictionary, with the tolerance of test_kpm_on_stencils,
    and bitwise with the prefetching form)."""
    wide = stencil_csr(2000, [(o, 1.0 / (50 + o)) for o in range(-20, 21)])
    ia, ja, a = stencil_csr(2000, [(-30, -1.0), (-1, -1.0), (0, 4.0), (1, -1.0), (30, -1.0)])
    ja, a = ja.copy(), a.copy()
    for r in range(0, 2000, 2):
        ja[ia[r]:ia[r + 1]] = ja[ia[r]:ia[r + 1]][::-1]
        a[ia[r]:ia[r + 1]] = a[ia[r]:ia[r + 1]][::-1]
    iv = [0.4, 2.9, -8.0, 8.0]
    X = O.seeded_normal(3 * 2000, 3).reshape(3, 2000)
    dX = E.DeviceBuffer.from_host(gpu_lib.lib, X)
    pol, mu = polynomial(gpu_lib, 7, 8.0)
    try:
        for m in (wide, (ia, ja, a)):
            gpu_lib.set_csr(*m)
            assert gpu_lib.row_pattern_count() > 0 and not gpu_lib.filter_stencil()
            assert np.array_equal(gpu_lib.chebav(pol, X[0]), O.cheb_av(pol.as_dict(), *m, X[0]))
            Y = gpu_lib.matvec_cols(X)
            for c in range(3):
                assert np.array_equal(Y[c], O.csr_matvec(*m, X[c]))
                assert np.array_equal(Y[c], gpu_lib.matvec(X[c]))
            for prec in (E.PREC_FP64, E.PREC_MIXED):
                Y = gpu_lib.chebav_multi([pol] * 3, X, prec)
                gpu_lib.set_filter_variant(0)
                assert np.array_equal(Y, gpu_lib.chebav_multi([pol] * 3, X, prec)), prec
                gpu_lib.set_filter_variant(-1)
            dots = gpu_lib.kpm_dots(21, iv, dX, 3)
            gpu_lib.lib.evslcu_set_kpm_prefetch(1)
            assert np.array_equal(dots, gpu_lib.kpm_dots(21, iv, dX, 3))
            gpu_lib.lib.evslcu_set_kpm_prefetch(0)
            gpu_lib.set_row_patterns(False)
            gpu_lib.set_csr(*m)
            assert np.max(np.abs(dots - gpu_lib.kpm_dots(21, iv, dX, 3))) <= 4 * 2000 * np.finfo(float).eps
            gpu_lib.set_row_patterns(True)
    finally:
        gpu_lib.set_filter_variant(-1)
        gpu_lib.lib.evslcu_set_kpm_prefetch(0)
        gpu_lib.set_row_patterns(True)


MULTI = ["cluster-over", "dropped-7", "eleven", "box-9", "lopsided", "two-rows-5", "two-rows-dropped",
         "two-rows-fp32-9", "two-rows-fp32-dropped"]


@pytest.mark.parametrize("blocks", [-1, 0])
@pytest.mark.parametrize("prec", [E.PREC_FP64, E.PREC_MIXED])
@pytest.mark.parametrize("shape", MULTI)
def test_stencil_columns_are_bitwise(gpu_lib, shape, prec, blocks):
    """Several columns with their own polynomials (degrees 1 to 9, so that
    columns end at different launches; 17 columns: two groups) equal the
    interleaved SELL-32 kernel's, in both precisions."""
    n, entries, drop = SHAPES[shape]
    gpu_lib.set_csr(*stencil_csr(n, entries, drop))
    bound = max(max(abs(v) for _, v in entries) * len(entries), 1.0)
    ncols = 17 if n < 20000 else 5
    X = O.seeded_normal(n * ncols, 4).reshape(ncols, n)
    made = [polynomial(gpu_lib, 1 + (5 * c) % 9, bound) for c in range(ncols)]
    pols = [p for p, _ in made]
    try:
        gpu_lib.lib.evslcu_set_stencil_cluster(blocks)
        gpu_lib.set_filter_variant(8)
        Y = gpu_lib.chebav_multi(pols, X, prec)
        gpu_lib.set_filter_variant(0)
        assert np.array_equal(Y, gpu_lib.chebav_multi(pols, X, prec))
    finally:
        gpu_lib.set_filter_variant(-1)
        gpu_lib.lib.evslcu_set_stencil_cluster(0)


def test_engine_batch_of_stencils_of_all_widths(gpu_lib):
    """Operators with masks of one and of two bytes, with and without a cluster,
    in one engine: the same eigenvalues as with each matrix's own filter."""
    box = [(o, -1.0 if o else 8.5) for o, _ in box9(33)]
    five = [(-40, -1.0), (-1, -1.0), (0, 4.2), (1, -1.0), (40, -1.0)]
    seven = [(-300, -1.0), (-17, -1.0), (-1, -1.0), (0, 6.4), (1, -1.0), (17, -1.0), (300, -1.0)]
    wide = [(o, -0.1 if o else 2.0) for o in range(-6, 7)]
    ops = [(1103, box, 16.5), (2000, five, 8.2), (5001, seven, 12.4), (900, wide, 3.2), (700, five, 8.2), (1500, box, 16.5)]
    mats = [gpu_lib.matrix(*stencil_csr(n, e)) for n, e, _ in ops]
    iv = [[0.30 * top, 0.31 * top, 0.0, top] for _, _, top in ops]
    pols = [gpu_lib.find_pol(i, max_deg=300) for i in iv]
    out = []
    for batch in (True, False):
        eng = gpu_lib.engine(len(ops), precision=E.PREC_FP64)
        eng.use_batch(batch)
        for t, (n, _, _) in enumerate(ops):
            eng.submit_slice(mats[t], iv[t], pols[t], 120, 1e-8, O.seeded_normal(n, t), t)
        eng.run()
        got = {}
        while (r := eng.pop()) is not None:
            got[r["tag"]] = r["lam"]
        eng.free()
        out.append(got)
    assert len(out[0]) == len(ops)
    for t in out[0]:
        assert np.array_equal(out[0][t], out[1][t]), t
    for m in mats:
        m.free()
    for p in pols:
        gpu_lib.free_pol(p)


@pytest.mark.parametrize("shape", ["cluster-over", "cluster-halo-rows", "cluster-loop"])
def test_long_filters_on_a_cluster_are_bitwise(gpu_lib, shape):
    """Degrees around the sizes at which a cluster filter's coefficients change
    place (63 and 511 in the launch's arguments, more on the device), with every
    remainder of the loop over three degrees."""
    n, entries, drop = SHAPES[shape]
    ia, ja, a = stencil_csr(n, entries, drop)
    gpu_lib.set_csr(ia, ja, a)
    v = O.seeded_normal(n, 3)
    try:
        for deg in (10, 35, 63, 64, 65, 511, 512, 700):
            pol, mu = polynomial(gpu_lib, deg, 1.2 * sum(abs(v) for _, v in entries))
            gpu_lib.set_filter_kernel("merged-stencil")
            before = gpu_lib.launch_count()
            y = gpu_lib.chebav(pol, v)
            assert gpu_lib.launch_count() - before == 1
            gpu_lib.set_filter_kernel(0)
            assert np.array_equal(y, gpu_lib.chebav(pol, v)), deg
    finally:
        gpu_lib.set_filter_kernel(-1)


def test_engine_batch_with_halos_of_most_of_a_block(gpu_lib):
    """Operators whose largest offset is a third to a half of their rows, beside
    one with short offsets, filtered together on clusters: the same eigenvalues
    as with each matrix's own filter."""
    five = lambda s: [(-s, -1.0), (-1, -1.0), (0, 4.2), (1, -1.0), (s, -1.0)]  # noqa: E731
    ops = [(700, five(230)), (1003, five(480)), (1600, five(40)), (2048, five(1000))]
    mats = [gpu_lib.matrix(*stencil_csr(n, e)) for n, e in ops]
    iv = [3.0, 3.1, 0.0, 8.4]
    pol = gpu_lib.find_pol(iv, max_deg=300)
    out = []
    for batch in (True, False):
        eng = gpu_lib.engine(len(ops), precision=E.PREC_FP64)
        eng.use_batch(batch)
        for t, (n, _) in enumerate(ops):
            eng.submit_slice(mats[t], iv, pol, 200, 1e-8, O.seeded_normal(n, t), t)
        eng.run()
        got = {}
        while (r := eng.pop()) is not None:
            got[r["tag"]] = r["lam"]
        assert (eng.batched_columns() > 0) == batch
        eng.free()
        out.append(got)
    assert len(out[0]) == len(ops) and sum(len(lam) for lam in out[0].values()) > 0
    for t in out[0]:
        assert np.array_equal(out[0][t], out[1][t]), t
    for m in mats:
        m.free()
    gpu_lib.free_pol(pol)


@pytest.mark.parametrize("blocks", [-1, 0, 1])
@pytest.mark.parametrize("shape", ["one-row", "tridiagonal", "cluster-over", "cluster-loop", "dropped-7", "eleven",
                                   "box-9", "two-rows-7"])
def test_kpm_on_stencils(gpu_lib, shape, blocks):
    """KPM sums on a merged stencil agree with the CSR kernel's to the rounding
    of sums of n products of unit vectors (|dots| <= 1: n eps, times 2 for the
    product identity and 2 for either side), and a probe's do not depend on
    the probes beside it."""
    n, entries, drop = SHAPES[shape]
    m = stencil_csr(n, entries, drop)
    bound = max(max(abs(v) for _, v in entries) * len(entries), 1.0)
    iv, M, nvec = [-0.2 * bound, 0.4 * bound, -bound, bound], 21, 7
    X = O.seeded_normal(n * nvec, 6).reshape(nvec, n)
    try:
        gpu_lib.lib.evslcu_set_stencil_cluster(blocks)
        gpu_lib.set_csr(*m)
        got = gpu_lib.kpm_dots(M, iv, E.DeviceBuffer.from_host(gpu_lib.lib, X), nvec)
        parts = [gpu_lib.kpm_dots(M, iv, E.DeviceBuffer.from_host(gpu_lib.lib, np.ascontiguousarray(X[a:b])), b - a)
                 for a, b in ((0, 1), (1, 6), (6, 7))]
        assert np.array_equal(got, np.concatenate(parts, axis=1))
        gpu_lib.set_row_patterns(False)
        gpu_lib.set_csr(*m)
        ref = gpu_lib.kpm_dots(M, iv, E.DeviceBuffer.from_host(gpu_lib.lib, X), nvec)
        assert np.max(np.abs(got - ref)) <= max(4 * n, 1000) * np.finfo(float).eps
    finally:
        gpu_lib.set_row_patterns(True)
        gpu_lib.lib.evslcu_set_stencil_cluster(0)


@pytest.mark.parametrize("shape", ["over-one-wave-7", "cluster-over"])
def test_filter_right_after_registration_on_the_device(gpu_lib, shape):
    """SetAMatrix_device_csr, then ChebAv on device vectors with nothing in
    between: the filter's first loads see the masks of the matrix just
    registered, not of the one before it (the pool gives both the same
    memory)."""
    n, entries, _ = SHAPES[shape]
    lib = gpu_lib.lib
    bound = sum(abs(v) for _, v in entries)
    pol, mu = polynomial(gpu_lib, 5, bound)
    v = O.seeded_normal(n, 3)
    dv, dy, dw = (E.DeviceBuffer.from_host(lib, a) for a in (v, v, np.zeros(3 * n)))
    full, thin = stencil_csr(n, entries), stencil_csr(n, entries, 3)
    refs = [O.cheb_av(pol.as_dict(), *m, v) for m in (full, thin)]
    try:
        lib.evslcu_set_stencil_cluster(-1)
        for i in range(12):
            gpu_lib.set_csr_device(*((full, thin)[i % 2]))
            assert lib.ChebAv(C.byref(pol), dv.ptr, dy.ptr, dw.ptr) == 0
            assert np.array_equal(dy.to_host(), refs[i % 2]), i
    finally:
        lib.evslcu_set_stencil_cluster(0)


@pytest.mark.parametrize("call", ["filter", "lanczos", "columns", "columns-fp32", "kpm", "engine"])
def test_cluster_waits_run_out_and_library_recovers(gpu_lib, call):
    """With a limit of one poll the blocks of the cluster kernels give up on
    their neighbours' rows: the call returns EVSLX_ERR_TIMEOUT (-105) with every
    block gone, and with the default limit the same call gives its result of
    before, bit for bit."""
    ia, ja, a = O.lap_csr(101, 97, 1)
    n = len(ia) - 1
    gpu_lib.set_csr(ia, ja, a)
    X = O.seeded_normal(4 * n, 8).reshape(4, n)
    iv = [0.5, 0.6, 0.0, 8.0]
    pol = gpu_lib.find_pol(iv)
    mat = gpu_lib.matrix(ia, ja, a)
    dX = E.DeviceBuffer.from_host(gpu_lib.lib, X)

    def engine():
        eng = gpu_lib.engine(1, precision=E.PREC_FP64)
        try:
            eng.submit_slice(mat, iv, pol, 400, 1e-8, X[0], 1)
            eng.run()
            return eng.pop()["lam"]
        finally:
            eng.free()

    run = {
        "filter": lambda: gpu_lib.chebav(pol, X[0]),
        "lanczos": lambda: gpu_lib.cheblan_nr(iv, 400, 1e-8, X[0], pol)[0],
        "columns": lambda: gpu_lib.chebav_multi([pol] * 4, X, E.PREC_FP64),
        "columns-fp32": lambda: gpu_lib.chebav_multi([pol] * 4, X, E.PREC_MIXED),
        "kpm": lambda: gpu_lib.kpm_dots(60, iv, dX, 4),
        "engine": engine,
    }[call]
    try:
        ref = run()
        assert len(ref) > 0 and np.all(np.isfinite(ref))
        gpu_lib.set_wait_limit(1)
        codes = []
        for _ in range(3):
            try:
                run()
                codes.append(0)
            except E.EvslError as e:
                codes.append(-105 if "returned -105" in str(e) else str(e))
                assert "within its bound" in gpu_lib.last_error()
        assert -105 in codes and all(c in (0, -105) for c in codes), codes
        gpu_lib.set_wait_limit(0)
        assert np.array_equal(run(), ref)
    finally:
        gpu_lib.set_wait_limit(0)
        mat.free()
        gpu_lib.free_pol(pol)


@pytest.mark.parametrize("blocks", [-1, 0])
@pytest.mark.parametrize("prec", [E.PREC_FP64, E.PREC_MIXED])
@pytest.mark.parametrize("shape", ["cluster-over", "two-rows-7"])
@pytest.mark.parametrize("shift", [0, 1, -1])
def test_columns_in_place(gpu_lib, shift, shape, prec, blocks):
    """Y on X itself, and each column's result on its neighbour's vector: the
    columns of separate vectors, degree 1 included."""
    n, entries, _ = SHAPES[shape]
    lib = gpu_lib.lib
    gpu_lib.set_csr(*stencil_csr(n, entries))
    bound = sum(abs(v) for _, v in entries)
    made = [polynomial(gpu_lib, deg, bound) for deg in (1, 2, 3, 1, 5)]
    pols = (E.PolParams * 5)(*[p for p, _ in made])
    X = O.seeded_normal(7 * n, 4).reshape(7, n)
    try:
        lib.evslcu_set_stencil_cluster(blocks)
        ref = gpu_lib.chebav_multi([p for p, _ in made], X[1:6], prec)
        buf = E.DeviceBuffer.from_host(lib, X)
        assert lib.evslx_chebav_multi(5, pols, buf.ptr + 8 * n, buf.ptr + 8 * n * (1 + shift), prec) == 0
        assert np.array_equal(buf.to_host(shape=X.shape)[1 + shift:6 + shift], ref)
    finally:
        lib.evslcu_set_stencil_cluster(0)


def test_forced_kernels_and_the_merged_stencil_are_told_apart(gpu_lib):
    """On a small grid the merged stencil filters in one launch and every other
    kernel in one per degree: forced, "merged-stencil" and the row-descriptor
    kernel are the ones that run, filter_stencil() says which is used, and a
    matrix without a merged stencil refuses it."""
    grid = O.lap_csr(40, 39, 1)
    wide = stencil_csr(2000, [(o, 1.0 / (50 + o)) for o in range(-20, 21)])
    pol, mu = polynomial(gpu_lib, 9, 8.0)

    def launches(kernel, v):
        gpu_lib.set_filter_kernel(kernel)
        gpu_lib.chebav(pol, v)  # (a first call may prepare the kernel's tables)
        before = gpu_lib.launch_count()
        gpu_lib.chebav(pol, v)
        return gpu_lib.launch_count() - before

    try:
        gpu_lib.set_csr(*grid)
        v = O.seeded_normal(1560, 3)
        assert gpu_lib.filter_stencil()
        assert launches(None, v) == 1 and launches("merged-stencil", v) == 1 and gpu_lib.filter_stencil()
        for kernel in ("sell-loop", "pattern-constant-rowdesc", "pattern-global-loop"):
            assert launches(kernel, v) == 9 and not gpu_lib.filter_stencil(), kernel
        gpu_lib.set_filter_kernel(None)
        gpu_lib.set_csr(*wide)
        assert gpu_lib.row_pattern_count() > 0 and not gpu_lib.filter_stencil()
        with pytest.raises(E.EvslError, match="not available"):
            launches("merged-stencil", O.seeded_normal(2000, 3))
    finally:
        gpu_lib.set_filter_kernel(None)


def _sets(n, offsets, sets):
    """Rows of `offsets`, the values one of `sets` multiples by row range."""
    ia, ja, a = stencil_csr(n, [(o, 5.0 if o == 0 else -1.0) for o in offsets])
    rows = np.repeat(np.arange(n), np.diff(ia))
    return ia, ja, a * (1.0 + 0.125 * (rows * sets // n))


LOOSE = {  # lists that no row has all of, and lists padded to the next width
    "six-sets": lambda n: _sets(n, (-97, -1, 0, 1, 97), 6),
    "two-sets": lambda n: _sets(n, (-97, -1, 0, 1, 97), 2),
    "tridiagonal": lambda n: _sets(n, (-1, 0, 1), 1),
    "thirteen": lambda n: _sets(n, range(-6, 7), 1),
    "box-27": lambda n: stencil_csr(n, box27(20, 400)),
}


@pytest.mark.parametrize("kind", sorted(LOOSE))
def test_loose_stencils_take_any_kernel_alike(gpu_lib, kind):
    """Operators whose stencil is timed among the other kernels: the filters and
    products of the default route equal the SELL kernels' and the oracle's, and
    KPM agrees with the general kernel's (the tolerance of test_kpm_on_stencils)."""
    n = 12001
    m = LOOSE[kind](n)
    gpu_lib.set_csr(*m)
    bound = float(np.abs(m[2]).max()) * 30
    X = O.seeded_normal(5 * n, 9).reshape(5, n)
    made = [polynomial(gpu_lib, deg, bound) for deg in (7, 4, 9, 2, 6)]
    pols = [p for p, _ in made]
    iv = [-0.2 * bound, 0.4 * bound, -bound, bound]
    dX = E.DeviceBuffer.from_host(gpu_lib.lib, X)
    try:
        assert np.array_equal(gpu_lib.chebav(pols[0], X[0]), O.cheb_av(pols[0].as_dict(), *m, X[0]))
        assert np.array_equal(gpu_lib.matvec(X[0]), O.csr_matvec(*m, X[0]))
        assert np.array_equal(gpu_lib.matvec_cols(X)[4], O.csr_matvec(*m, X[4]))
        for prec in (E.PREC_FP64, E.PREC_MIXED):
            Y = gpu_lib.chebav_multi(pols, X, prec)
            gpu_lib.set_filter_variant(0)
            assert np.array_equal(Y, gpu_lib.chebav_multi(pols, X, prec)), prec
            gpu_lib.set_filter_variant(-1)
        dots = gpu_lib.kpm_dots(20, iv, dX, 5)
        gpu_lib.set_row_patterns(False)
        gpu_lib.set_csr(*m)
        assert np.max(np.abs(dots - gpu_lib.kpm_dots(20, iv, dX, 5))) <= 4 * n * np.finfo(float).eps
    finally:
        gpu_lib.set_filter_variant(-1)
        gpu_lib.set_row_patterns(True)


def test_values_beyond_fp32_stay_in_their_rows(gpu_lib):
    """A value that is infinite in FP32, in the last rows only: FP32 columns are
    infinite or not a number where the general kernel's are, and equal elsewhere
    (an absent entry must not become 0 * inf)."""
    n = 2000
    ia, ja, a = stencil_csr(n, SHAPES["cluster-exact"][1])
    a = a.copy()
    a[ia[1900]:] *= 1e39
    gpu_lib.set_csr(ia, ja, a)
    made = [polynomial(gpu_lib, deg, 8.0) for deg in (3, 5)]
    pols = [p for p, _ in made]
    X = O.seeded_normal(2 * n, 4).reshape(2, n)
    try:
        Y = gpu_lib.chebav_multi(pols, X, E.PREC_MIXED)
        gpu_lib.set_filter_variant(0)
        ref = gpu_lib.chebav_multi(pols, X, E.PREC_MIXED)
    finally:
        gpu_lib.set_filter_variant(-1)
    assert np.array_equal(Y, ref, equal_nan=True)
    assert np.all(np.isfinite(Y[:, :1400])) and not np.any(np.isfinite(Y[:, 1900:]))


@pytest.mark.parametrize("columns", [1, 16])
def test_wide_lists_of_short_rows_do_not_take_the_stencil(gpu_lib, columns):
    """Six sets of coefficients make a list of 30 entries for rows of 5: the
    route taken is not the stencil, which costs about twice (16 columns) and
    three times (one) what the dictionary's kernel does."""
    import time

    n = 600000
    gpu_lib.set_csr(*_sets(n, (-775, -1, 0, 1, 775), 6))
    lib = gpu_lib.lib
    pol, mu = polynomial(gpu_lib, 40, 100.0)
    pols = (E.PolParams * columns)(*[pol] * columns)
    x, y = (E.DeviceBuffer.from_host(lib, np.zeros(n * columns)) for _ in range(2))
    w = E.DeviceBuffer(lib, 24 * n)

    def seconds(force):
        gpu_lib.set_filter_kernel("merged-stencil" if force else None)
        gpu_lib.set_filter_variant(8 if force else -1)
        best = np.inf
        for _ in range(4):
            t = time.perf_counter()
            if columns == 1:
                assert lib.ChebAv(C.byref(pol), x.ptr, y.ptr, w.ptr) == 0
            else:
                assert lib.evslx_chebav_multi(columns, pols, x.ptr, y.ptr, E.PREC_FP64) == 0
            best = min(best, time.perf_counter() - t)
        return best

    try:
        assert seconds(False) < 0.8 * seconds(True)
        gpu_lib.set_filter_kernel(None)
        assert columns > 1 or not gpu_lib.filter_stencil()
    finally:
        gpu_lib.set_filter_kernel(None)
        gpu_lib.set_filter_variant(-1)
