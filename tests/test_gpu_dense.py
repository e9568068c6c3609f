"""FP64 GEMM of the Ritz step (SRC/cheblanNr.c:333-399 forms the Ritz vectors
V(:,1:K) Y; evsl_dgemm_device is the reference's device BLAS entry point)
through the C ABI: the 128 x 128 tiled DFMA kernel (cp.async double
buffering, 8 x 8 accumulators per thread) against the 64 x 64 kernel -- both
form each entry as the FMA chain over k in order, so they agree bit for bit
-- and the default kernel on the FP64 tensor instruction against both and
numpy (1e-13 of the largest |C| entry): aligned and unaligned operands (odd
leading dimensions), ragged edges, beta 0 and 0.5.
"""
import ctypes as C
import os
import time

import numpy as np
import pytest

import evsl_b200

pytestmark = pytest.mark.gpu


def _gemm(lib, m, n, k, A, lda, B, ldb, Cm, ldc, alpha, beta, tiled):
    prev = lib.lib.evslcu_set_dgemm_tiled(int(tiled))
    dA = evsl_b200.DeviceBuffer.from_host(lib.lib, A)
    dB = evsl_b200.DeviceBuffer.from_host(lib.lib, B)
    dC = evsl_b200.DeviceBuffer.from_host(lib.lib, Cm)
    ci = lambda v: C.byref(C.c_int(v))  # noqa: E731
    cd = lambda v: C.byref(C.c_double(v))  # noqa: E731
    lib.lib.evsl_dgemm_device(b"N", b"N", ci(m), ci(n), ci(k), cd(alpha), C.c_void_p(dA.ptr), ci(lda),
                              C.c_void_p(dB.ptr), ci(ldb), cd(beta), C.c_void_p(dC.ptr), ci(ldc))
    out = dC.to_host(shape=Cm.shape)
    lib.lib.evslcu_set_dgemm_tiled(prev)
    return out


@pytest.mark.parametrize("m, n, k, pad", [(1000, 70, 333, 0), (1001, 64, 257, 0), (4096, 300, 1000, 0),
                                         (777, 129, 33, 3), (2048, 32, 16, 1), (513, 40, 1, 0)])
@pytest.mark.parametrize("beta", [0.0, 0.5])
def test_tiled_gemm_matches(gpu_lib, m, n, k, pad, beta):
    rng = np.random.default_rng(m + n + k)
    lda, ldb, ldc = m + pad, k + pad, m + pad
    A = rng.standard_normal((k, lda))  # column j of A is row j here (column-major storage)
    B = rng.standard_normal((n, ldb))
    C0 = rng.standard_normal((n, ldc))
    alpha = 1.0 if beta == 0.0 else -0.75
    got = _gemm(gpu_lib, m, n, k, A, lda, B, ldb, C0, ldc, alpha, beta, True)
    old = _gemm(gpu_lib, m, n, k, A, lda, B, ldb, C0, ldc, alpha, beta, False)
    assert np.array_equal(got, old)
    ref = alpha * (A[:, :m].T @ B[:, :k].T) + beta * C0[:, :m].T
    assert np.max(np.abs(got[:, :m].T - ref)) <= 1e-13 * np.max(np.abs(ref))
    # the padding rows of C are untouched
    assert np.array_equal(got[:, m:], C0[:, m:])


@pytest.mark.parametrize("n, m, b", [(20000, 100, 32), (5003, 45, 16), (40000, 33, 32)])
def test_block_cgs2_orthonormalises(gpu_lib, n, m, b):
    """Block Gram-Schmidt twice (the mixed-precision refinement's
    orthonormalisation; GEMM projections between blocks, CGS + DGKS as in
    SRC/misc_la.c:221-261 inside a block): the columns come out orthonormal to
    1e-13 and span the input columns (every input column is reproduced by its
    projection to 1e-12 of its norm), on well and badly conditioned inputs."""
    rng = np.random.default_rng(n + m)
    W0 = rng.standard_normal((m, n))  # row j = column j of the n x m block
    # a badly conditioned half: columns nearly dependent on the first ones
    W0[m // 2:] = W0[: m - m // 2] + 1e-6 * rng.standard_normal((m - m // 2, n))
    dW = evsl_b200.DeviceBuffer.from_host(gpu_lib.lib, W0)
    dH = evsl_b200.DeviceBuffer(gpu_lib.lib, 8 * m * m)
    dn = evsl_b200.DeviceBuffer(gpu_lib.lib, 8)
    gpu_lib.lib.evslcu_cgs_work_size.restype = C.c_size_t
    gpu_lib.lib.evslcu_cgs_work_size.argtypes = [C.c_int, C.c_int]
    work = evsl_b200.DeviceBuffer(gpu_lib.lib, 8 * int(gpu_lib.lib.evslcu_cgs_work_size(n, b)))
    fn = gpu_lib.lib.evslcu_block_cgs2
    fn.argtypes = [C.c_int, C.c_int, C.c_void_p, C.c_int, C.c_void_p, C.c_void_p, C.c_void_p]
    assert fn(n, m, dW.ptr, b, dH.ptr, dn.ptr, work.ptr) == 0
    Q = dW.to_host(shape=(m, n))
    G = Q @ Q.T
    assert np.max(np.abs(G - np.eye(m))) <= 1e-13
    P = (W0 @ Q.T) @ Q
    assert np.max(np.linalg.norm(W0 - P, axis=1) / np.linalg.norm(W0, axis=1)) <= 1e-12


@pytest.mark.parametrize("m, n, k, pad", [(1000, 70, 333, 0), (1001, 64, 257, 0), (4096, 300, 1000, 0),
                                         (777, 129, 33, 3), (2048, 32, 16, 1), (513, 40, 1, 0)])
@pytest.mark.parametrize("beta", [0.0, 0.5])
def test_mma_gemm_matches(gpu_lib, m, n, k, pad, beta):
    """The tall GEMM on the FP64 tensor instruction (mma.sync m8n8k4, same
    tiles and staging as the DFMA kernel, products summed in the
    instruction's order): within 1e-13 of numpy and of the DFMA kernel,
    aligned and unaligned operands, ragged edges, beta 0 and 0.5; the padding
    rows of C untouched."""
    rng = np.random.default_rng(m + 2 * n + k)
    lda, ldb, ldc = m + pad, k + pad, m + pad
    A = rng.standard_normal((k, lda))
    B = rng.standard_normal((n, ldb))
    C0 = rng.standard_normal((n, ldc))
    alpha = 1.0 if beta == 0.0 else -0.75
    got = _gemm(gpu_lib, m, n, k, A, lda, B, ldb, C0, ldc, alpha, beta, 2)
    dfma = _gemm(gpu_lib, m, n, k, A, lda, B, ldb, C0, ldc, alpha, beta, 1)
    ref = alpha * (A[:, :m].T @ B[:, :k].T) + beta * C0[:, :m].T
    scale = np.max(np.abs(ref))
    assert np.max(np.abs(got[:, :m].T - ref)) <= 1e-13 * scale
    assert np.max(np.abs(got - dfma)) <= 1e-13 * scale
    assert np.array_equal(got[:, m:], C0[:, m:])


@pytest.mark.parametrize("n, k", [(1, 1), (255, 7), (1025, 130), (40000, 17), (40001, 129), (80001, 33), (160001, 16),
                                 (3000, 2100)])
def test_gemv_of_every_column_split(gpu_lib, n, k):
    """y += A x and y = A^T x (the two products of a Gram-Schmidt pass) at the
    sizes where the split of the columns changes.  Either order of summation is
    within (k + 2) eps, or (n + 2) eps, times the sum of absolute products."""
    rng = np.random.default_rng(n + k)
    A = rng.standard_normal((k, n))  # column-major n x k
    x, y, z = rng.standard_normal(k), rng.standard_normal(n), rng.standard_normal(n)
    lib = gpu_lib.lib
    dA, dx, dy, dz = (evsl_b200.DeviceBuffer.from_host(lib, v) for v in (A, x, y, z))
    dh = evsl_b200.DeviceBuffer(lib, 8 * k)
    ci = lambda v: C.byref(C.c_int(v))  # noqa: E731
    cd = lambda v: C.byref(C.c_double(v))  # noqa: E731
    lib.evsl_dgemv_device(b"N", ci(n), ci(k), cd(-1.0), C.c_void_p(dA.ptr), ci(n), C.c_void_p(dx.ptr), ci(1), cd(1.0),
                          C.c_void_p(dy.ptr), ci(1))
    lib.evsl_dgemv_device(b"T", ci(n), ci(k), cd(1.0), C.c_void_p(dA.ptr), ci(n), C.c_void_p(dz.ptr), ci(1), cd(0.0),
                          C.c_void_p(dh.ptr), ci(1))
    eps = np.finfo(float).eps
    assert np.all(np.abs(dy.to_host() - (y - x @ A)) <= 2 * (k + 2) * eps * (np.abs(y) + np.abs(x) @ np.abs(A)))
    assert np.all(np.abs(dh.to_host() - A @ z) <= 2 * (n + 2) * eps * (np.abs(A) @ np.abs(z)))


@pytest.mark.parametrize("n, m, kind", [(1, 1, "random"), (2, 2, "random"), (9, 9, "random"), (70, 33, "random"),
                                        (515, 257, "random"), (1601, 40, "random"), (64, 64, "split"),
                                        (400, 90, "clusters")])
def test_tridiagonal_eigenvectors_on_gpu_are_the_hosts(gpu_lib, n, m, kind):
    """Inverse iteration with one thread per vector gives the host's vectors bit
    for bit, those of clusters (done on the host in both) included."""
    lib = gpu_lib.lib
    vp = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
    for f in (lib.evsl_trid_eigvecs, lib.evsl_trid_eigvecs_device, lib.evsl_trid_eigvals):
        f.restype = C.c_int
    lib.evsl_trid_eigvals.argtypes = [C.c_int, C.c_void_p, C.c_void_p, C.c_void_p]
    lib.evsl_trid_eigvecs.argtypes = [C.c_int, C.c_void_p, C.c_void_p, C.c_int, C.c_void_p, C.c_void_p, C.c_int]
    lib.evsl_trid_eigvecs_device.argtypes = [C.c_int, C.c_void_p, C.c_void_p, C.c_int, C.c_void_p, C.c_void_p]
    rng = np.random.default_rng(n + m)
    if kind == "clusters":  # four identical blocks: every eigenvalue four times
        b = n // 4
        d, e = np.tile(rng.uniform(-0.1, 1.0, b), 4), np.tile(np.r_[rng.uniform(0.01, 0.3, b - 1), 0.0], 4)
    else:
        d, e = rng.uniform(-0.1, 1.0, n), rng.uniform(0.01, 0.3, n)
        if kind == "split":
            e[n // 2] = 0.0
    w = np.zeros(n)
    assert lib.evsl_trid_eigvals(n, vp(d), vp(e), vp(w)) == 0
    sel = np.ascontiguousarray(w[n - m:])
    Z = np.zeros((m, n))
    dZ = evsl_b200.DeviceBuffer(lib, Z.nbytes)
    assert lib.evsl_trid_eigvecs(n, vp(d), vp(e), m, vp(sel), vp(Z), n) == 0
    assert lib.evsl_trid_eigvecs_device(n, vp(d), vp(e), m, vp(sel), C.c_void_p(dZ.ptr)) == 0
    assert np.array_equal(dZ.to_host(shape=Z.shape), Z)


def _eigvec_functions(lib):
    for f in (lib.evsl_trid_eigvecs, lib.evsl_trid_eigvecs_device, lib.evsl_trid_eigvals):
        f.restype = C.c_int
    lib.evsl_trid_eigvals.argtypes = [C.c_int, C.c_void_p, C.c_void_p, C.c_void_p]
    lib.evsl_trid_eigvecs.argtypes = [C.c_int, C.c_void_p, C.c_void_p, C.c_int, C.c_void_p, C.c_void_p, C.c_int]
    lib.evsl_trid_eigvecs_device.argtypes = [C.c_int, C.c_void_p, C.c_void_p, C.c_int, C.c_void_p, C.c_void_p]
    lib.evslcu_set_malloc_limit.argtypes = [C.c_size_t]
    return lambda a: a.ctypes.data_as(C.c_void_p)


@pytest.mark.parametrize("limit", [0, 2 << 20, 1 << 16])
def test_tridiagonal_eigenvectors_without_device_scratch(gpu_lib, limit):
    """With room for only some of the vectors at a time, and with room for none
    (the host's routine then), the vectors are the same; 30 pairs of close
    eigenvalues lie among lone ones."""
    lib = gpu_lib.lib
    vp = _eigvec_functions(lib)
    n, m = 600, 300
    rng = np.random.default_rng(7)
    d, e = rng.uniform(-0.1, 1.0, n), rng.uniform(0.01, 0.3, n)
    w = np.zeros(n)
    assert lib.evsl_trid_eigvals(n, vp(d), vp(e), vp(w)) == 0
    sel = np.ascontiguousarray(w[n - m:])
    sel[5:300:10] = sel[4:299:10] + 1e-9
    Z = np.zeros((m, n))
    assert lib.evsl_trid_eigvecs(n, vp(d), vp(e), m, vp(sel), vp(Z), n) == 0
    dZ = evsl_b200.DeviceBuffer(lib, Z.nbytes)
    try:
        lib.evslcu_set_malloc_limit(limit)
        assert lib.evsl_trid_eigvecs_device(n, vp(d), vp(e), m, vp(sel), C.c_void_p(dZ.ptr)) == 0
    finally:
        lib.evslcu_set_malloc_limit(0)
    assert np.array_equal(dZ.to_host(shape=Z.shape), Z)


@pytest.mark.skipif((os.cpu_count() or 1) < 4, reason="needs host cores to share the work")
def test_clustered_eigenvectors_share_the_host_threads(gpu_lib):
    """Vectors of clusters (here all: every eigenvalue is fourfold) are computed
    by several host threads: more processor time than time."""
    lib = gpu_lib.lib
    vp = _eigvec_functions(lib)
    n = 3000  # n vectors of n rows: work for four threads
    rng = np.random.default_rng(8)
    b = n // 4
    d, e = np.tile(rng.uniform(-0.1, 1.0, b), 4), np.tile(np.r_[rng.uniform(0.01, 0.3, b - 1), 0.0], 4)
    w = np.zeros(n)
    assert lib.evsl_trid_eigvals(n, vp(d), vp(e), vp(w)) == 0
    dZ = evsl_b200.DeviceBuffer(lib, 8 * n * n)
    t, c = time.perf_counter(), time.process_time()
    assert lib.evsl_trid_eigvecs_device(n, vp(d), vp(e), n, vp(w), C.c_void_p(dZ.ptr)) == 0
    t, c = time.perf_counter() - t, time.process_time() - c
    assert c > 1.5 * t, (c, t)
