"""The resident conjugate-gradient form at the edges of its sizes, against direct solves."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as spla

from ordito_b200 import _lib, linalg
from ordito_b200.array import CsrMatrix
from ordito_b200.device import DeviceArray

pytestmark = pytest.mark.gpu


def _operator(n: int, seed: int, wide_row: bool = True) -> sp.csr_matrix:
    """A diagonally dominant symmetric operator of neighbours at distance 1 and ~sqrt(n) (a
    dominance of 1.25: condition below 9), with one row and column of 40 entries, more than a
    thread of the resident form keeps in shared memory, or without."""
    rng = np.random.default_rng(seed)
    far = max(2, int(n**0.5))
    rows, cols = [], []
    for step in (1, far):
        at = np.arange(max(0, n - step))
        rows.append(at)
        cols.append(at + step)
    if n > 64 and wide_row:
        to = rng.choice(np.arange(2, n), size=40, replace=False)
        rows.append(np.full(40, 0))
        cols.append(to)
    i, j = np.concatenate(rows), np.concatenate(cols)
    off = sp.coo_matrix((-rng.uniform(0.5, 1.0, i.size), (i, j)), shape=(n, n)).tocsr()
    off = off + off.T
    diagonal = 1.25 * np.maximum(-np.asarray(off.sum(axis=1)).ravel(), 1.0)
    matrix = (off + sp.diags(diagonal)).tocsr()
    matrix.sort_indices()
    return matrix


# One CTA (1 to 1024 rows), a cluster (to 16 x 1024 at two rows a thread, then four), the grid at two
# rows a thread (148 x 1024), at four (148 x 2048), and the loop graph past it.
_SIZES = (1, 2, 31, 33, 1024, 1025, 2049, 16384, 16385, 26001, 32769, 151552, 151553, 303104, 303105)


@pytest.mark.parametrize("kind", ["diag", "chebyshev"])
@pytest.mark.parametrize("n", _SIZES)
def test_solve_at_every_form_edge(gpu, n: int, kind: str) -> None:
    host = _operator(n, n)
    matrix = CsrMatrix.from_host(host.indptr, host.indices, host.data, host.shape)
    rng = np.random.default_rng(n + 1)
    rhs, start = rng.normal(size=n), rng.normal(size=n)
    preconditioner = (linalg.chebyshev_preconditioner if kind == "chebyshev"
                      else linalg.jacobi_preconditioner)(matrix)
    tol = 1e-10
    results = []
    for _ in range(2):
        x = DeviceArray.from_host(start)
        _, residual, _ = linalg.solve_spd(matrix, DeviceArray.from_host(rhs), x, tol=tol,
                                          preconditioner=preconditioner)
        assert residual <= tol
        results.append(x.numpy())
    np.testing.assert_array_equal(results[0], results[1])
    # |b - A x| <= tol |b| (the recurrence's residual; its drift from the true one is of the order
    # of the rounding, 1e-16 times the ~25 rounds' terms, far below tol).
    assert np.linalg.norm(rhs - host @ results[0]) <= 1.01 * tol * np.linalg.norm(rhs)


# Every form on both sides of its edges, without a row that is longer than the others.
@pytest.mark.parametrize("kind", ["diag", "chebyshev"])
@pytest.mark.parametrize("n", [1024, 1025, 2049, 6144, 6145, 16384, 16385, 22528, 22529, 26624, 26625, 151553])
def test_solve_of_short_rows(gpu, n: int, kind: str) -> None:
    host = _operator(n, n, wide_row=False)
    _solves(host, kind)


def _solves(host: sp.csr_matrix, kind: str) -> None:
    n = host.shape[0]
    matrix = CsrMatrix.from_host(host.indptr, host.indices, host.data, host.shape)
    preconditioner = (linalg.chebyshev_preconditioner if kind == "chebyshev"
                      else linalg.jacobi_preconditioner)(matrix)
    rng = np.random.default_rng(n + 1)
    rhs, start = rng.normal(size=n), rng.normal(size=n)
    results = []
    for _ in range(2):
        x = DeviceArray.from_host(start)
        linalg.solve_spd(matrix, DeviceArray.from_host(rhs), x, tol=1e-10, preconditioner=preconditioner)
        results.append(x.numpy())
    np.testing.assert_array_equal(results[0], results[1])
    assert np.linalg.norm(rhs - host @ results[0]) <= 1.01e-10 * np.linalg.norm(rhs)


# Rows of 1 to ~40 entries (the last figure is the mean): past the seven every row has in place, past what
# fits in place, past what a thread lists alone (16), more than the list in shared memory holds; and one
# row of every column, of 3 000 in the larger ones.
@pytest.mark.parametrize("kind", ["diag", "chebyshev"])
@pytest.mark.parametrize(("n", "mean"), [(33, 8), (700, 9), (1024, 30), (1025, 9), (5000, 12), (16384, 20), (20000, 9),
                                         (22528, 12), (30000, 30), (160000, 9)])
def test_solve_of_irregular_rows(gpu, n: int, mean: int, kind: str) -> None:
    rng = np.random.default_rng(n + mean)
    per = np.minimum(rng.geometric(1.0 / (mean / 2), size=n), 40)
    i = np.repeat(np.arange(n), per)
    j = i + 1 + rng.integers(0, 60, size=i.size)
    keep = j < n
    i, j = i[keep], j[keep]
    every = np.arange(n) if n <= 5000 else rng.choice(n, size=3000, replace=False)
    every = every[every != n // 2]
    off = sp.coo_matrix((-rng.uniform(0.5, 1.0, i.size), (i, j)), shape=(n, n)).tocsr()
    off = off + sp.coo_matrix((np.full(every.size, -1e-3), (np.full(every.size, n // 2), every)), shape=(n, n)).tocsr()
    off = off + off.T
    diagonal = 1.25 * np.maximum(-np.asarray(off.sum(axis=1)).ravel(), 1.0)
    host = (off + sp.diags(diagonal)).tocsr()
    host.sort_indices()
    _solves(host, kind)


@pytest.mark.parametrize("n", [1500, 9000, 16384, 20000, 40000, 200000])
def test_scattered_rows(gpu, n: int) -> None:
    """Rows in random order: every CTA reads the others' rows, past what its halo and push list hold."""
    rng = np.random.default_rng(n)
    order = rng.permutation(n)
    host = _operator(n, 3)[order][:, order].tocsr()
    host.sort_indices()
    matrix = CsrMatrix.from_host(host.indptr, host.indices, host.data, host.shape)
    rhs = rng.normal(size=n)
    for preconditioner in (linalg.jacobi_preconditioner(matrix), linalg.chebyshev_preconditioner(matrix)):
        x = DeviceArray.zeros(n, np.float64)
        linalg.solve_spd(matrix, DeviceArray.from_host(rhs), x, tol=1e-10, preconditioner=preconditioner)
        assert np.linalg.norm(rhs - host @ x.numpy()) <= 1.01e-10 * np.linalg.norm(rhs)


@pytest.mark.parametrize("n", [1, 33, 1024, 1025, 16385, 32769, 151553, 303105])
def test_settle_at_every_form_edge(gpu, n: int) -> None:
    """The settled solve reaches every entry in its own precision: verified by the componentwise
    backward error the solver accepts iterates by, against a direct solve."""
    host = _operator(n, n + 7)
    matrix = CsrMatrix.from_host(host.indptr, host.indices, host.data, host.shape)
    rhs = np.random.default_rng(n).uniform(0.5, 1.5, size=n)
    x = DeviceArray.zeros(n, np.float64)
    linalg.solve_spd_settled(matrix, DeviceArray.from_host(rhs), x, check_rounds=16, change_tolerance=1e-6,
                             settle_rounds=192)
    got = x.numpy()
    # The iteration's operator holds float32 values (6e-8 each): a backward error of 1e-7, and a
    # componentwise condition below 9 for this dominance.
    scale = np.abs(host) @ np.abs(got) + np.abs(rhs)
    assert np.max(np.abs(rhs - host @ got) / scale) <= 2e-7
    if n <= 40000:
        want = spla.splu(host.tocsc()).solve(rhs)
        np.testing.assert_allclose(got, want, rtol=2e-6)


def test_rebound_state_solves_the_new_operator(gpu) -> None:
    """A kept state of the same shape takes another operator's values (and its wide row's)."""
    n = 3000
    first, second = _operator(n, 1), _operator(n, 1)
    second.data = second.data * 1.5
    rhs = np.random.default_rng(0).normal(size=n)
    for host in (first, second, first):
        matrix = CsrMatrix.from_host(host.indptr, host.indices, host.data, host.shape)
        x = DeviceArray.zeros(n, np.float64)
        linalg.solve_spd(matrix, DeviceArray.from_host(rhs), x, tol=1e-12)
        assert np.linalg.norm(rhs - host @ x.numpy()) <= 1e-11 * np.linalg.norm(rhs)
        matrix.release()


@pytest.mark.parametrize("countdown", [1, 2, 3])
def test_refused_allocation_leaves_the_state_whole(gpu, countdown: int) -> None:
    """A first solve whose buffers are refused, then one on the same state, by the form that makes
    buffers at its first solve (the grid's)."""
    n = 40001
    host = _operator(n, 5)
    matrix = CsrMatrix.from_host(host.indptr, host.indices, host.data, host.shape)
    solver = linalg._solver(matrix, "diag", False, 1)
    rhs = np.random.default_rng(1).normal(size=n)
    d_rhs, x = DeviceArray.from_host(rhs), DeviceArray.zeros(n, np.float64)
    _lib.call("ob_fail_allocation", countdown)
    try:
        solver.solve(d_rhs.ptr, x.ptr, 1e-10, 1000)
    except MemoryError:
        pass
    finally:
        _lib.call("ob_fail_allocation", 0)
    x.fill_zero()
    solver.solve(d_rhs.ptr, x.ptr, 1e-10, 1000)
    assert np.linalg.norm(rhs - host @ x.numpy()) <= 1.01e-10 * np.linalg.norm(rhs)


def test_info_only_reads(gpu) -> None:
    """The copy's entries are 0 until a call has made the copy, again 0 after a rebind, and asking
    launches nothing (it has no stream to order work on)."""
    host = _operator(5000, 2)
    matrix = CsrMatrix.from_host(host.indptr, host.indices, host.data, host.shape)
    solver = linalg._solver(matrix, "diag", False, 1)

    def entries() -> int:
        info = (ctypes.c_longlong * 6)()
        launches = _lib.launch_count()
        _lib.call("ob_pcg_info", solver.handle, info)
        assert _lib.launch_count() == launches
        assert (info[0], info[2]) == (5000, host.nnz)
        return int(info[5])

    assert entries() == 0
    ms = ctypes.c_float(0.0)
    _lib.call("ob_pcg_time_matvec", solver.handle, 1, ctypes.byref(ms), None)
    built = entries()
    assert built >= host.nnz
    solver.rebind(matrix)
    assert entries() == 0
    _lib.call("ob_pcg_time_matvec", solver.handle, 1, ctypes.byref(ms), None)
    assert entries() == built


def test_rebind_returns_with_the_operator_copied(gpu) -> None:
    """Another stream may overwrite the caller's arrays once ob_pcg_rebind has returned, however much
    work its own stream still has before the copies."""
    n = 30001
    host = _operator(n, 4)
    matrix = CsrMatrix.from_host(host.indptr, host.indices, host.data, host.shape)
    other = CsrMatrix.from_host(host.indptr, host.indices, 3.0 * host.data, host.shape)
    solver = linalg._solver(matrix, "diag", False, 1)
    rhs = np.random.default_rng(2).normal(size=n)
    d_rhs, x = DeviceArray.from_host(rhs), DeviceArray.zeros(n, np.float64)
    busy_in, busy_out = DeviceArray.zeros(64 * n, np.float64), DeviceArray.zeros(64 * n, np.float64)
    streams = [ctypes.c_void_p(0), ctypes.c_void_p(0)]
    for stream in streams:
        _lib.call("ob_stream_create", ctypes.byref(stream))
    _lib.call("ob_device_synchronize")
    try:
        for _ in range(400):  # some tens of milliseconds ahead of the copies
            _lib.call("ob_spmv", n, matrix.offsets.ptr, matrix.columns.ptr, matrix.values.ptr, busy_in.ptr,
                      busy_out.ptr, 64, streams[0])
        _lib.call("ob_pcg_rebind", solver.handle, other.offsets.ptr, other.columns.ptr, other.values.ptr, other.nnz,
                  streams[0])
        _lib.call("ob_memcpy", other.values.ptr, matrix.values.ptr, 8 * other.nnz, 2, streams[1], 0)
        _lib.call("ob_pcg_solve", solver.handle, d_rhs.ptr, x.ptr, 1e-10, 1000, None, None, streams[0])
        for stream in streams:
            _lib.call("ob_stream_synchronize", stream)
    finally:
        for stream in streams:
            _lib.call("ob_stream_destroy", stream)
    assert np.linalg.norm(rhs - 3.0 * (host @ x.numpy())) <= 1.01e-10 * np.linalg.norm(rhs)


@pytest.mark.parametrize(("n", "kind"), [(3000, "diag"), (20000, "diag"), (20000, "chebyshev"), (40001, "diag"),
                                         (40001, "chebyshev")])
def test_a_wait_given_up_is_reported_once(gpu, n: int, kind: str) -> None:
    """Waits between a cluster's and a grid's blocks that run out at once: the solve returns, the
    status says so, by the next solve that reads back where this one does not, and the state goes on
    (its loop graph's settle too: 20 000 rows under Chebyshev)."""
    host = _operator(n, 6, wide_row=False)
    matrix = CsrMatrix.from_host(host.indptr, host.indices, host.data, host.shape)
    solver = linalg._solver(matrix, kind, False, 1)
    rhs = np.random.default_rng(3).normal(size=n)
    d_rhs, x = DeviceArray.from_host(rhs), DeviceArray.zeros(n, np.float64)
    rounds, residual = ctypes.c_int(0), ctypes.c_double(0.0)

    def solve(read_back: bool = True) -> int:
        x.fill_zero()
        return _lib.lib.ob_pcg_solve(solver.handle, d_rhs.ptr, x.ptr, 1e-10, 1000,
                                     ctypes.byref(rounds) if read_back else None,
                                     ctypes.byref(residual) if read_back else None, None)

    _lib.call("ob_pcg_wait_limit", solver.handle, 0)
    try:
        for _ in range(3):
            assert solve() == _lib.OB_ERR_TIMEOUT
        assert solve(read_back=False) == _lib.OB_OK
    finally:
        _lib.call("ob_pcg_wait_limit", solver.handle, -1)
    assert solve(read_back=False) == _lib.OB_OK
    assert solve() == _lib.OB_ERR_TIMEOUT  # the unread one's
    assert solve() == _lib.OB_OK
    assert np.linalg.norm(rhs - host @ x.numpy()) <= 1.01e-10 * np.linalg.norm(rhs)
    x.fill_zero()
    solver.settle(d_rhs.ptr, x.ptr, 16, 1e-6, 192, 1000)
    assert np.linalg.norm(rhs - host @ x.numpy()) <= 1e-6 * np.linalg.norm(rhs)


def test_rebound_state_takes_its_form_anew(gpu) -> None:
    """Operators of one shape whose rows lie in order and scattered: the cluster's, then the grid's form,
    with and without reading anything back."""
    n = 12000
    rng = np.random.default_rng(0)
    ordered = _operator(n, 8, wide_row=False)
    order = rng.permutation(n)
    scattered = ordered[order][:, order].tocsr()
    scattered.sort_indices()
    solver = None
    rhs = rng.normal(size=n)
    d_rhs = DeviceArray.from_host(rhs)
    for host in (scattered, ordered, ordered, scattered, scattered, ordered):
        matrix = CsrMatrix.from_host(host.indptr, host.indices, host.data, host.shape)
        if solver is None:
            solver = linalg._solver(matrix, "chebyshev", False, 1)
        else:
            solver.rebind(matrix)
        for outputs in (False, True):
            x = DeviceArray.zeros(n, np.float64)
            if outputs:
                solver.solve(d_rhs.ptr, x.ptr, 1e-10, 1000)
            else:
                _lib.call("ob_pcg_solve", solver.handle, d_rhs.ptr, x.ptr, 1e-10, 1000, None, None, None)
            assert np.linalg.norm(rhs - host @ x.numpy()) <= 1.01e-10 * np.linalg.norm(rhs)
