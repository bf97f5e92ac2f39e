"""The pool of kept solver states, with fakes in the device's place."""

from __future__ import annotations

import collections
import ctypes
import threading

import pytest

from ordito_b200 import linalg


class _State(linalg.NativeSolver):
    def __init__(self, shape_key: tuple) -> None:
        self.handle = ctypes.c_void_p(1)
        self.shape_key = shape_key
        self.pooled = False
        self.rebound = 0

    def rebind(self, matrix) -> None:
        self.rebound += 1

    def close(self) -> None:
        self.handle = ctypes.c_void_p(0)


class _Matrix:
    """An operator whose entry count, once asked for, has another operator collected."""

    nrow = 10

    def __init__(self, collected: list) -> None:
        self._solvers = {}
        self.collected = collected

    @property
    def nnz(self) -> int:
        for state in self.collected:
            linalg.retire_solver(state)
        return 30


@pytest.fixture()
def pool(monkeypatch):
    monkeypatch.setattr(linalg, "_KEPT", type(linalg._KEPT)())
    monkeypatch.setattr(linalg, "_RETIRED", collections.deque(), raising=False)
    monkeypatch.setattr(linalg, "_KEPT_LOCK", threading.Lock())
    return linalg._KEPT


def _within(seconds: float, call) -> None:
    thread = threading.Thread(target=call, daemon=True)
    thread.start()
    thread.join(seconds)
    assert not thread.is_alive(), "the call waits for its own thread"


def test_a_state_retired_while_another_is_looked_up(pool) -> None:
    key = (10, 30, "diag", True, 1)
    wanted, other = _State(key), _State((10, 31, "diag", True, 1))
    linalg.retire_solver(wanted)
    matrix = _Matrix([other])
    _within(10.0, lambda: linalg._solver(matrix, "diag", True, 1))
    assert matrix._solvers[("diag", True, 1)] is wanted and wanted.rebound == 1 and not wanted.pooled
    assert list(pool.values()) == [other] and other.pooled


def test_a_state_retired_under_the_lock_is_pooled_after_it(pool) -> None:
    state = _State((10, 30, "diag", True, 1))

    def retire() -> None:
        with linalg._KEPT_LOCK:
            linalg.retire_solver(state)  # a collection between two statements under the lock
        assert not pool
        linalg._pool_retired()

    _within(10.0, retire)
    assert list(pool.values()) == [state]


def test_the_pool_is_bounded_and_closes_what_it_drops(pool) -> None:
    states = [_State((10, n, "diag", True, 1)) for n in range(linalg._KEPT_LIMIT + 3)]
    for state in states:
        linalg.retire_solver(state)
    assert list(pool.values()) == states[3:]
    assert all(not s.handle.value and not s.pooled for s in states[:3])
    again = _State(states[5].shape_key)
    linalg.retire_solver(again)
    assert not states[5].handle.value and pool[again.shape_key] is again
