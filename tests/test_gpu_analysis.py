"""The analysis started beside a settled solve: the same tree, and given up safely."""

from __future__ import annotations

import ctypes
import gc
import time

import numpy as np
import pytest

from ordito_b200 import _lib, creation
from ordito_b200 import heat as gheat
from ordito_b200.cholesky import CholeskyAnalysis, OperatorFactorization
from ordito_b200.device import DeviceArray
from ordito_b200.mesh import Trimesh

pytestmark = pytest.mark.gpu


def _nodes(analysis: CholeskyAnalysis) -> np.ndarray:
    out = np.zeros((analysis.supernodes, 4), dtype=np.int32)
    _lib.call("ob_chol_analysis_nodes", analysis.handle, out.ctypes.data_as(ctypes.c_void_p))
    return out


@pytest.mark.parametrize("shape", [(24, 12), (300, 200)])
def test_analysis_ahead_is_the_analysis(gpu, shape: tuple[int, int]) -> None:
    v, f = creation.jittered_torus(*shape, seed=1)
    mesh = Trimesh(v, f.reshape(-1))
    heat = mesh.heat_solver(method="meshlab").operators.heat_system
    plain = CholeskyAnalysis(heat, mesh.vertices)
    slot = OperatorFactorization(heat, mesh.vertices)
    slot.analyse_ahead()
    slot.analyse_ahead()  # one at a time
    assert not slot.exceeds_budget()
    assert slot.analysis.factor_entries == plain.factor_entries
    np.testing.assert_array_equal(_nodes(slot.analysis), _nodes(plain))
    assert slot.factor()


def test_abandoned_analyses_leave_nothing_behind(gpu) -> None:
    for seed in range(6):
        v, f = creation.jittered_torus(300, 200 + seed, seed=seed)
        mesh = Trimesh(v, f.reshape(-1))
        slot = OperatorFactorization(mesh.heat_solver(method="meshlab").operators.heat_system, mesh.vertices)
        slot.analyse_ahead()
        slot.release()  # the mesh's arrays go right after
        mesh.dispose()
        del slot, mesh


def _held() -> int:
    count = ctypes.c_int(0)
    _lib.call("ob_chol_analyses_held", ctypes.byref(count))
    return count.value


@pytest.mark.parametrize("wait", [0.0, 0.002, 0.02, 1.5])
def test_abandoned_analysis_is_let_go(gpu, wait: float) -> None:
    """One given up at once, under way, or after it has finished leaves no analysis behind, without
    another being abandoned."""
    v, f = creation.jittered_torus(300, 210, seed=3)
    mesh = Trimesh(v, f.reshape(-1))
    slot = OperatorFactorization(mesh.heat_solver(method="meshlab").operators.heat_system, mesh.vertices)
    gc.collect()
    before = _held()
    slot.analyse_ahead()
    time.sleep(wait)
    if wait >= 1.0:
        assert _held() == before + 1  # finished, and not taken
    slot.drop_analysis_ahead()
    for _ in range(200):
        if _held() == before:
            break
        time.sleep(0.01)
    assert _held() == before
    assert slot.factor()  # its own analysis, made in place
    slot.release()


def test_a_failed_settled_solve_gives_its_analysis_up(gpu, monkeypatch) -> None:
    v, f = creation.jittered_torus(300, 210, seed=4)
    mesh = Trimesh(v, f.reshape(-1))
    solver = mesh.heat_solver(method="meshlab")
    rhs = DeviceArray.zeros(v.shape[0], np.float64)

    def fail(*args, **kwargs):
        raise RuntimeError("the solve failed")

    monkeypatch.setattr(gheat, "_ANALYSE_AHEAD_ROWS", 1000)
    monkeypatch.setattr(gheat.twl, "solve_spd_settled", fail)
    with pytest.raises(RuntimeError, match="the solve failed"):
        solver.diffuse(rhs, rhs)
    assert solver._kept("heat")["factorization"]._pending is None


def test_large_queries_ahead_and_in_place_agree(gpu, monkeypatch) -> None:
    """The drop-in call on a mesh whose settled iterate is rejected, and on one whose is kept."""
    torus, sheet = creation.jittered_torus(300, 230, seed=2), creation.flat_grid((280, 250))
    for v, f in (torus, sheet):
        plain = gheat.heat_geodesic(v, f.reshape(-1), np.array([7], dtype=np.int32)).numpy()
        with monkeypatch.context() as patch:
            patch.setattr(gheat, "_ANALYSE_AHEAD_ROWS", 1000)
            ahead = gheat.heat_geodesic(v, f.reshape(-1), np.array([7], dtype=np.int32)).numpy()
        # The factored passes add split tiles' products atomically: the order, so the rounding, varies.
        np.testing.assert_allclose(ahead, plain, rtol=0, atol=1e-11 * np.abs(plain).max())
