"""The operator pattern at the edges of its row-block sort, bit for bit against the oracle."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import heat_path as hp
from ordito_b200 import creation
from ordito_b200.laplacian import mesh_operator_pattern

pytestmark = pytest.mark.gpu


def _fan(ring: int) -> tuple[np.ndarray, int]:
    """A hub on ``ring`` faces: a row of 2 ring + 1 keys."""
    at = 1 + np.arange(ring)
    return np.stack((np.zeros(ring, dtype=int), at, 1 + at % ring), 1), ring + 1


def _random(n_faces: int, n: int, low: int, high: int, seed: int) -> tuple[np.ndarray, int]:
    return np.random.default_rng(seed).integers(low, high, size=(n_faces, 3)), n


_CASES = {
    # Rows of one block of 128, one less, one more; a mesh of several blocks.
    "127": lambda: _random(250, 127, 0, 127, 0),
    "128": lambda: _random(250, 128, 0, 128, 1),
    "129": lambda: _random(250, 129, 0, 129, 2),
    "torus": lambda: (creation.torus(61, 37)[1], 61 * 37),
    # Rows at, and one key past, the longest a thread sorts (96 keys: 2 x 47 + 1 = 95, 2 x 48 + 1 = 97).
    "fan47": lambda: _fan(47),
    "fan48": lambda: _fan(48),
    # One run of 1 024 keys, two, and runs merged to an odd count.
    "fan511": lambda: _fan(511),
    "fan512": lambda: _fan(512),
    "fan5000": lambda: _fan(5000),
    # A block of rows past the shared memory (60 keys a row).
    "crowded": lambda: _random(4000, 256, 0, 256, 3),
    # Repeated corners, indices outside the vertices, unreferenced vertices.
    "degenerate": lambda: _random(600, 40, 0, 12, 4),
    "outside": lambda: _random(400, 100, -20, 130, 5),
    "all_outside": lambda: _random(50, 10, 10, 40, 6),
    "one_vertex": lambda: (np.zeros((3, 3), dtype=int), 1),
}


@pytest.mark.parametrize("name", sorted(_CASES))
def test_pattern_is_bit_exact_at_the_edges(gpu, name: str) -> None:
    faces, n = _CASES[name]()
    faces = np.ascontiguousarray(faces, dtype=np.int32)
    want = hp.mesh_operator_pattern(faces, n)
    got = mesh_operator_pattern(faces.reshape(-1), n)
    nnz = int(want["offsets"][-1])
    np.testing.assert_array_equal(got.offsets.numpy(), want["offsets"])
    np.testing.assert_array_equal(got.columns.numpy()[:nnz], want["columns"][:nnz])
    np.testing.assert_array_equal(got.run_start.numpy()[:nnz], want["run_start"][:nnz])
    np.testing.assert_array_equal(got.keys.numpy(), want["keys"])
    np.testing.assert_array_equal(got.order.numpy(), want["order"])
