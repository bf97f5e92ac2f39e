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
    # Rows a warp sorts.
    "fan47": lambda: _fan(47),
    "fan48": lambda: _fan(48),
    # The longest row of 256 threads (1 023 keys), the shortest of a CTA (1 025), tiles merged to an odd count.
    "fan511": lambda: _fan(511),
    "fan512": lambda: _fan(512),
    "fan5000": lambda: _fan(5000),
    # A block of rows past the shared memory (60 keys a row).
    "crowded": lambda: _random(4000, 256, 0, 256, 3),
    # The longest row a thread sorts and the shortest of a warp (23 and 25 keys), of a warp and of 256 threads
    # (127 and 129), of one tile and of two (4 095 and 4 097).
    "fan11": lambda: _fan(11),
    "fan12": lambda: _fan(12),
    "fan63": lambda: _fan(63),
    "fan64": lambda: _fan(64),
    "fan2047": lambda: _fan(2047),
    "fan2048": lambda: _fan(2048),
    "fan10300": lambda: _fan(10300),
    # Rows of 3 to some hundreds of keys beside one another, in and past the shared memory.
    "uneven": lambda: (np.concatenate([_fan(r)[0] + 1500 * (r > 40) for r in (20, 30, 200, 400, 700)]), 3000),
    "crowded_hub": lambda: (np.concatenate((_random(9000, 300, 0, 300, 7)[0], _fan(299)[0])), 300),
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
