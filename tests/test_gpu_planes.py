"""The divergence over corner planes and the packed shift's chunks, at their edges."""

from __future__ import annotations

import numpy as np
import pytest

from ordito_b200 import _lib, creation
from ordito_b200.device import DeviceArray
from ordito_b200.heat import corner_planes, mesh_corner_planes
from ordito_b200.mesh import Trimesh
from tests import meshes

pytestmark = pytest.mark.gpu


def _sliver() -> tuple[np.ndarray, np.ndarray]:
    """A strip of faces 1e4 times as long as high, and a face of no area."""
    top = np.array([[i * 1.0, 1e-4 * (i % 2), 0.1 * i] for i in range(40)])
    f = np.array([[i, i + 1, i + 2] for i in range(38)] + [[0, 0, 1]])
    return top.astype(np.float32), f.astype(np.int32)


_MESHES = {
    "bumpy": meshes.bumpy_sphere,
    "sheet": lambda: creation.flat_grid((23, 17)),
    "octahedron": creation.octahedron,
    "sliver": _sliver,
}


# 1, 2 and 4 columns a thread: odd strides, even ones, multiples of 4; pad columns past k.
@pytest.mark.parametrize("k,stride", [(1, 1), (1, 2), (2, 2), (3, 4), (5, 5), (6, 6), (64, 64)])
@pytest.mark.parametrize("name", sorted(_MESHES))
def test_planes_match_the_terms(gpu, name: str, k: int, stride: int) -> None:
    v, f = _MESHES[name]()
    n = v.shape[0]
    mesh = Trimesh(v, f.reshape(-1))
    face = mesh.face_terms
    offsets, slots = mesh.corner_index
    terms = DeviceArray.empty((mesh.n_faces, 18), np.float64)
    _lib.call("ob_face_gradient_terms", mesh.vertices.ptr, mesh.faces.ptr, mesh.n_faces, face.normals.ptr,
              face.areas.ptr, face.cot.ptr, terms.ptr, None)
    planes = corner_planes(terms, mesh.faces, slots, mesh.n_faces)
    rng = np.random.default_rng(k)
    field = np.zeros((n, stride))
    field[:, :k] = np.exp(-5.0 * rng.random((n, k)))
    order = rng.permutation(n).astype(np.int32)
    pinned = np.zeros(n, dtype=np.uint8)
    pinned[order[0]] = 1
    d_order, d_pinned = DeviceArray.from_host(order), DeviceArray.from_host(pinned)
    for u_iperm, out_iperm, mask in ((None, None, None), (d_order, d_order, d_pinned)):
        outs = {}
        for scale in (0, -900):
            u = DeviceArray.from_host(np.ldexp(field, scale).reshape(-1))
            tail = (n, k, u.ptr, stride, u_iperm and u_iperm.ptr)
            for form in ("terms", "planes"):
                out = DeviceArray.empty(n * stride, np.float64)
                head = (terms.ptr, mesh.faces.ptr, offsets.ptr, slots.ptr) if form == "terms" else (planes.ptr, offsets.ptr)
                _lib.call(f"ob_grad_div_{form}", *head, *tail, out.ptr, stride, out_iperm and out_iperm.ptr,
                          mask and mask.ptr, None)
                outs[form, scale] = out.numpy()
        # The unit gradient is scale-free, its power-of-two rescaling exact.
        assert np.array_equal(outs["planes", 0], outs["planes", -900])
        # Both forms in float64: the unit gradient loses u's rounding over the gradient's size, up to
        # 1e4 on the slivers' short side, so 1e-16 x 1e4 x a few, over the largest term.
        tolerance = 1e-10 if name == "sliver" else 1e-12
        want = outs["terms", 0]
        np.testing.assert_allclose(outs["planes", 0], want, rtol=tolerance, atol=tolerance * np.abs(want).max())


@pytest.mark.parametrize("name", sorted(_MESHES))
def test_planes_of_the_mesh_are_the_terms_planes(gpu, name: str) -> None:
    """The planes made from the mesh itself against those from its face terms, and in another numbering."""
    v, f = _MESHES[name]()
    mesh = Trimesh(v, f.reshape(-1))
    face = mesh.face_terms
    slots = mesh.corner_index[1]
    terms = DeviceArray.empty((mesh.n_faces, 18), np.float64)
    _lib.call("ob_face_gradient_terms", mesh.vertices.ptr, mesh.faces.ptr, mesh.n_faces, face.normals.ptr,
              face.areas.ptr, face.cot.ptr, terms.ptr, None)
    order = np.random.default_rng(0).permutation(v.shape[0]).astype(np.int32)
    for numbering in (np.arange(v.shape[0], dtype=np.int32), order):
        ids = DeviceArray.from_host(numbering[f.reshape(-1)])
        want = corner_planes(terms, ids, slots, mesh.n_faces).numpy().reshape(-1, 6)
        got = mesh_corner_planes(mesh.vertices, mesh.faces, ids, face.normals, face.areas, face.cot, slots,
                                 mesh.n_faces).numpy().reshape(-1, 6)
        np.testing.assert_array_equal(got[:, 5].view(np.int64), want[:, 5].view(np.int64))
        # The same float64 formulas: a few roundings of a corner's largest coefficient, which the frame's
        # division by a sliver's height (1e-4 of its length) carries on.
        scale = np.abs(want[:, :5]).max(axis=1, keepdims=True)
        assert np.all(np.abs(got[:, :5] - want[:, :5]) <= 1e-11 * scale)


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("k", [1, 2, 4])
def test_planes_carry_what_is_not_finite(gpu, k: int, bad: float) -> None:
    """A NaN or infinite value shows at every corner that reads it, as in the terms form, also where the
    face's other two values are equal."""
    v, f = creation.flat_grid((9, 7))
    n = v.shape[0]
    mesh = Trimesh(v, f.reshape(-1))
    face = mesh.face_terms
    offsets, slots = mesh.corner_index
    terms = DeviceArray.empty((mesh.n_faces, 18), np.float64)
    _lib.call("ob_face_gradient_terms", mesh.vertices.ptr, mesh.faces.ptr, mesh.n_faces, face.normals.ptr,
              face.areas.ptr, face.cot.ptr, terms.ptr, None)
    planes = corner_planes(terms, mesh.faces, slots, mesh.n_faces)
    faces = f.reshape(-1, 3)
    for at in range(0, n, 5):
        field = np.zeros((n, k))
        field[at, k - 1] = bad
        u, out = DeviceArray.from_host(field.reshape(-1)), DeviceArray.empty(n * k, np.float64)
        _lib.call("ob_grad_div_planes", planes.ptr, offsets.ptr, n, k, u.ptr, k, None, out.ptr, k, None, None, None)
        got = ~np.isfinite(out.numpy().reshape(n, k))
        want = np.zeros((n, k), dtype=bool)
        want[np.unique(faces[(faces == at).any(axis=1)]), k - 1] = True  # the vertex and its neighbours
        np.testing.assert_array_equal(got, want)


# A chunk is 512 rows: one less, one, one more, and several, beside a mesh of three vertices.
@pytest.mark.parametrize("k", [1, 3, 16])
def test_packed_shift_over_chunk_edges(gpu, k: int) -> None:
    sizes = np.array([3, 511, 512, 513, 1025, 2600], dtype=np.int32)
    offsets = np.concatenate(([0], np.cumsum(sizes))).astype(np.int32)
    n, stride = int(offsets[-1]), k + (k & 1)
    rng = np.random.default_rng(k)
    phi = rng.normal(size=(n, stride))
    order = rng.permutation(n).astype(np.int32)
    sources = np.array([[int(rng.integers(0, s)) if c < k - 1 or m % 2 == 0 else -1 for c in range(k)]
                        for m, s in enumerate(sizes)], dtype=np.int32)
    want = np.zeros((k, n))
    for m in range(sizes.size):
        rows = order[offsets[m]:offsets[m + 1]]
        for c in range(k):
            if sources[m, c] < 0:
                continue
            field = phi[rows, c]
            shift = field[sources[m, c]]
            want[c, offsets[m]:offsets[m + 1]] = field - shift if field.mean() - shift >= 0 else shift - field
    d_phi, d_order = DeviceArray.from_host(phi.reshape(-1)), DeviceArray.from_host(order)
    d_offsets, d_sources = DeviceArray.from_host(offsets), DeviceArray.from_host(sources.reshape(-1))
    sums = DeviceArray.empty(2 * k * sizes.size, np.float64)
    out = DeviceArray.empty((k, n), np.float64)
    _lib.call("ob_shift_packed", d_phi.ptr, n, stride, d_order.ptr, d_offsets.ptr, sizes.size, d_sources.ptr, k,
              sums.ptr, out.ptr, None)
    np.testing.assert_allclose(out.numpy(), want, rtol=1e-14, atol=1e-14)
