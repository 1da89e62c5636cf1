"""The candidate search's faces in their own planes: needles down to corner angles
near the limit of a usable normal, faces as long as the mesh (decided from the
corners instead), both side by side, thresholds from far below the edges to
the largest allowed, at three scales.  Everything must equal sym_verification bit
for bit."""
import numpy as np
import pytest

from mitra_algo_gb300.mesh import mirrored_heightfield, prepare
from mitra_algo_gb300.types import Mesh, Options
from test_gpu_verify_resident import compare, gpu, records, rotation  # noqa: F401

pytestmark = pytest.mark.gpu


def grid(nx, ny, dx, dy, noise, seed):
    g = np.random.default_rng(seed)
    x, y = np.meshgrid(np.arange(nx) * dx, np.arange(ny) * dy, indexing="ij")
    v = np.stack([x.ravel(), y.ravel(), np.zeros(nx * ny)])
    v += g.normal(size=v.shape) * noise * np.array([[dx], [dy], [min(dx, dy)]])
    i, j = np.meshgrid(np.arange(nx - 1), np.arange(ny - 1), indexing="ij")
    a = (i * ny + j).ravel()
    f = np.concatenate([np.stack([a, a + ny, a + 1]), np.stack([a + 1, a + ny, a + ny + 1])], 1)
    return v, f.astype(np.int32)


MESHES = {
    "cube": lambda: (np.array([[x, y, z] for x in (0, 1) for y in (0, 1) for z in (0, 1)], float).T,
                     np.array([[0, 1, 3], [0, 3, 2], [4, 6, 7], [4, 7, 5], [0, 4, 5], [0, 5, 1],
                               [2, 3, 7], [2, 7, 6], [0, 2, 6], [0, 6, 4], [1, 5, 7], [1, 7, 3]], np.int32).T),
    "needles": lambda: grid(40, 30, 1.0, 1e-2, 0.2, 1),
    "sharp": lambda: grid(24, 24, 1.0, 2e-5, 0.2, 2),
    "limit": lambda: grid(16, 16, 1.0, 1.5e-6, 0.3, 3),
    "long": lambda: grid(3, 60, 10.0, 1e-1, 0.2, 4),
}


@pytest.mark.parametrize("threshold", [1e-4, 0.02, 0.49])
@pytest.mark.parametrize("scale", [1e-3, 1.0, 500.0])
@pytest.mark.parametrize("name", [*MESHES, "mixed"])
def test_faces_in_their_planes(gpu, name, scale, threshold):  # noqa: F811
    if name == "mixed":
        m = mirrored_heightfield(size=20, bumps=4, seed=5)
        cube_v, cube_f = MESHES["cube"]()
        v = np.concatenate([m.vertices, 3 * cube_v + 2.0], 1)
        f = np.concatenate([m.faces, cube_f + m.vertices.shape[1]], 1).astype(np.int32)
    else:
        v, f = MESHES[name]()
    o = Options(verify_threshold=threshold)
    p = prepare(Mesh(v * scale, f), o)
    c = np.asarray(p.context.center)
    tau = threshold * p.context.box_size
    moves = []
    for k, (axis, angle) in enumerate([((0, 0, 1), np.pi), ((0, 1, 0), np.pi), ((1, 2, 3), 0.7)]):
        R = rotation(axis, angle)
        moves.append((R, c - R @ c + (0.3 * k) * tau * np.array([0.2, -0.5, 1.0])))
    moves += [(np.eye(3), tau * np.array([2.5, 0.1, 0.5])), (np.eye(3), v[:, 5] * scale - v[:, 2] * scale)]
    compare(gpu, p, o, records(rigid=moves, planes=[((1, 0, 0), -c[0]), ((0, 0, 1), -c[2] + 0.5 * tau)]))
