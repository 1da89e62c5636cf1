"""Motions that are not orthonormal: matrices whose large products cancel, so the image
lies on the mesh with the rounding of terms many times its size, and scaled plane
normals.  Everything must equal sym_verification bit for bit."""
import numpy as np
import pytest

from mitra_algo_gb300.mesh import prepare
from mitra_algo_gb300.types import Mesh, Options
from test_gpu_verify_resident import compare, gpu, records  # noqa: F401

pytestmark = pytest.mark.gpu


def sheet(n, at):
    """A rough n x n sheet across (1, -1, 0), `at` from the origin."""
    g = np.random.default_rng(5)
    x, y = np.meshgrid(np.linspace(-1, 1, n), np.linspace(-1, 1, n), indexing="ij")
    i, j = np.meshgrid(np.arange(n - 1), np.arange(n - 1), indexing="ij")
    a = (i * n + j).ravel()
    f = np.concatenate([np.stack([a, a + n, a + 1]), np.stack([a + 1, a + n, a + n + 1])], 1)
    across, along, up = np.array([1, -1, 0]) / 2 ** 0.5, np.array([1, 1, 0]) / 2 ** 0.5, np.array([0, 0, 1.0])
    v = np.outer(along, x.ravel() + at) + np.outer(up, y.ravel()) + np.outer(across, g.normal(0, 1e-4, n * n))
    return Mesh(v, f.astype(np.int32)), across, along, up


@pytest.mark.parametrize("at", [0.0, 4.0, 300.0])
@pytest.mark.parametrize("shear", [1, 20, 200, 1000, 3000, 20000, 1e9, 1e38])
def test_sheared(gpu, shear, at):  # noqa: F811
    mesh, across, along, up = sheet(90, at)
    o = Options(verify_threshold=0.02)
    p = prepare(mesh, o)
    g = np.random.default_rng(7)
    moves = []
    for s in range(6):
        t = along * (0.25 + 0.01 * s) + up * 0.07
        moves.append((np.eye(3) + shear * np.outer(across + 0.3 * g.normal(size=3), across), t))
        moves.append((np.eye(3) + shear * np.outer(along, across), t))
    moves = [(r, t - (r @ (at * along) - at * along)) for r, t in moves]
    cl = records(rigid=moves, planes=[(along, -at), (up, 0.01)])
    cl.plane_normal[-2:] *= min(shear, 1e30)  # the plane's side by a scaled normal
    cl.plane_offset[-2:] *= min(shear, 1e30)
    compare(gpu, p, o, cl)
