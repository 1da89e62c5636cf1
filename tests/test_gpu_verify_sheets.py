"""FP64 distances sorted by region over the rows of a block: one to four coincident
sheets (so every row has that many faces at one distance, all of one region, more
than a region's list holds with three or four), their normals alike or opposed,
row counts around a block of 256, images over, on and between the faces.
Everything must equal sym_verification bit for bit."""
import numpy as np
import pytest

from mitra_algo_gb300.mesh import prepare
from mitra_algo_gb300.types import Mesh, Options
from test_gpu_verify_flat import grid
from test_gpu_verify_resident import compare, gpu, records, rotation  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flip", [False, True])
@pytest.mark.parametrize("sheets", [1, 2, 3, 4])
@pytest.mark.parametrize("nx,ny", [(5, 17), (8, 8), (16, 16), (11, 7), (40, 13)])
def test_coincident_sheets(gpu, nx, ny, sheets, flip):  # noqa: F811
    v, f = grid(nx, ny, 1.0, 0.8, 0.1, nx)
    verts = np.concatenate([v] * sheets, 1)
    faces = np.concatenate([(f[::-1] if flip and k % 2 else f) + k * v.shape[1] for k in range(sheets)], 1)
    o = Options(verify_threshold=0.02)
    p = prepare(Mesh(verts, faces.astype(np.int32)), o)
    c = np.asarray(p.context.center)
    turn = rotation((0, 0, 1), np.pi)
    step = np.array([1.0, 0, 0])
    moves = [(turn, c - turn @ c), (turn, c - turn @ c + np.array([0, 0, 0.05])),
             (np.eye(3), step), (np.eye(3), step + np.array([0.31, 0.17, 0.02])),
             (np.eye(3), v[:, 1] - v[:, 0]), (np.eye(3), 2 * step + np.array([0, 0, 1e-9]))]
    compare(gpu, p, o, records(rigid=moves, planes=[((1, 0, 0), -c[0])]))
