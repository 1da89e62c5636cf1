"""The FP64 decisions of the resident verification where most of them are
made: images at, next to and between the corners of faces, around vertices of
4 to 17 faces (the lists hold 16) whose normals
disagree, at three scales.  Everything must equal sym_verification bit for
bit, as in tests/test_gpu_verify_resident.py."""
import numpy as np
import pytest

from mitra_algo_gb300.mesh import prepare
from mitra_algo_gb300.types import Mesh, Options
from test_gpu_verify_resident import compare, fan_pair_mesh, gpu, records  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1e-3, 1.0, 300.0])
@pytest.mark.parametrize("valence", [4, 6, 8, 9, 15, 16, 17])
def test_corner_ties(gpu, valence, scale):  # noqa: F811
    base = fan_pair_mesh((valence,) * 3)
    p = prepare(Mesh(base.vertices * scale, base.faces), Options())
    o = Options(verify_threshold=0.01)
    eye, moves = np.eye(3), []
    for step in ((0, 0, 0), (1e-9, 0, 0), (0, 0, 1e-6), (0, 0, 3e-4), (2e-5, -1e-5, 2e-4),
                 (0.02, 0.01, 0.01)):
        moves.append((eye, scale * (np.array([5.0, 0.0, 0.0]) + step)))
    got, _ = compare(gpu, p, o, records(rigid=moves))
    assert got.coverage[0] > 0
