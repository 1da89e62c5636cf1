"""sym_verification on hard geometry against the oracle, which has no FP32 in it: needles
down to the limit of a usable normal, faces as long as the mesh, coincident
sheets with normals alike or opposed, fans of more faces than a leaf holds, folded and
degenerate faces.  Lists, coverage and rms bit for bit.  (The resident form is
compared with sym_verification; what the two share is pinned here.)"""
import numpy as np
import pytest

from mitra_algo_gb300.mesh import mirrored_heightfield, prepare
from mitra_algo_gb300.types import Mesh, Options
from oracle import oracle
from test_gpu_verify_flat import MESHES, grid
from test_gpu_verify_resident import assert_identical, fan_pair_mesh, gpu, records, rotation  # noqa: F401

pytestmark = pytest.mark.gpu


def mixed():
    m = mirrored_heightfield(size=20, bumps=4, seed=5)
    v, f = MESHES["cube"]()
    return (np.concatenate([m.vertices, 3 * v + 2.0], 1),
            np.concatenate([m.faces, f + m.vertices.shape[1]], 1))


def sheets(flip):
    v, f = grid(11, 13, 1.0, 0.8, 0.1, 11)
    parts = [(f[::-1] if flip and k % 2 else f) + k * v.shape[1] for k in range(3)]
    return np.concatenate([v] * 3, 1), np.concatenate(parts, 1)


def fans():
    m = fan_pair_mesh((17, 16, 9, 4))
    return m.vertices, m.faces


def folded():
    """Faces folded onto each other within 1e-9, some of no area and some that nearly are."""
    v, f = grid(14, 14, 1.0, 1.0, 0.3, 9)
    v[2, ::3] *= 1e-9
    v[:, 1::14] = v[:, ::14] + 1e-9
    v[:, 5::28] = 0.5 * (v[:, 4::28] + v[:, 6::28])
    return v, f


CASES = {**{k: MESHES[k] for k in MESHES}, "mixed": mixed, "sheets": lambda: sheets(False),
         "opposed": lambda: sheets(True), "fans": fans, "folded": folded}


@pytest.mark.parametrize("threshold", [1e-4, 0.02, 0.3])
@pytest.mark.parametrize("scale", [1e-3, 1.0, 500.0])
@pytest.mark.parametrize("name", CASES)
def test_equal_to_the_oracle(gpu, name, scale, threshold):  # noqa: F811
    v, f = CASES[name]()
    o = Options(verify_threshold=threshold)
    p = prepare(Mesh(np.asarray(v) * scale, np.asarray(f, np.int32)), o)
    c = np.asarray(p.context.center)
    tau = threshold * p.context.box_size
    moves = []
    for k, (axis, angle) in enumerate([((0, 0, 1), np.pi), ((0, 1, 0), np.pi), ((1, 2, 3), 0.7)]):
        r = rotation(axis, angle)
        moves.append((r, c - r @ c + (0.3 * k) * tau * np.array([0.2, -0.5, 1.0])))
    step = scale * (v[:, 1] - v[:, 0])
    moves += [(np.eye(3), tau * np.array([2.5, 0.1, 0.5])), (np.eye(3), step), (np.eye(3), 3.3 * step),
              (np.eye(3), scale * np.array([5.0, 0, 0])), (np.eye(3), scale * np.array([5.0, 0, 3e-4]))]
    cl = records(rigid=moves, planes=[((1, 0, 0), -c[0]), ((0, 0, 1), -c[2] + 0.5 * tau)])
    assert_identical(gpu.verification(p.mesh, p.topology, cl, p.context, o),
                     oracle.OracleBackend().verification(p.mesh, p.topology, cl, p.context, o))
