"""The FP64 rows of the resident verification by how many of each kind there
are: images moved by exactly twice the threshold (FP32 cannot decide the test,
the row has no candidates and searches), images on vertices and edges whose
faces disagree, and all of them in one call, on meshes of a few to some
thousand vertices.  Everything must equal sym_verification bit for bit."""
import numpy as np
import pytest

from mitra_algo_gb300.mesh import motif_torus, prepare
from mitra_algo_gb300.types import Options
from test_gpu_verify_resident import compare, gpu, records, rotation  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kinds", ["search", "rows", "both"])
@pytest.mark.parametrize("nu,nv", [(8, 4), (11, 3), (31, 16), (64, 33)])
def test_rows_by_kind(gpu, nu, nv, kinds):  # noqa: F811
    mesh = motif_torus(R=1.0, r=0.3, nu=nu, nv=nv, copies=1, mirrored=0, noise=0.05, seed=nu)
    o = Options(verify_threshold=0.01)
    p = prepare(mesh, o)
    tau = o.verify_threshold * p.context.box_size
    c = np.asarray(p.context.center)
    turn = rotation((0, 0, 1), 2 * np.pi / nu)
    search = [(np.eye(3), np.array([2 * tau, 0, 0])), (np.eye(3), np.array([0, -2 * tau, 0]))]
    rows = [(turn, c - turn @ c), (np.eye(3), mesh.vertices[:, 5] - mesh.vertices[:, 3]),
            (rotation((0, 0, 1), np.pi), c - rotation((0, 0, 1), np.pi) @ c)]
    motions = {"search": search, "rows": rows, "both": search + rows}[kinds]
    compare(gpu, p, o, records(rigid=motions, planes=[((1, 0, 0), 0.0)]))
