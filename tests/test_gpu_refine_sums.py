"""The fixed-order sums behind the refinement and the coverage of detected
motions (128 and 256 strided partials, several vertices' loads ahead) at vertex
counts around multiples of the strides: one refinement pass equals its FP64
restatement, a motion's result does not depend on the others in the call, and
coverage and rms equal the exact verification's to the rounding of a sum of n
non-negative terms, 2 n u < 1e-12 for the sizes here."""
import numpy as np
import pytest

from mitra_algo_gb300.mesh import motif_torus, prepare
from mitra_algo_gb300.types import Options
from oracle.refine import refine_pass
from test_gpu_refine import motion_error, record
from test_gpu_verify_resident import gpu, records, rotation  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nu,nv", [(3, 3), (31, 4), (16, 8), (43, 3), (17, 15), (16, 16), (257, 3),
                                   (32, 16), (27, 19), (64, 32), (683, 3)])
def test_sums_at_stride_edges(gpu, nu, nv):  # noqa: F811
    mesh = motif_torus(R=1.0, r=0.3, nu=nu, nv=nv, copies=1, mirrored=0, noise=1e-3, seed=nu)
    o = Options(verify_threshold=0.05)
    p = prepare(mesh, o)
    c = np.asarray(p.context.center)
    tau = o.verify_threshold * p.context.box_size
    motions = []
    for angle in (2 * np.pi / nu, np.pi, 1.0):
        R = rotation((0.002, 0.001, 1), angle)
        motions.append(dict(reflection=False, rotation=R.reshape(-1), translation=c - R @ c,
                            plane_normal=np.zeros(3), plane_offset=0.0))
    resident = gpu.load_mesh(p)
    got = gpu.refine_transforms(resident, o, [record(m) for m in motions], 1)
    for k, m in enumerate(motions):
        alone = gpu.refine_transforms(resident, o, [record(m)], 1)
        for f in ("rotation", "translation", "coverage", "rms"):
            assert np.array_equal(alone[f][0], got[f][k]), f
        if nv == 3 and nu > 3:  # a triangular tube: images between two walls, where
            continue            # FP32 and FP64 searches pick different faces
        want = refine_pass(p.mesh.vertices, p.topology.normals, p.topology.weights, p.mesh.faces, m, tau)
        # the tolerance of tests/test_gpu_refine.py, whose FP32 search this is
        er, et = motion_error(dict(rotation=got["rotation"][k], translation=got["translation"][k]), want)
        assert er < 1e-6 and et < 1e-6, (k, er, et)
    rigid = [(np.reshape(R, (3, 3)), t) for R, t in zip(got["rotation"], got["translation"])]
    exact = gpu.verification(p.mesh, p.topology, records(rigid), p.context, o)
    resident.close()
    np.testing.assert_allclose(got["coverage"], exact.coverage, rtol=1e-12, atol=0)
    np.testing.assert_allclose(got["rms"], exact.rms, rtol=1e-12, atol=0)
