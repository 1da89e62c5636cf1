"""The exact verification's FP32 shortcuts where FP32 leaves its range or its
accuracy: meshes from 1e-20 to 1e15 in size, far from the origin, flat faces,
exact mirrors of a grid (every image ties between faces), motions that are not
finite.  Equal to the oracle bit for bit."""
import numpy as np
import pytest

from mitra_algo_gb300.mesh import mirrored_heightfield, motif_torus, prepare
from mitra_algo_gb300.types import Mesh, ModelContext, Options
from oracle import oracle
from test_gpu_verify_resident import records

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    from mitra_algo_gb300 import Gb300Backend
    b = Gb300Backend(0)
    yield b
    b.close()


@pytest.mark.parametrize("shift", [0.0, 1e3])
@pytest.mark.parametrize("scale", [1e-20, 1e-12, 1e-3, 1.0, 1e15])
@pytest.mark.parametrize("kind", ["grid", "torus", "flat"])
def test_scales_equal_the_oracle(gpu, kind, scale, shift):
    if kind == "torus":
        m = motif_torus(nu=48, nv=24, copies=4, mirrored=1, noise=3e-3, seed=3)
    else:
        m = mirrored_heightfield(size=33, bumps=4, seed=5)
    v = m.vertices.copy()
    if kind == "flat":
        v[2] *= 1e-9
    p = prepare(Mesh(v, m.faces), Options())  # the topology of the mesh at unit scale
    move = np.array([shift, 0.5 * shift, 0.0])
    mesh = Mesh((v + move[:, None]) * scale, p.mesh.faces)
    ctx = ModelContext(p.context.box_size * scale, tuple((np.asarray(p.context.center) + move) * scale))
    o = Options(verify_threshold=0.02)
    c = np.asarray(ctx.center)
    turn = np.array([[0, -1.0, 0], [1.0, 0, 0], [0, 0, 1.0]])
    rigid = [(turn, c - turn @ c), (np.eye(3), np.array([1e-2 * scale, 0, 0])), (turn * np.nan, np.zeros(3)),
             (turn, np.array([np.inf, 0, 0]))]
    planes = [((1, 0, 0), -shift * scale), ((1, 1e-3, 0), -shift * scale)]
    got = gpu.verification(mesh, p.topology, records(rigid[:3], planes), ctx, o)
    want = oracle.OracleBackend().verification(mesh, p.topology, records(rigid[:3], planes), ctx, o)
    for k in ("coverage", "rms", "patches_a_groups", "patches_b_groups"):
        assert np.array_equal(getattr(got, k), getattr(want, k), equal_nan=k in ("coverage", "rms")), k
    for k in ("side_a", "side_b", "patches_a", "patches_b"):
        g, w = getattr(got, k), getattr(want, k)
        assert np.array_equal(g.offsets, w.offsets) and np.array_equal(g.indices, w.indices), k
    # An image at infinity lies beyond the threshold the device's search starts
    # from, so its motion is not supported (the oracle starts from infinity and
    # compares NaN); the other motions' results are as without it.
    with_inf = gpu.verification(mesh, p.topology, records(rigid, planes), ctx, o)
    assert with_inf.coverage[3] == 0
    assert np.array_equal(np.delete(with_inf.coverage, 3), got.coverage, equal_nan=True)
