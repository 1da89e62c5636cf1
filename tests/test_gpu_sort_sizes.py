"""The one-block sort and scan (up to 8,192 keys and 16,384 values) and the passes
over the whole device at the sizes where the one gives way to the other, through
what is built on them: the device's mesh preparation (corner, ring and edge
sorts, stable by construction) and the pairing (64-bit keys with ties) must
equal the host's preparation and the reference's acceptance of every pair."""
import numpy as np
import pytest

from helpers import features_from
from mitra_algo_gb300.mesh import prepare
from mitra_algo_gb300.types import Mesh, ModelContext, Options
from test_gpu_pairing_cells import accepted_partners

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    from mitra_algo_gb300 import Gb300Backend
    b = Gb300Backend(0)
    yield b
    b.close()


def strip(nf, seed):
    """A closed-up triangle strip of nf faces (3 nf corners, 6 nf ring entries)."""
    g = np.random.default_rng(seed)
    nv = nf + 2
    t = np.linspace(0, 40, nv)
    v = np.stack([np.cos(t) * (1 + 0.01 * t), np.sin(t) * (1 + 0.01 * t), 0.2 * t + 0.1 * (np.arange(nv) % 2)])
    v += g.normal(size=v.shape) * 1e-3
    i = np.arange(nf)
    f = np.stack([i, np.where(i % 2, i + 2, i + 1), np.where(i % 2, i + 1, i + 2)]).astype(np.int32)
    return Mesh(v, f)


# corners 3 nf and ring entries 6 nf around 1,024 .. 8,192 (keys) and 16,384
@pytest.mark.parametrize("nf", [1, 2, 170, 171, 341, 342, 682, 683, 1365, 1366, 2730, 2731, 5461, 5462])
def test_preparation(gpu, nf):
    o = Options()
    host, dev = prepare(strip(nf, nf), o), gpu.prepare(strip(nf, nf), o)
    np.testing.assert_array_equal(dev.mesh.faces, host.mesh.faces)
    t, u = dev.topology, host.topology
    for x, y in ((t.normals, u.normals), (t.face_normals, u.face_normals), (t.weights, u.weights),
                 (t.neighbors.offsets, u.neighbors.offsets), (t.neighbors.indices, u.neighbors.indices),
                 (t.incident_faces.offsets, u.incident_faces.offsets),
                 (t.incident_faces.indices, u.incident_faces.indices)):
        assert np.array_equal(x, y, equal_nan=True)


@pytest.mark.parametrize("samples", [2, 31, 1023, 1024, 1025, 2049, 4096, 8191, 8192, 8193, 12800, 12801, 16385])
def test_pairs(gpu, samples):
    rng = np.random.default_rng(samples)
    n = samples + 17
    pos = rng.uniform(-1, 1, (3, n))
    k0 = rng.normal(0, 1, n)
    k0[: n // 4] = np.round(k0[: n // 4], 2)  # equal keys
    k0[n // 2: n // 2 + 3] = [0.0, -0.0, 1e-300][:min(3, n - n // 2)]
    k1 = k0 + rng.uniform(0, 0.5, n)
    t = 0.2 if samples < 100 else 0.01
    sel = rng.permutation(n)[:samples].astype(np.int32)
    got = gpu.pairing(Mesh(pos, np.zeros((3, 0), np.int32)), features_from({"kmin": k0, "kmax": k1}, n), sel,
                      ModelContext(1.0), Options(pair_threshold=t, max_pairs=10 ** 9))
    ordinal = np.empty(n, np.int64)
    ordinal[sel] = np.arange(sel.size)
    ga, gb = ordinal[got.a], ordinal[got.b]
    starts = np.searchsorted(ga, np.arange(sel.size + 1))
    for a in range(0, sel.size, max(1, sel.size // 300)):
        assert np.array_equal(gb[starts[a]:starts[a + 1]], accepted_partners(a, sel, pos, k0, k1, t, 0.03)), a
