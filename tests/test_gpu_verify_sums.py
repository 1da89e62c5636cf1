"""The serial sums of the verification (coverage, rms) and the result lists on
inputs where a parallel form of them can go wrong: vertex counts around the
sums' tile (4,096 addends), weights that tie in the rounding, span many
binades, vanish, are negative or not finite, sets without members.  Equal to
the oracle bit for bit."""
import dataclasses

import numpy as np
import pytest

from mitra_algo_gb300.mesh import motif_torus, prepare
from mitra_algo_gb300.types import Options
from oracle import oracle
from test_gpu_verify_resident import records

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    from mitra_algo_gb300 import Gb300Backend
    b = Gb300Backend(0)
    yield b
    b.close()


def weights(kind, n, rng):
    if kind == "ties":  # quarter units around powers of two
        return rng.integers(0, 9, n) * 2.0 ** rng.integers(-54, 0, n).astype(float)
    if kind == "spread":
        return 10.0 ** rng.uniform(-300, 300, n)
    if kind == "zeros":
        return np.where(rng.random(n) < 0.9, 0.0, rng.random(n))
    if kind == "tiny":
        return rng.random(n) * 1e-310
    if kind == "negative":
        return rng.normal(size=n)
    if kind == "nonfinite":
        w = rng.random(n)
        w[n // 2] = np.inf
        w[3 * n // 4] = np.nan
        return w
    return rng.random(n)


@pytest.mark.parametrize("nu,nv", [(24, 12), (64, 64), (241, 17), (90, 91)])
@pytest.mark.parametrize("kind", ["plain", "ties", "spread", "zeros", "tiny", "negative", "nonfinite"])
def test_sums_equal_the_oracle(gpu, kind, nu, nv):
    rng = np.random.default_rng(nu)
    o = Options(verify_threshold=0.02)
    p = prepare(motif_torus(nu=nu, nv=nv, copies=4, mirrored=1, noise=1e-3, seed=nu), o)
    topo = dataclasses.replace(p.topology, weights=weights(kind, nu * nv, rng))
    a, c, s = 2 * np.pi / 4, np.cos(2 * np.pi / 4), np.sin(2 * np.pi / 4)
    turn = np.array([[c, -s, 0], [s, c, 0], [0, 0, 1.0]])
    # a symmetry, a motion with no support, one off the surface
    rec = records(rigid=[(turn, np.zeros(3)), (np.eye(3), np.array([9.0, 0, 0])),
                         (turn, np.array([0.02 * a, 0, 0]))], planes=[((1, 0, 0), 0.0)])
    got = gpu.verification(p.mesh, topo, rec, p.context, o)
    want = oracle.OracleBackend().verification(p.mesh, topo, rec, p.context, o)
    for k in ("coverage", "rms", "patches_a_groups", "patches_b_groups"):
        assert np.array_equal(getattr(got, k), getattr(want, k), equal_nan=k in ("coverage", "rms")), k
    for k in ("side_a", "side_b", "patches_a", "patches_b"):
        g, w = getattr(got, k), getattr(want, k)
        assert np.array_equal(g.offsets, w.offsets) and np.array_equal(g.indices, w.indices), k
