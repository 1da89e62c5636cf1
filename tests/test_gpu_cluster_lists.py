"""The exact clustering's vote lists at their edges: windows of a few votes, of
more than 32 (one gathered group) and more than 1,024 (no list is kept), means
that travel several bandwidths (the list is made anew), counts around a warp,
coordinates far from the origin, one kind only.  Clusters, memberships and RNG
state equal the oracle's bit for bit."""
import numpy as np
import pytest

from mitra_algo_gb300.types import ModelContext, Options, Rng, Votes
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    from mitra_algo_gb300 import Gb300Backend
    b = Gb300Backend(0)
    yield b
    b.close()


def votes_of(descriptor, kind):
    q = kind.size
    eye = np.repeat(np.eye(3).reshape(9, 1), q, axis=1)
    return Votes(np.arange(q, dtype=np.int32), kind.astype(np.uint8), eye, np.zeros((3, q)),
                 np.zeros((3, q)), np.zeros(q), descriptor)


@pytest.mark.parametrize("shape", ["clumps", "dense", "slope", "far", "same"])
@pytest.mark.parametrize("q,planes", [(1, 1), (31, 0), (33, 33), (200, 60), (2500, 2400), (2500, 30)])
def test_lists_equal_the_oracle(gpu, shape, q, planes):
    rng = np.random.default_rng(q + planes)
    kind = (np.arange(q) < planes)[rng.permutation(q)]
    d = rng.uniform(-0.4, 0.4, (12, q))
    if shape == "dense":  # whole windows of more than 1,024 votes
        d = rng.normal(0, 0.004, (12, q))
    elif shape == "slope":  # density rising along one axis: means travel
        d = rng.normal(0, 0.003, (12, q))
        d[2] = d[9] = 0.5 * np.sqrt(rng.random(q))
    elif shape == "clumps":
        d = rng.uniform(-0.4, 0.4, (12, 40))[:, rng.integers(0, 40, q)] + rng.normal(0, 0.004, (12, q))
    elif shape == "far":
        d = 500 + rng.normal(0, 0.01, (12, q))
    elif shape == "same":
        d = np.repeat(d[:, :1], q, axis=1)
    d[4:, kind] = 0
    o = Options(bandwidth=0.05, max_clusters=50, max_iterations=60, seed=9)
    ctx = ModelContext(2.0, (0.1, 0.2, 0.3))
    r1, r2 = Rng(9), oracle.rng(9)
    got = gpu.clustering(votes_of(d, kind), ctx, o, r1)
    want = oracle.OracleBackend().clustering(votes_of(d, kind), ctx, o, r2)
    assert r1 == r2 and got.limited_iterations == want.limited_iterations
    assert np.array_equal(got.votes.offsets, want.votes.offsets)
    assert np.array_equal(got.votes.indices, want.votes.indices)
    for k in ("reflection", "rotation", "translation", "plane_normal", "plane_offset"):
        assert np.array_equal(getattr(got, k), getattr(want, k), equal_nan=True), k
