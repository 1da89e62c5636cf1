"""The exact clustering's memory and its two forms of the supports: rows of hit counts
up to 16,384 votes of a kind, rows of bits and a second run of the used
trajectories above.  Both sides of that line, lists that leave the device in one
piece and in several, supports of whole words and of single votes: clusters,
memberships and RNG state equal the oracle's bit for bit, and the workspace stays
within its three pieces of at most 1 GiB (rows, a piece of the lists, the clusters'
counts) and the votes themselves."""
import numpy as np
import pytest

from mitra_algo_gb300.types import ModelContext, Options, Rng
from oracle import oracle
from test_gpu_cluster_lists import votes_of

pytestmark = pytest.mark.gpu


def descriptors(shape, q):
    rng = np.random.default_rng(q)
    d = rng.uniform(-0.4, 0.4, (12, q))
    if shape == "same":
        return np.repeat(d[:, :1], q, axis=1)
    of = rng.integers(0, 3000, q)
    if shape == "runs":  # neighbours in vote order share a window
        of.sort()
    return d[:, :3000][:, of] + rng.normal(0, 0.002, (12, q))


@pytest.mark.parametrize("shape,q,planes", [
    ("clumps", 16384, 0), ("clumps", 16385, 0), ("runs", 16385, 1), ("runs", 17001, 17000),
    ("clumps", 18000, 1000), ("same", 16384, 0), ("same", 16500, 16500), ("same", 24001, 1)])
def test_supports_and_memory(shape, q, planes):
    from mitra_algo_gb300 import Gb300Backend
    gpu = Gb300Backend(0, profile=True)  # a workspace of its own
    try:
        kind = (np.arange(q) < planes)[np.random.default_rng(q).permutation(q)]
        d = descriptors(shape, q)
        d[4:, kind] = 0
        o = Options(bandwidth=0.05, max_clusters=50, max_iterations=60, seed=9)
        ctx = ModelContext(2.0, (0.1, 0.2, 0.3))
        r1, r2 = Rng(9), oracle.rng(9)
        got = gpu.clustering(votes_of(d, kind), ctx, o, r1)
        peak = gpu.take_metrics()[-1]["peak_buffer_bytes"]
        want = oracle.OracleBackend().clustering(votes_of(d, kind), ctx, o, r2)
    finally:
        gpu.close()
    assert r1 == r2 and got.limited_iterations == want.limited_iterations
    assert np.array_equal(got.votes.offsets, want.votes.offsets)
    assert np.array_equal(got.votes.indices, want.votes.indices)
    for k in ("reflection", "rotation", "translation", "plane_normal", "plane_offset"):
        assert np.array_equal(getattr(got, k), getattr(want, k), equal_nan=True), k
    assert peak < (3 << 30) + 1024 * q
