"""The bookkeeping kernels of the mean-shift loops (active seeds ranked by many
blocks, chunk lists and plan scanned by one, seeds updated eight to a block) at
their edges: seed counts around 32, 128, 2,048 (the most that are sorted) and
4,096, vote counts from one chunk to some hundred, every kernel and precision.

Every seed of the bulk ends at a mode of the planted set: the modes must be the
planted centres, to the FP32 tolerance of tests/test_gpu_meanshift.py (1e-5 of a
unit scale), each found once, and two runs of the same call must agree bit for
bit (no order of arrival enters a result)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    from mitra_algo_gb300 import Gb300Backend
    b = Gb300Backend(0)
    yield b
    b.close()


def planted(votes, modes, seed):
    """`modes` centres at least 1.2 apart, each with an equal share of the votes
    in symmetric pairs within 0.02, so a centre is its mode's mean exactly."""
    g = np.random.default_rng(seed)
    grid = np.stack(np.meshgrid(*[[-0.6, 0.6]] * 6), -1).reshape(-1, 6)
    centres = grid[g.permutation(len(grid))[:modes]]
    pairs = max(1, votes // (2 * modes))
    d = g.uniform(-0.01, 0.01, size=(modes, pairs, 6))
    v = np.concatenate([centres[:, None] + d, centres[:, None] - d], 1).reshape(-1, 6)
    return v[g.permutation(len(v))], centres


@pytest.mark.parametrize("precision,kernel", [("bf16", "epanechnikov"), ("fp32", "epanechnikov"),
                                              ("bf16", "gaussian"), ("fp64", "epanechnikov")])
@pytest.mark.parametrize("seeds", [1, 31, 32, 33, 127, 128, 129, 2047, 2048, 2049, 4095, 4097])
def test_seed_counts(gpu, seeds, precision, kernel):
    votes, centres = planted(max(2 * seeds, 9000), 6, seeds)
    pick = np.random.default_rng(seeds + 1).choice(len(votes), seeds, replace=False)
    out = gpu.meanshift6(votes, pick, 0.1, precision, 100, 30, kernel)
    again = gpu.meanshift6(votes, pick, 0.1, precision, 100, 30, kernel)
    for a, b in zip(out[:2], again[:2]):
        assert np.array_equal(a, b)
    means = np.asarray(out[0])[:, :6]
    near = np.abs(means[:, None] - centres[None]).max(-1)
    assert np.array_equal(near.argmin(1), np.abs(votes[pick][:, None] - centres[None]).max(-1).argmin(1))
    assert near.min(1).max() < 1e-5


@pytest.mark.parametrize("votes", [6, 127, 128, 129, 32767, 32769, 98303, 98306])
def test_vote_counts(gpu, votes):
    v, centres = planted(votes, 3, votes)
    pick = np.arange(min(len(v), 200))
    for precision in ("bf16", "fp32"):
        out = gpu.meanshift6(v, pick, 0.1, precision, 100, 30, "epanechnikov")
        means = np.asarray(out[0])[:, :6]
        near = np.abs(means[:, None] - centres[None]).max(-1)
        assert np.array_equal(near.argmin(1), np.abs(v[pick][:, None] - centres[None]).max(-1).argmin(1))
        assert near.min(1).max() < 1e-5


@pytest.mark.parametrize("precision,kernel", [("fp32", "epanechnikov"), ("fp32", "gaussian"),
                                              ("fp64", "epanechnikov"), ("bf16", "epanechnikov")])
@pytest.mark.parametrize("votes", [3000, 40000])  # direct, and by work items
def test_iteration_limits(gpu, votes, precision, kernel):
    """The host looks at the seeds every few iterations only: whatever the limit
    relative to that, it is kept, and a limit past the last iteration changes
    nothing, also with a polish that finds seeds still moving."""
    g = np.random.default_rng(votes)
    v = g.normal(size=(votes, 6)) * 0.2
    pick = g.choice(votes, 300, replace=False)
    long = gpu.meanshift6(v, pick, 0.3, precision, 500, 0, kernel)
    total = long[2][0]
    assert 3 < total < 500
    for limit in [1, 2, 3, 4, 5, 6, 7, 8, 9, total - 1, total, total + 1, total + 9]:
        out = gpu.meanshift6(v, pick, 0.3, precision, limit, 0, kernel)
        assert out[2][0] == min(limit, total)
        if limit >= total:
            assert np.array_equal(out[0], long[0]) and np.array_equal(out[1], long[1])
    for limit in (1, 2, 5):  # the polish goes on with moving seeds
        ends = [gpu.meanshift6(v, pick, 0.3, precision, limit, polish, kernel) for polish in (200, 201, 203)]
        assert ends[0][2][1] < 200
        for e in ends[1:]:
            assert e[2] == ends[0][2]
            assert np.array_equal(e[0], ends[0][0]) and np.array_equal(e[1], ends[0][1])


def test_tensor_kernel_time(gpu):
    """The tensor kernel's own time is taken on the device, launch by launch:
    positive, below the phase's, as many launches as iterations."""
    from mitra_algo_gb300.mesh import motif_sphere, prepare
    from mitra_algo_gb300.types import Options
    mesh = motif_sphere(level=4, bumps=12, folds=5, partial_shift=0.4, noise=1e-3, seed=0)
    o = Options(sample_ratio=0.5, pair_threshold=0.25, bandwidth=0.1, max_pairs=10 ** 7, max_votes=10 ** 8)
    r = gpu.load_mesh(prepare(mesh, o))
    d = gpu.detect_fast(r, None, o, precision="bf16", seeds=128, max_iterations=60, polish_iterations=30)
    r.close()
    assert d["tc_launches"] == d["iterations"] > 0
    assert 0 < d["tc_kernel_ms"] < d["bulk_ms"]
