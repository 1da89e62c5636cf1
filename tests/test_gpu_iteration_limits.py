"""Iteration limits far beyond what the seeds need: same result, traces and counts as
with a limit of some hundred, and not a byte more of workspace."""
import numpy as np
import pytest

from mitra_algo_gb300 import Gb300Backend, Options
from mitra_algo_gb300.mesh import motif_sphere

pytestmark = pytest.mark.gpu
LIMITS = ((400, 400), (200_000_000, 200_000_000))


def peak(gpu):
    return gpu.take_metrics()[-1]["peak_buffer_bytes"]


@pytest.mark.parametrize("precision", ["fp32", "bf16", "fp64"])
def test_modes(precision):
    gpu = Gb300Backend(0, profile=True)
    g = np.random.default_rng(2)
    votes = np.concatenate([c + g.normal(0, 0.01, (500, 6)) for c in g.uniform(-1, 1, (6, 6))])
    got = []
    for limit in LIMITS:
        means, state, iterations = gpu.meanshift6(votes, np.arange(0, 3000, 13), 0.06, precision, *limit)
        got.append((means, state, iterations, peak(gpu)))
    gpu.close()
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])
    assert got[0][2:] == got[1][2:]


@pytest.mark.parametrize("precision", ["fp32", "bf16"])
def test_detection(precision):
    gpu = Gb300Backend(0, profile=True)
    m = motif_sphere(level=4, noise=1e-3, seed=1)
    o = Options(sample_ratio=2000 / m.vertex_count, pair_threshold=0.05, bandwidth=0.1, max_pairs=10 ** 8,
                max_votes=10 ** 9, max_clusters=4)
    resident = gpu.load_mesh_raw(m, o)
    got = []
    for limit in LIMITS:
        r = gpu.detect_fast(resident, None, o, precision=precision, seeds=128, max_iterations=limit[0],
                            polish_iterations=limit[1], reference_seeds=8)
        got.append([r[k] for k in ("iterations", "polish_iterations", "bulk_trace", "polish_trace", "seed_iterations",
                                   "mean_shift_pairs", "modes", "support", "rotation", "translation",
                                   "mode_error_max", "tc_launches", "tc_evaluations")] + [peak(gpu)])
        assert r["seed_iterations"] == sum(r["bulk_trace"]) + sum(r["polish_trace"])
        if precision == "bf16":  # launches of some microseconds each, within their phase
            assert 1e-3 * r["iterations"] < r["tc_kernel_ms"] < r["bulk_ms"]
    resident.close()
    gpu.close()
    assert got[0] == got[1]
