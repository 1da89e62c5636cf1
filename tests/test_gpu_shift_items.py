"""The FP32 mean shift's work items at their edges: vote counts around a run
(16), a chunk (128) and a block of chunks (32,768), seed counts around a warp
(32) and a tile (128), on both sides of the rule that chooses listed items.
Compared with the FP64 restatement (oracle/meanshift6.py) after one plain step
from the same seeds: 1e-5 relative, the bound of tests/test_gpu_meanshift.py."""
import numpy as np
import pytest

from oracle.meanshift6 import meanshift6

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    from mitra_algo_gb300 import Gb300Backend
    b = Gb300Backend(0)
    yield b
    b.close()


def case(q, k, seed):
    """Half the votes in a tight cluster, so windows hold several votes."""
    rng = np.random.default_rng(seed)
    votes = np.concatenate([rng.normal(0.3, 0.02, (q // 2, 6)), rng.uniform(-1, 1, (q - q // 2, 6))])
    votes = votes.astype(np.float32).astype(np.float64)[rng.permutation(q)]
    return votes, np.sort(rng.choice(q, k, replace=False))


@pytest.mark.parametrize("kernel", ["epanechnikov", "gaussian"])
@pytest.mark.parametrize("q,k", [(1, 1), (15, 3), (16, 16), (17, 17), (127, 31), (129, 33), (1000, 129),
                                 (32769, 32), (33000, 160), (70001, 8200), (900001, 640)])
def test_steps_match_fp64(gpu, kernel, q, k):
    votes, seeds = case(q, k, q + k)
    means, _, _ = gpu.meanshift6(votes, seeds, 0.15, "fp32", 1, 0, kernel)
    pick = slice(None) if q < 2000 else slice(0, None, max(1, k // 40))
    ref, _, _ = meanshift6(votes, seeds[pick], 0.15, 1, 0, kernel=kernel)
    err = np.linalg.norm(means[pick] - ref, axis=1) / np.maximum(np.linalg.norm(ref, axis=1), 1e-300)
    assert err.max() <= 1e-5, err.max()
