"""mean_shift_pairs, the seed-vote evaluations of the mean shift: the (tile, chunk) pairs
within the bandwidth of some seed of the tile, whichever route an iteration takes.
In the first iteration the FP32 form and the tensor kernel start from the same
seeds, so their chunks are the same; the tensor kernel counts a whole last chunk per
tile that takes it, the FP32 form its votes."""
import pytest

from mitra_algo_gb300 import Gb300Backend, Options
from mitra_algo_gb300.mesh import motif_sphere, motif_torus

pytestmark = pytest.mark.gpu
CHUNK = 128


@pytest.fixture(scope="module")
def gpu():
    b = Gb300Backend(0)
    yield b
    b.close()


# up to 32,768 (tile, chunk) pairs the direct grid, the last ones the work items
@pytest.mark.parametrize("mesh,samples,seeds,bandwidth,blocks", [
    ("sphere", 400, 1, 0.1, 0), ("sphere", 400, 64, 0.1, 0), ("sphere", 2000, 128, 0.02, 0),
    ("sphere", 2000, 129, 0.1, 0), ("sphere", 3000, 300, 0.1, 0), ("sphere", 3000, 300, 0.1, 1),
    ("torus", 2500, 700, 0.05, 7), ("torus", 2500, 1000, 0.2, 1), ("torus", 4000, 2048, 0.1, 0)])
def test_first_iteration(gpu, mesh, samples, seeds, bandwidth, blocks):
    m = motif_sphere(level=5, noise=1e-3, seed=1) if mesh == "sphere" else \
        motif_torus(nu=171, nv=85, copies=12, mirrored=2, bumps=2, noise=5e-4, seed=2)
    o = Options(sample_ratio=samples / m.vertex_count, pair_threshold=0.05, bandwidth=bandwidth,
                max_pairs=10 ** 8, max_votes=2 * 10 ** 9 - 1, max_clusters=4)
    resident = gpu.load_mesh_raw(m, o)
    run = {p: gpu.detect_fast(resident, None, o, precision=p, seeds=seeds, max_iterations=1,
                              polish_iterations=0, verify=False,
                              tuning={"simt_blocks_per_sm": blocks} if blocks else None)
           for p in ("fp32", "bf16")}
    resident.close()
    votes, tiles = run["fp32"]["votes"], -(-seeds // CHUNK)
    want = run["bf16"]["tc_evaluations"]
    missing = CHUNK * (-votes % CHUNK)  # of a tile that takes the last chunk
    got = run["fp32"]["mean_shift_pairs"]
    assert votes > CHUNK and want % CHUNK ** 2 == 0
    assert (want - got) in {t * missing for t in range(tiles + 1)}, (votes, got, want)
