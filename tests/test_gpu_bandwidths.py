"""Bandwidths whose squares lie at the ends of FP32 and beyond: the weights' quotient
d^2 / h^2 stays what the division gives, so a window that holds one vote leaves its
seed where it is, and one that holds every vote with weight 1 takes it to their
mean.  And the quotients themselves against the division, bit for bit."""
import subprocess

import numpy as np
import pytest

from mitra_algo_gb300 import build

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    from mitra_algo_gb300 import Gb300Backend
    b = Gb300Backend(0)
    yield b
    b.close()


def votes_of(q):
    g = np.random.default_rng(q)
    centres = g.uniform(-1, 1, (4, 6))
    return (centres[np.arange(q) % 4] + g.normal(0, 0.01, (q, 6))).astype(np.float32).astype(np.float64)


# 1,200 votes: the direct grid; 70,000 with 8,192 seeds: the work items
@pytest.mark.parametrize("q,k", [(1200, 33), (70000, 8192)])
@pytest.mark.parametrize("kernel", ["epanechnikov", "gaussian"])
@pytest.mark.parametrize("h", [1e-23, 1e-22, 1e-21, 3e-20, 1e-19, 1e-18, 5e-10, 1e-9, 2e-9])
def test_tiny(gpu, h, kernel, q, k):
    v = votes_of(q)
    seeds = np.linspace(0, q - 1, k).astype(np.int64)
    means, _, _ = gpu.meanshift6(v, seeds, h, "fp32", 6, 3, kernel)
    assert np.array_equal(means, v[seeds])


@pytest.mark.parametrize("q,k", [(1200, 33), (70000, 8192)])
@pytest.mark.parametrize("kernel", ["epanechnikov", "gaussian"])
@pytest.mark.parametrize("h", [1e8, 1.0e9, 1.1e9, 2e9, 1e18, 1.3e19, 1.8e19, 1.9e19, 1e20, 1e30, 1e200])
def test_huge(gpu, h, kernel, q, k):
    v = votes_of(q)
    seeds = np.linspace(0, q - 1, k).astype(np.int64)
    means, state, _ = gpu.meanshift6(v, seeds, h, "fp32", 6, 3, kernel)
    assert np.all(state == 1)
    # FP32 sums of q terms of at most 3 in runs of at least 16 votes: q / 16 + 16 + 16
    # roundings of 6e-8 of a partial sum, over the q votes
    assert np.max(np.abs(means - v.mean(0))) < 3 * 6e-8 * (q / 16 + 32)


def test_quotients(tmp_path):
    tool = tmp_path / "quotient_check"
    source = build.HERE.parent / "tests" / "quotient_check.cu"
    subprocess.run([build.nvcc(), "-O3", "-std=c++17", "--fmad=true", *build.ARCH, "-I", str(build.SRC),
                    "-o", str(tool), str(source)], check=True)
    r = subprocess.run([str(tool)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
