"""Kernels that need more than 48 KB of dynamic shared memory, with several contexts in
one process.  The limit belongs to a device, so every context asks for its own,
and once: a context on another device of the process must not find it unset.  With
one device that is seen at the runtime: a shim in front of cudaFuncSetAttribute
notes the kernel of each call and passes the call on."""
import os
import shutil
import subprocess
import sys
from collections import Counter
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

SHIM = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stdio.h>
#include <stdlib.h>
int cudaFuncSetAttribute(const void *kernel, int attribute, int value) {
  void *runtime = dlopen("libcudart.so.13", RTLD_NOLOAD | RTLD_LAZY);  /* the library's own */
  int (*next)(const void *, int, int) = dlsym(runtime, "cudaFuncSetAttribute");
  FILE *f = fopen(getenv("SHARED_LIMITS"), "a");
  fprintf(f, "%p\n", kernel);
  fclose(f);
  return next(kernel, attribute, value);
}
"""
# sorts of 1,025 to 8,192 keys (each of their instances), the tensor kernel and its
# self-test, twice in each of two contexts
CHILD = """
import numpy as np
from mitra_algo_gb300 import Gb300Backend, Options
from mitra_algo_gb300.mesh import mirrored_heightfield
votes = np.random.default_rng(1).normal(0, 0.05, (3000, 6))
ones = lambda *shape: np.full(shape, 0x3f80, np.uint16)
for _ in range(2):
    gpu = Gb300Backend(0)
    for _ in range(2):
        for size in (24, 40, 60):
            gpu.load_mesh_raw(mirrored_heightfield(size=size, bumps=3, seed=1), Options()).close()
        gpu.meanshift6(votes, np.arange(64), 0.2, "bf16", 5, 2)
        gpu.tc_selftest(ones(128, 16), ones(128, 16), ones(128, 128), ones(16, 128))
    gpu.close()
"""


def test_every_context_asks_once(tmp_path):
    cc = shutil.which("gcc") or shutil.which("cc")
    if not cc:
        pytest.skip("no C compiler")
    (tmp_path / "shim.c").write_text(SHIM)
    shim, log = tmp_path / "shim.so", tmp_path / "calls"
    subprocess.run([cc, "-shared", "-fPIC", "-o", shim, tmp_path / "shim.c", "-ldl"], check=True)
    env = {**os.environ, "LD_PRELOAD": str(shim), "SHARED_LIMITS": str(log),
           "PYTHONPATH": str(Path(__file__).resolve().parents[1])}
    subprocess.run([sys.executable, "-c", CHILD], env=env, check=True, timeout=300)
    calls = Counter(log.read_text().split())
    assert len(calls) >= 5 and set(calls.values()) == {2}
