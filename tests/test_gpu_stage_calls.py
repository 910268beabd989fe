"""GPU tests of the stage calls' own resources: a set-up call that fails once,
and calls from two threads."""
import os
import subprocess
import sys
import textwrap
import threading

import numpy as np
import pytest

import hptracing_b200 as H
from tests import scenes as S

pytestmark = pytest.mark.gpu

# A cudaMemPoolCreate that fails the first time.
SHIM = """
#define _GNU_SOURCE
#include <dlfcn.h>
int cudaMemPoolCreate(void** pool, const void* props) {
  static int calls = 0;
  if (calls++ == 0) return 2; /* cudaErrorMemoryAllocation */
  void* lib = dlopen("libcudart.so.12", RTLD_NOW | RTLD_NOLOAD);
  int (*real)(void**, const void*) = dlsym(lib, "cudaMemPoolCreate");
  return real(pool, props);
}
"""

CALLER = """
import numpy as np
import hptracing_b200 as H
from tests import scenes as S
mesh, nodes, leaf = S.make_scene(0)
scene = H.Scene(mesh, nodes, leaf)
o, d = S.aabb_random_rays(mesh, 100, 1)
try:
    scene.intersect(o, d)
    print("no failure")
except RuntimeError as e:
    print("failed once")
print(int((scene.intersect(o, d)[0] >= 0).sum()))
"""


def test_a_pool_that_failed_once_is_made_by_the_next_call(built, tmp_path):
    if H.device_count() == 0:
        pytest.skip("no CUDA device")
    (tmp_path / "shim.c").write_text(SHIM)
    shim = str(tmp_path / "shim.so")
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", shim, str(tmp_path / "shim.c"), "-ldl"], check=True)
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", textwrap.dedent(CALLER)], cwd=root, capture_output=True, text=True,
                       env=dict(os.environ, LD_PRELOAD=shim, PYTHONPATH=root), timeout=300)
    mesh, nodes, leaf = S.make_scene(0)
    hits = int((H.Scene(mesh, nodes, leaf).intersect(*S.aabb_random_rays(mesh, 100, 1))[0] >= 0).sum())
    assert r.stdout.split("\n")[:2] == ["failed once", str(hits)], r.stdout + r.stderr[-2000:]


def test_stage_calls_from_two_threads(built):
    if H.device_count() == 0:
        pytest.skip("no CUDA device")
    mesh, nodes, leaf = S.make_scene(0)
    scene = H.Scene(mesh, nodes, leaf)
    rays = [S.aabb_random_rays(mesh, 3000 + 997 * k, k) for k in range(4)]
    want = [scene.intersect(*r) for r in rays]
    got = [None] * 4

    def work(k):
        for _ in range(5):
            got[k] = scene.intersect(*rays[k])

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for w, g in zip(want, got):
        assert all(np.array_equal(a, b) for a, b in zip(w, g))
