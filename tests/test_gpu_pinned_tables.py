"""Iterations where the host has no pinned memory left for the CFL and norm
tables: the same bits through pageable memory, and no CUDA error left behind.
cudaMallocHost is interposed in a process of its own."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))

SHIM = r"""
#include <dlfcn.h>
#include <stddef.h>
static int refuse, refused;
void shim_refuse(int on) { refuse = on; refused = 0; }
int shim_refused(void) { return refused; }
int cudaMallocHost(void **p, size_t n) {
  static int (*real)(void **, size_t);
  if (!real) /* the runtime that is loaded already, with its users' own scope */
    real = (int (*)(void **, size_t))dlsym(dlopen("libcudart.so.12", RTLD_LAZY | RTLD_NOLOAD),
                                           "cudaMallocHost");
  if (!refuse) return real(p, n);
  refused++;
  *p = NULL;
  return 2; /* cudaErrorMemoryAllocation */
}
"""

RUN = r"""
import ctypes, sys
sys.path[:0] = [{here!r}, {root!r}]
import numpy as np
from helpers import assert_bitwise
from minifs_b200 import grid as gr, meshgen
from minifs_b200.solver import BatchSolver, Solver
shim = ctypes.CDLL({shim!r})
p = gr.make_params(mach=0.5, alpha=2.0, cfl_start=10.0)
pg = gr.prepare(meshgen.cube_mesh(4, jitter=0.1, seed=2), p, bump_amp=0.05, bump_sigma=0.15)
for make in (lambda: Solver(pg, p), lambda: BatchSolver([pg, pg], [p, p])):
    a, b = make(), make()
    for s in (a, b):
        s.calculate_gradient()
    for n in (3, 300):  # the first tables, and larger ones
        shim.shim_refuse(1)
        na = a.iterate(n)
        assert shim.shim_refused() == 1
        shim.shim_refuse(0)
        assert_bitwise(na.reshape(-1), b.iterate(n).reshape(-1), f"norms of {{n}}")
    a.step(), b.step()
    assert_bitwise(a.download("q"), b.download("q"), "state")
    a.close(), b.close()
print("done")
"""


def test_iterate_without_pinned_memory(tmp_path):
    src, shim = tmp_path / "shim.c", tmp_path / "shim.so"
    src.write_text(SHIM)
    subprocess.run(["gcc", "-O1", "-D_GNU_SOURCE", "-shared", "-fPIC", "-o", str(shim), str(src),
                    "-ldl"], check=True)
    code = RUN.format(here=HERE, root=os.path.dirname(HERE), shim=str(shim))
    p = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, LD_PRELOAD=str(shim)))
    assert p.returncode == 0 and p.stdout.strip() == "done", (p.returncode, p.stderr[-2000:])
