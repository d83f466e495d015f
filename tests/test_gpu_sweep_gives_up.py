"""Sweeps whose waits give up, on chunks of many more levels than there are
level barriers: the call reports it, the kernel ends, and the context goes on
with the bits of one that never timed out.  A warp that gave up may not arrive
at its level's barrier: the order of the arrivals is all that keeps their
count within the barrier's."""
import pytest

from helpers import assert_bitwise
from minifs_b200 import _lib, grid as gr, meshgen
from minifs_b200.solver import BatchSolver, Solver

pytestmark = pytest.mark.gpu

MESHES = {
    "long": lambda: meshgen.box_mesh(2, 2, 200, lz=100.0, jitter=0.1, seed=4),
    "cube": lambda: meshgen.cube_mesh(14, jitter=0.15, seed=7),
    "prisms": lambda: meshgen.hexprism_mesh(7, 6, 40, jitter=0.1, seed=5),
}


def prepared(name):
    p = gr.make_params(mach=0.5, alpha=2.0, cfl_start=10.0)
    return gr.prepare(MESHES[name](), p, bump_amp=0.05, bump_sigma=0.15), p


def made(make, kind, chunking):
    lib = _lib.load()
    assert lib.mfg_set_sweep_kernel(kind) == 0 and lib.mfg_set_chunking(chunking) == 0
    try:
        return make()
    finally:
        lib.mfg_set_sweep_kernel(-1)
        lib.mfg_set_chunking(-1)


def check(make, kind, chunking):
    s, ref = made(make, kind, chunking), made(make, kind, chunking)
    assert s.info()["sweep_mode"] == 1 and s.info()["sweep_chunks"] >= 2, s.info()
    for x in (s, ref):
        x.calculate_gradient()
    for spin in (200_000, 1_000_000):
        assert s.selftest_sweep_timeout(spin) == -4
        for x in (s, ref):
            x.iterate(2)
        for f in ("q", "res", "dq", "dqdx"):
            assert_bitwise(s.download(f), ref.download(f), f"{f} after a time-out of {spin}")
    for x in (s, ref):
        x.close()


@pytest.mark.parametrize("chunking", [0, 4], ids=["vote", "transverse"])
@pytest.mark.parametrize("kind", [0, 1], ids=["deep", "wide"])
@pytest.mark.parametrize("name", list(MESHES))
def test_context_goes_on_after_waits_gave_up(name, kind, chunking):
    pg, p = prepared(name)
    for precision in ("fp64", "mixed"):
        check(lambda: Solver(pg, p, precision=precision), kind, chunking)


def test_batch_goes_on_after_waits_gave_up():
    both = [prepared(name) for name in ("long", "cube")]
    check(lambda: BatchSolver([pg for pg, _ in both], [p for _, p in both]), 0, 0)
