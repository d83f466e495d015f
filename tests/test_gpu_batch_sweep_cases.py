"""A batch's case ids in the persistent sweeps' tables: more cases than the
sweeps keep on the SM, cases of 6 cells beside larger ones, each with its own
flow and its own LimitTimeStep ratio, tables built on the host and (after the
autotuner's rebuilds) on the device: the bits of the one-launch-per-level
sweeps, which read a cell's case by its index."""
import pytest

from helpers import assert_bitwise

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("count", [2, 131])
def test_case_ids_of_host_and_device_tables(count, precision):
    from minifs_b200 import grid as gr, meshgen
    from minifs_b200.solver import BatchSolver
    grids, params = [], []
    for k in range(count):
        m = meshgen.cube_mesh(1 + k % 5, jitter=0.1, seed=k)
        p = gr.make_params(mach=0.3 + 0.004 * k, alpha=0.1 * (k % 7), cfl_start=5.0 + k % 11,
                           ratio_dtmax=2.0 if k % 3 == 0 else 1.0e80)
        grids.append(gr.prepare(m, p, bump_amp=0.05, bump_sigma=0.15))
        params.append(p)
    host, tuned, ref = (BatchSolver(grids, params, precision=precision) for _ in range(3))
    tuned.autotune(1)
    ref.set_sweep_mode(0)
    for s in (host, tuned, ref):
        s.set_sweep_mode(0 if s is ref else 1)
        s.calculate_gradient()
        s.iterate(4)
    for f in ("q", "res", "dt", "diag", "dq", "dqdx"):
        want = ref.download(f)
        assert_bitwise(host.download(f), want, f"host tables: {f}")
        assert_bitwise(tuned.download(f), want, f"device tables: {f}")
    for s in (host, tuned, ref):
        s.close()
