"""A pinned state buffer is the caller's again when the call that took it
returns, also where nothing of the call waits for the device: sweeps of one
launch per level (no error word to read), no outputs, no norms."""
import numpy as np
import pytest

from helpers import assert_bitwise
from minifs_b200 import grid as gr, meshgen, solver as sv
from test_gpu_sweep_turns import renumbered

pytestmark = pytest.mark.gpu


def pinned(q):
    import torch
    t = torch.empty(q.size, dtype=torch.float64, pin_memory=True).numpy()
    t[:] = q
    return t


def spoil(q):
    """The last quarter first: a copy under way reads it last."""
    q[-(q.size // 4):] = 7.0
    q[:] = 7.0


@pytest.fixture(scope="module")
def large():
    """64^3 x 6 cells in random order: few levels (few launches), 64 MB of state."""
    p = gr.make_params(mach=0.5, alpha=2.0, cfl_start=10.0)
    prep = gr.DevicePrep(renumbered(meshgen.cube_mesh(64, jitter=0.1, seed=7), 7))
    q = prep.init_flow(p, bump_center=(0.4, 0.5, 0.6))
    s = sv.Solver.from_device_prep(prep, p, q)
    prep.close()
    s.set_sweep_mode(0)
    yield s, q
    s.close()


@pytest.mark.parametrize("n", [0, 1, 2])
def test_state_in_of_iterate_host(large, n):
    s, q = large
    for k in range(2):  # the second time with every table and stream there
        mine = pinned(q * (1.0 + 1e-3 * np.sin(np.arange(q.size))))
        s.sync()
        s.upload_q(mine)
        s.sync()
        s.iter_done = 0
        s.iterate(n)
        want = s.download("q")
        s.iter_done = 0
        s.iterate_host(n, mine, None, None)
        spoil(mine)
        assert_bitwise(s.download("q"), want, f"{n} iterations, time {k}")


def test_upload_before_iterate(large):
    s, q = large
    mine = pinned(q)
    for k in range(2):
        mine[:] = q
        s.iter_done = 0
        s.upload_q(mine)
        s.iterate(1, norms=False)
        spoil(mine)
        got = s.download("q")
        s.upload_q(q)
        s.sync()
        s.iter_done = 0
        s.iterate(1)
        assert_bitwise(got, s.download("q"), f"time {k}")


def test_upload_before_a_batch_s_time_step():
    p = [gr.make_params(mach=m, alpha=2.0, cfl_start=10.0) for m in (0.4, 0.6)]
    pg = [gr.prepare(meshgen.cube_mesh(36, jitter=0.1, seed=k), x, device=0)
          for k, x in enumerate(p)]
    s = sv.BatchSolver(pg, p)
    q = s.download("q")
    mine = pinned(q)
    for k in range(2):
        mine[:] = q * (1.0 + 0.01 * k)
        want = mine.copy()
        s.sync()
        s.upload_q(mine)
        s.compute_timestep()
        spoil(mine)
        assert_bitwise(s.download("q"), want, f"time {k}")
    s.close()
