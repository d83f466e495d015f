"""Chunk assignments of sweeps with few cells per level, planned on the host:
a level smaller than the chunks' count is not spread over all of them."""
import numpy as np
import pytest

from test_chunk_plan import T_XY, T_XZ, T_YZ, dependencies, plan, sweep_tables


@pytest.mark.parametrize("fwd", [True, False], ids=["forward", "backward"])
@pytest.mark.parametrize("n", [3, 6])
def test_small_levels_take_fewer_chunks_and_stay_monotone(n, fwd):
    t = sweep_tables(n, fwd=fwd)
    P = 148
    rc, a, (pa, pb), est = plan(t, P, 16, -1)
    assert est > 0 and a.min() >= 0 and a.max() < P
    if rc in (T_XY, T_XZ, T_YZ):
        assert 1 <= pa * pb <= P and a.max() < pa * pb
        for lab in (a % pa, a // pa):
            d = np.sign([lab[c] - lab[e] for c, e in dependencies(t)])
            assert (d >= 0).all() or (d <= 0).all()
    # the model's own choice is never slower, by the model, than a forced one
    for force in (0, 4):
        assert est <= plan(t, P, 16, force)[3] * (1 + 1e-12)
    assert len(np.unique(a)) < P
