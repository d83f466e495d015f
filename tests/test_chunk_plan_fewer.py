"""Sweeps of few cells per level take fewer chunks than the SMs offer: each
holds half a warp's item or more of the widest level, where a grid of all the
chunks, or the vote, would leave it less; and the model's choice is shorter
than the vote."""
import numpy as np
import pytest

from test_chunk_plan import T_XY, T_XZ, T_YZ, VOTE, plan, sweep_tables

ITEM = 16  # tetrahedra of a warp's item


@pytest.mark.parametrize("fwd", [True, False], ids=["forward", "backward"])
@pytest.mark.parametrize("n", [3, 6, 8])
def test_chunks_hold_half_an_item_of_the_widest_level(n, fwd):
    t = sweep_tables(n, fwd=fwd)
    widest = int(np.diff(t[2]).max())
    for P in (24, 48, 148):
        most = -(-2 * widest // ITEM)
        assert most < P * 3 // 4  # no grid near P chunks is within it
        rc, a, (pa, pb), est = plan(t, P, ITEM, -1)
        assert rc in (T_XY, T_XZ, T_YZ) and pa * pb <= most, (P, rc, pa, pb)
        assert len(np.unique(a)) <= most
        rc, a, _, est_vote = plan(t, P, ITEM, VOTE)
        assert rc == VOTE and len(np.unique(a)) > most
        assert est < est_vote
