"""Which increments the persistent sweeps take from a block's ring: levels of
more cells per chunk than the ring has rows.  Two cells of one level then share
a row, and their warps write it in no order, so neither the tables built on the
host nor those built on the device may read such a row, whatever the length of
the level that reads.  The tables' counts against the rule written out, and the
bits of the one-launch-per-level sweeps."""
import numpy as np
import pytest

from helpers import assert_bitwise
from minifs_b200 import _lib, grid as gr, meshgen
from minifs_b200.solver import Solver
from test_chunk_plan import VOTE, plan
from test_gpu_sweep_turns import renumbered

RING = 512  # rows


def large():
    p = gr.make_params(mach=0.5, alpha=2.0, cfl_start=10.0)
    return renumbered(meshgen.cube_mesh(48, jitter=0.1, seed=7), 7), p


def records(f2c, C, P, fwd):
    """A sweep's records by where their increment comes from: the ring, the
    chunk's own cells otherwise, other chunks; and how many rows of the first
    kind would be had without the order within a level."""
    f = np.asarray(f2c).reshape(-1, 2)
    pairs = f[(f < C).all(1)]
    a = np.concatenate([pairs[:, 0], pairs[:, 1]])
    b = np.concatenate([pairs[:, 1], pairs[:, 0]])
    face = np.tile(np.flatnonzero((f < C).all(1)), 2)  # a cell's records are in face order
    dep = np.flatnonzero((b < a) if fwd else (b > a))
    dep = dep[np.argsort(face[dep], kind="stable")]
    a, b = a[dep], b[dep]
    count = np.bincount(a, minlength=C)
    if not fwd:  # the ghosts' faces are swept backward
        count += np.bincount(f[(f >= C).any(1), 0], minlength=C)
    level = np.zeros(C, np.int64)
    while True:
        new = np.zeros(C, np.int64)
        np.maximum.at(new, a, level[b] + 1)
        if (new == level).all():
            break
        level = new
    cells = np.lexsort((np.arange(C), level)).astype(np.int32)
    L = int(level.max()) + 1
    lptr = np.searchsorted(level[cells], np.arange(L + 1)).astype(np.int32)
    place = np.empty(C, np.int64)
    place[cells] = np.arange(C)
    order = np.argsort(place[a], kind="stable")
    sptr = np.zeros(C + 1, np.int32)
    sptr[1:] = np.cumsum(np.bincount(place[a], minlength=C))
    t = (C, L, lptr, cells, sptr, b[order].astype(np.int32), [np.zeros(C)] * 3)
    rc, chunk, _, _ = plan(t, P, 16, VOTE, geo=False)
    assert rc == VOTE
    # chunk by chunk, level by level, cells of many records first
    at = np.lexsort((np.arange(C), -count, level, chunk))
    pos = np.empty(C, np.int64)
    pos[at] = np.arange(C)
    last = np.iinfo(np.int64).max

    def level_at(p, own):
        """The level of the cell at position p, if it is of chunk `own`."""
        inside = (p >= 0) & (p < C)
        c = at[np.clip(p, 0, C - 1)]
        return np.where(inside & (chunk[c] == own), level[c], last)

    same = chunk[a] == chunk[b]
    later = level_at(pos[b] + RING, chunk[b]) <= level[a]
    mixed = level_at(pos[b] - RING, chunk[b]) == level[b]
    ring = same & ~later & ~mixed
    return (int(ring.sum()), int((same & ~ring).sum()), int((~same).sum()),
            int((same & ~later & mixed).sum()))


def test_such_rows_exist_on_this_mesh():
    mesh, p = large()
    m = gr.prepare(mesh, p)
    for fwd in (True, False):
        assert records(m.arrays["f2c"], m.n_cell, 148, fwd)[3] > 1000


@pytest.mark.gpu
@pytest.mark.parametrize("built", ["host", "device"])
def test_tables_and_bits(built):
    mesh, p = large()
    pg = gr.prepare(mesh, p, bump_amp=0.05, bump_sigma=0.15, device=0)
    lib = _lib.load()
    assert lib.mfg_set_sweep_kernel(0) == 0 and lib.mfg_set_chunking(VOTE) == 0
    try:
        if built == "host":
            s = Solver(pg, p)
        else:
            prep = gr.DevicePrep(mesh)
            s = Solver.from_device_prep(prep, p, pg.q0)
            prep.close()
    finally:
        lib.mfg_set_sweep_kernel(-1)
        lib.mfg_set_chunking(-1)
    info = s.info()
    assert info["sweep_mode"] == 1
    for k, fwd in enumerate((True, False)):
        want = records(pg.arrays["f2c"], pg.n_cell, info["sweep_chunks"], fwd)
        assert want[3] > 1000
        got = tuple(info[f"sweep_{w}_records"][k] for w in ("ring", "global", "cross"))
        assert got == want[:3], ("forward" if fwd else "backward", got, want)
    ref = Solver(pg, p)
    ref.set_sweep_mode(0)
    for x in (s, ref):
        x.calculate_gradient()
        x.iterate(3)
    for f in ("q", "dq", "dqdx"):
        assert_bitwise(s.download(f), ref.download(f), f)
    s.close()
    ref.close()
