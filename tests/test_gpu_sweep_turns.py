"""The persistent sweeps' turns at the sizes where they can go wrong, against
the one-launch-per-level sweeps and the CPU oracle: the same bits in every
field (the quotients are correctly rounded and every sum keeps its order, so
no tolerance)."""
import numpy as np
import pytest

from helpers import assert_bitwise, oracle_from
from minifs_b200 import _lib, grid as gr, meshgen
from minifs_b200.solver import Solver

pytestmark = pytest.mark.gpu


def renumbered(mesh, seed):
    f2c = np.asarray(mesh.f2c).reshape(-1, 2)
    new = np.random.default_rng(seed).permutation(mesh.n_cell).astype(np.int32)
    out = np.where(f2c >= 0, new[np.maximum(f2c, 0)], f2c).astype(np.int32)
    return meshgen.RawMesh(x=mesh.x, y=mesh.y, z=mesh.z, nnpf=mesh.nnpf, f2n=mesh.f2n,
                           f2c=np.ascontiguousarray(out.reshape(-1)), n_cell=mesh.n_cell,
                           n_bface=mesh.n_bface, patches=mesh.patches)


# (mesh, flow, bump): what each reaches
CASES = {
    # one chunk, items of a few cells, levels of one item
    "six cells": (lambda: meshgen.cube_mesh(1, jitter=0.1, seed=2), {}, 0.05),
    # levels of a few cells, more levels than the segment starts kept on the SM
    "long": (lambda: meshgen.box_mesh(2, 2, 200, lz=100.0, jitter=0.1, seed=4), {}, 0.05),
    # every record count in every level, most increments older than the ring
    "renumbered": (lambda: renumbered(meshgen.cube_mesh(13, jitter=0.15, seed=7), 7), {}, 0.05),
    # dividends and velocities of exact zeros
    "aligned": (lambda: meshgen.cube_mesh(9, jitter=0.0, seed=1), {"alpha": 0.0}, 0.0),
    # increments that the limiter cuts
    "limited": (lambda: meshgen.cube_mesh(10, jitter=0.15, seed=8), {"cfl_start": 1000.0}, 0.4),
    # three records a cell and more: the eight-record tables
    "prisms": (lambda: meshgen.hexprism_mesh(7, 6, 5, jitter=0.15, seed=5), {}, 0.05),
    "merged": (lambda: meshgen.merged_hex_mesh(8, 7, 6, jitter=0.15, seed=5), {}, 0.05),
}


def prepared(name):
    mesh, flow, bump = CASES[name]
    p = gr.make_params(**{"mach": 0.5, "alpha": 2.0, "cfl_start": 10.0, **flow})
    return p, gr.prepare(mesh(), p, bump_amp=bump, bump_sigma=0.15)


def run(p, pg, iters, precision="fp64", kind=-1, chunking=-1, mode=1):
    lib = _lib.load()
    assert lib.mfg_set_sweep_kernel(kind) == 0 and lib.mfg_set_chunking(chunking) == 0
    try:
        s = Solver(pg, p, precision=precision)
    finally:
        lib.mfg_set_sweep_kernel(-1)
        lib.mfg_set_chunking(-1)
    info = s.info()
    s.set_sweep_mode(mode)
    s.calculate_gradient()
    out = {"norms": s.iterate(iters).reshape(-1)}
    s.step()  # the routines by themselves
    out |= {f: s.download(f) for f in ("q", "res", "dt", "diag", "dq", "dqdx", "dqdy", "dqdz")}
    s.close()
    return info, out


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("name", list(CASES))
def test_turns_same_bits_as_per_level(name, precision):
    p, pg = prepared(name)
    _, ref = run(p, pg, 3, precision, mode=0)
    for kind in (0, 1):          # one block an SM, two
        for chunking in (0, 4):  # vote, transverse
            info, out = run(p, pg, 3, precision, kind, chunking)
            assert info["sweep_mode"] == 1, (name, info)
            if name == "long":
                assert min(info["fw_levels"], info["bw_levels"]) > 512, info
            for f in ref:
                assert_bitwise(out[f], ref[f], f"{name} kind {kind} chunks {chunking}: {f}")


@pytest.mark.parametrize("name", ["six cells", "renumbered", "aligned", "limited"])
def test_turns_and_node_values_same_bits_as_oracle(name):
    """8, 2744, 1000 and 1331 nodes: whole blocks of node pairs, partial ones
    and an odd count."""
    p, pg = prepared(name)
    o = oracle_from(pg.arrays, p.as_dict() | {"cfl_nstep": p.cfl_nstep}, pg.q0,
                    (pg.n_node, pg.n_face, pg.n_cell, pg.n_bface))
    _, out = run(p, pg, 3)
    o.calculate_gradient()
    o.iterate(3)
    o.step()
    for f, want in (("q", o.q), ("res", o.res), ("dqdx", o.dqdx)):
        assert_bitwise(out[f], want, f"{name}: {f}")


def test_tables_grow_between_calls():
    """300 iterations in one call (the CFL and norm tables grow from their
    first size) against calls of 1, 7 and 292."""
    p, pg = prepared("six cells")
    a, b = Solver(pg, p), Solver(pg, p)
    for s in (a, b):
        s.calculate_gradient()
    na = a.iterate(300)
    nb = np.concatenate([b.iterate(k) for k in (1, 7, 292)])
    assert_bitwise(nb.reshape(-1), na.reshape(-1), "norms")
    assert_bitwise(b.download("q"), a.download("q"), "state")
    a.close()
    b.close()
