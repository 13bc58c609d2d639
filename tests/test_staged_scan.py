"""The neighbour scan's staged rows (csrc/particle_ops.cuh) against the oracle: a warp's particles in one
row of cells, with 1 to 48 particles a cell, so that a row's candidates (three to a warp's worth of
cells) lie on both sides of 32 per lane and of the 96 that are staged, from odd and even places, next
to warps that cross rows and a last warp that is not full. Lists, density and the state after each of
two steps: 0 ulp."""
import numpy as np
import pytest

from liquidsimulation_b200 import abi, scenes
from liquidsimulation_b200.solver import batch_from_scenes, from_scene

pytestmark = pytest.mark.gpu
H = 0.04


def row_scene(per_cell, odd, solver, cells=12):
    rng = np.random.Generator(np.random.PCG64([per_cell, odd]))
    p = scenes._params(H / 2, solver, stiffness=1e-3)
    out = []
    for (cx, cy), n in (((10, 10), per_cell), ((10, 11), per_cell), ((11, 10), 1)):
        for cz in range(5, 5 + cells):
            k = n + (odd if cz == 5 else 0)
            out.append((np.array([cx, cy, cz]) + 0.02 + 0.96 * rng.random((k, 3))) * H)
    pos = np.concatenate(out).astype(np.float32)
    box = scenes.Collider("box", (0.5, 0.5, 0.5), (0.5, 0.5, 0.5), True)
    return scenes.Scene("row", p, pos, np.zeros_like(pos), [box], 1e-4, 2, domain=((0, 0, 0), (1, 1, 1)), spacing=H / 2)


def same(a, b):
    return np.array_equal(np.ascontiguousarray(a).view(np.uint32), np.ascontiguousarray(b).view(np.uint32))


@pytest.mark.parametrize("odd", [0, 1])
@pytest.mark.parametrize("per_cell", [1, 4, 10, 11, 16, 17, 31, 32, 33, 48])
def test_rows(oracle_mod, per_cell, odd):
    for solver in (abi.LSP_SOLVER_SPH, abi.LSP_SOLVER_PCISPH):
        sc = row_scene(per_cell, odd, solver)
        g, o = from_scene(sc), oracle_mod.OracleSolver(sc)
        g._call("lsp_profile", 1)   # the separate kernels
        b = batch_from_scenes([sc, sc])
        b.set_launch(True, 128, 0)
        for step in range(2):
            g.update(sc.dt)
            b.update(sc.dt)
            o.step(sc.dt)
            oo, io = o.neighbors()
            for off, idx in (g.neighbors(), b.neighbors(1)):
                assert np.array_equal(off, oo) and np.array_equal(idx, io), step
            for f in (abi.FIELD_DENSITY, abi.FIELD_PRESSURE, abi.FIELD_POSITION, abi.FIELD_VELOCITY):
                assert same(g.read(f), o.get(f)) and same(b.read(1, f), o.get(f)), (step, f)
        g.close()
        b.close()
        o.close()
