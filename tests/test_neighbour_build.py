"""The neighbour build where its masks, groups and shared-memory column have their edges, against
the oracle: lists of 1 entry and of lengths around the multiples of 4, rows of more than 32
particles (several masks a row), lists that need more masks than a thread's column holds, and
particle counts that fill the arrays exactly (the scan reads past the end of a row). Lists,
densities and the state after each step: 0 ulp."""
import numpy as np
import pytest

from liquidsimulation_b200 import abi, scenes
from liquidsimulation_b200.solver import batch_from_scenes, from_scene

pytestmark = pytest.mark.gpu


def cluster_scene(n, spread, seed, solver=abi.LSP_SOLVER_SPH):
    """n particles in a cube of edge spread * h in the middle of the unit box (h = 0.04)."""
    rng = np.random.Generator(np.random.PCG64([n, seed]))
    p = scenes._params(0.02, solver, stiffness=1e-3)
    pos = (0.5 + (rng.random((n, 3)) - 0.5) * spread * 0.04).astype(np.float32)
    box = scenes.Collider("box", (0.5, 0.5, 0.5), (0.5, 0.5, 0.5), True)
    return scenes.Scene("cluster", p, pos, np.zeros_like(pos), [box], 1e-4, 2, domain=((0, 0, 0), (1, 1, 1)), spacing=0.02)


# (count, spread): single particles; sparse; dense rows; more masks than a column (12 of 32
# candidates); 256 and 512 fill the arrays.
CASES = [(1, 1.0), (2, 0.1), (5, 0.5), (33, 0.5), (97, 0.9), (256, 1.5), (512, 2.5), (700, 0.6), (1500, 2.0)]


def same(a, b):
    return np.array_equal(np.ascontiguousarray(a).view(np.uint32), np.ascontiguousarray(b).view(np.uint32))


@pytest.mark.parametrize("n,spread", CASES)
def test_lists_and_density(oracle_mod, n, spread):
    sc = cluster_scene(n, spread, 1)
    g, o = from_scene(sc), oracle_mod.OracleSolver(sc)
    for step in range(2):
        st = g.update(sc.dt)
        o.step(sc.dt)
        og, ig = g.neighbors()
        oo, io = o.neighbors()
        assert np.array_equal(og, oo) and np.array_equal(ig, io), step
        assert st.max_neighbors == int(np.diff(oo).max())
        for f in (abi.FIELD_DENSITY, abi.FIELD_PRESSURE, abi.FIELD_POSITION, abi.FIELD_VELOCITY):
            assert same(g.read(f), o.get(f)), (step, f)
    g.close()
    o.close()


@pytest.mark.parametrize("threads", [128, 256, 512, 1024])
def test_batch_matches_the_single_scenes(oracle_mod, threads):
    scs = [cluster_scene(n, spread, 2) for n, spread in CASES]
    b = batch_from_scenes(scs)
    b.set_launch(True, threads, 0)
    b.update(scs[0].dt)
    for k, sc in enumerate(scs):
        o = oracle_mod.OracleSolver(sc)
        o.step(sc.dt)
        og, ig = b.neighbors(k)
        oo, io = o.neighbors()
        assert np.array_equal(og, oo) and np.array_equal(ig, io), k
        for f in (abi.FIELD_DENSITY, abi.FIELD_POSITION, abi.FIELD_VELOCITY):
            assert same(b.read(k, f), o.get(f)), (k, f)
        o.close()
    b.close()
