"""The SPH pressure force's exact forms and their fallback, one launch and separate kernels, against the
oracle (0 ulp): a scene whose positions are in range, and the same scene with a particle far outside it
(IEEE division and square root for the whole step), at sizes of both paths."""
import numpy as np
import pytest

from liquidsimulation_b200 import abi, scenes
from liquidsimulation_b200.solver import from_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side", [(5, 4, 6), (12, 13, 11), (36, 33, 35)])
@pytest.mark.parametrize("far", [False, True])
@pytest.mark.parametrize("separate", [False, True])
def test_sph_steps(oracle_mod, side, far, separate):
    rng = np.random.Generator(np.random.PCG64(side[0]))
    sc = scenes.small_box_scene(n_side=side, s=0.6 / max(side), solver=abi.LSP_SOLVER_SPH, obstacles=False,
                                negative_pressure_factor=0.3)
    sc.colliders = []
    sc.positions = (sc.positions + rng.uniform(-1e-3, 1e-3, sc.positions.shape)).astype(np.float32)
    sc.velocities = rng.uniform(-0.2, 0.2, sc.positions.shape).astype(np.float32)
    if far:
        sc.positions = np.concatenate([sc.positions, [[1.0e8, 0.5, 0.5]]]).astype(np.float32)
        sc.velocities = np.concatenate([sc.velocities, [[0.0, 0.0, 0.0]]]).astype(np.float32)
    g, o = from_scene(sc), oracle_mod.OracleSolver(sc)
    if separate:
        g._call("lsp_profile", 1)
    for step in range(2):
        g.update(5e-4)
        o.step(5e-4)
        for f in (abi.FIELD_POSITION, abi.FIELD_VELOCITY, abi.FIELD_DENSITY, abi.FIELD_PRESSURE):
            a, b = g.read(f), o.get(f)
            assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), (step, f)
    g.close()
    o.close()
