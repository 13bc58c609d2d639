"""The non-pressure pass's exact division over its velocity range: components of 0 and of magnitudes
around the positions' lower bound (2^-28), the velocities' (2^-57) and below it, where the pass keeps
IEEE division, in the one-launch step and in the separate kernels, against the oracle (0 ulp)."""
import numpy as np
import pytest

from liquidsimulation_b200 import abi, scenes
from liquidsimulation_b200.solver import from_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("separate", [False, True])
@pytest.mark.parametrize("exponents", [(-27, -29), (-40, -57), (-56, -57), (-57, -58), (-1, -57), (-1, -120), (-60, -149)])
def test_small_velocities(oracle_mod, exponents, separate):
    rng = np.random.Generator(np.random.PCG64(abs(exponents[0]) * 1000 + abs(exponents[1])))
    sc = scenes.small_box_scene(n_side=(8, 9, 7), keep_initial_velocity=1, pci_max_iterations=4, viscosity=3.5,
                                gravity=(0.0, 0.0, 0.0))
    e = rng.choice(exponents, sc.positions.shape)
    v = np.ldexp(rng.uniform(1.0, 2.0, e.shape), e) * rng.choice([-1.0, 0.0, 1.0], e.shape)
    sc.velocities = v.astype(np.float32)
    g, o = from_scene(sc), oracle_mod.OracleSolver(sc)
    if separate:
        g._call("lsp_profile", 1)
    for step in range(2):
        g.update(sc.dt)
        o.step(sc.dt)
        for f in (abi.FIELD_POSITION, abi.FIELD_VELOCITY, abi.FIELD_HALF_VELOCITY, abi.FIELD_PRESSURE):
            a, b = g.read(f), o.get(f)
            assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), (step, f)
    g.close()
    o.close()
