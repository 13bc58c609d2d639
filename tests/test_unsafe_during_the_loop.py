"""The one-launch step's force walk when a prediction leaves the range of the exact division in the middle
of a step, so that the word that chooses between the walk's two instances is set while other blocks
may be reading it: a lattice symmetric about x = 0, whose middle plane stays at x = 0 in the first
prediction and gets the rounding of the pressure sums, far below 2^-28, in the next. Every lane
count, against the separate kernels (all fields, 0 ulp) and the oracle."""
import numpy as np
import pytest

from liquidsimulation_b200 import abi, scenes
from liquidsimulation_b200.solver import from_scene
from test_small_step import bits, compare

pytestmark = pytest.mark.gpu


def symmetric(counts, s=0.02):
    sc = scenes.small_box_scene(n_side=counts, s=s, obstacles=False, surface_tension=0.0, pci_min_iterations=4)
    k, j, i = np.meshgrid(*[np.arange(c) for c in counts[::-1]], indexing="ij")
    x = np.stack([i.ravel() - counts[0] // 2, j.ravel() + 1, k.ravel() + 1], axis=1) * np.float32(0.9 * s)
    sc.positions = x.astype(np.float32)
    sc.velocities = np.zeros_like(sc.positions)
    sc.colliders = []
    sc.domain = ((-1.0, 0.0, 0.0), (1.0, 1.0, 1.0))
    sc.dt = 0.0005
    return sc


# 16, 8, 4 and 2 lanes per particle.
@pytest.mark.parametrize("counts", [(11, 9, 9), (17, 17, 17), (21, 21, 25), (31, 25, 29)])
def test_middle_plane(oracle_mod, counts):
    sc = symmetric(counts)
    s, o = from_scene(sc), oracle_mod.OracleSolver(sc)
    st = s.update(sc.dt)
    assert st.iterations >= 4 and o.step(sc.dt).iterations == st.iterations
    x = np.abs(s.read(abi.FIELD_PRED_POSITION).reshape(-1, 3)[:, 0])
    assert np.any((x > 0) & (x < 2.0 ** -28))
    for f in (abi.FIELD_POSITION, abi.FIELD_VELOCITY, abi.FIELD_PRED_POSITION, abi.FIELD_PRED_PRESSURE_FORCE):
        assert np.array_equal(bits(s.read(f)), bits(o.get(f))), f
    s.close()
    o.close()
    compare(sc, 2)
