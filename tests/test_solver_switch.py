"""A solver that steps as PCISPH and then as SPH (lsp_set_params): the fields of the prediction keep the
last PCISPH step's values through the SPH steps, whichever of the two buffers of predicted positions
its last iteration left them in, on both routes of the step; switched back, it steps as a fresh
solver given its state does."""
import ctypes

import numpy as np
import pytest

from liquidsimulation_b200 import abi, scenes
from liquidsimulation_b200.solver import from_scene
from test_small_step import bits

pytestmark = pytest.mark.gpu

FIELDS = [abi.FIELD_PRED_POSITION, abi.FIELD_PRED_HALF_VELOCITY, abi.FIELD_PRED_PRESSURE_FORCE, abi.FIELD_PRED_DENSITY,
          abi.FIELD_DENSITY_ERROR]


def as_solver(s, solver):
    p = s.params
    p.solver = solver
    s._call("lsp_set_params", ctypes.byref(p))


@pytest.mark.parametrize("separate", [0, 1])
@pytest.mark.parametrize("iterations", [1, 2, 3, 4])
def test_predictions_survive_sph_steps(iterations, separate):
    # No gravity, no particle near a cell's face (multiples of 0.04) and a time step too short to reach one:
    # the particles keep their order on the device, which the fields of an earlier step are read in.
    sc = scenes.small_box_scene(n_side=(8, 9, 10), pci_min_iterations=iterations, pci_max_iterations=iterations,
                                gravity=(0.0, 0.0, 0.0), obstacles=False)
    sc.positions = sc.positions + np.float32(0.007)
    s = from_scene(sc)
    s._call("lsp_profile", separate)
    dt = 1e-6
    for _ in range(2):
        assert s.update(dt).iterations == iterations
    want = [bits(s.read(f)).copy() for f in FIELDS]
    as_solver(s, abi.LSP_SOLVER_SPH)
    for _ in range(2):
        s.update(dt)
        for f, w in zip(FIELDS, want):
            assert np.array_equal(bits(s.read(f)), w), f
    as_solver(s, abi.LSP_SOLVER_PCISPH)
    twin = from_scene(sc)
    twin.update(dt)
    twin.write_state(*s.read_state())
    assert s.update(dt).iterations == twin.update(dt).iterations
    for f in FIELDS + [abi.FIELD_POSITION, abi.FIELD_VELOCITY]:
        assert np.array_equal(bits(s.read(f)), bits(twin.read(f))), f
    s.close()
    twin.close()
