"""Which steps run as one launch (small_step_lanes): on both sides of the rule's edges, by the number of
kernels a step launches."""
import numpy as np
import pytest

from liquidsimulation_b200 import abi, scenes
from liquidsimulation_b200.solver import from_scene
from test_small_step import launches

pytestmark = pytest.mark.gpu


def block(n, solver):
    side = int(np.ceil(n ** (1.0 / 3.0))) + 1
    sc = scenes.small_box_scene(n_side=(side, side, side), s=0.8 / side, solver=solver, pci_max_iterations=4)
    sc.positions, sc.velocities = sc.positions[:n].copy(), sc.velocities[:n].copy()
    return sc


def step_launches(sc, setup=lambda s: None):
    s = from_scene(sc)
    setup(s)
    counts = []
    for _ in range(3):
        before = launches(s)
        s.update(sc.dt)
        counts.append(launches(s) - before)
    s.close()
    return min(counts)      # a step that grows its lists launches twice


@pytest.mark.parametrize("solver", [abi.LSP_SOLVER_SPH, abi.LSP_SOLVER_PCISPH])
@pytest.mark.parametrize("n,one", [(1, True), (37888, True), (37889, False)])
def test_particles(n, one, solver):
    assert (step_launches(block(n, solver)) == 1) == one


@pytest.mark.parametrize("edge,one", [(4.0, True), (4.2, False)])
def test_cells(edge, one):
    # h = 0.04: a cube of 4.0 has 101^3 cells (below 2^20), one of 4.2 has 106^3.
    sc = scenes.small_box_scene(n_side=(9, 10, 11))
    sc.domain = ((0.0, 0.0, 0.0), (edge, edge, edge))
    assert (step_launches(sc) == 1) == one


@pytest.mark.parametrize("setup", ["profile", "record", "guess", "host loop"])
def test_what_needs_the_separate_kernels(setup):
    sc = scenes.small_box_scene(n_side=(9, 10, 11), loop_mode=abi.LSP_LOOP_HOST if setup == "host loop" else 0)
    calls = {"profile": lambda s: s._call("lsp_profile", 1), "record": lambda s: s.mlp_record(True),
             "guess": lambda s: s.set_warm_start(abi.LSP_WARM_MLP), "host loop": lambda s: None}
    assert step_launches(sc, calls[setup]) > 3
