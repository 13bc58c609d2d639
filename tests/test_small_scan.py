"""The one-launch step's cell scan on both sides of its rule (few cells: each block sums the counts
before its own run; more: block sums and a barrier), against the separate kernels over three steps, so
that counts which were not cleared would show: every field, the lists and the grid bit for bit. 990
particles take blocks of 128 threads, whose 12 rounds of 8 entries are 12,288 entries."""
import pytest

import test_small_batch
import test_small_step
from liquidsimulation_b200 import abi, scenes

pytestmark = pytest.mark.gpu
H = 0.04


@pytest.mark.parametrize("solver", [abi.LSP_SOLVER_SPH, abi.LSP_SOLVER_PCISPH])
@pytest.mark.parametrize("dims", [(6, 6, 8), (16, 32, 23), (16, 32, 24), (40, 30, 35)])
def test_scan(dims, solver):
    sc = scenes.small_box_scene(n_side=(9, 10, 11), solver=solver)
    sc.domain = ((0.0, 0.0, 0.0), tuple((d - 0.5) * H for d in dims))
    test_small_step.compare(sc, 3)
    other = scenes.small_box_scene(n_side=(7, 9, 8), solver=solver)
    test_small_batch.compare([sc, other, sc], 3)
