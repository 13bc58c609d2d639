"""What the batch's autotuner reports is what it keeps: a batch given the reported shape launches the same
kernels a step as the tuned one, and the chosen entry's time is the least of those listed. A small
batch (one launch a step at the default shape), SPH, and a batch whose loop takes blocks of its own
size at the default shape."""
import numpy as np
import pytest

from liquidsimulation_b200 import abi, scenes
from liquidsimulation_b200.solver import batch_from_scenes
from test_small_batch import boxes

pytestmark = pytest.mark.gpu


def launches(b, dt):
    before = b.launch_count()
    b.update(dt)
    return b.launch_count() - before


@pytest.mark.parametrize("solver", [abi.LSP_SOLVER_SPH, abi.LSP_SOLVER_PCISPH])
@pytest.mark.parametrize("counts", [(300, 1000, 700), (9000,) * 6])
def test_reported_shape_is_what_runs(solver, counts):
    scs = boxes(counts, solver)
    dt = scs[0].dt
    a, b = batch_from_scenes(scs), batch_from_scenes(scs)
    a.update(dt)
    b.update(dt)
    t, _ = a.autotune(dt, repeats=3)
    shapes = [(t.cand_threads[k], t.cand_loop_blocks[k]) for k in range(t.candidates)]
    assert len(set(shapes)) == len(shapes) and shapes.count((256, 0)) == 1
    chosen = (t.threads, t.loop_blocks)
    assert t.cand_ms[shapes.index(chosen)] == min(t.cand_ms[k] for k in range(t.candidates))
    kept = a.get_launch()
    assert (kept["threads"], kept["loop_blocks"]) == chosen
    if max(counts) <= 1000:
        assert chosen == (256, 0)       # one launch against ten
    b.set_launch(True, *chosen)
    b.update(dt)                        # the tuner's step (a step that grows its lists launches twice)
    for _ in range(3):
        na, nb = launches(a, dt), launches(b, dt)
        assert na == nb
    assert (na <= 2) == (max(counts) <= 1000 and chosen == (256, 0))
    a.close()
    b.close()
