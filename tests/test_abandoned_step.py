"""A one-launch step (csrc/small_step.cu) whose wait at one of its barriers runs out: the call reports
LSP_ERR_TIMEOUT, the state is bit for bit that before the call, the unfinished lists and grid are
refused, and the following steps equal those of a solver that never gave up (0 ulp). At every
barrier of the grid build, the lists and the loop, in few and in many cells, as the first step and
later ones, for single scenes and for one scene of a batch (graph and direct launches)."""
import numpy as np
import pytest

from liquidsimulation_b200 import abi, scenes
from liquidsimulation_b200.solver import batch_from_scenes, from_scene

pytestmark = pytest.mark.gpu

FIELDS = [abi.FIELD_POSITION, abi.FIELD_VELOCITY, abi.FIELD_HALF_VELOCITY, abi.FIELD_OLD_HALF_VELOCITY,
          abi.FIELD_FIRST_STEP]


def bits(a):
    return np.ascontiguousarray(a, np.float32).view(np.uint32)


def scene(solver, seed=1, edge=None, side=(9, 10, 11)):
    kw = dict(pci_min_iterations=3) if solver == abi.LSP_SOLVER_PCISPH else {}
    sc = scenes.small_box_scene(n_side=side, solver=solver, seed=seed, **kw)
    if edge:
        sc.domain = ((0.0, 0.0, 0.0), (edge, edge, edge))
    return sc


def refused(code, call, *args):
    with pytest.raises(abi.LspError) as e:
        call(*args)
    assert e.value.code == code


# The grid's phases, the lists and the pressure phase have six barriers (seven in many cells); a PCISPH
# step of three iterations has 11 or 12.
# h = 0.04: a cube of 0.8 has 9,261 cells (few for blocks of 128 threads: 12,288), the unit cube 17,576.
CASES = [(abi.LSP_SOLVER_SPH, 0.8, 6), (abi.LSP_SOLVER_SPH, None, 7), (abi.LSP_SOLVER_PCISPH, 0.8, 11),
         (abi.LSP_SOLVER_PCISPH, None, 12)]


@pytest.mark.parametrize("solver,edge,barriers", CASES)
@pytest.mark.parametrize("before", [0, 1, 2])
def test_single_scene(solver, edge, barriers, before):
    import ctypes
    sc = scene(solver, edge=edge)
    for barrier in range(1, barriers + 1):
        s, twin = from_scene(sc), from_scene(sc)
        for _ in range(before):
            s.update(sc.dt)
            twin.update(sc.dt)
        want = [bits(s.read(f)) for f in FIELDS]
        refused(abi.LSP_ERR_TIMEOUT, s._call, "lsp_stalled_step", ctypes.c_float(sc.dt), barrier)
        for f, w in zip(FIELDS, want):
            assert np.array_equal(bits(s.read(f)), w), (barrier, f)
        refused(abi.LSP_ERR_STATE, s.neighbors)
        refused(abi.LSP_ERR_STATE, s.grid)
        for _ in range(2):
            sa, sb = s.update(sc.dt), twin.update(sc.dt)
            assert sa.iterations == sb.iterations and sa.max_neighbors == sb.max_neighbors
        for f in FIELDS:
            assert np.array_equal(bits(s.read(f)), bits(twin.read(f))), (barrier, f)
        for a, b in zip(s.neighbors() + s.grid(), twin.neighbors() + twin.grid()):
            assert np.array_equal(a, b), barrier
        s.close()
        twin.close()


@pytest.mark.parametrize("solver,edge,barriers", [CASES[0], CASES[2]])
@pytest.mark.parametrize("graph", [True, False])
@pytest.mark.parametrize("before", [0, 3])
def test_scene_of_a_batch(solver, edge, barriers, graph, before):
    import ctypes
    scs = [scene(solver, seed, edge, side=(7 + seed, 8, 9)) for seed in range(3)]
    dt = scs[0].dt
    for barrier in range(1, barriers + 1):
        b, twin = batch_from_scenes(scs), batch_from_scenes(scs)
        b.set_launch(graph, 256, 0)
        for _ in range(before):
            b.update(dt)
            twin.update(dt)
        want = [[bits(b.read(k, f)) for f in FIELDS] for k in range(3)] if before else None
        refused(abi.LSP_ERR_TIMEOUT, b._call, "lsp_batch_stalled_step", ctypes.c_float(dt), 1, barrier)
        for k in range(3):
            for f, w in zip(FIELDS, want[k] if want else []):
                assert np.array_equal(bits(b.read(k, f)), w), (barrier, k, f)
            refused(abi.LSP_ERR_STATE, b.neighbors, k)
            refused(abi.LSP_ERR_STATE, b.grid, k)
        for _ in range(2):
            sa, sb = b.update(dt), twin.update(dt)
            assert [x.iterations for x in sa] == [x.iterations for x in sb]
        for k in range(3):
            for f in FIELDS:
                assert np.array_equal(bits(b.read(k, f)), bits(twin.read(k, f))), (barrier, k, f)
            for x, y in zip(b.neighbors(k) + b.grid(k), twin.neighbors(k) + twin.grid(k)):
                assert np.array_equal(x, y), (barrier, k)
        b.close()
        twin.close()


RESULTS = [abi.FIELD_DENSITY, abi.FIELD_PRESSURE, abi.FIELD_PRED_DENSITY, abi.FIELD_DENSITY_ERROR,
           abi.FIELD_PRED_POSITION, abi.FIELD_PRED_HALF_VELOCITY, abi.FIELD_PRED_PRESSURE_FORCE,
           abi.FIELD_NEIGHBOR_COUNT]


@pytest.mark.parametrize("barrier", [2, 6, 9])
def test_results_of_a_step_that_gave_up(barrier):
    """They are neither the last step's (other slots, partly overwritten) nor a step's at all."""
    import ctypes
    sc = scene(abi.LSP_SOLVER_PCISPH)
    s, twin = from_scene(sc), from_scene(sc)
    b = batch_from_scenes([sc, sc])
    for x in (s, twin, b):
        x.update(sc.dt)
    refused(abi.LSP_ERR_TIMEOUT, s._call, "lsp_stalled_step", ctypes.c_float(sc.dt), barrier)
    refused(abi.LSP_ERR_TIMEOUT, b._call, "lsp_batch_stalled_step", ctypes.c_float(sc.dt), 1, barrier)
    for f in RESULTS:
        refused(abi.LSP_ERR_STATE, s.read, f)
        for k in range(2):
            refused(abi.LSP_ERR_STATE, b.read, k, f)
    assert np.array_equal(bits(s.read(abi.FIELD_SPEED_SQUARED)), bits(twin.read(abi.FIELD_SPEED_SQUARED)))
    for x in (s, twin, b):
        x.update(sc.dt)
    for f in RESULTS:
        for got in (s.read(f), b.read(0, f), b.read(1, f)):
            assert np.array_equal(bits(got), bits(twin.read(f))), f
    for x in (s, twin, b):
        x.close()


def test_what_is_refused():
    import ctypes
    sc = scene(abi.LSP_SOLVER_PCISPH)
    s, twin = from_scene(sc), from_scene(sc)
    refused(abi.LSP_ERR_INVALID, s._call, "lsp_stalled_step", ctypes.c_float(sc.dt), 0)
    s._call("lsp_profile", 1)
    refused(abi.LSP_ERR_STATE, s._call, "lsp_stalled_step", ctypes.c_float(sc.dt), 1)
    s._call("lsp_profile", 0)
    s._call("lsp_stalled_step", ctypes.c_float(sc.dt), 1000)      # fewer barriers: an ordinary step
    twin.update(sc.dt)
    for f in FIELDS:
        assert np.array_equal(bits(s.read(f)), bits(twin.read(f)))
    b = batch_from_scenes([sc, sc])
    b.set_launch(True, 128, 0)
    refused(abi.LSP_ERR_STATE, b._call, "lsp_batch_stalled_step", ctypes.c_float(sc.dt), 0, 1)
    refused(abi.LSP_ERR_INVALID, b._call, "lsp_batch_stalled_step", ctypes.c_float(sc.dt), 2, 1)
    for x in (s, twin, b):
        x.close()
