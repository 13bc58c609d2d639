"""Solvers and batches stepped at once from several host threads: whichever route each step takes beside
the others (one launch or the separate kernels), every scene ends with the bits it has when it is
stepped alone, and several solvers of small scenes share the chip instead of queueing for it."""
import threading
import time

import numpy as np
import pytest

from liquidsimulation_b200 import abi, scenes
from liquidsimulation_b200.solver import batch_from_scenes, from_scene
from test_small_step import launches

pytestmark = pytest.mark.gpu

FIELDS = [abi.FIELD_POSITION, abi.FIELD_VELOCITY, abi.FIELD_HALF_VELOCITY, abi.FIELD_DENSITY, abi.FIELD_PRESSURE]


def bits(a):
    return np.ascontiguousarray(a, np.float32).view(np.uint32)


def together(calls):
    """Runs the calls at once, each in its thread; returns the seconds they took."""
    start = threading.Barrier(len(calls) + 1)
    failed = []

    def go(call):
        start.wait()
        try:
            call()
        except Exception as e:                 # noqa: BLE001 - reported below
            failed.append(e)

    threads = [threading.Thread(target=go, args=(c,)) for c in calls]
    for t in threads:
        t.start()
    start.wait()
    t0 = time.perf_counter()
    for t in threads:
        t.join()
    assert not failed, failed
    return time.perf_counter() - t0


def block(side, solver, seed=1):
    # stiffness 0.5: the plain SPH scenes stay finite over the steps taken here.
    return scenes.small_box_scene(n_side=(side,) * 3, s=0.8 / (side + 1), solver=solver, seed=seed, obstacles=False,
                                  stiffness=0.5)


def test_results_do_not_depend_on_the_others():
    kinds = [(8, abi.LSP_SOLVER_SPH), (17, abi.LSP_SOLVER_PCISPH), (23, abi.LSP_SOLVER_PCISPH), (31, abi.LSP_SOLVER_SPH),
             (23, abi.LSP_SOLVER_SPH), (45, abi.LSP_SOLVER_PCISPH)]
    scs = [block(side, solver, k) for k, (side, solver) in enumerate(kinds)]
    batch = [block(9, abi.LSP_SOLVER_PCISPH, 20 + k) for k in range(6)]
    steps = 12

    def make():
        return [from_scene(sc) for sc in scs], [batch_from_scenes(batch) for _ in range(2)]

    def step(x, dt):
        for _ in range(steps):
            x.update(dt)

    alone, at_once = make(), make()
    for s, sc in zip(alone[0], scs):
        before = launches(s)
        step(s, sc.dt)
        if sc.n <= 37888:
            assert launches(s) - before <= steps + 3        # one launch a step, and the lists' growth
    for b in alone[1]:
        step(b, batch[0].dt)
    together([lambda s=s, sc=sc: step(s, sc.dt) for s, sc in zip(at_once[0], scs)] +
             [lambda b=b: step(b, batch[0].dt) for b in at_once[1]])
    for a, b in zip(alone[0], at_once[0]):
        for f in FIELDS:
            assert np.array_equal(bits(a.read(f)), bits(b.read(f))), f
        for x, y in zip(a.neighbors(), b.neighbors()):
            assert np.array_equal(x, y)
    for a, b in zip(alone[1], at_once[1]):
        for k in range(len(batch)):
            for f in FIELDS:
                assert np.array_equal(bits(a.read(k, f)), bits(b.read(k, f))), (k, f)
    for group in alone + at_once:
        for x in group:
            x.close()


@pytest.mark.parametrize("solver", [abi.LSP_SOLVER_SPH, abi.LSP_SOLVER_PCISPH])
@pytest.mark.parametrize("side", [17, 23, 31])
def test_eight_solvers_share_the_chip(solver, side):
    """Eight solvers stepped at once take no longer (a quarter for the clock) than eight whose steps are
    separate kernels anyway, by a grid box of more than 2^20 cells, which costs those a longer scan
    besides. Queueing for the chip they took two to four times as long."""
    sc = block(side, solver)
    wide = block(side, solver)
    edge = 104 * 2 * 0.8 / (side + 1)               # h is two spacings
    wide.domain = ((0.0, 0.0, 0.0), (edge,) * 3)
    took = []
    for scene in (sc, wide):
        solvers = [from_scene(scene) for _ in range(8)]
        for s in solvers:
            s.step_many(sc.dt, 2)
        before = launches(solvers[0])
        solvers[0].update(sc.dt)
        assert (launches(solvers[0]) - before <= 2) == (scene is sc)     # alone: one launch
        took.append(min(together([lambda s=s: s.step_many(sc.dt, 40) for s in solvers]) for _ in range(3)))
        for s in solvers:
            s.close()
    assert took[0] <= 1.25 * took[1]
