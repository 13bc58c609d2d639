"""The one-launch step of small batches (csrc/small_step.cu) against the separate kernels, which an
explicit launch shape keeps in use: every field, the neighbour lists, the grids and the statistics of
every scene bit for bit (0 ulp), for scenes of unequal sizes and rules, at the counts where the rule
changes the lanes per particle (592 blocks of 128 threads, at 16, 8, 4 or 2 lanes a particle), at the
largest grid of a scene's blocks, and through list growth, the pressure history and the autotuner."""
import numpy as np
import pytest

from fuzz_scenes import random_scene
from liquidsimulation_b200 import abi, scenes
from liquidsimulation_b200.solver import batch_from_scenes
from test_batch import FIELDS_PCI, FIELDS_SPH

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a).view(np.uint32)


def compare(scs, steps, setup=lambda b: None, small=True, lists=True):
    a, b = batch_from_scenes(scs), batch_from_scenes(scs)
    b.set_launch(True, 128, 0)
    for x in (a, b):
        setup(x)
    pci = scs[0].params.solver == abi.LSP_SOLVER_PCISPH
    for step in range(steps):
        before = a.launch_count()
        sa, sb = a.update(scs[0].dt), b.update(scs[0].dt)
        if step and small is not None:
            # One launch, and one more for each time the lists grow.
            assert (a.launch_count() - before <= 3) == small
        for k in range(len(scs)):
            for name in ("iterations", "converged", "max_density_error_ratio", "max_neighbors", "escaped",
                         "warm_start_used", "warm_start_tried"):
                assert getattr(sa[k], name) == getattr(sb[k], name), (step, k, name)
            for f in FIELDS_PCI if pci else FIELDS_SPH:
                assert np.array_equal(bits(a.read(k, f)), bits(b.read(k, f))), (step, k, f)
            if lists:
                for x, y in zip(a.neighbors(k), b.neighbors(k)):
                    assert np.array_equal(x, y), (step, k)
                for x, y in zip(a.grid(k), b.grid(k)):
                    assert np.array_equal(x, y), (step, k)
    a.close()
    b.close()


def boxes(counts, solver=abi.LSP_SOLVER_PCISPH):
    out = []
    for n in counts:
        side = int(np.ceil(n ** (1.0 / 3.0))) + 1
        sc = scenes.small_box_scene(n_side=(side, side, side), s=0.8 / side, solver=solver, pci_max_iterations=4)
        sc.positions, sc.velocities = sc.positions[:n].copy(), sc.velocities[:n].copy()
        out.append(sc)
    return out


@pytest.mark.parametrize("seed", range(8))
def test_fuzz_scenes_of_a_solver(seed):
    scs = []
    k = 0
    solver = abi.LSP_SOLVER_SPH if seed % 4 == 3 else abi.LSP_SOLVER_PCISPH
    while len(scs) < 5:
        sc = random_scene(100 * seed + k)[0]
        k += 1
        if sc.params.solver == solver and sc.params.warm_start == abi.LSP_WARM_ZERO and sc.params.pci_max_iterations >= 1:
            scs.append(sc)
    compare(scs, 3)


@pytest.mark.parametrize("counts,small", [
    ((1, 31, 700, 1), True), ((2368, 2368), True), ((2368, 2369), True), ((4736, 4737), True),
    ((9472, 9473), True), ((18944, 18944), True), ((18944, 18945), False),
    ((64,) * 592, True), ((8,) * 593, False)])
@pytest.mark.parametrize("solver", [abi.LSP_SOLVER_SPH, abi.LSP_SOLVER_PCISPH])
def test_counts_at_the_rules_edges(counts, small, solver):
    scs = boxes(counts[:4], solver)
    scs = scs if len(counts) <= 4 else [scs[0]] * len(counts)
    compare(scs, 2, small=small, lists=sum(counts) < 10000 and len(counts) <= 4)


@pytest.mark.parametrize("edge,small", [(1.86, True), (1.90, False)])
def test_largest_grid(edge, small):
    # h = 0.04; 100 particles at 16 lanes are 13 blocks, which may scan 13 * 8192 = 106,496 cells: a
    # cube of 1.86 has 47^3 = 103,823, one of 1.90 has 48^3.
    a, b = scenes.small_box_scene(n_side=(5, 5, 4)), scenes.small_box_scene(n_side=(6, 10, 5))
    a.domain = ((0.0, 0.0, 0.0), (edge, edge, edge))
    compare([a, b], 2, small=small)


def test_lists_that_grow_and_history():
    rng = np.random.Generator(np.random.PCG64(3))
    a, b = boxes((300, 900))
    b.positions = (0.5 + 0.02 * rng.standard_normal((900, 3))).astype(np.float32)
    a.velocities = rng.uniform(-0.5, 0.5, a.positions.shape).astype(np.float32)
    compare([a, b], 3, setup=lambda x: x.set_warm_start(abi.LSP_WARM_AUTO), small=None)


def test_autotune_and_direct_launches():
    scs = scenes.batched_dam_breaks(seed=4, scenes=5, nmin=300, nmax=3000)
    # Direct launches instead of the captured graph, on both sides.
    compare(scs, 3, setup=lambda x: x.set_launch(False, x.get_launch()["threads"], 0))
    a, b = batch_from_scenes(scs), batch_from_scenes(scs)
    a.autotune(scs[0].dt, repeats=2)
    b.update(scs[0].dt)
    a.update(scs[0].dt)
    b.update(scs[0].dt)
    for k in range(len(scs)):
        for f in FIELDS_PCI:
            assert np.array_equal(bits(a.read(k, f)), bits(b.read(k, f))), (k, f)
    a.close()
    b.close()


@pytest.mark.parametrize("counts", [(8192,) * 5, (8191,) * 5, (30000, 9000, 1025)])
def test_blocks_of_the_loop_over_large_scenes(counts):
    """Scenes of 8,192 particles on average take the loop's 1024-thread blocks at the default shape."""
    compare(boxes(counts), 2, small=False, lists=False)
