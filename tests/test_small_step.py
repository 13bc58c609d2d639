"""The one-launch step of small scenes (csrc/small_step.cu) against the separate kernels, which the
per-class profile keeps in use: every field, the neighbour lists, the grid and the step's statistics
bit for bit (0 ulp), over the fuzz generator's parameter sets, at the particle counts where the rule
changes the lanes per particle (148 SMs of 512 threads: 16 lanes up to 4,736 particles, 8 to 9,472,
4 to 18,944, 2 to 37,888), at the rule's largest grid, and through list growth, first steps, moved
colliders and the pressure history."""
import numpy as np
import pytest

from fuzz_scenes import random_scene
from liquidsimulation_b200 import abi, scenes
from liquidsimulation_b200.solver import from_scene

pytestmark = pytest.mark.gpu

FIELDS = range(14)


def bits(a):
    return np.ascontiguousarray(a).view(np.uint32)


def launches(s):
    import ctypes
    n = ctypes.c_int64()
    s._call("lsp_launch_count", ctypes.byref(n))
    return n.value


def compare(sc, steps, setup=lambda s: None, between=lambda s, k: None, lists=True, expect_small=True):
    a, b = from_scene(sc), from_scene(sc)
    b._call("lsp_profile", 1)          # the profile needs the separate kernels
    for s in (a, b):
        setup(s)
    for k in range(steps):
        before = launches(a)
        sa, sb = a.update(sc.dt), b.update(sc.dt)
        if expect_small:
            assert launches(a) - before <= 3, "the one-launch step did not run"
        for name in ("iterations", "converged", "max_density_error_ratio", "max_neighbors", "escaped",
                     "warm_start_used", "warm_start_tried"):
            assert getattr(sa, name) == getattr(sb, name), (k, name)
        pci = sc.params.solver == abi.LSP_SOLVER_PCISPH
        for f in FIELDS:
            if not pci and f in (abi.FIELD_PRED_DENSITY, abi.FIELD_DENSITY_ERROR, abi.FIELD_PRED_POSITION,
                                 abi.FIELD_PRED_HALF_VELOCITY, abi.FIELD_PRED_PRESSURE_FORCE):
                continue
            assert np.array_equal(bits(a.read(f)), bits(b.read(f))), (k, f)
        if lists:
            for x, y in zip(a.neighbors(), b.neighbors()):
                assert np.array_equal(x, y), k
            for x, y in zip(a.grid(), b.grid()):
                assert np.array_equal(x, y), k
        between(a, k)
        between(b, k)
    a.close()
    b.close()


@pytest.mark.parametrize("seed", range(40))
def test_fuzz_scenes(seed):
    sc = random_scene(seed)[0]
    compare(sc, 3)


@pytest.mark.parametrize("n", [1, 31, 4736, 4737, 9472, 9473, 18944, 18945, 37888])
@pytest.mark.parametrize("solver", [abi.LSP_SOLVER_SPH, abi.LSP_SOLVER_PCISPH])
def test_counts_at_the_rules_edges(n, solver):
    side = int(np.ceil(n ** (1.0 / 3.0))) + 1
    sc = scenes.small_box_scene(n_side=(side, side, side), s=0.8 / side, solver=solver, pci_max_iterations=4)
    sc.positions, sc.velocities = sc.positions[:n].copy(), sc.velocities[:n].copy()
    compare(sc, 2, lists=n < 10000)


@pytest.mark.parametrize("edge,small", [(4.0, True), (4.2, False)])
def test_largest_grid(edge, small):
    # h = 0.04: a cube of 4.0 has 101^3 cells (below 2^20), one of 4.2 has 106^3.
    sc = scenes.small_box_scene(n_side=(9, 10, 11))
    sc.domain = ((0.0, 0.0, 0.0), (edge, edge, edge))
    compare(sc, 2, expect_small=small)


def test_lists_that_grow():
    rng = np.random.Generator(np.random.PCG64(3))
    sc = scenes.small_box_scene(n_side=(6, 6, 6), pci_max_iterations=3)
    sc.positions = (0.5 + 0.02 * rng.standard_normal((900, 3))).astype(np.float32)
    sc.velocities = np.zeros_like(sc.positions)
    compare(sc, 2)


@pytest.mark.parametrize("keep", [0, 1])
def test_initial_velocities_and_history(keep):
    rng = np.random.Generator(np.random.PCG64(4))
    sc = scenes.small_box_scene(n_side=(10, 9, 8), keep_initial_velocity=keep, pci_max_iterations=12)
    sc.velocities = rng.uniform(-0.5, 0.5, sc.positions.shape).astype(np.float32)

    def move(s, k):
        s.update_static_collision_sphere(2, (0.3, 0.1 + 0.01 * k, 0.6), 0.1)
        if k == 1:
            s.add_particles(np.array([[0.7, 0.7, 0.7]], np.float32))

    # LSP_WARM_AUTO keeps the pressure history while its steps start from zero pressure.
    compare(sc, 4, setup=lambda s: s.set_warm_start(abi.LSP_WARM_AUTO), between=move)


def test_no_grid_box_and_escaped_particles():
    sc = scenes.small_box_scene(n_side=(8, 8, 8), obstacles=False)
    sc.colliders = []
    sc.domain = None
    compare(sc, 3)
    sc.domain = ((0.1, 0.1, 0.1), (0.15, 0.15, 0.15))
    compare(sc, 2)
