"""State and field transfers between the solver and host memory, small (kernels on pinned memory or the
pinned stage) and large (copies): pinned, pageable, misaligned and mixed buffers, single scenes and
batches, at counts around the 256-row blocks and the limits of the stage (1 MB) and of the direct
transfers (8 MB). Exact equality."""
import ctypes

import numpy as np
import pytest
import torch

from liquidsimulation_b200 import abi, scenes
from liquidsimulation_b200.solver import batch_from_scenes, from_scene

pytestmark = pytest.mark.gpu

FP, IP = ctypes.POINTER(ctypes.c_float), ctypes.POINTER(ctypes.c_int32)


def buffer(count, dtype, kind, shift):
    """count values in pinned or pageable memory, `shift` elements after a 16-byte boundary."""
    t = torch.empty(count + shift + 8, dtype=torch.float32, pin_memory=kind == "pinned")
    a = t.numpy()
    lead = (-a.ctypes.data // 4) % 4 + shift
    return t, a[lead:lead + count].view(dtype)


def scene(n):
    side = int(np.ceil(n ** (1.0 / 3.0)))
    sc = scenes.small_box_scene(n_side=(side, side, side), s=0.9 / (side + 1), obstacles=False, pci_max_iterations=2)
    sc.positions, sc.velocities = sc.positions[:n].copy(), sc.velocities[:n].copy()
    return sc


def ptrs(arrs):
    return [a.ctypes.data_as(IP if a.dtype == np.int32 else FP) for a in arrs]


# 20,164 rows of 52 bytes fill the stage; 161,319 the direct transfers' limit.
COUNTS = [1, 255, 256, 257, 1000, 20164, 20165, 161319, 161320]
KINDS = [("pinned", 0), ("pinned", 1), ("pageable", 0), ("pageable", 3), ("mixed", 0)]


@pytest.mark.parametrize("n", COUNTS)
@pytest.mark.parametrize("kind,shift", KINDS)
def test_round_trip(n, kind, shift):
    rng = np.random.Generator(np.random.PCG64(n))
    sc = scene(n)
    s = from_scene(sc)
    s.update(sc.dt)                      # the particles are in cell order now
    lib, h = abi.load_library(), s._h
    keep, src, dst = [], [], []
    for c in range(5):
        k = ("pinned" if c % 2 else "pageable") if kind == "mixed" else kind
        for group in (src, dst):
            t, a = buffer(n * (1 if c == 4 else 3), np.int32 if c == 4 else np.float32, k, shift)
            keep.append(t)
            group.append(a)
        if c == 4:
            src[c][...] = rng.integers(0, 2, n)
        else:
            src[c][...] = rng.normal(0.5, 0.1, 3 * n)
        dst[c].view(np.uint32)[...] = 0xdeadbeef
    abi.check(lib, lib.lsp_write_state(h, *ptrs(src), n))
    abi.check(lib, lib.lsp_read_state(h, *ptrs(dst), n))
    for a, b in zip(src, dst):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    for d in dst:
        d.view(np.uint32)[...] = 0
    abi.check(lib, lib.lsp_read_particles(h, *ptrs(dst[:2]), n))
    assert np.array_equal(dst[0], src[0]) and np.array_equal(dst[1], src[1])
    abi.check(lib, lib.lsp_read_particles(h, None, dst[2].ctypes.data_as(FP), n))
    assert np.array_equal(dst[2], src[1])
    for f, want in ((abi.FIELD_POSITION, src[0]), (abi.FIELD_HALF_VELOCITY, src[2]), (abi.FIELD_OLD_HALF_VELOCITY, src[3]),
                    (abi.FIELD_FIRST_STEP, src[4].astype(np.float32))):
        out = dst[3][:want.size]
        abi.check(lib, lib.lsp_read_field(h, f, out.ctypes.data_as(FP), n))
        assert np.array_equal(out, want)
    s.close()


@pytest.mark.parametrize("kind,shift", KINDS)
def test_batch_round_trip(kind, shift):
    rng = np.random.Generator(np.random.PCG64(1))
    scs = [scene(n) for n in (5, 300, 1025)]
    b = batch_from_scenes(scs)
    b.update(scs[0].dt)
    lib, n = abi.load_library(), b.total
    keep, src, dst = [], [], []
    for c in range(5):
        k = ("pinned" if c % 2 else "pageable") if kind == "mixed" else kind
        for group in (src, dst):
            t, a = buffer(n * (1 if c == 4 else 3), np.int32 if c == 4 else np.float32, k, shift)
            keep.append(t)
            group.append(a)
        src[c][...] = rng.integers(0, 2, n) if c == 4 else rng.normal(0.5, 0.1, 3 * n)
    abi.check(lib, lib.lsp_batch_write_state(b._h, *ptrs(src), n))
    abi.check(lib, lib.lsp_batch_read_state(b._h, *ptrs(dst), n))
    for x, y in zip(src, dst):
        assert np.array_equal(x.view(np.uint32), y.view(np.uint32))
    base = 0
    for k, sc in enumerate(scs):
        assert np.array_equal(b.positions(k).ravel(), src[0][3 * base:3 * (base + sc.n)])
        base += sc.n
    b.close()


def test_counts_are_still_checked():
    sc = scene(100)
    s = from_scene(sc)
    s.update(sc.dt)
    x = np.empty(300, np.float32)
    lib = abi.load_library()
    assert lib.lsp_read_particles(s._h, x.ctypes.data_as(FP), x.ctypes.data_as(FP), 99) == abi.LSP_ERR_INVALID
    assert lib.lsp_read_field(s._h, abi.FIELD_POSITION, x.ctypes.data_as(FP), 101) == abi.LSP_ERR_INVALID
    s.close()
