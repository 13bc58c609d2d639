"""A read-back into device memory gathers a row per thread: the three components of a field take
hardly longer than one (25 us and 21 us at 990,000 particles; through shared memory, which is for host
memory across the link, 35). Both reads share the launch, the copy and the wait."""
import ctypes
import time

import pytest
import torch

from liquidsimulation_b200 import abi, scenes
from liquidsimulation_b200.solver import from_scene

pytestmark = pytest.mark.gpu


def test_positions_into_device_memory():
    sc = scenes.small_box_scene(n_side=(100, 100, 99), s=0.008, solver=abi.LSP_SOLVER_SPH)
    s, lib, n = from_scene(sc), abi.load_library(), len(sc.positions)
    s.update(1e-6)
    out = torch.zeros(3 * n, device="cuda")
    torch.cuda.synchronize()
    ptr = ctypes.cast(out.data_ptr(), ctypes.POINTER(ctypes.c_float))
    best = {}
    for _ in range(80):
        for f in (abi.FIELD_DENSITY, abi.FIELD_POSITION):
            t = time.perf_counter()
            abi.check(lib, lib.lsp_read_field(s._h, f, ptr, n))
            best[f] = min(best.get(f, 1.0), time.perf_counter() - t)
    s.close()
    assert best[abi.FIELD_POSITION] < 1.4 * best[abi.FIELD_DENSITY], best
