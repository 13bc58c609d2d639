"""State and field transfers with buffers in device memory, which the copies have always taken (unified
addressing): they must not be touched by the host. Single scenes and batches, alone and mixed with
host buffers, below and above the limit of the pinned stage (1 MB). Exact equality."""
import ctypes

import numpy as np
import pytest
import torch

from liquidsimulation_b200 import abi
from liquidsimulation_b200.solver import batch_from_scenes, from_scene
from test_host_transfers import scene

pytestmark = pytest.mark.gpu

FP, IP = ctypes.POINTER(ctypes.c_float), ctypes.POINTER(ctypes.c_int32)


def buffers(n, where):
    """Five state arrays; where: "device", or "mixed" with every other one in host memory."""
    out = []
    for c in range(5):
        host = where == "mixed" and c % 2 == 0
        out.append(torch.zeros(n * (1 if c == 4 else 3), dtype=torch.int32 if c == 4 else torch.float32,
                               device="cpu" if host else "cuda"))
    torch.cuda.synchronize()
    return out


def ptrs(ts):
    return [ctypes.cast(t.data_ptr(), IP if t.dtype == torch.int32 else FP) for t in ts]


def state(n, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    return [rng.normal(0.5, 0.1, 3 * n).astype(np.float32) for _ in range(4)] + [rng.integers(0, 2, n).astype(np.int32)]


def equal(ts, arrs):
    torch.cuda.synchronize()
    return all(np.array_equal(t.cpu().numpy(), a) for t, a in zip(ts, arrs))


@pytest.mark.parametrize("n", [300, 30000])
@pytest.mark.parametrize("where", ["device", "mixed"])
def test_single_scene(n, where):
    sc = scene(n)
    s, lib = from_scene(sc), abi.load_library()
    s.update(sc.dt)
    want = state(n, n)
    src, dst = buffers(n, where), buffers(n, where)
    for t, a in zip(src, want):
        t.copy_(torch.from_numpy(a))
    torch.cuda.synchronize()
    abi.check(lib, lib.lsp_write_state(s._h, *ptrs(src), n))
    abi.check(lib, lib.lsp_read_state(s._h, *ptrs(dst), n))
    assert equal(dst, want)
    x, v = buffers(n, where)[:2]
    abi.check(lib, lib.lsp_read_particles(s._h, *ptrs([x, v]), n))
    assert equal([x, v], want[:2])
    h = buffers(n, "device")[0]
    abi.check(lib, lib.lsp_read_field(s._h, abi.FIELD_HALF_VELOCITY, *ptrs([h]), n))
    assert equal([h], want[2:3])
    s.close()


@pytest.mark.parametrize("where", ["device", "mixed"])
def test_batch(where):
    scs = [scene(n) for n in (40, 300)]
    b, lib = batch_from_scenes(scs), abi.load_library()
    b.update(scs[0].dt)
    n = b.total
    want = state(n, 5)
    src, dst = buffers(n, where), buffers(n, where)
    for t, a in zip(src, want):
        t.copy_(torch.from_numpy(a))
    torch.cuda.synchronize()
    abi.check(lib, lib.lsp_batch_write_state(b._h, *ptrs(src), n))
    abi.check(lib, lib.lsp_batch_read_state(b._h, *ptrs(dst), n))
    assert equal(dst, want)
    x = buffers(300, "device")[0]
    abi.check(lib, lib.lsp_batch_read_field(b._h, 1, abi.FIELD_POSITION, *ptrs([x]), 300))
    assert equal([x], [want[0][120:]])
    b.close()
