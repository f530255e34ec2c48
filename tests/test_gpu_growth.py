"""Kept workspaces under calls of slowly growing size: a few allocations for
the whole run, not one or more per call.  Allocations show as changes of the
kept blocks, or of the device's free memory."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class Workspace(ctypes.Structure):
    _fields_ = [("dev", ctypes.c_void_p), ("host", ctypes.c_void_p), ("dev_len", ctypes.c_size_t),
                ("host_len", ctypes.c_size_t)]


def test_workspace_growth():
    import maise_b200

    lib = maise_b200.load_library()
    lib.mb_ws_grow.argtypes = [ctypes.POINTER(Workspace), ctypes.c_size_t, ctypes.c_size_t]
    lib.mb_ws_free.argtypes = [ctypes.POINTER(Workspace)]
    ws = Workspace()
    seen = set()
    need = 100_000
    for _ in range(100):  # 2% a step: 7.2 times the first size at the end
        need = need + need // 50
        assert lib.mb_ws_grow(ctypes.byref(ws), need, need // 2) == 0
        assert ws.dev_len >= need and ws.host_len >= need // 2
        seen.add((ws.dev_len, ws.host_len))
    dev, host = ws.dev_len, ws.host_len
    assert lib.mb_ws_grow(ctypes.byref(ws), need // 3, need // 3) == 0  # never shrinks
    assert (ws.dev_len, ws.host_len) == (dev, host)
    lib.mb_ws_free(ctypes.byref(ws))
    # a block at least doubles: at most 1 + log2(7.2) = 3.8 sizes of each, so 12 is generous
    assert len(seen) <= 12
    assert dev <= 2 * need and host <= need


def test_generations_of_growing_size():
    import torch

    from maise_b200.surrogate import Surrogate

    rng = np.random.default_rng(1)
    pop = [dict(X=rng.uniform(0, 8, (30, 3)), LAT=8.0 * np.eye(3), atmn=np.sort(rng.integers(0, 3, 30)).astype(np.int32))
           for _ in range(2000)]
    torch.cuda.synchronize()
    sur = Surrogate(3)
    free = []
    for S in range(200, 2001, 150):
        sur.screen(pop[:S])
        free.append(torch.cuda.mem_get_info()[0])
    sur.close()
    # 13 calls from 200 to 2000 structures: inputs, features and rows at least double, 1 + log2(10) = 4.3 sizes each,
    # mostly at the same calls
    assert len(set(free)) <= 7
