"""md_system_set_fields / md_system_get_fields with columns that touch, or lie at a constant
distance, but are page-locked one by one or not at all: a copy may not span two of them, and
what lies between them stays as it is."""
import ctypes as C
import mmap

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("locked", [(0, 1, 2), (0, 2), (1,), "whole", ()])
@pytest.mark.parametrize("gap", [0, 4096])
def test_columns_locked_apart(md, locked, gap):
    import torch

    n, size = 4096, 4096 * 8  # whole pages
    rt = torch.cuda.cudart()
    block = mmap.mmap(-1, 3 * (size + gap))
    rows = np.frombuffer(block, np.float64).reshape(3, n + gap // 8)
    cols = rows[:, :n]
    rows[:, n:] = -1.0
    spans = ([(rows[0].ctypes.data, 3 * (size + gap))] if locked == "whole"
             else [(cols[k].ctypes.data, size) for k in locked])
    want = np.random.default_rng(3).uniform(-6, 6, (3, n))
    s = md.System(n, [12.0, 12.0, 12.0])
    fields = (C.c_int * 3)(md.FIELD_VX, md.FIELD_VY, md.FIELD_VZ)
    ptrs = (C.POINTER(C.c_double) * 3)(*[c.ctypes.data_as(C.POINTER(C.c_double)) for c in cols])
    for p, length in spans:
        assert int(rt.cudaHostRegister(p, length, 0)) == 0
    try:
        cols[:] = want
        md._check(md.lib().md_system_set_fields(s.handle, 3, fields, ptrs))
        assert np.array_equal(s.velocities, want.T)
        cols[:] = 0.0
        md._check(md.lib().md_system_get_fields(s.handle, 3, fields, ptrs))
        assert np.array_equal(cols, want) and np.all(rows[:, n:] == -1.0)
    finally:
        for p, _ in spans:
            rt.cudaHostUnregister(p)
