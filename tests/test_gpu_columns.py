"""md_system_set_fields / md_system_get_fields over the host layouts that are copied
differently: columns end to end, rows of a larger array, unrelated columns, descending
addresses and a repeated field; after a re-sort of the device order too."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
DP = C.POINTER(C.c_double)


def pointers(cols):
    return (DP * len(cols))(*[c.ctypes.data_as(DP) for c in cols])


def layouts(k, n):
    yield "end to end", list(np.zeros((k, n)))
    yield "rows", [r[3:3 + n] for r in np.zeros((k, n + 40))]
    yield "separate", [np.zeros(n + 7 * i)[:n] for i in range(k)]
    yield "descending", list(np.zeros((k, n)))[::-1]
    mixed = np.zeros((k + 2, n))
    yield "two runs", [mixed[i if i < k // 2 else i + 2] for i in range(k)]


@pytest.mark.parametrize("n", [1, 255, 256, 2048])
@pytest.mark.parametrize("resort", [False, True])
def test_columns_round_trip(md, n, resort):
    rng = np.random.default_rng(n)
    fields = [md.FIELD_VZ, md.FIELD_X, md.FIELD_MASS, md.FIELD_Y, md.FIELD_Z, md.FIELD_FX,
              md.FIELD_FY, md.FIELD_FZ, md.FIELD_CHARGE, md.FIELD_VX, md.FIELD_VY]
    s = md.System(n, [12.0, 12.0, 12.0])
    if resort:
        s.positions = rng.uniform(-6, 6, (n, 3))
        md.VerletList([12.0] * 3, 2.5, 0.3).build(s)
    L = md.lib()
    for name, cols in layouts(len(fields), n):
        want = rng.uniform(-6, 6, (len(fields), n))
        want[2] = np.abs(want[2]) + 0.5
        for c, w in zip(cols, want):
            c[:] = w
        codes = (C.c_int * len(fields))(*fields)
        md._check(L.md_system_set_fields(s.handle, len(fields), codes, pointers(cols)))
        for other, out in layouts(len(fields), n):
            md._check(L.md_system_get_fields(s.handle, len(fields), codes, pointers(out)))
            assert all(np.array_equal(o, w) for o, w in zip(out, want)), (name, other)
        assert np.array_equal(s.velocities[:, 2], want[0]) and np.array_equal(s.masses, want[2])
    twice = (C.c_int * 13)(*([md.FIELD_X] * 13))  # more columns than there are fields
    out = list(np.zeros((13, n)))
    md._check(L.md_system_get_fields(s.handle, 13, twice, pointers(out)))
    assert all(np.array_equal(o, want[1]) for o in out)
