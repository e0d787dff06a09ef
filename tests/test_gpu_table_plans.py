"""Planned tables where the builder's paths part: identity planes (no map) of one word and of two, with unused leading variables and
with fixed coordinates, cubes shorter than a span of entries and one entry past it, and the entry that takes the caller's own maps."""
import numpy as np
import pytest

import tables_util as T

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    from intelligenceregulation_b200 import backend

    d = backend.B200Backend(device=0)
    yield d
    d.ctx.close()


@pytest.fixture(scope="module")
def committed(dev):
    data = np.random.default_rng(98).integers(0, T.P, size=64 << 10, dtype=np.uint64)
    store, _ = dev.try_commit(10, 2, data, 12)
    yield store, data
    store.free()


def _cases():
    fixed = [("fixed", (12345678901, 987654321)), ("fixed", (5, T.P - 1))]
    for n in (0, 1, 9, 10, 11, 13):
        cube = [("rho", v) for v in range(n)]
        yield n, cube, [(3, (1, 0))]
        yield n, cube, [(5, (1, 0)), (1 << 14, (0, 1))]
        yield n, cube, [(5, (1, 0)), (7, (2, 1)), (9, (0, 1))]
        yield n, fixed + cube, [(1, (1, 0))]
        yield n, fixed + cube, [(1, (1, 0)), (77, (0, 1))]
        if n > 3:
            yield n, cube[2:], [(3, (1, 0))]
            yield n, cube[::-1], [(3, (1, 0)), (4, (0, 1))]
            yield n, [("flip", v) for v in range(n)], [(3, (1, 0))]


@pytest.mark.parametrize("case", list(_cases()), ids=lambda c: f"{c[0]}-{len(c[1])}-{len(c[2])}")
def test_a_plane_both_ways(dev, oracle, committed, case):
    from intelligenceregulation_b200 import backend

    store, data = committed
    n, coords, slices = case
    want = oracle.priv_table(coords, slices, data, n)
    t = backend.B200Tables(dev.ctx, 2, n)
    t.plan_plane(0, store, coords, slices)
    used, xlo, inv_lo, inv_hi, zbits, eqf = backend.plane_maps(n, coords)
    sl = np.array([[off, cf[0], cf[1]] for off, cf in slices], dtype=np.uint64)
    nz = zbits.size
    dev.ctx.check(dev.ctx.lib.hl_b200_tables_plane(t.h, 1, store.h, None, 0, used, xlo, backend._ptr(inv_lo), backend._ptr(inv_hi),
                                                   backend._ptr(zbits) if nz else None, nz, backend._ptr(eqf) if nz else None, backend._ptr(sl), sl.shape[0], 0))
    assert (t.read(0) == want).all() and (t.read(1) == want).all()
    t.free()


def test_refusals(dev, committed):
    from intelligenceregulation_b200 import backend

    t = backend.B200Tables(dev.ctx, 1, 10)
    with pytest.raises(ValueError):
        t.plan_plane(0, committed[0], [("rho", 1), ("flip", 1)], [(0, (1, 0))])
    for coords, off in (([("rho", 10)], 0), ([("rho", v) for v in range(10)], (64 << 10) - 1023)):  # outside the cube; past the rows
        with pytest.raises(backend.DeviceError):
            t.plan_plane(0, committed[0], coords, [(off, (1, 0))])
    with pytest.raises(backend.DeviceError):
        t.plan_eq(0, np.zeros((4, 2), dtype=np.uint64), 7)
    t.free()
