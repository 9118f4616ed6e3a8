"""Grids to and from the host: reading a field of the host's own type (lem_get_field)
into memory that was never written, into memory that was, and into memory of which
only some pages were; and how the conversions of the other fields are split.

A copy straight into fresh pages waits for each of them (6.5 ms for 9 MB, where
the staging takes 0.5), and one through the staging takes three times as long as
a direct one where the pages are mapped.  The bounds of the times lie between the
ratios measured with the right path and with the wrong one.
"""
import ctypes
import mmap
import time

import numpy as np
import pytest

from parallem_gb300 import scenario as S

pytestmark = pytest.mark.gpu

PAGE = mmap.PAGESIZE


@pytest.fixture(scope="module")
def lem():
    from parallem_gb300 import build, lem
    build.build()
    lem.load()
    return lem


def model(lem, n):
    dem = S.make_dem(n, 0.7, 900.0, 0.02, 5, 2, 3)
    m = lem.Model(dem, 30.0, 800.0, 9.0)
    m.set_state(S.initial_state(dem, 30.0, 800.0, 9.0))
    m.flow_direction()
    m.flow_accumulation(lem.STEP_CONTRIB)
    m.synchronize()
    return m


def fresh(nbytes):
    return np.frombuffer(mmap.mmap(-1, nbytes), np.uint8)


def read(lem, m, field, buf):
    t = time.perf_counter()
    assert lem.load().lem_get_field(m.h, lem.FIELDS[field], ctypes.c_void_p(buf.ctypes.data)) == 0
    return time.perf_counter() - t


@pytest.mark.parametrize("n", [7, 100, 515])
def test_values_do_not_depend_on_where_they_go(lem, n):
    m = model(lem, max(n, 16))
    for field, dtype in (("dem", np.float64), ("contrib", np.int32), ("watershed", np.int32), ("dem_routed", np.float64)):
        want = m.get(field)
        mapped = fresh(want.nbytes + 4 * PAGE)
        mapped[:] = 1
        some = fresh(want.nbytes + 4 * PAGE)
        some[::3 * PAGE] = 1
        for buf in (mapped, some, fresh(want.nbytes + 4 * PAGE)):
            for off in (0, 24, PAGE - 8):  # within a page, across its end
                read(lem, m, field, buf[off:])
                np.testing.assert_array_equal(buf[off:off + want.nbytes].view(dtype).reshape(want.shape), want)
    m.close()


def test_fresh_memory_is_not_written_page_by_page(lem):
    """16.8 MB: fresh pages 102 times as long as mapped ones by a direct copy, 6 times through the staging."""
    m = model(lem, 2048)
    n = 2048 * 2048 * 4
    mapped = fresh(n)
    mapped[:] = 1
    t_mapped = min(read(lem, m, "contrib", mapped) for _ in range(9))
    t_fresh = min(read(lem, m, "contrib", fresh(n)) for _ in range(9))
    assert t_fresh < 25 * t_mapped
    m.close()


def test_a_large_array_in_use_is_written_directly(lem):
    """Per byte, 134 MB against 16.8 MB of mapped memory: 2.8 times as long through the staging, 0.9 times directly."""
    t = []
    for n, field, size in ((2048, "contrib", 4), (4096, "dem", 8)):
        m = model(lem, n)
        buf = fresh(n * n * size)
        buf[:] = 1
        t.append(min(read(lem, m, field, buf) for _ in range(9)) / buf.nbytes)
        m.close()
    assert t[1] < 1.6 * t[0]


def test_codes_of_a_larger_grid_take_no_longer_per_cell(lem):
    """Setting codes at 1500 x 1500 against 800 x 800 cells: 1.04 to 1.23 times as long per cell when threads narrow
    a quarter of a million cells each, 0.62 to 0.68 times when each has twice as many."""
    t = []
    for n in (800, 1500):
        m = model(lem, n)
        fd = m.get("fd")
        best = 1.0
        for _ in range(40):
            a = time.perf_counter()
            assert lem.load().lem_set_field(m.h, lem.FIELDS["fd"], ctypes.c_void_p(fd.ctypes.data)) == 0
            best = min(best, time.perf_counter() - a)
        t.append(best / fd.size)
        m.close()
    assert t[1] < t[0]
