"""The tile waves at the sizes where their tables end, against the FP64 oracle.

* Coarse waves: a comb of trunk channels whose tiles give one outlet a program
  of fewer than 32, of 32 to 64 and of more than 64 nodes, with more inputs than
  a warp gathers at once.
* The general wave (several receivers): slopes on which few cells start ready,
  on grids of a few cells and of many blocks.
* The stateless accumulation, tiled and by the general wave, and the tiled
  contributing counts.
* Spill heights: boundaries that tie, on few edges (one block) and on many.
* Ids of flats that lie on the edge of a grid without a nodata ring.

The tolerances are those of tests/test_gpu_parity.py.
"""
import numpy as np
import pytest

from parallem_gb300 import scenario as S
from tests.helpers import NODATA, ringed
from tests.test_gpu_parity import check_fa, check_fd, libs, pair, run_steps  # noqa: F401

pytestmark = pytest.mark.gpu


def comb(h, w, spacing):
    """Trunk channels flowing south every `spacing` columns, fed row by row from both sides."""
    y, x = np.mgrid[0:h, 0:w]
    off = np.abs((x + 5) % spacing - spacing // 2)
    z = 900.0 - 0.3 * y + 1.0 * off + 1e-3 * np.random.default_rng(3).random((h, w))
    return ringed(z, 2)


@pytest.mark.parametrize("spacing", [8, 32, 64, 200])
def test_programs_of_every_size_class(libs, spacing):
    run_steps(libs, comb(150, 170, spacing), 2, np.full(2, 900.0), np.full(2, 9.0), False)


def tilted(h, w, dy, dx):
    """A plane with a gentle undulation: no pits, few sources, several receivers per cell."""
    y, x = np.mgrid[0:h, 0:w]
    z = 500.0 + dy * y + dx * x + 3.0 * np.sin(x / 17.0) * np.cos(y / 23.0)
    return ringed(z, 2)


@pytest.mark.parametrize("shape,slope", [((30, 30), (1.0, 0.7)), ((97, 65), (-1.0, 1.2)), ((64, 131), (0.8, -1.0))])
@pytest.mark.parametrize("props", [0, 1])
def test_general_wave_with_several_receivers(libs, shape, slope, props):
    if props == 0 and max(shape) > 30:
        pytest.skip("every receiver takes the whole flow: it overflows on long paths")
    run_steps(libs, tilted(*shape, *slope), 1, np.full(1, 900.0), np.full(1, 9.0), False,
              params=dict(flow_direction_type=1, mfd_proportions=props))


@pytest.mark.parametrize("n", [5, 40, 333])
def test_general_wave_along_one_path_of_all_cells(libs, n):
    """Codes that run boustrophedon through every cell, with one negative weight: the general wave, whose other
    warps wait for all of it."""
    oracle, lem = libs
    dem = ringed(np.full((n, n), 500.0), 2)
    fd = np.full(dem.shape, -9999, np.int32)
    for r in range(n):
        row = fd[2 + r, 2:2 + n]
        row[:] = 1 if r % 2 == 0 else 16
        row[-1 if r % 2 == 0 else 0] = 4
    st = S.initial_state(dem, 30.0, 800.0, 9.0)
    g = lem.Model(dem, 30.0, 800.0, 9.0)
    g.set_state(st)
    g.flow_direction()
    stone = st["stone"].copy()
    stone[2, 2] = 300.0  # runs off less than nothing
    g.set("stone", stone)
    g.set("fd", fd)
    g.set("sfd", fd)
    g.flow_accumulation(lem.STEP_CONTRIB)
    g.synchronize()
    inside = dem[2:-2, 2:-2] != NODATA

    def along(a):  # in path order
        a = a[2:-2, 2:-2].copy()
        a[1::2] = a[1::2, ::-1]
        return a.reshape(-1)

    assert inside.all() and g.totals()["fa_uncomputed"] == 0
    w = along(g.get("runoff"))
    assert w[0] < 0
    want = np.concatenate([w[:1], np.cumsum(w[1:])])  # a negative sum of donors counts as none
    # fp32 weights summed as float pairs: the accumulation tolerance of the parity tests
    np.testing.assert_allclose(along(g.get("fa")), want, rtol=1e-5, atol=0)
    np.testing.assert_array_equal(along(g.get("contrib")), np.arange(1, n * n + 1))
    g.close()


# a strip whose tiles the tables do not hold (the general wave), ragged grids, a code with two receivers
@pytest.mark.parametrize("shape,double", [((1, 40), False), ((3, 40000), False), ((33, 31), False), ((257, 130), False),
                                          ((65, 97), True)])
def test_stateless_accumulation_on_ragged_grids(libs, shape, double):
    torch = pytest.importorskip("torch")
    from parallem_gb300 import lem
    rng = np.random.default_rng(shape[0])
    h, w = shape
    dem = rng.random(shape) + 500.0
    dem[rng.random(shape) < 0.05] = NODATA
    inside = dem != NODATA
    weight = np.where(inside, rng.random(shape) + 0.1, -9999.0)
    # every cell drains east or south-east (to a cell inside, or off the grid): a forest
    step = {1: (0, 1), 2: (1, 1)}
    code = np.where(rng.random(shape) < 0.7, 1, 2).astype(np.int32)
    if double:
        code[h // 2, w // 3] = 3
    code[~inside] = -9999
    want = np.where(inside, weight, 0.0)
    for x in range(w):
        for y in range(h):
            for bit, (dy, dx) in step.items():
                if not inside[y, x] or not code[y, x] & bit:
                    continue
                if y + dy < h and x + dx < w and inside[y + dy, x + dx]:
                    want[y + dy, x + dx] += want[y, x]
    t = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (code, weight, dem)]
    out = torch.full(shape, -1.0, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    rc = lem.load().lem_accumulate_flow_noalloc(t[0].data_ptr(), t[1].data_ptr(), t[2].data_ptr(), out.data_ptr(), w,
                                                h, None)
    assert rc == 0
    # fp32 weights summed as float pairs: the accumulation tolerance of the parity tests
    np.testing.assert_allclose(out.cpu().numpy(), want, rtol=1e-5, atol=0)


@pytest.mark.parametrize("n", [31, 97, 300])
def test_contributing_counts_of_tiled_steps(libs, n):
    from parallem_gb300 import lem
    dem = S.make_dem(n, 0.7, 800.0, 0.03, n, 2, 17)
    o, g, mask = pair(libs, dem, 900.0, 9.0, None, None)
    g.flow_direction()
    g.flow_accumulation(lem.STEP_CONTRIB)
    g.synchronize()
    o.flow_direction()
    o.flow_accumulation()
    check_fa(o, g, mask, contrib=True)


@pytest.mark.parametrize("n", [40, 300])
def test_spill_heights_of_tied_boundaries(libs, n):
    z = S.make_dem(n, 0.6, 60.0, 0.02, n, 2, 5, depressions=n // 4)
    # whole metres: many boundaries tie; above zero, since the reference takes a spill height of 0 for none
    z = np.where(z == NODATA, NODATA, np.floor(z) + 100.0)
    run_steps(libs, z, 1, np.full(1, 900.0), np.full(1, 9.0), False)


@pytest.mark.parametrize("n", [12, 65, 200])
def test_ids_of_winding_closed_flats(libs, n):
    z = tilted(n, n, 0.8, 0.5)
    # a winding pit floor as long as the grid has room for: every cell of it is a sink of one basin
    for i, y in enumerate(range(4, n - 5, 3)):
        z[y, 4:n - 4] = 50.0
        z[y:min(y + 4, n - 5), 4 if i % 2 else n - 5] = 50.0
    run_steps(libs, z, 1, np.full(1, 900.0), np.full(1, 9.0), False)


def edge_lakes(h, w):
    """A grid without a nodata ring: a closed flat over cell (0, 0), and flats and single pits on its other
    edges, each at a height of its own, some of them reaching into the grid.  The ids of the corner's flat
    are above those of the flat in row 0 and below those of the flats further down."""
    y, x = np.mgrid[0:h, 0:w]
    z = 500.0 + 0.8 * y + 0.5 * x + 3.0 * np.sin(x / 17.0) * np.cos(y / 23.0)
    z[0:3, 0:3] = 50.0          # the corner
    z[0, 10:13] = 300.0         # row 0 only: none of its cells has an id
    z[0, 18] = 301.0
    z[0:2, 22:25] = 302.0       # row 0, reaching in
    z[h - 1, 5:8] = 303.0       # the last row
    z[h - 1, 11] = 304.0
    z[h - 2:h, 14:17] = 305.0   # reaching in
    z[8:11, w - 1] = 306.0      # the last column
    z[13, w - 1] = 307.0
    z[16:19, w - 2:w] = 308.0   # reaching in
    z[h - 2:h, w - 2:w] = 309.0  # the opposite corner
    return z


@pytest.mark.parametrize("shape", [(24, 30), (33, 64), (90, 131)])
def test_ids_of_flats_on_the_edges_of_a_grid_without_a_ring(libs, shape):
    z = edge_lakes(*shape)
    o, g, mask = pair(libs, z, 900.0, 9.0, None, None)
    o.flow_direction()
    o.flow_accumulation()
    soil = g.get("soilM")
    for _ in range(10):  # the order in which the sinks are visited differs from call to call
        g.set("soilM", soil)  # runoff changes soil moisture
        g.flow_direction()
        g.flow_accumulation()
        g.synchronize()
        check_fd(o, g, mask)
        np.testing.assert_array_equal(g.get("watershed") == 0, o["watershed"] == 0)
        np.testing.assert_array_equal(g.get("dem_routed"), o["dem_routed"])
        check_fa(o, g, mask)


@pytest.mark.parametrize("n,most", [(64, 1435508), (1024, 363404948)])
def test_records_of_the_coarse_waves_take_no_memory_of_their_own(libs, n, most):
    """`most`: the bytes of a grid whose coarse waves kept 12 bytes a cell (records and links take 20)."""
    oracle, lem = libs
    b = lem.Batch(n, n, 30.0, max_dems=1)
    assert b.device_bytes() <= most
    b.close()
