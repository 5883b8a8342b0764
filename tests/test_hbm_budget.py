"""Triangle runs near their HBM budget: ring maps come in as many batches as the budget asks for, whatever the
context's buffers hold from the grid upload and from earlier runs, and the batches change no result."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MB = 1 << 20
DU = 1.0
MAP_BYTES = {"fp64": 8, "bf16x3": 4, "mixed": 7}  # per map value; the mixed path's also have block exponents


def _grid(nn, nc, hi, seed):
    """Random cells inside every ring (|U| < hi cells), nothing elsewhere."""
    rng = np.random.default_rng(seed)
    gv, counts = np.zeros((nn, nn // 2 + 1, nc), np.complex128), np.zeros((nn, nn // 2 + 1, nc))
    rows = np.r_[0:hi + 1, nn - hi:nn]
    shape = (len(rows), hi + 1, nc)
    gv[rows, :hi + 1] = rng.standard_normal(shape) + 1j * rng.standard_normal(shape)
    counts[rows, :hi + 1] = 1.0
    return gv, counts


def _slot(precision, ng, nc):
    """Bytes of one ring slot of one map set, and of its share of the map builder's intermediate."""
    kp = (ng * ng + 255) // 256 * 256
    return MAP_BYTES[precision] * nc * kp + 8 * nc + 4 * (kp // 256 + 1), 16 * ng * (ng // 3 + 1) * nc


def _estimator(precision, gv, counts, edges, nc10, budget=0):
    import amber_b200
    est = amber_b200.Estimator(precision=precision, hbm_budget=budget)
    est.load_grid(gv, counts, DU, 0)
    est.set_rings(edges[:-1], edges[1:])
    est.set_channels(nc10)
    return est


@pytest.mark.parametrize("precision,nn,nc,reserve", [("bf16x3", 256, 128, 64), ("mixed", 512, 256, 64 + 512)])
def test_batches_leave_out_the_staged_grid_upload(precision, nn, nc, reserve):
    """The buffer a grid was staged in stays held: a budget with room for four and a half of a group's 24 rings
    beside it runs the group in batches."""
    gv, counts = _grid(nn, nc, 40, 5)
    edges = np.linspace(4.0, 40.0, 25)
    tri = np.array([(23, r, r) for r in range(24)], np.int32)
    with _estimator(precision, gv, counts, edges, 7) as est:
        want = est.triangles(tri)
        maps, y = _slot(precision, est.ng1(23), nc)
    budget = 2 * 24 * gv.size + (reserve + 2) * MB + 9 * (maps + y) // 2
    with _estimator(precision, gv, counts, edges, 7, budget) as est:
        got = est.triangles(tri)
    np.testing.assert_array_equal(got[0], want[0])
    np.testing.assert_array_equal(got[1], want[1])


@pytest.mark.parametrize("precision,nn,nc,hi,reserve", [("fp64", 256, 32, 120, 64), ("mixed", 512, 56, 240, 64 + 512)])
def test_batches_count_the_mask_maps_of_an_earlier_run(precision, nn, nc, hi, reserve):
    """A run without mask sums after one with them: the mask maps still held are given back where the budget, which
    holds one map set of all eight rings, needs their room."""
    gv, counts = _grid(nn, nc, hi, 6)
    edges = np.linspace(4.0, hi, 9)
    tri = np.array([(7, r, r) for r in range(8)], np.int32)
    with _estimator(precision, gv, counts, edges, 3) as est:
        want = est.triangles(tri)
        maps, y = _slot(precision, est.ng1(7), nc)
    budget = 2 * 24 * gv.size + (reserve + 2) * MB + 8 * (maps + y)
    with _estimator(precision, gv, counts, edges, 3, budget) as est:
        est.run(np.array([(7, 6, 5), (7, 6, 4)], np.int32), want_v2=True)
        got = est.triangles(tri)
    np.testing.assert_array_equal(got[1], want[1])
    # FP64 units depend on the room for partial tiles: other groupings of the same sums
    np.testing.assert_allclose(got[0], want[0], rtol=0, atol=1e-10 * np.abs(want[0]).max())


def test_maps_leave_room_for_the_split_bf16_tiles():
    """Partial tiles larger than the reserve, beside them room for three of eight rings: batches, not all rings first."""
    gv, counts = _grid(120, 64, 56, 9)
    edges = np.linspace(4.0, 56.0, 9)
    tri = np.array([(7, r, r) for r in range(8)], np.int32)
    with _estimator("bf16x3", gv, counts, edges, 63) as est:
        want = est.triangles(tri)
        maps, y = _slot("bf16x3", est.ng1(7), 64)
    tiles = 8 * 64 * 19 * 127 ** 2  # anchors, pixel chunks on 148 SMs, lag cells
    budget = 24 * gv.size + tiles + 32 * MB + 32 * (maps + y) // 10
    with _estimator("bf16x3", gv, counts, edges, 63, budget) as est:
        got = est.triangles(tri)
    np.testing.assert_array_equal(got[0], want[0])


@pytest.mark.parametrize("precision", ["bf16x3", "mixed", "fp64"])
def test_a_run_that_fits_fits_again(precision):
    """The partial tiles a run leaves held do not turn the same run away: a budget for just over a triangle's rings."""
    gv, counts = _grid(60, 86, 28, 8)
    edges = np.array([2.0, 15.0, 28.0])
    with _estimator(precision, gv, counts, edges, 42) as est:
        maps, y = _slot(precision, est.ng1(1), 86)
    budget = 2 * 24 * gv.size + (64 + 512 * (precision == "mixed") + 1) * MB + 31 * (maps + y) // 10
    with _estimator(precision, gv, counts, edges, 42, budget) as est:
        first = est.triangles([(1, 1, 0)])
        again = est.triangles([(1, 1, 0)])
    for a, b in zip(again, first):
        np.testing.assert_array_equal(a, b)


def test_failed_run_leaves_no_results():
    """A run refused for its arguments keeps the last run's results; one that failed on the device has none."""
    import amber_b200
    gv, counts = _grid(512, 16, 240, 7)
    with _estimator("fp64", gv, counts, np.array([2.0, 6.0, 200.0, 240.0]), 3, 2 * 24 * gv.size + 84 * MB) as est:
        one = est.triangles([(0, 0, 0)], want_v2=True)
        with pytest.raises(amber_b200.AmberError):
            est.run([(0, 0, 3)])
        again = est.fetch(want_v2=True)
        for a, b in zip(again, one):
            np.testing.assert_array_equal(a, b)
        with pytest.raises(amber_b200.AmberError):
            est.run([(0, 0, 0), (2, 2, 2)])  # the second triangle's maps exceed the budget
        assert est.last_run_shape()[0] == 0
        assert len(est.fetch()[0]) == 0
        with pytest.raises(amber_b200.AmberError):
            est.cyl_bs(n_cut=1)
