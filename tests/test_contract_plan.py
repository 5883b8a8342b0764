"""The contraction's work-unit plan at its edges, on the device: tiles whose lag window is just below, at and
above a whole number of 8-row blocks and of tiles, windows that leave most of a tile out of the channel range,
and a budget that leaves the FP64 path little room for partial tiles."""
import numpy as np
import pytest

import oracle
from amber_b200 import synth

pytestmark = pytest.mark.gpu

WINDOWS = [
    (7, 3, None),          # nclen 7: one 8-row block a slot, 16 slots
    (9, 4, [4]),           # nclen 9: two blocks a slot, the second nearly empty
    (12, 11, None),        # nclen 23, half of every window outside the band
    (33, 31, [0, 32]),     # nclen 63: two slots of 64 rows
    (34, 32, None),        # nclen 65: one slot, the first past the packed tiles
    (48, 47, [5]),         # nclen 95: N = 96
    (66, 64, None),        # nclen 129: two tiles an axis, 72 + 57 lags
    (150, 63, [140]),      # nclen 127, 150 channels: two anchor blocks of 75
]


def _real(nc, nc10, flagged):
    return synth.tiny(32, nc, seed=900 + nc, nbins=3, hi=10.0, nc10=nc10, flagged=flagged)


def _fp64_error(real, **opts):
    import amber_b200
    with amber_b200.Estimator(precision="fp64", **opts) as est:
        _, res = amber_b200.estimate(real, version=2, est=est)
    _, ores = oracle.estimate(real, version=2, with_absscale=True)
    worst = 0.0
    for r, o in zip(res, ores):
        np.testing.assert_array_equal(r["numdnu"], o["numdnu"])
        worst = max(worst, (np.abs(r["bldnu"] - o["bldnu"]) / (o["absscale"] + 1e-300)).max(),
                    (np.abs(r["numtri"] - o["numtri"]) / (o["absscale_i"] + 1e-300)).max())
    return worst


# tolerance of the FP64 path's contract: 1e-10 of the sum of |products| per lag cell
@pytest.mark.parametrize("nc,nc10,flagged", WINDOWS)
def test_fp64_windows_against_oracle(nc, nc10, flagged):
    assert _fp64_error(_real(nc, nc10, flagged)) <= 1e-10


def test_fp64_partial_tiles_keep_to_the_budget():
    """A budget without room for every job's partial tiles at once splits the launch rather than failing."""
    real = synth.tiny(48, 16, seed=77, nbins=4, hi=20.0, nc10=7)
    assert _fp64_error(real, hbm_budget=108 << 20) <= 1e-10


def _digits(x, n, rounded):
    """Base-254 digits of x; every residual rounded to float32 as the device's fused op leaves it."""
    out = []
    for i in range(n):
        d = np.rint(x if i == 0 else 254.0 * x)
        x = (x if i == 0 else 254.0 * x) - d
        if rounded:
            x = x.astype(np.float32).astype(np.float64)
        out.append(d)
    return out


def _fixed_point(m, w, nc10, classes):
    """The mixed path's arithmetic restated: per 256-pixel block one exponent a ring, three digits of ring 2,
    three or four of the float32 product of rings 1 and 3, the digit classes below ``classes`` summed exactly."""
    m = [(x * w[:, None]).astype(np.float32).astype(np.float64) for x in m]
    nc, k = m[0].shape
    nclen = 2 * nc10 + 1
    out = np.zeros((nclen, nclen))
    for x0 in range(0, k, 256):
        b = [x[:, x0:x0 + 256] for x in m]
        e = [int(np.frexp(np.abs(x).max())[1]) if np.abs(x).max() > 0 else 0 for x in b]
        u = (b[0].astype(np.float32) * np.float32(127.0 * 2.0 ** -(e[0] + e[2]))).astype(np.float64)
        t = (b[1].astype(np.float32) * np.float32(127.0 * 2.0 ** -e[1])).astype(np.float64)
        q = _digits(t, 3, True)
        for p1 in range(nc):
            if w[p1] == 0:
                continue
            lo, hi = max(0, p1 - nc10), min(nc, p1 + nc10 + 1)
            p = _digits(u[p1] * b[2][lo:hi], 3 if classes == 3 else 4, True)
            s = sum(254.0 ** -(i + j) * (q[i][lo:hi] @ p[j].T)
                    for i in range(3) for j in range(len(p)) if i + j < classes)
            out[lo - p1 + nc10:hi - p1 + nc10, lo - p1 + nc10:hi - p1 + nc10] += s * 2.0 ** sum(e) / 127.0 ** 2
    return out


# The device's sums of digits are exact, so it differs from the restatement only where a map value sits so near
# a float32 rounding boundary that the two FP64 transforms (1e-15 apart) round it apart: at most a few of ~1e6
# values, 6e-8 of one product each, far below 1e-9 of the largest cell's sum of |products|; a row, column or
# anchor left out or counted twice shows at 1e-2.
@pytest.mark.parametrize("nc,nc10,flagged", WINDOWS)
def test_mixed_windows_against_the_fixed_point_restatement(nc, nc10, flagged):
    import amber_b200
    real = _real(nc, nc10, flagged)
    _, res = amber_b200.estimate(real, precision="mixed", version=2)
    _, ores = oracle.estimate(real, version=2, with_absscale=True)
    gv, mask = oracle.normalize(real.gv, real.counts)
    w = np.zeros(nc)
    w[real.uf_chans] = 1.0
    maps = {}
    for r, o in zip(res, ores):
        for d, (src, classes, key, scale) in enumerate(((gv, 3, "bldnu", "absscale"), (mask, 4, "numtri", "absscale_i"))):
            m = []
            for ring in (r["r1"], r["r2"], r["r3"]):
                at = (d, ring, r["ng1"])
                if at not in maps:
                    maps[at] = oracle.ring_maps(src, real.ulow[ring], real.uhigh[ring], r["ng1"], mask=d == 1)
                m.append(maps[at])
            want = _fixed_point(m, w, nc10, classes)
            got = r[key].reshape(want.shape)
            assert np.abs(got - want).max() <= 1e-9 * np.abs(o[scale]).max(), (r["r1"], r["r2"], r["r3"], key)


# Two tiles an axis whose first is 97 lags or wider: the mask maps' four accumulators do not fit beside their A buffers
# (N = 112 and 128), so they run two sweeps, in tiles of 104 + 89 and of 128 + 123 lags.
@pytest.mark.parametrize("nc,nc10,flagged", [(110, 96, [50]), (126, 125, None)])
def test_mixed_windows_of_two_wide_tiles(nc, nc10, flagged):
    test_mixed_windows_against_the_fixed_point_restatement(nc, nc10, flagged)


@pytest.mark.parametrize("nc,nc10,version", [(40, 19, 2), (24, 11, 2), (20, 19, 1), (33, 31, 2)])
def test_paired_triangles_equal_single_ones(nc, nc10, version):
    """Triangles with the same first and third ring may run as pairs on one formed operand; run one at a time they
    never do.  The digit sums are exact either way, so the lag arrays are equal bit for bit."""
    import amber_b200
    real = synth.tiny(96, nc, seed=55 + nc, nbins=8, hi=44.0, nc10=nc10, flagged=[3])
    with amber_b200.Estimator(precision="mixed") as est:
        est.load_grid(real.gv, real.counts, real.du, real.flag_key)
        est.set_rings(real.ulow, real.uhigh)
        est.set_channels(real.nc10, real.uf_chans)
        tri = est.calcr()[:, :3].astype(np.int32)
        last = tri[tri[:, 0] == 7]  # one r1 group: its ten triangles share a launch, four of them in two pairs
        bl, _, nt = est.triangles(last, want_v2=version == 2)
        for i, t in enumerate(last):
            one, _, none = est.triangles(t[None], want_v2=version == 2)
            np.testing.assert_array_equal(bl[i], one[0])
            if version == 2:
                np.testing.assert_array_equal(nt[i], none[0])
