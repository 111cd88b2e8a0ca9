"""The fixed-point weights and contraction of the FP64 path.

On the CPU: csrc/fx_weight.cuh, compiled for the host, against 60-digit decimal
values.  A bisquare weight carries two truncated squares relative to
rho >= 2^60 (2^-59), the truncated product with 2^124 / rho and its own square,
2^-57 in all; a gaussian weight adds the granularity of the squared distance
relative to rho >= 2^53.5, up to 2^-53 of the exponent.

On the GPU: criteria and fits against the oracle at the drop-in's bars (criteria
1e-9, beta 1e-10 relative), at the edges of the 128-row blocks, the 16-point
tiles, the 1024-point scale blocks and the 64-column groups, and where the FP64
kernel has to take over (weights far below 1, wide dynamic range, rounded
coordinates)."""
import ctypes
import os
import random
import subprocess
from decimal import Decimal, getcontext

import numpy as np
import pytest

import oracle as O
from parity_util import col_rel

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("fx") / "fx_host.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", os.path.join(HERE, "arith", "fx_host.cpp"), "-o", so],
                   check=True)
    lib = ctypes.CDLL(so)
    lib.fx_weight.restype = ctypes.c_uint64
    lib.fx_weight.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.c_double, ctypes.c_int, ctypes.c_int64, ctypes.c_int64]
    lib.fx_geo_weight.restype = ctypes.c_uint64
    lib.fx_geo_weight.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.c_double, ctypes.c_void_p, ctypes.c_void_p]
    lib.fx_ratio63.restype = ctypes.c_uint64
    lib.fx_ratio63.argtypes = [ctypes.c_uint64, ctypes.c_uint64]
    lib.fx_square.restype = ctypes.c_uint64
    lib.fx_square.argtypes = [ctypes.c_uint64]
    return lib


@pytest.mark.parametrize("gauss", [0, 1])
@pytest.mark.parametrize("ratio", [1e-6, 1e-3, 0.1, 1.0, 1.7, 300.0])  # threshold over extent
def test_weights_against_decimal(host, gauss, ratio):
    getcontext().prec = 60
    rng = random.Random(int(ratio * 1e7) + gauss)
    for it in range(400):
        extent = 2.0 ** rng.uniform(-20, 30)
        r = extent * ratio * rng.uniform(0.5, 1.0) if it % 8 else 2.0 ** rng.randint(-8, 8)
        scale = 60 - int(np.floor(np.log2(max(extent, r / ratio))))
        reach = (9.4 if gauss else 1.02) * (rng.random() if it % 3 else rng.random() ** 0.1)
        a = rng.uniform(0, 6.283)
        dx, dy = (int(reach * r * f * 2.0 ** scale) for f in (np.cos(a), np.sin(a)))
        if max(abs(dx), abs(dy)) >> 61:
            continue
        q = (Decimal(dx) ** 2 + Decimal(dy) ** 2) / Decimal(2) ** (2 * scale) / Decimal(r) ** 2
        want = (-q / 2).exp() if gauss else ((1 - q) ** 2 if q < 1 else Decimal(0))
        got = Decimal(host.fx_weight(gauss, it % 5 == 0, r, scale, dx, dy)) / Decimal(2) ** 62
        bound = Decimal(2) ** -60 + want * (q + 1) * Decimal(2) ** -53 if gauss else Decimal(2) ** -57
        assert abs(got - want) <= bound, (gauss, r, scale, dx, dy, got, want)
    assert host.fx_weight(gauss, 0, 1.5, 60, 0, 0) in (1 << 62, (1 << 62) - 1, (1 << 62) - 2)


@pytest.mark.parametrize("r", [0.0, -1.0, float("inf"), float("nan"), 5e-324])
def test_no_weight_without_a_threshold(host, r):
    assert host.fx_weight(0, 0, r, 10, 5, 5) == 2 ** 64 - 1
    assert host.fx_weight(1, 0, r, 10, 5, 5) == 2 ** 64 - 1


def _sincos(x):
    """sin and cos of a Decimal by their Taylor series (|x| <= 4)."""
    s, c, t, k = Decimal(0), Decimal(0), Decimal(1), 0
    while abs(t) > Decimal(10) ** -55:
        (s, c) = (s, c + t) if k % 2 == 0 else (s + t, c)
        t = t * x / (k + 1) * (-1 if k % 2 == 1 else 1)
        k += 1
    return s, c


def _asin(x):
    """asin of a small Decimal (x <= 1/2) by its series."""
    t, s, k = x, x, 1
    while t > Decimal(10) ** -55:
        t = t * x * x * k / (k + 1)
        k += 2
        s += t / k
    return s


def _great_circle2(lon1, lat1, lon2, lat2):
    """(squared distance in km, chord) of the reference's formula, unit vectors times 2^61."""
    (so1, co1), (sa1, ca1), (so2, co2), (sa2, ca2) = map(_sincos, (lon1, lat1, lon2, lat2))
    e1, e2 = (ca1 * co1, ca1 * so1, sa1), (ca2 * co2, ca2 * so2, sa2)
    S = sum((a - b) ** 2 for a, b in zip(e1, e2)) / 4
    C = 1 - S
    w = _asin(S.sqrt())
    R = (S * C).sqrt() / w
    f = 1 / Decimal("298.257223563")
    D = 2 * w * Decimal("6378.137")
    D *= 1 + f * (3 * R - 1) / (2 * C) * ((sa1 + sa2) / 2) ** 2 - f * (3 * R + 1) / (2 * S) * ((sa1 - sa2) / 2) ** 2
    q = [[int((v * 2 ** 61).to_integral_value()) for v in e] for e in (e1, e2)]
    return D, 2 * S.sqrt(), q


@pytest.mark.parametrize("gauss", [0, 1])
@pytest.mark.parametrize("span", [0.02, 1.0, 12.0, 50.0])  # degrees
def test_great_circle_weights_against_decimal(host, gauss, span):
    """The unit vectors' rounding (2^-62 a component, against the chord), the polynomials (2^-54) and the
    granularity of the squared distance (gaussian 2^-51 of the exponent), doubled in the square."""
    getcontext().prec = 60
    rng = random.Random(int(span * 100) + gauss)
    done = 0
    for it in range(150):
        lon, lat = rng.uniform(-3.1, 3.1), rng.uniform(-1.5, 1.5)
        near = np.radians(span) * rng.random()
        a = rng.uniform(0, 6.283)
        other = (lon + near * np.cos(a) / max(np.cos(lat), 0.1), min(1.57, max(-1.57, lat + near * np.sin(a))))
        D, chord, (q1, q2) = _great_circle2(*map(Decimal, (lon, lat) + other))
        if chord > Decimal("0.999") or chord < Decimal(10) ** -6:
            continue
        r = float(D) * rng.uniform(0.15 if gauss else 0.95, 4.0)
        q = (D / Decimal(r)) ** 2
        want = (-q / 2).exp() if gauss else ((1 - q) ** 2 if q < 1 else Decimal(0))
        v1, v2 = (ctypes.c_int64 * 3)(*q1), (ctypes.c_int64 * 3)(*q2)
        got = Decimal(host.fx_geo_weight(gauss, it % 5 == 0, r, v1, v2)) / 2 ** 62
        rel = 4 * Decimal(2) ** -62 / chord + Decimal(2) ** -52
        bound = Decimal(2) ** -60 + (want * q if gauss else 2 * min(q, 1)) * rel + (want * Decimal(2) ** -51 if gauss else 0)
        assert abs(got - want) <= bound, (gauss, r, lon, lat, other, got, want)
        done += 1
    assert done > 60
    same = (ctypes.c_int64 * 3)(2 ** 60, 2 ** 60, 3 ** 37)
    assert host.fx_geo_weight(gauss, 0, 25.0, same, same) >= (1 << 62) - 2


def test_ratio(host):
    rng = random.Random(3)
    for _ in range(200000):
        den = rng.getrandbits(rng.randint(1, 63)) or 1
        num = rng.randint(0, den)
        assert abs(host.fx_ratio63(num, den) - (num << 63) // den) <= 8, (num, den)
    assert host.fx_ratio63(0, 0) == 0


def test_square(host):
    for w in (0, 1, 1 << 31, (1 << 62) - 1, 1 << 62, 0x123456789abcdef0 >> 3):
        assert abs(host.fx_square(w) - (w * w >> 62)) <= 1


def problem(n, p, seed, extent=100.0, offset=0.0):
    rng = np.random.default_rng(seed)
    x = np.column_stack([np.ones(n), rng.standard_normal((n, p - 1))]) if p > 1 else np.ones((n, 1))
    coords = offset + rng.uniform(0, extent, (n, 2))
    return x, x.sum(1) + rng.normal(0, 0.3, n), coords


def engine(x, y, coords, geographic=False):
    from libgwmodel_gb300 import Engine
    e = Engine(0)
    e.set_data(x, y, coords, geographic)
    return e


def check(x, y, coords, cases, fit=True, geographic=False):
    e, ref = engine(x, y, coords, geographic), O.Problem(x, y, coords, geographic=geographic)
    for adaptive, kernel, bw in cases:
        for crit in (O.AIC, O.CV):
            want, _ = ref.criterion(bw, adaptive, kernel, crit)
            got = e.criterion(bw, adaptive, kernel, crit)
            assert abs(got - want) <= 1e-9 * abs(want), (adaptive, kernel, bw, crit, got, want)
        if fit:
            betas, se, shat, qdiag, S = e.fit(bw, adaptive, kernel)
            rb, rse, rshat, rq, rS = ref.fit_core(bw, adaptive, kernel)[:5]
            assert col_rel(betas, rb) <= 1e-10
            assert col_rel(se, rse) <= 1e-9
            np.testing.assert_allclose(shat, rshat, rtol=1e-9)
            np.testing.assert_allclose(qdiag, rq, rtol=1e-9)


@pytest.mark.gpu
@pytest.mark.parametrize("n,p", [(17, 2), (127, 1), (128, 4), (129, 5), (1023, 3), (1025, 9), (600, 10), (900, 17),
                                 (700, 21), (640, 25)])
def test_contraction_edges(n, p):
    x, y, coords = problem(n, p, n + p)
    check(x, y, coords, [(True, O.BISQUARE, max(n // 2, min(n - 1, 3 * p))), (True, O.GAUSSIAN, max(n // 3, min(n - 1, 2 * p))),
                         (False, O.GAUSSIAN, 40.0), (False, O.BISQUARE, 160.0)])


@pytest.mark.gpu
def test_thresholds_above_the_extent_and_large_offsets():
    x, y, coords = problem(500, 3, 7, extent=3.0, offset=5e6)  # rounded in the last bits
    check(x, y, coords, [(False, O.GAUSSIAN, 1e4), (False, O.BISQUARE, 900.0), (True, O.BISQUARE, 700.0),
                         (True, O.GAUSSIAN, 60)])


@pytest.mark.gpu
def test_rows_without_a_weight_near_one():
    """Leave-one-out rows six to nine bandwidths from their neighbours: gaussian weights of 1e-8 to 1e-18.
    An intercept alone: with covariates such rows' local systems have condition numbers above 1e8, where the
    FP64 oracle itself is 2e-9 off the criterion's value in 200-bit arithmetic."""
    x, y, coords = problem(400, 1, 8)
    coords[:6] = 160.0 + np.arange(6)[:, None] * 30.0
    check(x, y, coords, [(False, O.GAUSSIAN, 7.0)], fit=False)


@pytest.mark.gpu
@pytest.mark.parametrize("which", ["one", "tile", "half"])
@pytest.mark.parametrize("scale", [1e-3, 1e9])
def test_wide_dynamic_range(scale, which):
    """A covariate that is 1e7 times larger at one point, within one cluster or at every second point: one scale
    per block would cost the other points their bits."""
    x, y, coords = problem(1500, 3, 9)
    x[:, 2] *= scale
    far = {"one": [700], "tile": np.hypot(*(coords - 50).T) < 8, "half": slice(None, None, 2)}[which]
    x[far, 2] *= 1e7
    check(x, y, coords, [(True, O.BISQUARE, 200)], fit=False)


@pytest.mark.gpu
def test_coordinates_far_finer_than_the_extent():
    """A cluster 1e-9 of the extent wide: integer coordinates would round it."""
    x, y, coords = problem(600, 3, 10, extent=1e-4)
    coords[500:] *= 1e9
    check(x, y, coords, [(True, O.GAUSSIAN, 60), (True, O.GAUSSIAN, 25)], fit=False)


@pytest.mark.gpu
def test_predictions_near_and_far():
    x, y, coords = problem(900, 4, 11)
    rng = np.random.default_rng(12)
    at = np.concatenate([rng.uniform(0, 100, (130, 2)), rng.uniform(300, 320, (3, 2)), [[1e7, 1e7]]])
    e, ref = engine(x, y, coords), O.Problem(x, y, coords)
    for adaptive, kernel, bw in [(True, O.BISQUARE, 90), (True, O.GAUSSIAN, 90), (False, O.GAUSSIAN, 1e7)]:
        assert col_rel(e.predict(at, bw, adaptive, kernel), ref.predict(at, bw, adaptive, kernel)) <= 1e-10
    near = at[:130]  # 15 bandwidths beyond them the far ones' weights underflow
    assert col_rel(e.predict(near, 20.0, False, O.GAUSSIAN), ref.predict(near, 20.0, False, O.GAUSSIAN)) <= 1e-10


def degrees(coords, lon0, lat0, span):
    return np.column_stack([lon0 + coords[:, 0] * span / 100, lat0 + coords[:, 1] * span / 200])


@pytest.mark.gpu
@pytest.mark.parametrize("n,p,lon0,lat0,span", [(129, 2, 0.0, 40.0, 0.5), (1025, 9, -10.0, 35.0, 40.0),
                                                (640, 17, 170.0, -60.0, 25.0),   # across the antimeridian
                                                (700, 4, 0.0, 84.0, 12.0),       # to the pole
                                                (500, 3, -60.0, -30.0, 120.0)])  # wider than the cap: FP64 weights
def test_geographic_contraction(n, p, lon0, lat0, span):
    x, y, coords = problem(n, p, n + p)
    g = degrees(coords, lon0, lat0, span)
    g[:, 0] = np.where(g[:, 0] > 180, g[:, 0] - 360, g[:, 0])
    check(x, y, g, [(True, O.BISQUARE, n // 2), (True, O.GAUSSIAN, n // 3), (False, O.GAUSSIAN, 30.0 * span)],
          geographic=True)


@pytest.mark.gpu
def test_geographic_predictions():
    x, y, coords = problem(900, 4, 21)
    g = degrees(coords, 5.0, 45.0, 10.0)
    rng = np.random.default_rng(22)
    near = np.column_stack([rng.uniform(5, 15, 140), rng.uniform(45, 50, 140)])
    far = np.concatenate([near[:20], [[-170.0, -40.0]]])  # outside the cap
    e, ref = engine(x, y, g, True), O.Problem(x, y, g, geographic=True)
    for at in (near, far):
        for kernel in (O.BISQUARE, O.GAUSSIAN):
            assert col_rel(e.predict(at, 90, True, kernel)[:20], ref.predict(at, 90, True, kernel)[:20]) <= 1e-10


@pytest.mark.gpu
@pytest.mark.parametrize("geographic", [False, True])
@pytest.mark.parametrize("kernel", [O.GAUSSIAN, O.BISQUARE])
def test_infinite_bandwidth(kernel, geographic):
    """Every pair has weight 1, in the first call on the data and in those after it: criteria, a fit with S and
    qDiag, predictions, then a finite bandwidth."""
    x, y, coords = problem(300, 3, 31)
    g = degrees(coords, 5.0, 45.0, 10.0) if geographic else coords
    e, ref = engine(x, y, g, geographic), O.Problem(x, y, g, geographic=geographic)
    inf = float("inf")
    for bw in (inf, inf, 900.0 if geographic else 120.0, inf):
        for crit in (O.AIC, O.CV):
            want, _ = ref.criterion(bw, False, kernel, crit)
            got = e.criterion(bw, False, kernel, crit)
            assert abs(got - want) <= 1e-9 * abs(want), (bw, crit, got, want)
        for store in (True, False):
            betas, se, shat, qdiag, S = e.fit(bw, False, kernel, store)
            rb, rse, rshat, rq, rS = ref.fit_core(bw, False, kernel, store)
            assert col_rel(betas, rb) <= 1e-10
            assert col_rel(se, rse) <= 1e-9
            np.testing.assert_allclose(shat, rshat, rtol=1e-9)
            np.testing.assert_allclose(qdiag, rq, rtol=1e-9)
            assert np.abs(S - rS).max() <= 1e-9 * np.abs(rS).max()
        assert col_rel(e.predict(g[:40] + 0.01, bw, False, kernel), ref.predict(g[:40] + 0.01, bw, False, kernel)) <= 1e-10


@pytest.mark.gpu
@pytest.mark.parametrize("n,p,geographic,kernel", [(3000, 9, True, O.GAUSSIAN), (3000, 5, False, O.GAUSSIAN),
                                                   (2000, 17, False, O.BISQUARE)])
def test_timeout_is_reported_and_engine_recovers(n, p, geographic, kernel):
    """With a limit of one poll the contraction's pipeline waits run out: the kernel waits for its own MMAs, commits
    and bulk copies, frees its tensor memory and sets the error flag; criterion, fit and prediction fail with that
    error, and the next call on the same engine returns the value it returned before."""
    from libgwmodel_gb300 import GwgpuError
    x, y, coords = problem(n, p, n + p)
    g = degrees(coords, 5.0, 45.0, 20.0) if geographic else coords
    e = engine(x, y, g, geographic)
    calls = [lambda: e.criterion(n // 2, True, kernel, O.AIC), lambda: e.criterion(n // 2, True, kernel, O.CV),
             lambda: e.fit(n // 2, True, kernel, False)[0], lambda: e.predict(g[:300], n // 2, True, kernel)]
    want = [f() for f in calls]
    for f, w in zip(calls, want):
        e.set_tc_wait_limit(1)
        with pytest.raises(GwgpuError, match="timed out"):
            f()
        e.set_tc_wait_limit(0)
        assert np.array_equal(f(), w)


@pytest.mark.gpu
@pytest.mark.parametrize("geographic", [False, True])
@pytest.mark.parametrize("n,kernel", [(129, O.BISQUARE), (129, O.GAUSSIAN), (701, O.BISQUARE), (701, O.GAUSSIAN)])
def test_hat_matrix_entries(n, kernel, geographic):
    """S whole, and its last row where it is not stored (fixed-point weights there): 1e-9 of the largest entry."""
    x, y, coords = problem(n, 4, n)
    g = degrees(coords, 5.0, 45.0, 10.0) if geographic else coords
    e, ref = engine(x, y, g, geographic), O.Problem(x, y, g, geographic=geographic)
    want = ref.fit_core(n // 2, True, kernel)
    for store in (True, False):
        got = e.fit(n // 2, True, kernel, store)
        S = want[4] if store else ref.fit_core(n // 2, True, kernel, False)[4]
        assert got[4].shape == S.shape
        assert np.abs(got[4] - S).max() <= 1e-9 * np.abs(S).max()
        np.testing.assert_allclose(got[3], want[3], rtol=1e-9)
