"""The refinement of the mixed form: residuals from the fixed-point sums of the FP32 weights, and from the
double-float pass for rows where a column rests on weights near 2^-62, at the mixed form's bar against FP64
(coefficients 1e-6 relative)."""
import numpy as np
import pytest

import oracle as O
from libgwmodel_gb300 import Engine, Precision
from parity_util import col_rel

pytestmark = pytest.mark.gpu


def fit_both(x, y, c, geographic, bw, adaptive, kernel):
    out = []
    for precision in (Precision.FP64, Precision.Mixed):
        e = Engine(0)
        e.set_data(x, y, c, geographic)
        e.set_precision(precision)
        out.append(e.fit(bw, adaptive, kernel, False)[0])
    return out


def points(n, seed, geographic):
    rng = np.random.default_rng(seed)
    c = rng.uniform(0, 100, (n, 2))
    return rng, c, np.column_stack([c[:, 0] / 10, 40 + c[:, 1] / 10]) if geographic else c


@pytest.mark.parametrize("geographic", [False, True])
@pytest.mark.parametrize("kernel", [O.GAUSSIAN, O.EXPONENTIAL, O.BISQUARE, O.TRICUBE, O.BOXCAR])
@pytest.mark.parametrize("n", [127, 1030])
def test_every_kernel(kernel, geographic, n):
    rng, _, c = points(n, n, geographic)
    x = np.asfortranarray(np.column_stack([np.ones(n), rng.standard_normal((n, 3))]))
    y = x.sum(1) + rng.normal(0, 0.3, n)
    bw, adaptive = n // 2, True
    if kernel == O.BOXCAR:
        # the step at an adaptive threshold, the distance of a point, is FP32's to decide: a fixed
        # bandwidth in the widest gap between the pairs' distances instead
        ref = O.Problem(x, y, c, geographic=geographic)
        d = np.sort(np.concatenate([ref.distance_row(i) for i in range(n)]))
        d = d[(d > np.quantile(d, 0.4)) & (d < np.quantile(d, 0.42))]
        i = np.argmax(np.diff(d))
        bw, adaptive = 0.5 * (d[i] + d[i + 1]), False
    b64, bmx = fit_both(x, y, c, geographic, bw, adaptive, kernel)
    assert col_rel(bmx, b64) <= 1e-6


@pytest.mark.parametrize("geographic", [False, True])
@pytest.mark.parametrize("kernel,bw", [(O.GAUSSIAN, 9.0), (O.GAUSSIAN, 12.0), (O.EXPONENTIAL, 2.0)])
def test_indicator_without_an_intercept(kernel, bw, geographic):
    """Nothing is centred, so the indicator's sums rest on weights down to 1e-21 far from its region."""
    n = 600
    rng, c, at = points(n, 2, geographic)
    x = np.asfortranarray(np.column_stack([1.0 + 0.3 * rng.standard_normal(n), c[:, 0] > 80]))
    y = x @ [1.0, 3.0] + rng.normal(0, 0.3, n)
    b64, bmx = fit_both(x, y, at, geographic, bw * (10.0 if geographic else 1.0), False, kernel)
    assert col_rel(bmx, b64) <= 1e-6
