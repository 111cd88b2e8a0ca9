"""Covariates that are zero near a location: the sums of such a column rest on small weights.

Fixed-point weights have an absolute unit (2^-62), FP64 weights keep their bits down to 1e-300, so rows where a
column of X has only far support must take FP64 sums: criteria, fits and predictions against the oracle at the
drop-in's bars (criteria and standard errors 1e-9, coefficients 1e-10 relative)."""
import numpy as np
import pytest

import oracle as O
from libgwmodel_gb300 import Engine
from parity_util import col_rel, rel
from test_gpu_mgwr import assert_parity, build

pytestmark = pytest.mark.gpu


def problem(n, seed, geographic, edge=80.0):
    """X = (1, normal, indicator of the eastern edge), on [0, 100]^2 or 10 x 10 degrees."""
    rng = np.random.default_rng(seed)
    c = rng.uniform(0, 100, (n, 2))
    x = np.asfortranarray(np.column_stack([np.ones(n), rng.standard_normal(n), c[:, 0] > edge]))
    y = x @ [1.0, 1.0, 3.0] + rng.normal(0, 0.3, n)
    if geographic:
        c = np.column_stack([c[:, 0] / 10, 40 + c[:, 1] / 10])
    return x, y, np.asfortranarray(c)


def engine(x, y, c, geographic):
    e = Engine(0)
    e.set_data(x, y, c, geographic)
    return e


def check(e, ref, bw, adaptive, kernel, at=None):
    for repeat in range(2):  # the first call on new data takes a route of its own
        for crit in (O.AIC, O.CV):
            want = ref.criterion(bw, adaptive, kernel, crit)[0]
            got = e.criterion(bw, adaptive, kernel, crit)
            assert abs(got - want) <= 1e-9 * abs(want), (bw, kernel, crit, repeat, got, want)
    betas, se, shat = e.fit(bw, adaptive, kernel)[:3]
    rb, rse, rshat = ref.fit_core(bw, adaptive, kernel)[:3]
    assert col_rel(betas, rb) <= 1e-10, (bw, kernel)
    assert col_rel(se, rse) <= 1e-9, (bw, kernel)
    assert rel(shat, rshat) <= 1e-9, (bw, kernel)
    if at is not None:
        assert col_rel(e.predict(at, bw, adaptive, kernel), ref.predict(at, bw, adaptive, kernel)) <= 1e-10


@pytest.mark.parametrize("geographic", [False, True])
@pytest.mark.parametrize("bw,adaptive", [(6.0, False), (8.0, False), (10.0, False), (15.0, False), (20, True)])
def test_indicator_far_from_most_rows(bw, adaptive, geographic):
    n = 600
    x, y, c = problem(n, 1, geographic)
    e, ref = engine(x, y, c, geographic), O.Problem(x, y, c, geographic=geographic)
    at = c[::7] + 0.01
    # 10 degrees of longitude at 45 degrees: 8 to 11 km a unit
    check(e, ref, bw * (10.0 if geographic and not adaptive else 1.0), adaptive, O.GAUSSIAN, at)


@pytest.mark.parametrize("geographic", [False, True])
def test_bisquare_rows_that_reach_the_region_with_their_rim(geographic):
    """The smallest bandwidth at which every row reaches the indicator's points, 0.2% beyond: weights of 1e-5 and
    squares of 1e-10 carry the column in the farthest rows."""
    n = 1500
    x, y, c = problem(n, 2, geographic)
    e, ref = engine(x, y, c, geographic), O.Problem(x, y, c, geographic=geographic)
    bw = 1.002 * max(ref.distance_row(i)[x[:, 2] > 0].min() for i in range(n))
    check(e, ref, bw, False, O.BISQUARE)


@pytest.mark.parametrize("n,p,bw", [(3001, 3, 12.0), (1100, 1, 3.0), (2049, 11, 16.0)])
def test_some_blocks_of_many(n, p, bw):
    """Marked blocks are recomputed from a list, their tiles split: partial blocks and tiles, column counts of the
    narrow form (p = 1: an uncentred column alone) and of several groups, rows marked in one region only."""
    x, y, c = problem(n, 7, False)
    rng = np.random.default_rng(p)
    if p == 1:  # small where it is not 1, so that no system is singular
        x = np.asfortranarray(np.where(x[:, 2:] > 0, 1.0, 1e-2 * (1.0 + rng.random((n, 1)))))
        y = x[:, 0] + rng.normal(0, 0.1, n)
    else:
        x = np.asfortranarray(np.column_stack([x, rng.standard_normal((n, p - 3))]))
    check(engine(x, y, c, False), O.Problem(x, y, c), bw, False, O.GAUSSIAN, c[::11] + 0.01)


@pytest.mark.parametrize("p", [11, 24])
def test_indicator_among_many_columns(p):
    """Column groups after the first and the warp form of the solve (p > 20)."""
    n = 700
    x, y, c = problem(n, 3, False)
    rng = np.random.default_rng(p)
    x = np.asfortranarray(np.column_stack([x, rng.standard_normal((n, p - 3))]))
    check(engine(x, y, c, False), O.Problem(x, y, c), 9.0 if p == 11 else 14.0, False, O.GAUSSIAN)


@pytest.mark.parametrize("geographic", [False, True])
@pytest.mark.parametrize("kernel,bw,store", [(O.GAUSSIAN, 6.0, False), (O.GAUSSIAN, 9.0, False), (O.BISQUARE, None, True)])
def test_hat_matrix_of_an_indicator(kernel, bw, store, geographic):
    """s_ij = w_ij v_i . x_j with v_i = A_i^-1 x_i as large as the column's weights are small: qDiag and S."""
    n = 600
    x, y, c = problem(n, 4, geographic)
    e, ref = engine(x, y, c, geographic), O.Problem(x, y, c, geographic=geographic)
    bw = bw * (10.0 if geographic else 1.0) if bw else 1.002 * max(ref.distance_row(i)[x[:, 2] > 0].min() for i in range(n))
    want = ref.fit_core(bw, False, kernel, True)
    for repeat in range(2):
        got = e.fit(bw, False, kernel, store)
        np.testing.assert_allclose(got[3], want[3], rtol=1e-9)
        if store:
            assert np.abs(got[4] - want[4]).max() <= 1e-9 * np.abs(want[4]).max()


@pytest.mark.parametrize("elsewhere", [0.0, 0.1])
@pytest.mark.parametrize("geographic", [False, True])
def test_multiscale_with_a_sparse_uncentred_column(elsewhere, geographic):
    """One-variable systems of a column that is 0, or small, away from its region: coefficients, and the traces of
    the hat matrix that its updates leave."""
    n = 400
    x, y, c = problem(n, 6, geographic)
    rng = np.random.default_rng(8)
    x = np.asfortranarray(np.column_stack([np.ones(n), np.where(x[:, 2] > 0, 1.0, elsewhere * rng.standard_normal(n))]))
    y = x @ [1.0, 3.0] + rng.normal(0, 0.3, n)
    unit = 10.0 if geographic else 1.0
    bw0 = [30.0 * unit, 7.0 * unit]
    kw = dict(adaptive=[0, 0], kernel=[O.GAUSSIAN] * 2, centered=[0, 0])
    # init Specified, approach AIC; the first variable's weight also spans the search of the initial fit
    ref = O.Problem(x, y, c, geographic=geographic).mgwr(bw0=bw0, init_type=[2, 2], approach=[1, 1], select_threshold=[1e-5] * 2,
                                                         max_iteration=4, lower=20.0 * unit, upper=60.0 * unit, **kw)
    alg = build(x, y, c, bw0=bw0, init=[2, 2], approach=[1, 1], geographic=geographic, max_iteration=4,
                lower=20.0 * unit, upper=60.0 * unit, **kw)
    alg.fit()
    assert_parity(alg, ref, capped=4)
