"""A served request gives the engine's own result bit for bit: how sums are split over the device follows from the
request's shape, not from what may be kept in memory."""
import numpy as np
import pytest

from libgwmodel_gb300 import Engine, Precision, datasets
from libgwmodel_gb300.serve import FIT, Server

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,p,bw,precision", [(2500, 17, 300.0, Precision.FP64), (4101, 4, 4000.0, Precision.Mixed),
                                              (9000, 9, 8000.0, Precision.Mixed)])
def test_served_fit_is_the_engines(n, p, bw, precision):
    pb = datasets._plain_problem(np.random.default_rng(n), n, p, False, "bits")
    srv = Server(0, hbm_budget_gb=40, slots=1)
    res, betas = srv.wait(srv.submit(pb, kind=FIT, bandwidth=bw, precision=precision))
    srv.close()
    e = Engine(0)
    e.set_data(pb.x, pb.y, pb.coords, pb.geographic)
    e.set_precision(precision)
    want, _, shat, _, _ = e.fit(bw, pb.adaptive, pb.kernel, store_s=False)
    assert res.status == 0
    assert np.array_equal(betas, want) and np.array_equal(list(res.shat), shat)


def test_the_splits_are_taken():
    """One more launch than with all tiles in one chunk, which leaves nothing to split."""
    pb = datasets._plain_problem(np.random.default_rng(1), 4101, 4, False, "splits")
    e = Engine(0)
    e.set_data(pb.x, pb.y, pb.coords, pb.geographic)
    e.set_precision(Precision.Mixed)

    def launches():
        e.criterion(4000.0, True, pb.kernel, 0)
        e.reset_stats()
        e.criterion(4000.0, True, pb.kernel, 0)
        return e.stats()["kernel_launches"]

    split = launches()
    e.set_flush_tiles(1 << 20)
    assert split == launches() + 1
