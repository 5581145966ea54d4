"""Launch groups of an ensemble: a member's E-phase threads are the ones asked for,
and only automatic counts are the batch's to choose."""

import numpy as np
import pytest

import cases as CS
from casebuild import build_product

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("first,groups", [(dict(e_threads=384, e_producer_warps=4), 2), (dict(), 1)], ids=["asked", "automatic"])
def test_asked_for_e_threads_are_kept(first, groups):
    from ionosphere_fdtd_b200 import Ensemble
    from ionosphere_fdtd_b200.engine import Tuning

    case = CS.CASES["plasma_drude_s2"]
    members = [build_product(case, "float32", tuning=Tuning(**t)) for t in (first, dict(e_threads=256, e_producer_warps=4))]
    alone = build_product(case, "float32", tuning=Tuning(staging=1))
    with Ensemble(members) as ens:
        assert ens.launch_layout()["groups"] == groups
        ens.step(35)
    alone.step(35)
    for m in members:
        for f in ("er", "et", "hr", "ht"):
            np.testing.assert_array_equal(m.to_numpy(getattr(m, f)), alone.to_numpy(getattr(alone, f)), err_msg=f)
