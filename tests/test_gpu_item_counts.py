"""A problem alone (its work items on teams of four warps), among some hundred
and among some thousand (eigenvalues on teams, then on pairs): the launches
differ by the number of items, the values do not, bit for bit.  (The scan is
not trimmed here: with 594 units on 592 schedulers the trim drops the last
unit of the first two problems, whose eigenvalues then settle from other
brackets.)"""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def untrimmed(gpu):
    import ncpa_gpu

    old = os.environ.get("NCPA_SCAN_TRIM")
    os.environ["NCPA_SCAN_TRIM"] = "0"
    try:
        ctx = ncpa_gpu.Context(0)
    finally:
        if old is None:
            del os.environ["NCPA_SCAN_TRIM"]
        else:
            os.environ["NCPA_SCAN_TRIM"] = old
    yield ctx
    ctx.close()


@pytest.mark.parametrize("wide,group", [(0, 0), (0, 1), (1, 0)])
@pytest.mark.parametrize("n_f,n_az,nz", [(1, 296, 700), (1, 297, 700), (8, 80, 700), (48, 75, 500)])
def test_values_do_not_depend_on_the_batch(untrimmed, analytic_profile, wide, group, n_f, n_az, nz):
    import ncpa_gpu

    gpu = untrimmed
    prof = gpu.load_profile(analytic_profile)
    prm = ncpa_gpu.default_params(nz_grid=nz, turnoff_wkb=1, want_group_speed=group,
                                  method=ncpa_gpu.METHOD_WMOD if wide else 0)
    freqs = list(np.linspace(0.02, 0.06, n_f)) if n_f > 1 else [0.05]
    az = list(np.linspace(0.0, 359.0, n_az))
    m = gpu.solve(prof, prm, freqs, az)
    for f, a in ((0, 0), (n_f - 1, n_az - 1), (n_f // 2, n_az // 3)):
        alone = gpu.solve(prof, prm, [freqs[f]], [az[a]])
        x, y = m.problem(f * n_az + a), alone.problem(0)
        assert x.M == y.M > 0
        for name in ("kr", "ki", "vs", "vr", "vg"):
            assert np.array_equal(getattr(x, name), getattr(y, name))
        alone.close()
    m.close()
    prof.close()
