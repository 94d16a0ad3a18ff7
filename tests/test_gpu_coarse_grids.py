"""Grids so coarse against the wavelength that the work items sweep the rows as
they are: few items (teams of four warps), many (a warp each) and a mix with
items on panels, in one batch of azimuths.  Every value is finite, counts are
the oracle's, and a problem of the batch has the values it has alone, bit for
bit (without the scan's trim, which changes brackets)."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def untrimmed():
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
@pytest.mark.parametrize("freq,nz,n_az", [(0.1, 150, 3), (0.1, 150, 600), (0.5, 800, 90), (1.0, 2500, 60),
                                          (0.5, 4100, 3)])
def test_coarse_grids(untrimmed, analytic_profile, wide, group, freq, nz, n_az):
    import ncpa_gpu
    from oracle import oracle as O

    gpu = untrimmed
    az = list(np.linspace(0.0, 357.0, n_az))
    prof = gpu.load_profile(analytic_profile)
    par = ncpa_gpu.default_params(nz_grid=nz, turnoff_wkb=1, want_group_speed=group,
                                  method=ncpa_gpu.METHOD_WMOD if wide else 0)
    m = gpu.solve(prof, par, [freq], az)
    for v in m.all_modes()[1:]:
        assert np.all(np.isfinite(v))
    prm = O.EssParams(Nz_grid=nz, turnoff_WKB=True)
    pp = O.prepare(O.read_profile(analytic_profile), prm)
    for a in (0, n_az // 2, n_az - 1):
        o = O.solve_problem_wmod(pp, prm, freq, az[a]) if wide else O.solve_problem(pp, prm, freq, az[a])
        alone = gpu.solve(prof, par, [freq], [az[a]])
        g, h = m.problem(a), alone.problem(0)
        assert g.M == h.M == o.M > 0
        for name in ("kr", "ki", "vs", "vr", "vg"):
            assert np.array_equal(getattr(g, name), getattr(h, name))
        alone.close()
    m.close()
    prof.close()
