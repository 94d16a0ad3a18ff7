"""Windows so narrow (a wavenumber filter, or a low column whose fastest layers
are close to its slowest) that their panels are wide in rows, at frequencies
where a chain grows or decays by many orders within a chunk of blocks.

Against the oracle: counts identical, Re k within 1e-9 relative or the
conditioning floor, Im k and V_s V_r 1e-6 relative (V_s V_r to 1e-12 of the
largest), as in the other parity tests."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps


def _check(gpu, arrays, freq, nz, wide, c=None, top=None):
    import ncpa_gpu
    from oracle import oracle as O

    z, u, v, T, p, rho = arrays
    kw = dict(wvnum_filter=1, c_min=c[0], c_max=c[1]) if c else {}
    if top:
        kw["maxheight_km"] = top
    prof = gpu.profile_from_arrays(*arrays)
    m = gpu.solve(prof, ncpa_gpu.default_params(nz_grid=nz, turnoff_wkb=1, max_modes=20000,
                                                method=ncpa_gpu.METHOD_WMOD if wide else 0, **kw), [freq], [90.0])
    g = m.problem(0)
    m.close()
    prof.close()
    prm = O.EssParams(Nz_grid=nz, turnoff_WKB=True, wvnum_filter=c is not None, c_min=c[0] if c else 0.0,
                      c_max=c[1] if c else 0.0, maxheight_km=top or 150.0)
    pp = O.prepare(O.Profile(z, "m", {"U": (u, "m/s"), "V": (v, "m/s"), "T": (T, "K"), "P": (p, "Pa"),
                                      "RHO": (rho, "kg/m3")}, {}), prm)
    o = O.solve_problem_wmod(pp, prm, freq, 90.0) if wide else O.solve_problem(pp, prm, freq, 90.0)
    assert g.M == o.M
    if o.M == 0:
        return 0
    tol = np.maximum(1e-9, 8 * EPS * (4.0 / o.dz ** 2) / (2 * o.kr ** 2))
    assert np.all(np.abs(g.kr - o.kr) / o.kr <= tol)
    assert np.allclose(g.ki, o.ki, rtol=1e-6, atol=1e-18)
    assert np.allclose(g.vs * g.vr, o.vs * o.vr, rtol=1e-6, atol=1e-12 * np.abs(o.vs * o.vr).max())
    return o.M


@pytest.mark.parametrize("wide", [0, 1])
@pytest.mark.parametrize("nz", [5000, 5417, 6000])
def test_filters_2hz(gpu, wide, nz):
    import workloads

    arrays = workloads.perturbed_profile(np.random.default_rng([3, 977]))
    rng = np.random.default_rng(nz)
    found = _check(gpu, arrays, 2.0, nz, wide, (330.0, 330.1)) + _check(gpu, arrays, 2.0, nz, wide, (331.3, 331.4))
    for width in (0.05, 0.1, 0.2, 0.5, 1.0, 2.0):
        for c in rng.uniform(300.0, 345.0, 4):
            found += _check(gpu, arrays, 2.0, nz, wide, (c, c + width))
    assert found > 20


@pytest.mark.parametrize("wide", [0, 1])
def test_filters_8hz(gpu, wide):
    import workloads

    arrays = workloads.perturbed_profile(np.random.default_rng([3, 978]))
    assert _check(gpu, arrays, 8.0, 20000, wide, (320.0, 320.1)) + _check(gpu, arrays, 8.0, 20000, wide, (309.0, 309.4)) > 0


@pytest.mark.parametrize("wide", [0, 1])
@pytest.mark.parametrize("freq,nz", [(2.0, 5000), (8.0, 20000)])
def test_low_column(gpu, wide, freq, nz):
    import workloads

    arrays = workloads.perturbed_profile(np.random.default_rng([3, 13]))
    assert _check(gpu, arrays, freq, nz, wide, top=95.0) > 0
