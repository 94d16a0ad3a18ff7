"""Modes that live between two of the rows (every 128th) where the chains of the
mode values are joined: short grids, grids of a few rows to a wavelength, wind
layers at high frequency.  Values without vectors, full vectors, ESS and wide
angle, items on panels and by rows.

Against the oracle, whose twist is chosen among all rows, for every mode: Re k
within 1e-9 relative or the conditioning floor, Im k and V_s V_r 1e-6 relative
(V_s V_r to 1e-12 of the largest), group speeds 1e-6, vectors 1e-6 of a mode's
largest value: the tolerances of the other parity tests."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps


def _oracle(arrays, nz, freq, az, wide, **kw):
    from oracle import oracle as O

    z, u, v, T, p, rho = arrays
    prm = O.EssParams(Nz_grid=nz, turnoff_WKB=True)
    pp = O.prepare(O.Profile(z, "m", {"U": (u, "m/s"), "V": (v, "m/s"), "T": (T, "K"), "P": (p, "Pa"),
                                      "RHO": (rho, "kg/m3")}, {}), prm)
    return O.solve_problem_wmod(pp, prm, freq, az) if wide else O.solve_problem(pp, prm, freq, az, **kw)


def _check(g, o):
    assert g.M == o.M > 0
    tol = np.maximum(1e-9, 8 * EPS * (4.0 / o.dz ** 2) / (2 * o.kr ** 2))
    assert np.all(np.abs(g.kr - o.kr) / o.kr <= tol)
    assert np.allclose(g.ki, o.ki, rtol=1e-6, atol=1e-18)
    assert np.allclose(g.vs * g.vr, o.vs * o.vr, rtol=1e-6, atol=1e-12 * np.abs(o.vs * o.vr).max())


@pytest.mark.parametrize("wide", [0, 1])
@pytest.mark.parametrize("freq,nz,n_az", [(0.03, 100, 2), (0.03, 127, 2), (0.03, 128, 2), (0.03, 129, 2), (0.04, 120, 2),
                                          (0.1, 150, 3), (0.1, 150, 600), (0.1, 300, 2), (0.5, 800, 60)])
def test_short_grids(gpu, wide, freq, nz, n_az):
    import ncpa_gpu
    import workloads

    arrays = workloads.si_arrays()
    az = list(np.linspace(0.0, 357.0, n_az))
    prof = gpu.profile_from_arrays(*arrays)
    m = gpu.solve(prof, ncpa_gpu.default_params(nz_grid=nz, turnoff_wkb=1, want_group_speed=1 - wide,
                                                method=ncpa_gpu.METHOD_WMOD if wide else 0), [freq], az)
    for a in (0, n_az // 2, n_az - 1):
        o = _oracle(arrays, nz, freq, az[a], wide, **({} if wide else dict(want_group=True)))
        g = m.problem(a)
        _check(g, o)
        if not wide:
            assert np.allclose(g.vg, o.vg, rtol=1e-6)
    m.close()
    prof.close()


@pytest.mark.parametrize("nz,freqs", [(300, [0.1, 0.15]), (129, [0.03, 0.05])])
def test_vectors(gpu, nz, freqs):
    import ncpa_gpu
    import workloads

    arrays = workloads.perturbed_profile(np.random.default_rng([3, 17]))
    prof = gpu.profile_from_arrays(*arrays)
    m = gpu.solve(prof, ncpa_gpu.default_params(nz_grid=nz, turnoff_wkb=1, want_vectors=1), freqs, [90.0])
    for p, f in enumerate(freqs):
        o = _oracle(arrays, nz, f, 90.0, 0, want_full=True)
        g, v = m.problem(p), m.vectors(p, nz)
        _check(g, o)
        top = np.abs(o.vfull).max(axis=0)
        sgn = np.sign((v * o.vfull).sum(axis=0))
        assert np.max(np.abs(v * sgn - o.vfull) / top) <= 1e-6
    m.close()
    prof.close()


def test_wind_layers(gpu):
    """layers of 1.3 km at 2 Hz: modes a few tens of rows wide on a grid of 10000"""
    import ncpa_gpu
    import workloads

    z, u, v, T, p, rho = workloads.perturbed_profile(np.random.default_rng([3, 5]))
    arrays = (z, u + 30.0 * np.sin(2 * np.pi * z / 1300.0 + 5), v, T, p, rho)
    prof = gpu.profile_from_arrays(*arrays)
    m = gpu.solve(prof, ncpa_gpu.default_params(nz_grid=10000, turnoff_wkb=1), [2.0], [70.0])
    _check(m.problem(0), _oracle(arrays, 10000, 2.0, 70.0, 0))
    m.close()
    prof.close()
