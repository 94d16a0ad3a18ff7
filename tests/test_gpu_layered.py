"""Finely layered winds at high frequency: blocks with two wells and a barrier
between them, whose levels come in pairs closer than a panel (see
test_panel_counts.py).  Counts identical to the oracle's, Re k within 1e-9
relative or the conditioning floor, as in the other parity tests."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps


@pytest.mark.parametrize("freq,nz,length,amp,wide", [(2.0, 20000, 500.0, 10.0, 0), (2.0, 20000, 500.0, 10.0, 1),
                                                     (2.0, 12000, 500.0, 10.0, 0), (4.0, 20000, 500.0, 10.0, 0)])
def test_layers_vs_oracle(gpu, freq, nz, length, amp, wide):
    import ncpa_gpu
    import workloads
    from oracle import oracle as O

    z, u, v, T, p, rho = workloads.perturbed_profile(np.random.default_rng([3, 5]))
    u = u + amp * np.sin(2 * np.pi * z / length + 5)
    prof = gpu.profile_from_arrays(z, u, v, T, p, rho)
    m = gpu.solve(prof, ncpa_gpu.default_params(nz_grid=nz, turnoff_wkb=1, max_modes=8000,
                                                method=ncpa_gpu.METHOD_WMOD if wide else 0), [freq], [70.0])
    g = m.problem(0)
    m.close()
    prof.close()
    prm = O.EssParams(Nz_grid=nz, turnoff_WKB=True)
    pp = O.prepare(O.Profile(z, "m", {"U": (u, "m/s"), "V": (v, "m/s"), "T": (T, "K"), "P": (p, "Pa"),
                                      "RHO": (rho, "kg/m3")}, {}), prm)
    o = O.solve_problem_wmod(pp, prm, freq, 70.0) if wide else O.solve_problem(pp, prm, freq, 70.0)
    assert g.M == o.M
    tol = np.maximum(1e-9, 8 * EPS * (4.0 / o.dz ** 2) / (2 * o.kr ** 2))
    assert np.all(np.abs(g.kr - o.kr) / o.kr <= tol)
