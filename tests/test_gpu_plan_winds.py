"""A plan whose profile's winds grow between replays far beyond those that its
records were sized for: items without panels, which the graph was captured
without.  Counts identical to the oracle's, Re k within 1e-9 relative or the
conditioning floor, Im k, V_s V_r and TL of a fresh solve as in the other parity
tests (a fresh solve has other records, so not bit for bit)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps


def atmosphere():
    import workloads

    return workloads.perturbed_profile(np.random.default_rng([3, 11]))


def oracle(arrays, nz, freq, az):
    from oracle import oracle as O

    z, u, v, T, p, rho = arrays
    prm = O.EssParams(Nz_grid=nz, turnoff_WKB=True)
    pp = O.prepare(O.Profile(z, "m", {"U": (u, "m/s"), "V": (v, "m/s"), "T": (T, "K"), "P": (p, "Pa"),
                                      "RHO": (rho, "kg/m3")}, {}), prm)
    return O.solve_problem(pp, prm, freq, az)


def same(g, o):
    assert g.M == o.M > 0
    tol = np.maximum(1e-9, 8 * EPS * (4.0 / o.dz ** 2) / (2 * o.kr ** 2))
    assert np.all(np.abs(g.kr - o.kr) / o.kr <= tol)


@pytest.mark.parametrize("tune", [False, True])
@pytest.mark.parametrize("freq,nz", [(0.5, 1000), (0.5, 3000)])
def test_plan_after_a_change_of_winds(gpu, freq, nz, tune):
    import ncpa_gpu

    full = atmosphere()
    z, u, v, T, p, rho = full
    calm = (z, 0 * u, 0 * v, np.full_like(T, 300.0), 1.2 * 300.0 * 287.0 * np.exp(-z / 8000.0), 1.2 * np.exp(-z / 8000.0))
    prof = gpu.profile_from_arrays(*calm)
    prm = ncpa_gpu.default_params(nz_grid=nz, turnoff_wkb=1)
    with gpu.plan([(prof, [freq], 70.0)], prm, tl=(50, 1000.0), tune=tune) as plan:
        plan.run()
        prof.update(*full)
        for _ in range(2):
            plan.run()
            g = plan.modes().problem(0)
            same(g, oracle(full, nz, freq, 70.0))
            tl = plan.tl()
        m = gpu.solve(prof, prm, [freq], [70.0])
        h = m.problem(0)
        assert np.allclose(g.ki, h.ki, rtol=1e-6, atol=1e-18)
        assert np.allclose(g.vs * g.vr, h.vs * h.vr, rtol=1e-6, atol=1e-12 * np.abs(h.vs * h.vr).max())
        for a, b in zip(tl, m.tl1d(50, 1000.0)):
            assert np.abs(a - b).max() <= 1e-6 * np.abs(b).max()
        m.close()
    prof.close()
