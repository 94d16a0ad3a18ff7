"""A broadband batch of more than a thousand scan units on a context as it is
created: the modes of every eighth problem are those of the problem solved
alone, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nz", [5000, 2500])
def test_broadband_problems_as_alone(gpu, analytic_profile, nz):
    import ncpa_gpu
    import workloads

    prof = gpu.load_profile(analytic_profile)
    prm = ncpa_gpu.default_params(nz_grid=nz, turnoff_wkb=1)
    freqs = workloads.broadband_freqs(256, 0.5)
    m = gpu.solve(prof, prm, freqs, [90.0])
    for i in range(7, 256, 8):
        alone = gpu.solve(prof, prm, [freqs[i]], [90.0])
        x, y = m.problem(i), alone.problem(0)
        assert x.M == y.M > 0
        for name in ("kr", "ki", "vs", "vr"):
            assert np.array_equal(getattr(x, name), getattr(y, name))
        alone.close()
    m.close()
    prof.close()
