"""1-D transmission loss where its mode tiles end (64 modes) and where the
tiles get blocks of their own (few problems and ranges): one mode tile less and
more, one range, ranges around a block's 256, many ranges (no split).

Against an FP64 NumPy sum of the same modes: the phases k r reach 1e4 rad,
rounded to 1e-12 of a term by either side and by the powers' 2^6 ulps, so 1e-10
of the sum of the terms' magnitudes.  One problem alone and in a batch that
runs without the split agree bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PI = np.pi


@pytest.mark.parametrize("freq,nz", [(0.02, 2000), (0.1, 4000), (0.5, 8000)])
@pytest.mark.parametrize("nr,dr,lossless", [(1, 1000.0, False), (255, 1000.0, True), (256, 1000.0, False),
                                            (257, 1000.0, False), (1000, 500.0, False), (80000, 10.0, False)])
def test_tiles(gpu, analytic_profile, freq, nz, nr, dr, lossless):
    import ncpa_gpu

    prof = gpu.load_profile(analytic_profile)
    prm = ncpa_gpu.default_params(nz_grid=nz, turnoff_wkb=1)
    m = gpu.solve(prof, prm, [freq], [90.0])
    g = m.problem(0)
    re, im, inc = m.tl1d(nr, dr, lossless=lossless)
    k = g.kr + 1j * (0.0 if lossless else g.ki)
    r = (np.arange(nr) + 1) * dr
    P, S, I = np.zeros(nr, complex), np.zeros(nr), np.zeros(nr)
    for kk, v in zip(k, g.vs * g.vr):
        t = v * np.exp(1j * kk * r) / np.sqrt(kk)
        P += t
        S += np.abs(t)
        I += np.abs(t) ** 2
    C = 1000.0 * 4 * PI * 1j * np.exp(-1j * PI / 4) / np.sqrt(8 * PI * r)
    assert np.max(np.abs(re[0] + 1j * im[0] - C * P) / (np.abs(C) * S)) < 1e-10
    assert np.allclose(inc[0], np.abs(C) * np.sqrt(I), rtol=1e-10)
    if nr == 1000:  # enough problems for a launch without the split
        b = gpu.solve(prof, prm, [freq], list(np.linspace(0.0, 350.0, 79)) + [90.0])
        out = b.tl1d(nr, dr, lossless=lossless)
        for x, y in zip(out, (re, im, inc)):
            assert np.array_equal(x[79], y[0])
        b.close()
    m.close()
    prof.close()
