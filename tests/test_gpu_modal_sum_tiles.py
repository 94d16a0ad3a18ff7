"""The FP64 modal sum where its tiles end: heights around the 64 of a block,
ranges around its 16, 24 or 32 and around the 32 tiles of a coarse phase, mode
counts that are no multiple of a step, both layouts, with and without loss.

Against an FP64 NumPy sum of the same modes.  The phase k r reaches 40 rad
per km x 2000 km of ranges at most, 1e4 to 1e5 rad, whose rounding is 1e-11
of a term on either side: 1e-10 of the terms' magnitude, as for the sum's
other tests."""
import numpy as np
import pytest

from test_gpu_modal_sum import _ref_sum

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[(0.05, 1500), (0.5, 8000)])
def solved(gpu, analytic_profile, request):
    import ncpa_gpu

    freq, nz = request.param
    prof = gpu.load_profile(analytic_profile)
    m = gpu.solve(prof, ncpa_gpu.default_params(nz_grid=nz, want_vectors=1, turnoff_wkb=1), [freq], [90.0])
    yield m, m.problem(0), m.vectors(0, nz), nz
    m.close()
    prof.close()


@pytest.mark.parametrize("n_rcv,n_ranges,dr,lossless", [
    (1, 1, 1000.0, False), (63, 15, 1000.0, False), (64, 16, 1000.0, True), (65, 17, 1000.0, False),
    (129, 33, 1000.0, False), (7, 511, 500.0, True), (7, 512, 500.0, False), (7, 513, 500.0, False),
    (64, 8000, 100.0, False), (64, 14209, 100.0, False), (64, 20000, 100.0, True), (1024, 50, 1000.0, False)])
def test_receiver_sum_tiles(solved, n_rcv, n_ranges, dr, lossless):
    m, g, v, nz = solved
    h = np.arange(n_rcv) * (nz // 2) // n_rcv * g.dz
    idx = np.ceil(h / g.dz).astype(int)  # the grid row at or above a receiver
    P, S = _ref_sum(g.kr, g.ki, g.vs, v[idx, :], n_ranges, dr, lossless)
    p = m.tl_multi(0, h, n_ranges, dr, method=m.SUM_FP64, lossless=lossless)
    assert np.max(np.abs(p - P) / S) < 1e-10


@pytest.mark.parametrize("n_ranges,dr", [(1, 1000.0), (31, 1000.0), (65, 2000.0), (1025, 500.0)])
def test_2d_sum_tiles(solved, n_ranges, dr):
    m, g, v, nz = solved
    z, re, im = m.tl2d(0, n_ranges, dr)
    idx = np.rint(z / g.dz).astype(int)
    P, S = _ref_sum(g.kr, g.ki, g.vs, v[idx, :], n_ranges, dr)
    assert re.shape == (n_ranges, len(z))
    assert np.max(np.abs(re + 1j * im - P.T) / S.T) < 1e-10
