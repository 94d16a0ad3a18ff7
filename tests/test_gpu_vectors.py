"""The mode functions at every row (want_vectors) where the chunks they are
filled in end: less than a chunk of 128 rows, one row around a chunk and around
a coarser block, rows swept as they are, several problems of one solve with
different mode counts.

Against the oracle's vectors: 1e-6 of a mode's largest value, the tolerance of
the mode values in the other parity tests.  A mode is positive where it is
largest; the values at the source and receiver rows are those of vs and vr to
1e-9 of the largest (computed from another block's end)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("freqs,nz,zs,zr", [
    ([0.02, 0.01], 100, 0.0, 0.0), ([0.03], 127, 0.0, 0.0), ([0.03], 128, 1.2, 30.0), ([0.03], 129, 0.0, 0.0),
    ([0.05, 0.03], 257, 20.0, 5.0), ([0.05], 513, 12.3, 4.1), ([0.25, 0.1, 0.01], 4097, 3.21, 20.7),
    ([0.04], 120, 0.0, 0.0), ([2.0], 6007, 0.0, 1.0)])
def test_vectors_vs_oracle(gpu, analytic_profile, freqs, nz, zs, zr):
    import ncpa_gpu
    from oracle import oracle as O

    oprm = O.EssParams(Nz_grid=nz, turnoff_WKB=True, sourceheight_km=zs, receiverheight_km=zr)
    prof = gpu.load_profile(analytic_profile)
    m = gpu.solve(prof, ncpa_gpu.default_params(nz_grid=nz, turnoff_wkb=1, want_vectors=1, sourceheight_km=zs,
                                                receiverheight_km=zr), freqs, [75.0, 200.0])
    for p in range(2 * len(freqs)):
        f, az = freqs[p // 2], [75.0, 200.0][p % 2]
        o = O.solve_problem(O.prepare(O.read_profile(analytic_profile), oprm), oprm, f, az, want_full=True)
        g, v = m.problem(p), m.vectors(p, nz)
        assert g.M == o.M and v.shape == (nz, o.M) == o.vfull.shape
        if o.M == 0:
            continue
        top = np.abs(o.vfull).max(axis=0)
        at = np.abs(v).argmax(axis=0)
        assert np.all(v[at, np.arange(o.M)] > 0)
        sgn = np.sign((v * o.vfull).sum(axis=0))
        assert np.max(np.abs(v * sgn - o.vfull) / top) <= 1e-6
        i_s, i_r = int(np.ceil(zs * 1000.0 / g.dz)), int(np.ceil(zr * 1000.0 / g.dz))
        assert np.max(np.abs(v[i_s] - g.vs) / top) <= 1e-9
        assert np.max(np.abs(v[i_r] - g.vr) / top) <= 1e-9
    m.close()
    prof.close()
