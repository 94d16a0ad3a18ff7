"""The wide-angle eigen-solve on panel expansions against the oracle where its
blocks, chunks and panels end: one row around two and four blocks, short
blocks, rows inside a block, and the full vectors.

Tolerances are those of the other wide-angle tests (counts identical, Re k
within 1e-9 relative or the conditioning floor, Im k and V_s V_r 1e-6
relative), full vectors 1e-6 of a mode's largest value."""
import numpy as np
import pytest

from test_gpu_wmod import _check_modes, _wmod

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("freq,nz,zs,zr", [
    (0.03, 255, 0.0, 0.0), (0.03, 256, 0.0, 0.0), (0.03, 257, 0.0, 0.0), (0.05, 511, 0.0, 0.0),
    (0.05, 513, 12.3, 4.1), (0.25, 4097, 3.21, 20.7), (1.0, 3001, 0.0, 0.0), (0.01, 6000, 0.0, 0.0)])
def test_grid_edges_vs_oracle(gpu, analytic_profile, freq, nz, zs, zr):
    from oracle import oracle as O

    prm = O.EssParams(Nz_grid=nz, turnoff_WKB=True, sourceheight_km=zs, receiverheight_km=zr)
    o = O.solve_problem_wmod(O.prepare(O.read_profile(analytic_profile), prm), prm, freq, 75.0, want_full=True)
    prof = gpu.load_profile(analytic_profile)
    kw = dict(nz_grid=nz, turnoff_wkb=1, sourceheight_km=zs, receiverheight_km=zr)
    m = gpu.solve(prof, _wmod(**kw), [freq], [75.0])
    g = m.problem(0)
    assert o.M > 0
    _check_modes(g, o)
    mv = gpu.solve(prof, _wmod(want_vectors=1, **kw), [freq], [75.0])
    _check_modes(mv.problem(0), o)
    v = mv.vectors(0, nz)
    top = np.abs(o.vfull).max(axis=0)
    assert np.all(v[np.abs(v).argmax(axis=0), np.arange(o.M)] > 0)
    sgn = np.sign((v * o.vfull).sum(axis=0))
    assert np.max(np.abs(v * sgn - o.vfull) / top) <= 1e-6
    for x in (m, mv, prof):
        x.close()
