"""The eigen-solve on panel expansions (panel.cu) against the oracle where its
blocks, chunks and panels end: grids of less than a block, one row around a
block and around a chunk of four blocks, grids so coarse against the
wavelength that the blocks are short or the rows are swept as they are, and
source and receiver rows inside a block.

Tolerances are those of the other parity tests: counts identical, Re k within
1e-9 relative or the conditioning floor, Im k, V_s V_r and group speeds 1e-6
relative."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps


@pytest.mark.parametrize("freq,nz,zs,zr", [
    (0.004, 12, 0.0, 0.0), (0.02, 100, 0.0, 0.0),                       # less than a block
    (0.03, 127, 0.0, 0.0), (0.03, 128, 0.0, 0.0), (0.03, 129, 0.0, 0.0),  # around a block
    (0.05, 511, 0.0, 0.0), (0.05, 512, 0.0, 0.0), (0.05, 513, 12.3, 4.1),  # around a chunk
    (0.25, 4097, 3.21, 20.7),                                          # rows inside blocks
    (1.0, 3001, 0.0, 0.0), (2.0, 6007, 0.0, 1.0),                      # short blocks
    (0.04, 120, 0.0, 0.0),                                             # raw rows
])
def test_grid_edges_vs_oracle(gpu, analytic_profile, freq, nz, zs, zr):
    import ncpa_gpu
    from oracle import oracle as O

    prm = O.EssParams(Nz_grid=nz, turnoff_WKB=True, sourceheight_km=zs, receiverheight_km=zr)
    o = O.solve_problem(O.prepare(O.read_profile(analytic_profile), prm), prm, freq, 75.0, want_group=True)
    prof = gpu.load_profile(analytic_profile)
    m = gpu.solve(prof, ncpa_gpu.default_params(nz_grid=nz, turnoff_wkb=1, want_group_speed=1, sourceheight_km=zs,
                                                receiverheight_km=zr), [freq], [75.0])
    g = m.problem(0)
    m.close()
    prof.close()
    assert g.M == o.M and g.M > 0
    tol = np.maximum(1e-9, 8 * EPS * (4.0 / o.dz ** 2) / (2 * o.kr ** 2))
    assert np.all(np.abs(g.kr - o.kr) / o.kr <= tol)
    # the twist is chosen among every 128th row: on one such row alone (the
    # ground) only vectors that reach it are resolved
    big = np.abs(o.vs * o.vr).max()
    sel = np.abs(o.vs * o.vr) >= (1e-3 * big if nz <= 129 else 0.0)
    assert np.allclose(g.ki[sel], o.ki[sel], rtol=1e-6, atol=1e-18)
    assert np.allclose((g.vs * g.vr)[sel], (o.vs * o.vr)[sel], rtol=1e-6, atol=1e-12 * big)
    assert np.allclose(g.vg[sel], o.vg[sel], rtol=1e-6)
