"""Knot and grid fields of several groups in one launch: profiles whose knots
fill a block's 125 intervals exactly, one less and one more, one to seventeen
frequencies (a block takes 8, the grid fields 16), different grids, several
azimuths, all in one batch.  Against the oracle (the tolerances of the other
parity tests) and, bit for bit, against each job alone."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps


def _subset(src, dst, n):
    """n of the profile's levels, first and last included"""
    with open(src) as f:
        lines = f.readlines()
    head = [x for x in lines if x.lstrip().startswith("#")]
    rows = [x for x in lines if x.strip() and not x.lstrip().startswith("#")]
    pick = np.unique(np.rint(np.linspace(0, len(rows) - 1, n)).astype(int))
    assert len(pick) == n
    with open(dst, "w") as f:
        f.writelines(head + [rows[i] for i in pick])
    return dst


@pytest.mark.parametrize("wide", [0, 1])
def test_groups_vs_alone_and_oracle(gpu, analytic_profile, workdir, wide):
    import ncpa_gpu
    from oracle import oracle as O

    sizes = [(125, 1, 3000, [75.0]), (126, 8, 3000, [75.0, 200.0]), (127, 9, 4096, [10.0]), (251, 17, 2500, [75.0]),
             (252, 2, 3001, [75.0, 100.0, 330.0])]
    jobs, paths = [], []
    for n, nf, nz, az in sizes:
        p = _subset(analytic_profile, os.path.join(str(workdir), "levels_%d.dat" % n), n)
        paths.append(p)
        jobs.append((gpu.load_profile(p), list(np.linspace(0.03, 0.1, nf)), az, nz))
    prm = ncpa_gpu.default_params(turnoff_wkb=1, method=ncpa_gpu.METHOD_WMOD if wide else 0)
    m = gpu.solve_jobs(jobs, prm)
    q = 0
    for (n, nf, nz, az), (prof, f, _, _), path in zip(sizes, jobs, paths):
        alone = gpu.solve_jobs([(prof, f, az, nz)], prm)
        for k in range(nf * len(az)):
            a, b = m.problem(q + k), alone.problem(k)
            assert a.M == b.M > 0
            for name in ("kr", "ki", "vs", "vr"):
                assert np.array_equal(getattr(a, name), getattr(b, name))
        k = nf * len(az) - 1  # the last frequency and azimuth
        op = O.EssParams(Nz_grid=nz, turnoff_WKB=True)
        solve = O.solve_problem_wmod if wide else O.solve_problem
        o = solve(O.prepare(O.read_profile(path), op), op, f[-1], az[-1])
        g = m.problem(q + k)
        assert g.M == o.M
        tol = np.maximum(1e-9, 8 * EPS * (4.0 / o.dz ** 2) / (2 * o.kr ** 2))
        assert np.all(np.abs(g.kr - o.kr) / o.kr <= tol)
        assert np.allclose(g.ki, o.ki, rtol=1e-6, atol=1e-18)
        assert np.allclose(g.vs * g.vr, o.vs * o.vr, rtol=1e-6, atol=1e-12 * np.abs(o.vs * o.vr).max())
        alone.close()
        q += nf * len(az)
    m.close()
    for prof, _, _, _ in jobs:
        prof.close()
