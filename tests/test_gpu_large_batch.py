"""A batch whose panel expansions exceed 32 GB is solved in parts: the device
memory that a context takes stays bounded, and every problem's modes are those
of the problem solved alone, bit for bit, on both sides of the cuts."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("group,n_az", [(0, 1700), (1, 1200)])
def test_large_batch_in_parts(analytic_profile, group, n_az):
    import torch
    import ncpa_gpu

    torch.cuda.init()
    with ncpa_gpu.Context(0) as ctx:
        prof = ctx.load_profile(analytic_profile)
        prm = ncpa_gpu.default_params(nz_grid=20000, turnoff_wkb=1, max_modes=2000, want_group_speed=group)
        az = np.linspace(0.0, 359.0, n_az)
        alone = {i: ctx.solve(prof, prm, [2.0], [az[i]]) for i in (0, 1, n_az // 3, n_az // 2, 2 * n_az // 3, n_az - 2, n_az - 1)}
        ctx.synchronize()
        free = torch.cuda.mem_get_info(0)[0]
        m = ctx.solve(prof, prm, [2.0], az)
        taken = free - torch.cuda.mem_get_info(0)[0]
        off, kr, ki, vs, vr, vg = m.all_modes()
        assert off[-1] > 900 * n_az
        for i, a in alone.items():
            g = a.problem(0)
            for x, y in zip((kr, ki, vs, vr, vg), (g.kr, g.ki, g.vs, g.vr, g.vg)):
                assert np.array_equal(x[off[i]:off[i + 1]], y)
            a.close()
        m.close()
        prof.close()
    assert taken < 37e9  # 34.4 of records, rows and mode arrays; with records for all problems 42 and more
