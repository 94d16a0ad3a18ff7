"""Results in pageable memory (staged through the context's page-locked ring)
against the same call into page-locked memory (written directly), bit for bit,
at the sizes where the staging changes: parts that share one wait (128 KB in
all), one chunk of 256 KB and a little more, more than the 16 MB ring."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nr", [1, 5461, 5462, 32768, 32769, 699050, 699051, 1500001])
def test_pageable_equals_page_locked(gpu, analytic_profile, nr):
    import torch
    import ncpa_gpu

    prof = gpu.load_profile(analytic_profile)
    m = gpu.solve(prof, ncpa_gpu.default_params(nz_grid=1000, turnoff_wkb=1), [0.02], [90.0])
    direct = [torch.zeros((1, nr), dtype=torch.float64).pin_memory().numpy() for _ in range(3)]
    m.tl1d(nr, 10.0, out=direct)
    for _ in range(2):
        for a, b in zip(m.tl1d(nr, 10.0), direct):
            assert np.array_equal(a, b)
    mixed = [np.zeros((1, nr)), torch.zeros((1, nr), dtype=torch.float64).pin_memory().numpy(), np.zeros((1, nr))]
    m.tl1d(nr, 10.0, out=mixed)
    for a, b in zip(mixed, direct):
        assert np.array_equal(a, b)
    m.close()
    prof.close()
