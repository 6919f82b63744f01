"""Upload and download kernels at the edges of their grid: record and field
counts around one CTA's words, one round of 32 and of 128 CTAs x 256 threads x 8 words and
past it, from and to page-locked memory, come back unchanged."""
from __future__ import annotations

import numpy as np
import pytest

from _helpers import small_muller
from coupledwateranimation_gb300 import Sim
from coupledwateranimation_gb300._abi import PARTICLE_DTYPE, check, ptr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 63, 64, 2047, 2049, 16383, 16385, 65536, 65537])
def test_round_trip(lib, n):
    import torch

    rng = np.random.default_rng(n)
    sc = small_muller((n, 1, 1), 0.02, (n, 3))
    sc.desc.box_hi[0] = 0.02 * n + 1.0
    rec = torch.empty(n * 64, dtype=torch.uint8, pin_memory=True)
    back = torch.empty(n * 64, dtype=torch.uint8, pin_memory=True)
    rec.numpy().view(np.float32)[...] = rng.uniform(0.0, 1.0, 16 * n)
    u = torch.from_numpy(rng.uniform(-1, 1, (3, n)).astype(np.float32)).pin_memory()
    v = torch.empty((3, n), dtype=torch.float32, pin_memory=True)
    with Sim(sc.desc) as sim:
        sim.upload_particles(0, rec.numpy().view(PARTICLE_DTYPE))
        sim.upload_wave(0, u.numpy())
        check(lib.cwa_download_particles(sim.handle, 0, ptr(back), n), "download")
        check(lib.cwa_download_wave(sim.handle, 0, ptr(v), None, n, 3), "download")
    assert np.array_equal(back.numpy(), rec.numpy())
    assert np.array_equal(v.numpy(), u.numpy())


@pytest.mark.parametrize("pinned", [True, False])
@pytest.mark.parametrize("nx", [1, 7, 682, 683, 349526])
def test_one_field_fills_both_levels(lib, nx, pinned):
    import torch

    sc = small_muller((3, 3, 3), 0.02, (nx, 3))
    u = torch.from_numpy(np.random.default_rng(nx).uniform(-1, 1, (3, nx)).astype(np.float32))
    u = u.pin_memory() if pinned else u
    with Sim(sc.desc) as sim:
        sim.upload_wave(0, u.numpy())
        a, b = sim.download_wave(0)
    assert np.array_equal(a, u.numpy())
    assert np.array_equal(b, u.numpy())
