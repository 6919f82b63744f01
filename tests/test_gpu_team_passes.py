"""The several-lanes-a-particle forms of the density and force passes (small
sims) against the one-thread forms (which the work-queue option keeps), bit
for bit, at the particle counts where the rule changes and with dense spots:
row windows that pass bit 63 of their masks from the cell-based start, and
windows of more than 64 candidates."""
from __future__ import annotations

import numpy as np
import pytest

from _helpers import bits, load_scene, records_f32, small_muller
from coupledwateranimation_gb300 import PREC_COMPENSATED, PREC_FP32, PREC_FP64, Sim

pytestmark = pytest.mark.gpu


def _scene(n, zsub):
    sc = small_muller((37, 37, 37), 0.02, (48, 40), zsub=zsub, seed=n)
    sc.desc.n_particles = n
    sc.particles = sc.particles[:n].copy()
    rng = np.random.default_rng(n)
    sc.particles["vel"][:, :3] = rng.uniform(-0.5, 0.5, (n, 3)).astype(np.float32)
    for count, at in ((min(n // 8, 90), (0.41, 0.43, 0.37)), (min(n // 8, 40), (0.31, 0.33, 0.30))):
        k = rng.choice(n, count, replace=False)
        sc.particles["pos"][k, :3] = np.float32(at) + rng.uniform(-0.004, 0.004, (count, 3)).astype(np.float32)
    return sc


@pytest.mark.parametrize("prec", [PREC_FP32, PREC_COMPENSATED, PREC_FP64])
@pytest.mark.parametrize("zsub", [1, 4])
@pytest.mark.parametrize("n", [1, 33, 1000, 24 * 1024, 24 * 1024 + 1])
def test_team_forms_equal_one_thread_forms(lib, n, zsub, prec):
    sc = _scene(n, zsub)
    out = []
    for queue in (0, 1):
        with Sim(sc.desc, precision=prec, nb_queue=queue) as sim:
            load_scene(sim, 0, sc)
            for _ in range(2):
                sim.grid()
                sim.rho_pres()
                sim.force()
                first = records_f32(sim.download_particles(0))
                sim.integrate()
                sim.wave()
            sim.synchronize()
            out.append((first, records_f32(sim.download_particles(0))))
    assert np.array_equal(bits(out[0][0]), bits(out[1][0]))
    assert np.array_equal(bits(out[0][1]), bits(out[1][1]))
