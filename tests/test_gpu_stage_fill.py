"""Staged candidate segments of odd length, whose last pair is filled up: the
staged density pass against the unstaged one, bit for bit and many times over,
with stages that hold other tiles' candidates from before (the work queue)
or another CTA's (more particles than the several-lanes forms take)."""
from __future__ import annotations

import numpy as np
import pytest

from _helpers import bits, load_scene, records_f32, small_muller
from coupledwateranimation_gb300 import PREC_COMPENSATED, PREC_FP32, Sim

pytestmark = pytest.mark.gpu


def _scene(n, zsub):
    """n particles at random places: segments of all lengths, half of them odd."""
    sc = small_muller((30, 30, 30), 0.02, (32, 32), zsub=zsub, seed=7)
    rng = np.random.default_rng(n + zsub)
    sc.desc.n_particles = n
    sc.particles = sc.particles[:n].copy()
    sc.particles["pos"][:, :3] = rng.uniform(0.05, 0.6, (n, 3)).astype(np.float32)
    return sc


@pytest.mark.parametrize("prec", [PREC_FP32, PREC_COMPENSATED])
@pytest.mark.parametrize("zsub", [1, 4])
@pytest.mark.parametrize("queue", [0, 1])
def test_odd_segments(lib, queue, zsub, prec):
    sc = _scene(26000, zsub)

    def passes(times, **kw):
        with Sim(sc.desc, precision=prec, nb_queue=queue, **kw) as sim:
            load_scene(sim, 0, sc)
            for _ in range(times):
                sim.grid()
                sim.rho_pres()
                sim.force()
                yield bits(records_f32(sim.download_particles(0)))

    want = next(passes(1, nb_stage=-1))
    for got in passes(20):
        assert np.array_equal(got, want)
