"""Dense spots on cell borders, where the density pass counts a particle's
mask bits from its row windows' starts and force forms those windows again:
the windows have to be the same in both kernels, or force takes wrong
neighbours.  Against the float64 oracle, in the one-thread forms (work queue)
and the several-lanes forms."""
from __future__ import annotations

import numpy as np
import pytest

from _helpers import load_scene, records_f32, rel_inf, small_muller
from coupledwateranimation_gb300 import PREC_COMPENSATED, PREC_FP64, Sim

pytestmark = pytest.mark.gpu
TOL = 1e-5  # the neighbour passes' bound


def _scene(zsub, shift):
    """Two spots of one column, 60 particles above 40, around cell corners; a
    third of the coordinates lie on a border or `shift` steps of a float off."""
    sc = small_muller((9, 9, 9), 0.02, (16, 16), zsub=zsub, seed=3)
    d = sc.desc
    rng = np.random.default_rng(zsub)
    edge = np.float32([d.cell_size, d.cell_size, d.cell_size / zsub])
    lo = np.float32(list(d.box_lo))
    k = rng.permutation(d.n_particles)[:100]
    pos = (lo + edge * np.float32([9, 10, 9 * zsub])) + rng.uniform(-0.004, 0.004, (100, 3)).astype(np.float32)
    pos[60:, 2] -= np.float32(1.2) * edge[2]
    border = (lo + np.round((pos - lo) / edge).astype(np.float32) * edge).astype(np.float32)
    for _ in range(abs(shift)):
        border = np.nextafter(border, np.float32(np.sign(shift)) * np.float32(np.inf))
    sc.particles["pos"][k, :3] = np.where(rng.random((100, 3)) < 1.0 / 3.0, border, pos)
    sc.particles["vel"][:, :3] = rng.uniform(-0.5, 0.5, (d.n_particles, 3)).astype(np.float32)
    return sc


@pytest.mark.parametrize("prec", [PREC_COMPENSATED, PREC_FP64])
@pytest.mark.parametrize("shift", [-1, 0, 1])
@pytest.mark.parametrize("zsub", [1, 4])
@pytest.mark.parametrize("queue", [0, 1])
def test_windows_of_dense_spots(lib, orc, queue, zsub, shift, prec):
    sc = _scene(zsub, shift)
    with Sim(sc.desc, precision=prec, nb_queue=queue) as sim:
        load_scene(sim, 0, sc)
        u_n, _ = sim.download_wave(0)
        ref = orc.to_f64(records_f32(sim.download_particles(0)))
        sim.grid()
        sim.rho_pres()
        sim.force()
        got = records_f32(sim.download_particles(0))
    orc.rho_pres(sc.desc, ref, u_n.astype(np.float64))
    orc.force(sc.desc, ref, u_n.astype(np.float64))
    assert np.max(np.abs(got[:, 12] - ref[:, 12]) / np.abs(ref[:, 12])) <= TOL
    for c in range(3):
        assert rel_inf(got[:, 8 + c], ref[:, 8 + c]) <= TOL, c
