"""The 2D family's grid passes at the sizes where their kernels change (cells
of one scan CTA, more cells, ragged particle counts, cells of more than 32
members) against the CPU restatement: one substep's density and force from the
same state within 1e-5, and passes called out of the frame's order."""
from __future__ import annotations

import numpy as np
import pytest

from coupledwateranimation_gb300 import _abi
from coupledwateranimation_gb300.sim2d import Sim2D, defaults2d

pytestmark = pytest.mark.gpu
TOL = 1e-5


def _rel_inf(got, want):
    got, want = np.asarray(got, np.float64), np.asarray(want, np.float64)
    return float(np.abs(got - want).max() / max(np.abs(want).max(), 1e-30))


def _params(n, cells):
    p = defaults2d()
    p.n_particles, p.init_columns = n, 1
    p.grid_cells[0], p.grid_cells[1] = cells
    return p


def _state(n, seed):
    rng = np.random.default_rng(seed)
    s = np.zeros(n, _abi.PARTICLE2D_DTYPE)
    s["pos"][:, 0] = rng.uniform(0.05, 9.5, n)
    s["pos"][:, 1] = rng.uniform(0.05, 9.5, n)
    s["pos"][: n // 4, :2] = rng.uniform(4.0, 4.6, (n // 4, 2))  # a crowd: cells of many members
    s["pos"][:, 3] = 1.0
    s["vel"][:, :2] = rng.uniform(-0.5, 0.5, (n, 2))
    s["acc"][:, 3] = 1000.0
    return s


@pytest.mark.parametrize("n", [1, 255, 1000, 8193])
@pytest.mark.parametrize("cells", [(1, 1), (16, 32), (63, 65), (64, 64), (70, 90)])
def test_one_substep(lib, orc, n, cells):
    p = _params(n, cells)
    if n / (cells[0] * cells[1]) > 1000:
        pytest.skip("cells above the stable-order limit")
    state = _state(n, n + cells[0])
    with Sim2D(p) as sim:
        sim.splash()
        sim.upload_particles(state)
        wave = sim.download_wave()
        sim.run_pass("grid")
        sim.run_pass("density")
        dens = sim.download_particles()
        sim.run_pass("force")
        forc = sim.download_particles()
    want_d = orc.density_2d(p, state, wave)
    assert np.max(np.abs(dens["acc"][:, 3] - want_d["acc"][:, 3]) / want_d["acc"][:, 3]) <= TOL
    want_f = orc.force_2d(p, dens, wave, grid_from=state)
    for k in range(2):
        assert _rel_inf(forc["acc"][:, k], want_f["acc"][:, k]) <= TOL


@pytest.mark.parametrize("n", [300, 5000])
def test_passes_out_of_order(lib, n):
    """grid, force without density; grid, density twice; frames between: the
    same bits as a sim brought to the same state by upload."""
    p = _params(n, (32, 32))
    p.wave_cells = 128
    with Sim2D(p) as a, Sim2D(p) as b:
        a.splash()
        b.splash()
        a.upload_particles(_state(n, 1))
        for names in (("grid", "force"), ("grid", "density", "density", "force"), ("grid", "density", "force")):
            b.upload_particles(a.download_particles())
            b.upload_wave(a.download_wave())
            for s in (a, b):
                for name in names:
                    s.run_pass(name)
            assert np.array_equal(a.download_particles().view(np.uint8), b.download_particles().view(np.uint8))
            a.step(1)
