"""The colour pass without an environment map (sprites shaded pixel by pixel)
at the edges of its tiles: images off multiples of the tile, sprites of one
pixel to many tiles, tile lists around 32 and past the shared-memory sort's 512
entries, particles alone and with the surface, against the CPU restatement, as
the frame tests compare: same fragments, colours within 2 counts on 99.8% of
the pixels."""
from __future__ import annotations

import numpy as np
import pytest

from _helpers import load_scene, records_f32, small_muller
from coupledwateranimation_gb300 import Sim
from coupledwateranimation_gb300.sim import render_defaults

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(1, 1), (33, 18), (160, 91)])
@pytest.mark.parametrize("point", [1.0, 7.5, 40.0])
@pytest.mark.parametrize("lattice,surface", [((3, 3, 3), 1), ((16, 12, 14), 0), ((16, 12, 14), 1)])
def test_frames(lib, orc, size, point, lattice, surface):
    sc = small_muller(lattice, 0.03, (24, 20), seed=9)
    cam, prm = render_defaults(*size)
    prm.point_size, prm.surface_res, prm.draw_surface = point, 40, surface
    with Sim(sc.desc) as sim:
        load_scene(sim, 0, sc)
        got = sim.render(0, camera=cam, params=prm)
        pos = records_f32(sim.download_particles(0))[:, :4]
        u, _ = sim.download_wave(0)
    want = orc.render(pos, u, cam, prm)
    off = np.abs(got.astype(int) - want.astype(int)).max(axis=2)
    assert got.shape == want.shape
    assert np.mean(off <= 2) >= 0.998
