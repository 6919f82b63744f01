"""PBD boxes whose partner lists are long: one large box of the highest index
touches hundreds of lower ones, below, between and past the list sizes that
the post pass treats differently, against the float32 CPU restatement bit for
bit; and grids of one and several scan tiles."""
from __future__ import annotations

import numpy as np
import pytest

from coupledwateranimation_gb300.pbd import PbdSim, make_boxes, pbd_defaults

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 60, 66, 400])
@pytest.mark.parametrize("slots", [0, 65, 512])
def test_long_partner_lists(lib, orc, n, slots):
    p = pbd_defaults()
    p.n_boxes = n
    p.max_contacts = slots
    for a in range(3):
        p.grid_cells[a] = 6
    boxes = make_boxes(p, 5)
    small = np.float32(0.02)
    boxes["hw"][:-1, :3] = small
    boxes["rm"][:-1] = np.float32(1.0) / (small * small * small)
    boxes["hw"][-1, :3] = 0.6  # around the origin: every other box lies inside it
    boxes["rm"][-1] = np.float32(1.0) / np.float32(0.6 * 0.6 * 0.6)
    boxes["x"][-1, :3] = 0.0
    assert orc.pbd_step(p, boxes, 1)["n"][-1] == n - 1
    with PbdSim(p) as sim:
        sim.upload(boxes)
        sim.step(3)
        got = sim.download()
    assert np.array_equal(got.view(np.uint8), orc.pbd_step(p, boxes, 3).view(np.uint8))


@pytest.mark.parametrize("cells", [(20, 20, 20), (21, 20, 20), (8, 32, 32)])
def test_scan_tile_edges(lib, orc, cells):
    p = pbd_defaults()
    p.n_boxes = 1500
    p.max_contacts = 512  # long boxes in the flat grid touch many others
    for a in range(3):
        p.grid_cells[a] = cells[a]
    boxes = make_boxes(p, 6)
    with PbdSim(p) as sim:
        sim.upload(boxes)
        sim.step(4)
        got = sim.download()
    assert np.array_equal(got.view(np.uint8), orc.pbd_step(p, boxes, 4).view(np.uint8))
