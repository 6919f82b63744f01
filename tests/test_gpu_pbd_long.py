"""Boxes whose partner lists are served by the whole block: lists spread over
several windows of box numbers, several such boxes in one block and in the last
block, against the float32 CPU restatement bit for bit; and the time of a floor
over thousands of boxes beside that of the same boxes without contact to it."""
from __future__ import annotations

import time

import numpy as np
import pytest

from coupledwateranimation_gb300.pbd import PbdSim, make_boxes, pbd_defaults

pytestmark = pytest.mark.gpu


def _floors(n, floors, slots, cells, y=0.0, thin=1):
    """n - floors small boxes about the plane y = 0 and `floors` slabs of the
    highest indexes; of the small ones only every `thin`-th near the plane."""
    p = pbd_defaults()
    p.n_boxes, p.max_contacts = n, slots
    for a in range(3):
        p.grid_cells[a] = cells
    b = make_boxes(p, 5)
    rng = np.random.default_rng(n)
    small = np.float32(0.02 if n < 30000 else 0.002)
    b["hw"][:, :3] = small
    b["rm"] = np.float32(1.0) / (small * small * small)
    b["x"][:, :3] = rng.uniform(-0.97, 0.97, (n, 3)).astype(np.float32)
    far = np.arange(n) % thin != 0
    b["x"][:, 1] = np.where(far, rng.uniform(0.3, 0.97, n), rng.uniform(-0.05, 0.05, n)).astype(np.float32)
    b["v"] = 0.0
    for k in range(floors):
        b["hw"][n - 1 - k, :3] = (0.9, 0.04, 0.9)
        b["x"][n - 1 - k, :3] = (0.0, y + 0.01 * k, 0.0)
        b["rm"][n - 1 - k] = 1e-3
    return p, b


@pytest.mark.parametrize("n,floors,slots,cells,thin", [
    (129, 1, 16, 8, 1), (130, 3, 48, 8, 1), (1500, 2, 64, 8, 1), (4097, 1, 4096, 8, 1),
    (131073, 1, 64, 16, 97), (300000, 2, 64, 16, 641)])
def test_floors(lib, orc, n, floors, slots, cells, thin):
    p, boxes = _floors(n, floors, slots, cells, thin=thin)
    want = orc.pbd_step(p, boxes, 2)
    with PbdSim(p) as sim:
        sim.upload(boxes)
        sim.step(2)
        got = sim.download()
    assert got["n"][-1] > min(slots, 64)  # the floor's list is long
    assert np.array_equal(got.view(np.uint8), want.view(np.uint8))


def test_floor_costs_no_search_of_all_pairs(lib):
    """A floor over 4095 boxes with the default 64 slots: its partners took a
    search of every pair, 3400 us a step, where the same boxes without contact
    take 57; the block's walk of the floor's cells brings it to about 500."""
    us = []
    for y in (0.0, 0.9):
        p, boxes = _floors(4096, 1, 64, 16, y=y)
        with PbdSim(p) as sim:
            best = 1e9
            for _ in range(5):
                sim.upload(boxes)
                sim.step(1)
                sim.download()
                t = time.perf_counter()
                sim.step(4)
                sim.download()
                best = min(best, (time.perf_counter() - t) / 4 * 1e6)
            us.append(best)
    assert us[0] < 20 * us[1], us
