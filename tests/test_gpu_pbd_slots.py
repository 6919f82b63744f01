"""More contact slots than 32 bits index (n_boxes x max_contacts above 2^31):
contacts of boxes whose slots lie past that, against the same boxes with few
slots a box, byte for byte."""
from __future__ import annotations

import numpy as np
import pytest

from coupledwateranimation_gb300._abi import PBD_BOX_DTYPE
from coupledwateranimation_gb300.pbd import PbdSim, pbd_defaults

pytestmark = pytest.mark.gpu

N, WIDE = 1 << 22, 520
TOUCHING = 4096  # boxes at the list's end, one for each of the 4096 before them


def _boxes(p):
    b = np.zeros(N, PBD_BOX_DTYPE)
    side = 162  # a lattice whose boxes are far apart
    k = np.arange(N)
    for a, q in enumerate((k % side, k // side % side, k // side**2)):
        b["x"][:, a] = -0.98 + 1.96 * q / (side - 1)
    b["x"][-TOUCHING:] = b["x"][-2 * TOUCHING:-TOUCHING] + np.float32(0.0004)
    hw = np.float32(0.001)
    b["hw"][:, :3] = hw
    b["rm"] = np.float32(1.0) / (hw * hw * hw)
    return b


def test_slots_past_32_bits(lib):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available() or torch.cuda.mem_get_info()[0] < 130 << 30:
        pytest.skip("needs 130 GB of free device memory")
    p = pbd_defaults()
    p.n_boxes = N
    for a in range(3):
        p.grid_cells[a] = 128
    boxes, out = _boxes(p), []
    assert (N - 2 * TOUCHING) * WIDE > 2**31  # every touching box's slots lie past 2^31
    for slots in (8, WIDE):
        p.max_contacts = slots
        with PbdSim(p) as sim:
            sim.upload(boxes)
            sim.step(1)
            assert sim.pair_count() == TOUCHING
            sim.step(1)
            out.append(sim.download())
    assert np.array_equal(out[0].view(np.uint8), out[1].view(np.uint8))
