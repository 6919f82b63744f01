"""A box upload whose item buffers do not fit: the call is refused with
CWA_ERR_OOM, the sim does not step on buffers it does not have, and the same
or another upload works once there is room."""
from __future__ import annotations

import numpy as np
import pytest

from coupledwateranimation_gb300 import CwaError
from coupledwateranimation_gb300._abi import CWA_ERR_INVALID_ARG, CWA_ERR_OOM
from coupledwateranimation_gb300.pbd import PbdSim, make_boxes, pbd_defaults

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def test_refused_upload(lib):
    p = pbd_defaults()
    p.n_boxes, p.max_contacts = 1 << 18, 8
    for a in range(3):
        p.grid_cells[a] = 64
    boxes = make_boxes(p, 3)
    boxes["hw"][:, :3] = np.float32(0.002)
    boxes["rm"] = np.float32(1.0) / np.float32(0.002) ** 3
    large = boxes.copy()
    large["hw"][-1, :3] = 0.22  # 16 cells a side: 2^18 x 4096 items, 17 GB
    large["rm"][-1] = 1.0
    with PbdSim(p) as sim, PbdSim(p) as other:
        for s in (sim, other):
            s.upload(boxes)
            s.step(1)
            s.download()
        torch.cuda.empty_cache()
        room = torch.empty(max(torch.cuda.mem_get_info()[0] - (6 << 30), 0), dtype=torch.uint8, device="cuda")
        for _ in range(2):
            with pytest.raises(CwaError) as ei:
                sim.upload(large)
            assert ei.value.status == CWA_ERR_OOM
            with pytest.raises(CwaError) as ei:
                sim.step(1)
            assert ei.value.status == CWA_ERR_INVALID_ARG
        del room
        torch.cuda.empty_cache()
        for s in (sim, other):
            s.upload(boxes)
            s.step(2)
        assert np.array_equal(sim.download().view(np.uint8), other.download().view(np.uint8))
        sim.upload(large)
        sim.step(1)
        assert np.isfinite(sim.download()["x"]).all()
