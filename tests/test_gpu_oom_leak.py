"""A refused device allocation fails its own call alone: the CUDA error it
leaves behind must not be taken for one of the launches that follow (a 2D
frame would return an error after its particles had been counted, and count
them again when called once more)."""
from __future__ import annotations

import numpy as np
import pytest

from _helpers import bits, load_scene, records_f32, small_muller
from coupledwateranimation_gb300 import CwaError, Sim
from coupledwateranimation_gb300._abi import CWA_ERR_OOM
from coupledwateranimation_gb300.pbd import PbdSim, make_boxes, pbd_defaults
from coupledwateranimation_gb300.sim2d import Sim2D, defaults2d

pytestmark = pytest.mark.gpu
OOM = CWA_ERR_OOM


def _refused():
    p = pbd_defaults()
    p.n_boxes, p.max_contacts = 1 << 22, 4096  # 820 GB of contact slots
    with pytest.raises(CwaError) as ei:
        PbdSim(p)
    assert ei.value.status == OOM


def test_next_calls_are_unaffected(lib):
    sc = small_muller((6, 6, 6), 0.03, (64, 48))
    p2, pb = defaults2d(), pbd_defaults()
    pb.n_boxes = 300
    boxes, out = make_boxes(pb, 4), []
    for refuse in (False, True):
        with Sim2D(p2) as a, Sim(sc.desc) as b, PbdSim(pb) as c:
            load_scene(b, 0, sc)
            c.upload(boxes)
            state = a.download_particles()
            for step in (lambda: a.upload_particles(state), lambda: a.step(2), lambda: a.run_pass("grid"),
                         lambda: a.run_pass("density"), lambda: a.run_pass("force"), lambda: b.step(2), b.grid,
                         b.rho_pres, b.force, lambda: b.wave_advance(5), lambda: c.step(2)):
                if refuse:
                    _refused()
                step()
            out.append((a.download_particles(), bits(records_f32(b.download_particles(0))), c.download()))
    for x, y in zip(*out):
        assert np.array_equal(x.view(np.uint8), y.view(np.uint8))
