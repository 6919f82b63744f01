"""The wave advance's variants by name: each name of the list selects the
kernel that the header documents under it, and the 128 x 32 box with its walk
in shared memory, once the default, is among them with its own steps."""
from __future__ import annotations

import numpy as np
import pytest

from _helpers import bits, load_scene, small_muller
from coupledwateranimation_gb300 import Sim
from coupledwateranimation_gb300._abi import WAVE_BLOCKS


def test_names_match_the_header():
    import re
    from pathlib import Path
    text = (Path(__file__).resolve().parent.parent / "include" / "cwa.h").read_text()
    named = {k: int(v) for k, v in re.findall(r"CWA_WAVE_BLOCK_(\w+) = (\d+)", text)}
    assert named.pop("COUNT") == len(WAVE_BLOCKS)
    assert sorted(named.values()) == list(range(len(WAVE_BLOCKS)))
    assert {k.lower() if k == "STRIP" else k: v for k, v in named.items()} == {n: k for k, n in enumerate(WAVE_BLOCKS)}


@pytest.mark.gpu
@pytest.mark.parametrize("wave", [(64, 64), (333, 217)])
def test_box_32x4(lib, wave):
    """Launches of four steps and single passes for the rest, where the strips
    take 10 steps in two launches; the same bits as the strips."""
    sc = small_muller((4, 4, 4), 0.02, wave)
    got, launches = [], []
    for name in ("32x4", "strip"):
        with Sim(sc.desc, wave_block=WAVE_BLOCKS.index(name)) as sim:
            load_scene(sim, 0, sc)
            l0 = sim.launch_count
            sim.wave_advance(10)
            sim.synchronize()
            launches.append(sim.launch_count - l0)
            got.append(bits(np.stack(sim.download_wave(0))))
    assert launches == [2 + 2, 2]
    assert np.array_equal(got[0], got[1])
