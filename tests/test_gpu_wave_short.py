"""Wave advances of fewer than four steps: single passes, which allocate
nothing (the allocation hook would fail the first), leave the three buffers
where they are and the captured step graphs in use; from four steps on the
strips, in launches of 4 to 8 steps."""
from __future__ import annotations

import numpy as np
import pytest

from _helpers import bits, load_scene, small_muller
from coupledwateranimation_gb300 import Sim

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3])
def test_short_advances_need_no_memory(lib, n):
    sc = small_muller((6, 6, 6), 0.03, (125, 64), seed=4)
    with Sim(sc.desc) as a, Sim(sc.desc) as b:
        for s in (a, b):
            load_scene(s, 0, sc)
            s.step(3)
        fields = set()
        for _ in range(3):
            v = a.device_view(0)
            fields |= {v.wave_u_n, v.wave_u_nm1}
            assert lib.cwa_debug_fail_alloc(0) == 0
            try:
                a.wave_advance(n)
            finally:
                lib.cwa_debug_fail_alloc(-1)
            for _ in range(n):
                b.wave()
            for s in (a, b):
                s.step(2)
        v = a.device_view(0)
        assert len(fields | {v.wave_u_n, v.wave_u_nm1}) <= 3
        assert np.array_equal(bits(np.stack(a.download_wave(0))), bits(np.stack(b.download_wave(0))))


@pytest.mark.parametrize("wave", [(64, 48), (61, 200)])
def test_launches(lib, wave):
    sc = small_muller((1, 1, 1), 0.03, wave, seed=4)
    with Sim(sc.desc) as a, Sim(sc.desc) as b:
        for s in (a, b):
            load_scene(s, 0, sc)
        for n in (4, 5, 8, 9, 12, 16, 17, 25):
            l0 = a.launch_count
            a.wave_advance(n)
            assert a.launch_count - l0 == (n + 7) // 8
            for _ in range(n):
                b.wave()
            assert np.array_equal(bits(np.stack(a.download_wave(0))), bits(np.stack(b.download_wave(0)))), n
