"""The wave advance's default form (register strips, 2 to 8 steps a launch)
against single wave passes, bit for bit, at the edges of its strips: widths
around the strips' 112 and 120 output columns and off multiples of 4, heights
around the smallest strip and where strips split, every remainder of the step
count, a line source on a strip's border, damping with and without coupling."""
from __future__ import annotations

import numpy as np
import pytest

from coupledwateranimation_gb300 import Sim

from _helpers import bits, load_scene, small_muller, small_reference

pytestmark = pytest.mark.gpu


def _same(scenes, n):
    sims = [Sim([sc.desc for sc in scenes]) for _ in range(2)]
    try:
        for s in sims:
            for k, sc in enumerate(scenes):
                load_scene(s, k, sc)
        sims[0].wave_advance(n)
        for _ in range(n):
            sims[1].wave()
        for k in range(len(scenes)):
            for a, b in zip(sims[0].download_wave(k), sims[1].download_wave(k)):
                assert np.array_equal(bits(a), bits(b))
        for s in sims:
            s.synchronize()
    finally:
        for s in sims:
            s.close()


@pytest.mark.parametrize("nx", [1, 3, 111, 112, 113, 116, 120, 121, 224, 226, 241])
@pytest.mark.parametrize("nz", [1, 7, 31, 32, 95])
def test_strip_edges(lib, nx, nz):
    _same([small_muller((3, 3, 3), 0.03, (nx, nz), seed=nx + nz)], 15)


@pytest.mark.parametrize("nx", [123, 127, 128, 129, 130, 131, 136, 239, 240, 242, 243, 249, 351, 353])
@pytest.mark.parametrize("n", [8, 4])  # 8 and 4 columns of halo
def test_first_and_last_strip(lib, nx, n):
    _same([small_muller((3, 3, 3), 0.03, (nx, 37), seed=nx)], n)


@pytest.mark.parametrize("widths", [(128, 64), (130, 64), (64, 131, 252)])  # of four, and mixed, in one launch
def test_widths_of_a_batch(lib, widths):
    _same([small_muller((3, 3, 3), 0.03, (nx, 40), seed=nx) for nx in widths], 8)


@pytest.mark.parametrize("n", [2, 3, 4, 5, 6, 7, 8, 9, 23])
@pytest.mark.parametrize("atten", [1.0, 0.97])
def test_steps_and_damping(lib, n, atten):
    sc = small_muller((3, 3, 3), 0.03, (229, 130), seed=n)
    sc.desc.wave_atten = atten
    _same([sc, small_muller((3, 3, 3), 0.03, (64, 40), seed=n + 1)], n)


@pytest.mark.parametrize("nx", [64, 224, 225, 240])  # the source column nx / 2 inside a strip and on its border
@pytest.mark.parametrize("preset", ["reference", "muller"])
def test_line_source(lib, nx, preset):
    sc = small_reference(512) if preset == "reference" else small_muller((3, 3, 3), 0.03, (nx, 50), seed=3)
    sc.desc.wave_nx, sc.desc.wave_nz, sc.desc.wave_mode = nx, 50, 0.5
    sc.wave = np.random.default_rng(nx).uniform(-0.02, 0.02, (50, nx)).astype(np.float32)
    _same([sc], 13)
