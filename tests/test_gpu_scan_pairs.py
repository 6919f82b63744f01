"""The candidate scan over staged candidates in pairs against the scan of
unstaged ones, bit for bit: row windows of 31 to 129 candidates (both sides of
the mask words and of the 64 bits), beginning at even and odd places of the
stage, alone and behind another scene."""
from __future__ import annotations

import numpy as np
import pytest

from _helpers import bits, load_scene, records_f32, small_muller
from coupledwateranimation_gb300 import PREC_COMPENSATED, PREC_FP32, Sim

pytestmark = pytest.mark.gpu


def _passes(scenes, k, prec, **kw):
    with Sim([sc.desc for sc in scenes], precision=prec, nb_queue=1, **kw) as sim:
        for j, sc in enumerate(scenes):
            load_scene(sim, j, sc)
        sim.grid()
        sim.rho_pres()
        sim.force()
        return records_f32(sim.download_particles(k))


def _spot(count, below, zsub):
    """`below` particles in the column under the spot of `count` in one z cell."""
    sc = small_muller((9, 9, 9), 0.02, (16, 16), zsub=zsub, seed=count)
    rng = np.random.default_rng(100 * count + below)
    n = sc.desc.n_particles
    pos = sc.particles["pos"]
    k = rng.permutation(n)[: count + below]
    pos[k[:count], :3] = np.float32((0.41, 0.43, 0.37)) + rng.uniform(-0.002, 0.002, (count, 3)).astype(np.float32)
    pos[k[count:], :3] = np.float32((0.41, 0.43, 0.31)) + rng.uniform(-0.002, 0.002, (below, 3)).astype(np.float32)
    return sc


@pytest.mark.parametrize("prec", [PREC_FP32, PREC_COMPENSATED])
@pytest.mark.parametrize("zsub", [1, 4])
@pytest.mark.parametrize("below", [0, 1, 2])
@pytest.mark.parametrize("count", [31, 32, 33, 34, 63, 64, 65, 66, 97, 129])
def test_pairs_equal_the_scalar_scan(lib, count, below, zsub, prec):
    sc = _spot(count, below, zsub)
    odd = small_muller((3, 3, 3), 0.03, (8, 8), seed=1)
    ref = _passes([sc], 0, prec, nb_stage=-1)
    for got in (_passes([sc], 0, prec), _passes([odd, sc], 1, prec), _passes([sc], 0, prec, nb_threads=64)):
        assert np.array_equal(bits(got), bits(ref))
