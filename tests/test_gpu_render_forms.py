"""The two forms of the colour walk against each other, byte for byte: with an
environment map every fragment goes through the queue, without one sprites are
shaded pixel by pixel; a map of zeros, not drawn as background, gives both the
same colour terms.  And the blend's quotient by 255 against the division."""
from __future__ import annotations

from fractions import Fraction

import numpy as np
import pytest

from _helpers import load_scene, small_muller, small_reference
from coupledwateranimation_gb300 import Sim
from coupledwateranimation_gb300.sim import render_defaults


def _rounded(x: Fraction) -> np.float32:
    """x to the nearest float, ties to even (x >= 0, in the normal range)."""
    if x == 0:
        return np.float32(0)
    f = np.float32(float(x))
    near = [np.nextafter(f, np.float32(-np.inf)), f, np.nextafter(f, np.float32(np.inf))]
    return min(near, key=lambda v: (abs(Fraction(float(v)) - x), int(v.view(np.uint32)) & 1))


def test_quotient_by_255():
    """n / 255 as reciprocal product and one residual correction, each
    operation rounded once, equals the division for every 8-bit n."""
    r = _rounded(Fraction(1, 255))
    exact = lambda v: Fraction(float(v))  # noqa: E731
    for n in range(256):
        q = _rounded(n * exact(r))
        residual = n - exact(q) * 255
        e = np.float32(float(residual))
        assert exact(e) == residual  # a float, whatever its rounding
        assert _rounded(exact(e) * exact(r) + exact(q)) == _rounded(Fraction(n, 255)), n


@pytest.mark.gpu
@pytest.mark.parametrize("size", [(33, 18), (160, 91), (320, 240), (641, 359)])
@pytest.mark.parametrize("point", [1.0, 7.5, 40.0])
@pytest.mark.parametrize("scene,surface", [("muller", 0), ("muller", 1), ("reference", 1)])
def test_forms_are_equal(lib, size, point, scene, surface):
    sc = small_muller((20, 16, 18), 0.03, (64, 48), seed=9) if scene == "muller" else small_reference()
    cam, prm = render_defaults(*size)
    prm.point_size, prm.surface_res, prm.draw_surface, prm.draw_skybox = point, 60, surface, 0
    with Sim(sc.desc) as sim:
        load_scene(sim, 0, sc)
        for steps in (0, 3):
            sim.step(steps)
            plain = sim.render(0, camera=cam, params=prm)
            with Sim(sc.desc) as other:
                load_scene(other, 0, sc)
                other.step(3 if steps else 0)
                other.set_skybox(np.zeros((6, 2, 2, 4), np.uint8))
                queued = other.render(0, camera=cam, params=prm)
            assert len(np.unique(plain.reshape(-1, 4), axis=0)) > 3
            assert np.array_equal(plain, queued)
