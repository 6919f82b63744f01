"""The 2D family on either side of the sizes where its grid changes its kernels,
its cells and its particles times cells, against the CPU restatement; and
where a frame's wave substeps change theirs, against single passes."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_sph2d_grid import TOL, _params, _rel_inf, _state
from coupledwateranimation_gb300.sim2d import Sim2D, defaults2d

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,cells", [(4096, (1, 1279)), (4096, (1, 1280)), (40000, (26, 32)), (40400, (26, 32)),
                                     (300, (1, 1279)), (300, (40, 32))])
def test_grid_rule(lib, orc, n, cells):
    """1280 counters in one launch, 1281 in two; 40,000 x 833 counters below
    2^25, 40,400 above."""
    p = _params(n, cells)
    state = _state(n, n)
    state["pos"][: n // 4, :2] = state["pos"][n // 4: 2 * (n // 4), :2] + np.float32(0.01)  # no crowd
    with Sim2D(p) as sim:
        sim.splash()
        sim.upload_particles(state)
        wave = sim.download_wave()
        sim.run_pass("grid")
        sim.run_pass("density")
        dens = sim.download_particles()
        sim.run_pass("force")
        forc = sim.download_particles()
    want_d = orc.density_2d(p, state, wave)
    assert np.max(np.abs(dens["acc"][:, 3] - want_d["acc"][:, 3]) / want_d["acc"][:, 3]) <= TOL
    want_f = orc.force_2d(p, dens, wave, grid_from=state)
    for k in range(2):
        assert _rel_inf(forc["acc"][:, k], want_f["acc"][:, k]) <= TOL


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("substeps", [1, 2, 5])
@pytest.mark.parametrize("cells", [3, 1023, 1024, 1025, 2049])
def test_wave_rule(lib, cells, substeps, kind):
    p = defaults2d(kind)
    p.n_particles, p.init_columns = 64, 8
    p.sph_substeps, p.wave_substeps, p.wave_cells = 0, substeps, cells
    names = ("wave_iterate",) if kind else ("wave_predict", "wave_correct")
    with Sim2D(p) as a, Sim2D(p) as b:
        a.splash()
        b.splash()
        a.step(3)
        for _ in range(3 * substeps):
            for name in names:
                b.run_pass(name)
        assert np.array_equal(a.download_wave().view(np.uint32), b.download_wave().view(np.uint32))
        if kind:
            assert np.array_equal(a.download_wave_prev().view(np.uint32), b.download_wave_prev().view(np.uint32))
