"""The warp-aggregated count under keys that repeat in every way a warp can
hold them: the point grid's order against a stable sort of the cells, and the
time of a grid with half the points in one cell, between the others."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_scan_tiles import _Grid
from coupledwateranimation_gb300 import _abi

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
DIMS = (64, 64, 100)


def _grid(lib, cell):
    """Points in the middle of the given cells (x-major)."""
    n = len(cell)
    pos = np.zeros((n, 4), np.float32)
    for a, q in enumerate((cell // 6400, cell // 100 % 64, cell % 100)):
        pos[:, a] = (q + 0.5) / 64
    return _Grid(lib, torch.from_numpy(pos).cuda(), DIMS, 1.0 / 64)


def _one_hash(count):
    """Cells whose keys agree in the bits that group a warp's lanes."""
    k = np.arange(64 * 64 * 100, dtype=np.uint64)
    return k[((k * np.uint64(0x9E3779B1)) & np.uint64(0xFFFFFFFF)) >> np.uint64(27) == 5][:count].astype(np.int64)


def _patterns():
    rng = np.random.default_rng(8)
    yield "one point", np.array([77])
    yield "sorted", np.sort(rng.integers(0, 40, 5003))
    yield "two in turn", 7 + 9 * (np.arange(2047) % 2)
    yield "few at random", rng.integers(0, 9, 5000) * 41000
    yield "all distinct", rng.permutation(409600)[:5001]
    for m in (2, 3, 5, 40):
        yield f"{m} of one hash", rng.choice(_one_hash(m), min(5003, 900 * m))
    yield "one hash among others", np.where(rng.random(4099) < 0.5, rng.choice(_one_hash(4), 4099),
                                            rng.integers(0, 409600, 4099))
    yield "half in one", np.where(np.arange(2001) % 2 == 0, 409599, rng.integers(0, 409600, 2001))


@pytest.mark.parametrize("name,cell", list(_patterns()), ids=lambda v: v if isinstance(v, str) else "")
def test_order(lib, name, cell):
    g = _grid(lib, cell)
    for _ in range(2):
        g.build()
    assert g.status() == _abi.CWA_OK
    want = torch.from_numpy(cell).cuda()
    assert torch.equal(g.cell_of.long(), want)
    assert torch.equal(g.index.long(), torch.sort(want, stable=True).indices)


def test_half_the_points_in_one_cell(lib):
    """1.2 times the time of scattered points; 8 times when each of them took
    an atomic of its own."""
    n = 1000003
    rng = np.random.default_rng(1)
    scattered = rng.integers(0, 409600, n)
    ms = []
    for cell in (scattered, np.where(np.arange(n) % 2 == 0, 5, scattered)):
        g, best = _grid(lib, cell), float("inf")
        for _ in range(8):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            g.build()
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b))
        ms.append(best)
    assert ms[1] < 3 * ms[0], ms
