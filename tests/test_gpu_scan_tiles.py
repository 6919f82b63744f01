"""Grids of many scan tiles: the point grid and the boxes on either side of the
tile counts where the scan of the counts changes its form, and the time of a
grid whose tiles' totals cost more than its cells when each tile adds them up."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from coupledwateranimation_gb300 import _abi
from coupledwateranimation_gb300.pbd import PbdSim, make_boxes, pbd_defaults

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


class _Grid:
    def __init__(self, lib, pos, dims, edge, skew=0):
        nc = int(np.prod(dims))
        self.lib, self.pos, self.dims, self.edge, self.nc = lib, pos, (C.c_int32 * 3)(*dims), edge, nc
        self.size = lib.cwa_grid_workspace_bytes(len(pos), nc)
        self.ws = torch.empty(self.size, dtype=torch.uint8, device="cuda")
        self.start = torch.empty(nc + 1 + skew, dtype=torch.int32, device="cuda")[skew:]
        self.index = torch.empty(len(pos), dtype=torch.int32, device="cuda")
        self.cell_of = torch.empty(len(pos), dtype=torch.int32, device="cuda")
        self.lo = (C.c_float * 3)(0.0, 0.0, 0.0)
        self.stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)

    def build(self):
        _abi.check(self.lib.cwa_grid_build(
            _abi.ptr(self.pos), len(self.pos), self.lo, self.edge, self.dims, _abi.ptr(self.start),
            _abi.ptr(self.index), _abi.ptr(self.cell_of), _abi.ptr(self.ws), self.size, self.stream), "cwa_grid_build")

    def status(self):
        return self.lib.cwa_grid_status(len(self.pos), self.nc, _abi.ptr(self.ws), self.stream)


def _points(n, dims, edge, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.rand(n, 4, generator=g, device="cuda") * torch.tensor([*(d * edge for d in dims), 1.0], device="cuda")


@pytest.mark.parametrize("skew", [0, 1])
@pytest.mark.parametrize("dims", [(47, 178481, 1), (256, 256, 128), (3, 4, 700000), (1, 1, 67108869)])
def test_point_grid(lib, dims, skew):
    """1024 tiles, 1025 tiles, 1026 tiles and 8193 (a second round of the
    totals' scan); the starts on a 16-byte boundary and off it."""
    edge = 1.0 / max(dims)
    pos = _points(50001, dims, edge, 1)
    g = _Grid(lib, pos, dims, edge, skew)
    g.build()
    assert g.status() == _abi.CWA_OK
    key = g.cell_of.long()
    assert torch.equal(g.index.long(), torch.sort(key, stable=True).indices)
    cells, counts = torch.unique(key, return_counts=True)
    full = torch.zeros(g.nc + 1, dtype=torch.int32, device="cuda")
    full[cells + 1] = counts.int()
    assert torch.equal(g.start, torch.cumsum(full, 0, dtype=torch.int32))
    pos[7, 1] = float("nan")
    g.build()
    assert g.status() == _abi.CWA_ERR_NONFINITE


@pytest.mark.parametrize("cells", [(256, 256, 128), (204, 204, 204)])
def test_boxes(lib, orc, cells):
    p = pbd_defaults()
    p.n_boxes = 700
    for a in range(3):
        p.grid_cells[a] = cells[a]
    boxes = make_boxes(p, 9)
    boxes["hw"][:, :3] *= np.float32(0.1)
    with PbdSim(p) as sim:
        sim.upload(boxes)
        sim.step(3)
        got = sim.download()
    assert np.array_equal(got.view(np.uint8), orc.pbd_step(p, boxes, 3).view(np.uint8))


def test_cost_grows_with_the_cells(lib):
    """2^30 cells against 2^27, eight times as many: 7 times the time; 27 when
    every tile added up the totals before it."""
    us = []
    for dims in ((512, 512, 512), (1024, 1024, 1024)):
        g = _Grid(lib, _points(100000, dims, 1.0 / dims[0], 2), dims, 1.0 / dims[0])
        best = float("inf")
        for _ in range(4):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            g.build()
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b))
        us.append(best)
        del g
    assert us[1] < 14 * us[0], us
