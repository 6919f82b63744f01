"""The neighbour-pass options on small sims: an option of the one-thread forms
that is set runs those forms (by the kernels that the passes queue), none set
the several-lanes forms; all of them the same bits, and the tuner times the
several-lanes form as the options at entry."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from _helpers import bits, load_scene, records_f32, small_muller
from coupledwateranimation_gb300 import PREC_COMPENSATED, PREC_FP32, PREC_FP64, Sim

pytestmark = pytest.mark.gpu
ONE_THREAD = [{"nb_stage": 1}, {"nb_stage": -1}, {"nb_threads": 32}, {"nb_threads": 64}, {"nb_threads": 96},
              {"nb_threads": 128}, {"nb_scan_minb": 6}, {"nb_scan_minb": 8}, {"nb_force_minb": 6}, {"nb_queue": 1}]


class _KernelNode(C.Structure):  # CUDA_KERNEL_NODE_PARAMS
    _fields_ = [("func", C.c_void_p), ("dims", C.c_uint * 7), ("params", C.c_void_p), ("extra", C.c_void_p),
                ("kern", C.c_void_p), ("ctx", C.c_void_p)]


def _kernels(sim, fn):
    """Names of the kernels that fn queues on the sim's stream: captured into a
    graph that is never run, and read from its nodes."""
    cu = C.CDLL("libcuda.so.1")

    def ok(err):
        assert err == 0, err

    stream, graph, n = C.c_void_p(sim.device_view(0).stream), C.c_void_p(), C.c_size_t()
    ok(cu.cuStreamBeginCapture_v2(stream, 1))
    fn()
    ok(cu.cuStreamEndCapture(stream, C.byref(graph)))
    ok(cu.cuGraphGetNodes(graph, None, C.byref(n)))
    nodes = (C.c_void_p * n.value)()
    ok(cu.cuGraphGetNodes(graph, nodes, C.byref(n)))
    names = []
    for node in nodes:
        kind, p, name = C.c_int(), _KernelNode(), C.c_char_p()
        ok(cu.cuGraphNodeGetType(C.c_void_p(node), C.byref(kind)))
        if kind.value == 0:
            ok(cu.cuGraphKernelNodeGetParams_v2(C.c_void_p(node), C.byref(p)))
            ok(cu.cuFuncGetName(C.byref(name), C.c_void_p(p.func)) if p.func
               else cu.cuKernelGetName(C.byref(name), C.c_void_p(p.kern)))
            names.append(name.value.decode())
    ok(cu.cuGraphDestroy(graph))
    return " ".join(names)


@pytest.mark.parametrize("zsub", [1, 4])
@pytest.mark.parametrize("prec", [PREC_FP32, PREC_COMPENSATED, PREC_FP64])
def test_options_reach_their_kernels(lib, prec, zsub):
    sc = small_muller((17, 16, 15), 0.02, (48, 40), zsub=zsub, seed=41)
    got = []
    for kw in [{}] + ONE_THREAD:
        with Sim(sc.desc, precision=prec, **kw) as sim:
            load_scene(sim, 0, sc)
            sim.step(2)
            sim.grid()
            names = _kernels(sim, lambda: (sim.rho_pres(), sim.force()))
            assert ("k_rho_team" in names) == (not kw), (kw, names)
            assert ("k_scan_cands" in names) == bool(kw), (kw, names)
            assert ("k_force_team" in names) == (not kw and prec == PREC_COMPENSATED), (kw, names)
            sim.rho_pres()
            sim.force()
            got.append(bits(records_f32(sim.download_particles(0))))
    for kw, g in zip(ONE_THREAD, got[1:]):
        assert np.array_equal(g, got[0]), kw


@pytest.mark.parametrize("prec,n", [(PREC_FP32, 24576), (PREC_COMPENSATED, 24576), (PREC_FP64, 8192)])
def test_limit_of_the_several_lanes_forms(lib, prec, n):
    sc = small_muller((30, 30, 30), 0.02, (16, 16), seed=2)
    for count in (n, n + 1):
        sc.desc.n_particles = count
        with Sim(sc.desc, precision=prec) as sim:
            sim.upload_particles(0, sc.particles[:count].copy())
            sim.upload_wave(0, sc.wave)
            sim.grid()
            assert ("k_rho_team" in _kernels(sim, sim.rho_pres)) == (count == n)


def test_tuner_keeps_the_faster_form(lib):
    sc = small_muller((16, 16, 16), 0.02, (64, 64), zsub=1)
    with Sim(sc.desc) as sim:
        load_scene(sim, 0, sc)
        sim.step(2)
        rep = sim.autotune(trial_steps=4)
        assert rep["entry_ms"] > 0 and rep["best_ms"] <= rep["entry_ms"]
        knobs = ("nb_stage", "nb_scan_minb", "nb_force_minb", "nb_threads")
        if min(t["ms"] for t in rep["tried"]) > 0.985 * rep["entry_ms"]:
            assert not any(rep["best"][k] for k in knobs)  # four lanes stay
        else:
            assert rep["best"]["nb_threads"] in (64, 128)
        assert {k: sim.options()[k] for k in knobs} == {k: rep["best"][k] for k in knobs}
