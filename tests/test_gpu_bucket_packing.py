"""Bucket calls of the C ABI at counts that put one to four systems on a warp of
the factor kernel, each tracer with its own inverse-Compton row: 64 tracers
against the oracle (1e-10), and the same 64 tiled to larger calls bit for bit the
same wherever they land."""
import ctypes as C

import numpy as np
import pytest

import pyoracle
from conftest import load_package
from golden_io import rel_err

load_package()
from croma_fp_b200 import config, ref_abi, synth  # noqa: E402
from test_gpu_ref_abi import _coeff, _pipeline_input  # noqa: E402

pytestmark = pytest.mark.gpu

N, STEPS, DT = 64, 9, 2.0e-4


def _call(abi, grids, bg, ric, m1, p1, mass, crp, cre, windowed):
    cgp, cge = abi.grid(*grids[0]), abi.grid(*grids[1])
    ws = abi.lib.cuda_pipeline_workspace_create()
    assert ws
    try:
        ci, keep = _coeff(np.ascontiguousarray(bg), np.ascontiguousarray(ric), m1, p1, mass, np.zeros(crp.shape[0], np.uint8))
        pin = _pipeline_input(abi, cgp, cge, ci, STEPS, DT, windowed, *((2, 6) if windowed else (0, STEPS)), ws)
        zero = np.zeros_like(crp)
        pin.crp_init, pin.cre_init = ref_abi.dptr(crp), ref_abi.dptr(cre)
        pin.qpi_batch, pin.qepri_batch = ref_abi.dptr(zero), ref_abi.dptr(zero)
        out = np.empty_like(crp), np.empty_like(cre)
        rc = abi.lib.run_tracer_pipeline(C.byref(pin), None, ref_abi.dptr(out[0]), ref_abi.dptr(out[1]), None, None, None, None)
        assert rc == 0, abi.error()
        return out
    finally:
        abi.lib.cuda_pipeline_workspace_destroy(ws)


@pytest.mark.parametrize("nb,windowed", [(128, False), (128, True), (256, False), (512, True)])
def test_packing_keeps_a_tracers_bits(nb, windowed):
    cfg = config.config1(nb=nb)
    o = pyoracle.Oracle(cfg)
    abi = ref_abi.RefAbi(nb)
    assert abi.lib.croma_b200_set_model(1, 1, 0.3, 0.0) == 0   # ASA
    w = synth.Workload(cfg, N, 100, seed=9)
    gp, ge = o.grid(0), o.grid(1)
    crp, cre = synth.initial_state((gp[0], gp[1]), (ge[0], ge[1]), N, cfg.species)
    bg, mass = w.background(7), w.mass
    row, m1, p1 = o.ic_row(0.6)
    own = 1.0 + 0.01 * np.arange(N)   # each tracer's own row
    ric, m1, p1 = np.ascontiguousarray(row[:, None] * own), m1 * own, p1 * own
    o_crp, o_cre, zero = crp.copy(), cre.copy(), np.zeros_like(crp)
    o.evolve_segment(STEPS, DT, windowed, *((2, 6) if windowed else (0, STEPS)), bg, ric, m1, p1, zero, zero, o_crp, o_cre,
                     mass=mass, dis=np.zeros(N, np.uint8))
    grids = (gp, ge)
    g = _call(abi, grids, bg, ric, m1, p1, mass, crp, cre, windowed)
    assert rel_err(g[0], o_crp) <= 1e-10 and rel_err(g[1], o_cre) <= 1e-10
    # 2,368 warps: one to four systems each, with one set of factors or two
    for n in (1101, 2303, 3301, 4503, 9473) if nb == 128 else (1201, 2411):
        pick = np.arange(n) % N
        t = _call(abi, grids, bg[:, pick], ric[:, pick], m1[pick], p1[pick], mass[pick], crp[pick], cre[pick], windowed)
        assert np.array_equal(t[0], g[0][pick]) and np.array_equal(t[1], g[1][pick]), n
