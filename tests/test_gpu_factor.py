"""The factor kernel's row forms against the oracle, over the grids and
diffusion coefficients that choose between them: vanishing coefficients at the
low end of the grid (exp(-1/p) underflows below p ~ 1e-3), coefficients that
cross the reference's 1e-200 floor inside the grid, no diffusion, the filled and
the off form of a centred window, per-segment launches (eta cap); packed and
small runs, the per-step path's raw rows, at every bin count."""
import numpy as np
import pytest

import pyoracle
from conftest import load_package
from golden_io import rel_err

load_package()
from croma_fp_b200 import config, native, synth  # noqa: E402

pytestmark = pytest.mark.gpu

CASES = {
    "low_end": dict(pmin=-3.2, pemin=-3.1, dpp_mode="asa"),
    "floor": dict(dpp_mode="direct_tacc", t_acc_direct_gyr=1e208),
    "off": dict(dpp_mode="off"),
    "window_low_end": dict(pmin=-3.2, pemin=-3.1, dpp_mode="asa", reacc_window_mode=1, f_eddy=0.002),
    "window": dict(dpp_mode="ttd", reacc_window_mode=1, f_eddy=0.002),
    "cap": dict(dpp_mode="asa", eta_dpp_cap=1e-3),
    "odd_segments": dict(dpp_mode="asa", coeff_interp_max_segments=3, reacc_window_mode=1, f_eddy=0.002),
}


RUNS = [(128, 67, "fused"), (128, 5, "fused"), (256, 65, "fused"), (128, 67, "plain")]
WIDE = [(512, 65, "fused"), (512, 9, "plain")]


@pytest.mark.parametrize("name,nb,n,path", [(k, *r) for k in sorted(CASES) for r in RUNS] +
                         [(k, *r) for k in ("floor", "window_low_end") for r in WIDE])
def test_row_forms_match_oracle(name, nb, n, path):
    cfg = config.config1(nb=nb, nsub_max=16, **CASES[name])
    w = synth.Workload(cfg, n, 100, seed=nb + n)
    o = pyoracle.Oracle(cfg)
    fp = native.TracerFP(cfg, path=path)
    try:
        gp, ge = fp.grid(0), fp.grid(1)
        crp, cre = synth.initial_state((gp[0], gp[1]), (ge[0], ge[1]), n, cfg.species)
        q = np.zeros_like(crp)
        o_crp, o_cre = crp.copy(), cre.copy()
        args = w.snapshot_args(41)
        o.snapshot(*args, q, q, o_crp, o_cre, mass=w.mass)
        fp.set_state(crp, cre, mass=w.mass)
        fp.snapshot(*args, sync=True)
        g_crp, g_cre = fp.get_state()
    finally:
        fp.close()
    assert np.all(np.isfinite(o_cre)) and np.any(o_cre != cre)
    assert rel_err(g_crp, o_crp) <= 1e-10
    assert rel_err(g_cre, o_cre) <= 1e-10
