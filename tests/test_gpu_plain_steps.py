"""The per-step path against the oracle at every bin count: one tracer, a few,
an odd number; with and without sources; windowed segments, whose sub-steps
change coefficient sets; the resident rows are the per-step results."""
import numpy as np
import pytest

import pyoracle
from conftest import load_package
from golden_io import rel_err

load_package()
from croma_fp_b200 import config, native, synth  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("window", [0, 1])
@pytest.mark.parametrize("source", [False, True])
@pytest.mark.parametrize("nb,n", [(128, 1), (128, 37), (256, 3), (256, 33), (512, 1), (512, 5)])
def test_per_step_path(nb, n, source, window):
    extra = dict(reacc_window_mode=1, f_eddy=0.002) if window else {}
    cfg = config.config1(nb=nb, nsub_max=24, **extra)
    w = synth.Workload(cfg, n, 100, seed=3 * nb + n)
    o = pyoracle.Oracle(cfg)
    crp, cre = synth.initial_state((o.grid(0)[0], o.grid(0)[1]), (o.grid(1)[0], o.grid(1)[1]), n, cfg.species)
    q = np.zeros_like(crp)
    qp, qe = (3.0 * crp, 5.0 * cre) if source else (q, q)
    args = w.snapshot_args(41)
    o_crp, o_cre = crp.copy(), cre.copy()
    o.snapshot(*args, qp, qe, o_crp, o_cre, mass=w.mass)
    fp = native.TracerFP(cfg, path="plain")
    try:
        fp.set_state(crp, cre, *((qp, qe) if source else ()), mass=w.mass)
        fp.snapshot(*args, sync=True)
        g_crp, g_cre = fp.get_state()
    finally:
        fp.close()
    assert np.any(o_crp != crp) and np.any(o_cre != cre)
    assert rel_err(g_crp, o_crp) <= 1e-10
    assert rel_err(g_cre, o_cre) <= 1e-10
