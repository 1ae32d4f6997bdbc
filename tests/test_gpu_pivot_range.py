"""Pivots far above one: a magnetic field that takes the diagonal to 2^184 ..
2^211, where eight rows' continuants leave the range of a double and four stay in
it.  The electrons lose everything but what the secondary source gives them in
the sub-step, so the bins above the lowest hold the source's stationary flux;
against the oracle on every bin down to 1e-100 of the largest."""
import numpy as np
import pytest

import pyoracle
from conftest import load_package
from golden_io import rel_err

load_package()
from croma_fp_b200 import config, native, synth  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb,n,path", [(128, 67, "fused"), (128, 5, "fused"), (128, 67, "plain"), (256, 65, "fused"),
                                       (512, 65, "fused"), (512, 9, "plain")])
def test_huge_pivots_match_oracle(nb, n, path):
    cfg = config.config1(nb=nb, nsub_max=10)
    w = synth.Workload(cfg, n, 100, seed=nb + n)
    cur, nxt, *when = w.snapshot_args(41)
    cur, nxt = cur.copy(), nxt.copy()
    cur[2] = nxt[2] = 1e30   # G
    o = pyoracle.Oracle(cfg)
    fp = native.TracerFP(cfg, path=path)
    try:
        gp, ge = fp.grid(0), fp.grid(1)
        crp, cre = synth.initial_state((gp[0], gp[1]), (ge[0], ge[1]), n, cfg.species)
        q = np.zeros_like(crp)
        o_crp, o_cre = crp.copy(), cre.copy()
        o.snapshot(cur, nxt, *when, q, q, o_crp, o_cre, mass=w.mass)
        fp.set_state(crp, cre, mass=w.mass)
        fp.snapshot(cur, nxt, *when, sync=True)
        g_crp, g_cre = fp.get_state()
    finally:
        fp.close()
    assert np.all(np.isfinite(o_cre)) and np.mean(o_cre > 1e-100 * o_cre.max()) > 0.5
    assert rel_err(g_cre, o_cre, floor_frac=1e-100) <= 1e-10
    assert rel_err(g_crp, o_crp) <= 1e-10
