"""DSA injection where a block looks at one, two and eight tracers, with a
ragged last block: tracers repeat in a cycle of 47 and must come out as the
oracle's 47 (the parity tolerance: the sums run in another order)."""
import numpy as np
import pytest

import pyoracle
from conftest import load_package
from golden_io import rel_err

load_package()
from croma_fp_b200 import config, native, synth  # noqa: E402

pytestmark = pytest.mark.gpu
CYCLE = 47


@pytest.mark.parametrize("reacc", ["off", "positive_delta", "drury83"])
@pytest.mark.parametrize("n", [1, 47, 4735, 4737, 18947])
def test_injection_over_block_sizes(n, reacc):
    cfg = config.config1(nb=128)
    w = synth.Workload(cfg, CYCLE, 100, seed=7)
    args = w.snapshot_args(25)
    sh = synth.shocks(args[0], 25, 7, fraction=0.5)
    prm = config.DsaParams(reacc_eta_cap=0.1 if reacc == "drury83" else 0.0)
    o = pyoracle.Oracle(cfg)
    crp, cre = synth.initial_state((o.grid(0)[0], o.grid(0)[1]), (o.grid(1)[0], o.grid(1)[1]), CYCLE,
                                   "electron_proton")
    o_crp, o_cre = crp.copy(), cre.copy()
    q = np.zeros_like(crp)
    dis = np.zeros(CYCLE, np.uint8)
    code = native.TracerFP.DSA_REACC[reacc]
    shocked = o.dsa_inject(prm, sh, w.mass, 1.0, args[5], 1, code, o_crp, o_cre, q, q.copy(), dis)
    at = np.arange(n) % CYCLE

    def tile(x):
        return np.ascontiguousarray(np.asarray(x)[at])

    fp = native.TracerFP(cfg)
    try:
        fp.set_state(tile(crp), tile(cre), mass=tile(w.mass))
        fp.set_dsa(prm)
        count = fp.dsa_inject({k: tile(v) if isinstance(v, np.ndarray) else v for k, v in sh.items()}, 1.0, args[5],
                              "tracer_state", reacc)
        g_crp, g_cre = fp.get_state()
    finally:
        fp.close()
    changed = np.any(o_cre != cre, axis=1) | np.any(o_crp != crp, axis=1)
    assert changed.sum() == shocked > 5
    assert count == changed[at].sum()
    assert rel_err(g_crp, tile(o_crp)) <= 1e-10
    assert rel_err(g_cre, tile(o_cre)) <= 1e-10
