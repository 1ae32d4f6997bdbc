"""DSA injection by a whole block a tracer (small runs, few shocks) and by two
warps a tracer (three shocked tracers of a block's eight and more): a tracer's
spectra are the same bits either way, and the oracle's to the parity bar."""
import numpy as np
import pytest

import pyoracle
from conftest import load_package
from golden_io import rel_err

load_package()
from croma_fp_b200 import config, native, synth  # noqa: E402

pytestmark = pytest.mark.gpu
CYCLE, BLOCKS_PER_SM = 47, 16


def _inject(cfg, prm, w, args, sh, crp, cre, at, reacc):
    fp = native.TracerFP(cfg)
    try:
        fp.set_state(crp[at], cre[at], mass=w.mass[at])
        fp.set_dsa(prm)
        count = fp.dsa_inject({k: np.ascontiguousarray(v[at]) if isinstance(v, np.ndarray) else v for k, v in sh.items()},
                              1.0, args[5], "tracer_state", reacc)
        return count, *fp.get_state()
    finally:
        fp.close()


@pytest.mark.parametrize("reacc", ["off", "positive_delta", "drury83"])
@pytest.mark.parametrize("nb,fraction", [(128, 1.0), (128, 0.3), (512, 1.0)])
def test_teams_give_the_same_bits(nb, fraction, reacc):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    cfg = config.config1(nb=nb)
    w = synth.Workload(cfg, CYCLE, 100, seed=7)
    args = w.snapshot_args(25)
    sh = synth.shocks(args[0], 25, 7, fraction=fraction)
    prm = config.DsaParams(reacc_eta_cap=0.1 if reacc == "drury83" else 0.0)
    o = pyoracle.Oracle(cfg)
    crp, cre = synth.initial_state((o.grid(0)[0], o.grid(0)[1]), (o.grid(1)[0], o.grid(1)[1]), CYCLE, cfg.species)
    o_crp, o_cre, q, dis = crp.copy(), cre.copy(), np.zeros_like(crp), np.zeros(CYCLE, np.uint8)
    shocked = o.dsa_inject(prm, sh, w.mass, 1.0, args[5], 1, native.TracerFP.DSA_REACC[reacc], o_crp, o_cre, q, q.copy(), dis)
    assert shocked >= (CYCLE if fraction == 1.0 else 5) * 0.5
    count, b_crp, b_cre = _inject(cfg, prm, w, args, sh, crp, cre, np.arange(CYCLE), reacc)   # a block a tracer
    assert count == shocked and rel_err(b_crp, o_crp) <= 1e-10 and rel_err(b_cre, o_cre) <= 1e-10
    at = np.arange(8 * BLOCKS_PER_SM * sms + 3) % CYCLE                                       # eight tracers a block
    _, t_crp, t_cre = _inject(cfg, prm, w, args, sh, crp, cre, at, reacc)
    assert np.array_equal(t_crp, b_crp[at]) and np.array_equal(t_cre, b_cre[at])
