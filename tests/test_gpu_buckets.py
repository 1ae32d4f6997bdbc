"""Buckets of equal (nsub, n_on), numbered by their first tracer, members in
tracer order: the one-block build and the sorts it gives way to above 4,096
tracers, at the edges of warps, blocks and tables, with one key (the cap on the sub-steps) and with many."""
import numpy as np
import pytest

from conftest import load_package

load_package()
from croma_fp_b200 import config, native, synth  # noqa: E402

pytestmark = pytest.mark.gpu

CASES = {
    "one": dict(nsub_max=10),
    "capped": dict(nsub_max=64),
    "many": dict(nsub_max=4096, reacc_window_mode=1, f_eddy=0.002),
}


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("n", [1, 31, 33, 64, 1023, 1025, 2049, 4095, 4096, 4097])
def test_buckets_in_first_appearance_order(name, n):
    cfg = config.config1(nb=128, **CASES[name])
    w = synth.Workload(cfg, n, 100, seed=n)
    args = list(w.snapshot_args(41))
    if name == "many":   # densities (sub-steps) and eddy times (window) over decades
        rng = np.random.default_rng(n)
        args[0] = args[0].copy()
        args[0][0] *= 10.0 ** rng.uniform(-2.0, 2.0, n)
        args[0][4] *= 10.0 ** rng.uniform(-2.0, 2.0, n)
    fp = native.TracerFP(cfg)
    try:
        gp, ge = fp.grid(0), fp.grid(1)
        crp, cre = synth.initial_state((gp[0], gp[1]), (ge[0], ge[1]), n, cfg.species)
        fp.set_state(crp, cre, mass=w.mass)
        fp.snapshot(*args, sync=True)
        s = fp.schedule()
    finally:
        fp.close()
    number, ids = {}, []
    for key in zip(s["nsub"].tolist(), s["non"].tolist()):
        ids.append(number.setdefault(key, len(number)))
    ids = np.array(ids)
    assert (len(number) > 1) == (name == "many" and n > 1)
    assert s["nbuckets"] == len(number)
    assert np.array_equal(s["bucket_ids"], ids)
    assert np.array_equal(s["bucket_indices"], np.argsort(ids, kind="stable"))
