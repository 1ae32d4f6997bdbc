"""Which steps kernel a run takes: the packed one from 64 tracers on, uncalibrated
(tuned, no variant timed), also where one context crosses the line both ways; the
tuner below it; a tracer's spectra the same to the parity bar (1e-10) on either
side, and bit for bit wherever both runs take the packed one."""
import numpy as np
import pytest

from conftest import load_package
from golden_io import Case, rel_err

load_package()
from croma_fp_b200 import native  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _no_switches(monkeypatch):
    monkeypatch.delenv("CROMA_CUDA_TRIDIAG", raising=False)
    monkeypatch.delenv("CROMA_B200_STEPS_VARIANT", raising=False)


def _run(fp, case, n):
    d = case.d
    pick = np.arange(n) % d["crp0"].shape[0]
    fp.set_state(d["crp0"][pick], d["cre0"][pick], mass=d["mass"][pick])
    cur, nxt, *rest = case.snapshot_args(0)
    fp.snapshot(cur[:, pick], nxt[:, pick] if nxt is not None else None, *rest, sync=True)
    return fp.get_state(), [fp.tuning(s) for s in (0, 1)]


@pytest.mark.parametrize("name", ["c1_asa128", "c1_asa256", "c4_asa512"])
def test_packed_from_64_tracers_on_across_the_line(name):
    case = Case(name)
    fp = native.TracerFP(case.cfg, path="fused")
    states = []
    try:
        for n in (64, 63, 64, 63, 200):
            state, tunes = _run(fp, case, n)
            states.append((n, state))
            for t in tunes:
                timed = [v for v in t["variant_ms"].values() if v is not None]
                assert t["tuned"] == 1
                if n >= 64:
                    assert t["solver"] == "thomas-scan-packed" and not timed
                else:
                    assert t["solver"] != "thomas-scan-packed" and timed
    finally:
        fp.close()
    (_, a), (_, b), (_, a2), (_, b2), (_, c) = states
    for s in (0, 1):
        assert np.array_equal(a[s], a2[s]) and np.array_equal(b[s], b2[s])   # either side again
        assert np.array_equal(a[s], c[s][:64])                               # a larger run of the same tracers
        if np.any(a[s]):
            assert rel_err(b[s], a[s][:63]) <= 1e-10


def test_packed_is_not_calibrated_at_16384_tracers():
    case = Case("c1_asa128")
    fp = native.TracerFP(case.cfg, path="fused")
    try:
        _, tunes = _run(fp, case, 16384)
    finally:
        fp.close()
    for t in tunes:
        assert t["tuned"] == 1 and t["solver"] == "thomas-scan-packed"
        assert all(v is None for v in t["variant_ms"].values())
