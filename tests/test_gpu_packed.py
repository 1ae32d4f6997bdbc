"""The packed steps kernel (the FP64 on-chip path from 64 tracers on): the
golden fixtures tiled past that line, at tracer counts that leave a warp's
groups, a block's warps and the order kernels' blocks partly filled, against
the reference's spectra (bar 1e-10, as everywhere), each copy of a tracer bit
for bit the same wherever it landed; chunked runs bit for bit the unchunked
one; and a tracer with NaN spectra leaving its warp's others alone."""
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


def _tiled(case, n, limit=None, spoil=None):
    d = case.d
    pick = np.arange(n) % d["crp0"].shape[0]
    crp, cre = d["crp0"][pick], d["cre0"][pick]
    if spoil is not None:
        cre[spoil] = np.nan
    fp = native.TracerFP(case.cfg, path="fused")
    try:
        if limit is not None:
            fp.set_workspace_limit(limit)
        fp.set_state(crp, cre, mass=d["mass"][pick])
        cur, nxt, *rest = case.snapshot_args(0)
        fp.snapshot(cur[:, pick], nxt[:, pick] if nxt is not None else None, *rest, sync=spoil is None)
        solver = fp.tuning(1)["solver"]
        out = fp.get_state() if spoil is None else _raw(fp)
    finally:
        fp.close()
    assert solver == "thomas-scan-packed"
    return pick, out


def _raw(fp):
    """The spectra whatever the error word says."""
    crp, cre = np.empty((fp.ntracer, fp.nb)), np.empty((fp.ntracer, fp.nb))
    try:
        fp.get_state(crp, cre)
    except native.CromaError:
        pass
    return crp, cre


# uneven sub-steps, a centred window (on and off sets), both with an eta cap's
# one-segment launches, no interpolation, and every bin count with secondaries;
# counts: just past the line, an odd one, and (128 bins) past the one-block order
@pytest.mark.parametrize("name,n", [("c0_direct", 65), ("c0_narrow", 67), ("c0_narrow", 16417), ("c0_last", 64),
                                    ("c1_asa128", 131), ("c1_narrow_window", 77), ("c2_ttd_spect_window", 95),
                                    ("c1_etacap", 101), ("c1_asa256", 65), ("c1_asa256", 97), ("c4_asa512", 66)])
def test_packed_matches_reference(name, n):
    c = Case(name)
    pick, (crp, cre) = _tiled(c, n)
    first = np.array([np.flatnonzero(pick == p)[0] for p in pick])
    assert np.array_equal(cre, cre[first]) and np.array_equal(crp, crp[first])
    assert rel_err(cre, c.d["cre_0"][pick]) <= 1e-10
    if np.any(c.d["crp_0"]):
        assert rel_err(crp, c.d["crp_0"][pick]) <= 1e-10


@pytest.mark.parametrize("name,n,limit", [("c0_narrow", 203, 9e6), ("c1_asa256", 75, 8e6), ("c4_asa512", 66, 9e6)])
def test_chunks_do_not_change_a_bit(name, n, limit):
    c = Case(name)
    _, (crp, cre) = _tiled(c, n)
    _, (crp2, cre2) = _tiled(c, n, limit=limit)
    assert np.array_equal(crp, crp2) and np.array_equal(cre, cre2)


@pytest.mark.parametrize("name", ["c0_narrow", "c1_asa256"])
def test_nan_tracer_stays_alone(name):
    c = Case(name)
    _, (crp, cre) = _tiled(c, 70)
    _, (crp2, cre2) = _tiled(c, 70, spoil=41)
    keep = np.arange(70) != 41
    assert np.array_equal(cre[keep], cre2[keep]) and np.array_equal(crp, crp2)
    assert np.all(np.isnan(cre2[41]))
