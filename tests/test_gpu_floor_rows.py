"""Systems with rows below the floor of the diffusion coefficient (1e-200), which
the factor kernel takes by a copy of its face loop that knows their forms: what
shares a warp with them keeps its bits, and they do not cost the call more than
the rows are worth.  Their values are held against the oracle in
test_gpu_factor.py."""
import numpy as np
import pytest
import torch

from conftest import load_package

load_package()
from croma_fp_b200 import config, native, synth  # noqa: E402

pytestmark = pytest.mark.gpu

LOW = dict(pmin=-3.2, pemin=-3.1)   # exp(-1/p) underflows in the lowest bins


def _run(cfg, n, quiet, path="fused"):
    """The spectra after a snapshot; tracers in `quiet` have no turbulence, so the off form, which no bin takes to the floor."""
    w = synth.Workload(cfg, n, 100, seed=31)
    cur, nxt, *when = w.snapshot_args(41)
    cur, nxt = cur.copy(), nxt.copy()
    cur[5, quiet] = nxt[5, quiet] = 0.0
    fp = native.TracerFP(cfg, path=path)
    try:
        gp, ge = fp.grid(0), fp.grid(1)
        crp, cre = synth.initial_state((gp[0], gp[1]), (ge[0], ge[1]), n, cfg.species)
        fp.set_state(crp, cre, mass=w.mass)
        fp.snapshot(cur, nxt, *when, sync=True)
        return fp.get_state()
    finally:
        fp.close()


# one segment slot a launch (eta cap, one segment): neighbouring tracers share a warp below 512 bins
@pytest.mark.parametrize("nb,n,path,kw", [(128, 67, "fused", dict(eta_dpp_cap=1e-3)),
                                          (128, 67, "plain", dict(eta_dpp_cap=1e-3)),
                                          (128, 67, "fused", dict(coeff_interp_max_segments=1)),
                                          (256, 65, "fused", dict(eta_dpp_cap=1e-3))])
def test_neighbours_of_floor_rows_keep_their_bits(nb, n, path, kw):
    cfg = config.config1(nb=nb, nsub_max=16, dpp_mode="asa", **LOW, **kw)
    quiet = np.arange(n) % 3 != 1
    every = np.ones(n, bool)
    mixed, alone = _run(cfg, n, quiet, path), _run(cfg, n, every, path)
    for a, b in zip(mixed, alone):
        assert np.all(np.isfinite(a)) and np.array_equal(a[quiet], b[quiet])
    assert np.any(mixed[1][~quiet] != alone[1][~quiet])


@pytest.mark.parametrize("nb,n", [(128, 4096), (512, 1024)])
def test_floor_rows_cost_no_multiple(nb, n):
    """Tolerance: the grid below p = 1e-3 changes the coefficients' part of a call, under half of it, whose rows take
    some selects more and Coulomb terms in their slower range, so far less than a second call; 3 to 4 calls when those
    systems' rows were formed one by one."""
    def time(**grid):
        cfg = config.config1(nb=nb, nsub_max=500, dpp_mode="asa", **grid)
        w = synth.Workload(cfg, n, 100, seed=3)
        fp = native.TracerFP(cfg, path="fused")
        try:
            gp, ge = fp.grid(0), fp.grid(1)
            crp, cre = synth.initial_state((gp[0], gp[1]), (ge[0], ge[1]), n, cfg.species)
            fp.set_state(crp, cre, mass=w.mass)
            cur, nxt, *when = w.snapshot_args(41)
            cur, nxt = (torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (cur, nxt))
            torch.cuda.synchronize()
            stream, times = torch.cuda.ExternalStream(fp.stream()), []
            for _ in range(8):
                e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
                e[0].record(stream)
                fp.snapshot(cur.data_ptr(), nxt.data_ptr(), *when, sync=False)
                e[1].record(stream)
                e[1].synchronize()
                times.append(e[0].elapsed_time(e[1]))
            return min(times)
        finally:
            fp.close()

    assert time(**LOW) <= 2.0 * time()
