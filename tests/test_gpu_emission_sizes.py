"""The resident emission over run sizes: a tracer's emissivities do not depend
on how many others the run holds -- bit for bit the same with 37 tracers
(32-row GEMM tiles, frequencies split over blocks, blocks whose tracers span
many log-B planes) and with 20,011 (128-row tiles, unsplit, staged planes) --
and the synchrotron sums equal the interpolated table's in numpy on spectra
with cut-offs, at fields below, inside and above the table's range."""
import numpy as np
import pytest

from conftest import load_package

load_package()
from croma_fp_b200 import config, native, synth  # noqa: E402

pytestmark = pytest.mark.gpu

SETUP = dict(nfreq=7, nu_min_s=7.0, nu_max_s=10.0, ntheta_pitch=32, nlogb=48, logb_min=-3.0, logb_max=1.0,
             nbins_ic=70, nu_min_ic=17.0, nu_max_ic=29.0, nbins_gamma=9, egamma_min=-3.0, egamma_max=4.0, nbins_nu=64,
             enu_min=-3.0, enu_max=4.0)


def _run(cfg, crp, cre, bg, table=False):
    fp = native.TracerFP(cfg, path="fused")
    try:
        fp.emission_setup(**SETUP)
        fp.set_state(crp, cre, mass=np.full(crp.shape[0], 1e7))
        out = fp.emission_run(bg, 0.4)
        tab = fp.emission_table("synch", (SETUP["nlogb"], SETUP["nfreq"], cfg.nb)) if table else None
    finally:
        fp.close()
    return out, tab


@pytest.mark.parametrize("nb", [128, 512])
def test_run_size_does_not_change_a_bit(nb):
    cfg = config.config1(nb=nb)
    n, big = 37, 20011
    rng = np.random.default_rng(nb)
    fp = native.TracerFP(cfg, path="fused")
    gp, ge = fp.grid(0), fp.grid(1)
    fp.close()
    crp, cre = synth.initial_state((gp[0], gp[1]), (ge[0], ge[1]), n, cfg.species)
    crp *= rng.uniform(0.5, 2.0, (n, 1))
    cre *= np.exp(-ge[0] / 10.0 ** rng.uniform(1.0, 6.0, (n, 1)))
    cre[3, nb // 3:] = 0.0
    bg = synth.background(n, 12, 5)
    bg[2, :4] = (1e-12, 1e-3, 1e-9, 1e-5)      # below, above and at the ends of the table
    small, tab = _run(cfg, crp, cre, bg, table=True)
    pick = rng.integers(0, n, big)
    pick[:n] = np.arange(n)
    large, _ = _run(cfg, crp[pick], cre[pick], np.ascontiguousarray(bg[:, pick]))
    for k in small:
        assert np.all(np.isfinite(small[k])) and np.array_equal(large[k], small[k][pick]), k

    # the synchrotron shape in numpy: table interpolated in log K, bins 2 .. first non-positive N[j + 1]
    inv = (SETUP["nlogb"] - 1) / (SETUP["logb_max"] - SETUP["logb_min"])
    u = (np.log10(bg[2] / 1e-6) - SETUP["logb_min"]) * inv
    ib = np.clip(np.floor(u).astype(int), 0, SETUP["nlogb"] - 2)
    tw = np.clip(u - ib, 0.0, 1.0)[:, None, None]
    a, b = tab[ib], tab[ib + 1]
    both = (a > 0) & (b > 0)
    with np.errstate(divide="ignore", invalid="ignore"):
        K = np.where(both & (tw > 0) & (tw < 1), np.exp((1 - tw) * np.log(a) + tw * np.log(b)), (1 - tw) * a + tw * b)
    j = np.arange(nb)
    stop = np.array([next((m for m in range(2, nb - 1) if not row[m + 1] > 0.0), nb - 1) for row in cre])
    use = (j >= 2) & (j < stop[:, None])
    want = bg[2][:, None] * np.einsum("tj,tfj->tf", np.where(use, cre * ge[1], 0.0), K)
    # the prefactor is one number; each value is a sum of at most nb positive
    # terms of ~1e-15 relative error each (and exactly zero where all are)
    want *= small["syn"][0, 0] / want[0, 0]
    assert np.all(np.abs(small["syn"] - want) <= 1e-12 * want)
