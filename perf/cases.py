"""The work that users of this framework have it do, as cases that can be timed.

A case is one pass through a public entry point:

  snapshot  TracerFP.snapshot: one snapshot of resident spectra from device
            backgrounds (the call of a run's main loop)
  pipeline  the whole per-snapshot sequence on resident spectra:
            TracerFP.dsa_inject, emission_run_device, snapshot
  host      TracerFP.snapshot_host: host spectra to host spectra
  bucket    run_tracer_pipeline of the reference-compatible C ABI: one bucket
            and segment from host arrays to host arrays, as a CROMA host calls it

The configurations are this repository's own (config.config0, 1, 2, 4 and
tracer_10k); inputs follow the distributions of its synthetic histories.
Successive passes on a state walk along the run's timeline (every pass has its
own redshifts, so its own inverse-Compton cooling row) and start the run again
from the seed spectra at the timeline's end.
"""
import ctypes as C
import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
DEVICE = "cuda"
F64 = torch.float64

NSNAP, FIRST = 100, 30      # the timeline z = 1 .. 0 and the snapshot that a state starts at
NBG = 4                     # distinct background snapshots of a state, used in turn
MASS = 1.0e7                # tracer mass, solar masses
BUCKET_STEPS = 31           # sub-steps of one segment of a capped snapshot (500 / 16)
SHOCK_FRACTION = 0.05


def load_package():
    """The package (its folder's name is not an identifier)."""
    if "croma_fp_b200" not in sys.modules:
        folder = os.path.join(ROOT, "croma-fp_b200")
        spec = importlib.util.spec_from_file_location("croma_fp_b200", os.path.join(folder, "__init__.py"),
                                                      submodule_search_locations=[folder])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["croma_fp_b200"] = mod
        spec.loader.exec_module(mod)
    from croma_fp_b200 import config, native, ref_abi
    return config, native, ref_abi


# ---------------------------------------------------------------- the cases
def _case(name, kind, cfg, nb, nt, path="fused", reacc="off"):
    return {"name": name, "kind": kind, "cfg": cfg, "nb": nb, "ntracer": nt, "path": path, "reacc": reacc}


def listed():
    return [
        # the smallest run: a few tracers followed on their own, where latency and launches count
        _case("snap128_64", "snapshot", "direct", 128, 64),
        # uneven sub-steps (nsub 11 .. 500): most tracers are done early
        _case("snap128_uneven", "snapshot", "uneven", 128, 30011),
        # the reference's run of its 10,000 real tracers: centred reacceleration window, eta cap, no sub-step cap
        _case("snap128_window", "snapshot", "tracer_10k", 128, 10000),
        # the electron-only precision workload, TTD reacceleration
        _case("snap128_ttd", "snapshot", "ttd", 128, 131072),
        # protons and electrons with secondaries: an odd count that does not fill the chip
        _case("snap256_999", "snapshot", "asa", 256, 999),
        # the batching workload at its own size
        _case("snap256_65536", "snapshot", "asa", 256, 65536),
        # the finest grid, evolve alone
        _case("snap512_4096", "snapshot", "asa", 512, 4096),
        # the whole pipeline for a small run, shocks reaccelerating the spectra
        _case("pipe512_1500", "pipeline", "asa", 512, 1500, reacc="positive_delta"),
        # the whole pipeline in bulk: the largest case
        _case("pipe512_131072", "pipeline", "asa", 512, 131072),
        # the per-step path (the reference's data contract, TracerFP's default)
        _case("plain256_4096", "snapshot", "asa", 256, 4096, path="plain"),
        # spectra kept by a host program
        _case("host256_16384", "host", "asa", 256, 16384),
        # the drop-in call of a CROMA host
        _case("bucket256_2048", "bucket", "asa", 256, 2048),
    ]


def draw(rng):
    """One more case of the same ranges; tracer counts spread over their logarithm, odd ones among them."""
    kind = rng.choice(["snapshot", "snapshot", "snapshot", "snapshot", "pipeline", "pipeline", "plain", "fp32r", "host",
                       "bucket"])
    nb = rng.choice([128, 256, 512])
    top = {"snapshot": 131072, "pipeline": 131072, "plain": 16384, "fp32r": 32768, "host": 32768, "bucket": 8192}[kind]
    top = top * 128 // nb if kind != "pipeline" else top * 128 // max(nb, 256)
    n = int(round(math.exp(rng.uniform(math.log(64), math.log(top)))))
    cfg = "asa" if kind in ("pipeline", "bucket") else rng.choice(["asa", "asa", "direct", "ttd", "uneven"])
    if kind == "snapshot" and nb == 128 and rng.random() < 0.25:
        cfg, n = "tracer_10k", min(n, 32768)
    reacc = rng.choice(["off", "off", "positive_delta", "drury83"]) if kind == "pipeline" else "off"
    c = _case("", "snapshot" if kind in ("plain", "fp32r") else kind, cfg, nb, n,
              path=kind if kind in ("plain", "fp32r") else "fused", reacc=reacc)
    del c["name"]
    return c


def run_config(case):
    """The RunConfig fields of a case (config.py's configurations at the case's bin count)."""
    base = dict(nb=case["nb"], nsub_max=500)
    return {"asa": ("config1", base), "direct": ("config0", base), "ttd": ("config2", base),
            "uneven": ("config0", dict(base, pemin=1.0, pemax=3.0)),
            "tracer_10k": ("tracer_10k", dict(nb=case["nb"]))}[case["cfg"]]


def both_species(case):
    return case["cfg"] == "asa"


# ---------------------------------------------------------------- inputs, from the seed alone
K_C, K_GYR, K_MP, K_ME, K_GEV, K_KPC, K_MPC = 2.999e10, 3.1536e16, 0.938, 0.511e-3, 1.6e-3, 3.0857e21, 3.0857e24
KB_EV, MU = 8.62e-5, 0.59


def timeline():
    """Redshifts and cosmic-time steps (Gyr) of the snapshots: flat LCDM, H0 = 70 km/s/Mpc, Omega_m = 0.3."""
    z = np.linspace(1.0, 0.0, NSNAP)
    t = 2.0 / (3.0 * math.sqrt(0.7)) * np.arcsinh(math.sqrt(0.7 / 0.3) * (1.0 + z) ** -1.5) / (7.0e6 / K_MPC) / K_GYR
    return z, np.diff(t), t - t[0]


def backgrounds(nt, gen, nsnap=NBG):
    """[nsnap][8][nt]: n_gas, kT, B, div v, L_turb, dv, c_s, beta of the synthetic histories' distributions."""
    def log_uniform(lo, hi):
        u = torch.rand((nsnap, nt), generator=gen, device=DEVICE, dtype=F64)
        return 10.0 ** (math.log10(lo) + (math.log10(hi) - math.log10(lo)) * u)

    n_gas, temp, b_ug = log_uniform(1e-5, 1e-2), log_uniform(1e6, 1e8), log_uniform(0.01, 10.0)
    div_v = 1e-17 * torch.randn((nsnap, nt), generator=gen, device=DEVICE, dtype=F64)
    l_cm = 150.0 * K_KPC
    cs = torch.sqrt(5.0 / 3.0 * KB_EV * temp / (MU * 0.938e9)) * K_C
    dv = torch.minimum(log_uniform(1e-18, 1e-16) * l_cm, 0.5 * cs)
    b = torch.maximum(torch.sqrt(4.0 * math.pi * 0.05 * n_gas * (1.6e-24 * MU) * dv * dv), b_ug * 1e-6)
    beta = n_gas * KB_EV * temp * 1.6e-12 / (b * b / (8.0 * math.pi))
    return torch.stack([n_gas, KB_EV * temp * 1e-9, b, div_v * K_GYR, torch.full_like(b, l_cm / K_MPC), dv, cs, beta],
                       dim=1).contiguous()


def momenta(lo, hi, nb):
    """p and dp of the log grid (momentum_bin: 10^a, a accumulated; the last dp reaches two steps up, as there)."""
    da, a, v = (hi - lo) / nb, lo - (hi - lo) / nb, []
    for _ in range(nb + 2):
        v.append(10.0 ** a)
        a += da
    q = np.array(v + [10.0 ** a])
    p = q[1:nb + 1]
    dp = 0.5 * (q[2:nb + 2] - q[:nb])
    dp[-1] = 0.5 * (q[nb + 2] - q[nb - 1])
    return p, dp


def grids(case):
    fields = {"direct": (-2, 6, -1, 6), "asa": (-2, 6, -1, 6), "ttd": (-2, 6, -1, 6), "uneven": (-2, 6, 1, 3),
              "tracer_10k": (-1, 8, -0.5, 6)}[case["cfg"]]
    return momenta(fields[0], fields[1], case["nb"]), momenta(fields[2], fields[3], case["nb"])


def spectra(case, gen):
    """Seed spectra [nt][nb] (protons, electrons): power laws with the reference's template cut-offs, each tracer's
    slope, amplitude and upper cut-off its own, as tracers in the middle of a run have them."""
    nt = case["ntracer"]
    (pp, _), (pe, _) = grids(case)

    def u(lo, hi):
        return lo + (hi - lo) * torch.rand((nt, 1), generator=gen, device=DEVICE, dtype=F64)

    out = []
    for p, inj, amp in ((pp, 1.0, 1.0e58), (pe, 10.0, 1.0e57)):
        x = torch.from_numpy(p).to(DEVICE)[None, :]
        slope, scale, cut = u(2.2, 2.8), 10.0 ** u(-1.0, 1.0), 10.0 ** u(4.0, 6.0)
        out.append(amp * scale * torch.exp(-slope * torch.log(x) - inj / x - x / cut))
    if not both_species(case):
        out[0] = torch.zeros_like(out[0])
    return out


def shock_fields(bg, gen):
    """Shock fields of one snapshot: Mach U[2, 5] on 5 % of the tracers, the upstream state the tracer's own."""
    nt = bg.shape[1]
    hit = torch.rand(nt, generator=gen, device=DEVICE, dtype=F64) < SHOCK_FRACTION
    mach = torch.where(hit, 2.0 + 3.0 * torch.rand(nt, generator=gen, device=DEVICE, dtype=F64), 0.0)
    return {"mach": mach, "prestemp": bg[1] * 1e9 / KB_EV, "presden": bg[0] * (1.6e-24 * MU),
            "shock_side_code": torch.where(hit, 1.0, 99.0).to(F64)}


def inputs(case, seed):
    gen = torch.Generator(device=DEVICE)
    gen.manual_seed(int(seed))
    bg = backgrounds(case["ntracer"], gen)
    crp, cre = spectra(case, gen)
    return gen, bg, crp, cre


# ---------------------------------------------------------------- states and passes
class DeviceArray:
    """A float64 device block of a context as torch sees it; it keeps the context open."""

    def __init__(self, ptr, shape, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f8", "data": (ptr, False), "version": 3}


class State:
    """What a program keeps between the passes of one case."""

    def __init__(self, case):
        self.case, self.k = case, 0
        self.z, self.dt, self.elapsed = timeline()

    def now(self):
        """(background pair, snapshot index) of the next pass."""
        k = self.k
        self.k += 1
        return k % NBG, (k + 1) % NBG, FIRST + k % (NSNAP - 1 - FIRST)


def _resident(case, seed):
    config, native, _ = load_package()
    s = State(case)
    name, fields = run_config(case)
    gen, s.bg, s.crp0, s.cre0 = inputs(case, seed)
    nt, nb = case["ntracer"], case["nb"]
    s.fp = native.TracerFP(getattr(config, name)(**fields), path=case["path"])
    s.fp.set_state_broadcast(nt, np.zeros(nb), np.zeros(nb), MASS)
    s.stream = torch.cuda.ExternalStream(s.fp.stream())
    a, b = s.fp.state_device()
    s.crp = torch.as_tensor(DeviceArray(a, (nt, nb), s.fp), device=DEVICE)
    s.cre = torch.as_tensor(DeviceArray(b, (nt, nb), s.fp), device=DEVICE)
    torch.cuda.synchronize()
    s.crp.copy_(s.crp0)
    s.cre.copy_(s.cre0)
    if case["kind"] == "pipeline":
        s.fp.set_dsa(config.DsaParams())
        s.fp.emission_setup(**native.EMISSION_CONFIG4)
        s.shocks = [shock_fields(s.bg[i], gen) for i in range(NBG)]
        s.eps = {k: torch.empty((nt, 64), dtype=F64, device=DEVICE) for k in ("syn", "ic", "gamma", "nu")}
    torch.cuda.synchronize()
    return s


def _host(case, seed):
    config, native, _ = load_package()
    s = State(case)
    name, fields = run_config(case)
    _, bg, crp, cre = inputs(case, seed)
    nt, nb = case["ntracer"], case["nb"]
    s.fp = native.TracerFP(getattr(config, name)(**fields), path=case["path"])
    s.bg = [np.ascontiguousarray(x) for x in bg.cpu().numpy()]
    s.crp, s.cre = (x.cpu().pin_memory().numpy() for x in (crp, cre))   # page-locked, so that the copies overlap
    s.mass = np.full(nt, MASS)
    return s


ABI = {}   # a program has one binding per bin count


class Workspace:
    """A pipeline workspace of the C ABI."""

    def __init__(self, abi):
        self.abi, self.ws = abi, abi.lib.cuda_pipeline_workspace_create()
        if not self.ws:
            raise RuntimeError(abi.error())

    def __del__(self):
        self.abi.lib.cuda_pipeline_workspace_destroy(self.ws)


def _bucket(case, seed):
    config, _, ref_abi = load_package()
    s = State(case)
    nt, nb = case["ntracer"], case["nb"]
    s.abi = ABI.setdefault(nb, None) or ref_abi.RefAbi(nb)
    ABI[nb] = s.abi
    if s.abi.lib.croma_b200_set_model(1, 1, 0.3, 0.0) != 0:   # ASA, as config1
        raise RuntimeError(s.abi.error())
    _, bg, crp, cre = inputs(case, seed)
    s.crp0, s.cre0 = crp.cpu().numpy(), cre.cpu().numpy()
    (pp, dpp), (pe, dpe) = grids(case)
    rp, re = pp[1] / pp[0], pe[1] / pe[0]
    s.gp = s.abi.grid(pp, dpp, K_MP * np.sqrt(1 + pp * pp), pp[0] / rp, pp[-1] * rp)
    s.ge = s.abi.grid(pe, dpe, K_ME * np.sqrt(1 + pe * pe), pe[0] / re, pe[-1] * re)
    row = ic_row(float(s.z[FIRST]), pe)
    s.ric = np.ascontiguousarray(np.repeat(row[:, None], nt, axis=1))
    s.edge = np.full(nt, row[0]), np.full(nt, row[-1])
    s.mass, s.dis = np.full(nt, MASS), np.zeros(nt, np.uint8)
    s.f = [np.ascontiguousarray(x) for x in bg[0].cpu().numpy()]
    ci = ref_abi.FpCoeffBatchInput()
    ci.ncell, ci.epmax = nt, 1.0e7
    for name, x in zip(("n_gas", "kbt", "b_field", "divv_gyr", "l_turb_mpc", "dv_imc", "cs", "beta_pl"), s.f):
        setattr(ci, name, ref_abi.dptr(x))
    ci.tracer_mass_msun, ci.disable_adiabatic = ref_abi.dptr(s.mass), ref_abi.u8ptr(s.dis)
    ci.rad_ic_batch, ci.rad_ic_m1, ci.rad_ic_p1 = ref_abi.dptr(s.ric), ref_abi.dptr(s.edge[0]), ref_abi.dptr(s.edge[1])
    s.ws = Workspace(s.abi)
    p = s.abi.PipelineInput()
    p.ncell, p.nstep = nt, BUCKET_STEPS
    p.fp_cadence_steps = p.diff_cadence_steps = p.adv_cadence_steps = 1
    p.on_start_step, p.on_end_step = 0, BUCKET_STEPS
    p.dt, p.epmax, p.psi_value, p.mach_limit_value, p.transport_mode = float(s.dt[FIRST]) / 500.0, 1.0e7, 0.5, 0.5, 1
    p.crp_grid, p.cre_grid, p.coeff_in = C.pointer(s.gp), C.pointer(s.ge), C.pointer(ci)
    p.crp_init, p.cre_init, p.workspace = ref_abi.dptr(s.crp0), ref_abi.dptr(s.cre0), s.ws.ws
    s.crp, s.cre = np.empty_like(s.crp0), np.empty_like(s.cre0)
    s.out = ref_abi.dptr(s.crp), ref_abi.dptr(s.cre)
    s.ci, s.pin, s.times = ci, p, ref_abi.FpCudaPipelineTimes()
    return s


def prepare(case, seed):
    return {"snapshot": _resident, "pipeline": _resident, "host": _host, "bucket": _bucket}[case["kind"]](case, seed)


def run(s):
    kind = s.case["kind"]
    if kind == "bucket":
        if s.abi.lib.run_tracer_pipeline(C.byref(s.pin), None, *s.out, None, None, None, C.byref(s.times)) != 0:
            raise RuntimeError(s.abi.error())
        return {"crp": s.crp, "cre": s.cre}
    cur, nxt, i = s.now()
    when = float(s.z[i]), float(s.z[i + 1]), True, float(s.dt[i]), float(s.elapsed[i])
    if kind == "host":
        s.fp.snapshot_host(s.crp, s.cre, s.bg[cur], s.bg[nxt], *when, mass=s.mass)
        return {"crp": s.crp, "cre": s.cre}
    if i == FIRST and s.k > 1:   # the run starts again
        with torch.cuda.stream(s.stream):
            s.crp.copy_(s.crp0)
            s.cre.copy_(s.cre0)
    out = {"crp": s.crp, "cre": s.cre}
    bg = s.bg[cur].data_ptr()
    if kind == "pipeline":
        shocks = {k: v.data_ptr() for k, v in s.shocks[cur].items()}
        s.fp.dsa_inject(dict(shocks, on_device=1, has_dsa=0), 1.0, when[3], "tracer_state", s.case["reacc"])
        s.fp.emission_run_device(bg, when[0], **{k: t.data_ptr() for k, t in s.eps.items()})
        out.update(s.eps)
    s.fp.snapshot(bg, s.bg[nxt].data_ptr(), *when, sync=False)
    return out


def work(case):
    """Bytes: spectra in and out, the backgrounds (and shock fields, emissivities) once.  Flops: three multiply-adds
    a row and sub-step (right-hand side and the two sweeps of a factored solve), ~40 operations a row and segment for
    its coefficients, the secondary source's half-filled product per segment, the emissivities' products."""
    nt, nb = case["ntracer"], case["nb"]
    species = 2 if both_species(case) else 1
    steps = {"uneven": 90, "tracer_10k": 700}.get(case["cfg"], 500)
    nseg = 16 if case["cfg"] != "uneven" else 8
    if case["kind"] == "bucket":
        steps, nseg = BUCKET_STEPS, 1
    nbytes = 8.0 * nt * (2 * species * nb + 16)
    flops = float(nt) * nb * (species * (6.0 * steps + 40.0 * nseg) + (nseg * nb if species == 2 else 0))
    if case["kind"] == "pipeline":
        nbytes += 8.0 * nt * (4 * 64 + 4)
        flops += float(nt) * nb * 64 * (3 * 2 + 4)
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------- the same in plain torch, 64 bits
def ic_row(z, p):
    """Inverse-Compton cooling rate per bin at redshift z: the CMB integral of rad_IC_cool / b_IC (GeV-free units)."""
    meg, re = 9.11e-28, 2.82e-13
    pref = 8.0 * math.pi * K_C ** 3 * (meg / 6.63e-27) ** 3

    def density(e):
        x = e * meg * K_C * K_C / (1.38e-16 * 2.757 * (1.0 + z))
        return pref * e * e / (np.exp(x) - 1.0)

    def slope(e):
        t = 1.38e-16 * 2.757 * (1.0 + z)
        ex = math.exp(e * meg * K_C * K_C / t)
        return pref * e / (ex - 1.0) * (2.0 - e * meg * K_C * K_C * ex / (t * (ex - 1.0)))

    tiny, ep = 10.0 ** -5.5, 1.38e-16 / (meg * 3.0e10 * 3.0e10) * 2.725 * (1.0 + z)
    ends = []
    for new in (0.01 * ep, 10.0 * ep):
        e = 1.0
        while abs(new - e) > tiny * e:
            e = new
            new = e - (float(density(e)) - float(density(ep)) * tiny) / slope(e)
        ends.append(new)
    da = 0.05
    n = int(round((math.log10(ends[1]) - math.log10(ends[0])) / da))
    e0 = torch.from_numpy(np.concatenate([[ends[0]], 10.0 ** (math.log10(ends[0]) + da * np.arange(1, n + 1))]))[None, :]
    g = torch.sqrt(1.0 + torch.from_numpy(p) ** 2)[:, None]
    emax = g * 4.0 * e0 * g / (1.0 + 4.0 * e0 * g)
    count = torch.round((torch.log10(emax) - torch.log10(e0)) / da)

    def kernel(eps):
        kap = eps / (4.0 * e0 * g * (g - eps))
        t = 4.0 * e0 * kap * g
        k = torch.where(kap > 0, kap, torch.ones_like(kap))
        c = 2 * k * torch.log(k) + (1 + 2 * k) * (1 - k) + t * t / (2 * (1 + t)) * (1 - k)
        return torch.where(kap > 0, 2.0 * math.pi * re * re * K_C / (g * g * e0) * c, torch.zeros_like(kap))

    eps, total = e0 + 0 * g, torch.zeros_like(emax)
    val = kernel(eps)
    for i in range(1, int(count.max()) + 1):
        new = 10.0 ** (torch.log10(e0) + da * i) + 0 * g
        vnew = kernel(new)
        total = torch.where(i <= count, total + 0.5 * (eps * val + new * vnew) * (new - eps), total)
        eps, val = new, vnew
    f = total * torch.from_numpy(density(e0.numpy()))
    return (0.5 * (f[:, 1:] + f[:, :-1]) * (e0[:, 1:] - e0[:, :-1])).sum(1).numpy() * K_GYR


def pp_cross_section(p):
    """Kamae's inelastic pp -> pion cross section (all pions), p in GeV/c, with the reference's parameters."""
    e = np.sqrt(K_MP * K_MP + p * p)
    t, x = e - K_MP, np.log10(p)
    bump = 23.10 + 6.454 * x ** 2 - 5.764 * x ** 3 - 23.63 * np.exp(-94.75 * (x + 0.02667) ** 2)
    nond = np.select([p < 1, p < 1.3, p < 2.4, p < 10],
                     [0, 0.57 * np.abs(x / 0.1176) ** 1.2 * bump,
                      (11.34 * np.abs(0.3829 - x) + 23.72 * np.abs(0.1176 - x)) / (0.3829 - 0.1176), bump],
                     28.5 - 6.133 * x + 1.464 * x ** 2)
    dd = 1.498 + 2.0 * np.log10(30.0 * np.maximum(x - 0.25, 1e-300)) + 3.155 * x ** 2 - 1.042 * x ** 3
    diff = np.select([p < 2.25, p < 3.2, p < 100], [0, np.sqrt(np.abs(x - 0.3522) / 0.1530) * dd, dd], 5.922 + 1.632 * x)
    dres = np.select([e < 1.4, e < 1.6, e < 1.8, e < 10],
                     [0, 0.0834 * e ** 10, 9.5 * np.exp(-5.5 * (e - 1.68) ** 2), 3134.0 * e ** -10.0], 0)
    res = np.select([e < 1.6, e < 1.9, e < 2.3, e < 20],
                    [0, 0.0004257 * e ** 14, 4.5 * np.exp(-7.0 * (e - 2.1) ** 2), 503.5 * e ** -6.0], 0)
    r0 = 1.0 / (0.007 + 0.1 * np.log(t) / t + 0.3 / t ** 2)
    rp = 1.0 / (0.00717 + 0.0652 * np.log(t) / t + 0.162 / t ** 2)
    rm = 1.0 / (0.00456 + 0.0846 / t ** 0.5 + 0.577 / t ** 1.5)
    return (nond + diff + dres + res) * 1e-27 * (1.0 + rp / r0 + rm / r0)


def coulomb_p(n, kbt, p):
    """Proton Coulomb loss rate at momenta p for gas density n and temperature kbt."""
    gamma = torch.sqrt(1.0 + p * p)
    k = lambda x: 0.5 * math.sqrt(math.pi) * torch.erf(torch.sqrt(x)) - torch.sqrt(x) * torch.exp(-x)  # noqa: E731
    xp = (gamma * K_MP - K_MP) / kbt
    thermal = 1.0 - kbt / (2.0 * K_MP * (gamma - 1.0))
    s = k(xp * (K_ME / K_MP)) + k(xp) * (K_ME / K_MP)
    return K_GYR * K_C / (K_MP * K_GEV) * s * n * (1.0 + p * p) / (p * p) * thermal.clamp(min=0.0) * 3.5e-29


def coulomb_e(n, p):
    return 3.05e-29 * n * (1.0 + torch.log(p / n) / 74.8) / (K_ME * K_GEV) * K_C * K_GYR * (1.0 + p * p) / (p * p)


def synch(b, p):
    return 4.8e-4 * p * p * (b * 1e6 / 3.2) ** 2 * 9.11e-28 * 3.0e10 * 3.1536e16


def schedule(case, bg, dt, row, pp, pe):
    """Sub-steps, sub-steps with the reacceleration on, and coefficient segments of every tracer."""
    n, kbt, b, dvv, lt, dv = (bg[k] for k in range(6))
    t = torch.full_like(n, math.inf)
    for p in (pp[0], pp[-1]):
        t = torch.minimum(t, (p / (coulomb_p(n, kbt, p) + dvv * p / 3.0)).abs())
    for p, r in ((pe[0], row[0]), (pe[-1], row[-1])):
        t = torch.minimum(t, (p / (synch(b, p) + r + coulomb_e(n, p) + dvv * p / 3.0)).abs())
    wide = case["cfg"] == "tracer_10k"
    target = torch.minimum((0.5 if wide else 0.25) * t, torch.full_like(t, dt / 10.0))
    scale = 10.0 ** torch.floor(torch.log10(target))
    ladder = torch.tensor([1.0, 1.25, 1.6, 2.0, 2.5, 3.2, 4.0, 5.0, 6.4, 8.0], dtype=F64, device=n.device)
    at = (torch.bucketize(target / scale, ladder, right=True) - 1).clamp(min=0)
    used = torch.minimum(ladder[at] * scale, target)
    nsub = torch.ceil(dt / used).clamp(10.0, 1.0e6).long()
    on = torch.ones_like(n)
    if wide:
        x = 2.0 * (lt * K_MPC / dv / K_GYR) / dt
        bins = torch.tensor([1 / 8, 1 / 4, 1 / 3, 1 / 2, 1.0], dtype=F64, device=n.device)
        on = torch.where(x < 1.0, bins[(x[:, None] - bins[None, :]).abs().argmin(1)], on)
    else:
        nsub = nsub.clamp(max=500)
    non = torch.minimum(torch.floor(nsub.double() * on + 0.5).long().clamp(min=1), nsub)
    nseg = (2 ** torch.floor(torch.log2((nsub // 4).double()))).long().clamp(1, 16)
    return nsub, non, nseg


def face_weights(w):
    """The Chang-Cooper weights of a face: w+ = w / (1 - exp(-w)), w- = w / (exp(w) - 1), by series near 0."""
    a = w.abs()
    small = a < 0.1
    den = 1.0 + w * w / 24.0 + w ** 4 / 1920.0
    big = a / -torch.expm1(-torch.where(small, torch.ones_like(a), a))
    less = big * torch.exp(-a)
    return (torch.where(small, torch.exp(0.5 * w) / den, torch.where(w >= 0, big, less)),
            torch.where(small, torch.exp(-0.5 * w) / den, torch.where(w >= 0, less, big)))


def dpp_rate(case, g):
    """1 / (4 t_acc) of every tracer from its background."""
    n, kbt, b, dvv, lt, dv, cs, beta = g
    mach = torch.minimum(dv / cs, torch.full_like(cs, 0.5))
    big_l = lt * K_MPC
    if case["cfg"] in ("direct", "uneven"):
        tacc = torch.full_like(cs, 0.3)
    elif case["cfg"] == "ttd":
        x = cs / K_C
        theta = x ** 4 / 4.0 + x * x - (1.0 + 2.0 * x * x) * torch.log(x) - 1.25
        tacc = 2.5e-3 / (x * theta) / (mach / 0.5) ** 4 * (big_l / (300.0 * K_KPC)) / (cs / 1.5e8)
    else:
        tacc = math.sqrt(6.0 / 5.0) / 12.0 * (K_C / cs / cs) * big_l / torch.sqrt(beta) / mach ** 3 * 0.125 / K_GYR
    return 0.25 / tacc, tacc


def factor(p, dp, radp, dpp, dt, rate):
    """Thomas factors (1/d, a/d, c/d), each [nb][nt], of the Chang-Cooper matrix."""
    bb = radp - 2.0 / p * dpp
    x = p[1:] - p[:-1]
    wp, wm = face_weights((bb[:-1] + bb[1:]) / (dpp[:-1] + dpp[1:]) * x)
    flow = 0.5 * (dpp[:-1] + dpp[1:]) / x
    k = dt / dp
    a, c, b = torch.zeros_like(bb), torch.zeros_like(bb), 1.0 + dt * rate
    a[1:], c[:-1] = k[1:] * flow * wm, k[:-1] * flow * wp
    b = b.expand_as(bb).clone()
    b[1:] += k[1:] * flow * wp
    b[:-1] += k[:-1] * flow * wm
    inv, h, q = torch.empty_like(b), torch.empty_like(b), torch.empty_like(b)
    for i in range(p.shape[0]):
        d = b[i] - a[i] * q[i - 1] if i else b[i]
        inv[i] = 1.0 / d
        h[i], q[i] = a[i] * inv[i], c[i] * inv[i]
    return inv, h, q


def sweep(f, y):
    """M^-1 y with the factors f."""
    inv, h, q = f
    y = y * inv
    for i in range(1, y.shape[0]):
        torch.addcmul(y[i], h[i], y[i - 1], out=y[i])
    for i in range(y.shape[0] - 2, -1, -1):
        torch.addcmul(y[i], q[i], y[i + 1], out=y[i])
    return y


def exact(case, seed):
    """The spectra after the first pass, by the plain sweeps in 64 bits.  Not restated: the secondary electrons of the
    two-species cases (their source is a table of nested pion integrals), and the whole pipeline, whose shocks change
    the spectra before the update."""
    if case["kind"] == "pipeline":
        return None
    _, bg, crp, cre = inputs(case, seed)
    z, dts, _ = timeline()
    (pp, dpp), (pe, dpe) = grids(case)
    dt, bucket = float(dts[FIRST]), case["kind"] == "bucket"
    row, row1 = (torch.from_numpy(ic_row(float(z[FIRST + k]), pe)).to(DEVICE)[:, None] for k in (0, 1))
    pp, dpp, pe, dpe = (torch.from_numpy(v).to(DEVICE)[:, None] for v in (pp, dpp, pe, dpe))
    nt = case["ntracer"]
    if bucket:
        nsub = non = torch.full((nt,), BUCKET_STEPS, device=DEVICE)
        nseg, step_dt = torch.ones_like(nsub), torch.full((nt,), dt / 500.0, dtype=F64, device=DEVICE)
    else:
        nsub, non, nseg = schedule(case, bg[0], dt, row[:, 0], pp[:, 0], pe[:, 0])
        step_dt = dt / nsub.double()
    steps_all = int(nsub.max()) * (2 if case["cfg"] == "tracer_10k" else 1)
    if 2 * case["nb"] * steps_all > 1_000_000:
        return None
    sp = 0 if both_species(case) else 1
    p, dp = ((pp, dpp), (pe, dpe))[sp]
    if sp == 0:
        sig = pp_cross_section(K_MP * pp[:, 0].cpu().numpy())
        j = int(np.argmax(sig[:case["nb"] - 100] > 0)) + 2
        sig[:j + 1] = sig[j]
        sig = torch.from_numpy(sig).to(DEVICE)[:, None] / (1.0 + torch.exp(-5.0 * (pp - pp[j])))
    u = (crp if sp == 0 else cre).t().contiguous()
    on0 = (nsub - non) // 2
    ek = ((K_ME * torch.sqrt(1.0 + pe * pe) - K_ME) * K_GEV * dpe)[2:-2]
    for k in range(int(nseg.max())):
        live = k < nseg
        lo, hi = (k * nsub) // nseg, ((k + 1) * nsub) // nseg
        count = torch.where(live, hi - lo, torch.zeros_like(lo))
        alpha = torch.where(nseg > 1, (k + 0.5) / nseg.double(), torch.zeros_like(step_dt))
        g = bg[0] + alpha * (bg[1] - bg[0])
        n, kbt, b, dvv, lt, dv = (g[i] for i in range(6))
        rate, tacc = dpp_rate(case, g)
        if case["cfg"] == "tracer_10k":   # the turbulent energy caps the reacceleration
            power = 0.5 * MASS * 1.99e33 * dv ** 3 / (lt * K_MPC)
            eta = (ek * u[2:-2]).sum(0) / (power * tacc * K_GYR)
            rate = torch.where(eta > 0.1, rate * 0.1 / eta, rate)
        shape = p * p * torch.exp(-1.0 / p)
        if sp == 0:
            shape = shape * torch.exp(-K_MP * torch.sqrt(1.0 + p * p) / 1.0e7)
            radp = coulomb_p(n, kbt, p) + dvv / 3.0 * p
            loss = sig * 0.5 * K_C * n * K_GYR
        else:
            radp = synch(b, p) + (row + alpha * (row1 - row)) + coulomb_e(n, p) + dvv / 3.0 * p
            loss = torch.full_like(n, 1e-100)
        on = factor(p, dp, radp, shape * rate, step_dt, loss)
        windowed = case["cfg"] == "tracer_10k"
        off = factor(p, dp, radp, p * p / 4.0e5 + 0 * n, step_dt, loss) if windowed else None
        sl = torch.maximum(on0, lo) - lo
        el = sl + (torch.minimum(on0 + non, hi) - torch.maximum(on0, lo)).clamp(min=0)
        for i in range(int(count.max())):
            new = sweep(on, u)
            if windowed:
                new = torch.where((i >= sl) & (i < el), new, sweep(off, u))
            u = torch.where(i < count, new, u)
    u = u.t().contiguous()
    return {"crp": u, "cre": None} if sp == 0 else {"crp": torch.zeros_like(u), "cre": u}
