"""The work a psvWave-GB300 program does, as timed cases through the public API.

A case is a dict of plain values. Two surveys give the physical scales, both
from the repository's own workloads: "lab" (dx = 1.249 m, dt = 0.25 ms,
2000 / 800 / 1500 background with an inclusion, Ricker 50 Hz: the documented
inversion set-up) and "field" (dx = 5 m, dt = 0.4 ms, layered 1500-4500 m/s,
Ricker 15-25 Hz). Kinds of work:

* forward   -- set the medium, simulate one shot, read the seismograms;
* gradient  -- one FWI gradient with the reference's adjoint kernels, on host
               arrays as the reference's L-BFGS-B workflow calls it;
* exact     -- misfit and exact discrete gradient through the torch layer;
* batch     -- shots of many models of uneven sizes together;
* judge     -- misfits of many chains' states (Monte Carlo, batched forward);
* triples   -- exact misfit gradients at many states in parallel threads
               (training sets, plain HMC);
* predict, train -- the surrogate network's inference and training step.

FP32 models compute wave fields, seismograms and kernels to FP32 accuracy
and hand them out in FP64 containers, as the reference's API does; a program
that runs them keeps the results as FP32, so the cases return them so. FP64
models' results stay FP64.
"""
import math

import numpy as np
import torch
import torch.nn.functional as F
from torch.utils.checkpoint import checkpoint

import psvwave_gb300 as psv
from psvwave_gb300 import surrogate, torch_ops, workloads

DEV = "cuda:0"

# Typical seismogram amplitude of a survey's synthetics, for the scale of
# observed data (the integrated velocity over the cell area).
AMPLITUDE = {"lab": 1000.0, "field": 3.0, "mc": 1500.0}


def listed():
    return [
        # A first run on a toy grid (the test configuration's size), host
        # arrays in and out: call overhead and per-step latency.
        dict(name="forward_tiny", kind="forward", survey="lab", nxi=48, nzi=36, np=10, nt=400,
             shots=1, per_shot=1, nr=7, host=True),
        # One shot of a mid-size survey, of a ragged size near the
        # differentiation workload's grid.
        dict(name="forward_mid", kind="forward", survey="field", nxi=1003, nzi=397, np=50,
             nt=2000, shots=1, per_shot=1, nr=200, host=False),
        # One shot on the benchmark's large grid, with its full-tensor source.
        dict(name="forward_large", kind="forward", survey="field", nxi=2000, nzi=800, np=50,
             nt=2000, shots=1, per_shot=1, nr=400, host=False),
        # One iteration of the documented inversion (single precision), and
        # the same in the reference's own precision.
        dict(name="gradient_small", kind="gradient", survey="lab", nxi=200, nzi=100, np=25,
             nt=4000, shots=1, per_shot=2, nr=19, precision="fp32"),
        dict(name="gradient_small_fp64", kind="gradient", survey="lab", nxi=200, nzi=100, np=25,
             nt=2000, shots=1, per_shot=2, nr=19, precision="fp64"),
        # Multi-shot inversion gradients on the mid-size grid: the reference's
        # adjoint kernels, and the exact adjoint with checkpoints.
        dict(name="gradient_mid", kind="gradient", survey="field", nxi=1000, nzi=400, np=50,
             nt=1200, shots=8, per_shot=1, nr=200, precision="fp32"),
        dict(name="exact_mid", kind="exact", survey="field", nxi=1000, nzi=400, np=50, nt=1200,
             shots=8, per_shot=1, nr=200, ck=100),
        # Many models of uneven, odd sizes, one to four shots each.
        dict(name="batch_uneven", kind="batch", models=64, lo_x=200, hi_x=800, lo_z=100,
             hi_z=400, np=25, nt=250, nr=50),
        # One sampler iteration's judged states (128 chains).
        dict(name="judge", kind="judge", states=128, nt=2000),
        # A slice of a training set: exact gradients in parallel threads.
        dict(name="triples", kind="triples", states=32, nt=2000),
        # One leapfrog step's network call, and one training step's batch.
        dict(name="predict", kind="predict", states=128),
        dict(name="train", kind="train", states=256),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _steps(rng, lo, hi):
    """A number of time steps, a multiple of the snapshot interval (10)."""
    return 10 * _log_int(rng, lo // 10, hi // 10)


def draw(rng):
    kind = rng.choice(["forward", "forward", "gradient", "gradient", "exact", "batch", "judge",
                       "triples", "predict", "train"])
    if kind == "forward":
        survey = rng.choice(["lab", "field"])
        return dict(kind=kind, survey=survey, nxi=_log_int(rng, 40, 2000),
                    nzi=_log_int(rng, 36, 800), np=rng.randint(10, 50),
                    nt=_steps(rng, 300, 2000), shots=1, per_shot=rng.randint(1, 2),
                    nr=_log_int(rng, 3, 400), host=rng.random() < 0.5)
    if kind == "gradient":
        if rng.random() < 0.35:
            return dict(kind=kind, survey="lab", nxi=_log_int(rng, 60, 300),
                        nzi=_log_int(rng, 60, 200), np=rng.randint(10, 30),
                        nt=_steps(rng, 200, 1000), shots=rng.randint(1, 2),
                        per_shot=rng.randint(1, 2), nr=_log_int(rng, 5, 60), precision="fp64")
        return dict(kind=kind, survey=rng.choice(["lab", "field"]), nxi=_log_int(rng, 60, 1000),
                    nzi=_log_int(rng, 60, 400), np=rng.randint(10, 50),
                    nt=_steps(rng, 200, 1200), shots=rng.randint(1, 8), per_shot=1,
                    nr=_log_int(rng, 5, 200), precision="fp32")
    if kind == "exact":
        return dict(kind=kind, survey=rng.choice(["lab", "field"]), nxi=_log_int(rng, 60, 1000),
                    nzi=_log_int(rng, 60, 400), np=rng.randint(10, 50),
                    nt=_steps(rng, 200, 1200), shots=rng.randint(1, 8), per_shot=1,
                    nr=_log_int(rng, 5, 200), ck=rng.choice([40, 100, 150]))
    if kind == "batch":
        return dict(kind=kind, models=_log_int(rng, 4, 64), lo_x=rng.randint(100, 300),
                    hi_x=rng.randint(400, 800), lo_z=rng.randint(60, 150),
                    hi_z=rng.randint(200, 400), np=rng.randint(15, 30),
                    nt=_steps(rng, 150, 250), nr=_log_int(rng, 5, 60))
    if kind in ("judge", "triples"):
        return dict(kind=kind, states=_log_int(rng, 1, 128 if kind == "judge" else 32),
                    nt=_steps(rng, 400, 2000))
    return dict(kind=kind, states=_log_int(rng, 1, 512))


# ---- geometry, media and data ------------------------------------------------

SURVEYS = {"lab": dict(dx=1.249, dt=2.5e-4, f=50.0, delay=24, z=10),
           "field": dict(dx=5.0, dt=4e-4, f=20.0, delay=0, z=5),
           "mc": dict(dx=1.249, dt=2e-4, f=15.0, delay=0, z=10)}


def _params(case, nxi=None, nzi=None, shots=None):
    s = SURVEYS[case.get("survey", "field")]
    nxi, nzi = nxi or case["nxi"], nzi or case["nzi"]
    shots, per, nr = shots or case.get("shots", 1), case.get("per_shot", 1), case["nr"]
    n = shots * per
    return dict(nt=case["nt"], nx_inner=nxi, nz_inner=nzi, nx_inner_boundary=10,
                nz_inner_boundary=10, dx=s["dx"], dz=s["dx"], dt=s["dt"],
                np_boundary=case["np"], np_factor=0.015, scalar_rho=2000.0, scalar_vp=2500.0,
                scalar_vs=1445.0, npx=1, npz=1, peak_frequency=s["f"], source_timeshift=0.0,
                delay_cycles_per_shot=s["delay"] if per > 1 else 0, n_sources=n,
                ix_sources=[int(nxi * (k + 0.5) / n) for k in range(n)],
                iz_sources=[s["z"] + 5] * n, moment_angles=[45.0 + 15.0 * (k % 2) for k in range(n)],
                which_source_to_fire_in_which_shot=[list(range(k * per, (k + 1) * per))
                                                    for k in range(shots)],
                nr=nr, ix_receivers=[int(2 + (nxi - 4) * r / max(1, nr - 1)) for r in range(nr)],
                iz_receivers=[s["z"]] * nr, snapshot_interval=10)


def _generator(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _medium(survey, nx, nz, npb, seed):
    """(vp, vs, rho) [nx][nz], float64 on the GPU."""
    gen = _generator(seed)
    coarse = torch.randn((1, 1, nx // 20 + 3, nz // 20 + 3), generator=gen, device=DEV,
                         dtype=torch.float64)
    smooth = F.interpolate(coarse, size=(nx, nz), mode="bicubic", align_corners=True)[0, 0]
    if survey == "lab":
        u = torch.rand(2, generator=gen, device=DEV, dtype=torch.float64)
        x = torch.arange(nx, device=DEV, dtype=torch.float64)[:, None]
        z = torch.arange(nz, device=DEV, dtype=torch.float64)[None, :]
        inside = ((x - nx * (0.3 + 0.4 * u[0])) ** 2 + (z - nz * (0.3 + 0.4 * u[1])) ** 2) < 225.0
        f = (1 + 0.1 * inside) * (1 + 0.01 * smooth)
        return 2000.0 * f, 800.0 * f, 1500.0 * (1 + 0.1 * inside)
    vps = (1500.0 + 2700.0 * torch.rand(30, generator=gen, device=DEV,
                                        dtype=torch.float64)).sort().values
    inner = nz - 2 * npb
    depth = (torch.arange(nz, device=DEV) - npb).clamp(0, inner - 1)
    vp = vps[(depth * 30 // inner).clamp(max=29)][None, :] * (1 + 0.02 * smooth)
    return vp.contiguous(), (vp / 1.73).contiguous(), (310.0 * vp ** 0.25).contiguous()


def _observed(case, seed):
    """Recorded data [2][shots][nr][nt] (float64, GPU): a direct and two
    reflected Ricker arrivals per trace with the survey's moveout, and noise."""
    s = SURVEYS[case["survey"]]
    gen = _generator(seed + 7)
    p = _params(case)
    shots, nr, nt = case["shots"], case["nr"], case["nt"]
    xs = torch.tensor([p["ix_sources"][k * case.get("per_shot", 1)] for k in range(shots)],
                      device=DEV, dtype=torch.float64) * s["dx"]
    xr = torch.tensor(p["ix_receivers"], device=DEV, dtype=torch.float64) * s["dx"]
    t = torch.arange(nt, device=DEV, dtype=torch.float64) * s["dt"]
    off = (xs[:, None] - xr[None, :]).abs()
    r = torch.rand((2, 3), generator=gen, device=DEV, dtype=torch.float64)
    out = torch.zeros((2, shots, nr, nt), device=DEV, dtype=torch.float64)
    for c in range(2):
        for k in range(3):
            t0 = 1.4 / s["f"] + 0.25 * k * nt * s["dt"] * (0.5 + r[c, k])
            arr = torch.sqrt(t0 ** 2 + (off / (1600.0 + 800.0 * r[c, k])) ** 2)
            a = (math.pi * s["f"] * (t[None, None, :] - arr[..., None])) ** 2
            out[c] += (0.6 ** k) * (1 - 2 * a) * torch.exp(-a)
    out += 0.01 * torch.randn(out.shape, generator=gen, device=DEV, dtype=torch.float64)
    return out * AMPLITUDE[case["survey"]]


def _mc_case(case):
    """The Monte Carlo workload's geometry as a case of this file's shape."""
    return dict(case, survey="mc", nxi=200, nzi=100, np=25, nr=19, shots=1, per_shot=2)


def _mc_observed(case, seed):
    return _observed(_mc_case(case), seed)


def _states(case, seed):
    gen = _generator(seed)
    return 0.5 * torch.randn((case["states"], 3, 20, 10), generator=gen, device=DEV)


def _batch_sizes(case, seed):
    """(nx_inner, nz_inner, shots) of each model; the sizes are the case's,
    the media the seed's."""
    rng = np.random.default_rng(1000 * case["models"] + case["nt"])
    return [(int(rng.integers(case["lo_x"], case["hi_x"] + 1)),
             int(rng.integers(case["lo_z"], case["hi_z"] + 1)), int(rng.integers(1, 5)))
            for _ in range(case["models"])]


def _net_data(case, seed):
    """Network parameters and a batch of features and normalised targets."""
    gen = _generator(seed)
    B = case["states"]
    z = torch.randn((B, 3, 20, 10), generator=gen, device=DEV)
    m = torch.randn(B, generator=gen, device=DEV)
    g = torch.randn((B, 3, 20, 10), generator=gen, device=DEV)
    w = surrogate.init_params(seed % 100003)
    n_last = surrogate.CNN_LAYERS[-1][0] * surrogate.CNN_LAYERS[-1][1] * 9 + \
        surrogate.CNN_LAYERS[-1][1]
    w[-n_last:] *= 30.0  # a trained network's last layer is not near zero
    return z, m, g, w


# ---- prepare, run, work ------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    st = dict(case=case)
    if kind in ("forward", "gradient", "exact"):
        p = _params(case)
        m = psv.fdModel.from_parameters(p, precision=case.get("precision", "fp32"))
        med = _medium(case["survey"], m.nx, m.nz, m.np_boundary, seed)
        if kind == "forward" and case["survey"] == "field":
            m.set_moment(np.repeat(workloads.c1_moment(), m.n_sources, axis=0))
        if kind != "forward":
            m.set_observed_data_device(*_observed(case, seed))
        if kind == "gradient" or case.get("host"):
            med = tuple(a.cpu().numpy() for a in med)
        if kind == "exact":
            med = tuple(a.float().requires_grad_(True) for a in med)
        st.update(model=m, medium=med)
    elif kind == "batch":
        st["models"], st["batch"] = [], psv.Batch()
        for k, (nxi, nzi, shots) in enumerate(_batch_sizes(case, seed)):
            m = psv.fdModel.from_parameters(_params(case, nxi, nzi, shots))
            m.set_parameter_fields_device(*_medium("field", m.nx, m.nz, m.np_boundary,
                                                   1000 * seed + k))
            st["batch"].add_all_shots(m)
            st["models"].append(m)
        st["batch"].autotune()
    elif kind in ("judge", "triples"):
        mean, sigma = workloads.c4_prior()
        p = workloads.c4_params(nt=case["nt"])
        nx, nz = p["nx_inner"] + 2 * p["np_boundary"], p["nz_inner"] + 2 * p["np_boundary"]
        coarse = surrogate.CoarseParam(nx, nz, p["np_boundary"], mean, sigma)
        obs = _mc_observed(case, seed).cpu().numpy()
        st.update(z=_states(case, seed),
                  post=surrogate.FDPosterior(p, coarse, (obs[0], obs[1]), 1.0,
                                             min(case["states"], 128 if kind == "judge" else 16)))
    else:
        z, m, g, w = _net_data(case, seed)
        net = surrogate.SurrogateNet(max_batch=512)
        net.set_params(w)
        st.update(net=net, z=z, m=m, g=g, x=net.features(z))
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "forward":
        m = st["model"]
        if case["host"]:
            m.set_parameter_fields(*st["medium"])
            m.forward_simulate(0, store_fields=False)
            return [a.astype(np.float32) for a in m.get_synthetic_data()]
        m.set_parameter_fields_device(*st["medium"])
        m.forward_simulate(0, store_fields=False)
        return [a.float() for a in m.get_synthetic_data_device()]
    if kind == "gradient":
        m = st["model"]
        m.set_parameter_fields(*st["medium"])
        misfit, g = m.compute_gradients()
        return [misfit, g if case["precision"] == "fp64" else g.astype(np.float32)]
    if kind == "exact":
        for t in st["medium"]:
            t.grad = None
        loss = torch_ops.l2_misfit(st["model"], *st["medium"], checkpoint_every=case["ck"])
        loss.backward()
        return [loss.item()] + [t.grad for t in st["medium"]]
    if kind == "batch":
        st["batch"].forward()
        out = [m.get_synthetic_data_device() for m in st["models"]]
        return [torch.cat([a[c].reshape(-1) for a in out]).float() for c in range(2)]
    if kind == "judge":
        return st["post"].misfits(st["z"]).astype(np.float32)
    if kind == "triples":
        _, mis, g = surrogate.triples_at(st["post"], st["z"])
        return [mis.float(), g]
    if kind == "predict":
        m, g = st["net"].predict(st["z"])
        return [m.float(), g]
    loss, d = st["net"].loss_grad(st["x"], st["m"], st["g"])
    return [loss, d]


# Floating-point operations of one cell and time step of the staggered
# scheme: four derivatives of 5 operations in each half step, the stress
# combinations and updates (16), the velocity updates (8), the taper (5).
STEP_FLOPS = 69
# Network multiply-adds per state: 200 nodes x 9 taps x channel pairs.
NET_FLOPS = 2 * 200 * 9 * (5 * 32 + 32 * 64 + 64 * 64 + 64 * 4)


def work(case):
    """Bytes: the media, data and states read and the results written.
    Operations: the time steps these need (a gradient: the forward, the
    recomputed forward or the correlation, and the adjoint)."""
    kind = case["kind"]
    if kind in ("forward", "gradient", "exact"):
        nx, nz = case["nxi"] + 2 * case["np"], case["nzi"] + 2 * case["np"]
        cells, data = nx * nz, 2 * case["shots"] * case["nr"] * case["nt"] * 8
        steps = cells * case["nt"] * case["shots"]
        if kind == "forward":
            return {"bytes": 24 * cells + data, "flops": STEP_FLOPS * steps}
        per = 2 if kind == "gradient" else 3
        return {"bytes": 48 * cells + data, "flops": per * STEP_FLOPS * steps}
    if kind == "batch":
        steps = sum((a + 2 * case["np"]) * (b + 2 * case["np"]) * s
                    for a, b, s in _batch_sizes(case, 0)) * case["nt"]
        data = sum(s for _, _, s in _batch_sizes(case, 0)) * 2 * case["nr"] * case["nt"] * 8
        return {"bytes": data + 24 * steps // case["nt"], "flops": STEP_FLOPS * steps}
    B = case["states"]
    if kind in ("judge", "triples"):
        steps = B * 250 * 150 * case["nt"]
        return {"bytes": B * 2400 * (1 if kind == "judge" else 2) + 2 * 19 * case["nt"] * 8,
                "flops": (1 if kind == "judge" else 3) * STEP_FLOPS * steps}
    if kind == "predict":
        return {"bytes": B * (3 + 3) * 800, "flops": B * NET_FLOPS}
    return {"bytes": B * (5 + 3) * 800 + 4 * surrogate._num_params(), "flops": 3 * B * NET_FLOPS}


# ---- the same in plain 64-bit torch ------------------------------------------

class _Plain:
    """The staggered-grid scheme in plain torch, float64, for a batch of
    simulations ([S][nx][nz] fields): S shots of one medium ([nx][nz]) or S
    media ([S][nx][nz]) of one shot."""

    def __init__(self, p, media, shots, moment=None):
        self.p = p
        npb, dt = p["np_boundary"], p["dt"]
        vp, vs, rho = media
        self.vp, self.vs, self.rho = vp, vs, rho
        self.lm, self.mu, self.b = rho * vp ** 2, rho * vs ** 2, 1.0 / rho
        self.la = self.lm - 2 * self.mu
        nx, nz = vp.shape[-2:]
        self.nx, self.nz = nx, nz
        ix = torch.arange(nx, device=DEV, dtype=torch.float64)[:, None]
        iz = torch.arange(nz, device=DEV, dtype=torch.float64)[None, :]
        c = torch.minimum(torch.minimum(ix + 1, nx - ix), torch.minimum(iz + 1, nz - iz))
        self.taper = torch.exp(-(p["np_factor"] * (npb - c.clamp(max=npb))) ** 2)[2:-2, 2:-2]
        self.h, self.dt, self.nt = p["dx"], dt, p["nt"]
        # Source patterns and wavelets by position in the shot's list.
        src = [p["which_source_to_fire_in_which_shot"][k] for k in shots]
        self.S = len(shots)
        t = torch.arange(self.nt, device=DEV, dtype=torch.float64) * dt
        f = p["peak_frequency"]
        self.sources = []
        for pos in range(max(len(s) for s in src)):
            a = (math.pi * f * (t - 1.4 / f - p["delay_cycles_per_shot"] * pos / f)) ** 2
            px = torch.zeros((self.S, nx, nz), device=DEV, dtype=torch.float64)
            pz = torch.zeros_like(px)
            for k, s in enumerate(src):
                i = s[pos]
                r = p["moment_angles"][i] * 3.14159265 / 180.0
                M = np.array([[math.cos(r), -math.sin(r)], [-math.sin(r), -math.cos(r)]]) * 1e15
                if moment is not None:
                    M = moment[i]
                x, z, h4 = p["ix_sources"][i] + npb, p["iz_sources"][i] + npb, self.h ** 4
                for dx_, dz_, w in ((-1, 0, -M[0, 0]), (0, 0, M[0, 0]), (-1, 1, M[0, 1] / 4),
                                    (0, 1, M[0, 1] / 4), (-1, -1, -M[0, 1] / 4),
                                    (0, -1, -M[0, 1] / 4)):
                    px[k, x + dx_, z + dz_] += w / h4
                for dx_, dz_, w in ((0, -1, -M[1, 1]), (0, 0, M[1, 1]), (1, -1, M[1, 0] / 4),
                                    (1, 0, M[1, 0] / 4), (-1, -1, -M[1, 0] / 4),
                                    (-1, 0, -M[1, 0] / 4)):
                    pz[k, x + dx_, z + dz_] += w / h4
            self.sources.append(((1 - 2 * a) * torch.exp(-a) * dt, px, pz))
        self.rx = torch.tensor(p["ix_receivers"], device=DEV) + npb
        self.rz = torch.tensor(p["iz_receivers"], device=DEV) + npb

    def zero(self, S):
        return tuple(torch.zeros((S, self.nx, self.nz), device=DEV, dtype=torch.float64)
                     for _ in range(5))

    def _d(self, f, axis, forward):
        """Fourth-order staggered difference on the interior [2, n - 2)."""
        n = f.shape[axis]
        o = (lambda k: f.narrow(axis, 2 + k, n - 4))
        g = (lambda d: d.narrow(-1, 2, self.nz - 4) if axis == -2 else d.narrow(-2, 2, self.nx - 4))
        if forward:
            d = (9.0 / 8.0) * (o(1) - o(0)) + (1.0 / 24.0) * (o(-1) - o(2))
        else:
            d = (9.0 / 8.0) * (o(0) - o(-1)) + (1.0 / 24.0) * (o(-2) - o(1))
        return g(d) / self.h

    def _advance(self, f, rate, sign):
        pad = self.taper * (f[:, 2:-2, 2:-2] + (sign * self.dt) * rate)
        return F.pad(pad, (2, 2, 2, 2))

    def half(self, a):
        return a[..., 2:-2, 2:-2]

    def step(self, state, it, sign=1.0):
        vx, vz, txx, tzz, txz = state
        ex, ez = self._d(vx, -2, True), self._d(vz, -1, False)
        g = self._d(vx, -1, True) + self._d(vz, -2, False)
        lm, la, mu, b = (self.half(a) for a in (self.lm, self.la, self.mu, self.b))
        txx, tzz = self._advance(txx, lm * ex + la * ez, sign), \
            self._advance(tzz, la * ex + lm * ez, sign)
        txz = self._advance(txz, mu * g, sign)
        ax = self._d(txx, -2, False) + self._d(txz, -1, False)
        az = self._d(txz, -2, True) + self._d(tzz, -1, True)
        vx, vz = self._advance(vx, b * ax, sign), self._advance(vz, b * az, sign)
        if sign > 0:
            for w, px, pz in self.sources:
                vx = vx + w[it] * px * self.b
                vz = vz + w[it] * pz * self.b
        return vx, vz, txx, tzz, txz

    def record(self, state):
        return torch.stack([state[0][:, self.rx, self.rz], state[1][:, self.rx, self.rz]])

    def forward(self, every=0):
        """Seismograms [2][S][nr][nt] and the snapshots taken every `every`
        steps (lists of states)."""
        S = self.S if self.vp.dim() == 2 else self.vp.shape[0]
        state, rec, snaps = self.zero(S), [], []
        for it in range(self.nt):
            if every and it % every == 0:
                snaps.append(state)
            rec.append(self.record(state))
            state = self.step(state, it)
        return torch.stack(rec, -1).cumsum(-1) * self.dt / self.h ** 2, snaps

    def misfit(self, obs, segment=40):
        """L2 misfit per medium or shot, differentiable in the medium."""
        S = self.S if self.vp.dim() == 2 else self.vp.shape[0]
        state, rec = self.zero(S), []

        def chunk(i0, i1, *s):
            out = []
            for it in range(i0, i1):
                out.append(self.record(s))
                s = self.step(s, it)
            return (torch.stack(out, -1),) + tuple(s)

        for i0 in range(0, self.nt, segment):
            r, *state = checkpoint(chunk, i0, min(self.nt, i0 + segment), *state,
                                   use_reentrant=False)
            rec.append(r)
        u = torch.cat(rec, -1).cumsum(-1) * self.dt / self.h ** 2
        return 0.5 * self.dt * ((obs - u) ** 2).sum((0, 2, 3))

    def kernels(self, obs):
        """Misfit and the reference's adjoint kernels for (vp, vs, rho)."""
        si = self.p["snapshot_interval"]
        u, snaps = self.forward(si)
        adj = u - obs
        r = self.la / self.lm
        den = (self.lm - self.la * r) ** 2
        k_rho, k_lam, k_mu = (torch.zeros_like(self.vp) for _ in range(3))
        state = self.zero(self.S)
        lin = self.rx * self.nz + self.rz
        area = self.h ** 2
        for it in range(self.nt - 1, -1, -1):
            if it % si == 0:
                avx, avz, axx, azz, axz = snaps.pop()
                vx, vz, txx, tzz, txz = state
                fxx, fzz = txx - tzz * r, tzz - txx * r
                hxx, hzz = axx - azz * r, azz - axx * r
                w = si * self.dt
                k_rho -= w * (avx * vx + avz * vz).sum(0)
                k_lam += w * ((hxx + hzz) * (fxx + fzz) / den).sum(0)
                k_mu += 2 * w * ((fxx * hxx + fzz * hzz) / den
                                 + txz * axz / (2 * self.mu ** 2)).sum(0)
            vx, vz, *t = self.step(state, it, -1.0)
            bi = self.dt * self.b.reshape(-1)[lin] / area
            for v, a in ((vx, adj[0, :, :, it]), (vz, adj[1, :, :, it])):
                v.view(self.S, -1).index_add_(1, lin, bi * a)
            state = (vx, vz, *t)
        f0 = self.p["np_boundary"] + 10
        free = torch.zeros_like(self.vp)
        free[f0:self.nx - f0, f0:self.nz - f0] = 1
        k_rho, k_lam, k_mu = k_rho * free, k_lam * free, k_mu * free
        g_vp = 2 * self.vp * k_lam * self.rho
        g_vs = (2 * self.vs * k_mu - 4 * self.vs * k_lam) * self.rho
        g_rho = k_rho + (self.vp ** 2 - 2 * self.vs ** 2) * k_lam + self.vs ** 2 * k_mu
        vec = [g[f0:self.nx - f0, f0:self.nz - f0].t().reshape(-1) for g in (g_vp, g_vs, g_rho)]
        return float(0.5 * self.dt * (adj ** 2).sum()), torch.cat(vec)


def _plain_fields(z):
    """(vp, vs, rho) [B][250][150] of coarse states [B][3][20][10]."""
    mean, sigma = (torch.tensor(a, device=DEV, dtype=torch.float64) for a in workloads.c4_prior())
    theta = mean + sigma * z
    inner = F.interpolate(theta, size=(200, 100), mode="bilinear", align_corners=False)
    f = F.pad(inner, (25, 25, 25, 25), mode="replicate")
    return f[:, 0], f[:, 1], f[:, 2]


def _plain_net(w, x):
    """The network's output [B][4][20][10] and its parameters, in float64;
    weights are held in BF16, biases in FP32."""
    off, params = 0, []
    for l, (cin, cout) in enumerate(surrogate.CNN_LAYERS):
        k = torch.tensor(w[off:off + cout * cin * 9], device=DEV).bfloat16().double()
        b = torch.tensor(w[off + cout * cin * 9:off + cout * cin * 9 + cout], device=DEV).double()
        off += cout * cin * 9 + cout
        params += [k.requires_grad_(True), b.requires_grad_(True)]
        d = (1, 2, 4, 1)[l]
        # the 3 x 3 taps as one matrix product
        cols = F.unfold(x, 3, dilation=d, padding=d)
        x = (k.view(cout, cin * 9) @ cols + b[:, None]).view(-1, cout, 20, 10)
        x = torch.relu(x) if l < 3 else x
    return x, params


def exact(case, seed):
    kind = case["kind"]
    if kind in ("forward", "gradient", "exact"):
        p = _params(case)
        nx, nz = case["nxi"] + 2 * case["np"], case["nzi"] + 2 * case["np"]
        med = _medium(case["survey"], nx, nz, case["np"], seed)
        if kind == "forward":
            mom = np.repeat(workloads.c1_moment(), len(p["ix_sources"]), axis=0) \
                if case["survey"] == "field" else None
            with torch.no_grad():
                u, _ = _Plain(p, med, [0], mom).forward()
            return [u[0], u[1]]
        obs = _observed(case, seed)
        shots = list(range(case["shots"]))
        if kind == "gradient":
            with torch.no_grad():
                return list(_Plain(p, med, shots).kernels(obs))
        med = [a.float().double().requires_grad_(True) for a in med]
        loss = _Plain(p, med, shots).misfit(obs).sum()
        loss.backward()
        return [loss.item()] + [a.grad for a in med]
    if kind == "batch":
        outs = ([], [])
        with torch.no_grad():
            for k, (nxi, nzi, shots) in enumerate(_batch_sizes(case, seed)):
                p = _params(case, nxi, nzi, shots)
                med = _medium("field", nxi + 2 * case["np"], nzi + 2 * case["np"], case["np"],
                              1000 * seed + k)
                u, _ = _Plain(p, med, list(range(shots))).forward()
                for c in range(2):
                    outs[c].append(u[c].reshape(-1))
        return [torch.cat(o) for o in outs]
    if kind in ("judge", "triples"):
        obs = _mc_observed(case, seed)
        p = workloads.c4_params(nt=case["nt"])
        z = _states(case, seed).double()
        if kind == "judge":
            with torch.no_grad():
                return _Plain(p, _plain_fields(z), [0]).misfit(obs)
        z.requires_grad_(True)
        mis = _Plain(p, _plain_fields(z), [0]).misfit(obs)
        mis.sum().backward()
        return [mis.detach(), z.grad]
    z, m, g, w = _net_data(case, seed)
    xc = torch.linspace(-1.0, 1.0, 20, device=DEV)[:, None].expand(20, 10)
    zc = torch.linspace(-1.0, 1.0, 10, device=DEV)[None, :].expand(20, 10)
    coords = torch.stack([xc, zc]).expand(case["states"], 2, 20, 10)
    y, params = _plain_net(w, torch.cat([z, coords], 1).double())
    my, gy = y[:, 3].sum((1, 2)), y[:, :3]
    if kind == "predict":
        return [my.detach(), gy.detach()]
    loss = ((my - m.double()) ** 2).mean() + ((gy - g.double()) ** 2).mean()
    loss.backward()
    return [loss.item(), torch.cat([t.grad.reshape(-1) for t in params])]
