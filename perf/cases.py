"""What the framework's speed is measured on: simulations as users run them.

Every case goes through the public entry points -- ``model.run()`` of the 2D
and 3D models and ``TissueBatch.run()`` -- in the precisions, stencils and
tracker set-ups that they are used with.  Three kinds of pass:

* ``chunk``: a program that holds an initialised model in mid-simulation and
  advances it by ``steps`` time steps (``run(initialize=False)`` after moving
  ``t_max``), as programs do that steer, save or watch a simulation between
  chunks; the state stays on the device and is what the pass returns;
* ``whole``: a complete ``model.run()`` from the initial values -- weights,
  stimulus, trackers, all steps -- and the outputs read back on the host;
* ``batch``: many tissues of different sizes, models and stencils advanced
  together by ``TissueBatch.run(initialize=False)``.

float64 is the models' default precision; float32 is what users choose for
speed.  Tissues carry diffuse fibrosis; anisotropic ones have smooth fibers.
The states are smooth mixtures of rest and excitation, so that all phases of
the action potential are met in one tissue.
"""
import math
import random

import numpy as np
import torch

import finitewave_gb300 as fg

DT, DR = 0.01, 0.25

# parameters as in the models' papers and defaults, for exact()
_P = {
    "ap": dict(a=0.1, k=8.0, eap=0.01, mu_1=0.2, mu_2=0.3),
    "ms": dict(tau_close=150.0, tau_open=120.0, tau_in=0.3, tau_out=6.0, u_gate=0.13),
    "fk": dict(tau_d=0.172, tau_o=12.5, tau_r=130.0, tau_si=127.0, tau_v_m=18.2, tau_v_p=10.0,
               tau_w_m=80.0, tau_w_p=1020.0, k=10.0, u_c=0.13, uc_si=0.85),
    "bo": dict(u_o=0.0, u_u=1.55, theta_v=0.3, theta_w=0.13, theta_v_m=0.006, theta_o=0.006,
               tau_v1_m=60, tau_v2_m=1150, tau_v_p=1.4506, tau_w1_m=60, tau_w2_m=15, k_w_m=65,
               u_w_m=0.03, tau_w_p=200, tau_fi=0.11, tau_o1=400, tau_o2=6, tau_so1=30.0181,
               tau_so2=0.9957, k_so=2.0458, u_so=0.65, tau_s1=2.7342, tau_s2=16, k_s=2.0994,
               u_s=0.9087, tau_si=1.8875, tau_w_inf=0.07, w_inf_=0.94),
}
_D_MODEL = {"tp06": 0.154, "crn": 0.154, "lr91": 0.1}

# state variables after u: (name, value at rest, value when excited)
_STATE = {
    "ap": [("v", 0.0, 2.0)],
    "ms": [("h", 1.0, 0.1)],
    "fk": [("v", 1.0, 0.05), ("w", 1.0, 0.5)],
    "bo": [("v", 1.0, 0.02), ("w", 1.0, 0.4), ("s", 0.02, 0.7)],
    "tp06": [("cai", 7e-5, 9e-5), ("casr", 1.3, 1.1), ("cass", 7e-5, 4e-4), ("nai", 7.67, 7.8),
             ("Ki", 138.3, 137.9), ("m", 0.002, 0.98), ("h", 0.75, 0.01), ("j", 0.75, 0.02),
             ("xr1", 0.001, 0.6), ("xr2", 0.95, 0.2), ("xs", 0.004, 0.3), ("r", 0.001, 0.9),
             ("s", 0.99, 0.1), ("d", 0.001, 0.95), ("f", 0.99, 0.5), ("f2", 0.99, 0.6),
             ("fcass", 0.99, 0.7), ("rr", 0.99, 0.8), ("oo", 0.0, 1e-5)],
    "crn": [("nai", 11.2, 11.4), ("ki", 139.0, 138.7), ("cai", 1.02e-4, 6e-4), ("caup", 1.6, 1.5),
            ("carel", 1.1, 0.6), ("m", 0.003, 0.98), ("h", 0.965, 0.01), ("j_", 0.978, 0.02),
            ("d", 1.4e-4, 0.9), ("f", 0.999, 0.6), ("oa", 6e-4, 0.8), ("oi", 0.999, 0.05),
            ("ua", 0.0035, 0.8), ("ui", 0.9987, 0.98), ("xr", 3.3e-5, 0.3), ("xs", 0.0187, 0.4),
            ("fca", 0.775, 0.4), ("irel", 0.0, 0.001), ("vrel", 0.999, 0.5), ("urel", 0.001, 0.4),
            ("wrel", 0.9, 0.6)],
    "lr91": [("m", 0.002, 0.98), ("h", 0.983, 0.01), ("j", 0.995, 0.02), ("d", 3e-6, 0.9),
             ("f", 0.999, 0.5), ("x", 0.0057, 0.5), ("cai", 2e-4, 4e-3)],
}
_REST = {"ap": (0.0, 1.0), "ms": (0.0, 0.95), "fk": (0.0, 0.95), "bo": (0.0, 1.4),
         "tp06": (-84.5, 25.0), "crn": (-81.0, 20.0), "lr91": (-84.5, 25.0)}
# concentrations keep 8 bytes a node in float32 as well
_CONC = {"tp06": ("cai", "casr", "cass", "nai", "Ki"), "crn": ("nai", "ki", "cai", "caup", "carel"),
         "lr91": ("cai",)}

_CLASSES = {("ap", 2): fg.AlievPanfilov2D, ("ap", 3): fg.AlievPanfilov3D,
            ("ms", 2): fg.MitchellSchaeffer2D, ("ms", 3): fg.MitchellSchaeffer3D,
            ("fk", 2): fg.FentonKarma2D, ("fk", 3): fg.FentonKarma3D,
            ("bo", 2): fg.BuenoOrovio2D, ("bo", 3): fg.BuenoOrovio3D,
            ("tp06", 2): fg.TP062D, ("tp06", 3): fg.TP063D,
            ("crn", 2): fg.Courtemanche2D, ("crn", 3): fg.Courtemanche3D,
            ("lr91", 2): fg.LuoRudy912D, ("lr91", 3): fg.LuoRudy913D}


def _case(name=None, **kw):
    c = dict(kind="chunk", model="ap", prec="float32", ni=128, nj=128, nk=0, fibers="none",
             fibrosis=0.1, steps=100, track="none")
    c.update(kw)
    return dict(name=name, **c) if name else c


def listed():
    return [
        # the first program of a user: a small isotropic sheet in the default
        # precision, one plane wave, activation map and two probes
        _case("ap2d_f64_whole", kind="whole", prec="float64", ni=100, nj=100, steps=1000,
              fibrosis=0.0, track="act+probe"),
        # a fibrotic anisotropic sheet in the default precision
        _case("ap2d_f64_sheet", prec="float64", ni=600, nj=601, fibers="smooth", fibrosis=0.2,
              steps=50, track="act"),
        # the benchmark's sheet: 4096 x 4096, anisotropic, 20 % fibrosis
        _case("ap2d_f32_large", ni=4096, nj=4096, fibers="smooth", fibrosis=0.2, steps=100,
              track="act"),
        # a small float32 sheet, where launches and their gaps count
        _case("ms2d_f32_small", model="ms", ni=250, nj=256, steps=400, track="act"),
        # a ragged sheet of a model with two state variables
        _case("fk2d_f32_ragged", model="fk", ni=777, nj=1011, fibers="smooth", steps=200,
              track="act"),
        # an ECG recorded during a whole float32 run
        _case("ap2d_f32_ecg", kind="whole", ni=320, nj=300, fibers="smooth", steps=1000,
              track="ecg"),
        # a 3D block whose fibers turn out of the plane (all 19 weights)
        _case("ap3d_f32_aniso", ni=256, nj=240, nk=60, fibers="smooth", steps=50),
        # an isotropic 3D block of the minimal ventricular model
        _case("bo3d_f32_iso", model="bo", ni=130, nj=128, nk=100, steps=50),
        # the detailed ventricular model in the default precision
        _case("tp06_2d_f64", model="tp06", prec="float64", ni=192, nj=190, fibers="smooth",
              steps=20),
        # the detailed atrial model in float32, odd sizes
        _case("crn2d_f32", model="crn", ni=511, nj=387, fibers="smooth", steps=50),
        # a transmural slab of the detailed ventricular model: fibers turn
        # with depth and stay in the plane
        _case("tp06_3d_f32_slab", model="tp06", ni=256, nj=256, nk=40, fibers="layers", steps=30),
        # sixteen tissues of different sizes, models and stencils together
        _case("batch_f32", kind="batch", ni=16, nj=64, nk=1024, steps=100, track="lat", mix=4),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    pick = rng.choice(["whole", "f64", "f32", "f32", "3d", "detailed64", "detailed32", "slab",
                       "batch"])
    fibrosis = round(rng.uniform(0.0, 0.3), 3)
    if pick == "whole":
        return _case(kind="whole", model=rng.choice(["ap", "fk", "ms"]), prec="float64",
                     ni=_log(rng, 48, 160), nj=_log(rng, 48, 160),
                     fibers=rng.choice(["none", "smooth"]), steps=rng.randrange(300, 1000),
                     fibrosis=fibrosis, track=rng.choice(["act+probe", "ecg"]))
    if pick == "f64":
        return _case(model=rng.choice(["ap", "ms", "fk", "bo"]), prec="float64",
                     ni=_log(rng, 128, 600), nj=_log(rng, 128, 600),
                     fibers=rng.choice(["none", "smooth"]), fibrosis=fibrosis,
                     steps=rng.randrange(25, 50), track="act")
    if pick == "f32":
        ni, nj = _log(rng, 96, 4000), _log(rng, 96, 4000)
        if rng.random() < 0.4:
            nj = max(96, nj - nj % 16)
        return _case(model=rng.choice(["ap", "ms", "fk"]), ni=ni, nj=nj,
                     fibers=rng.choice(["none", "smooth"]), fibrosis=fibrosis,
                     steps=rng.randrange(60, 100), track="act")
    if pick == "3d":
        return _case(model=rng.choice(["ap", "ms", "fk", "bo"]), ni=_log(rng, 60, 256),
                     nj=_log(rng, 60, 240), nk=_log(rng, 16, 60),
                     fibers=rng.choice(["none", "smooth", "layers"]), fibrosis=fibrosis,
                     steps=rng.randrange(20, 50))
    if pick == "detailed64":
        return _case(model=rng.choice(["tp06", "crn", "lr91"]), prec="float64",
                     ni=_log(rng, 64, 190), nj=_log(rng, 64, 190),
                     fibers=rng.choice(["none", "smooth"]), fibrosis=fibrosis,
                     steps=rng.randrange(10, 20))
    if pick == "detailed32":
        return _case(model=rng.choice(["tp06", "crn", "lr91"]), ni=_log(rng, 96, 510),
                     nj=_log(rng, 96, 380), fibers=rng.choice(["none", "smooth"]),
                     fibrosis=fibrosis, steps=rng.randrange(25, 50))
    if pick == "slab":
        return _case(model=rng.choice(["tp06", "crn"]), ni=_log(rng, 64, 250),
                     nj=_log(rng, 64, 250), nk=rng.randrange(12, 40),
                     fibers=rng.choice(["layers", "none", "smooth"]), fibrosis=fibrosis,
                     steps=rng.randrange(10, 24))
    return _case(kind="batch", ni=rng.randrange(4, 16), nj=64, nk=_log(rng, 160, 1000),
                 steps=rng.randrange(50, 100), track="lat", mix=rng.randrange(1 << 20))


# ------------------------------------------------------------------ inputs

def _dim(c):
    return 3 if c["nk"] else 2


def _shape(c):
    return (c["ni"], c["nj"], c["nk"]) if c["nk"] else (c["ni"], c["nj"])


def _dev():
    return torch.device("cuda", torch.cuda.current_device())


def _smooth(shape, rng):
    """A smooth field in [0, 1]: a sum of plane waves of 1 to 6 periods."""
    axes = [torch.linspace(0, 1, n, dtype=torch.float64, device=_dev()) for n in shape]
    f = torch.zeros(shape, dtype=torch.float64, device=_dev())
    for _ in range(5):
        arg = rng.uniform(0, 2 * math.pi)
        for d, x in enumerate(axes):
            v = 2 * math.pi * rng.uniform(-6, 6) * x
            arg = arg + v.reshape([-1 if k == d else 1 for k in range(len(shape))])
        f += torch.sin(arg)
    return torch.sigmoid(2.0 * f)


def _inputs(c, seed):
    """Mesh (int8), fibers or None, and the state as float64 tensors."""
    shape, dim = _shape(c), _dim(c)
    rng = random.Random(seed * 7919 + 17)
    gen = torch.Generator(device=_dev())
    gen.manual_seed(seed * 104729 + 5)
    mesh = 1 + (torch.rand(shape, generator=gen, device=_dev()) < c["fibrosis"]).to(torch.int8)
    for d in range(dim):
        mesh.select(d, 0).zero_()
        mesh.select(d, shape[d] - 1).zero_()
    fibers = None
    if c["fibers"] != "none":
        if c["fibers"] == "layers":
            t = torch.linspace(-math.pi / 3, math.pi / 3, shape[-1], dtype=torch.float64,
                               device=_dev()).expand(shape) + rng.uniform(-0.2, 0.2)
        else:
            t = (2 * _smooth(shape, rng) - 1) * (math.pi / 4)
        if dim == 2:
            fibers = torch.stack([torch.cos(t), torch.sin(t)], -1)
        else:
            p = (2 * _smooth(shape, rng) - 1) * (math.pi / 6) if c["fibers"] == "smooth" \
                else torch.zeros_like(t)
            fibers = torch.stack([torch.cos(t) * torch.cos(p), torch.sin(t) * torch.cos(p),
                                  torch.sin(p)], -1)
    state = None
    if c["kind"] != "whole":
        rest, up = _REST[c["model"]]
        a, b = _smooth(shape, rng), _smooth(shape, rng)
        state = {"u": rest + (up - rest) * a}
        for k, (name, lo, hi) in enumerate(_STATE[c["model"]]):
            x = (b, 0.5 * (a + b), 1 - (1 - a) * (1 - 0.5 * b))[k % 3]
            state[name] = lo + (hi - lo) * x
    return mesh, fibers, state


def _init_u(model):
    return float(getattr(model, "init_u", 0.0))


def _build(c, seed, mesh, fibers):
    shape, dim = _shape(c), _dim(c)
    tissue = fg.CardiacTissue2D(shape) if dim == 2 else fg.CardiacTissue3D(shape)
    tissue.mesh = mesh.cpu().numpy()
    model = _CLASSES[c["model"], dim]()
    if fibers is not None:
        tissue.fibers = fibers.cpu().numpy()
        model.stencil = fg.AsymmetricStencil2D() if dim == 2 else fg.AsymmetricStencil3D()
        model.stencil.D_al, model.stencil.D_ac = 1.0, 0.111
    model.cardiac_tissue = tissue
    model.dt, model.dr = DT, DR
    model.npfloat = c["prec"]
    model.prog_bar = False
    model.t_max = (c["steps"] - 0.5) * DT
    trackers = {}
    seq = fg.TrackerSequence()
    if "act" in c["track"]:
        tr = fg.ActivationTime2DTracker() if dim == 2 else fg.ActivationTime3DTracker()
        tr.threshold = 0.5
        trackers["act"] = tr
    if c["track"] == "lat":
        tr = fg.LocalActivationTime2DTracker()
        tr.threshold = 0.5
        trackers["lat"] = tr
    if "probe" in c["track"]:
        tr = fg.ActionPotential2DTracker()
        tr.cell_ind = _cells(c)
        trackers["probe"] = tr
    if c["track"] == "ecg":
        tr = fg.ECG2DTracker(_leads(c))
        tr.step = 10
        trackers["ecg"] = tr
    for tr in trackers.values():
        seq.add_tracker(tr)
    if trackers:
        model.tracker_sequence = seq
    if c["kind"] == "whole":
        stims = fg.StimSequence()
        stims.add_stim(fg.StimVoltageCoord2D(0, 1.0, 0, c["ni"], 1 + seed % 5, 9 + seed % 5))
        model.stim_sequence = stims
    return model, trackers


def _cells(c):
    return [[c["ni"] // 2, c["nj"] // 4], [c["ni"] // 3, c["nj"] // 2]]


def _leads(c):
    return np.array([[c["ni"] * 0.5, -8.0, 10.0], [c["ni"] * 0.25, c["nj"] * 0.5, 25.0],
                     [c["ni"] + 20.0, c["nj"] + 20.0, 15.0], [c["ni"] * 0.5, c["nj"] * 1.2, 12.0]])


def _set_state(model, mesh, state):
    """What a program loads into an initialised model; nodes outside the
    tissue keep the initial potential."""
    myo = mesh == 1
    model.u = torch.where(myo, state["u"], torch.full_like(state["u"], _init_u(model))).cpu().numpy()
    for name, x in state.items():
        if name != "u":
            setattr(model, name, x.cpu().numpy())


def _tissues(c):
    """The batch's tissues: sides log-uniform in [nj, nk], `ni` of them."""
    rng = random.Random(c["mix"])
    out = []
    for _ in range(c["ni"]):
        side = _log(rng, c["nj"], c["nk"])
        out.append(_case(model=rng.choice(["ap", "ms", "fk"]), ni=side, nj=side,
                         fibers=rng.choice(["none", "smooth"]),
                         fibrosis=round(rng.uniform(0.0, 0.3), 3), steps=c["steps"], track="lat"))
    return out


def prepare(case, seed):
    if case["kind"] == "batch":
        parts = []
        for k, c in enumerate(_tissues(case)):
            mesh, fibers, state = _inputs(c, seed * 64 + k)
            model, trackers = _build(c, seed, mesh, fibers)
            model.initialize()
            _set_state(model, mesh, state)
            parts.append((model, trackers["lat"]))
        return {"case": case, "parts": parts, "batch": fg.TissueBatch([m for m, _ in parts])}
    mesh, fibers, state = _inputs(case, seed)
    model, trackers = _build(case, seed, mesh, fibers)
    if case["kind"] == "chunk":
        model.initialize()
        _set_state(model, mesh, state)
    return {"case": case, "model": model, "trackers": trackers}


def _on_device(model):
    """The state where the program keeps it between chunks: on the device."""
    return {n: model._dev[n] for n in ["u"] + list(model._state_names)}


def run(state):
    c = state["case"]
    if c["kind"] == "batch":
        for m, _ in state["parts"]:
            m.t_max = m.t + (c["steps"] - 0.5) * m.dt
        state["batch"].run(initialize=False)
        return [dict(_on_device(m), count=tr._count) for m, tr in state["parts"]]
    m = state["model"]
    if c["kind"] == "whole":
        m.run()
        out = {n: np.asarray(getattr(m, n)) for n in ["u"] + list(m._state_names)}
        out.update({k: tr.output for k, tr in state["trackers"].items()})
        return out
    m.t_max = m.t + (c["steps"] - 0.5) * m.dt
    m.run(initialize=False)
    out = _on_device(m)
    if "act" in state["trackers"]:
        out["act"] = state["trackers"]["act"]._act_step
    return out


# operations of one node's ionic update, an exponential or division counted
# as one
_OPS = {"ap": 18, "ms": 12, "fk": 30, "bo": 50, "tp06": 640, "crn": 640, "lr91": 260}


def work(case):
    """Inputs (state, mesh, fibers) read once and outputs (state, records)
    written once per pass; the operations of every step."""
    if case["kind"] == "batch":
        parts = [work(c) for c in _tissues(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    n = float(np.prod(_shape(case)))
    b = 8 if case["prec"] == "float64" else 4
    dim, aniso = _dim(case), case["fibers"] != "none"
    conc = _CONC.get(case["model"], ())
    per = b + sum(8 if s[0] in conc else b for s in _STATE[case["model"]])
    rec = 0 if case["track"] in ("none", "ecg") else 4
    nw = (9 if dim == 2 else 19) if aniso else (5 if dim == 2 else 7)
    reads = (0 if case["kind"] == "whole" else per) + 1 + (dim * b if aniso else 0)
    myo = n * (1.0 - case["fibrosis"])
    return {"bytes": n * (reads + per + rec),
            "flops": myo * case["steps"] * (2 * nw - 1 + _OPS[case["model"]])}


# ------------------------------------------------------------------ exact
# The same simulations in float64 with plain torch operations.

def _at(x, off):
    """x at the node displaced by `off` (the outer ring is never a myocyte)."""
    return torch.roll(x, [-o for o in off], list(range(x.dim())))


def _weights(mesh, fibers, D_model):
    """{offset: weight}: finite-difference weights of the diffusion step."""
    dim, shape = mesh.dim(), mesh.shape
    m = (mesh == 1).double()
    zero = (0,) * dim
    w = {zero: torch.zeros(shape, dtype=torch.float64, device=mesh.device)}

    def unit(a, s):
        return tuple(s if d == a else 0 for d in range(dim))

    def add(off, v):
        w[off] = w[off] + v if off in w else v

    def both(p, q):
        return tuple(x + y for x, y in zip(p, q))
    if fibers is None:
        for a in range(dim):
            for s in (1, -1):
                m0, m1 = _at(m, unit(a, s)), _at(m, unit(a, -s))
                add(unit(a, s), m0 * (m0 + (m1 == 0).double()))
        total = sum(v for k, v in w.items() if k != zero)
        w[zero] = -total
    else:
        D_al, D_ac = 1.0, 0.111
        for a in range(dim):
            for b in range(dim):
                D = D_ac * float(a == b) + (D_al - D_ac) * fibers[..., a] * fibers[..., b]
                half = 0.5 * (D + _at(D, unit(a, 1)))
                for s in (1, -1):
                    face = half if s == 1 else _at(half, unit(a, -1))
                    ea, eb, nb = unit(a, s), unit(b, 1), unit(b, -1)
                    if a == b:
                        q = face * _at(m, ea)
                        add(ea, q)
                        add(zero, -q)
                        continue
                    offs = [both(ea, nb), nb, ea, zero, both(ea, eb), eb]
                    ms = [_at(m, o) for o in offs]
                    hi, lo = ms[2] + ms[3] + ms[4] + ms[5], ms[0] + ms[1] + ms[2] + ms[3]
                    ok = (ms[2] > 0) & (ms[3] > 0) & (hi >= 3) & (lo >= 3)
                    f = s * torch.where(ok, face, torch.zeros_like(face))
                    hi, lo = hi.clamp(min=1), lo.clamp(min=1)
                    for k, o in enumerate(offs):
                        g = torch.zeros_like(f)
                        if k < 4:
                            g = g - ms[k] / lo
                        if k >= 2:
                            g = g + ms[k] / hi
                        add(o, f * g)
    scale = D_model * DT / DR ** 2
    w = {k: v * scale for k, v in w.items()}
    w[zero] = w[zero] + 1.0
    return w


def _diffuse(u, w):
    return sum(_at(u, off) * v for off, v in w.items())


def _gate(x, inf, tau):
    return inf - (inf - x) * torch.exp(-DT / tau)


def _ionic_ap(u, un, s):
    p = _P["ap"]
    v = s["v"]
    v = v - DT * (p["eap"] + p["mu_1"] * v / (p["mu_2"] + u)) * (v + p["k"] * u * (u - p["a"] - 1))
    s["v"] = v
    return un + DT * (-p["k"] * u * (u - p["a"]) * (u - 1) - u * v)


def _ionic_ms(u, un, s):
    p = _P["ms"]
    h = s["h"]
    h = h + torch.where(u < p["u_gate"], DT * (1 - h) / p["tau_open"], -DT * h / p["tau_close"])
    s["h"] = h
    return un + DT * (h * u * u * (1 - u) / p["tau_in"] - u / p["tau_out"])


def _ionic_fk(u, un, s):
    p = _P["fk"]
    h1, h2 = (p["u_c"] - u >= 0).double(), (u - p["u_c"] >= 0).double()
    v = s["v"] + DT * (h1 * (1 - s["v"]) / p["tau_v_m"] - h2 * s["v"] / p["tau_v_p"])
    w = s["w"] + DT * (h1 * (1 - s["w"]) / p["tau_w_m"] - h2 * s["w"] / p["tau_w_p"])
    s["v"], s["w"] = v, w
    j_fi = -v * h2 * (1 - u) * (u - p["u_c"]) / p["tau_d"]
    j_so = u * h1 / p["tau_o"] + h2 / p["tau_r"]
    j_si = -v * (1 + torch.tanh(p["k"] * (u - p["uc_si"]))) / (2 * p["tau_si"])
    return un + DT * (-j_fi - j_so - j_si)


def _ionic_bo(u, un, s):
    p = _P["bo"]
    one = torch.ones_like(u)
    v, w = s["v"], s["w"]
    v_inf = (u < p["theta_v_m"]).double()
    tau_vm = torch.where(u < p["theta_v_m"], p["tau_v1_m"] * one, p["tau_v2_m"] * one)
    s["v"] = v = v + DT * torch.where(u < p["theta_v"], (v_inf - v) / tau_vm, -v / p["tau_v_p"])
    w_inf = torch.where(u < p["theta_o"], 1 - u / p["tau_w_inf"], p["w_inf_"] * one)
    tau_wm = p["tau_w1_m"] + (p["tau_w2_m"] - p["tau_w1_m"]) * (
        1 + torch.tanh(p["k_w_m"] * (u - p["u_w_m"]))) / 2
    s["w"] = w = w + DT * torch.where(u < p["theta_w"], (w_inf - w) / tau_wm, -w / p["tau_w_p"])
    tau_s = torch.where(u < p["theta_w"], p["tau_s1"] * one, p["tau_s2"] * one)
    s["s"] = s["s"] + DT * ((1 + torch.tanh(p["k_s"] * (u - p["u_s"]))) / 2 - s["s"]) / tau_s
    hv, hw = (u >= p["theta_v"]).double(), (u >= p["theta_w"]).double()
    j_fi = -v * hv * (u - p["theta_v"]) * (p["u_u"] - u) / p["tau_fi"]
    tau_o = torch.where(u < p["theta_o"], p["tau_o1"] * one, p["tau_o2"] * one)
    tau_so = p["tau_so1"] + (p["tau_so2"] - p["tau_so1"]) * (
        1 + torch.tanh(p["k_so"] * (u - p["u_so"]))) / 2
    j_so = (u - p["u_o"]) * (1 - hw) / tau_o + hw / tau_so
    j_si = -hw * w * s["s"] / p["tau_si"]
    return un + DT * (-j_fi - j_so - j_si)


def _fast_na(u, aj):
    """h and j rates shared by the detailed models: (ah, bh, j alpha)."""
    e = torch.exp
    return aj * (u + 37.78) / (1 + e(0.311 * (u + 79.23)))


def _ionic_tp06(u, un, s):
    e, log, sqrt = torch.exp, torch.log, torch.sqrt
    F, R, T, RTONF, cap = 96485.3415, 8314.472, 310.0, 26.71376, 0.185
    Vc, Vsr, Vss = 0.016404, 0.001094, 0.00005468
    ko, cao, nao = 5.4, 2.0, 140.0
    RT = R * T
    cai, casr, cass, nai, Ki = s["cai"], s["casr"], s["cass"], s["nai"], s["Ki"]
    Ek, Ena = RTONF * log(ko / Ki), RTONF * log(nao / nai)
    Eks = RTONF * log((ko + 0.03 * nao) / (Ki + 0.03 * nai))
    Eca = 0.5 * RTONF * log(cao / cai)
    tau_m = 1 / (1 + e((-60 - u) / 5)) * (0.1 / (1 + e((u + 35) / 5)) + 0.1 / (1 + e((u - 50) / 200)))
    m_inf = 1 / (1 + e((-56.86 - u) / 9.03)) ** 2
    up = u >= -40.0
    zero = torch.zeros_like(u)
    ah = torch.where(up, zero, 0.057 * e(-(u + 80) / 6.8))
    bh = torch.where(up, 0.77 / (0.13 * (1 + e(-(u + 10.66) / 11.1))),
                     2.7 * e(0.079 * u) + 310000.0 * e(0.3485 * u))
    aj = torch.where(up, zero, _fast_na(u, -25428.0 * e(0.2444 * u) - 6.948e-06 * e(-0.04391 * u)))
    bj = torch.where(up, 0.6 * e(0.057 * u) / (1 + e(-0.1 * (u + 32))),
                     0.02424 * e(-0.01052 * u) / (1 + e(-0.1378 * (u + 40.14))))
    h_inf = 1 / (1 + e((u + 71.55) / 7.43)) ** 2
    s["m"] = _gate(s["m"], m_inf, tau_m)
    s["h"] = _gate(s["h"], h_inf, 1 / (ah + bh))
    s["j"] = _gate(s["j"], h_inf, 1 / (aj + bj))
    ina = 14.838 * s["m"] ** 3 * s["h"] * s["j"] * (u - Ena)
    tau_d = (1.4 / (1 + e((-35 - u) / 13)) + 0.25) * (1.4 / (1 + e((u + 5) / 5))) + 1 / (1 + e((50 - u) / 20))
    tau_f = 1102.5 * e(-(u + 27) ** 2 / 225) + 200 / (1 + e((13 - u) / 10)) + 180 / (1 + e((u + 30) / 10)) + 20
    tau_f2 = 600 * e(-(u + 25) ** 2 / 170) + 31 / (1 + e((25 - u) / 10)) + 16 / (1 + e((u + 30) / 10))
    q = (cass / 0.05) ** 2
    s["d"] = _gate(s["d"], 1 / (1 + e((-8 - u) / 7.5)), tau_d)
    s["f"] = _gate(s["f"], 1 / (1 + e((u + 20) / 7)), tau_f)
    s["f2"] = _gate(s["f2"], 0.67 / (1 + e((u + 35) / 7)) + 0.33, tau_f2)
    s["fcass"] = _gate(s["fcass"], 0.6 / (1 + q) + 0.4, 80 / (1 + q) + 2)
    z = 2 * (u - 15) * F / RT
    ical = (3.98e-5 * s["d"] * s["f"] * s["f2"] * s["fcass"] * 4 * (u - 15) * (F * F / RT) *
            (0.25 * e(z) * cass - cao) / torch.expm1(z))
    s["s"] = _gate(s["s"], 1 / (1 + e((u + 20) / 5)),
                   85 * e(-(u + 45) ** 2 / 320) + 5 / (1 + e((u - 20) / 5)) + 3)
    s["r"] = _gate(s["r"], 1 / (1 + e((20 - u) / 6)), 9.5 * e(-(u + 40) ** 2 / 1800) + 0.8)
    ito = 0.294 * s["r"] * s["s"] * (u - Ek)
    s["xr1"] = _gate(s["xr1"], 1 / (1 + e((-26 - u) / 7)),
                     450 / (1 + e((-45 - u) / 10)) * (6 / (1 + e((u + 30) / 11.5))))
    s["xr2"] = _gate(s["xr2"], 1 / (1 + e((u + 88) / 24)),
                     3 / (1 + e((-60 - u) / 20)) * (1.12 / (1 + e((u - 60) / 20))))
    ikr = 0.153 * math.sqrt(ko / 5.4) * s["xr1"] * s["xr2"] * (u - Ek)
    s["xs"] = _gate(s["xs"], 1 / (1 + e((-5 - u) / 14)),
                    1400 / sqrt(1 + e((5 - u) / 6)) / (1 + e((u - 35) / 15)) + 80)
    iks = 0.392 * s["xs"] ** 2 * (u - Eks)
    ak1 = 0.1 / (1 + e(0.06 * (u - Ek - 200)))
    bk1 = (3 * e(0.0002 * (u - Ek + 100)) + e(0.1 * (u - Ek - 10))) / (1 + e(-0.5 * (u - Ek)))
    ik1 = 5.405 * ak1 / (ak1 + bk1) * (u - Ek)
    ncx = (1000 / (87.5 ** 3 + nao ** 3) / (1.38 + cao) / (1 + 0.1 * e(-0.65 * u * F / RT)) *
           (e(0.35 * u * F / RT) * nai ** 3 * cao - e(-0.65 * u * F / RT) * nao ** 3 * cai * 2.5))
    rec = 1 / (1 + 0.1245 * e(-0.1 * u * F / RT) + 0.0353 * e(-u * F / RT))
    inak = 2.724 * (ko / (ko + 1.0)) * (nai / (nai + 40.0)) * rec
    ipca = 0.1238 * cai / (0.0005 + cai)
    ipk = 0.0146 / (1 + e((25 - u) / 5.98)) * (u - Ek)
    ibna, ibca = 0.00029 * (u - Ena), 0.000592 * (u - Eca)
    k_sr = 2.5 - 1.5 / (1 + (1.5 / casr) ** 2)
    k1, k2 = 0.15 / k_sr, 0.045 * k_sr
    s["rr"] = s["rr"] + DT * (0.005 * (1 - s["rr"]) - k2 * cass * s["rr"])
    s["oo"] = k1 * cass ** 2 * s["rr"] / (0.060 + k1 * cass ** 2)
    irel = 0.102 * s["oo"] * (casr - cass)
    ileak, iup = 0.00036 * (casr - cai), 0.006375 / (1 + 0.00025 ** 2 / cai ** 2)
    ixfer = 0.0038 * (cass - cai)
    dsr = DT * (iup - irel - ileak)
    dss = DT * (-ixfer * (Vc / Vss) + irel * (Vsr / Vss) - ical * cap / (2 * Vss * F))
    b = 10.0 - 10.0 * casr / (casr + 0.3) - dsr - casr + 0.3
    c = 0.3 * (10.0 * casr / (casr + 0.3) + dsr + casr)
    s["casr"] = (sqrt(b * b + 4 * c) - b) / 2
    b = 0.4 - 0.4 * cass / (cass + 0.00025) - dss - cass + 0.00025
    c = 0.00025 * (0.4 * cass / (cass + 0.00025) + dss + cass)
    s["cass"] = (sqrt(b * b + 4 * c) - b) / 2
    s["nai"] = nai - DT * (ina + ibna + 3 * inak + 3 * ncx) * cap / (Vc * F)
    s["Ki"] = Ki - DT * (ik1 + ito + ikr + iks - 2 * inak + ipk) * cap / (Vc * F)
    return un - DT * (ikr + iks + ik1 + ito + ina + ibna + ical + ibca + inak + ncx + ipca + ipk)


def _ionic_crn(u, un, s):
    e, log, sqrt = torch.exp, torch.log, torch.sqrt
    F, T, R = 96485.0, 310.0, 8314.0
    Vj = 20100 * 0.68
    Vup, Vrel = Vj * 0.06 * 0.92, Vj * 0.06 * 0.08
    cao, nao, ko = 1.8, 140.0, 5.4
    RT = R * T
    nai, ki, cai, caup, carel = s["nai"], s["ki"], s["cai"], s["caup"], s["carel"]
    ena, ek = RT / F * log(nao / nai), RT / F * log(ko / ki)
    eca = RT / (2 * F) * log(cao / cai)
    am = 0.32 * (u + 47.13) / -torch.expm1(-0.1 * (u + 47.13))
    am = torch.where(u == -47.13, torch.full_like(u, 3.2), am)
    bm = 0.08 * e(-u / 11)
    s["m"] = _gate(s["m"], am / (am + bm), 1 / (am + bm))
    up = u >= -40
    zero = torch.zeros_like(u)
    ah = torch.where(up, zero, 0.135 * e(-(80 + u) / 6.8))
    bh = torch.where(up, 1 / (0.13 * (1 + e(-(u + 10.66) / 11.1))),
                     3.56 * e(0.079 * u) + 310000 * e(0.35 * u))
    aj = torch.where(up, zero, _fast_na(u, -127140 * e(0.2444 * u) - 3.474e-05 * e(-0.04391 * u)))
    bj = torch.where(up, 0.3 * e(-2.535e-07 * u) / (1 + e(-0.1 * (u + 32))),
                     0.1212 * e(-0.01052 * u) / (1 + e(-0.1378 * (u + 40.14))))
    s["h"] = _gate(s["h"], ah / (ah + bh), 1 / (ah + bh))
    s["j_"] = _gate(s["j_"], aj / (aj + bj), 1 / (aj + bj))
    ina = 7.8 * s["m"] ** 3 * s["h"] * s["j_"] * (u - ena)
    ik1 = 0.09 * (u - ek) / (1 + e(0.07 * (u + 80)))
    ao = 0.65 / (e(-(u + 10) / 8.5) + e(-(u - 30) / 59.0))
    bo = 0.65 / (2.5 + e((u + 82) / 17.0))
    tau = 1 / (3 * (ao + bo))
    tau_oi = 1 / (3 * (1 / (18.53 + e((u + 113.7) / 10.95)) + 1 / (35.56 + e(-(u + 1.26) / 7.44))))
    s["oa"] = _gate(s["oa"], 1 / (1 + e(-(u + 20.47) / 17.54)), tau)
    s["oi"] = _gate(s["oi"], 1 / (1 + e((u + 43.1) / 5.3)), tau_oi)
    ito = 0.1652 * s["oa"] ** 3 * s["oi"] * (u - ek)
    gkur = 0.005 + 0.05 / (1 + e(-(u - 15) / 13.0))
    tau_ui = 1 / (3 * (1 / (21 + e(-(u - 185) / 28.0)) + e((u - 158) / 16.0)))
    s["ua"] = _gate(s["ua"], 1 / (1 + e(-(u + 30.3) / 9.6)), tau)
    s["ui"] = _gate(s["ui"], 1 / (1 + e((u - 99.45) / 27.48)), tau_ui)
    ikur = gkur * s["ua"] ** 3 * s["ui"] * (u - ek)
    axr = 0.0003 * (u + 14.1) / -torch.expm1(-(u + 14.1) / 5)
    bxr = 7.3898e-05 * (u - 3.3328) / torch.expm1((u - 3.3328) / 5.1237)
    s["xs"] = _gate(s["xs"], 1 / (1 + e(-(u + 14.1) / 6.5)), 1 / (axr + bxr))
    ikr = 0.0294 * s["xs"] * (u - ek) / (1 + e((u + 15) / 22.4))
    axs = 4e-05 * (u - 19.9) / -torch.expm1(-(u - 19.9) / 17)
    bxs = 3.5e-05 * (u - 19.9) / torch.expm1((u - 19.9) / 9)
    s["xr"] = _gate(s["xr"], 1 / sqrt(1 + e(-(u - 19.9) / 12.7)), 1 / (2 * (axs + bxs)))
    iks = 0.129 * s["xr"] ** 2 * (u - ek)
    ex = e(-(u + 10) / 6.24)
    tau_d = -torch.expm1(-(u + 10) / 6.24) / (0.035 * (u + 10) * (1 + ex))
    tau_f = 9 / (0.0197 * e(-(0.0337 ** 2) * (u + 10) ** 2) + 0.02)
    s["d"] = _gate(s["d"], 1 / (1 + e(-(u + 10) / 8.0)), tau_d)
    s["f"] = _gate(s["f"], 1 / (1 + e((u + 28) / 6.9)), tau_f)
    s["fca"] = _gate(s["fca"], 1 / (1 + cai / 0.00035), torch.full_like(u, 2.0))
    ical = 0.1238 * s["d"] * s["f"] * s["fca"] * (u - 65)
    sg = (math.exp(nao / 67.3) - 1) / 7.0
    fnak = 1 / (1 + 0.1245 * e(-0.1 * F * u / RT) + 0.0365 * sg * e(-F * u / RT))
    inak = 0.6 * fnak / (1 + (10 / nai) ** 1.5) * (ko / (ko + 1.5))
    fwd, rev = e(0.35 * F * u / RT), e(-0.65 * F * u / RT)
    ncx = 1600 * (fwd * nai ** 3 * cao - rev * nao ** 3 * cai) / (
        (87.5 ** 3 + nao ** 3) * (1.38 + cao) * (1 + 0.1 * rev))
    ibca, ibna = 0.00113 * (u - eca), 0.000674 * (u - ena)
    ipca = 0.275 * cai / (cai + 0.0005)
    Fn = 1e-12 * Vrel * s["irel"] - 5e-13 / F * (0.5 * ical - 0.2 * ncx)
    ef = e(-(Fn - 3.4175e-13) / 1.367e-15)
    tau_w = 6 * -torch.expm1(-(u - 7.9) / 5) / ((1 + 0.3 * e(-(u - 7.9) / 5)) * (u - 7.9))
    s["urel"] = _gate(s["urel"], 1 / (1 + ef), torch.full_like(u, 8.0))
    s["vrel"] = _gate(s["vrel"], 1 - 1 / (1 + e(-(Fn - 6.835e-14) / 1.367e-15)), 1.91 + 2.09 / (1 + ef))
    s["wrel"] = _gate(s["wrel"], 1 - 1 / (1 + e(-(u - 40) / 17.0)), tau_w)
    s["irel"] = irel = 30 * s["urel"] ** 2 * s["vrel"] * s["wrel"] * (carel - cai)
    itr = (caup - carel) / 180
    iup, leak = 0.005 / (1 + 0.00092 / cai), caup / 15 * 0.005
    s["caup"] = caup + DT * (iup - leak - itr * (Vrel / Vup))
    s["nai"] = nai + DT * (-3 * inak - 3 * ncx - ibna - ina) / (F * Vj)
    s["ki"] = ki + DT * (2 * inak - ik1 - ito - ikur - ikr - iks) / (F * Vj)
    b1 = (2 * ncx - ipca - ical - ibca) / (2 * F * Vj) + (Vup * (leak - iup) + irel * Vrel) / Vj
    b2 = 1 + 0.07 * 0.0005 / (cai + 0.0005) ** 2 + 0.05 * 0.00238 / (cai + 0.00238) ** 2
    s["cai"] = cai + DT * b1 / b2
    s["carel"] = carel + DT * (itr - irel) / (1 + 10.0 * 0.8 / (carel + 0.8) ** 2)
    return un - DT * (ina + ik1 + ito + ikur + ikr + iks + ical + ipca + inak + ncx + ibna + ibca)


def _ionic_lr91(u, un, s):
    e = torch.exp
    RTF = 8.314 * 310.0 / 96.5
    up = u >= -40.0
    zero = torch.zeros_like(u)

    def step(x, a, b):
        return x + DT * (a - (a + b) * x)
    ah = torch.where(up, zero, 0.135 * e(-(80 + u) / 6.8))
    bh = torch.where(up, 1 / (0.13 * (1 + e(-(u + 10.66) / 11.1))), 3.56 * e(0.079 * u) + 3.1e5 * e(0.35 * u))
    aj = torch.where(up, zero, _fast_na(u, -1.2714e5 * e(0.2444 * u) - 3.474e-5 * e(-0.04391 * u)))
    bj = torch.where(up, 0.3 * e(-2.535e-07 * u) / (1 + e(-0.1 * (u + 32))),
                     0.1212 * e(-0.01052 * u) / (1 + e(-0.1378 * (u + 40.14))))
    am = 0.32 * (u + 47.13) / -torch.expm1(-0.1 * (u + 47.13))
    s["m"] = step(s["m"], am, 0.08 * e(-u / 11))
    s["h"], s["j"] = step(s["h"], ah, bh), step(s["j"], aj, bj)
    ina = 23.0 * s["m"] ** 3 * s["h"] * s["j"] * (u - RTF * math.log(140.0 / 18.0))
    isi = 0.09 * s["d"] * s["f"] * (u - (7.7 - 13.0287 * torch.log(s["cai"])))
    ad = 0.095 * e(-0.01 * (u - 5)) / (1 + e(-0.072 * (u - 5)))
    bd = 0.07 * e(-0.017 * (u + 44)) / (1 + e(0.05 * (u + 44)))
    af = 0.012 * e(-0.008 * (u + 28)) / (1 + e(0.15 * (u + 28)))
    bf = 0.0065 * e(-0.02 * (u + 30)) / (1 + e(-0.2 * (u + 30)))
    s["d"], s["f"] = step(s["d"], ad, bd), step(s["f"], af, bf)
    s["cai"] = s["cai"] + DT * (-0.0001 * isi + 0.07 * (0.0001 - s["cai"]))
    E_K = RTF * math.log((5.4 + 0.01833 * 140.0) / (145.0 + 0.01833 * 18.0))
    Xi = torch.where(u > -100, 2.837 * torch.expm1(0.04 * (u + 77)) / ((u + 77) * e(0.04 * (u + 35))),
                     torch.ones_like(u))
    ik = 0.282 * s["x"] * Xi * (u - E_K)
    s["x"] = step(s["x"], 0.0005 * e(0.083 * (u + 50)) / (1 + e(0.057 * (u + 50))),
                  0.0013 * e(-0.06 * (u + 20)) / (1 + e(-0.04 * (u + 20))))
    E1 = RTF * math.log(5.4 / 145.0)
    ak = 1.02 / (1 + e(0.2385 * (u - E1 - 59.215)))
    bk = (0.49124 * e(0.08032 * (u - E1 + 5.476)) + e(0.06175 * (u - E1 - 594.31))) / (
        1 + e(-0.5143 * (u - E1 + 4.753)))
    ik1 = 0.6047 * ak / (ak + bk) * (u - E1)
    ikp = 0.0183 / (1 + e((7.488 - u) / 5.98)) * (u - E1)
    return un - DT * (ina + isi + ik1 + ikp + 0.03921 * (u + 59.87) + ik)


_IONIC = {"ap": _ionic_ap, "ms": _ionic_ms, "fk": _ionic_fk, "bo": _ionic_bo,
          "tp06": _ionic_tp06, "crn": _ionic_crn, "lr91": _ionic_lr91}


def _exact_one(c, seed, data_seed):
    mesh, fibers, state = _inputs(c, data_seed)
    myo = mesh == 1
    init = {"tp06": -84.5, "crn": -84.5, "lr91": -84.5}.get(c["model"], 0.0)
    f32 = c["prec"] == "float32"
    conc = _CONC.get(c["model"], ())
    names = [n for n, _, _ in _STATE[c["model"]]]
    if c["kind"] == "whole":
        start = {"v": 1.0 if c["model"] == "fk" else 0.0, "h": 1.0, "w": 1.0}
        state = {n: torch.full(_shape(c), start[n], dtype=torch.float64, device=_dev()) for n in names}
        state["u"] = torch.zeros(_shape(c), dtype=torch.float64, device=_dev())
    u = torch.where(myo, state["u"], torch.full_like(state["u"], init))
    s = {n: state[n] for n in names}
    if f32:
        u = u.float().double()
        s = {n: x if n in conc else x.float().double() for n, x in s.items()}
    w = _weights(mesh, fibers, _D_MODEL.get(c["model"], 1.0))
    probes, ecg = [], []
    if c["track"] == "ecg":
        ii, jj = torch.meshgrid(*[torch.arange(n, dtype=torch.float64, device=_dev()) for n in _shape(c)],
                                indexing="ij")
        inv = [torch.where(myo, 1 / (((x - ii) ** 2 + (y - jj) ** 2 + z * z) * DR), torch.zeros_like(ii))
               for x, y, z in _leads(c)]
    for n in range(c["steps"]):
        if c["kind"] == "whole" and n == 0:
            y = 1 + seed % 5
            box = torch.zeros_like(myo)
            box[:, y:y + 8] = True
            u = torch.where(myo & box, torch.ones_like(u), u)
        un = _diffuse(u, w)
        if "probe" in c["track"]:
            probes.append(torch.stack([u[i, j] for i, j in _cells(c)]))
        if c["track"] == "ecg" and n % 10 == 0:
            ecg.append(torch.stack([((un - u) * k).sum() for k in inv]))
        old = dict(s)
        un = _IONIC[c["model"]](u, un, s)
        s = {k: torch.where(myo, s[k], old[k]) for k in s}
        u = torch.where(myo, un, u)
    out = {"u": u}
    for n in names:
        if f32 and n in conc:
            hi = s[n].float().double()
            out[n] = torch.stack([hi, s[n] - hi], -1)
        else:
            out[n] = s[n]
    if probes:
        out["probe"] = torch.stack(probes)
    if ecg:
        out["ecg"] = torch.stack(ecg)
    if "act" in c["track"]:
        out["act"] = None   # whole steps: compared as they are
    return out


def exact(case, seed):
    if case["kind"] == "batch":
        return [dict(_exact_one(c, seed, seed * 64 + k), count=None)
                for k, c in enumerate(_tissues(case))]
    return _exact_one(case, seed, seed)
