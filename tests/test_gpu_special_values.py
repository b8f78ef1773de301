"""GPU: the models' updates at potentials, parameters and time steps where an
expression of theirs has no finite value, against the CPU oracle's."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fg():
    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for -m gpu tests")
    import finitewave_gb300 as fg
    return fg


def _node_update(fg, model, prec, u, state, dt=0.01, **params):
    """One fw_ionic pass over the nodes; returns the host values of u and the
    state."""
    m = getattr(fg, model)()
    m.npfloat = prec
    for k, v in params.items():
        setattr(m, k, v)
    t = np.float64 if prec == "float64" else np.float32
    uu = torch.as_tensor(u.astype(t), device="cuda")
    un = uu.clone()
    arrs = []
    for i, name in enumerate(m._state_names):
        if fg._ffi.state_is_pair(m._model_id, m._precision(), i):
            from finitewave_gb300.model import _split_pair
            arrs.append(torch.as_tensor(_split_pair(state[name]), device="cuda"))
        else:
            arrs.append(torch.as_tensor(state[name].astype(t), device="cuda"))
    ptr = (ctypes.c_void_p * len(arrs))(*[a.data_ptr() for a in arrs])
    par = (ctypes.c_double * len(m._param_names))(*m._params())
    idx = torch.arange(u.size, device="cuda")
    fg._ffi.call("fw_ionic", m._model_id, m._precision(), un.data_ptr(),
                 uu.data_ptr(), ptr, idx.data_ptr(), u.size, dt, par,
                 torch.cuda.current_stream().cuda_stream)
    out = {"u": un.cpu().numpy().astype(np.float64)}
    for name, a in zip(m._state_names, arrs):
        a = a.cpu().numpy().astype(np.float64)
        out[name] = a[:, 0] + a[:, 1] if a.ndim == 2 else a
    return out


def _oracle_update(oracle, name, u, state, **params):
    un = u.copy()
    st = {k: v.copy() for k, v in state.items()}
    with np.errstate(all="ignore"):
        oracle._ionic(name, st, un, u, np.arange(u.size), 0.01,
                      dict(oracle.MODELS[name]["params"], **params))
    return dict(st, u=un)


def _state(fg, model, n):
    """Gates of 0.1 and the initial concentrations."""
    m = getattr(fg, model)()
    return {s: np.full(n, float(getattr(m, "init_" + m._init_names.get(s, s)))
                       if fg._ffi.state_is_pair(m._model_id, fg._ffi.F32, i) else 0.1)
            for i, s in enumerate(m._state_names)}


# potentials at which a rate or a current is 0 / 0
# (Courtemanche's alpha_m has its limit written out at -47.13)
POLES = [("Courtemanche2D", "crn", [-14.1, 3.3328, 19.9, -10.0, 7.9, -47.13], 5),
         ("LuoRudy912D", "lr91", [-47.13, -77.0], 2), ("TP062D", "tp06", [15.0], 1)]


@pytest.mark.parametrize("model,name,poles,nans", POLES)
def test_float64_poles(fg, oracle, model, name, poles, nans):
    """At the pole itself every variable is NaN exactly where the
    reference-order update's is, and right next to it finite exactly where
    that one's is."""
    p = np.array(poles)
    u = np.concatenate([p, np.nextafter(p, -1e3), np.nextafter(p, 1e3), p + 1e-9])
    state = _state(fg, model, u.size)
    got = _node_update(fg, model, "float64", u, state)
    want = _oracle_update(oracle, name, u, state)
    assert np.any([np.isnan(w) for w in want.values()], axis=0).sum() == nans
    for k in want:
        assert np.array_equal(np.isnan(got[k]), np.isnan(want[k])), k
        assert np.array_equal(np.isfinite(got[k]), np.isfinite(want[k])), k
    # away from the pole by 1e-9 a difference quotient keeps six digits
    for k in want:
        a, b = got[k][-p.size:], want[k][-p.size:]
        assert np.all(np.abs(a - b) <= 1e-5 * np.maximum(1, np.abs(b))), k


def test_pole_warns(fg):
    """A stimulus that sets such a potential is reported by the run."""
    t = fg.CardiacTissue2D((12, 13))
    m = fg.Courtemanche2D()
    m.dt, m.dr, m.t_max, m.cardiac_tissue = 0.01, 0.25, 0.01, t
    seq = fg.StimSequence()
    seq.add_stim(fg.StimVoltageCoord2D(0, -10.0, 0, 12, 0, 13))
    m.stim_sequence = seq
    with pytest.warns(RuntimeWarning, match="inf or NaN"):
        m.run()
    assert np.isnan(np.asarray(m.u)[1:-1, 1:-1]).all()


# a pump blocked by an infinite half-saturation, constants of zero, and a
# temperature at which the reversal exponents leave the in-range update's
PARAMS = [("TP062D", "tp06", dict(Kup=np.inf)), ("TP062D", "tp06", dict(KpCa=np.inf)),
          ("TP062D", "tp06", dict(k3=0.0, EC=0.0)),
          ("TP062D", "tp06", dict(gna=0.0, gto=0.0)), ("TP062D", "tp06", dict(T=3.0)),
          ("TP062D", "tp06", dict(n_=40.0)),
          ("Courtemanche2D", "crn", dict(kmnai=0.0)), ("Courtemanche2D", "crn", dict(kup=np.inf)),
          ("Courtemanche2D", "crn", dict(T=3.0)), ("Courtemanche2D", "crn", dict(caupmax=np.inf)),
          ("Courtemanche2D", "crn", dict(nao=5e4))]


# (float32 leaves its own range at T = 3 and n = 40 in any order)
@pytest.mark.parametrize("model,name,params,prec",
                         [(*p, "float64") for p in PARAMS] +
                         [(*p, "float32") for p in PARAMS[:4]])
def test_unusual_parameters(fg, oracle, model, name, params, prec):
    """One step with such parameters: finite where the reference-order update
    is, with the value it has there."""
    assert all(v in oracle.MODELS[name]["params"] for v in params)
    u = np.linspace(-95.0, 60.0, 700).astype(np.float32).astype(np.float64)
    state = _state(fg, model, u.size)
    if prec == "float32":
        state = {k: v.astype(np.float32).astype(np.float64) for k, v in state.items()}
    got = _node_update(fg, model, prec, u, state, **params)
    want = _oracle_update(oracle, name, u, state, **params)
    assert any(np.isfinite(w).all() for w in want.values())
    # float64: exponents up to 4e3 carry half an ulp of themselves; float32:
    # 1e-3 of a value is far above one step's error, far below a lost term
    tol = 1e-9 if prec == "float64" else 1e-3
    for k in want:
        w, g = want[k], got[k]
        fine = np.isfinite(w)
        assert np.array_equal(np.isfinite(g), fine), k
        assert np.all(np.abs(g - w)[fine] <= tol * np.maximum(1.0, np.abs(w[fine]))), k


@pytest.mark.parametrize("prec", ["float64", "float32"])
@pytest.mark.parametrize("model", ["BuenoOrovio2D", "TP062D", "Courtemanche2D", "LuoRudy912D"])
def test_step_of_zero(fg, model, prec):
    """An ionic pass with dt = 0 changes no potential and no gate that is
    integrated (the others go to the value they have at dt = 0: themselves)."""
    m = getattr(fg, model)()
    n = 500
    u = np.linspace(0.0, 1.5, n) if model == "BuenoOrovio2D" else np.linspace(-95, 60, n)
    u = u.astype(np.float32).astype(np.float64)
    state = {k: v.astype(np.float32).astype(np.float64)
             for k, v in _state(fg, model, n).items()}
    got = _node_update(fg, model, prec, u, state, dt=0.0)
    assert np.array_equal(got["u"], u)
    for k in m._state_names:
        if k not in ("oo", "irel"):   # algebraic: not integrated
            # one rounding where a new value is formed as inf - (inf - x)
            eps = 2.0 ** -50 if prec == "float64" else 2.0 ** -21
            assert np.all(np.abs(got[k] - state[k]) <= eps * np.maximum(1, np.abs(state[k]))), k


@pytest.mark.parametrize("prec", ["float64"])
def test_calcium_far_out(fg, oracle, prec):
    """TP06's calcium spaces from concentrations below minus their buffers'
    constants (a simulation that blows up) and from empty ones: the root that
    the reference-order quadratic takes."""
    n = 400
    gen = np.random.default_rng(2)
    state = _state(fg, "TP062D", n)
    state["cass"] = np.concatenate([-np.logspace(-5, 0, n // 2), np.logspace(-9, 0, n // 2)])
    state["casr"] = np.concatenate([gen.uniform(-3, -0.01, n // 2), gen.uniform(0.01, 8, n // 2)])
    state["rr"], state["oo"] = np.zeros(n), np.zeros(n)
    u = np.linspace(-90, 40, n)
    got = _node_update(fg, "TP062D", prec, u, state)
    want = _oracle_update(oracle, "tp06", u, state)
    for k in want:
        w, g = want[k], got[k]
        assert np.array_equal(np.isfinite(g), np.isfinite(w)), k
        # the reference's own root cancels up to eight digits of a calcium
        # of 1e-9 against its buffer of 0.4
        fine = np.isfinite(w)
        assert np.all(np.abs(g - w)[fine] <= 1e-9 * np.maximum(1.0, np.abs(w[fine]))), k


@pytest.mark.parametrize("model,name", [
    ("TP062D", "tp06"), ("Courtemanche2D", "crn"), ("LuoRudy912D", "lr91")])
def test_states_not_finite(fg, oracle, model, name):
    """One state variable of a node infinite, NaN, 0 or negative (a simulation
    that blows up): the others are finite where the reference-order update's
    are."""
    m = getattr(fg, model)()
    values = [np.inf, -np.inf, np.nan, 0.0, -0.5]
    names = list(m._state_names)
    n = len(names) * len(values)
    state = _state(fg, model, n)
    for i, k in enumerate(names):
        state[k][i * len(values):(i + 1) * len(values)] = values
    u = np.full(n, -31.25)
    got = _node_update(fg, model, "float64", u, state)
    want = _oracle_update(oracle, name, u, state)
    for k in want:
        ok = np.isfinite(got[k]) | ~np.isfinite(want[k])
        bad = [(names[i // len(values)], values[i % len(values)]) for i in np.flatnonzero(~ok)]
        assert not bad, (k, bad)
