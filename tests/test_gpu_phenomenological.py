"""GPU: one float32 step of the phenomenological models against the float64
step of the same nodes, over potentials across every threshold."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

MODELS = ["AlievPanfilov2D", "MitchellSchaeffer2D", "FentonKarma2D", "Barkley2D",
          "BuenoOrovio2D"]


def _step(fg, model, prec, u, state):
    dt = np.float64 if prec == "float64" else np.float32
    m = getattr(fg, model)()
    m.npfloat = prec
    un = torch.as_tensor(u.astype(dt), device="cuda")
    uu = un.clone()
    arrs = [torch.as_tensor(s.astype(dt), device="cuda") for s in state]
    idx = torch.arange(u.size, device="cuda")
    ptr = (ctypes.c_void_p * len(arrs))(*[a.data_ptr() for a in arrs])
    par = (ctypes.c_double * len(m._param_names))(*m._params())
    fg._ffi.call("fw_ionic", m._model_id, m._precision(), un.data_ptr(),
                 uu.data_ptr(), ptr, idx.data_ptr(), u.size, 0.01, par,
                 torch.cuda.current_stream().cuda_stream)
    return [un.cpu().numpy()] + [a.cpu().numpy() for a in arrs]


@pytest.mark.parametrize("model", MODELS)
def test_float32_step(model):
    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for -m gpu tests")
    import finitewave_gb300 as fg
    gen = np.random.default_rng(5)
    # (thresholds themselves round to float32 and may fall on either side)
    u = gen.uniform(-0.1, 1.6, 200000).astype(np.float32).astype(np.float64)
    m = getattr(fg, model)()
    state = [gen.uniform(0, 1, u.size).astype(np.float32).astype(np.float64)
             for _ in m._state_names]
    got, want = _step(fg, model, "float32", u, state), _step(fg, model, "float64", u, state)
    for g, w in zip(got, want):
        # a result is its old value (at most 1.7) plus at most dt times rates
        # of up to 60 (1 / tau_d, ten of them for 1 / tau_in and eap): a few
        # roundings of 2^-24 of each
        assert np.abs(g - w).max() < 12 * 2.0 ** -24 * max(1.7, float(np.abs(w).max()))
        assert np.sqrt(np.mean((g - w) ** 2)) < 2.0 ** -24 * max(1.0, float(np.sqrt(np.mean(w * w))))


@pytest.mark.parametrize("model", MODELS)
def test_float32_step_not_finite(model):
    """NaN stays NaN and infinities raise no finite potential."""
    import finitewave_gb300 as fg
    u = np.array([np.nan, np.inf, -np.inf])
    m = getattr(fg, model)()
    state = [np.full(3, 0.5) for _ in m._state_names]
    un = _step(fg, model, "float32", u, state)[0]
    assert not np.isfinite(un).any()
