"""GPU: one float32 step of the phenomenological models against the float64
step of the same nodes, over potentials across every threshold."""
import ctypes
import subprocess

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


SRC = r"""
#include "fw_models.cuh"
template <class M>
struct Args {
    const float *u;
    float *un;
    void *state[M::NS];
    float params[M::NP + M::ND];
    int n;
};
// FUSED: the update of the fused and batched kernels; else the expressions
// with their quotients, under the same compiler options
template <class M, bool FUSED>
__global__ void k(Args<M> a)
{
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= a.n) return;
    const auto P = fw::load_params<float, M::NP>(a.params);
    auto st = M::template load<float>(a.state, p);
    if constexpr (FUSED) a.un[p] = M::update_fused(a.u[p], a.un[p], st, P, 0.01f);
    else a.un[p] = M::template update<float>(a.u[p], a.un[p], st, P, 0.01f);
    M::template store<float>(a.state, p, st);
}
template <class M>
static int run(int fused, const float *u, float *un, void *const *state,
               const double *params, int n)
{
    Args<M> a;
    a.u = u;
    a.un = un;
    for (int i = 0; i < M::NS; ++i) a.state[i] = state[i];
    fw::fill_params<M, float>(a.params, params, 0.01);
    a.n = n;
    if (fused) k<M, true><<<(n + 127) / 128, 128>>>(a);
    else k<M, false><<<(n + 127) / 128, 128>>>(a);
    return (int)cudaDeviceSynchronize();
}
extern "C" __attribute__((visibility("default"))) int
step(int model, int fused, const float *u, float *un, void *const *state,
     const double *params, int n)
{
    return model == 0 ? run<fw::ModelMS>(fused, u, un, state, params, n)
         : model == 1 ? run<fw::ModelFK>(fused, u, un, state, params, n)
                      : run<fw::ModelBK>(fused, u, un, state, params, n);
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    from finitewave_gb300 import _build
    d = tmp_path_factory.mktemp("phen")
    src, out = str(d / "p.cu"), str(d / "libp.so")
    with open(src, "w") as f:
        f.write(SRC)
    subprocess.run([_build.nvcc()] + _build.ARCH + _build.UNITS["fw_fused_ms.cu"] +
                   ["-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-shared",
                    "--expt-relaxed-constexpr", "-I" + _build.INCLUDE,
                    "-I" + _build.CSRC, "-o", out, src], check=True)
    return ctypes.CDLL(out)


@pytest.mark.parametrize("index,model", list(enumerate(MODELS[1:4])))
def test_fused_update(lib, index, model):
    """The update of the fused kernels (products with reciprocals of the
    parameters) and the expressions with quotients, compiled alike, against
    the float64 step."""
    import finitewave_gb300 as fg
    gen = np.random.default_rng(5)
    u = gen.uniform(-0.1, 1.6, 200000).astype(np.float32).astype(np.float64)
    m = getattr(fg, model)()
    state = [gen.uniform(0, 1, u.size).astype(np.float32).astype(np.float64)
             for _ in m._state_names]
    want = _step(fg, model, "float64", u, state)
    par = (ctypes.c_double * len(m._param_names))(*m._params())
    got = []
    for fused in (1, 0):
        un = torch.as_tensor(u.astype(np.float32), device="cuda")
        uu = un.clone()
        arrs = [torch.as_tensor(s.astype(np.float32), device="cuda") for s in state]
        ptr = (ctypes.c_void_p * len(arrs))(*[a.data_ptr() for a in arrs])
        assert lib.step(index, fused, ctypes.c_void_p(uu.data_ptr()),
                        ctypes.c_void_p(un.data_ptr()), ptr, par, u.size) == 0
        got.append([un.cpu().numpy()] + [a.cpu().numpy() for a in arrs])
    for g, q, w in zip(*got, want):
        # old value (at most 1.7) plus dt times rates of up to 60, a few
        # roundings of 2^-24 of each, as for the plain step; approximate
        # reciprocals add one of each quotient
        assert np.abs(g - w).max() < 14 * 2.0 ** -24 * max(1.7, float(np.abs(w).max()))
        # the two forms differ by no more than the quotients' roundings do
        assert np.sqrt(np.mean((g - w) ** 2)) <= 1.01 * np.sqrt(np.mean((q - w) ** 2)) + 2.0 ** -40


@pytest.mark.parametrize("model", ["BuenoOrovio2D", "MitchellSchaeffer2D", "FentonKarma2D",
                                   "Barkley2D"])
def test_float32_step_far_out(model):
    """Potentials of a simulation that blows up: finite where every term of
    the float64 step's fits float32, with its value."""
    import finitewave_gb300 as fg
    u = -np.logspace(1, 12 if model in ("MitchellSchaeffer2D", "Barkley2D") else 36, 200)
    u = u.astype(np.float32).astype(np.float64)
    m = getattr(fg, model)()
    state = [np.full(u.size, 0.5) for _ in m._state_names]
    got, want = _step(fg, model, "float32", u, state), _step(fg, model, "float64", u, state)
    for g, w in zip(got, want):
        assert np.isfinite(g).all()
        assert np.all(np.abs(g - w) <= 1e-4 * np.maximum(1.0, np.abs(w)))


@pytest.mark.parametrize("model", MODELS)
def test_float32_step_state_not_finite(model):
    """A state variable that is NaN or infinite makes the same variables not
    finite as in float64."""
    import finitewave_gb300 as fg
    m = getattr(fg, model)()
    values = [np.nan, np.inf, -np.inf]
    for u0 in (0.001, 0.05, 0.2, 0.9):
        n = len(m._state_names) * 3
        state = [np.full(n, 0.5) for _ in m._state_names]
        for i in range(len(state)):
            state[i][3 * i:3 * i + 3] = values
        u = np.full(n, np.float32(u0), dtype=np.float64)
        for g, w in zip(_step(fg, model, "float32", u, state),
                        _step(fg, model, "float64", u, state)):
            assert np.array_equal(np.isfinite(g), np.isfinite(w))


@pytest.mark.parametrize("model", MODELS)
def test_float32_step_nan_as_float64(model):
    """Infinite potentials and NaN, and the state after them, are NaN and
    infinite where the float64 step's are."""
    import finitewave_gb300 as fg
    m = getattr(fg, model)()
    u = np.repeat([np.nan, np.inf, -np.inf], 2)
    state = [np.tile([0.0, 0.5], 3) for _ in m._state_names]
    for _ in range(3):
        got, want = _step(fg, model, "float32", u, state), _step(fg, model, "float64", u, state)
        for g, w in zip(got, want):
            assert np.array_equal(np.isnan(g), np.isnan(w))
            assert np.array_equal(np.isinf(g), np.isinf(w))
        u, state = want[0].astype(np.float64), [w.astype(np.float64) for w in want[1:]]
