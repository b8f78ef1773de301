"""GPU: the exponentials, logarithms and reciprocals of the detailed models
(csrc/fw_math.cuh), compiled into a small library of their own, against
extended-precision values, and the models' in-range updates against their
updates in the reference's order."""
import ctypes
import os
import subprocess

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SRC = r"""
#include "fw_models_big.cuh"
template <class T>
__global__ void k_eval(int fn, const T *x, T *y, int n)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const T v = x[i];
    using namespace fw::dm;
    if constexpr (sizeof(T) == 8)
        if (fn == 5) { y[i] = ex_limited(v); return; }
    y[i] = fn == 0 ? ex(v) : fn == 1 ? lg(v) : fn == 2 ? rcp(v)
           : fn == 3 ? rsq(v) : fn == 4 ? FW_EX(v, 1 / 7.43) : x_over_expm1(v, ex(v));
}
// one step of every node by the model's update and by its update in the
// reference's order
template <class M, class T>
struct Args {
    const T *u;
    T *un;
    void *state[M::NS];
    T params[M::NP + M::ND];
    int n;
};
template <class M, class T, bool REF>
__global__ void k_update(Args<M, T> a)
{
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= a.n) return;
    const auto P = fw::load_params<T, M::NP + M::ND>(a.params);
    auto st = M::template load<T>(a.state, p);
    if constexpr (REF) a.un[p] = M::template update_ref<T>(a.u[p], a.un[p], st, P, (T)0.01);
    else a.un[p] = M::template update<T>(a.u[p], a.un[p], st, P, (T)0.01);
    M::template store<T>(a.state, p, st);
}
template <class M>
static int run(int ref, const float *u, float *un, void *const *state,
               const double *params, int n)
{
    Args<M, float> a;
    a.u = u;
    a.un = un;
    for (int i = 0; i < M::NS; ++i) a.state[i] = state[i];
    fw::fill_params<M, float>(a.params, params, 0.01);
    a.n = n;
    if (ref) k_update<M, float, true><<<(n + 127) / 128, 128>>>(a);
    else k_update<M, float, false><<<(n + 127) / 128, 128>>>(a);
    return (int)cudaDeviceSynchronize();
}
extern "C" __attribute__((visibility("default"))) int
update(int model, int ref, const float *u, float *un, void *const *state,
       const double *params, int n)
{
    return model == 0 ? run<fw::ModelTP06>(ref, u, un, state, params, n) : -1;
}
extern "C" __attribute__((visibility("default"))) int
eval(int fn, int f64, const void *x, void *y, int n)
{
    if (f64) k_eval<double><<<(n + 255) / 256, 256>>>(fn, (const double *)x, (double *)y, n);
    else k_eval<float><<<(n + 255) / 256, 256>>>(fn, (const float *)x, (float *)y, n);
    return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for -m gpu tests")
    from finitewave_gb300 import _build
    d = tmp_path_factory.mktemp("math")
    src, out = str(d / "m.cu"), str(d / "libm.so")
    with open(src, "w") as f:
        f.write(SRC)
    subprocess.run([_build.nvcc()] + _build.ARCH +
                   _build.UNITS["fw_step_detailed_tp06_f32.cu"] +
                   ["-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-shared",
                    "--expt-relaxed-constexpr", "-I" + _build.INCLUDE,
                    "-I" + _build.CSRC, "-o", out, src], check=True)
    return ctypes.CDLL(out)


def _eval(lib, fn, x):
    d = torch.as_tensor(x, device="cuda")
    y = torch.empty_like(d)
    assert lib.eval(fn, int(x.dtype == np.float64), ctypes.c_void_p(d.data_ptr()),
                    ctypes.c_void_p(y.data_ptr()), x.size) == 0
    return y.cpu().numpy()


def _rel(got, want):
    return float(np.max(np.abs((got.astype(np.longdouble) - want) / want)))


EPS = 2.0 ** -53


@pytest.mark.skipif(np.finfo(np.longdouble).nmant < 62,
                    reason="needs a long double wider than double")
def test_float64_functions(lib):
    gen = np.random.default_rng(1)
    ld = np.longdouble
    for span in (1e-3, 1.0, 60.0, 600.0):
        x = gen.uniform(-span, span, 400000)
        # 1.5 ulp and the rounding of the polynomial's last term
        assert _rel(_eval(lib, 0, x), np.exp(x.astype(ld))) < 3.1 * EPS
        # the scale 1 / 7.43 is rounded once: half an ulp of the argument
        z = x.astype(ld) / ld("7.43")
        assert _rel(_eval(lib, 4, x), np.exp(z)) < (3.1 + span / 7.43) * EPS
    assert _eval(lib, 0, np.zeros(1))[0] == 1.0
    x = np.array([-1e6, -700.0, -690.0, 690.0, 1e9])
    y = _eval(lib, 5, x)
    assert np.all(y[:3] < 1e-299) and np.all(y[:3] > 0) and np.all(np.isfinite(y))
    x = np.exp(gen.uniform(-300, 300, 400000))
    assert _rel(_eval(lib, 2, x), 1 / x.astype(ld)) < 3.1 * EPS
    assert _rel(_eval(lib, 2, -x), -1 / x.astype(ld)) < 3.1 * EPS
    assert _rel(_eval(lib, 3, x), 1 / np.sqrt(x.astype(ld))) < 3.1 * EPS
    want = np.log(x.astype(ld))
    err = np.abs(_eval(lib, 1, x).astype(ld) - want) / np.maximum(1, np.abs(want))
    assert float(err.max()) < 3.1 * EPS
    # the ends of the table's intervals and the arguments left to CUDA's log
    x = np.concatenate([1 + np.arange(129) / 128.0, np.nextafter(1 + np.arange(1, 129) / 128.0, 0)])
    want = np.log(x.astype(ld))
    assert float(np.max(np.abs(_eval(lib, 1, x).astype(ld) - want))) < 3.1 * EPS
    y = _eval(lib, 1, np.array([0.0, -1.0, np.inf, 5e-320]))
    assert y[0] == -np.inf and np.isnan(y[1]) and y[2] == np.inf
    assert abs(y[3] - np.log(5e-320)) < 1e-12


def test_float32_quotients(lib):
    """x / (e^x - 1) of the float32 form on both sides of the switch."""
    x = np.linspace(-80, 80, 1000001).astype(np.float32)
    x = np.concatenate([x, np.linspace(-0.6, 0.6, 400001).astype(np.float32)])
    x = x[x != 0]
    want = x.astype(np.float64) / np.expm1(x.astype(np.float64))
    got = _eval(lib, 6, x)
    rel = np.abs(got - want) / np.abs(want)
    # the exponential's argument x log2(e) is rounded once (|x| 2^-24), its
    # instruction adds two ulps, e - 1 loses at most 1 / (1 - e^-1/2) = 2.5
    # of them; the reciprocal and the product one each
    assert float(np.max(rel / (1 + np.abs(x)))) < 9 * 2.0 ** -24
    assert _eval(lib, 6, np.zeros(1, np.float32))[0] == 1.0


def _arrays(fg, m, u, state):
    """Device arrays of u, u_new and the state in the model's precision."""
    dt = np.float64 if m.npfloat == "float64" else np.float32
    un = torch.as_tensor(u.astype(dt), device="cuda")
    arrs = []
    for i, name in enumerate(m._state_names):
        if fg._ffi.state_is_pair(m._model_id, m._precision(), i):
            from finitewave_gb300.model import _split_pair
            arrs.append(torch.as_tensor(_split_pair(state[name]), device="cuda"))
        else:
            arrs.append(torch.as_tensor(state[name].astype(dt), device="cuda"))
    ptr = (ctypes.c_void_p * len(arrs))(*[a.data_ptr() for a in arrs])
    par = (ctypes.c_double * len(m._param_names))(*m._params())
    return un.clone(), un, arrs, ptr, par


def _host(m, un, arrs):
    out = {"u": un.cpu().numpy().astype(np.float64)}
    for name, a in zip(m._state_names, arrs):
        a = a.cpu().numpy().astype(np.float64)
        out[name] = a[:, 0] + a[:, 1] if a.ndim == 2 else a
    return out


def _node_update(fg, model, prec, u, state):
    """One fw_ionic pass over the nodes."""
    m = getattr(fg, model)()
    m.npfloat = prec
    uu, un, arrs, ptr, par = _arrays(fg, m, u, state)
    idx = torch.arange(u.size, device="cuda")
    fg._ffi.call("fw_ionic", m._model_id, m._precision(), un.data_ptr(),
                 uu.data_ptr(), ptr, idx.data_ptr(), u.size, 0.01, par,
                 torch.cuda.current_stream().cuda_stream)
    return _host(m, un, arrs)


def _oracle_update(oracle, model, u, state):
    """The same pass by the CPU oracle, in float64."""
    spec = oracle.MODELS[model]
    un = u.copy()
    st = {k: v.copy() for k, v in state.items()}
    oracle._ionic(model, st, un, u, np.arange(u.size), 0.01, spec["params"])
    return dict(st, u=un)


def _state(fg, model, u, gen):
    m = getattr(fg, model)()
    state = {}
    for i, s in enumerate(m._state_names):
        v = float(getattr(m, "init_" + m._init_names.get(s, s)))
        if fg._ffi.state_is_pair(m._model_id, fg._ffi.F32, i):
            state[s] = v * gen.uniform(0.8, 1.25, u.size)
        elif s == "irel":
            state[s] = gen.uniform(0, 0.01, u.size)
        else:
            state[s] = gen.uniform(0, 0.2, u.size)
    return state


MODELS = [("TP062D", "tp06"), ("Courtemanche2D", "crn"), ("LuoRudy912D", "lr91")]


@pytest.mark.parametrize("model,name", MODELS)
def test_update_against_oracle(lib, oracle, model, name):
    """Every state variable after one float64 step, over potentials inside,
    around the branches of and outside the in-range update, with gates in
    [0, 0.2] (so that no calcium current empties its space in a step) and
    concentrations around their values."""
    import finitewave_gb300 as fg
    gen = np.random.default_rng(11)
    edges = np.array([-40.0, -100.0, 129.9, 130.0, -130.0, 131.0])
    u = np.concatenate([gen.uniform(-120, 100, 60000), gen.uniform(-180, 180, 2000),
                        np.repeat(edges, 8), np.repeat(edges + 1e-3, 8),
                        gen.uniform(-600, 600, 2000), [399.9, 400.0, -400.0]])
    state = _state(fg, model, u, gen)
    got = _node_update(fg, model, "float64", u, state)
    want = _oracle_update(oracle, name, u, state)
    for k in want:
        w, g = want[k], got[k]
        fine = np.isfinite(w)
        assert np.array_equal(np.isfinite(g), fine), k
        d = np.abs(g - w)[fine] / np.maximum(np.abs(w[fine]), 1.0 if k == "u" else 1e-3)
        # exponents up to 600 / 5 carry 120 half-ulps of their argument; the
        # subspace calcium's quadratic cancels four digits, the difference
        # quotients up to nine next to their poles
        assert np.quantile(d, 0.99) < 2e-13 and d.max() < 1e-8, (k, d.max())


@pytest.mark.parametrize("model,name", MODELS[:1])
def test_float32_update_no_less_exact(lib, oracle, model, name):
    """The float32 update against the float64 oracle is, variable by
    variable, no further off than the update in the reference's order is
    (half as far again at most, for the last bits that fall otherwise, and
    one rounding)."""
    import finitewave_gb300 as fg
    gen = np.random.default_rng(11)
    u = np.concatenate([gen.uniform(-120, 100, 200000),
                        np.repeat([-40.0, -100.0], 100)])
    u = u.astype(np.float32).astype(np.float64)
    state = {k: v if k in ("nai", "Ki", "ki", "cai", "casr", "cass", "caup", "carel")
             else v.astype(np.float32).astype(np.float64)
             for k, v in _state(fg, model, u, gen).items()}
    want = _oracle_update(oracle, name, u, state)
    off = []
    for ref in (0, 1):
        m = getattr(fg, model)()
        m.npfloat = "float32"
        uu, un, arrs, ptr, par = _arrays(fg, m, u, state)
        assert lib.update([n for _, n in MODELS].index(name), ref,
                          ctypes.c_void_p(uu.data_ptr()), ctypes.c_void_p(un.data_ptr()),
                          ptr, par, u.size) == 0
        got = _host(m, un, arrs)
        off.append({k: np.abs(got[k] - want[k]) /
                    np.maximum(np.abs(want[k]), 1.0 if k == "u" else 1e-3) for k in want})
    for k in want:
        new, old = off[0][k], off[1][k]
        for f in (lambda d: np.sqrt(np.mean(d * d)), lambda d: np.quantile(d, 0.99)):
            assert f(new) <= 1.5 * f(old) + 2.0 ** -24, (k, f(new), f(old))


@pytest.mark.skipif(np.finfo(np.longdouble).nmant < 62,
                    reason="needs a long double wider than double")
@pytest.mark.parametrize("span,bound", [(1.0, 1.5), (60.0, 1.5), (600.0, 2.5), (699.0, 2.5)])
def test_float64_exponential_ulps(lib, span, bound):
    """Units in the last place of the result: half each for the table and the
    last sum, the series' remainder r^5 / 120 at the largest r of the range."""
    gen = np.random.default_rng(3)
    x = gen.uniform(-span, span, 1000000)
    want = np.exp(x.astype(np.longdouble))
    ulp = np.spacing(want.astype(np.float64)).astype(np.longdouble)
    err = np.abs(_eval(lib, 0, x).astype(np.longdouble) - want) / ulp
    assert float(err.max()) < bound
