"""GPU: TP06's in-range update is, variable by variable, no further off than
its update in the reference's order: the fast sodium gate and the open
fraction against extended precision in float64, and with the concentrations
that float32 accumulates against the float64 oracle in float32."""
import ctypes
import subprocess

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SRC = r"""
#include "fw_models_big.cuh"
using M = fw::ModelTP06;
template <class T>
struct Args {
    const T *u;
    T *un;
    void *state[M::NS];
    T params[M::NP + M::ND];
    int n;
};
template <class T, bool REF>
__global__ void k(Args<T> a)
{
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= a.n) return;
    const auto P = fw::load_params<T, M::NP + M::ND>(a.params);
    auto st = M::load<T>(a.state, p);
    if constexpr (REF) a.un[p] = M::update_ref<T>(a.u[p], a.un[p], st, P, (T)0.01);
    else a.un[p] = M::update<T>(a.u[p], a.un[p], st, P, (T)0.01);
    M::store<T>(a.state, p, st);
}
template <class T>
static int run(int ref, const void *u, void *un, void *const *state,
               const double *params, int n)
{
    Args<T> a;
    a.u = (const T *)u;
    a.un = (T *)un;
    for (int i = 0; i < M::NS; ++i) a.state[i] = state[i];
    fw::fill_params<M, T>(a.params, params, 0.01);
    a.n = n;
    if (ref) k<T, true><<<(n + 127) / 128, 128>>>(a);
    else k<T, false><<<(n + 127) / 128, 128>>>(a);
    return (int)cudaDeviceSynchronize();
}
extern "C" __attribute__((visibility("default"))) int
update(int f64, int ref, const void *u, void *un, void *const *state,
       const double *params, int n)
{
    return f64 ? run<double>(ref, u, un, state, params, n)
               : run<float>(ref, u, un, state, params, n);
}
"""


@pytest.fixture(scope="module")
def libs(tmp_path_factory):
    """(precision, reference order) -> library.  The update with the options
    of its unit; the reference's order in float64 without contraction, as the
    reference evaluates it."""
    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for -m gpu tests")
    from finitewave_gb300 import _build
    d = tmp_path_factory.mktemp("tp06")
    src = str(d / "t.cu")
    with open(src, "w") as f:
        f.write(SRC)
    made = {}
    for name, flags in (("f32", _build.UNITS["fw_step_detailed_tp06_f32.cu"]),
                        ("f64", _build.UNITS["fw_step_detailed_tp06_f64.cu"]),
                        ("ref", ["--fmad=false"])):
        out = str(d / ("lib%s.so" % name))
        subprocess.run([_build.nvcc()] + _build.ARCH + flags +
                       ["-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-shared",
                        "--expt-relaxed-constexpr", "-I" + _build.INCLUDE,
                        "-I" + _build.CSRC, "-o", out, src], check=True)
        made[name] = ctypes.CDLL(out)
    return {("float64", 0): made["f64"], ("float64", 1): made["ref"],
            ("float32", 0): made["f32"], ("float32", 1): made["f32"]}


# a variable's value at rest and up, as in a tissue in activity
RANGE = dict(cai=(7e-5, 9e-5), casr=(1.3, 1.1), cass=(7e-5, 4e-4), nai=(7.67, 7.8),
             Ki=(138.3, 137.9), m=(0.002, 0.98), h=(0.75, 0.01), j=(0.75, 0.02),
             xr1=(0.001, 0.6), xr2=(0.95, 0.2), xs=(0.004, 0.3), r=(0.001, 0.9),
             s=(0.99, 0.1), d=(0.001, 0.95), f=(0.99, 0.5), f2=(0.99, 0.6),
             fcass=(0.99, 0.7), rr=(0.99, 0.8), oo=(0.0, 1e-5))


def _nodes(n, dtype):
    gen = np.random.default_rng(5)
    a, b = gen.uniform(0, 1, n), gen.uniform(0, 1, n)
    u = (-84.5 + 109.5 * a).astype(dtype).astype(np.float64)
    state = {}
    for k, (name, (lo, hi)) in enumerate(RANGE.items()):
        x = (b, 0.5 * (a + b), 1 - (1 - a) * (1 - 0.5 * b))[k % 3]
        state[name] = lo + (hi - lo) * x
    return u, state


def _both(libs, fg, prec, u, state):
    """u_new and the state after one step by the update and by its form in
    the reference's order, and the state as it went in."""
    from finitewave_gb300.model import _split_pair
    m = fg.TP062D()
    m.npfloat = prec
    t = np.float64 if prec == "float64" else np.float32
    out, went = [], {}
    for ref in (0, 1):
        uu = torch.as_tensor(u.astype(t), device="cuda")
        un, arrs = uu.clone(), []
        for i, name in enumerate(m._state_names):
            pair = fg._ffi.state_is_pair(m._model_id, m._precision(), i)
            x = _split_pair(state[name]) if pair else state[name].astype(t)
            went[name] = x.astype(np.float64).sum(-1) if pair else x.astype(np.float64)
            arrs.append(torch.as_tensor(x, device="cuda"))
        ptr = (ctypes.c_void_p * len(arrs))(*[a.data_ptr() for a in arrs])
        par = (ctypes.c_double * len(m._param_names))(*m._params())
        assert libs[prec, ref].update(int(prec == "float64"), ref,
                                      ctypes.c_void_p(uu.data_ptr()),
                                      ctypes.c_void_p(un.data_ptr()), ptr, par, u.size) == 0
        got = {"u": un.cpu().numpy()}
        for name, a in zip(m._state_names, arrs):
            a = a.cpu().numpy().astype(np.float64)
            got[name] = a.sum(-1) if a.ndim == 2 else a
        out.append(got)
    return out[0], out[1], went, m


def _rms(got, want):
    d = got.astype(np.longdouble) - want
    return float(np.sqrt((d * d).sum() / (want * want).sum()))


@pytest.mark.skipif(np.finfo(np.longdouble).nmant < 62,
                    reason="needs a long double wider than double")
def test_float64(libs):
    import finitewave_gb300 as fg
    u, state = _nodes(100000, np.float64)
    new, ref, went, m = _both(libs, fg, "float64", u, state)
    ld = np.longdouble
    U, e = u.astype(ld), np.exp
    s = {k: v.astype(ld) for k, v in went.items()}
    tau_m = 1 / (1 + e((-60 - U) / 5)) * (0.1 / (1 + e((U + 35) / 5)) + 0.1 / (1 + e((U - 50) / 200)))
    m_inf = 1 / (1 + e((ld(-56.86) - U) / ld(9.03))) ** 2
    kcasr = m.maxsr - (m.maxsr - m.minsr) / (1 + (m.EC / s["casr"]) ** 2)
    rr = s["rr"] + ld(0.01) * (m.k4 * (1 - s["rr"]) - m.k2_ * kcasr * s["cass"] * s["rr"])
    k1 = m.k1_ / kcasr * s["cass"] ** 2
    want = {"m": m_inf - (m_inf - s["m"]) * e(-ld(0.01) / tau_m), "oo": k1 * rr / (m.k3 + k1)}
    for k, w in want.items():
        assert _rms(new[k], w) <= 1.002 * _rms(ref[k], w), (k, _rms(new[k], w), _rms(ref[k], w))


def test_float32(libs, oracle):
    import finitewave_gb300 as fg
    u, state = _nodes(200000, np.float32)
    new, ref, went, _ = _both(libs, fg, "float32", u, state)
    un, st = u.copy(), {k: v.copy() for k, v in went.items()}
    oracle._ionic("tp06", st, un, u, np.arange(u.size), 0.01, oracle.MODELS["tp06"]["params"])
    want = dict(st, u=un)
    for k in ("u", "m", "oo", "nai", "Ki", "casr"):
        a, b = _rms(new[k], want[k].astype(np.longdouble)), _rms(ref[k], want[k].astype(np.longdouble))
        assert a <= 1.002 * b, (k, a, b)
