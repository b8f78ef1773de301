"""GPU: ECG trackers (on-device reduction, fw_ecg_tracker / fw_ecg) against
the reference's golden ECG traces.  Float64: the diffusion is the
reference's (bitwise), the sum over myocytes is a parallel reduction in a
different order, so the traces agree to rounding (1e-12 of the trace's
scale).  Float32: within 1e-3 of the scale."""
import ctypes

import numpy as np
import pytest
import torch

import cases

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gc():
    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for -m gpu tests")
    from finitewave_gb300 import _ffi
    _ffi.load()
    import gpu_cases
    return gpu_cases


@pytest.mark.parametrize("npfloat,rtol", [("float64", 1e-12),
                                          ("float32", 1e-3)])
@pytest.mark.parametrize("dim", [2, 3])
def test_ecg_traces(gc, dim, npfloat, rtol):
    case, g = cases.ecg(dim)
    r = gc.run(case, npfloat=npfloat)
    ecg = np.asarray(r["trackers"][0])
    assert ecg.shape == g["ecg"].shape
    scale = np.abs(g["ecg"]).max()
    assert np.abs(ecg - g["ecg"]).max() <= rtol * scale
    if npfloat == "float64":
        assert np.array_equal(r["u"], g["u"])


def test_fw_ecg_callable(gc):
    """fw_ecg on a state of the 2D case equals the oracle's compute_ecg."""
    from finitewave_gb300 import _ffi
    from oracle import oracle
    case, _ = cases.ecg(2)
    model, _ = gc.build(case)
    model.initialize()
    rng = np.random.default_rng(3)
    u0 = rng.uniform(0, 1, model._shape())
    model.u = u0
    coords = np.array([[25, 2, 0], [10, -3, 1.5], [3, 3, 0]], np.float64)
    out = torch.zeros(3, dtype=torch.float64, device="cuda")
    ni, nj = model._shape()
    # coords stay in host memory (they are passed to the kernel by value)
    _ffi.call("fw_ecg", _ffi.ISO5, _ffi.F64, model._dev["u"].data_ptr(),
              model.weights.data_ptr(), model._myo_d.data_ptr(), ni, nj, 1,
              coords.ctypes.data, 3, model.dr, out.data_ptr(),
              torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    w = oracle.weights("iso5", case["mesh"], 1.0, case["dt"], case["dr"])
    idx = np.flatnonzero(case["mesh"] == 1).astype(np.int64)
    u_tr = np.zeros_like(u0)
    oracle._diffuse("iso5", u_tr, u0, w, idx)
    ref = oracle._ecg(u_tr, u0, coords, case["dr"], idx, u0.shape)
    np.testing.assert_allclose(out.cpu().numpy(), ref, rtol=1e-12,
                               atol=1e-15 * np.abs(ref).max())
    cd = torch.as_tensor(coords, device="cuda")
    with pytest.raises(_ffi.FwError, match="host memory"):
        _ffi.call("fw_ecg", _ffi.ISO5, _ffi.F64, model._dev["u"].data_ptr(),
                  model.weights.data_ptr(), model._myo_d.data_ptr(), ni, nj,
                  1, cd.data_ptr(), 3, model.dr, out.data_ptr(),
                  torch.cuda.current_stream().cuda_stream)


@pytest.mark.parametrize("shape", [(5, 7), (33, 130), (4, 5, 6), (17, 9, 35)])
@pytest.mark.parametrize("n_leads", [1, 3, 5, 8])
def test_fw_ecg_lead_counts(gc, shape, n_leads):
    """Every lead of one to eight gets its own sum, on grids from one warp's
    work to several CTAs'.  n terms of either sign summed in float64, in any
    order, differ by at most n eps of the sum of their magnitudes."""
    from finitewave_gb300 import _ffi
    from oracle import oracle
    rng = np.random.default_rng(n_leads)
    st, dim = ("iso5", 2) if len(shape) == 2 else ("iso7", 3)
    mesh = np.ones(shape, np.int8)
    for a in range(dim):
        edge = [slice(None)] * dim
        for e in (0, -1):
            edge[a] = e
            mesh[tuple(edge)] = 0
    u = rng.uniform(-1, 1, shape)
    w = oracle.weights(st, mesh, 1.0, 0.001, 0.25)
    coords = np.zeros((n_leads, 3))
    coords[:, :dim] = rng.uniform(-9, -2, (n_leads, dim))
    out = torch.zeros(n_leads, dtype=torch.float64, device="cuda")
    ud, wd, md = (torch.as_tensor(np.ascontiguousarray(x), device="cuda")
                  for x in (u, np.moveaxis(w, -1, 0), mesh))
    ni, nj, nk = (*shape, 1)[:3]
    _ffi.call("fw_ecg", _ffi.ISO5 if dim == 2 else _ffi.ISO7, _ffi.F64,
              ud.data_ptr(), wd.data_ptr(), md.data_ptr(), ni, nj, nk,
              coords.ctypes.data, n_leads, 0.25, out.data_ptr(),
              torch.cuda.current_stream().cuda_stream)
    idx = np.flatnonzero(mesh == 1).astype(np.int64)
    u_tr = np.zeros_like(u)
    oracle._diffuse(st, u_tr, u, w, idx)
    ref = oracle._ecg(u_tr, u, coords, 0.25, idx, shape)
    inner = np.argwhere(mesh == 1)
    got = out.cpu().numpy()
    for c in range(n_leads):
        d = ((inner - coords[c, :dim]) ** 2).sum(1) * 0.25
        bound = (np.abs(u_tr - u)[mesh == 1] / d).sum()
        assert abs(got[c] - ref[c]) <= (len(idx) + 8) * 2.3e-16 * bound
