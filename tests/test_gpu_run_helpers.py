"""GPU: the helpers around a run's steps -- the comparison of the potential
buffers at non-myocytes and the row copies of the batches -- against torch,
at sizes around their vector widths."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ffi():
    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for -m gpu tests")
    from finitewave_gb300 import _ffi
    return _ffi


def _stream():
    return torch.cuda.current_stream().cuda_stream


@pytest.mark.parametrize("prec", ["float32", "float64"])
@pytest.mark.parametrize("n,offset", [(1, 0), (15, 0), (16, 0), (17, 0), (1000003, 0),
                                      (4099, 1), (4096, 3)])
def test_nonmyo_differ(ffi, prec, n, offset):
    gen = np.random.default_rng(n)
    dt = getattr(torch, prec)
    base = torch.as_tensor((gen.random(n + offset) < 0.5).astype(np.int8), device="cuda")
    myo = base[offset:]
    myo[0] = 0
    u0 = torch.randn(n, dtype=dt, device="cuda")
    u1 = torch.where(myo != 0, u0 + 1, u0)
    code = ffi.F64 if prec == "float64" else ffi.F32

    def differ(a, b):
        flag = torch.zeros(1, dtype=torch.int32, device="cuda")
        ffi.call("fw_nonmyo_differ", myo.data_ptr(), a.data_ptr(), b.data_ptr(), code, n,
                 flag.data_ptr(), _stream())
        return int(flag.item())
    assert differ(u0, u1) == 0
    off = torch.nonzero(myo == 0).view(-1)
    for p in {int(off[0]), int(off[-1]), int(off[len(off) // 2])}:
        v = u1.clone()
        v[p] += 1
        assert differ(u0, v) == 1
        v[p] = float("nan")
        assert differ(v, v) == 1      # NaN is not equal to itself
    z = torch.zeros(n, dtype=dt, device="cuda")
    assert differ(z, -z) == 0


@pytest.mark.parametrize("n_copies", [1, 64, 65, 130])
def test_copy_rows(ffi, n_copies):
    gen = np.random.default_rng(n_copies)
    rows, want, keep = [], [], []
    for i in range(n_copies):
        dt = (torch.float32, torch.uint8)[int(gen.integers(2))]
        b = 4 if dt == torch.float32 else 1
        ni, nj = int(gen.integers(1, 90)), int(gen.integers(1, 200))
        if i % 3 == 0:
            nj = -(-nj // 16) * 16
        ps, pd = nj + int(gen.integers(0, 20)), nj + int(gen.integers(0, 20))
        if i % 5 == 0:
            ps = pd = -(-nj // 16) * 16
        src = torch.randint(0, 200, (ni, ps), device="cuda").to(dt)
        dst = torch.full((ni, pd), 7, device="cuda").to(dt)
        out = dst.clone()
        out[:, :nj] = src[:, :nj]
        rows.append((src.data_ptr(), dst.data_ptr(), ni, nj * b, ps * b, pd * b))
        want.append(out)
        keep.append((src, dst))
    arr = (ffi.Rows * n_copies)(*rows)
    ffi.call("fw_copy_rows", arr, n_copies, _stream())
    for (src, dst), out in zip(keep, want):
        assert torch.equal(dst, out)


def test_bad_arguments(ffi):
    lib = ffi.load()
    t = torch.zeros(64, dtype=torch.int32, device="cuda")
    assert lib.fw_nonmyo_differ(None, t.data_ptr(), t.data_ptr(), ffi.F32, 4,
                                t.data_ptr(), None) == -1
    assert lib.fw_copy_rows(None, 1, None) == -1
    arr = (ffi.Rows * 1)((t.data_ptr(), t.data_ptr() + 128, 2, 16, 8, 16))
    assert lib.fw_copy_rows(arr, 1, None) == -1
    assert lib.fw_copy_rows(None, 0, None) == 0


@pytest.mark.parametrize("kind,nw,centre", [(0, 5, 2), (1, 9, 4)])
@pytest.mark.parametrize("ni,nj", [(1, 1), (3, 17), (40, 255), (5, 1000), (4200, 33)])
def test_pack_rows(ffi, kind, nw, centre, ni, nj):
    kind = (ffi.ISO5, ffi.ANISO9)[kind]
    w = torch.randn((nw, ni, nj), device="cuda")
    pitch = -(-nj // 16) * 16
    out = torch.full((ni, pitch, nw - 1), 9.0, device="cuda")
    cen = torch.full((ni, pitch), 9.0, device="cuda")
    ffi.call("fw_pack_rows", kind, w.data_ptr(), ni, nj, pitch, out.data_ptr(),
             cen.data_ptr(), _stream())
    want = torch.zeros((ni, pitch, nw - 1), device="cuda")
    want[:, :nj] = w[[q for q in range(nw) if q != centre]].permute(1, 2, 0)
    c = torch.zeros((ni, pitch), device="cuda")
    c[:, :nj] = w[centre]
    assert torch.equal(out, want) and torch.equal(cen, c)
