"""GPU: the myocytes-first node list of the plain form (fw_node_list) and
the listed steps against the grid-order steps, bit for bit."""
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


# sizes around the warp, the scan's CTA and its 4096-node chunk
@pytest.mark.parametrize("n", [1, 31, 33, 256, 4095, 4096, 4097, 12289, 2500000])
@pytest.mark.parametrize("p", [0.0, 0.3, 1.0])
def test_node_list(fg, n, p):
    gen = np.random.default_rng(n)
    myo = (gen.random(n) < p).astype(np.int8)
    d = torch.as_tensor(myo, device="cuda")
    out = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    scratch = torch.empty(n // 4096 + 2, dtype=torch.int32, device="cuda")
    fg._ffi.call("fw_node_list", d.data_ptr(), n, out.data_ptr(),
                 scratch.data_ptr(), torch.cuda.current_stream().cuda_stream)
    want = np.concatenate([np.flatnonzero(myo), np.flatnonzero(myo == 0)])
    assert np.array_equal(out.cpu().numpy(), want)


def _model(fg, cls, npfloat, shape, special):
    gen = np.random.default_rng(3)
    tissue = (fg.CardiacTissue2D if len(shape) == 2
              else fg.CardiacTissue3D)(shape)
    tissue.mesh = np.where(gen.random(shape) < 0.25, 2, 1).astype(np.int8)
    if special:
        tissue.special_boundaries = (gen.random(shape) < 0.1).astype(np.int8)
    m = cls()
    m.dt, m.dr, m.t_max, m.npfloat = 0.01, 0.25, 0.2, npfloat
    m.form = "plain"
    m.cardiac_tissue = tissue
    seq = fg.StimSequence()
    box = [b for n in shape for b in (0, n // 2)]
    stim = fg.StimVoltageCoord2D if len(shape) == 2 else fg.StimVoltageCoord3D
    seq.add_stim(stim(0.03, 20.0 if m._model_id in m._DETAILED_MODELS else 1.0,
                      *box))
    m.stim_sequence = seq
    trs = fg.TrackerSequence()
    for t in (fg.ActivationTime2DTracker(), fg.LocalActivationTime2DTracker()):
        # the init potential is above one threshold and below the other, and
        # one tracker starts late, so non-myocytes are tracked as well
        t.threshold = -90.0 if m._model_id in m._DETAILED_MODELS else 0.5
        trs.add_tracker(t)
    trs.sequence[0].start_time = 0.05
    m.tracker_sequence = trs
    return m, trs.sequence


@pytest.mark.parametrize("special", [False, True])
@pytest.mark.parametrize("cls,npfloat,shape", [
    ("AlievPanfilov2D", "float64", (137, 145)), ("FentonKarma3D", "float64", (29, 34, 21)),
    ("TP062D", "float32", (133, 154)), ("Courtemanche3D", "float32", (27, 29, 33)),
    ("LuoRudy912D", "float64", (120, 175))])
def test_listed_steps_equal_grid_order(fg, cls, npfloat, shape, special):
    out = []
    for listed in (True, False):
        m, trs = _model(fg, getattr(fg, cls), npfloat, shape, special)
        m.initialize()
        assert m._nodes is not None
        if not listed:
            m._nodes = None
        m.run(initialize=False)
        out.append([getattr(m, n) for n in ["u", "u_new"] + list(m._state_names)] +
                   [t.output for t in trs])
    for a, b in zip(*out):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("cls,npfloat,shape", [
    ("AlievPanfilov2D", "float64", (141, 150)), ("TP062D", "float32", (141, 150))])
@pytest.mark.parametrize("start,step", [(0, 1), (0.04, 1), (0.03, 2), (0, 3)])
def test_listed_activation_at_non_myocytes(fg, cls, npfloat, shape, start, step):
    """Non-myocytes above the threshold in either potential buffer, trackers
    whose windows open late or skip steps: the activation steps are those of
    grid order."""
    out = []
    for listed in (True, False):
        gen = np.random.default_rng(5)
        t = fg.CardiacTissue2D(shape)
        t.mesh = np.where(gen.random(shape) < 0.3, 2, 1).astype(np.int8)
        m = getattr(fg, cls)()
        m.dt, m.dr, m.npfloat, m.cardiac_tissue = 0.01, 0.25, npfloat, t
        seq = fg.StimSequence()
        seq.add_stim(fg.StimVoltageCoord2D(0.05, 1.0, 20, 90, 20, 90))
        m.stim_sequence = seq
        trs = fg.TrackerSequence()
        for thr in (0.5, 0.8):
            tr = fg.ActivationTime2DTracker()
            tr.threshold = thr
            trs.add_tracker(tr)
        trs.sequence[1].start_time, trs.sequence[1].step = start, step
        m.tracker_sequence = trs
        m.t_max = 0.115
        m.initialize()
        for name in ("u", "u_new"):
            u = m._dev[name]
            r = torch.as_tensor(gen.random(shape), device=u.device, dtype=u.dtype)
            u.copy_(torch.where(m._myo_d.reshape(shape) == 0, r, u))
        if not listed:
            m._nodes = None
        m.run(initialize=False)
        out.append([np.asarray(tr.output) for tr in trs.sequence])
    for a, b in zip(*out):
        assert np.array_equal(a, b) and (a >= 0).any()


@pytest.mark.parametrize("cls,npfloat", [("AlievPanfilov2D", "float64"), ("TP062D", "float32")])
@pytest.mark.parametrize("how", ["in place", "replaced", "inference"])
def test_node_list_follows_the_flags(fg, cls, npfloat, how):
    """Myocyte flags cleared and set between two runs: the steps are those of
    grid order, on a grid that is large enough for the list."""
    out = []
    for listed in (True, False):
        with torch.inference_mode(how == "inference"):
            m, trs = _model(fg, getattr(fg, cls), npfloat, (150, 161), False)
            m.initialize()
            if not listed:
                m._nodes = None
            m.run(initialize=False)
            myo = m._myo_d if how != "replaced" else m._myo_d.clone()
            myo[20:60] = 0
            inner = myo[70:90, 1:-1]
            inner.copy_((torch.arange(inner.numel(), device=myo.device) % 3 > 0)
                        .to(torch.int8).reshape(inner.shape))
            m._myo_d = myo
            m.t_max = 0.4
            m.run(initialize=False)
            out.append([getattr(m, n) for n in ["u", "u_new"] + list(m._state_names)] +
                       [t.output for t in trs])
    for a, b in zip(*out):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("npfloat", ["float64", "float32"])
@pytest.mark.parametrize("shape,share", [((83, 81, 79), 0.05), ((27, 28, 26), 0.0),
                                         ((28, 27, 26), 0.999), ((30, 27, 25), 0.8)])
def test_listed_local_activation_at_non_myocytes(fg, npfloat, shape, share):
    """Local activation trackers at nodes that do not step, few and many (more
    than one round of 152 x 512 threads of four), with values on either side
    of the thresholds in each potential buffer: as in grid order."""
    out = []
    for listed in (True, False):
        gen = np.random.default_rng(7)
        t = fg.CardiacTissue3D(shape)
        t.mesh = np.where(gen.random(shape) < share, 1, 2).astype(np.int8)
        m = fg.TP063D()
        m.dt, m.dr, m.npfloat, m.cardiac_tissue, m.t_max = 0.01, 0.25, npfloat, t, 0.085
        trs = fg.TrackerSequence()
        for cls, thr in ((fg.LocalActivationTime3DTracker, 0.5),
                         (fg.LocalActivationTime3DTracker, 0.2),
                         (fg.ActivationTime3DTracker, 0.7)):
            tr = cls()
            tr.threshold = thr
            trs.add_tracker(tr)
        trs.sequence[1].start_time, trs.sequence[1].step = 0.03, 3
        m.tracker_sequence = trs
        m.initialize()
        for name in ("u", "u_new"):
            u = m._dev[name]
            r = torch.as_tensor(gen.random(shape), device=u.device, dtype=u.dtype)
            u.copy_(torch.where(m._myo_d.reshape(shape) == 0, r, u))
        if not listed:
            m._nodes = None
        m.run(initialize=False)
        out.append([tr._steps.cpu().numpy() for tr in trs.sequence[:2]] +
                   [tr._count.cpu().numpy() for tr in trs.sequence[:2]] +
                   [np.asarray(trs.sequence[2].output), m.u])
    for a, b in zip(*out):
        assert np.array_equal(a, b)
    assert (out[0][2] > 1).any()   # nodes that cross again and again
