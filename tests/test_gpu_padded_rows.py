"""GPU: fused runs on row-padded copies (rows of no multiple of 16 nodes)
against the same runs on the model's own arrays, bit for bit, with every
tracker, stimuli with masks, odd segment lengths and host writes between
segments; and the argument checks of padded rows."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture()
def env(tmp_path, monkeypatch):
    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for -m gpu tests")
    monkeypatch.setenv("FWGPU_AUTOTUNE_CACHE", str(tmp_path / "tune.json"))
    import finitewave_gb300 as fg
    from finitewave_gb300 import autotune
    autotune._memo.clear()
    yield fg, autotune
    autotune._memo.clear()


def _model(fg, cls, shape, aniso):
    gen = np.random.default_rng(shape[1])
    t = fg.CardiacTissue2D(shape)
    t.mesh = np.where(gen.random(shape) < 0.15, 2, 1).astype(np.int8)
    if aniso:
        a = gen.uniform(-1, 1, shape)
        t.fibers = np.stack([np.cos(a), np.sin(a)], -1)
    m = getattr(fg, cls)()
    m.dt, m.dr, m.npfloat, m.cardiac_tissue = 0.01, 0.25, "float32", t
    seq = fg.StimSequence()
    seq.add_stim(fg.StimVoltageMatrix2D(0, 1.0, gen.random(shape) < 0.2))
    seq.add_stim(fg.StimCurrentCoord2D(0.3, 5.0, 0.05, 0, shape[0] // 2, 0, shape[1]))
    m.stim_sequence = seq
    trs = fg.TrackerSequence()
    for tr in (fg.ActivationTime2DTracker(), fg.LocalActivationTime2DTracker(),
               fg.MultiVariable2DTracker()):
        trs.add_tracker(tr)
    trs.sequence[0].threshold = trs.sequence[1].threshold = 0.5
    trs.sequence[2].cell_ind = [[shape[0] // 2, shape[1] - 2], [0, 0], [3, 4]]
    trs.sequence[2].var_list = ["u", m._state_names[0]]
    m.tracker_sequence = trs
    return m


@pytest.mark.parametrize("choice", [(3, 4), (3, 3), (3, 8), (4, 4)])
@pytest.mark.parametrize("cls,shape,aniso", [
    ("AlievPanfilov2D", (70, 17), True), ("FentonKarma2D", (41, 131), False),
    ("MitchellSchaeffer2D", (133, 257), True), ("Barkley2D", (30, 999), True)])
def test_padded_rows_bits(env, cls, shape, aniso, choice):
    fg, autotune = env
    out = []
    for pad in (True, False):
        m = _model(fg, cls, shape, aniso)
        m.initialize()
        autotune._memo[autotune.key(m)] = {"variant": choice[0], "k": choice[1],
                                           "flat": [1, 4]}
        m.pad_rows = pad
        for steps in (65, 1, 100):       # padded, short, padded
            m.t_max = m.t + (steps - 0.5) * m.dt
            m.run(initialize=False)
            u = m.u
            u[1:4, 1:5] = 0.25 * (np.asarray(m.cardiac_tissue.mesh)[1:4, 1:5] == 1)
        assert (m._pad is not None) == pad
        # (u_new holds an earlier launch's potential, which depends on K)
        out.append([getattr(m, n) for n in ["u"] + list(m._state_names)] +
                   [m.tracker_sequence.sequence[0].output,
                    m.tracker_sequence.sequence[1].output,
                    *m.tracker_sequence.sequence[2].output.values()])
    for a, b in zip(*out):
        assert np.array_equal(a, b)


def test_tuner_times_padded_rows(env):
    fg, autotune = env
    m = _model(fg, "FentonKarma2D", (300, 301), True)
    m.initialize()
    u0 = m.u.copy()
    r = autotune.tune(m)
    assert "3/4" in r["ms"] and "1/4" in r["ms"] and tuple(r["flat"]) in autotune._CPASYNC
    assert np.array_equal(m.u, u0)
    m.pad_rows = False
    assert "3/4" not in autotune.tune(m)["ms"]


def test_pitch_arguments(env):
    fg, _ = env
    m = _model(fg, "AlievPanfilov2D", (40, 33), False)
    m.initialize()
    m.autotune = False
    a = m._bare_args()
    lib = fg._ffi.load()
    for form, variant, pitch in ((fg._ffi.FORM_PLAIN, 0, 48), (fg._ffi.FORM_FUSED, 1, 48),
                                 (fg._ffi.FORM_FUSED, 3, 40), (fg._ffi.FORM_FUSED, 3, 32),
                                 (fg._ffi.FORM_FUSED, 7, 48)):
        a.form, a.fused_variant, a.fused_k, a.pitch = form, variant, 4, pitch
        assert lib.fw_step(ctypes.byref(a), 0, 8, None) != 0
    torch.cuda.synchronize()


@pytest.mark.parametrize("change", ["weights", "no room"])
def test_padded_rows_follow_the_model(env, monkeypatch, change):
    """Weights written in place between two runs are the next run's weights,
    and a device without room for the copies runs on the model's arrays."""
    fg, autotune = env
    from finitewave_gb300 import batch
    out = []
    for pad in (True, False):
        m = _model(fg, "AlievPanfilov2D", (45, 150), True)
        m.pad_rows = pad
        m.initialize()
        autotune._memo[autotune.key(m)] = {"variant": 3, "k": 4, "flat": [1, 4]}
        if pad and change == "no room":
            def no_room(model):
                raise torch.cuda.OutOfMemoryError("no room")
            monkeypatch.setattr(batch, "_Mirror", no_room)
        m.t_max = 0.9
        m.run(initialize=False)
        if change == "weights":
            m.weights.mul_(0.99)
        m.t_max = 1.8
        m.run(initialize=False)
        assert (m._pad is not None) == (pad and change == "weights")
        out.append([m._dev[k].cpu().numpy().copy() for k in ("u", m._state_names[0])])
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("batch", [False, True])
def test_inference_mode(env, batch):
    """Runs under torch.inference_mode(), whose tensors count no writes: the
    same bits as outside it, also after weights written in place."""
    fg, autotune = env
    out = []
    for inference in (True, False):
        with torch.inference_mode(inference):
            m = _model(fg, "MitchellSchaeffer2D", (70, 121), True)
            m.tracker_sequence.sequence.pop()      # a batch takes no probes
            m.initialize()
            autotune._memo[autotune.key(m)] = {"variant": 3, "k": 4, "flat": [1, 4]}
            runner = fg.TissueBatch([m]) if batch else m
            m.t_max = 0.995
            runner.run(initialize=False)
            m.weights.mul_(0.99)
            m.t_max = 1.995
            runner.run(initialize=False)
            out.append([m.u, m.h] + [np.asarray(t.output)
                                     for t in m.tracker_sequence.sequence])
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


def test_padded_copies_end_with_the_model(env):
    """A model that ran on padded copies is freed with its last reference, its
    device memory with it, without the cycle collector; clones and a new
    initialize() start without the copies."""
    import gc
    import weakref
    fg, autotune = env
    gc.collect()
    before = torch.cuda.memory_allocated()
    t = fg.CardiacTissue2D((300, 301))
    m = fg.AlievPanfilov2D()
    m.dt, m.dr, m.npfloat, m.cardiac_tissue = 0.01, 0.25, "float32", t
    m.initialize()
    autotune._memo[autotune.key(m)] = {"variant": 3, "k": 4, "flat": [1, 4]}
    held = torch.cuda.memory_allocated()
    m.t_max = 0.995
    m.run(initialize=False)
    padded = m._pad is not None
    assert padded and torch.cuda.memory_allocated() > held
    c = m.clone()
    bare = getattr(c, "_pad", None) is None
    assert bare
    c.t_max = m.t_max = 1.995
    c.run(initialize=False)
    m.run(initialize=False)
    assert all(torch.equal(c._dev[k], m._dev[k]) for k in ("u", "v"))
    del c
    m.initialize()
    assert torch.cuda.memory_allocated() <= held
    m.t_max = 0.995
    m.run(initialize=False)
    gc.disable()
    try:
        gone = weakref.ref(m)
        del m
        assert gone() is None and torch.cuda.memory_allocated() <= before
    finally:
        gc.enable()


def _fake_times(monkeypatch, autotune, cpasync, tma, copies):
    """A tuner that finds these ms for 96 steps and for the copies."""
    monkeypatch.setattr(autotune, "_time_candidate",
                        lambda model, a, v, k, steps, stream: tma if v in (3, 4) else cpasync)
    monkeypatch.setattr(autotune, "_time_copies", lambda *a: copies)


def test_copies_are_dropped_where_they_lose(env, monkeypatch):
    fg, autotune = env
    m = _model(fg, "AlievPanfilov2D", (60, 77), False)
    m.initialize()
    _fake_times(monkeypatch, autotune, 1.0, 0.8, 0.3)
    m.t_max = 1.195
    m.run(initialize=False)
    assert m._pad is None and m._fused_choice == (1, 2)


def test_copies_from_the_measured_steps(env, monkeypatch):
    """0.5 ms saved in 96 steps make up for copies of 0.4 ms in 77 steps."""
    fg, autotune = env
    m = _model(fg, "AlievPanfilov2D", (60, 77), False)
    m.initialize()
    _fake_times(monkeypatch, autotune, 1.5, 1.0, 0.4)
    assert autotune.choose(m) == (3, 2) and autotune.flat(m) == ((1, 2), 77)
    for steps, padded in ((76, False), (77, True)):
        m._pad = None
        m.t_max = m.t + (steps - 0.5) * m.dt
        m.run(initialize=False)
        assert (m._pad is not None) == padded


def test_choice_without_copies_is_its_own(env, monkeypatch, tmp_path):
    """What a model that may not, or cannot, keep copies was given is not
    what the next model with copies gets."""
    fg, autotune = env
    from finitewave_gb300 import batch
    _fake_times(monkeypatch, autotune, 1.5, 1.0, 0.1)

    def no_room(model):
        raise torch.cuda.OutOfMemoryError("no room")
    for why in ("pad_rows", "no room"):
        autotune._memo.clear()
        monkeypatch.setenv("FWGPU_AUTOTUNE_CACHE", str(tmp_path / (why + ".json")))
        m = _model(fg, "AlievPanfilov2D", (60, 77), False)
        m.initialize()
        with monkeypatch.context() as mp:
            if why == "pad_rows":
                m.pad_rows = False
            else:
                mp.setattr(batch, "_Mirror", no_room)
            assert autotune.choose(m) == (1, 2)
            assert autotune.choose(m) == (1, 2)
        m = _model(fg, "AlievPanfilov2D", (60, 77), False)
        m.initialize()
        assert autotune.choose(m) == (3, 2), why
