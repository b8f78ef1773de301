"""GPU: plain steps captured in a CUDA graph -- the overlapped launches of
consecutive steps, the stimuli, probes, ECG samples and tip copies between
them -- against the same call made directly, bit for bit."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _model(fg, cls, npfloat, shape):
    gen = np.random.default_rng(3)
    t = (fg.CardiacTissue2D if len(shape) == 2 else fg.CardiacTissue3D)(shape)
    t.mesh = np.where(gen.random(shape) < 0.2, 2, 1).astype(np.int8)
    m = getattr(fg, cls)()
    m.dt, m.dr, m.npfloat, m.cardiac_tissue, m.t_max = 0.01, 0.25, npfloat, t, 0.195
    m.form = "plain"
    detailed = m._model_id in m._DETAILED_MODELS
    seq = fg.StimSequence()
    box = [b for n in shape for b in (0, n // 2)]
    seq.add_stim((fg.StimVoltageCoord2D if len(shape) == 2 else fg.StimVoltageCoord3D)
                 (0.05, 20.0 if detailed else 1.0, *box))
    m.stim_sequence = seq
    trs = fg.TrackerSequence()
    at, lat, probe = (fg.ActivationTime2DTracker(), fg.LocalActivationTime2DTracker(),
                      fg.MultiVariable2DTracker())
    at.threshold = lat.threshold = -40.0 if detailed else 0.5
    probe.cell_ind = [[5] * len(shape), [9] * len(shape)]
    probe.var_list = ["u", m._state_names[0]]
    ap = fg.ActionPotential2DTracker()
    ap.cell_ind = [[6] * len(shape)]
    for tr in (at, lat, probe, ap):
        trs.add_tracker(tr)
    if len(shape) == 2:
        ecg, tip = fg.ECG2DTracker(), fg.SpiralWaveCore2DTracker()
        ecg.measure_coords = np.array([[5.0, 6.0, 3.0]])
        ecg.step, tip.step, tip.threshold = 3, 2, at.threshold
        trs.add_tracker(ecg)
        trs.add_tracker(tip)
    m.tracker_sequence = trs
    return m


@pytest.mark.parametrize("cls,npfloat,shape", [
    ("AlievPanfilov2D", "float64", (60, 70)), ("AlievPanfilov2D", "float64", (141, 150)),
    ("TP062D", "float32", (141, 150)), ("FentonKarma2D", "float32", (60, 70)),
    ("Courtemanche3D", "float64", (27, 29, 31))])
def test_captured_steps(cls, npfloat, shape):
    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for -m gpu tests")
    import finitewave_gb300 as fg
    out = []
    for captured in (True, False):
        m = _model(fg, cls, npfloat, shape)
        m.initialize()
        m._nonmyo_equal = None
        seg = m._prepare_segment(1000)
        assert seg.n_seg == 20

        def steps(stream):
            fg._ffi.call("fw_step", ctypes.byref(seg.args), seg.n0, seg.n_seg,
                         stream.cuda_stream)
        if captured:
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g):
                steps(torch.cuda.current_stream())
            g.replay()
        else:
            steps(torch.cuda.current_stream())
        m._finish_segment(seg)
        torch.cuda.synchronize()
        m._check_status()
        trs = m.tracker_sequence.sequence
        r = {n: m._dev[n].cpu().numpy() for n in ["u", "u_new"] + list(m._state_names)}
        r.update(at=trs[0].output, lat=trs[1]._count.cpu().numpy(), ap=trs[3].output)
        r.update({"probe " + k: v for k, v in trs[2].output.items()})
        if len(trs) > 4:
            r["ecg"] = trs[4].output
            r["tip"] = trs[5]._u_prev.cpu().numpy()
        out.append(r)
    for k in out[1]:
        a, b = np.asarray(out[0][k]), np.asarray(out[1][k])
        if k == "ecg":      # one float64 atomic sum a CTA, in any order
            assert np.allclose(a, b, rtol=1e-9, atol=1e-12)
        else:
            assert np.array_equal(a, b), k
