"""GPU: both launch forms of the batched TMA kernels -- one kernel for all
groups, and a kernel per group from 64 tiles a CTA on -- against each tissue
run alone in the fused form, bit for bit."""
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


def _model(fg, name, aniso, n, seed, steps):
    gen = np.random.default_rng(seed)
    t = fg.CardiacTissue2D((n, n))
    t.mesh = np.where(gen.random((n, n)) < 0.1, 2, 1).astype(np.int8)
    m = {"ap": fg.AlievPanfilov2D, "ms": fg.MitchellSchaeffer2D,
         "fk": fg.FentonKarma2D}[name]()
    if aniso:
        a = gen.uniform(-1, 1, (n, n))
        t.fibers = np.stack([np.cos(a), np.sin(a)], -1)
    m.dt, m.dr, m.t_max, m.npfloat = 0.01, 0.25, (steps - 0.5) * 0.01, "float32"
    m.cardiac_tissue = t
    m.autotune = False
    seq = fg.StimSequence()
    seq.add_stim(fg.StimVoltageCoord2D(0, 1.0, 0, n, 1, 6))
    seq.add_stim(fg.StimVoltageCoord2D(0.05, 1.0, n // 2, n, 0, n // 2))
    m.stim_sequence = seq
    lat = fg.LocalActivationTime2DTracker()
    lat.threshold, lat.capacity = 0.5, 8
    trs = fg.TrackerSequence()
    trs.add_tracker(lat)
    m.tracker_sequence = trs
    return m


ALL = [("ap", False), ("ap", True), ("ms", False), ("ms", True), ("fk", False), ("fk", True)]


# tiles per group from one to a few hundred, groups missing, an odd step
# count and one launch; then more than 64 tiles a CTA
@pytest.mark.parametrize("kernel", ["tma", "pairs"])
@pytest.mark.parametrize("groups,sizes,steps", [
    (ALL, [20, 57, 130, 64, 33, 300], 21), ([ALL[5]], [24], 3),
    ([ALL[1], ALL[4]], [50, 900], 10), (ALL, [250] * 6, 1),
    (ALL * 2 + ALL[:2], [1000] * 14, 10)])
def test_batch_launch_forms(fg, kernel, groups, sizes, steps):
    def make():
        return [_model(fg, name, aniso, n, i, steps)
                for i, ((name, aniso), n) in enumerate(zip(groups, sizes))]
    got, want = make(), make()
    batch = fg.TissueBatch(got, kernel=kernel)
    batch.run()
    large = batch._batch.n_tiles >= 64 * batch._batch.grid
    assert large == (len(groups) == 14)
    for m, r in zip(got, want):
        r.form = "fused"
        r.run()
        for n in ["u"] + list(m._state_names):
            assert np.array_equal(getattr(m, n), getattr(r, n)), n
        a, b = (x.tracker_sequence.sequence[0] for x in (m, r))
        assert torch.equal(a._count, b._count) and torch.equal(a._activated, b._activated)


@pytest.mark.parametrize("kernel", ["tma", "pairs"])
def test_captured_launches_follow_the_groups(fg, kernel):
    """Tissues exchanged for others of the same sizes: as many tissues and
    tiles, other groups.  The captured launches of the first set are not
    replayed for the second."""
    batch = fg.TissueBatch(kernel=kernel)
    for names in (["ap", "ap", "ms"], ["ap", "ms", "fk"], ["fk", "fk", "fk"]):
        got = [_model(fg, n, True, 130, i, 21) for i, n in enumerate(names)]
        want = [_model(fg, n, True, 130, i, 21) for i, n in enumerate(names)]
        batch.models = got
        batch.run()
        for a, b in zip(got, want):
            b.form = "fused"
            b.run()
            for k in ["u"] + list(a._state_names):
                assert torch.equal(a._dev[k], b._dev[k]), (names, k)


def test_copies_of_models_that_left(fg):
    """A batch whose models are exchanged holds the copies of the present ones
    only."""
    import gc
    batch = fg.TissueBatch(graphs=False)
    held = []
    for seed in range(3):
        m = _model(fg, "ap", True, 500, seed, 3)
        batch.models = [m]
        batch.run()
        del m
        batch.models = []
        gc.collect()
        held.append(torch.cuda.memory_stats()["requested_bytes.all.current"])
    assert held[2] <= held[0] and len(batch._mirrors) == 1
